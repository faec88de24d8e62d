"""The dynamic shared memory of a kernel is granted once per solver (and so on
each device and in each context a solver is made in), not once per process: the
grant's bookkeeping against a fake of cudaFuncSetAttribute."""
import os
import shutil
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "finess_b200", "csrc")
CUDA_INC = os.path.join(os.environ.get("CUDA_HOME", "/usr/local/cuda"), "include")

SRC = r"""
#include <cstdio>
#include <cstring>
#include "fin_smem.h"
static int calls, fail;
static const void* last;
static int bytes;
extern "C" cudaError_t cudaFuncSetAttribute(const void* f, cudaFuncAttribute, int v)
{
    calls++; last = f; bytes = v;
    return fail ? cudaErrorInvalidValue : cudaSuccess;
}
template <int N> void kern(int) {}
template <int N> void many(fin::SmemGrants& g) { if constexpr (N > 0) { g.allow(kern<N>, 1000 + N); many<N - 1>(g); } }
#define CHECK(c) if (!(c)) { printf("line %d: %s\n", __LINE__, #c); return 1; }
int main()
{
    fin::SmemGrants a, b;
    memset(&a, 0, sizeof a);
    memset(&b, 0, sizeof b);
    CHECK(a.allow(kern<1>, 50000) == cudaSuccess && calls == 1 && bytes == 50000 && last == (const void*)kern<1>);
    CHECK(a.allow(kern<1>, 50000) == cudaSuccess && calls == 1);     // once a solver
    CHECK(a.allow(kern<2>, 60000) == cudaSuccess && calls == 2);     // each kernel
    CHECK(b.allow(kern<1>, 50000) == cudaSuccess && calls == 3);     // another solver: again
    fail = 1;
    CHECK(b.allow(kern<3>, 50000) == cudaErrorInvalidValue && calls == 4);
    fail = 0;
    CHECK(b.allow(kern<3>, 50000) == cudaSuccess && calls == 5);     // a refusal is not remembered
    calls = 0;
    memset(&a, 0, sizeof a);
    many<12>(a);
    CHECK(calls == 12);
    many<12>(a);
    CHECK(calls == 12 + 4);                                          // the last four of twelve are not held
    return 0;
}
"""


@pytest.mark.skipif(not shutil.which("g++") or not os.path.isdir(CUDA_INC), reason="needs g++ and CUDA headers")
def test_grants(tmp_path):
    src, exe = tmp_path / "g.cpp", tmp_path / "g"
    src.write_text(SRC)
    subprocess.check_call(["g++", "-std=c++17", "-I" + CSRC, "-I" + CUDA_INC, "-o", str(exe), str(src)])
    subprocess.check_call([str(exe)])


def test_no_grant_is_process_wide():
    """Solvers' launches hold no static flag about an attribute."""
    import re
    for f in ("finess_b200.cu", "fin_mhd.cu", "fin_hi.cu"):
        with open(os.path.join(CSRC, f)) as h:
            assert not re.search(r"static bool\s+\w+\s*=\s*false", h.read()), f
