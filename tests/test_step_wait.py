"""The host's wait for a step's result: bounded polling, then a stream
synchronisation; none of it polls under a schedule flag that asks for blocking
or yielding.  The logic against fakes of the CUDA calls; on the GPU, the
processor time of long steps under cudaDeviceScheduleBlockingSync, and more
solver threads than a process has cores to poll on."""
import os
import shutil
import subprocess
import sys

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "finess_b200", "csrc")
CUDA_INC = os.path.join(os.environ.get("CUDA_HOME", "/usr/local/cuda"), "include")

SRC = r"""
#include <cstdio>
#include "fin_wait.h"
static volatile unsigned long long num;
static unsigned flags;
static int syncs;
static cudaError_t sync_result, flag_result;
static unsigned long long set_in_sync;
extern "C" cudaError_t cudaGetDeviceFlags(unsigned* f) { *f = flags; return flag_result; }
extern "C" cudaError_t cudaStreamSynchronize(cudaStream_t)
{
    syncs++;
    if (set_in_sync) num = set_in_sync;
    return sync_result;
}
static double wait(unsigned long long seq, cudaError_t& e, bool& there)
{
    there = false;
    const auto t = std::chrono::steady_clock::now();
    e = fin::wait_number(&num, seq, nullptr, &there);
    return std::chrono::duration<double>(std::chrono::steady_clock::now() - t).count();
}
#define CHECK(c) if (!(c)) { printf("line %d: %s\n", __LINE__, #c); return 1; }
int main()
{
    cudaError_t e;
    bool there;
    num = 7;
    wait(7, e, there);
    CHECK(e == cudaSuccess && there && syncs == 0);              // already there: no call waits
    set_in_sync = 8;   // should the thread come late
    std::thread later([] { std::this_thread::sleep_for(std::chrono::microseconds(20)); num = 8; });
    wait(8, e, there);
    later.join();
    CHECK(e == cudaSuccess && there);
    syncs = 0;
    set_in_sync = 9;
    const double s = wait(9, e, there);
    CHECK(e == cudaSuccess && there && syncs == 1 && s >= 1e-3 && s < 1.0);   // a long wait is the runtime's
    for (unsigned f : {unsigned(cudaDeviceScheduleBlockingSync), unsigned(cudaDeviceScheduleYield)}) {
        flags = f | cudaDeviceMapHost;
        syncs = 0;
        num = 10;
        set_in_sync = 0;
        wait(10, e, there);
        CHECK(e == cudaSuccess && there && syncs == 1);          // asked for: no polling at all
    }
    flags = 0;
    syncs = 0;
    wait(11, e, there);
    CHECK(e == cudaSuccess && !there && syncs == 1);             // the stream ended without the number
    sync_result = cudaErrorLaunchFailure;
    wait(12, e, there);
    CHECK(e == cudaErrorLaunchFailure && !there);                // its error
    flag_result = cudaErrorInvalidDevice;
    syncs = 0;
    wait(13, e, there);
    CHECK(e == cudaErrorInvalidDevice && !there && syncs == 0);
    return 0;
}
"""


@pytest.mark.skipif(not shutil.which("g++") or not os.path.isdir(CUDA_INC), reason="needs g++ and CUDA headers")
def test_wait_logic(tmp_path):
    src, exe = tmp_path / "w.cpp", tmp_path / "w"
    src.write_text(SRC)
    subprocess.check_call(["g++", "-std=c++17", "-O2", "-pthread", "-I" + CSRC, "-I" + CUDA_INC, "-o", str(exe), str(src)])
    subprocess.check_call([str(exe)], timeout=60)


BLOCKING = r"""
import ctypes as C, sys, time
sys.path.insert(0, sys.argv[1])
cu = C.CDLL("libcuda.so.1")
assert cu.cuInit(0) == 0 and cu.cuDevicePrimaryCtxSetFlags_v2(0, 4) == 0   # CU_CTX_SCHED_BLOCKING_SYNC
import numpy as np
from finess_b200 import problems as P
from finess_b200.solver import Solver
from finess_b200.mhd import MhdSolver
p = P.riemann_params(n=3000)
pm = P.orszag_tang_params(n=1400)
with Solver(p) as s, MhdSolver(pm) as m:
    s.set_state(P.riemann_init(p))
    m.set_state(*P.mhd_random_state(pm, np.random.default_rng(1)))
    for f in (lambda: s.step_fixed(1e-7), lambda: m.step_fixed(1e-7)):
        f()
        w, c = time.perf_counter(), time.process_time()
        for _ in range(60):
            f()
        w, c = time.perf_counter() - w, time.process_time() - c
        print(c / w)
        assert c < 0.5 * w, (c, w)
"""


@pytest.mark.gpu
def test_long_steps_block_when_asked_to():
    """Steps of 2 to 4 ms: the caller sleeps most of the time (it polled all of it)."""
    r = subprocess.run([sys.executable, "-c", BLOCKING, ROOT], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stdout + r.stderr[-2000:]


@pytest.mark.gpu
def test_many_solver_threads():
    """Twice as many threads as cores (at least 16), a solver each: all end, with
    the states of a single thread."""
    import threading

    import numpy as np

    from finess_b200 import problems as P
    from finess_b200.solver import Solver
    p = P.riemann_params(n=64)
    q = P.random_riemann_state(p, np.random.default_rng(1))
    n = max(16, min(64, 2 * (os.cpu_count() or 8)))
    out = [None] * n

    def run(k):
        with Solver(p) as s:
            s.set_state(q)
            for _ in range(50):
                s.step_fixed(1e-4)
            out[k] = s.get_state()[0]

    t = [threading.Thread(target=run, args=(k,)) for k in range(n)]
    for x in t:
        x.start()
    for x in t:
        x.join(timeout=120)
    assert all(o is not None and np.array_equal(o, out[0]) for o in out)
