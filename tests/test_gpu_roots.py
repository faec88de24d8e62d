"""Error bounds and edge cases of fin_device.cuh's sqrt_fast and rsqrt_fast,
against roots in extended precision and CUDA's correctly rounded square root.

FP64 rsqrt_fast is one third-order step y (1 + e/2 + 3 e^2/8) from an
approximation y of relative error 2^-22: the series' rest, 5/16 e^3 with e up to
2^-21, is below 2^-64; e = 1 - x y y comes from the rounded product x y and so is
off by 2^-53, half of which reaches the result; the last fma rounds once, 2^-53.
Sum 1.5 * 2^-53.  sqrt_fast multiplies by x and rounds once more: 2.5 * 2^-53.
FP32 takes the hardware approximations, 2^-22 of the value."""
import ctypes as C
import os

import numpy as np
import pytest

from conftest import ROOT
from finess_b200 import problems as P
from finess_b200._abi import FIN_OK

pytestmark = pytest.mark.gpu
F64 = np.ctypeslib.ndpointer(dtype=np.float64, flags="C_CONTIGUOUS")


def _roots(x):
    """sqrt_fast, rsqrt_fast, __dsqrt_rn, FP32 sqrt_fast, FP32 rsqrt_fast of x."""
    lib = C.CDLL(os.path.join(ROOT, "tests", "apps", "libfin_phys_app.so"))
    lib.app_root_probe.argtypes = [F64, F64, C.c_int]
    x = np.ascontiguousarray(x, dtype=np.float64)
    out = np.zeros((5, x.size))
    assert lib.app_root_probe(x, out, x.size) == FIN_OK
    return out


def test_root_edge_cases():
    """A NaN of either sign and every negative number (but the zeros and the
    subnormals, which count as zero) give NaN, so that no speed of a failed
    state turns into a finite one."""
    bits = [0x7ff8000000000000, 0xfff8000000000000, 0x7ff0000000000001, 0xffffffffffffffff]
    nan = np.array(bits, dtype=np.uint64).view(np.float64)
    neg = np.array([-1.0, -1e-300, -1e300, -2.0 ** -1022, -np.inf])
    for bad in (nan, neg):
        s, r, _, s32, r32 = _roots(bad)
        assert np.all(np.isnan(s)), s
        assert np.all(np.isnan(r)), r
    s, _, _, s32, _ = _roots(np.concatenate([nan, [-1.0, -np.inf]]))
    assert np.all(np.isnan(s32))
    s, r, _, s32, _ = _roots([0.0, -0.0, 2.0 ** -1074, -2.0 ** -1074, 2.0 ** -1023])
    assert np.all(s == 0.0) and np.all(s32 == 0.0) and not np.any(np.isfinite(r))
    s, _, _, _, _ = _roots([np.inf])
    assert not np.isfinite(s[0])


@pytest.mark.skipif(np.finfo(np.longdouble).nmant < 63, reason="no extended precision on this host")
def test_root_error_bounds():
    rng = np.random.default_rng(12)
    e = rng.integers(-1000, 1000, 400000)
    x = np.ldexp(rng.uniform(1.0, 2.0, e.size), e)
    x = np.concatenate([x, [1.0, 2.0, 3.0, 4.0, 0.25, 1.4, 1e-300, 7e300, 2.0 ** -1022, 2.0 ** 1023],
                        np.nextafter(np.ldexp(1.0, np.arange(-40, 40)), 0), np.nextafter(np.ldexp(1.0, np.arange(-40, 40)), np.inf)])
    s, r, cuda, s32, r32 = _roots(x)
    root = np.sqrt(x.astype(np.longdouble))
    assert np.array_equal(cuda, np.sqrt(x))
    u, slack = 2.0 ** -53, 2.0 ** -62
    assert np.max(np.abs(r * root - 1)) <= 1.5 * u + slack
    assert np.max(np.abs(s / root - 1)) <= 2.5 * u + slack
    ok = (x > 1e-30) & (x < 1e30)
    root32 = np.sqrt(x[ok].astype(np.float32).astype(np.longdouble))
    assert np.max(np.abs(s32[ok] / root32 - 1)) <= 2.0 ** -22
    assert np.max(np.abs(r32[ok] * root32 - 1)) <= 2.0 ** -22


BAD = [np.uint64(b).view(np.float64) for b in (0x7ff8000000000000, 0xfff8000000000000)] + [np.inf, -np.inf]


@pytest.mark.parametrize("ga", [0, 1])
@pytest.mark.parametrize("m", range(5))
def test_euler_construct_l_reports_non_finite_states(oracle, m, ga):
    from finess_b200.solver import Solver
    p = P.riemann_params(n=33, global_alpha=ga)
    q = oracle.set_bnd(p, P.random_riemann_state(p, np.random.default_rng(m)))
    with Solver(p) as s:
        for bad in BAD:
            b = q.copy()
            b[p.mbc + 17, p.mbc + 5 + m, m] = bad
            with pytest.raises(RuntimeError, match="non-finite"):
                s.ConstructL(b)
        s.ConstructL(q)


@pytest.mark.parametrize("ga", [0, 1])
@pytest.mark.parametrize("m", range(8))
def test_mhd_construct_l_reports_non_finite_states(oracle, m, ga):
    from finess_b200.mhd import MhdSolver
    p = P.orszag_tang_params(n=33, global_alpha=ga)
    q, aux = oracle.mhd_set_bnd(p, *P.mhd_random_state(p, np.random.default_rng(m)))
    with MhdSolver(p) as s:
        for bad in BAD:
            b = q.copy()
            b[p.mbc + 17, p.mbc + 5 + m, m] = bad
            with pytest.raises(RuntimeError, match="non-finite"):
                s.ConstructL(b, aux)
        s.ConstructL(q, aux)
