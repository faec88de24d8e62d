"""Performance cases: the steps of a finite-difference WENO run as a program takes them.

A case names a path (the Euler steppers, one ConstructL call on host arrays, a
batch of uneven problems, ideal MHD), a grid and the number of accepted steps
of one pass.  ``prepare`` builds the solver and loads its first state, as a
program does once per run; ``run`` advances it by ``steps`` adaptive steps
through the public entry points and returns the whole state.  A pass goes on
from where the last one stopped, as a run does between two frames.

The states hold what a run meets after its first moments: smooth waves over
the whole domain, jumps (a bubble and a quarter plane of other density and
pressure), and a tenth of the domain with waves about ten cells long (the
compressed entropy waves and rolled-up contacts of the benchmark problems),
so that the learned indicator has smooth, troubled and marginal faces.

FP64 forms return the FP64 state where it lies on the device.  The FP32 and
hybrid forms compute in FP32: a program that picks them takes its fields in
float32, so those cases end with that copy.
"""
import ctypes as C
import math
from fractions import Fraction

import numpy as np
import torch

from finess_b200 import batch as B
from finess_b200 import _abi as A
from finess_b200.indicator import DEFAULT_MHD_WEIGHTS, DEFAULT_WEIGHTS
from finess_b200.mhd import MhdSolver
from finess_b200.solver import Solver

F64 = torch.float64
WENO = {"JS": A.FIN_WENO_JS, "Z": A.FIN_WENO_Z, "FD": A.FIN_WENO_FD}
PREC = {"fp64": A.FIN_PREC_FP64, "fp32": A.FIN_PREC_FP32, "hybrid": A.FIN_PREC_HYBRID}
METHOD = {"rk": A.FIN_TS_RK, "md": A.FIN_TS_MD, "lxw": A.FIN_TS_LXW}
BC = {"periodic": A.FIN_BC_PERIODIC, "transmissive": A.FIN_BC_TRANSMISSIVE}
# the benchmark's hybrid schedule: the indicator every 2nd step, a judge step every 50th
HYB_EVERY, HYB_JUDGE, HYB_TOL = 2, 50, 1e-3


def _euler(name, mx, my, steps, prec="fp64", weno="Z", method="rk", order=5, time_order=3, bcx="transmissive",
           bcy="transmissive", mpp=False, global_alpha=True):
    c = {"kind": "euler", "mx": mx, "my": my, "steps": steps, "prec": prec, "weno": weno, "method": method,
         "order": order, "time_order": time_order, "bcx": bcx, "bcy": bcy, "mpp": mpp, "global_alpha": global_alpha}
    return dict(c, name=name) if name else c


def listed():
    return [
        # one right-hand side on host arrays: what an application relinked against the building blocks asks
        # for at every stage of its own stepper
        {"name": "construct_l_host_300x257", "kind": "construct_l", "mx": 300, "my": 257, "weno": "JS",
         "global_alpha": True},
        # the smallest grids of a parameter sweep, run one at a time
        _euler("sweep_96x80_fp64", 96, 80, 20),
        # the isentropic vortex of the accuracy benchmark
        _euler("vortex_200_fp64", 200, 200, 20, weno="JS", bcx="periodic", bcy="periodic"),
        # the headline problem's size in the parity form and in the hybrid form
        _euler("riemann_4096_fp64", 4096, 4096, 1),
        _euler("riemann_4096_hybrid", 4096, 4096, 8, prec="hybrid"),
        # the shock / entropy-wave problem's shape (long, periodic in y) at an odd size, FP32 bulk
        _euler("shock_entropy_4001x515_fp32", 4001, 515, 2, prec="fp32", weno="JS", bcy="periodic"),
        # two-stage multiderivative steps of order 4
        _euler("multiderivative_1024x1000", 1024, 1000, 2, method="md", time_order=4),
        # Lax-Wendroff with the positivity limiter on a near-vacuum flow
        _euler("lxw_mpp_1023x1025", 1023, 1025, 2, method="lxw", mpp=True),
        # seventh-order space
        _euler("weno7_js_1024", 1024, 1024, 2, weno="JS", order=7, bcx="periodic", bcy="periodic"),
        # the uneven sweep, batched: many problems of unequal size to one end time
        {"name": "batch_48_hybrid", "kind": "batch", "problems": 48, "nmin": 64, "nmax": 512, "grid_seed": 7,
         "prec": "hybrid", "dt_total": 0.04},
        # ideal MHD with constrained transport, parity form and hybrid form
        {"name": "mhd_1024_fp64", "kind": "mhd", "mx": 1024, "my": 1024, "steps": 2, "prec": "fp64", "weno": "JS"},
        {"name": "mhd_1024_hybrid", "kind": "mhd", "mx": 1024, "my": 1024, "steps": 4, "prec": "hybrid", "weno": "JS"},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _grid(rng, lo, hi, cells):
    """An uneven grid of at most `cells` cells."""
    mx = _log_int(rng, lo, hi)
    return mx, min(_log_int(rng, lo, hi), max(lo, cells // mx))


def draw(rng):
    kind = rng.choice(["rk", "rk", "rk", "fp32", "hybrid", "hybrid", "lw", "order", "construct_l", "batch", "mhd"])
    bcx, bcy = rng.choice(["periodic", "transmissive"]), rng.choice(["periodic", "transmissive"])
    if kind in ("rk", "fp32", "hybrid"):
        mx, my = _grid(rng, 64, 4096, 1 << 23 if kind == "rk" else 1 << 24)
        steps = max(1, min(20, int((2.4e7 if kind == "rk" else 6e7) / (mx * my))))
        return _euler(None, mx, my, steps, prec="fp64" if kind == "rk" else kind, weno=rng.choice(["JS", "Z"]),
                      time_order=rng.choice([3, 3, 2, 4]) if kind == "rk" and steps > 4 else 3, bcx=bcx, bcy=bcy,
                      global_alpha=rng.choice([True, False]))
    if kind == "lw":
        mx, my = _grid(rng, 96, 3000, 1 << 21)
        method = rng.choice(["md", "lxw"])
        return _euler(None, mx, my, max(1, min(8, int(3e6 / (mx * my)))), weno=rng.choice(["JS", "Z"]), method=method,
                      time_order=4 if method == "md" else 3, mpp=method == "lxw" and rng.random() < 0.6, bcx=bcx, bcy=bcy)
    if kind == "order":
        mx, my = _grid(rng, 96, 2048, 1 << 21)
        return _euler(None, mx, my, max(1, min(6, int(3e6 / (mx * my)))), weno=rng.choice(["JS", "Z"]),
                      order=rng.choice([7, 7, 9]), bcx=bcx, bcy=bcy)
    if kind == "construct_l":
        mx, my = _grid(rng, 64, 1024, 1 << 19)
        return {"kind": "construct_l", "mx": mx, "my": my, "weno": rng.choice(["JS", "Z"]),
                "global_alpha": rng.choice([True, False])}
    if kind == "batch":
        return {"kind": "batch", "problems": rng.randint(8, 48), "nmin": 64, "nmax": _log_int(rng, 128, 512),
                "grid_seed": rng.randint(0, 1 << 20), "prec": rng.choice(["hybrid", "fp32", "fp64"]),
                "dt_total": 0.01}
    mx, my = _grid(rng, 96, 1536, 1 << 20)
    prec = rng.choice(["fp64", "fp32", "hybrid"])
    return {"kind": "mhd", "mx": mx, "my": my, "steps": max(1, min(6, int(2.5e6 / (mx * my)))), "prec": prec,
            "weno": rng.choice(["JS", "Z"])}


# ---- inputs ---------------------------------------------------------------

def _params(case):
    if case["kind"] == "mhd":
        return A.default_params(mx=case["mx"], my=case["my"], mbc=7, meqn=8, maux=1, xhigh=2 * math.pi, yhigh=2 * math.pi,
                                weno_version=WENO[case["weno"]], gamma=5.0 / 3.0, physics=A.FIN_PHYS_MHD,
                                precision=PREC[case["prec"]])
    if case["kind"] == "construct_l":
        case = dict(_euler(None, case["mx"], case["my"], 1, weno=case["weno"]), global_alpha=case["global_alpha"])
    bx, by = BC[case["bcx"]], BC[case["bcy"]]
    return A.default_params(mx=case["mx"], my=case["my"], mbc=5, xhigh=1.0, yhigh=case["my"] / case["mx"],
                            weno_version=WENO[case["weno"]], global_alpha=int(case["global_alpha"]),
                            space_order=case["order"], time_order=case["time_order"],
                            time_stepping_method=METHOD[case["method"]], mpp_limiter=int(case["mpp"]),
                            precision=PREC[case["prec"]], bc_xlow=bx, bc_xhigh=bx, bc_ylow=by, bc_yhigh=by,
                            # single-stage Lax-Wendroff and the two-stage methods step at smaller CFL numbers
                            desired_cfl=0.2 if case["method"] == "lxw" else 0.4,
                            max_cfl=0.25 if case["method"] == "lxw" else 0.45)


def _mesh(mx, my, gen):
    x = ((torch.arange(mx, dtype=F64, device="cuda") + 0.5) / mx)[:, None]
    y = ((torch.arange(my, dtype=F64, device="cuda") + 0.5) / my)[None, :]
    r = (torch.rand(64, generator=gen, dtype=F64)).tolist()
    return x, y, r


def _waves(x, y, r, k):
    """Three random plane waves of 1 to 6 periods, amplitude at most 1 in sum."""
    out = 0.0
    for n in range(3):
        a, b = 1 + int(3 * r[k + 3 * n]), 1 + int(3 * r[k + 3 * n + 1])
        out = out + torch.sin(2 * math.pi * (a * (n + 1) * x + b * y + r[k + 3 * n + 2])) / 3.0
    return out


def _rough(x, y, mx, my, r, k):
    """Waves about ten cells long inside a disc of a tenth of the domain."""
    inside = ((x - 0.3 - 0.4 * r[k]) ** 2 + (y - 0.3 - 0.4 * r[k + 1]) ** 2) < 0.032
    w = torch.sin(2 * math.pi * (x * mx / 9.3 + r[k + 2])) * torch.sin(2 * math.pi * (y * my / 10.7 + r[k + 3]))
    return torch.where(inside, w, torch.zeros((), dtype=F64, device="cuda"))


def _euler_state(mx, my, gamma, seed, vacuum=False):
    """Conserved interior planes (5, mx, my)."""
    gen = torch.Generator().manual_seed(int(seed))
    x, y, r = _mesh(mx, my, gen)
    rho = 1.0 + 0.25 * _waves(x, y, r, 0)
    u = 0.3 + 0.3 * _waves(x, y, r, 9)
    v = -0.2 + 0.3 * _waves(x, y, r, 18)
    p = 1.0 + 0.25 * _waves(x, y, r, 27)
    if vacuum:
        # two rarefactions moving apart: density and pressure close to zero between them
        u = torch.where(x < 0.5, -1.9, 1.9) + 0.1 * u
        p = 0.4 * p
    else:
        quarter = (x > 0.6 + 0.2 * r[40]) & (y > 0.6 + 0.2 * r[41])
        rho, p = torch.where(quarter, 0.6 * rho, rho), torch.where(quarter, 0.5 * p, p)
        bubble = ((x - 0.2 - 0.2 * r[42]) ** 2 + (y - 0.2 - 0.2 * r[43]) ** 2) < 0.01
        rho, p = torch.where(bubble, 1.8 * rho, rho), torch.where(bubble, 2.0 * p, p)
        rho = rho * (1.0 + 0.12 * _rough(x, y, mx, my, r, 44))
        u = u + 0.1 * _rough(x, y, mx, my, r, 50)
    u, v = u + 0.0 * rho, v + 0.0 * rho
    return torch.stack([rho, rho * u, rho * v, 0.0 * rho, p / (gamma - 1.0) + 0.5 * rho * (u * u + v * v)])


def _d4(a, axis, h):
    """4th-order central difference on a periodic grid (constrained transport's)."""
    return (torch.roll(a, 2, axis) - 8 * torch.roll(a, 1, axis) + 8 * torch.roll(a, -1, axis)
            - torch.roll(a, -2, axis)) * (1.0 / (12.0 * h))


def _mhd_state(mx, my, gamma, seed):
    """Conserved interior planes (8, mx, my) and the potential A3 whose curl is (B1, B2)."""
    gen = torch.Generator().manual_seed(int(seed))
    x, y, r = _mesh(mx, my, gen)
    rho = 1.4 + 0.4 * _waves(x, y, r, 0)
    u1, u2 = 0.5 * _waves(x, y, r, 9), 0.5 * _waves(x, y, r, 18)
    u3 = 0.1 * torch.sin(2 * math.pi * (x + r[30])) + 0.0 * y
    p = 1.6 + 0.4 * _waves(x, y, r, 27)
    rho = rho * (1.0 + 0.08 * _rough(x, y, mx, my, r, 44))
    # whole periods in y, so that the patch's cut edge is a jump of density only
    a3 = (0.5 * torch.cos(2 * math.pi * (2 * x + r[50])) + torch.cos(2 * math.pi * (y + r[51]))
          + 0.2 * torch.sin(2 * math.pi * (x + 2 * y + r[52])))
    h = (2 * math.pi / mx, 2 * math.pi / my)
    b1, b2 = _d4(a3, 1, h[1]), -_d4(a3, 0, h[0])
    b3 = 0.3 + 0.1 * torch.cos(2 * math.pi * (y + r[53])) + 0.0 * x
    e = p / (gamma - 1.0) + 0.5 * rho * (u1 * u1 + u2 * u2 + u3 * u3) + 0.5 * (b1 * b1 + b2 * b2 + b3 * b3)
    return torch.stack([rho, rho * u1, rho * u2, rho * u3, e, b1, b2, b3]), a3


def _index(n, halo, periodic):
    i = torch.arange(-halo, n + halo, device="cuda")
    return i % n if periodic else i.clamp(0, n - 1)


def _ghosted(q, halo, px, py):
    """Planes (m, mx, my) -> the same with `halo` ghost cells filled by the boundary conditions."""
    return q[:, _index(q.shape[1], halo, px)][:, :, _index(q.shape[2], halo, py)]


def _host(q, p):
    """The reference's ghosted (i, j, m) host array of interior planes."""
    g = _ghosted(q, p.mbc, p.bc_xlow == A.FIN_BC_PERIODIC, p.bc_ylow == A.FIN_BC_PERIODIC)
    return g.permute(1, 2, 0).contiguous().cpu().numpy()


def _first_dt(p, q):
    """desired_cfl min(dx, dy) / max wave speed."""
    ax, ay = (float(s.max()) for s in _cell_speeds(q, p.gamma))
    return p.desired_cfl * min((p.xhigh - p.xlow) / p.mx, (p.yhigh - p.ylow) / p.my) / max(ax, ay)


def _mhd_first_dt(p, q):
    s = max(float(_mhd_speed(q, q, n, p.gamma).max()) for n in (1, 2))
    return p.desired_cfl / (s * (p.mx / (p.xhigh - p.xlow) + p.my / (p.yhigh - p.ylow)))


def _sizes(case):
    rng = np.random.default_rng(case["grid_seed"])
    lo, hi = math.log(case["nmin"]), math.log(case["nmax"])
    return [int(round(math.exp(rng.uniform(lo, hi)))) for _ in range(case["problems"])]


def _batch_problem(case, k, n, seed):
    c = _euler(None, n, n, 1, prec=case["prec"])
    p = _params(c)
    return p, _euler_state(n, n, p.gamma, 1000003 * int(seed) + k)


def prepare(case, seed):
    if case["kind"] == "batch":
        probs = [_batch_problem(case, k, n, seed) for k, n in enumerate(_sizes(case))]
        b = B.Batch([p for p, _ in probs])
        if case["prec"] == "hybrid":
            W = np.load(DEFAULT_WEIGHTS)
            b.set_indicator(W["params"], float(W["z_threshold"]), HYB_JUDGE, HYB_TOL, HYB_EVERY)
        for k, (p, q) in enumerate(probs):
            b.set_state(k, _host(q, p))
        return {"case": case, "b": b, "dt": np.array([_first_dt(p, q) for p, q in probs]), "t": 0.0}
    p = _params(case)
    if case["kind"] == "mhd":
        q, a3 = _mhd_state(p.mx, p.my, p.gamma, seed)
        s = MhdSolver(p)
        if case["prec"] == "hybrid":
            W = np.load(DEFAULT_MHD_WEIGHTS)
            s.set_indicator(W["params"], float(W["z_threshold"]), HYB_JUDGE, HYB_TOL, HYB_EVERY)
        s.set_state(_host(q, p), _host(a3[None], p))
        return {"case": case, "s": s, "dtv": np.array([0.0, _mhd_first_dt(p, q), p.max_dt])}
    q = _euler_state(p.mx, p.my, p.gamma, seed, vacuum=bool(case.get("mpp")))
    s = Solver(p)
    if case["kind"] == "construct_l":
        return {"case": case, "s": s, "q": _host(q, p)}
    if case["prec"] == "hybrid":
        W = np.load(DEFAULT_WEIGHTS)
        s.set_indicator(W["params"], float(W["z_threshold"]), HYB_JUDGE, HYB_TOL, HYB_EVERY)
    s.set_state(_host(q, p))
    return {"case": case, "s": s, "dtv": np.array([0.0, _first_dt(p, q), p.max_dt])}


# ---- one pass -------------------------------------------------------------

class _DeviceArray:
    """A device buffer of the library as torch.as_tensor reads it (no copy);
    the tensor keeps this object, and with it the buffer's owner."""

    def __init__(self, owner, ptr, shape, strides):
        self.owner = owner
        self.__cuda_array_interface__ = {"data": (ptr, False), "shape": shape, "typestr": "<f8", "version": 3,
                                         "strides": tuple(8 * s for s in strides)}


def _state_view(s, mhd):
    ptr, plane = C.c_void_p(), C.c_size_t()
    p = s.p
    if mhd:   # the potential A3 is the ninth plane
        s._check(s.lib.fin_mhd_device_state(s.h, C.byref(ptr), C.byref(plane)))
    else:
        row = C.c_size_t()
        s.lib.fin_state_device_ptr(s.h, C.byref(ptr))
        s.lib.fin_device_layout(s.h, C.byref(plane), C.byref(row))
    m = 9 if mhd else 5
    return torch.as_tensor(_DeviceArray(s, ptr.value, (m, p.mx, p.my), (plane.value, p.my, 1)), device="cuda")


def run(state):
    case = state["case"]
    if case["kind"] == "construct_l":
        L, smax = state["s"].ConstructL(state["q"])
        return {"L": L, "smax": smax}
    if case["kind"] == "batch":
        state["t"] += case["dt_total"]
        state["dt"], steps = state["b"].solve(state["t"], state["dt"])
        f = np.float64 if case["prec"] == "fp64" else np.float32
        return {"q": [state["b"].get_state(k)[0].astype(f, copy=False) for k in range(case["problems"])], "steps": steps}
    s = state["s"]
    s.advance(1e30, state["dtv"], case["steps"])
    q = _state_view(s, case["kind"] == "mhd")
    if case["prec"] != "fp64":
        q = q.to(torch.float32)
        torch.cuda.current_stream().synchronize()   # the solver's next step writes these buffers on its own stream
    return {"q": q, "dt": torch.tensor(state["dtv"][1], dtype=q.dtype)}


def work(case):
    """Per step (a right-hand side): the state read and written once; per stage
    and face the projections of a 2r-point stencil, ten (MHD 16) reconstructions
    and the back projection, counted as multiplications and additions."""
    if case["kind"] == "batch":
        # the fastest wave of these states runs at about 2.5: steps of 0.4 / (2.5 n)
        upd = sum(n * n * max(1.0, case["dt_total"] * n * 2.5 / 0.4) for n in _sizes(case))
        return {"bytes": 80.0 * upd, "flops": 3 * 2 * 1300.0 * upd}
    cells = float(case["mx"] * case["my"])
    if case["kind"] == "construct_l":
        return {"bytes": 96.0 * cells, "flops": 2 * 1300.0 * cells}
    if case["kind"] == "mhd":
        return {"bytes": 144.0 * cells * case["steps"], "flops": 3 * 2 * 2600.0 * cells * case["steps"]}
    stages = {"rk": {2: 2, 3: 3, 4: 10}.get(case["time_order"]), "md": 2, "lxw": 1}[case["method"]]
    face = {5: 1300.0, 7: 2400.0, 9: 3800.0}[case["order"]] + (600.0 if case["method"] != "rk" else 0.0)
    return {"bytes": 80.0 * cells * case["steps"], "flops": 2 * face * stages * cells * case["steps"]}


# ---- the same in plain torch, 64 bits ---------------------------------------

def _prim(Q, g):
    rho = Q[0]
    u, v, w = Q[1] / rho, Q[2] / rho, Q[3] / rho
    return rho, u, v, w, (g - 1.0) * (Q[4] - 0.5 * rho * (u * u + v * v + w * w))


def _cell_speeds(Q, g):
    rho, u, v, _, p = _prim(Q, g)
    c = torch.sqrt(torch.abs(g * p / rho))
    return torch.abs(u) + c, torch.abs(v) + c


def _flux(Q, n, g):
    rho, u, v, w, p = _prim(Q, g)
    un = u if n == 1 else v
    F = [rho * un, rho * u * un, rho * v * un, rho * w * un, un * (Q[4] + p)]
    F[n] = F[n] + p
    return torch.stack(F)


_scheme_cache = {}


def _scheme(order):
    """Candidate stencils, linear weights and Jiang-Shu smoothness forms of
    WENO of an odd order, from the interpolating polynomials of the cell
    averages (exact fractions; the forms scaled as Balsara and Shu print them)."""
    if order in _scheme_cache:
        return _scheme_cache[order]
    r = (order + 1) // 2

    def poly(points):   # coefficients (power basis in x, cell 0 = [-1/2, 1/2]) per unit cell average
        n = len(points)
        M = [[(Fraction(2 * c + 1, 2) ** (k + 1) - Fraction(2 * c - 1, 2) ** (k + 1)) / (k + 1) for k in range(n)]
             + [Fraction(int(i == j)) for j in range(n)] for i, c in enumerate(points)]
        for i in range(n):
            piv = next(k for k in range(i, n) if M[k][i] != 0)
            M[i], M[piv] = M[piv], M[i]
            M[i] = [v / M[i][i] for v in M[i]]
            for k in range(n):
                if k != i and M[k][i] != 0:
                    M[k] = [a - M[k][i] * b for a, b in zip(M[k], M[i])]
        return [[M[k][n + j] for k in range(n)] for j in range(n)]   # [average j][power k]

    def at_half(P):
        return [sum(c * Fraction(1, 2) ** k for k, c in enumerate(row)) for row in P]

    def deriv(c):
        return [k * v for k, v in enumerate(c)][1:]

    def integral(a, b):
        s = Fraction(0)
        for i, u in enumerate(a):
            for j, v in enumerate(b):
                if (i + j) % 2 == 0:
                    s += u * v * 2 * Fraction(1, 2) ** (i + j + 1) / (i + j + 1)
        return s

    scale = {5: 1, 7: 240, 9: 5040}[order]
    cand, forms = [], []
    for k in range(r):
        P = poly(list(range(k - r + 1, k + 1)))
        cand.append(at_half(P))
        form = [[Fraction(0)] * r for _ in range(r)]
        D = P
        for _ in range(1, r):
            D = [deriv(row) for row in D]
            for i in range(r):
                for j in range(r):
                    form[i][j] += integral(D[i], D[j])
        forms.append([[float(v * scale) for v in row] for row in form])
    full = at_half(poly(list(range(1 - r, r))))
    lin, rest = [], list(full)
    for k in range(r):
        d = rest[k] / cand[k][0]
        lin.append(d)
        for j in range(r):
            rest[k + j] -= d * cand[k][j]
    out = ([[float(v) for v in row] for row in cand], [float(v) for v in lin], forms)
    _scheme_cache[order] = out
    return out


def _recon(u, order, ver, eps, pw):
    """WENO value at i+1/2 of the list of 2r-1 point values u."""
    cand, lin, forms = _scheme(order)
    r = len(lin)
    val, beta = [], []
    for k in range(r):
        s = u[k:k + r]
        val.append(sum(c * a for c, a in zip(cand[k], s)))
        # the forms annihilate constants: evaluate them on differences from the middle point
        d = [a - s[r // 2] for a in s]
        b = 0.0
        for i in range(r):
            for j in range(i, r):
                c = forms[k][i][j] * (1 if i == j else 2)
                if i != r // 2 and j != r // 2:
                    b = b + c * (d[i] * d[j])
        beta.append(b)
    if ver == "FD":
        return sum(g * v for g, v in zip(lin, val))
    if ver == "JS":
        w = [g * (eps + b) ** (-pw) for g, b in zip(lin, beta)]
    else:
        tau = torch.abs({3: lambda b: b[0] - b[2], 4: lambda b: b[0] + 3 * (b[1] - b[2]) - b[3],
                         5: lambda b: b[4] - b[0]}[r](beta))
        w = [g * (1.0 + (tau / (eps + b)) ** pw) for g, b in zip(lin, beta)]
    return sum(a * v for a, v in zip(w, val)) / sum(w)


def _faces(Q, F, n, order, ver, p, ag):
    """Numerical fluxes and speeds of the n+1 faces along axis 1 of Q, F
    (5, n + 2r, M) in the normal frame (rho, m_n, m_t, m_w, E)."""
    r, g = (order + 1) // 2, p.gamma
    Ql, Qr = Q[:, r - 1:r + n], Q[:, r:r + n + 1]
    Qa = 0.5 * (Ql + Qr)
    rho, u1, u2, u3, press = _prim(Qa, g)
    um2 = u1 * u1 + u2 * u2 + u3 * u3
    c, H = torch.sqrt(g * press / rho), (Qa[4] + press) / rho
    rl, ul, _, _, pl = _prim(Ql, g)
    rr, ur, _, _, pr = _prim(Qr, g)
    ua, ca = 0.5 * (ul + ur), torch.sqrt(torch.abs(g * 0.5 * (pl + pr) / rho))
    s1 = torch.minimum(ul - torch.sqrt(torch.abs(g * pl / rl)), ua - ca)
    s2 = torch.maximum(ur + torch.sqrt(torch.abs(g * pr / rr)), ua + ca)
    alpha = torch.clamp(torch.maximum(s1.abs(), s2.abs()), min=ag)
    la = p.alpha_scaling * alpha
    d = 2 * H - um2

    def left(v):
        tail = c * (v[4] - u2 * v[2] - u3 * v[3])
        return torch.stack([
            ((0.5 * um2 - H - u1 * c) * v[1] + (0.5 * um2 * (c - u1) + H * u1) * v[0] + tail) / (c * d),
            ((H - um2) * v[0] + u1 * v[1] + u2 * v[2] + u3 * v[3] - v[4]) * 2 / d,
            v[2] - u2 * v[0], v[3] - u3 * v[0],
            ((H - 0.5 * um2 - u1 * c) * v[1] + (0.5 * um2 * (c + u1) - H * u1) * v[0] + tail) / (c * d)])

    gp, gm = [], []
    for s in range(2 * r):
        w, f = left(Q[:, s:s + n + 1]), left(F[:, s:s + n + 1])
        gp.append(0.5 * (f + la * w))
        gm.append(0.5 * (f - la * w))
    W = _recon(gp[:2 * r - 1], order, ver, p.epsilon, p.power_param) + \
        _recon(gm[:0:-1], order, ver, p.epsilon, p.power_param)
    s = W[0] + W[1] + W[4]
    return torch.stack([s, (u1 - c) * W[0] + u1 * W[1] + (u1 + c) * W[4], u2 * s + W[2], u3 * s + W[3],
                        (H - u1 * c) * W[0] + 0.5 * um2 * W[1] + u2 * W[2] + u3 * W[3] + (H + u1 * c) * W[4]]), alpha


def _mhd_flux(Q, n, g):
    rho, B1, B2, B3 = Q[0], Q[5], Q[6], Q[7]
    u = [Q[1] / rho, Q[2] / rho, Q[3] / rho]
    Bm = 0.5 * (B1 * B1 + B2 * B2 + B3 * B3)
    p = (g - 1.0) * (Q[4] - 0.5 * rho * (u[0] ** 2 + u[1] ** 2 + u[2] ** 2) - Bm)
    un, Bn = u[n - 1], Q[4 + n]
    F = [rho * un] + [rho * un * u[k] - Bn * Q[5 + k] for k in range(3)]
    F[n] = F[n] + p + Bm
    F += [un * (Q[4] + p + Bm) - Bn * (u[0] * B1 + u[1] * B2 + u[2] * B3)]
    F += [un * Q[5 + k] - u[k] * Bn if k != n - 1 else torch.zeros_like(rho) for k in range(3)]
    return torch.stack(F)


def _mhd_speed(Ql, Qr, n, g):
    """max(|s1|, |s2|) of the MHD SetWaveSpd (the first magnetic component enters for either normal)."""
    def side(Q):
        rho = Q[0]
        p = (g - 1.0) * (Q[4] - 0.5 * (Q[1] ** 2 + Q[2] ** 2 + Q[3] ** 2) / rho
                         - 0.5 * (Q[5] ** 2 + Q[6] ** 2 + Q[7] ** 2))
        return rho, Q[n] / rho, p, Q[5], Q[6], Q[7]

    def fast(s):
        rho, _, p, b1, b2, b3 = s
        a2 = torch.abs(g * p / rho)
        t = a2 + (b1 * b1 + b2 * b2 + b3 * b3) / rho
        return torch.sqrt(0.5 * (t + torch.sqrt(torch.abs(t * t - 4 * a2 * b1 * b1 / rho))))
    l, r = side(Ql), side(Qr)
    a = [0.5 * (x + y) for x, y in zip(l, r)]
    ca = fast(a)
    return torch.maximum(torch.minimum(l[1] - fast(l), a[1] - ca).abs(), torch.maximum(r[1] + fast(r), a[1] + ca).abs())


def _mhd_faces(Q, n, nd, ver, p):
    """As _faces for ideal MHD (WENO5, local speeds); Q (8, n + 6, M) in the grid frame, normal nd."""
    g, gm1, t2 = p.gamma, p.gamma - 1.0, math.sqrt(2.0)
    Ql, Qr = Q[:, 2:n + 3], Q[:, 3:n + 4]
    alpha = _mhd_speed(Ql, Qr, nd, g)
    F = _mhd_flux(Q, nd, g)
    perm = [0, 1, 2, 3, 4, 5, 6, 7] if nd == 1 else [0, 2, 1, 3, 4, 6, 5, 7]
    Q, F = Q[perm], F[perm]
    Qa = 0.5 * (Q[:, 2:n + 3] + Q[:, 3:n + 4])
    rho = Qa[0]
    u = [Qa[k] / rho for k in (1, 2, 3)]
    Bv = [Qa[5], Qa[6], Qa[7]]
    um2 = 0.5 * (u[0] ** 2 + u[1] ** 2 + u[2] ** 2)
    press = gm1 * (Qa[4] - rho * um2 - 0.5 * (Bv[0] ** 2 + Bv[1] ** 2 + Bv[2] ** 2))
    sq, a2 = torch.sqrt(rho), g * press / rho
    a = torch.sqrt(a2)
    d = a2 + (Bv[0] ** 2 + Bv[1] ** 2 + Bv[2] ** 2) / rho
    disc = torch.sqrt(d * d - 4 * a2 * Bv[0] ** 2 / rho)
    cf, cs = torch.sqrt(0.5 * (d + disc)), torch.sqrt(0.5 * (d - disc))
    perp = Bv[1] ** 2 + Bv[2] ** 2
    none = perp <= 1e-12
    b1 = torch.where(Bv[0] < 0, -1.0, 1.0).to(F64)
    b2 = torch.where(none, 1 / t2, Bv[1] / torch.sqrt(perp))
    b3 = torch.where(none, 1 / t2, Bv[2] / torch.sqrt(perp))
    umb = none & (torch.abs(a2 - Bv[0] ** 2 / rho) <= 1e-12)
    dd = torch.sqrt(torch.abs(cf * cf - cs * cs))
    af = torch.where(umb, math.sin(math.atan(1.0) / 2), torch.sqrt(torch.abs(a2 - cs * cs)) / dd)
    as_ = torch.where(umb, math.cos(math.atan(1.0) / 2), torch.sqrt(torch.abs(cf * cf - a2)) / dd)

    def left(v):
        z = [(v[k + 1] - u[k] * v[0]) / rho for k in range(3)]
        zp = gm1 * (um2 * v[0] - u[0] * v[1] - u[1] * v[2] - u[2] * v[3] + v[4]
                    - Bv[0] * v[5] - Bv[1] * v[6] - Bv[2] * v[7])
        zt, zb = b1 * (b2 * z[1] + b3 * z[2]), b2 * v[6] + b3 * v[7]
        ft = (af * cf * z[0] - as_ * cs * zt) / (2 * a2)
        fe = af * zp / (2 * rho * a2) + as_ * zb / (2 * sq * a)
        st = (as_ * cs * z[0] + af * cf * zt) / (2 * a2)
        se = as_ * zp / (2 * rho * a2) - af * zb / (2 * sq * a)
        al, am = (b2 * z[2] - b3 * z[1]) / t2, (b2 * v[7] - b3 * v[6]) / (t2 * sq)
        return torch.stack([fe - ft, al + am, se - st, v[0] - zp / a2, v[5], se + st, al - am, fe + ft])

    la = p.alpha_scaling * alpha
    gp, gm = [], []
    for s in range(6):
        w, f = left(Q[:, s:s + n + 1]), left(F[:, s:s + n + 1])
        gp.append(0.5 * (f + la * w))
        gm.append(0.5 * (f - la * w))
    W = _recon(gp[:5], 5, ver, p.epsilon, p.power_param) + _recon(gm[:0:-1], 5, ver, p.epsilon, p.power_param)
    fs, ss, fd, sd = W[0] + W[7], W[2] + W[5], W[7] - W[0], W[5] - W[2]
    y0 = rho * (af * fs + as_ * ss) + W[3]
    yu = [af * cf * fd + as_ * cs * sd]
    tr = b1 * (af * cf * sd - as_ * cs * fd)
    yu += [b2 * tr - b3 * (W[1] + W[6]) / t2, b3 * tr + b2 * (W[1] + W[6]) / t2]
    yp = g * press * (af * fs + as_ * ss)
    br, bt = a * sq * (as_ * fs - af * ss), sq * (W[1] - W[6]) / t2
    yb = [W[4], b2 * br - b3 * bt, b3 * br + b2 * bt]
    out = [y0] + [rho * yu[k] + y0 * u[k] for k in range(3)]
    out += [um2 * y0 + rho * sum(u[k] * yu[k] for k in range(3)) + yp / gm1 + sum(Bv[k] * yb[k] for k in range(3))]
    return torch.stack(out + yb)[perm], alpha


def _chunks(M, n):
    step = max(1, (1 << 21) // max(1, n))
    return [(k, min(M, k + step)) for k in range(0, M, step)]


def _rhs(q, p, order, ver, px, py, ag, FG=None, want_faces=False):
    """ConstructL / ConstructLxWL: L, face speeds (and the face fluxes)."""
    r = (order + 1) // 2
    mhd = q.shape[0] == 8
    mx, my = q.shape[1:]
    dx, dy = (p.xhigh - p.xlow) / mx, (p.yhigh - p.ylow) / my
    Fx, sx = torch.empty((q.shape[0], mx + 1, my), dtype=F64, device="cuda"), torch.empty((mx + 1, my), dtype=F64, device="cuda")
    qx, qy = q[:, _index(mx, r, px)], q[:, :, _index(my, r, py)]
    for a, b in _chunks(my, mx):
        if mhd:
            Fx[:, :, a:b], sx[:, a:b] = _mhd_faces(qx[:, :, a:b], mx, 1, ver, p)
        else:
            f = _flux(qx[:, :, a:b], 1, p.gamma) if FG is None else FG[0][:, :, 3 + a:3 + b]
            Fx[:, :, a:b], sx[:, a:b] = _faces(qx[:, :, a:b], f, mx, order, ver, p, ag[0])
    Fy, sy = torch.empty((q.shape[0], mx, my + 1), dtype=F64, device="cuda"), torch.empty((mx, my + 1), dtype=F64, device="cuda")
    sw = [0, 2, 1, 3, 4]
    for a, b in _chunks(mx, my):
        Q = qy[:, a:b].transpose(1, 2)
        if mhd:
            f, s = _mhd_faces(Q, my, 2, ver, p)
            Fy[:, a:b] = f.transpose(1, 2)
        else:
            G = (_flux(Q, 2, p.gamma) if FG is None else FG[1][:, 3 + a:3 + b].transpose(1, 2))[sw]
            f, s = _faces(Q[sw], G, my, order, ver, p, ag[1])
            Fy[:, a:b] = f[sw].transpose(1, 2)
        sy[a:b] = s.transpose(0, 1)
    if want_faces:
        return Fx, Fy, sx, sy
    L = -(Fx[:, 1:] - Fx[:, :-1]) / dx - (Fy[:, :, 1:] - Fy[:, :, :-1]) / dy
    return L, sx, sy


def _integrated(q, p, px, py, dt, second=None):
    """ConstructIntegratedR on the 3-cell frame: with f_tt (one state), or the
    two-state form a1 f(q) + dt b1 f_t(q) + dt b2 f_t(q2)."""
    mx, my = q.shape[1:]
    g = p.gamma
    dx, dy = (p.xhigh - p.xlow) / mx, (p.yhigh - p.ylow) / my

    def sh(a, i, j):
        return a[:, 2 + i:a.shape[1] - 2 + i, 2 + j:a.shape[2] - 2 + j]

    def d1(a, ax, h):
        s = [sh(a, k, 0) if ax == 1 else sh(a, 0, k) for k in (-2, -1, 1, 2)]
        return ((s[0] - s[3]) / 12.0 + (s[2] - s[1]) * (2.0 / 3.0)) / h

    def d2(a, ax, h):
        s = [sh(a, k, 0) if ax == 1 else sh(a, 0, k) for k in (-2, -1, 0, 1, 2)]
        return ((-s[0] - s[4]) / 12.0 + (s[1] + s[3]) * (4.0 / 3.0) - s[2] * 2.5) / (h * h)

    def dxy(a):
        return (sh(a, 1, 1) - sh(a, -1, 1) - sh(a, 1, -1) + sh(a, -1, -1)) / (4 * dx * dy)

    def var(c, a):
        rho, u, m, E, P = c
        du = [(a[k + 1] - u[k] * a[0]) / rho for k in range(3)]
        uu = u[0] ** 2 + u[1] ** 2 + u[2] ** 2
        dpe = (g - 1) * (0.5 * uu * a[0] - u[0] * a[1] - u[1] * a[2] - u[2] * a[3])
        return du, dpe + (g - 1) * a[4], dpe

    def jac(n, c, a):
        rho, u, m, E, P = c
        du, dp, _ = var(c, a)
        out = [a[n]] + [a[n] * u[k] + m[n - 1] * du[k] + (dp if k + 1 == n else 0.0) for k in range(3)]
        return torch.stack(out + [(a[4] + dp) * u[n - 1] + (E + P) * du[n - 1]])

    def hess(n, c, a, b):
        # the energy row leaves the pressure's E dependence out of the cross terms, as the reference's Hessian does
        rho, u, m, E, P = c
        da, _, ea = var(c, a)
        db, _, eb = var(c, b)
        d2u = [-(da[k] * b[0] + db[k] * a[0]) / rho for k in range(3)]
        d2p = -(g - 1) * rho * sum(da[k] * db[k] for k in range(3))
        out = [torch.zeros_like(rho)] + [a[n] * db[k] + b[n] * da[k] + m[n - 1] * d2u[k] + (d2p if k + 1 == n else 0.0)
                                         for k in range(3)]
        return torch.stack(out + [(a[4] + ea) * db[n - 1] + (b[4] + eb) * da[n - 1] + d2p * u[n - 1]
                                  + (E + P) * d2u[n - 1]])

    def parts(s):
        Q = _ghosted(s, 5, px, py)
        f, gg = _flux(Q, 1, g), _flux(Q, 2, g)
        Qc = sh(Q, 0, 0)
        rho, u, v, w, P = _prim(Qc, g)
        c = (rho, [u, v, w], [Qc[1], Qc[2], Qc[3]], Qc[4], P)
        return Q, f, gg, c, d1(f, 1, dx) + d1(gg, 2, dy)

    Q, f, gg, c, w = parts(q)
    if second is None:
        fpg = (hess(1, c, d1(Q, 1, dx), w) + hess(2, c, d1(Q, 2, dy), w) + jac(1, c, d2(f, 1, dx) + dxy(gg))
               + jac(2, c, dxy(f) + d2(gg, 2, dy)))
        return [sh(a, 0, 0) + 0.5 * dt * (-jac(n, c, w) + dt / 3.0 * (jac(n, c, fpg) + hess(n, c, w, w)))
                for n, a in ((1, f), (2, gg))]
    q2, a1, b1, b2 = second
    _, _, _, c2, w2 = parts(q2)
    return [a1 * sh(a, 0, 0) - dt * b1 * jac(n, c, w) - dt * b2 * jac(n, c2, w2) for n, a in ((1, f), (2, gg))]


def _mpp_update(q, p, px, py, Fx, Fy, ag, dt):
    """The Lax-Wendroff update with the positivity limiter: Lax-Friedrichs
    fluxes, the density and the pressure step per cell, the limited update."""
    g = p.gamma
    mx, my = q.shape[1:]
    dtx, dty = dt * mx / (p.xhigh - p.xlow), dt * my / (p.yhigh - p.ylow)

    def lf(Q, n, a):
        f = _flux(Q, n, g)
        lo, hi = (slice(None, -1), slice(1, None))
        sl = (lambda t, k: t[:, k]) if n == 1 else (lambda t, k: t[:, :, k])
        return 0.5 * (sl(f, lo) + sl(f, hi)) + 0.5 * a * (sl(Q, lo) - sl(Q, hi))

    Lx, Ly = lf(q[:, _index(mx, 1, px)], 1, ag[0]), lf(q[:, :, _index(my, 1, py)], 2, ag[1])
    fh = [Fx[:, :-1], Fx[:, 1:], Fy[:, :, :-1], Fy[:, :, 1:]]
    fl = [Lx[:, :-1], Lx[:, 1:], Ly[:, :, :-1], Ly[:, :, 1:]]

    def upd(f):
        return q + dtx * (f[0] - f[1]) + dty * (f[2] - f[3])

    def pres(Q):
        return _prim(Q, g)[4]

    eps = 1e-12
    qlf = upd(fl)
    sgn = [dtx, -dtx, dty, -dty]
    ff = [sgn[k] * (fh[k][0] - fl[k][0]) for k in range(4)]
    tot = sum(torch.where(x < 0, x, torch.zeros_like(x)) for x in ff)
    one = torch.ones_like(tot)
    amin = [torch.where(x < 0, torch.minimum((eps - qlf[0]) / (tot - eps), one), one) for x in ff]
    scale = [one.clone() for _ in range(4)]
    for combo in range(16):
        on = [(combo >> (3 - k)) & 1 for k in range(4)]
        qh = upd([amin[k] * fh[k] + (1 - amin[k]) * fl[k] if on[k] else fl[k] for k in range(4)])
        ph = pres(qh)
        lo, hi, rate = torch.zeros_like(ph), one.clone(), torch.zeros_like(ph)
        bad = ph < 0
        if bool(bad.any()):
            for _ in range(9):
                rate = 0.5 * (lo + hi)
                ph = pres(rate * qh + (1 - rate) * qlf)
                hi, lo = torch.where(ph < 0, rate, hi), torch.where(ph < 0, lo, rate)
            res = torch.where(bad, torch.where(ph > 0, rate, lo), one)
            for k in range(4):
                if on[k]:
                    scale[k] = torch.minimum(scale[k], res)
    am = [scale[k] * amin[k] for k in range(4)]
    tx, ty = torch.ones((mx + 1, my), dtype=F64, device="cuda"), torch.ones((mx, my + 1), dtype=F64, device="cuda")
    tx[:-1], ty[:, :-1] = am[0], am[2]
    tx[1:], ty[:, 1:] = torch.cat([torch.minimum(tx[1:-1], am[1][:-1]), am[1][-1:]]), \
        torch.cat([torch.minimum(ty[:, 1:-1], am[3][:, :-1]), am[3][:, -1:]], 1)
    Hx, Hy = tx * (Fx - Lx) + Lx, ty * (Fy - Ly) + Ly
    return q - dtx * (Hx[:, 1:] - Hx[:, :-1]) - dty * (Hy[:, :, 1:] - Hy[:, :, :-1])


def _euler_steps(q, p, case, steps, dt, tend=None):
    """`steps` accepted adaptive steps (or up to tend) from q; (q, next dt, steps taken)."""
    order, ver = case["order"], case["weno"]
    px, py = case["bcx"] == "periodic", case["bcy"] == "periodic"
    mx, my = q.shape[1:]
    dx, dy = (p.xhigh - p.xlow) / mx, (p.yhigh - p.ylow) / my

    def alpha(s):
        return [float(a.max()) for a in _cell_speeds(s, p.gamma)] if case["global_alpha"] else [0.0, 0.0]

    t, taken = 0.0, 0
    while (taken < steps) if tend is None else (t < tend):
        if tend is not None and t + dt > tend:
            dt = tend - t
        S = [0.0, 0.0]

        def L(s, FG=None):
            l, sx, sy = _rhs(s, p, order, ver, px, py, alpha(s), FG)
            S[0], S[1] = max(S[0], float(sx[:-1].max())), max(S[1], float(sy[:, :-1].max()))
            return l
        if case["method"] == "md":
            q1 = q + 0.5 * dt * L(q, _integrated(q, p, px, py, 0.5 * dt))
            qn = q + dt * L(q1, _integrated(q, p, px, py, dt, (q1, 1.0, 1.0 / 6.0, 1.0 / 3.0)))
        elif case["method"] == "lxw" and not case["mpp"]:
            qn = q + dt * L(q, _integrated(q, p, px, py, dt))
        elif case["method"] == "lxw":
            ag = [float(a.max()) for a in _cell_speeds(q, p.gamma)]
            Fx, Fy, sx, sy = _rhs(q, p, order, ver, px, py, alpha(q), _integrated(q, p, px, py, dt), True)
            S = [max(ag[0], float(sx[:-1].max())), max(ag[1], float(sy[:, :-1].max()))]
            qn = _mpp_update(q, p, px, py, Fx, Fy, ag, dt)
        elif case["time_order"] == 2:
            q1 = q + dt * L(q)
            qn = 0.5 * q1 + 0.5 * q + 0.5 * dt * L(q1)
        elif case["time_order"] == 3:
            q1 = q + dt * L(q)
            q1 = 0.75 * q + 0.25 * q1 + 0.25 * dt * L(q1)
            qn = (2.0 / 3.0) * q1 + (1.0 / 3.0) * q + (2.0 / 3.0) * dt * L(q1)
        else:
            q1 = q
            for _ in range(5):
                q1 = q1 + dt / 6.0 * L(q1)
            q2 = (q + 9.0 * q1) / 25.0
            q1 = 15.0 * q2 - 5.0 * q1
            for _ in range(4):
                q1 = q1 + dt / 6.0 * L(q1)
            qn = q2 + 0.6 * q1 + 0.1 * dt * L(q1)
        cfl = max(dt * S[0] / dx, dt * S[1] / dy)
        if cfl <= p.max_cfl:
            q, t, taken = qn, t + dt, taken + 1
        dt = min(p.max_dt, dt * p.desired_cfl / cfl)
    return q, dt, taken


def _mhd_steps(q, a3, p, ver, steps, dt):
    mx, my = q.shape[1:]
    dx, dy = (p.xhigh - p.xlow) / mx, (p.yhigh - p.ylow) / my

    def hj(s, a):
        def recon(axis, h, sign):
            d = [(torch.roll(a, -k, axis) - torch.roll(a, 1 - k, axis)) / h for k in range(-2, 4)]   # d[m]: difference m - 2
            u = d[:5] if sign < 0 else d[:0:-1]
            return _recon(u, 5, ver, p.epsilon, p.power_param)
        u1, u2 = s[1] / s[0], s[2] / s[0]
        m1, m2 = max(1e-15, float(u1.abs().max())), max(1e-15, float(u2.abs().max()))
        xm, xp, ym, yp = recon(0, dx, -1), recon(0, dx, 1), recon(1, dy, -1), recon(1, dy, 1)
        return -u1 * 0.5 * (xm + xp) - u2 * 0.5 * (ym + yp) + m1 * 0.5 * (xp - xm) + m2 * 0.5 * (yp - ym)

    taken = 0
    while taken < steps:
        S = 0.0
        qs, as_ = q, a3
        for c0, cs, cl in ((1.0, 0.0, 1.0), (0.75, 0.25, 0.25), (1.0 / 3.0, 2.0 / 3.0, 2.0 / 3.0)):
            l, sx, sy = _rhs(qs, p, 5, ver, True, True, (0.0, 0.0))
            S = max(S, float(torch.maximum(sx[:-1], sy[:, :-1]).max()))
            la = hj(qs, as_)
            qs = (c0 * q + cs * qs if cs else q) + cl * dt * l
            as_ = (c0 * a3 + cs * as_ if cs else a3) + cl * dt * la
            qs[5], qs[6] = _d4(as_, 1, dy), -_d4(as_, 0, dx)
        cfl = dt * S * (1.0 / dx + 1.0 / dy)
        if cfl <= p.max_cfl:
            q, a3, taken = qs, as_, taken + 1
        dt = min(p.max_dt, dt * p.desired_cfl / cfl)
    return q, a3, dt


def exact(case, seed):
    """The FP64 full-WENO result (for the hybrid form too: its linear faces are its approximation)."""
    if case["kind"] == "batch":
        return None   # some thousand steps of small grids
    p = _params(case)
    out = torch.float64 if case.get("prec", "fp64") == "fp64" else torch.float32
    if case["kind"] == "mhd":
        q, a3 = _mhd_state(p.mx, p.my, p.gamma, seed)
        q, a3, dt = _mhd_steps(q, a3, p, case["weno"], case["steps"], _mhd_first_dt(p, q))
        return {"q": torch.cat([q, a3[None]]).to(out), "dt": torch.tensor(dt, dtype=out)}
    q = _euler_state(p.mx, p.my, p.gamma, seed, vacuum=bool(case.get("mpp")))
    if case["kind"] == "construct_l":
        ag = [float(a.max()) for a in _cell_speeds(q, p.gamma)] if case["global_alpha"] else [0.0, 0.0]
        px, py = p.bc_xlow == A.FIN_BC_PERIODIC, p.bc_ylow == A.FIN_BC_PERIODIC
        L, sx, sy = _rhs(q, p, 5, case["weno"], px, py, ag)
        b = p.mbc
        host = np.zeros(A.ghosted_shape(p))
        host[b:b + p.mx, b:b + p.my] = L.permute(1, 2, 0).cpu().numpy()
        sm = np.zeros(A.smax_shape(p))
        sm[b:b + p.mx + 1, b:b + p.my, 0] = sx.cpu().numpy()
        sm[b:b + p.mx, b:b + p.my + 1, 1] = sy.cpu().numpy()
        return {"L": host, "smax": sm}
    q, dt, _ = _euler_steps(q, p, case, case["steps"], _first_dt(p, q))
    return {"q": q.to(out), "dt": torch.tensor(dt, dtype=out)}
