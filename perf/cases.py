"""Timed cases of the library: what its users have it solve, through the public
entry points (``Solver``, ``HeatADI``, ``ChannelPoisson``, ``ChannelMomentum``),
with inputs made from a seed, a 64-bit answer in plain torch and the error a
correct implementation may show.

A case is a dict of plain values; ``listed()`` are the fixed ones, ``draw(rng)``
one more of the same ranges.  Arrays are row-interleaved [n_row, n_sys].
"""
import math

import numpy as np
import torch

from filtered_tdma_b200 import Solver
from filtered_tdma_b200 import _lib as L
from filtered_tdma_b200.heat import HeatADI
from filtered_tdma_b200.momentum import ChannelMomentum
from filtered_tdma_b200.poisson import ChannelPoisson

PI = math.pi
EPS_CONSTANT = 1.0e-3  # the Filtered solvers' eps constant: the applications pass dt


def listed():
    return [
        # one sweep of a 64^3 heat step on one rank (P = 1: the serial Thomas): the smallest call
        dict(name="serial_4096x64", kind="solve", method="pascal", n_sys=4096, n_row=64, P=1,
             periodic=False, dtype="f64", r_hi=10.0),
        # one rank again, at the Z sweep of a 256 x 384 x 512 grid
        dict(name="serial_98304x512", kind="solve", method="pascal", n_sys=98304, n_row=512, P=1,
             periodic=False, dtype="f64", r_hi=10.0),
        # the batch of the headline benchmark: 512^3 cells, 8 segments a system
        dict(name="pascal_262144x512", kind="solve", method="pascal", n_sys=262144, n_row=512,
             P=8, periodic=False, dtype="f64", r_hi=10.0),
        # the same batch stored in FP32
        dict(name="store32_262144x512", kind="solve", method="pascal", n_sys=262144, n_row=512,
             P=8, periodic=False, dtype="f32", r_hi=10.0),
        # a sweep of a 250^3 grid: a row count that no tile divides
        dict(name="pascal_62500x250", kind="solve", method="pascal", n_sys=62500, n_row=250, P=4,
             periodic=False, dtype="f64", r_hi=10.0),
        # periodic sweep of a 256^3 grid
        dict(name="periodic_65536x256", kind="solve", method="pascal", n_sys=65536, n_row=256,
             P=4, periodic=True, dtype="f64", r_hi=10.0),
        # few long systems
        dict(name="pascal_8192x4096", kind="solve", method="pascal", n_sys=8192, n_row=4096,
             P=16, periodic=False, dtype="f64", r_hi=10.0),
        # Filtered v2 where its truncation holds (rho <= 1/3)
        dict(name="filtered_65536x512", kind="solve", method="filtered_v2", n_sys=65536,
             n_row=512, P=8, periodic=False, dtype="f64", r_hi=1.0),
        # systems of 16 to 4096 rows in one call, a quarter of them periodic, tuned once
        dict(name="ragged_10000", kind="ragged", n_sys=10000, n_lo=16, n_hi=4096,
             periodic_frac=0.25, dtype="f64", tuned=True),
        # one step of the 3-D heat application
        dict(name="heat_256x384x512", kind="heat", ix=256, iy=384, iz=512, rho=0.25),
        # the wall-normal solves of a channel flow's FFT Poisson equation
        dict(name="poisson_128x128x192", kind="poisson", n1m=128, n2m=128, n3m=192, gamma=2.0),
        # the implicit viscous half step of one velocity component
        dict(name="momentum_256x256x256", kind="momentum", nx=256, ny=256, nz=256, comp=0,
             c=1.0e-3),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["serial", "pascal", "pascal", "periodic", "long", "store32", "filtered",
                       "ragged", "heat", "poisson", "momentum"])
    case = dict(kind="solve", method="pascal", periodic=False, dtype="f64",
                r_hi=rng.choice([1.0, 10.0]))
    if kind == "serial":
        n_row = _log_int(rng, 16, 512)
        case.update(n_sys=_log_int(rng, 256, min(131072, (1 << 24) // n_row)), n_row=n_row, P=1,
                    periodic=rng.random() < 0.25)
    elif kind == "pascal":
        n_row = rng.choice([_log_int(rng, 32, 512), 16 * rng.randint(2, 32)])
        case.update(n_sys=_log_int(rng, 1024, (1 << 25) // n_row), n_row=n_row,
                    P=rng.choice([2, 4, 8]))
    elif kind == "periodic":
        n_row = rng.choice([64, 128, 256, 512, 16 * rng.randint(3, 32), rng.randint(48, 512)])
        case.update(n_sys=_log_int(rng, 1024, (1 << 24) // n_row), n_row=n_row,
                    P=rng.choice([4, 8]), periodic=True)
    elif kind == "long":
        n_row = rng.choice([rng.randint(513, 2048), 16 * rng.randint(33, 128), 1024, 2048, 4096])
        n_sys = _log_int(rng, 512, (1 << 25) // n_row)
        # an odd batch of 4096-row systems is refused at P = 16
        case.update(n_sys=n_sys - n_sys % 2 if n_row == 4096 else n_sys, n_row=n_row, P=16)
    elif kind == "store32":
        n_row = 16 * rng.randint(2, 32)
        case.update(n_sys=4 * _log_int(rng, 1024, (1 << 24) // n_row), n_row=n_row, P=8,
                    dtype="f32")
    elif kind == "filtered":
        n_row = rng.choice([128, 256, 512, 512, rng.randint(100, 512)])
        case.update(method="filtered_v2", n_sys=_log_int(rng, 1024, (1 << 24) // n_row),
                    n_row=n_row, P=rng.choice([2, 4, 8]), r_hi=1.0)
    elif kind == "ragged":
        case = dict(kind="ragged", n_sys=_log_int(rng, 500, 10000), n_lo=rng.randint(3, 64),
                    n_hi=rng.choice([512, 1024, 4096]), periodic_frac=rng.choice([0.0, 0.25, 0.5]),
                    dtype=rng.choice(["f64", "f32"]), tuned=rng.random() < 0.5)
    elif kind == "heat":
        ix, iy, iz = 64 * rng.randint(1, 4), 64 * rng.randint(1, 5), 16 * _log_int(rng, 4, 20)
        case = dict(kind="heat", ix=ix, iy=iy, iz=iz, rho=rng.choice([0.25, 0.4]))
    elif kind == "poisson":
        case = dict(kind="poisson", n1m=2 * rng.randint(16, 96), n2m=2 * rng.randint(16, 96),
                    n3m=16 * rng.randint(3, 24), gamma=rng.choice([1.5, 2.0]))
    else:
        case = dict(kind="momentum", nx=rng.choice([64, 128, 256]), ny=rng.choice([64, 128, 256]),
                    nz=16 * rng.randint(4, 20), comp=rng.randrange(3), c=1.0e-3)
    return case


# ------------------------------------------------------------------- inputs
def _gen(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    return g


def _rand(g, *shape):
    return torch.rand(shape, generator=g, dtype=torch.float64, device="cuda")


def _solve_inputs(case, seed):
    """A, B, C, D of an implicit diffusion sweep: per-system r log-uniform in
    [0.1, r_hi], rows scaled by a smoothly stretched grid's metrics, D uniform."""
    g = _gen(seed)
    n_sys, n_row = case["n_sys"], case["n_row"]
    r = 10.0 ** (-1.0 + (math.log10(case["r_hi"]) + 1.0) * _rand(g, n_sys))
    k = torch.arange(n_row + 1, dtype=torch.float64, device="cuda")
    m = 1.0 + 0.1 * torch.cos(2.0 * PI * k / n_row + 2.0 * PI * _rand(g, 1))
    A = -m[:-1, None] * r
    C = -m[1:, None] * r
    B = 1.0 - A - C
    D = 2.0 * _rand(g, n_row, n_sys) - 1.0
    dt = torch.float32 if case["dtype"] == "f32" else torch.float64
    return [x.to(dt).contiguous() for x in (A, B, C, D)]


def _ragged_inputs(case, seed):
    """CSR batch: lengths log-uniform in [n_lo, n_hi] (the case's layout, the same
    for every seed), r log-uniform in [0.05, 20]."""
    n_sys, lo, hi = case["n_sys"], case["n_lo"], case["n_hi"]
    rng = np.random.default_rng(n_sys)
    n = np.floor(np.exp(rng.uniform(math.log(lo), math.log(hi), n_sys))).astype(np.int64)
    n = np.clip(n, lo, hi)
    per = (rng.uniform(size=n_sys) < case["periodic_frac"]).astype(np.uint8)
    rng = np.random.default_rng(seed)
    r = np.repeat(10.0 ** rng.uniform(math.log10(0.05), math.log10(20.0), n_sys), n)
    off = np.concatenate([[0], np.cumsum(n)]).astype(np.int64)
    d = rng.uniform(-1.0, 1.0, int(off[-1]))
    dt = np.float32 if case["dtype"] == "f32" else np.float64
    arrays = [torch.from_numpy(x.astype(dt)).cuda() for x in (-r, 1.0 + 2.0 * r, -r, d)]
    return arrays, off, per


def _heat_dt(case):
    dd = 2.0 / case["ix"]
    return case["rho"] / (1.0 - 2.0 * case["rho"]) * 2.0 * dd * dd


def _centres(n):
    return -1.0 + (torch.arange(n + 2, dtype=torch.float64, device="cuda") - 0.5) * (2.0 / n)


def _heat_inputs(case, seed):
    """A smooth field with small noise on the grid with ghosts."""
    g = _gen(seed)
    x, y, z = (_centres(case[k]) for k in ("ix", "iy", "iz"))
    th = (torch.sin(PI * z)[:, None, None] * torch.sin(PI * y)[None, :, None]
          * torch.sin(PI * x)[None, None, :])
    th += (torch.cos(PI * z)[:, None, None] * torch.cos(PI * y)[None, :, None]
           * torch.cos(PI * x)[None, None, :])
    return th + 0.1 * (2.0 * _rand(g, *th.shape) - 1.0)


def _poisson_inputs(case, seed):
    g = _gen(seed)
    shape = (case["n3m"], case["n2m"], case["n1m"] // 2 + 1)
    return torch.complex(2.0 * _rand(g, *shape) - 1.0, 2.0 * _rand(g, *shape) - 1.0)


def _momentum_inputs(case, seed):
    g = _gen(seed)
    return 2.0 * _rand(g, case["nz"] + 2, case["ny"] + 2, case["nx"] + 2) - 1.0


def prepare(case, seed):
    kind = case["kind"]
    if kind == "solve":
        A, B, C, D = _solve_inputs(case, seed)
        prec = L.FP32_STORE if case["dtype"] == "f32" else L.FP64
        s = Solver(case["method"], case["n_sys"], case["n_row"], case["P"], precision=prec)
        if case["method"] != "pascal":
            s.set_eps_constant(EPS_CONSTANT)
            s.set_rho(A, B, C, all_systems=True)
        X = torch.empty(D.shape, dtype=torch.float64, device="cuda")
        return dict(case=case, solver=s, arrays=(A, B, C, D), X=X)
    if kind == "ragged":
        arrays, off, per = _ragged_inputs(case, seed)
        prec = L.FP32_STORE if case["dtype"] == "f32" else L.FP64
        s = Solver("pascal", case["n_sys"], 64, 2, precision=prec)
        X = torch.empty(arrays[3].shape, dtype=torch.float64, device="cuda")
        if case["tuned"]:
            s.ragged_autotune(*arrays, X, off, per)
        else:  # the first call with a layout builds its plan
            s.solve_ragged(*arrays, X, off, per)
        return dict(case=case, solver=s, arrays=arrays, X=X, off=off, per=per)
    if kind == "heat":
        h = HeatADI(case["ix"], case["iy"], case["iz"], dt=_heat_dt(case))
        return dict(case=case, solver=h, theta=_heat_inputs(case, seed))
    if kind == "poisson":
        p = ChannelPoisson(case["n1m"], case["n2m"], case["n3m"], gamma=case["gamma"])
        rhs = _poisson_inputs(case, seed)
        return dict(case=case, solver=p, rhs=rhs, hat=torch.empty_like(rhs))
    m = ChannelMomentum(case["nx"], case["ny"], case["nz"])
    rhs = _momentum_inputs(case, seed)
    return dict(case=case, solver=m, rhs=rhs, q=torch.zeros_like(rhs))


def run(state):
    case, s = state["case"], state["solver"]
    kind = case["kind"]
    if kind == "solve":
        f = s.solve_f32 if case["dtype"] == "f32" else s.solve_out
        return f(*state["arrays"], state["X"], cyclic=case["periodic"])
    if kind == "ragged":
        return s.solve_ragged(*state["arrays"], state["X"], state["off"], state["per"])
    if kind == "heat":
        s.step(state["theta"], 1)
        return state["theta"]
    if kind == "poisson":  # the transform's output arrives in the array that is solved in place
        state["hat"].copy_(state["rhs"])
        return s.solve(state["hat"])
    return s.adi(case["comp"], state["rhs"], state["q"], case["c"])


def _ragged_rows(case):
    lo, hi = case["n_lo"], case["n_hi"]
    return case["n_sys"] * (hi - lo) / math.log(hi / lo)


def work(case):
    kind = case["kind"]
    if kind in ("solve", "ragged"):
        rows = case["n_sys"] * case["n_row"] if kind == "solve" else _ragged_rows(case)
        elem = 4 if case["dtype"] == "f32" else 8
        return {"bytes": rows * (4 * elem + 8), "flops": 8 * rows}
    if kind == "heat":  # three sweeps that each read and write the field
        cells = case["ix"] * case["iy"] * case["iz"]
        return {"bytes": 48 * cells, "flops": 40 * cells}
    if kind == "poisson":
        rows = case["n3m"] * case["n2m"] * (case["n1m"] // 2 + 1)
        return {"bytes": 32 * rows, "flops": 16 * rows}
    cells = case["nx"] * case["ny"] * case["nz"]
    return {"bytes": 48 * cells, "flops": 24 * cells}


def tolerance(case):
    kind = case["kind"]
    if kind == "solve" and case["P"] == 1:
        return "exact"  # the serial algorithm in the documented operation order
    if kind == "solve" and case["method"] != "pascal":
        # Filtered's own bound on what its truncation leaves out
        return {"rel": EPS_CONSTANT / case["n_row"] ** 2}
    if kind == "poisson":  # the matrix of mode (0, 0) has a condition number of about n3m^2
        return {"rel": 1.5e-11}
    # seen between the library and plain torch: 2e-16 (array solves), 4e-16
    # (heat), 1.1e-15 (momentum: stretched walls, three sweeps)
    return {"rel": 1e-15 if kind == "solve" else 4e-15}


# ------------------------------------------- the same in plain torch, 64 bits
def _thomas(A, B, C, D):
    """x of every system; A, B, C, D [n_row, n_sys] or [n_row, 1]."""
    n = D.shape[0]
    cp, dp = torch.empty_like(C), torch.empty_like(D)
    cp[0], dp[0] = C[0] / B[0], D[0] / B[0]
    for j in range(1, n):
        p = B[j] - A[j] * cp[j - 1]
        cp[j] = C[j] / p
        dp[j] = (D[j] - A[j] * dp[j - 1]) / p
    for j in range(n - 2, -1, -1):
        dp[j] -= cp[j] * dp[j + 1]
    return dp


def _thomas_periodic(A, B, C, D):
    """Rows 1.. as a plain system in x_0: x = u + x_0 v, then row 0 for x_0."""
    E = torch.zeros_like(A[1:])
    E[0] -= A[1]
    E[-1] -= C[-1]
    A1 = A[1:].clone()
    C1 = C[1:].clone()
    A1[0] = 0.0
    C1[-1] = 0.0
    u, v = _thomas(A1, B[1:], C1, D[1:]), _thomas(A1, B[1:], C1, E)
    x0 = (D[0] - A[0] * u[-1] - C[0] * u[0]) / (B[0] + A[0] * v[-1] + C[0] * v[0])
    return torch.cat([x0[None], u + x0 * v])


def _exact_ragged(case, seed):
    arrays, off, per = _ragged_inputs(case, seed)
    n = np.diff(off)
    out = torch.empty(int(off[-1]), dtype=torch.float64, device="cuda")
    order = np.argsort(n, kind="stable")
    for periodic in (0, 1):
        ids = order[per[order] == periodic]
        for part in np.array_split(ids, 16):  # systems of similar length, padded to the longest
            if not len(part):
                continue
            m = int(n[part].max())
            k = np.arange(m)[:, None]
            have = torch.from_numpy(k < n[part][None, :]).cuda()
            at = torch.from_numpy(np.minimum(off[part][None, :] + k, int(off[-1]) - 1)).cuda()
            A, B, C, D = (torch.where(have, x.double()[at], torch.full((), fill, dtype=torch.float64,
                                                                      device="cuda"))
                          for x, fill in zip(arrays, (0.0, 1.0, 0.0, 0.0)))
            last = torch.from_numpy(n[part] - 1).cuda()[None, :]
            c_last, a_first = C.gather(0, last), A[0].clone()
            C.scatter_(0, last, torch.zeros_like(c_last))
            A[0] = 0.0
            if periodic:  # Sherman-Morrison: T = T' + w z^T on the two corners
                g = -B[0].clone()
                z_last = a_first / g
                B[0] -= g
                B.scatter_(0, last, B.gather(0, last) - c_last * z_last)
                W = torch.zeros_like(D)
                W[0] = g
                W.scatter_(0, last, c_last)
                y, q = _thomas(A, B, C, D), _thomas(A, B, C, W)
                zy = y[0] + z_last * y.gather(0, last)[0]
                zq = q[0] + z_last * q.gather(0, last)[0]
                x = y - q * (zy / (1.0 + zq))
            else:
                x = _thomas(A, B, C, D)
            out[at[have]] = x[have]
    return out


def _const_sweep(D, base):
    """Rows -base, 1 + 2 base (+ base on the two wall rows), -base along axis 0."""
    n = D.shape[0]
    A = torch.full((n, 1), -base, dtype=torch.float64, device="cuda")
    B = torch.full((n, 1), 1.0 + 2.0 * base, dtype=torch.float64, device="cuda")
    B[0] += base
    B[-1] += base
    return _thomas(A, B, A, D.reshape(n, -1)).reshape(D.shape)


def _exact_heat(case, seed):
    """One theta-scheme ADI step with reflection ghosts 2 u_wall - u."""
    th = _heat_inputs(case, seed)
    ix, iy, iz = case["ix"], case["iy"], case["iz"]
    dt = _heat_dt(case)
    bx, by, bz = (dt / (2.0 * (2.0 / n) ** 2) for n in (ix, iy, iz))
    cx, cy, cz = (torch.cos(PI * _centres(n)[1:-1]) for n in (ix, iy, iz))
    cx, cy, cz = cx[None, None, :], cy[None, :, None], cz[:, None, None]
    f = th.clone()
    c = (slice(1, -1),) * 3
    t = th[c]
    walls = []  # base * (ghost + cell) of the low and high wall of each direction
    for axis, wall, base in ((0, -cx * cy, bz), (1, -cx * cz, by), (2, -cy * cz, bx)):
        for side, edge in ((0, 0), (-1, -1)):
            cell = t.select(axis, edge)
            ghost = 2.0 * wall.select(axis, 0) - cell
            f.select(axis, side)[1:-1, 1:-1] = ghost
            walls.append(base * (ghost + cell))
    rhs = (bx * (f[1:-1, 1:-1, 2:] + f[1:-1, 1:-1, :-2])
           + by * (f[1:-1, 2:, 1:-1] + f[1:-1, :-2, 1:-1])
           + bz * (f[2:, 1:-1, 1:-1] + f[:-2, 1:-1, 1:-1])
           + (1.0 - 2.0 * (bx + by + bz)) * t + dt * 3.0 * PI * PI * cx * cy * cz)
    for axis, base in ((0, bz), (1, by), (2, bx)):
        rhs.select(axis, 0).add_(walls[2 * axis])
        rhs.select(axis, -1).add_(walls[2 * axis + 1])
        rhs = _const_sweep(rhs.movedim(axis, 0).contiguous(), base).movedim(0, axis).contiguous()
    th[c] = rhs
    return th


def _metrics(n, length, gamma, periodic):
    """Cell sizes and centre spacings of an axis, ghosts included."""
    if gamma:
        xf = [0.5 * length * (1.0 - math.tanh(gamma * (1.0 - 2.0 * i / n)) / math.tanh(gamma))
              for i in range(n + 1)]
    else:
        xf = [length * i / n for i in range(n + 1)]
    xc = [0.0] + [0.5 * (xf[i - 1] + xf[i]) for i in range(1, n + 1)] + [0.0]
    xc[0] = xc[n] - length if periodic else 2.0 * xf[0] - xc[1]
    xc[n + 1] = xc[1] + length if periodic else 2.0 * xf[n] - xc[n]
    dx = [0.0] + [xf[i] - xf[i - 1] for i in range(1, n + 1)] + [0.0]
    dx[0], dx[n + 1] = (dx[n], dx[1]) if periodic else (dx[1], dx[n])
    dm = [0.0] + [xc[i] - xc[i - 1] for i in range(1, n + 2)]
    dm[0] = dm[n] if periodic else dm[1]
    return dx, dm


def _column(v):
    return torch.tensor(v, dtype=torch.float64, device="cuda")[:, None]


def _exact_poisson(case, seed):
    rhs = _poisson_inputs(case, seed)
    n1, n2, nz = case["n1m"], case["n2m"], case["n3m"]
    dz, dm = _metrics(nz, 2.0, case["gamma"], False)
    lx, ly = 4.0 * PI, 2.0 * PI
    kx = torch.arange(n1 // 2 + 1, dtype=torch.float64, device="cuda")
    ky = torch.arange(n2, dtype=torch.float64, device="cuda")
    lam = ((2.0 - 2.0 * torch.cos(2.0 * PI * ky / n2)) * (n2 / ly) ** 2)[:, None] \
        + ((2.0 - 2.0 * torch.cos(2.0 * PI * kx / n1)) * (n1 / lx) ** 2)[None, :]
    a = _column([0.0] + [1.0 / (dz[k + 1] * dm[k + 1]) for k in range(1, nz)])
    c = _column([1.0 / (dz[k + 1] * dm[k + 2]) for k in range(nz - 1)] + [0.0])
    lam = lam.reshape(1, -1).repeat_interleave(2, dim=1)
    A, C = (v.expand(nz, lam.shape[1]).contiguous() for v in (a, c))
    B = -(a + c) - lam
    D = torch.view_as_real(rhs).reshape(nz, -1).clone()
    for k in (0, 1):  # the pinned mean pressure
        A[0, k], B[0, k], C[0, k], D[0, k] = 0.0, 1.0, 0.0, 0.0
    return torch.view_as_complex(_thomas(A, B, C, D).reshape(*rhs.shape, 2))


def _exact_momentum(case, seed):
    """z, y, x sweeps of (1 - c d^2) with no-slip z walls, periodic in x and y."""
    f = _momentum_inputs(case, seed)[1:-1, 1:-1, 1:-1]
    comp, c = case["comp"], case["c"]
    for d, axis, n, length, gamma in ((2, 0, case["nz"], 2.0, 1.5), (1, 1, case["ny"], 2.0 * PI, 0),
                                      (0, 2, case["nx"], 4.0 * PI, 0)):
        dx, dm = _metrics(n, length, gamma, d != 2)
        rows = range(1, n + 1)
        if comp == d:
            ar = [1.0 / (dm[r] * dx[r - 1]) for r in rows]
            cr = [1.0 / (dm[r] * dx[r]) for r in rows]
        else:
            ar = [1.0 / (dx[r] * dm[r]) for r in rows]
            cr = [1.0 / (dx[r] * dm[r + 1]) for r in rows]
        A, C = -c * _column(ar), -c * _column(cr)
        B = 1.0 - A - C
        f = f.movedim(axis, 0).contiguous()
        D = f.reshape(n, -1).clone()
        if d == 2:
            if comp == 2:
                C[0], B[0], D[0] = 0.0, 1.0, 0.0
            else:
                B[0] -= A[0]
                B[-1] -= C[-1]
            A[0], C[-1] = 0.0, 0.0
            x = _thomas(A, B, C, D)
        else:
            x = _thomas_periodic(A, B, C, D)
        f = x.reshape(f.shape).movedim(0, axis)
    q = torch.zeros(case["nz"] + 2, case["ny"] + 2, case["nx"] + 2, dtype=torch.float64,
                    device="cuda")
    q[1:-1, 1:-1, 1:-1] = f
    return q


def exact(case, seed):
    kind = case["kind"]
    if kind == "solve":
        arrays = [x.double() for x in _solve_inputs(case, seed)]
        return (_thomas_periodic if case["periodic"] else _thomas)(*arrays)
    return {"ragged": _exact_ragged, "heat": _exact_heat, "poisson": _exact_poisson,
            "momentum": _exact_momentum}[kind](case, seed)
