"""The workloads whose speed and results are tracked, through the package's
public calls: whole levels of the explicit path (1D, 2D, 3D; one box or many;
FP64 and FP32 storage; the default and the general limiting), the per-box
Fluxes.H calls, a subcycled AMR hierarchy, the pressure solve, the IMEX step
and a rigid body.

listed() names the cases, draw(rng) gives another one of the same ranges,
prepare(case, seed) makes the inputs and handles a program holds before the
call, run(state) is one pass through the library, work(case) what a pass
cannot do without, and exact(case, seed) the same pass in 64 bits by plain
torch operations.
"""
import math

import numpy as np
import torch

from bamrex_b200 import _abi
from bamrex_b200.amr import Amr
from bamrex_b200.helmholtz import Helmholtz
from bamrex_b200.imex import Imex
from bamrex_b200.level import Level, Parm, compute_flux, conservative_update

LIMITERS = {"minbee": _abi.MINBEE, "van_leer": _abi.VAN_LEER, "van_albada": _abi.VAN_ALBADA,
            "superbee": _abi.SUPERBEE}
METHODS = {"muscl": _abi.MUSCL_HANCOCK, "slic": _abi.SLIC, "hllc": _abi.HLLC, "force": _abi.FORCE}
BCS = {"transmissive": _abi.BC_TRANSMISSIVE, "periodic": _abi.BC_PERIODIC, "reflective": _abi.BC_REFLECTIVE}
AMR_BLOCK = 32
DEV = "cuda" if torch.cuda.is_available() else "cpu"


# ------------------------------------------------------------------ the cases
def level_case(name, dim, nx, ny=1, nz=1, box=0, steps=4, precision="f64", limiter="minbee", method="muscl",
               gamma=1.4, limit="energy", bc="transmissive", drive="run", body=False):
    c = dict(kind="level", dim=dim, nx=nx, ny=ny, nz=nz, box=box, steps=steps, precision=precision, limiter=limiter,
             method=method, gamma=gamma, limit=limit, bc=bc, drive=drive, body=body)
    return dict(name=name, **c) if name else c


def listed():
    return [
        # a shock tube: the smallest runs, all launch latency
        level_case("sod_1d_400", 1, 400, steps=50, limiter="van_leer"),
        # the four-quadrant Riemann problem on one 4096^2 box, both precisions
        level_case("quadrant_2d_4096", 2, 4096, 4096, steps=8),
        level_case("quadrant_2d_4096_fp32", 2, 4096, 4096, steps=8, precision="f32"),
        # an ordinary level in max_grid_size boxes with ragged edges, stepped
        # by the host as an AMReX driver does (estTimeStep, advance)
        level_case("boxes_2d_64", 2, 1000, 1030, box=64, steps=8, limiter="van_leer", bc="reflective",
                   drive="advance"),
        # a 3D blast level of 64^3 boxes
        level_case("blast_3d_256", 3, 256, 256, 256, box=64, steps=4),
        # another gas and every component limited on its own ratio: the
        # general kernels
        level_case("general_2d", 2, 1024, 768, box=256, steps=4, limiter="van_albada", gamma=5.0 / 3.0,
                   limit="self", bc="periodic"),
        # the centred scheme on small ragged 3D boxes
        level_case("slic_3d", 3, 100, 80, 112, box=32, steps=4, method="slic", limiter="superbee",
                   bc="reflective"),
        # the per-box calls a host code with its own fabs makes: three face
        # fluxes and the unsplit update of one box
        dict(name="box_fluxes_3d", kind="box", dim=3, nx=64, ny=64, nz=64, method="muscl", limiter="van_leer"),
        # a subcycled three-level blast hierarchy, fixed grids between regrids
        dict(name="amr_blast_3d", kind="amr", dim=3, n0=128, steps=2, precision="f64"),
        # the low-Mach pressure equation, new density each solve
        dict(name="pressure_2d_2048", kind="pressure", nx=2048, ny=2048),
        # whole IMEX steps of a low-Mach state
        dict(name="imex_2d", kind="imex", nx=512, ny=384, steps=6),
        # flow past a cylinder: ghost-fluid fill and step
        level_case("cylinder_2d", 2, 1024, 1024, box=64, steps=4, body=True),
    ]


def _log_int(rng, lo, hi, odd=True):
    n = int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))
    if not odd:
        n = max(32, n // 32 * 32)
    return n


def draw(rng):
    kind = rng.choice(["level2"] * 5 + ["level3"] * 3 + ["level1", "general", "box", "amr", "pressure", "imex", "body"])
    lim = rng.choice(sorted(LIMITERS))
    bc = rng.choice(sorted(BCS))
    prec = rng.choice(["f64", "f64", "f32"])
    drive = rng.choice(["run", "advance"])
    if kind == "level1":
        return level_case(None, 1, _log_int(rng, 64, 100000), steps=rng.randint(8, 50), limiter=lim, bc=bc,
                          precision=prec)
    if kind == "level2":
        return level_case(None, 2, _log_int(rng, 100, 3500), _log_int(rng, 100, 3500), box=rng.choice([0, 0, 64, 128]),
                          steps=rng.randint(2, 6), limiter=lim, bc=bc, precision=prec, drive=drive)
    if kind == "level3":
        return level_case(None, 3, _log_int(rng, 30, 220), _log_int(rng, 30, 220), _log_int(rng, 30, 220),
                          box=rng.choice([0, 32, 48, 64]), steps=rng.randint(2, 4), limiter=lim, bc=bc, precision=prec,
                          drive=drive)
    if kind == "general":
        return level_case(None, 2, _log_int(rng, 100, 1500), _log_int(rng, 100, 1500), box=rng.choice([0, 64, 256]),
                          steps=rng.randint(2, 4), limiter=lim, gamma=rng.choice([5.0 / 3.0, 1.3]),
                          limit=rng.choice(["energy", "self"]), bc=bc, method=rng.choice(["muscl", "slic"]))
    if kind == "box":
        return dict(kind="box", dim=3, nx=_log_int(rng, 8, 100), ny=_log_int(rng, 8, 100), nz=_log_int(rng, 8, 100),
                    method=rng.choice(sorted(METHODS)), limiter=lim)
    if kind == "amr":
        dim = rng.choice([2, 3])
        return dict(kind="amr", dim=dim, n0=rng.choice([256, 512, 768] if dim == 2 else [64, 96, 128]),
                    steps=rng.randint(1, 3), precision=prec)
    if kind == "pressure":
        return dict(kind="pressure", nx=_log_int(rng, 128, 2048, odd=False), ny=_log_int(rng, 128, 2048, odd=False))
    if kind == "imex":
        return dict(kind="imex", nx=_log_int(rng, 128, 768, odd=False), ny=_log_int(rng, 128, 768, odd=False),
                    steps=rng.randint(2, 6))
    return level_case(None, 2, _log_int(rng, 256, 1500), _log_int(rng, 256, 1500), box=64, steps=rng.randint(2, 4),
                      limiter=lim, body=True)


# ------------------------------------------------------------------ inputs
def _gen(seed):
    return torch.Generator(device=DEV).manual_seed(int(seed))


def _centres(lo, n, total, gen_dev=DEV):
    """Cell centres of indices lo .. lo + n - 1 of `total` cells over [0, 1]."""
    return (torch.arange(lo, lo + n, dtype=torch.float64, device=gen_dev) + 0.5) / total


def _consv(q, gamma, eps=1.0):
    u = torch.empty_like(q)
    u[0] = q[0]
    u[1:-1] = q[0] * q[1:-1]
    u[-1] = q[-1] / (gamma - 1) + 0.5 * eps * q[0] * (q[1:-1] ** 2).sum(0)
    return u


def _grf(shape, corr, g):
    """Unit-variance periodic Gaussian random field, correlation length in cells."""
    w = torch.randn(shape, dtype=torch.float64, device=DEV, generator=g)
    ky = torch.fft.fftfreq(shape[0], dtype=torch.float64, device=DEV)[:, None]
    kx = torch.fft.rfftfreq(shape[1], dtype=torch.float64, device=DEV)[None]
    f = torch.fft.irfft2(torch.fft.rfft2(w) * torch.exp(-0.5 * (2 * math.pi * corr) ** 2 * (kx ** 2 + ky ** 2)), s=shape)
    return (f - f.mean()) / f.std()


def _shape(c):
    return (c["nz"], c["ny"], c["nx"])


def _level_state(c, seed):
    """The initial conserved state (NC, nz, ny, nx) of a level case."""
    g, D, (nz, ny, nx) = _gen(seed), c["dim"], _shape(c)
    r = torch.rand(64, dtype=torch.float64, device=DEV, generator=g).cpu()
    noise = torch.randn((nz, ny, nx), dtype=torch.float64, device=DEV, generator=g)
    X = _centres(0, nx, nx)[None, None, :]
    Y = _centres(0, ny, ny)[None, :, None]
    Z = _centres(0, nz, nz)[:, None, None]
    q = torch.zeros((D + 2, nz, ny, nx), dtype=torch.float64, device=DEV)
    if c["body"]:
        # a Mach 0.3 free stream with a smooth disturbance
        wave = torch.sin(2 * math.pi * (2 * X + r[0])) * torch.sin(2 * math.pi * (3 * Y + r[1]))
        q[0] = 1.0 + 0.05 * wave
        q[1] = 0.3 * math.sqrt(c["gamma"]) + 0.02 * torch.cos(2 * math.pi * (Y + r[2])) + 0 * X
        q[2] = 0.02 * torch.cos(2 * math.pi * (X + r[3])) + 0 * Y
        q[-1] = 1.0 + 0.03 * wave
        q[0] *= 1.0 + 1e-3 * noise
        return _consv(q, c["gamma"])
    if D == 1:
        # Sod's tube, the states and the diaphragm moved a little
        left = (X < 0.5 + 0.1 * (r[0] - 0.5)).expand(nz, ny, nx)
        q[0] = torch.where(left, 1.0 + 0.1 * float(r[1]), 0.125)
        q[-1] = torch.where(left, 1.0 + 0.1 * float(r[2]), 0.1)
    elif D == 2:
        # four quadrant states (rho, u, v, p), mild enough that no limiter
        # drives a cell into vacuum
        for k, m in enumerate([(X > 0.5) & (Y > 0.5), (X <= 0.5) & (Y > 0.5), (X <= 0.5) & (Y <= 0.5),
                               (X > 0.5) & (Y <= 0.5)]):
            m = m.expand(nz, ny, nx)
            a = [float(v) for v in r[4 * k:4 * k + 4]]
            for n, v in enumerate((0.5 + a[0], a[1] - 0.5, a[2] - 0.5, 0.5 + a[3])):
                q[n][m] = v
    else:
        # a spherical blast off the middle
        R2 = sum((W - 0.5 - 0.1 * (float(v) - 0.5)) ** 2 for W, v in zip((X, Y, Z), r[:3]))
        q[0] = 1.0
        q[-1] = torch.where(R2 < 0.2 ** 2, 10.0, 0.1)
    q[0] *= 1.0 + 1e-3 * noise
    return _consv(q, c["gamma"])


def _boxes(dim, n, size):
    """The domain of n = (nx, ny, nz) cells chopped into boxes of at most `size` per side."""
    cuts = [[(a, min(a + (size or m) - 1, m - 1)) for a in range(0, m, size or m)] for m in n]
    return [((x[0], y[0], z[0]), (x[1], y[1], z[1])) for z in cuts[2] for y in cuts[1] for x in cuts[0]]


def _pack(glob, boxes):
    """Box after box, inside a box the components slowest."""
    return torch.cat([glob[:, lo[2]:hi[2] + 1, lo[1]:hi[1] + 1, lo[0]:hi[0] + 1].reshape(-1) for lo, hi in boxes])


def _parm(c):
    D = c["dim"]
    own = c.get("limit", "energy") == "self"
    return Parm(D, adiabatic=c.get("gamma", 1.4), limiter=LIMITERS[c["limiter"]],
                limiter_indices=list(range(D + 2)) if own else None, limit_on_primv=[False] * (D + 2) if own else None)


# the AMR hierarchy: base n0 cells per side and two finer levels (ratio 2) of
# AMR_BLOCK-cell blocks around the blast front, up to two blocks merged in x
def _amr_boxes(c):
    D, n0, r0 = c["dim"], c["n0"], 0.2
    nb = [4 * n0 // AMR_BLOCK if d < D else 1 for d in range(3)]
    e = [(np.arange(m + 1) / m - 0.5) if d < D else np.zeros(2) for d, m in enumerate(nb)]
    near = [np.where((a[:-1] < 0) & (a[1:] > 0), 0.0, np.minimum(abs(a[:-1]), abs(a[1:]))) ** 2 for a in e]
    far = [np.maximum(abs(a[:-1]), abs(a[1:])) ** 2 for a in e]
    tot = lambda v: np.sqrt(v[2][:, None, None] + v[1][None, :, None] + v[0][None, None, :])  # noqa: E731
    fine = (tot(near) < r0 + 0.02) & (tot(far) > r0 - 0.02)
    pad = [(0, (-m) % 2 if d < D else 0) for d, m in enumerate(nb)][::-1]
    f = np.pad(fine, pad)
    for ax, d in ((2, 0), (1, 1), (0, 2)):
        if d < D:
            f = f.reshape(f.shape[:ax] + (f.shape[ax] // 2, 2) + f.shape[ax + 1:]).any(axis=ax + 1)
    mid = f.copy()  # one block more on every side
    for ax, d in ((2, 0), (1, 1), (0, 2)):
        if d < D:
            p = np.pad(mid, [(1, 1) if a == ax else (0, 0) for a in range(3)])
            n = mid.shape[ax]
            mid = np.take(p, range(n), ax) | np.take(p, range(1, n + 1), ax) | np.take(p, range(2, n + 2), ax)
    out = [_boxes(D, [n0 if d < D else 1 for d in range(3)], 64)]
    for mask in (mid, fine):
        bx = []
        nz, ny, nx = mask.shape
        for k in range(nz):
            for j in range(ny):
                i = 0
                while i < nx:
                    if not mask[k, j, i]:
                        i += 1
                        continue
                    w = 2 if i + 1 < nx and mask[k, j, i + 1] else 1
                    lo = [i, j, k]
                    ext = [w, 1, 1]
                    bx.append((tuple(lo[d] * AMR_BLOCK if d < D else 0 for d in range(3)),
                               tuple((lo[d] + ext[d]) * AMR_BLOCK - 1 if d < D else 0 for d in range(3))))
                    i += w
        out.append(bx)
    return out


def _amr_state(c, boxes, lev, seed):
    """The packed initial state of level lev: a blast with 1e-3 density noise."""
    D, n = c["dim"], c["n0"] << lev
    g = _gen(seed * 3 + lev)
    p_in = 5.0 + 10.0 * float(torch.rand(1, generator=_gen(seed), device=DEV, dtype=torch.float64))
    parts = []
    for lo, hi in boxes:
        s = [hi[d] - lo[d] + 1 for d in range(3)]
        ax = [_centres(lo[d], s[d], n) - 0.5 if d < D else torch.zeros(1, dtype=torch.float64, device=DEV)
              for d in range(3)]
        r2 = ax[2][:, None, None] ** 2 + ax[1][None, :, None] ** 2 + ax[0][None, None, :] ** 2
        q = torch.zeros((D + 2, s[2], s[1], s[0]), dtype=torch.float64, device=DEV)
        q[0] = 1.0 + 1e-3 * torch.randn(r2.shape, generator=g, device=DEV, dtype=torch.float64)
        q[-1] = torch.where(r2 < 0.2 ** 2, p_in, 0.1)
        parts.append(_consv(q, 1.4).reshape(-1))
    return torch.cat(parts)


def _pressure_inputs(c, seed):
    """Lognormal density (correlation length 32 cells) at Mach 0.01 and a smooth right-hand side."""
    g = _gen(seed)
    beta = torch.exp(-_grf((c["ny"], c["nx"]), 32, g))[None].contiguous()
    rhs = _grf((c["ny"], c["nx"]), 64, g)[None].contiguous()
    mach, dx = 0.01, 1.0 / c["nx"]
    return beta, rhs, mach * mach / 0.4, (0.8 * dx / mach) ** 2, dx


def _imex_inputs(c, seed):
    """Lognormal density, solenoidal velocity of peak 0.01, uniform pressure."""
    g, s = _gen(seed), (c["ny"], c["nx"])
    rho = torch.exp(_grf(s, 32, g))
    psi = _grf(s, 32, g)
    u = 0.5 * (psi.roll(-1, 0) - psi.roll(1, 0))
    v = -0.5 * (psi.roll(-1, 1) - psi.roll(1, 1))
    k = 0.01 / torch.sqrt(u * u + v * v).max()
    p = torch.full_like(rho, 1 / 1.4)
    U = _consv(torch.stack([rho, u * k, v * k, p])[:, None], 1.4)
    return U.cpu().numpy(), p[None].cpu().numpy()


def _box_input(c, seed):
    """One box with two ghost cells: a smooth state with noise; dt at CFL 0.5."""
    g = _gen(seed)
    s = (c["nz"] + 4, c["ny"] + 4, c["nx"] + 4)
    q = 1.0 + torch.rand((5,) + s, dtype=torch.float64, device=DEV, generator=g)
    q[1:4] = 2 * q[1:4] - 3
    return _consv(q, 1.4).contiguous(), 0.5 / 64 / 4.0


# ------------------------------------------------------------------ prepare and run
def prepare(case, seed):
    c, st = case, {"case": case}
    if c["kind"] == "level":
        D, n = c["dim"], (c["nx"], c["ny"], c["nz"])
        boxes = _boxes(D, n, c["box"])
        st["u0"] = _pack(_level_state(c, seed), boxes)
        st["out"] = torch.empty_like(st["u0"])
        bc = [BCS[c["bc"]]] * 3
        st["level"] = Level(D, (0, 0, 0), tuple(m - 1 for m in n), [0.0] * D, [1.0] * D, boxes, _parm(c),
                            method=METHODS[c["method"]], cfl=0.8, ngrow=4 if c["body"] else 2, bc_lo=bc, bc_hi=bc,
                            precision=_abi.FP32_STORAGE if c["precision"] == "f32" else _abi.FP64)
        if c["body"]:
            st["level"].set_body(dict(kind=_abi.SDF_CYLINDER, center=(0.5, 0.5, 0.0), axis=(0.0, 0.0, 1.0), radius=0.1))
    elif c["kind"] == "box":
        st["u"], st["dt"] = _box_input(c, seed)
        n = (c["nx"], c["ny"], c["nz"])
        st["flux"] = [torch.empty((5,) + tuple(n[q] + (q == d) for q in (2, 1, 0)), dtype=torch.float64, device=DEV)
                      for d in range(3)]
        st["new"] = torch.empty((5, n[2], n[1], n[0]), dtype=torch.float64, device=DEV)
        st["parm"] = _parm(c)
    elif c["kind"] == "amr":
        D, n0 = c["dim"], c["n0"]
        boxes = _amr_boxes(c)
        A = Amr(D, (0, 0, 0), tuple(n0 - 1 if d < D else 0 for d in range(3)), [0.0] * D, [1.0] * D, boxes[0],
                Parm(D, limiter=_abi.MINBEE), cfl=0.8, max_level=2, ref_ratio=2, blocking_factor=8, max_grid_size=64,
                phigrad=[0.1, 0.1], precision=_abi.FP32_STORAGE if c["precision"] == "f32" else _abi.FP64)
        st["u0"] = [_amr_state(c, b, lev, seed) for lev, b in enumerate(boxes)]
        torch.cuda.synchronize()
        for lev in (0, 1, 2):
            if lev:
                A.set_level_boxes(lev, boxes[lev])
            A.level(lev).copy_in_ptr(st["u0"][lev].data_ptr())
        st["amr"], st["out"] = A, [torch.empty_like(u) for u in st["u0"]]
    elif c["kind"] == "pressure":
        st["beta"], st["rhs"], a, B, dx = _pressure_inputs(c, seed)
        st["x"] = torch.zeros_like(st["rhs"])
        st["stream"] = torch.cuda.Stream()
        h = Helmholtz(2, (c["nx"], c["ny"]), [0.0, 0.0], [1.0, dx * c["ny"]], stream=st["stream"])
        h.setScalars(1.0, B, 0.0)
        h.setACoeffs(a)
        st["op"] = h
    else:
        st["U"], st["p"] = _imex_inputs(c, seed)
        n = (c["nx"], c["ny"])
        per = [_abi.BC_PERIODIC] * 3
        st["imex"] = Imex(2, n, [0.0, 0.0], [1.0, n[1] / n[0]], Parm(2), bc_lo=per, bc_hi=per, cfl=0.8)
    torch.cuda.synchronize()
    return st


def run(st):
    c = st["case"]
    if c["kind"] == "level":
        # set the state, take the steps, fetch the state
        lev = st["level"]
        lev.copy_in_ptr(st["u0"].data_ptr())
        t = 0.0
        if c["drive"] == "run":
            t, _ = lev.run(c["steps"])
        else:
            for _ in range(c["steps"]):
                dt = lev.estTimeStep()
                lev.advance(t, dt)
                t += dt
        lev.copy_out_ptr(st["out"].data_ptr())
        lev.sync()
        return {"state": st["out"], "time": t}
    if c["kind"] == "box":
        n = (c["nx"], c["ny"], c["nz"])
        bx = ((0, 0, 0), (n[0] - 1, n[1] - 1, n[2] - 1))
        s = torch.cuda.current_stream()
        h = [1.0 / 64] * 3
        for d in range(3):
            compute_flux(METHODS[c["method"]], d, 3, bx, st["flux"][d], (0, 0, 0), st["u"], (-2, -2, -2), h, st["dt"],
                         st["parm"], stream=s)
        conservative_update(3, bx, st["new"], (0, 0, 0), st["u"], (-2, -2, -2), st["flux"], [(0, 0, 0)] * 3, st["dt"],
                            [64.0] * 3, stream=s)
        return {"flux": st["flux"], "state": st["new"]}
    if c["kind"] == "amr":
        A = st["amr"]
        levels = [A.level(lev) for lev in range(3)]
        for lev, u in zip(levels, st["u0"]):
            lev.copy_in_ptr(u.data_ptr())
        dts = A.run(c["steps"])
        for lev, o in zip(levels, st["out"]):
            lev.copy_out_ptr(o.data_ptr())
        for lev in levels:
            lev.sync()
        return {"levels": st["out"], "dt": dts}
    if c["kind"] == "pressure":
        with torch.cuda.stream(st["stream"]):
            st["op"].setBCoeffsFromCell(st["beta"])
            st["x"].zero_()
            st["op"].solve_device(st["x"], st["rhs"])
        return st["x"]
    im = st["imex"]
    im.set_state(st["U"], st["p"])
    for _ in range(c["steps"]):
        im.step(im.est_time_step())
    U, p = im.get_state()
    return {"state": U, "pressure": p}


# ------------------------------------------------------------------ work
def _flops_per_cell_sweep(c):
    """Additions, multiplications, divisions and roots of one cell in one sweep."""
    return {"muscl": 270, "slic": 190, "hllc": 170, "force": 90}[c.get("method", "muscl")] + 10 * c.get("dim", 2)


def work(case):
    c = case
    if c["kind"] == "level":
        cells, size = c["nx"] * c["ny"] * c["nz"], 4 if c["precision"] == "f32" else 8
        # each sweep of a step reads the state once and writes it once
        return {"bytes": c["steps"] * c["dim"] * 2 * (c["dim"] + 2) * size * cells,
                "flops": c["steps"] * c["dim"] * cells * _flops_per_cell_sweep(c)}
    if c["kind"] == "box":
        cells = c["nx"] * c["ny"] * c["nz"]
        return {"bytes": 8 * 5 * (3 * (cells + cells) + 5 * cells), "flops": 3 * cells * _flops_per_cell_sweep(c)}
    if c["kind"] == "amr":
        size = 4 if c["precision"] == "f32" else 8
        cells = sum((1 << lev) * int(np.prod([hi[d] - lo[d] + 1 for d in range(3)]))
                    for lev, b in enumerate(_amr_boxes(c)) for lo, hi in b)
        return {"bytes": c["steps"] * c["dim"] * 2 * (c["dim"] + 2) * size * cells,
                "flops": c["steps"] * c["dim"] * cells * _flops_per_cell_sweep(c)}
    cells = c["nx"] * c["ny"]
    if c["kind"] == "pressure":
        # about a dozen iterations of two V-cycles of four smoothings (48 B a
        # cell and sweep, a third more on the coarser levels)
        return {"bytes": 12 * 2 * 4 * 48 * 4 // 3 * cells, "flops": 12 * 2 * 4 * 20 * 4 // 3 * cells}
    return {"bytes": c["steps"] * 40 * 48 * cells, "flops": c["steps"] * 40 * 20 * cells}


# ------------------------------------------------------------------ the same in 64 bits
def _prim(U, gamma):
    q = torch.empty_like(U)
    q[0] = U[0]
    q[1:-1] = U[1:-1] / U[0]
    q[-1] = (gamma - 1) * (U[-1] - 0.5 * U[0] * (q[1:-1] ** 2).sum(0))
    return q


def _phys(U, q, d):
    F = U * q[1 + d]
    F[0] = U[1 + d]
    F[1 + d] += q[-1]
    F[-1] = (U[-1] + q[-1]) * q[1 + d]
    return F


def _phi(num, den, lim):
    r = num / torch.where(den == 0, torch.ones_like(den), den)
    if lim == "minbee":
        f = torch.where(r > 1, torch.clamp(2 / (1 + r), max=1.0), r)
    elif lim == "van_leer":
        f = torch.minimum(2 * r / (1 + r), 2 / (1 + r))
    elif lim == "van_albada":
        f = torch.minimum(r * (1 + r) / (1 + r * r), 2 / (1 + r))
    else:
        f = torch.where(r <= 0.5, 2 * r, torch.where(r <= 1, torch.ones_like(r),
                                                     torch.clamp(torch.minimum(r, 2 / (1 + r)), max=2.0)))
    f = torch.where(r <= 0, torch.zeros_like(r), f)
    f = torch.where((den == 0) & (num != 0), torch.zeros_like(f), f)
    return torch.where((den == 0) & (num == 0), torch.ones_like(f), f)


def _hllc(L, R, d, gamma):
    qL, qR = _prim(L, gamma), _prim(R, gamma)
    rL, rR = qL[0].clamp(min=1e-14), qR[0].clamp(min=1e-14)
    pL, pR = qL[-1].clamp(min=1e-14), qR[-1].clamp(min=1e-14)
    uL, uR = qL[1 + d], qR[1 + d]
    cL, cR = torch.sqrt(gamma * pL / rL), torch.sqrt(gamma * pR / rR)
    z = (gamma - 1) / (2 * gamma)
    prr = ((cL + cR - 0.5 * (gamma - 1) * (uR - uL)) / (cL * pL ** -z + cR * pR ** -z)) ** (1 / z)
    g = (gamma + 1) / (2 * gamma)
    SL = uL - cL * torch.where(prr > pL, torch.sqrt(torch.clamp(1 + g * (prr / pL - 1), min=0)), 1.0)
    SR = uR + cR * torch.where(prr > pR, torch.sqrt(torch.clamp(1 + g * (prr / pR - 1), min=0)), 1.0)
    dL, dR = SL - uL, SR - uR
    Ss = (pR - pL + rL * uL * dL - rR * uR * dR) / (rL * dL - rR * dR)
    left = (SL >= 0) | (Ss >= 0)
    star = torch.where(left, SL < 0, SR >= 0)
    U, q, S = torch.where(left, L, R), torch.where(left, qL, qR), torch.where(left, SL, SR)
    F = _phys(U, q, d)
    w = q[0] * (S - q[1 + d])
    V = q.clone()
    V[0] = 1.0
    V[1 + d] = Ss
    V[-1] = U[-1] / q[0] + (Ss - q[1 + d]) * (Ss + q[-1] / w)
    return torch.where(star, F + S * (w / (S - Ss) * V - U), F)


def _force(L, R, d, gamma, dx, dt):
    fL, fR = _phys(L, _prim(L, gamma), d), _phys(R, _prim(R, gamma), d)
    H = 0.5 * (L + R) + dt / (2 * dx) * (fL - fR)
    return 0.5 * (0.5 * dx / dt * (L - R) + 0.5 * (fL + fR)) + 0.5 * _phys(H, _prim(H, gamma), d)


def _face_flux(W, d, gamma, dx, dt, method, lim, limit):
    """Fluxes of the faces of a state with two ghost cells along direction d."""
    ax = 3 - d
    n = W.shape[ax]
    cut = lambda a, b: W.narrow(ax, a, n - b)  # noqa: E731
    if method in ("muscl", "slic"):
        m, o, p = cut(0, 2), cut(1, 2), cut(2, 2)
        if limit == "energy":
            phi = _phi(o[-1] - m[-1], p[-1] - o[-1], lim)
        else:
            phi = _phi(o - m, p - o, lim)
        delta = 0.5 * phi * (0.5 * (o - m) + 0.5 * (p - o))
        L, R = o - delta, o + delta
        h = 0.5 * dt / dx * (_phys(R, _prim(R, gamma), d) - _phys(L, _prim(L, gamma), d))
        L, R = L - h, R - h
        k = n - 3
        left, right = R.narrow(ax, 0, k), L.narrow(ax, 1, k)
    else:
        left, right = W.narrow(ax, 1, n - 3), W.narrow(ax, 2, n - 3)
    if method in ("muscl", "hllc"):
        return _hllc(left, right, d, gamma)
    return _force(left, right, d, gamma, dx, dt)


def _ghosts(U, d, bc):
    ax, n = 3 - d, U.shape[3 - d]
    a, b = U.narrow(ax, 0, min(2, n)), U.narrow(ax, max(0, n - 2), min(2, n))
    if bc == "periodic":
        a, b = b, a
    elif bc == "reflective":
        a, b = a.flip(ax).clone(), b.flip(ax).clone()
        a[1 + d] *= -1
        b[1 + d] *= -1
    else:
        a, b = torch.cat([U.narrow(ax, 0, 1)] * 2, ax), torch.cat([U.narrow(ax, n - 1, 1)] * 2, ax)
    return torch.cat([a, U, b], ax)


def exact(case, seed):
    c = case
    if c["kind"] == "level" and not c["body"]:
        U, D, gamma = _level_state(c, seed), c["dim"], c["gamma"]
        n, t = (c["nx"], c["ny"], c["nz"]), 0.0
        for _ in range(c["steps"]):
            q = _prim(U, gamma)
            speed = (torch.sqrt(gamma * q[-1] / q[0]) + torch.sqrt((q[1:-1] ** 2).sum(0))).max()
            del q
            dt = 0.8 * min(1.0 / n[d] for d in range(D)) / float(speed)
            for d in range(D):
                F = _face_flux(_ghosts(U, d, c["bc"]), d, gamma, 1.0 / n[d], dt, c["method"], c["limiter"], c["limit"])
                m = n[d]
                U = U - dt * n[d] * (F.narrow(3 - d, 1, m) - F.narrow(3 - d, 0, m))
                del F
            t += dt
        return {"state": _pack(U, _boxes(D, n, c["box"])), "time": t}
    if c["kind"] == "box":
        u, dt = _box_input(c, seed)
        n = (c["nx"], c["ny"], c["nz"])
        new, fluxes = u[:, 2:-2, 2:-2, 2:-2].clone(), []
        for d in range(3):
            W = u
            for q in range(3):
                if q != d:
                    W = W.narrow(3 - q, 2, n[q])
            F = _face_flux(W, d, 1.4, 1.0 / 64, dt, c["method"], c["limiter"], "energy")
            fluxes.append(F)
            new -= dt * 64.0 * (F.narrow(3 - d, 1, n[d]) - F.narrow(3 - d, 0, n[d]))
        return {"flux": fluxes, "state": new}
    if c["kind"] == "pressure":
        return _pressure_exact(c, seed)
    return None


def _pressure_exact(c, seed):
    """a x - B div(b grad x) = rhs (periodic, b the mean of the two cells of a
    face) by conjugate gradients, preconditioned with the constant-coefficient
    operator in Fourier space."""
    beta, rhs, a, B, h = _pressure_inputs(c, seed)
    beta, rhs = beta[0], rhs[0]
    k = B / (h * h)
    bx, by = 0.5 * (beta + beta.roll(1, 1)), 0.5 * (beta + beta.roll(1, 0))

    def A(x):
        fx, fy = bx * (x - x.roll(1, 1)), by * (x - x.roll(1, 0))
        return a * x - k * (fx.roll(-1, 1) - fx + fy.roll(-1, 0) - fy)

    ny, nx = rhs.shape
    lam = (2 - 2 * torch.cos(2 * math.pi * torch.fft.fftfreq(ny, dtype=torch.float64, device=DEV)))[:, None] + \
          (2 - 2 * torch.cos(2 * math.pi * torch.fft.rfftfreq(nx, dtype=torch.float64, device=DEV)))[None]
    inv = 1 / (a + k * float(torch.exp(torch.log(beta).mean())) * lam)
    M = lambda r: torch.fft.irfft2(torch.fft.rfft2(r) * inv, s=(ny, nx))  # noqa: E731
    x = torch.zeros_like(rhs)
    r = rhs.clone()
    z = M(r)
    p, rz = z.clone(), (r * z).sum()
    for it in range(2000):
        q = A(p)
        al = rz / (p * q).sum()
        x += al * p
        r -= al * q
        if it % 50 == 49:
            r = rhs - A(x)
        if it % 10 == 9 and float(r.norm()) <= 1e-14 * float(rhs.norm()):
            break
        z = M(r)
        new = (r * z).sum()
        p = z + (new / rz) * p
        rz = new
    return x[None]
