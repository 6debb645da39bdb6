"""HLLC faces that are supersonic: the flux is the upwind state's own, whatever
the Mach number (HLLC.cpp:101-167 takes it as it stands).  The bars count
roundings, in ulps of 2^-52: the density's quotient (rho d) (1 / d) is 2, the
velocity 1.5, so the mass flux is within 4; the momentum adds a velocity and a
sum: 6; the energy flux is the sum of an energy (2) and a pressure (2 of the
energy at gamma 5/3, 3 in three dimensions) times a velocity: 8, taken of the
terms without their cancellation."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

ULP = 2.0 ** -52
MACHS = [1.5, 10.0, 1e2, 1e3, 1e4, 1e6, 1e9, 1e17]


def _rows(D, d, n, gamma, sign, cold, seed):
    """Uniform lines along d, one Mach number each (normal velocity of order
    one, or pressure of order one when not cold)."""
    rng = np.random.default_rng(seed)
    m = len(MACHS)
    grid = [1, 1, 1]
    grid[2 - d] = n
    if D > 1:
        grid[2 - (0 if d else 1)] = m
    line = [1, 1, 1]
    if D > 1:
        line[2 - (0 if d else 1)] = m
    mach = np.array(MACHS if D > 1 else [MACHS[seed % m]]).reshape(line)
    rho = rng.uniform(0.5, 2.0, line)
    p = rng.uniform(0.5, 2.0, line)
    v = mach * np.sqrt(gamma * p / rho)
    if cold:
        p, v = p / v ** 2, np.ones_like(v) * rng.uniform(1.0, 2.0, line)
        p *= v ** 2
    q = np.zeros((D + 2,) + tuple(line))
    q[0], q[1 + d], q[D + 1] = rho, sign * v, p
    for e in range(D):
        if e != d:
            q[1 + e] = rng.uniform(-0.5, 0.5, line) * v
    u = q.copy()
    u[1:1 + D] *= q[0]
    u[D + 1] = p / (gamma - 1) + 0.5 * rho * (q[1:1 + D] ** 2).sum(0)
    return np.ascontiguousarray(np.broadcast_to(u, (D + 2,) + tuple(grid)))


def _check(D, d, gamma, u, got):
    """Against the physical flux of u in extended precision; got's cells along
    d are faces of a uniform line, so u's line is compared as it is."""
    U = u.astype(np.longdouble)[(slice(None),) * (3 - d) + (slice(0, 1),)]
    g = np.longdouble(gamma)
    vel = U[1:1 + D] / U[0]
    kin = (U[1:1 + D] * vel).sum(0) / 2
    p = (g - 1) * (U[D + 1] - kin)
    F = np.empty_like(U)
    F[0] = U[1 + d]
    size = np.empty_like(U)  # the terms' size, without their cancellation
    for e in range(D):
        F[1 + e] = U[1 + d] * vel[e] + (p if e == d else 0)
        size[1 + e] = abs(U[1 + d] * vel[e]) + (abs(p) + (g - 1) * kin if e == d else 0)
    F[D + 1] = (U[D + 1] + p) * vel[d]
    size[D + 1] = (U[D + 1] + abs(p)) * abs(vel[d])
    size[0] = abs(U[1 + d])
    for c in range(D + 2):
        err = float(np.max(np.abs(got[c] - F[c]) / size[c]) / ULP)
        assert err <= (4 if c == 0 else 8 if c == D + 1 else 6), (c, err)


@pytest.mark.parametrize("cold", [False, True], ids=["pressure_one", "cold"])
@pytest.mark.parametrize("sign", [1, -1])
@pytest.mark.parametrize("method,gamma", [(0, 1.4), (0, 5.0 / 3.0), (0, 1.3), (1, 1.4), (1, 5.0 / 3.0)])
@pytest.mark.parametrize("D", [1, 2, 3])
def test_flux_of_uniform_lines(D, method, gamma, sign, cold):
    import torch

    import bamrex_b200 as bx
    n = 40
    for d in range(D):
        for seed in range(len(MACHS) if D == 1 else 2):
            u = _rows(D, d, n + 4, gamma, sign, cold, seed)
            lo = (0, 0, 0)
            shape = u.shape[:0:-1]  # cells along x, y, z
            hi = tuple(shape[e] - 1 - (4 if e == d else 0) for e in range(3))
            begin = tuple(-2 if e == d else 0 for e in range(3))
            faces = tuple(shape[e] - (3 if e == d else 0) for e in (2, 1, 0))
            ft = torch.full((D + 2,) + faces, float("nan"), dtype=torch.float64, device="cuda")
            v = np.max(np.abs(u[1 + d] / u[0]))
            bx.compute_flux(method, d, D, (lo, hi), ft, lo, torch.tensor(u, device="cuda"), begin, [0.01] * D,
                            1e-4 / v, bx.Parm(D, adiabatic=gamma, limiter=1))
            _check(D, d, gamma, u, ft.cpu().numpy())


@pytest.mark.parametrize("sign", [1, -1])
@pytest.mark.parametrize("D", [1, 2, 3])
def test_flux_between_states(D, sign):
    """compute_flux_LR's HLLC with the same state on both sides."""
    import torch

    import bamrex_b200 as bx
    n = 12
    for d in range(D):
        u = _rows(D, d, n + 2, 1.4, sign, True, 3)
        lo, shape = (0, 0, 0), u.shape[:0:-1]
        hi = tuple(shape[e] - 1 - (2 if e == d else 0) for e in range(3))
        begin = tuple(-1 if e == d else 0 for e in range(3))
        faces = tuple(shape[e] - (1 if e == d else 0) for e in (2, 1, 0))
        ft = torch.full((D + 2,) + faces, float("nan"), dtype=torch.float64, device="cuda")
        ut = torch.tensor(u, device="cuda")
        bx.compute_flux_LR(bx.HLLC, d, D, (lo, hi), ft, lo, ut, ut, begin, [0.01] * D, 1e-4, bx.Parm(D))
        _check(D, d, 1.4, u, ft.cpu().numpy())


def _regime(D, shape, mach, seed):
    """Plateaus of three cells, normal velocity of order one, pressures by the
    Mach number."""
    rng = np.random.default_rng(seed)
    coarse = [max(1, -(-n // 3)) if n > 1 else 1 for n in shape]
    up = lambda a: np.kron(a, np.ones([3 if n > 1 else 1 for n in shape]))[:shape[0], :shape[1], :shape[2]]  # noqa: E731
    q = np.zeros((D + 2,) + tuple(shape))
    q[0] = up(rng.uniform(0.5, 2.0, coarse))
    for e in range(D):
        q[1 + e] = 3.0 + up(rng.uniform(-0.5, 0.5, coarse)) / mach
    q[D + 1] = up(rng.uniform(0.5, 2.0, coarse)) * 9.0 / mach ** 2
    u = q.copy()
    u[1:1 + D] *= q[0]
    u[D + 1] = q[D + 1] / 0.4 + 0.5 * q[0] * (q[1:1 + D] ** 2).sum(0)
    return u


@pytest.mark.parametrize("mach", [1e2, 1e3, 1e4])
@pytest.mark.parametrize("method", [0, 1])
@pytest.mark.parametrize("D", [1, 2, 3])
def test_jumps_at_high_mach(oracle, D, method, mach):
    """Against the oracle by the parity bar of a step.  The bar covers the
    fluxes: the oracle's own pressure carries E's rounding, mach^2 of it."""
    import torch

    import bamrex_b200 as bx
    shape = [38, 17, 9][:D] + [1] * (3 - D)
    u = _regime(D, [shape[e] + (4 if e < D else 0) for e in (2, 1, 0)], mach, 7)
    lo, hi = (0, 0, 0), tuple(s - 1 for s in shape)
    begin = tuple(-2 if e < D else 0 for e in range(3))
    for d in range(D):
        ref = oracle.compute_flux(D, method, d, lo, hi, u, begin, [0.01] * D, 1e-5, oracle.Parm(D, limiter=1))
        ft = torch.full(ref.shape, float("nan"), dtype=torch.float64, device="cuda")
        bx.compute_flux(method, d, D, (lo, hi), ft, lo, torch.tensor(u, device="cuda"), begin, [0.01] * D, 1e-5,
                        bx.Parm(D, limiter=1))
        got = ft.cpu().numpy()
        for c in range(D + 2):
            assert np.max(np.abs(got[c] - ref[c])) <= 1e-12 * np.max(np.abs(ref[c])), (d, c)
