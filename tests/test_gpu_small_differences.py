"""Limiters on differences far below the size of the flow: components and
primitive variables limited on their own ratio pass through every exponent
ahead of a wave (transverse momentum falls by orders of magnitude per cell),
down to subnormal values and zero beside them.  Against the CPU oracle, which
divides the differences."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

RTOL = 1e-12  # the per-step parity bar, relative L-infinity per component
TINY = 200 * 5e-324  # roundings in the subnormal range, where a relative bar means nothing

# successive differences: 0, rising, falling, equal, of both signs, 1/2, 0 beside large
PATTERN = np.array([0, 0, 1, 2, 4, 5, 5, 0, -1, 3, 3.5, 3, 0, 0, 0, 2, 1000, 1001, 999.5, 0, -7, -7, -14, 1e-7, 0, 3])


def _limits(name, D):
    t = D + 1  # the limiting variable: a transverse momentum is D (the last one)
    return {"own": dict(limiter_indices=list(range(D + 2)) + [0] * (6 - D), limit_on_primv=[False] * 8),
            "primitive": dict(limiter_indices=[t] + list(range(1, D + 2)) + [0] * (6 - D),
                              limit_on_primv=[True] * (D + 2) + [False] * (6 - D)),
            "momentum": dict(limiter_indices=[D] * 8, limit_on_primv=[False] * 8)}[name]


def _state(D, d, n, scale, gamma):
    """Plateaus of three cells along d in pressure and normal velocity; the
    last momentum that is not along d follows the pattern times `scale`."""
    rng = np.random.default_rng(17)
    shape = [1, 1, 1]
    shape[2 - d] = n
    along = lambda a: a.reshape(shape)  # noqa: E731
    grid = tuple(n if 2 - e == 2 - d else (3 if e < D else 1) for e in (2, 1, 0))
    step = np.repeat(rng.uniform(0.5, 2.0, n), 3)[:n]
    u = np.zeros((D + 2,) + grid)
    u[0] = 1.25
    u[1 + d] = 1.25 * along(0.3 * step)
    t = D - 1 if d != D - 1 else 0
    u[1 + t] = along(scale * np.resize(PATTERN, n))
    u[D + 1] = along(step) / (gamma - 1) + 0.5 * u[1 + d] ** 2 / 1.25
    return u


@pytest.mark.parametrize("scale", [1.0, 1e-150, 1e-160, 1e-250, 1e-300, 1e-310])
@pytest.mark.parametrize("limit", ["own", "primitive", "momentum"])
@pytest.mark.parametrize("method,gamma", [(0, 5.0 / 3.0), (0, 1.4), (4, 1.4)])
@pytest.mark.parametrize("D", [2, 3])
def test_fluxes(oracle, D, method, gamma, limit, scale):
    import torch

    import bamrex_b200 as bx
    n, kw, dx, dt = 45, _limits(limit, D), [0.01] * D, 1e-4
    for limiter in range(4):
        for d in range(D):
            u = _state(D, d, n + 4, scale if scale < 1 else 1e-3, gamma)
            lo = (0, 0, 0)
            hi = tuple(n - 1 if e == d else (2 if e < D else 0) for e in range(3))
            begin = tuple(-2 if e == d else 0 for e in range(3))
            ref = oracle.compute_flux(D, method, d, lo, hi, u, begin, dx, dt,
                                      oracle.Parm(D, adiabatic=gamma, limiter=limiter, **kw))
            ft = torch.full(ref.shape, float("nan"), dtype=torch.float64, device="cuda")
            bx.compute_flux(method, d, D, (lo, hi), ft, lo, torch.tensor(u, device="cuda"), begin, dx, dt,
                            bx.Parm(D, adiabatic=gamma, limiter=limiter, **kw))
            got = ft.cpu().numpy()
            for c in range(D + 2):
                bar = RTOL * np.max(np.abs(ref[c])) + TINY
                assert np.max(np.abs(got[c] - ref[c])) <= bar, (limiter, d, c)


@pytest.mark.parametrize("limiter", range(4))
@pytest.mark.parametrize("scale", [1e-150, 1e-160, 1e-250])
def test_small_energies(oracle, scale, limiter):
    """The fast path (limiting on the energy) in gas without pressure to speak
    of: the flux is the clamp's sound speed times rounding, so the bar is
    RTOL times density times that speed."""
    import torch

    import bamrex_b200 as bx
    n = 45
    u = np.zeros((3, 1, 1, n + 4))
    u[0] = 1.0
    u[2, 0, 0] = scale * (2000 + np.resize(PATTERN, n + 4))
    lo, hi, begin, dx, dt = (0, 0, 0), (n - 1, 0, 0), (-2, 0, 0), [0.01], 1e-4
    ref = oracle.compute_flux(1, 0, 0, lo, hi, u, begin, dx, dt, oracle.Parm(1, limiter=limiter))
    ft = torch.full(ref.shape, float("nan"), dtype=torch.float64, device="cuda")
    bx.compute_flux(0, 0, 1, (lo, hi), ft, lo, torch.tensor(u, device="cuda"), begin, dx, dt, bx.Parm(1, limiter=limiter))
    assert np.max(np.abs(ft.cpu().numpy() - ref)) <= RTOL * np.sqrt(1.4 * 1e-14)


def jet(n):
    """A jet into gas at rest: its transverse momentum ahead of the waves runs
    down to the smallest numbers."""
    u = np.zeros((4, 1, n, n))
    u[0] = 1.0
    u[3] = 1.0 / (5.0 / 3.0 - 1.0)
    y, x = np.mgrid[0:n, 0:n]
    core = (x < n // 4) & (abs(y - n // 2) < n // 10)
    u[1, 0][core] = 2.0
    u[3, 0][core] += 2.0
    return u


@pytest.mark.parametrize("limiter", range(4))
def test_jet_steps(oracle, limiter):
    import bamrex_b200 as bx
    n, steps, gamma, kw = 96, 60, 5.0 / 3.0, _limits("own", 2)
    u0, box = jet(n), ((0, 0, 0), (n - 1, n - 1, 0))
    lev = bx.Level(2, (0, 0, 0), box[1], [0.0, 0.0], [1.0, 1.0], [box], bx.Parm(2, adiabatic=gamma, limiter=limiter, **kw),
                   cfl=0.5)
    lev.set_state(u0)
    _, done = lev.run(steps)
    got = lev.get_state()
    lev.close()
    lay = oracle.LevelLayout(2, (0, 0, 0), box[1], [box], 2, [1.0 / n] * 2)
    ref, _, dts = oracle.run_level(lay, u0, oracle.Parm(2, adiabatic=gamma, limiter=limiter, **kw), 0, 0.5, nsteps=steps)
    assert done == steps and np.isfinite(got).all()
    for c in range(4):
        assert np.max(np.abs(got[c] - ref[c])) <= steps * RTOL * np.max(np.abs(ref[c])), c
