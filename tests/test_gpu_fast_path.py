"""The fast FP64 MUSCL-Hancock / HLLC path in the regimes its rearranged
arithmetic distinguishes, against the CPU oracle (1e-12 relative L-infinity
per component, the parity bar of a step)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

RTOL = 1e-12


def _consv(D, q, eps, gamma=1.4):
    u = q.copy()
    u[1:1 + D] *= q[0]
    u[1 + D] = q[1 + D] / (gamma - 1) + 0.5 * eps * q[0] * (q[1:1 + D] ** 2).sum(0)
    return u


def _states(regime, D, shape, eps, seed, gamma=1.4):
    """Primitive plateaus of three cells (so that limited, unlimited and
    exactly flat differences all occur) with a little noise on half of them."""
    rng = np.random.default_rng(seed)
    nz, ny, nx = shape
    coarse = [max(1, -(-n // 3)) if n > 1 else 1 for n in (nz, ny, nx)]
    up = lambda a: np.kron(a, np.ones([3 if n > 1 else 1 for n in shape]))[:nz, :ny, :nx]  # noqa: E731
    q = np.zeros((D + 2,) + tuple(shape))
    q[0] = up(rng.uniform(0.5, 2.0, coarse))
    for d in range(D):
        q[1 + d] = up(rng.uniform(-0.5, 0.5, coarse))
    q[1 + D] = up(rng.uniform(0.5, 2.0, coarse))
    if regime == "supersonic_up":
        q[1:1 + D] += 6.0
    elif regime == "supersonic_down":
        q[1:1 + D] -= 6.0
    elif regime == "pressure_ratio":
        q[1 + D] *= up(np.where(rng.uniform(size=coarse) < 0.5, 1.0, 1e4))
    elif regime == "rest":
        q[1:1 + D] = 0.0
    if regime != "rest":
        q *= 1.0 + 1e-3 * up(rng.uniform(size=coarse) < 0.5) * rng.standard_normal(q.shape)
    return _consv(D, q, eps, gamma)


@pytest.mark.parametrize("regime", ["subsonic", "supersonic_up", "supersonic_down", "pressure_ratio", "rest"])
@pytest.mark.parametrize("limiter", [0, 1, 2, 3])
@pytest.mark.parametrize("D,eps", [(1, 1.0), (2, 1.0), (3, 0.5)])
def test_fluxes_by_regime(oracle, D, eps, limiter, regime):
    import torch

    import bamrex_b200 as bx
    shape = [38, 17, 9][:D] + [1] * (3 - D)
    g = [n + 4 if d < D else 1 for d, n in enumerate(shape)]
    u = _states(regime, D, (g[2], g[1], g[0]), eps, 11 * D + limiter)
    lo, hi = (0, 0, 0), tuple(n - 1 for n in shape)
    begin = tuple(-2 if d < D else 0 for d in range(3))
    dx, dt = [0.01] * D, 1e-5
    ut = torch.tensor(u, device="cuda")
    for d in range(D):
        ref = oracle.compute_flux(D, 0, d, lo, hi, u, begin, dx, dt,
                                  oracle.Parm(D, adiabatic=1.4, epsilon=eps, limiter=limiter))
        ft = torch.full(ref.shape, float("nan"), dtype=torch.float64, device="cuda")
        bx.compute_flux(0, d, D, (lo, hi), ft, lo, ut, begin, dx, dt,
                        bx.Parm(D, adiabatic=1.4, epsilon=eps, limiter=limiter))
        got = ft.cpu().numpy()
        for n in range(D + 2):
            scale = np.max(np.abs(ref[n]))
            assert np.max(np.abs(got[n] - ref[n])) <= RTOL * (scale if scale > 0 else 1.0), (d, n)


@pytest.mark.parametrize("regime", ["subsonic", "supersonic_up", "supersonic_down", "pressure_ratio", "rest"])
@pytest.mark.parametrize("gamma", [5.0 / 3.0, 1.5, 1.25, 1.3], ids=["k5", "k6", "k10", "pow"])
@pytest.mark.parametrize("limit", ["energy", "own", "primitive"])
def test_general_path_by_regime(oracle, limit, gamma, regime):
    """The general path: integer roots 1/z = 5, 6, 10 and pow(), limited on
    the energy, on each component's own ratio, and on primitive variables."""
    import torch

    import bamrex_b200 as bx
    D, shape = 2, (17, 38)
    kw = {"energy": {}, "own": dict(limiter_indices=list(range(4)) + [0] * 4, limit_on_primv=[False] * 8),
          "primitive": dict(limiter_indices=[3, 1, 2, 3] + [0] * 4, limit_on_primv=[True] * 4 + [False] * 4)}[limit]
    lo, hi, begin = (0, 0, 0), (shape[1] - 1, shape[0] - 1, 0), (-2, -2, 0)
    dx, dt = [0.01] * D, 1e-5
    for limiter in range(4):
        u = _states(regime, D, (1, shape[0] + 4, shape[1] + 4), 1.0, 5 + limiter, gamma)
        ut = torch.tensor(u, device="cuda")
        for d in range(D):
            ref = oracle.compute_flux(D, 0, d, lo, hi, u, begin, dx, dt,
                                      oracle.Parm(D, adiabatic=gamma, limiter=limiter, **kw))
            ft = torch.full(ref.shape, float("nan"), dtype=torch.float64, device="cuda")
            bx.compute_flux(0, d, D, (lo, hi), ft, lo, ut, begin, dx, dt,
                            bx.Parm(D, adiabatic=gamma, limiter=limiter, **kw))
            got = ft.cpu().numpy()
            for n in range(D + 2):
                scale = np.max(np.abs(ref[n]))
                assert np.max(np.abs(got[n] - ref[n])) <= RTOL * (scale if scale > 0 else 1.0), (limiter, d, n)


def test_gamma_beside_seven_fifths(oracle):
    """A gamma within 1e-12 of 1.4 but not its rounding: a request for the
    TMA kernels is still taken, by the general register kernels."""
    import bamrex_b200 as bx
    from bamrex_b200 import problems
    gamma = 1.4 * (1 + 2e-14)
    n = 24
    u0 = problems.quadrant_2d(n)
    lev = bx.Level(2, (0, 0, 0), (n - 1, n - 1, 0), [0.0, 0.0], [1.0, 1.0], [((0, 0, 0), (n - 1, n - 1, 0))],
                   bx.Parm(2, adiabatic=gamma, limiter=0), cfl=0.8, staging=bx.STAGING_TMA)
    assert [lev.staging(d) for d in range(2)] == [bx.STAGING_REGISTERS] * 2
    lev.set_state(u0)
    dt = lev.estTimeStep()
    lev.advance(0.0, dt)
    lay = oracle.LevelLayout(2, (0, 0, 0), (n - 1, n - 1, 0), [((0, 0, 0), (n - 1, n - 1, 0))], 2, lev.dx)
    ref, _, _ = oracle.run_level(lay, u0, oracle.Parm(2, adiabatic=gamma, limiter=0), 0, 0.8, nsteps=1, fixed_dt=dt)
    got = lev.get_state()
    for c in range(4):
        assert np.max(np.abs(got[c] - ref[c])) <= RTOL * np.max(np.abs(ref[c]))
