"""A state whose sound speed overflows to infinity ends a run or an estimate
with an error: the time step would be zero.  In every kernel that forms the
maximum: the stand-alone one, the sweeps', the short 1D run's."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _level(D, n, precision, method, gamma, boxes=None):
    import bamrex_b200 as bx
    hi = tuple(n - 1 if d < D else 0 for d in range(3))
    return bx.Level(D, (0, 0, 0), hi, [0.0] * D, [1.0] * D, boxes or [((0, 0, 0), hi)],
                    bx.Parm(D, adiabatic=gamma, limiter=1), method=method, cfl=0.5, precision=precision)


def _state(D, n, precision):
    """At rest, rho 0.1, E so large that gamma p / rho overflows and p does
    not."""
    shape = tuple(n if d < D else 1 for d in (2, 1, 0))
    u = np.zeros((D + 2,) + shape)
    u[0] = 0.1
    u[D + 1] = 1e38 if precision else 5e307
    return u


CASES = [(0, 0, 1.4), (0, 0, 5.0 / 3.0), (0, 5, 1.4), (0, 6, 1.4), (1, 0, 1.4), (1, 0, 5.0 / 3.0), (1, 5, 1.4), (1, 6, 1.4)]


@pytest.mark.parametrize("energy", ["overflow", "inf"])
@pytest.mark.parametrize("precision,method,gamma", CASES)
@pytest.mark.parametrize("D", [1, 2, 3])
def test_estimate_and_run_refuse(D, precision, method, gamma, energy):
    import bamrex_b200 as bx
    n = 24
    lev = _level(D, n, precision, method, gamma)
    u = _state(D, n, precision)
    if energy == "inf":
        u[D + 1] = 1.0
        u[D + 1].reshape(-1)[5] = np.inf
    lev.set_state(u)
    with pytest.raises(bx.BamrexError, match="non-finite time step"):
        lev.estTimeStep()
    with pytest.raises(bx.BamrexError, match="non-finite time step"):
        lev.run(2)
    lev.close()


@pytest.mark.parametrize("precision", [0, 1], ids=["fp64", "fp32_storage"])
@pytest.mark.parametrize("method", [5, 6], ids=["force", "lax_friedrichs"])
@pytest.mark.parametrize("D", [1, 2, 3])
def test_sweeps_report_it(D, method, precision):
    """FORCE and Lax-Friedrichs keep such a uniform state finite, so the
    maximum of the sweep's own updates is what the estimate reads."""
    import bamrex_b200 as bx
    n = 24
    lev = _level(D, n, precision, method, 1.4)
    u = _state(D, n, precision)
    lev.set_state(u)
    lev.advance(0.0, 1e-30 if precision else 1e-160)
    assert np.isfinite(lev.get_state()).all()
    with pytest.raises(bx.BamrexError, match="non-finite time step"):
        lev.estTimeStep()
    lev.close()
