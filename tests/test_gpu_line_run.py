"""Runs of a short 1D box in one launch: the same steps as the sweeps', at the
sizes around a warp's 30 cells, a block's 16 chunks and the line's last
length, with an even and an odd number of steps, a stop time, and a run
longer than one launch's steps.  A level that is being timed takes the
sweeps, which is what these compare against: FP32 storage bit for bit, FP64
by the parity bar of a step (1e-12 of the largest value) times the steps."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SIZES = [1, 3, 4, 5, 29, 30, 31, 60, 61, 400, 480, 481, 1201, 1920, 1921]


def _levels(n, bc, method, limiter, gamma, precision):
    import bamrex_b200 as bx
    out = []
    for timed in (False, True):
        lev = bx.Level(1, (0, 0, 0), (n - 1, 0, 0), [0.0], [1.0], [((0, 0, 0), (n - 1, 0, 0))],
                       bx.Parm(1, adiabatic=gamma, limiter=limiter), method=method, bc_lo=[bc] * 3, bc_hi=[bc] * 3,
                       precision=precision)
        lev.set_timing(timed)
        out.append(lev)
    return out


def _state(n, seed):
    from bamrex_b200 import problems
    u = problems.random_states(1, (1, 1, n), seed=seed)
    u[:, :, :, n // 2:] *= 0.35
    return u


def _same(a, b, precision, steps):
    for c in range(3):
        if precision:
            assert np.array_equal(a[c], b[c])
        else:
            assert np.max(np.abs(a[c] - b[c])) <= steps * 1e-12 * np.max(np.abs(b[c]))


@pytest.mark.parametrize("precision", [0, 1], ids=["fp64", "fp32_storage"])
@pytest.mark.parametrize("method,limiter,gamma", [(0, 0, 1.4), (0, 1, 1.4), (0, 2, 1.4), (0, 3, 1.4), (0, 1, 5.0 / 3.0),
                                                  (1, 0, 1.4), (4, 2, 1.4), (5, 0, 1.4), (6, 0, 1.4)])
def test_run_matches_sweeps(method, limiter, gamma, precision):
    for i, n in enumerate(SIZES):
        steps, bc = 3 + i % 2, i % 3
        one, ref = _levels(n, bc, method, limiter, gamma, precision)
        u = _state(n, 11 * n + method)
        got = []
        for lev in (one, ref):
            lev.set_state(u)
            t1, k1 = lev.run(steps)
            # a second run from the other buffer, ended by its stop time
            t2, k2 = lev.run(50, stop_time=t1 * (1 + 1.5 / steps), time=t1)
            got.append((t1, k1, t2, k2, lev.get_state()))
        assert got[0][1] == got[1][1] == steps and got[0][3] == got[1][3]
        rt = 0 if precision else 1e-12 * (steps + got[1][3])
        assert abs(got[0][0] - got[1][0]) <= rt * got[1][0] and abs(got[0][2] - got[1][2]) <= rt * got[1][2]
        _same(got[0][4], got[1][4], precision, steps + got[1][3])


def test_long_run_and_bad_state():
    one, ref = _levels(40, 0, 0, 1, 1.4, 1)
    u = _state(40, 5)
    got = []
    for lev in (one, ref):
        lev.set_state(u)
        got.append((lev.run(4099), lev.get_state()))
        assert lev.run(0, time=0.25) == (0.25, 0)
    assert got[0][0] == got[1][0] and np.array_equal(got[0][1], got[1][1])
    for bad in (np.nan, np.inf, -1.0):
        u[2, 0, 0, 7] = bad
        ends = []
        for lev in (one, ref):
            lev.set_state(u)
            try:
                ends.append(lev.run(3))
            except Exception as e:
                ends.append(str(e))
        assert ends[0] == ends[1], bad
