"""Which register kernel a level's x sweep takes by itself, on both sides of
the lines between them, and that the choice does not show in the results: the
automatic level's bits are those of either kernel asked for."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

ROWS, MARCH = 1, 2
OWN = dict(limiter_indices=[0, 1, 2, 3, 4, 0, 0, 0], limit_on_primv=[False] * 8)
# (dimension, method, gamma, limiting, precision): widest rows that march
CASES = [(2, 0, 1.4, None, 0, 20), (2, 0, 1.4, None, 1, 0), (3, 0, 1.4, None, 0, 12), (3, 0, 1.4, None, 1, 14),
         (3, 5, 1.4, None, 0, 14), (3, 6, 1.4, None, 1, 12), (3, 4, 1.4, None, 0, 16), (3, 1, 1.4, None, 1, 32),
         (3, 0, 5.0 / 3.0, None, 0, 24), (3, 0, 5.0 / 3.0, None, 1, 40), (3, 0, 1.4, OWN, 1, 100)]


@pytest.mark.parametrize("D,method,gamma,limiting,precision,line", CASES)
def test_line(D, method, gamma, limiting, precision, line):
    import bamrex_b200 as bx
    from bamrex_b200 import problems
    parm = bx.Parm(D, adiabatic=gamma, limiter=1, **(limiting or {}))
    for w, want in ((line, MARCH), (line + 1, ROWS)):
        if w == 0 or (limiting and want == ROWS):
            continue
        n = [2 * w, 12, 6 if D == 3 else 1]
        hi = tuple(m - 1 for m in n)
        boxes = [((0, 0, 0), (w - 1, hi[1], hi[2])), ((w, 0, 0), (2 * w - 1, hi[1], hi[2]))]
        u0 = problems.random_states(D, (n[2], n[1], n[0]), seed=w)
        outs = []
        for mode in (bx.XSWEEP_AUTO, bx.XSWEEP_ROWS, bx.XSWEEP_MARCH):
            lev = bx.Level(D, (0, 0, 0), hi, [0.0] * D, [1.0] * D, boxes, parm, method=method, cfl=0.4,
                           bc_lo=(1,) * 3, bc_hi=(1,) * 3, precision=precision, x_mode=mode)
            assert lev.x_mode == (want if mode == bx.XSWEEP_AUTO else mode)
            lev.set_state(u0)
            lev.run(3)
            outs.append(lev.get_state())
            lev.close()
        np.testing.assert_array_equal(outs[1], outs[0])
        np.testing.assert_array_equal(outs[2], outs[0])
