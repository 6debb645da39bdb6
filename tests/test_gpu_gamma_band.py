"""FP32 storage takes any 1/z near 7 by its exponential and logarithm, so a
gamma that misses 7/5 by more than its rounding (but by less than 1e-12) keeps
the fast kernels there, and gives the bits of 7/5: the constants agree in
single precision."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("staging", [0, 1, 2, 3], ids=["auto", "registers", "tma", "wave"])
@pytest.mark.parametrize("D", [1, 2, 3])
def test_fp32_keeps_the_fast_kernels(D, staging):
    import bamrex_b200 as bx
    from bamrex_b200 import problems
    if D == 1 and staging > 1:
        pytest.skip("the staged kernels are 2D and 3D")
    n = [4000, 96, 32][D - 1]
    hi = tuple(n - 1 if d < D else 0 for d in range(3))
    u0 = problems.random_states(D, tuple(n if d < D else 1 for d in (2, 1, 0)), seed=3)
    out, kinds = [], []
    for gamma in (1.4, 1.4 * (1 + 2e-14)):
        lev = bx.Level(D, (0, 0, 0), hi, [0.0] * D, [1.0] * D, bx.decompose(D, (0, 0, 0), hi, n), bx.Parm(D, adiabatic=gamma, limiter=1),
                       cfl=0.5, precision=bx.FP32_STORAGE, staging=staging)
        lev.set_state(u0)
        lev.run(3)
        kinds.append([lev.staging(d) for d in range(D)])
        out.append(lev.get_state())
        lev.close()
    assert kinds[0] == kinds[1]
    np.testing.assert_array_equal(out[1], out[0])
