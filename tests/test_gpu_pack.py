"""Copies between the level's fabs and the packed layout, and the stand-alone
wave-speed maximum, on boxes whose rows are shorter and longer than a warp and
whose cells do not fill a warp's group."""
import numpy as np
import pytest

import bamrex_b200 as bx
from bamrex_b200.level import Level, Parm

pytestmark = pytest.mark.gpu

LAYOUTS = {
    "1d_1": (1, [((0, 0, 0), (0, 0, 0))]),
    "1d_400": (1, [((0, 0, 0), (399, 0, 0))]),
    "1d_ragged": (1, [((0, 0, 0), (2, 0, 0)), ((3, 0, 0), (133, 0, 0)), ((134, 0, 0), (135, 0, 0))]),
    "2d_one": (2, [((0, 0, 0), (130, 4, 0))]),
    "2d_thin": (2, [((0, 0, 0), (0, 129, 0)), ((1, 0, 0), (2, 129, 0)), ((3, 0, 0), (34, 63, 0)),
                    ((3, 64, 0), (34, 129, 0))]),
    "2d_wide": (2, [((0, 0, 0), (4100, 2, 0)), ((0, 3, 0), (4100, 3, 0))]),
    "3d": (3, [((0, 0, 0), (4, 4, 4)), ((5, 0, 0), (37, 4, 4)), ((0, 5, 0), (37, 6, 4))]),
}


def _level(D, boxes, precision):
    hi = tuple(max(b[1][d] for b in boxes) for d in range(3))
    return Level(D, (0, 0, 0), hi, [0.0] * D, [1.0] * D, boxes, Parm(D, limiter=bx.MINBEE), cfl=0.7,
                 precision=precision)


@pytest.mark.parametrize("fp32", [False, True])
@pytest.mark.parametrize("name", sorted(LAYOUTS))
def test_copy_in_out_and_wave_speed(name, fp32):
    D, boxes = LAYOUTS[name]
    lev = _level(D, boxes, bx.FP32_STORAGE if fp32 else bx.FP64)
    rng = np.random.default_rng(7)
    n = int(lev.ncells)
    q = rng.uniform(1.0, 2.0, (D + 2, n))
    q[1:1 + D] -= 1.5
    u = q.copy()
    u[1:1 + D] *= q[0]
    u[D + 1] = q[D + 1] / 0.4 + 0.5 * q[0] * (q[1:1 + D] ** 2).sum(0)
    if fp32:
        u = u.astype(np.float32).astype(np.float64)
    packed, o = np.empty((D + 2) * n), 0
    for lo, hi in boxes:
        m = int(np.prod([hi[d] - lo[d] + 1 for d in range(3)]))
        packed[(D + 2) * o:(D + 2) * (o + m)] = u[:, o:o + m].reshape(-1)
        o += m
    lev.copy_in_ptr(packed.ctypes.data)
    out = np.full_like(packed, np.nan)
    lev.copy_out_ptr(out.ctypes.data)
    lev.sync()
    assert np.array_equal(out, packed)
    v = u[1:1 + D] / u[0]
    p = 0.4 * (u[D + 1] - 0.5 * u[0] * (v ** 2).sum(0))
    speed = (np.sqrt(1.4 * p / u[0]) + np.sqrt((v ** 2).sum(0))).max()
    ref = 0.7 * min(lev.dx) / speed
    # FP32 storage computes |u| + c in single precision: about ten roundings
    assert abs(lev.estTimeStep() - ref) <= (10 * 2.0 ** -24 if fp32 else 1e-14) * ref
