"""The rigid body's extrapolation sweeps of 2D regions by their number of
rows: one warp, a few warps one behind the other, more warps than that, and
rows around the warps' edges; against the CPU restatement, by the bar of
test_gpu_gfm.py (1e-12 of the largest value per component)."""
import pytest

from test_gpu_gfm import RTOL, _flow, rel_linf

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [(9, 8), (30, 33), (13, 37), (40, 68), (16, 69), (20, 101), (14, 132), (12, 150), (64, 64)],
                         ids=str)
def test_sweep_rows(oracle, n):
    import bamrex_b200 as bx
    from oracle import gfm_oracle as G
    h = 1.0 / 64  # square cells: an interface cell's reflection stays in the ghost cells
    box = ((0, 0, 0), (n[0] - 1, n[1] - 1, 0))
    lay = oracle.LevelLayout(2, (0, 0, 0), box[1], [box], 4, [h, h], bc_lo=(0,) * 3, bc_hi=(0,) * 3)
    lev = bx.Level(2, (0, 0), (n[0] - 1, n[1] - 1), [0.0] * 2, [n[0] * h, n[1] * h], [box], bx.Parm(2), ngrow=4,
                   bc_lo=[0] * 2, bc_hi=[0] * 2)
    # a slanted plane with the fluid in one corner: nearly all rows are swept
    x = dict(kind=bx.SDF_PLANE, center=(3.2 * h, 3.2 * h, 0.0), axis=(-1.0, -0.7, 0.0))
    body = None
    for sign in (1, -1):
        x["axis"] = (-sign * 1.0, -sign * 0.7, 0.0)
        shapes = [G.make_shape(x["kind"], x["center"], x["axis"], 0.0, False)]
        lev.set_body([x])
        if lev.body_counts()[1] > n[0] * n[1] // 3:
            body = G.Body(lay, shapes, bx.SDF_UNION, (0.0, 0.0))
            break
    assert body is not None
    u0 = _flow(2, n, seed=n[1])
    lev.set_state(u0)
    lev.fill_body_ghosts()
    got = lev.get_state()
    buf = lay.alloc()
    lay.scatter(buf, u0)
    lay.fill_boundary(buf)
    assert G.fill_rb(lay, buf, body, 0, 1.4, 1.0) == 0
    err = rel_linf(got, lay.gather(buf))
    assert err <= RTOL, err
    lev.close()
