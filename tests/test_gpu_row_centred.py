"""FORCE and Lax-Friedrichs on the x sweep by row groups, four positions to a
lane: rows around the sizes of a group, a warp's 30 owned groups and a box's
last chunk, paired and not, in the per-box call and on levels."""
import numpy as np
import pytest

from test_gpu_row_sweep import RTOL, WIDTHS, _input

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("method", [5, 6], ids=["force", "lax_friedrichs"])
@pytest.mark.parametrize("shift", [0, 1], ids=["paired", "unpaired"])
@pytest.mark.parametrize("D", [1, 2, 3])
def test_flux_and_update_by_width(oracle, D, shift, method):
    import torch

    import bamrex_b200 as bx
    dx, dt = [0.01] * D, 0.0005
    for w in WIDTHS:
        ny, nz = (3 if D > 1 else 1), (2 if D > 2 else 1)
        g = 2 + shift  # an odd ghost width puts cell lo at an odd element
        u = _input(D, (nz, ny, w + 2 * g), 7 * w + D)
        lo, hi = (0, 0, 0), (w - 1, ny - 1, nz - 1)
        begin = (-g, 0, 0)
        ref = oracle.compute_flux(D, method, 0, lo, hi, u, begin, dx, dt, oracle.Parm(D))
        ut = torch.tensor(u, device="cuda")
        ft = torch.full(ref.shape, float("nan"), dtype=torch.float64, device="cuda")
        out = torch.full((D + 2, nz, ny, w), float("nan"), dtype=torch.float64, device="cuda")
        bx.sweep_box(method, 0, D, (lo, hi), out, lo, ut, begin, dx, dt, bx.Parm(D), flux=ft, flux_begin=lo)
        got, new = ft.cpu().numpy(), out.cpu().numpy()
        want = u[:, :, :, g:g + w] - dt / dx[0] * (ref[:, :, :, 1:] - ref[:, :, :, :-1])
        for n in range(D + 2):
            assert np.max(np.abs(got[n] - ref[n])) <= RTOL * np.max(np.abs(ref[n])), (w, n)
            assert np.max(np.abs(new[n] - want[n])) <= RTOL * np.max(np.abs(want[n])), (w, n)


@pytest.mark.parametrize("precision", [0, 1], ids=["fp64", "fp32_storage"])
@pytest.mark.parametrize("method", [4, 5, 6], ids=["slic", "force", "lax_friedrichs"])
@pytest.mark.parametrize("cuts", [[0, 64, 97, 128, 131, 200], [0, 2, 5, 66, 130], [0, 1, 4, 30, 60, 90, 120]])
def test_boxes_step_like_one_box(cuts, method, precision):
    """Boxes of even and odd widths step bit for bit like one box."""
    import bamrex_b200 as bx
    from bamrex_b200 import problems
    nx, ny = cuts[-1], 24
    u0 = problems.quadrant_2d(nx, ny=ny)
    parts = [((a, y, 0), (b - 1, y + 11, 0)) for y in (0, 12) for a, b in zip(cuts, cuts[1:])]
    outs = []
    for boxes in ([((0, 0, 0), (nx - 1, ny - 1, 0))], parts):
        lev = bx.Level(2, (0, 0, 0), (nx - 1, ny - 1, 0), [0.0, 0.0], [1.0, 1.0], boxes, bx.Parm(2), method=method,
                       cfl=0.6, bc_lo=(1,) * 3, bc_hi=(1,) * 3, x_mode=bx.XSWEEP_ROWS, precision=precision)
        lev.set_state(u0)
        lev.run(3, use_graph=False)
        outs.append(lev.get_state())
        lev.close()
    np.testing.assert_array_equal(outs[1], outs[0])
