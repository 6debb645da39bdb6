"""The x sweep by row groups: rows around the sizes of a lane's group (4 or 2
positions), a warp's 30 owned groups and a box's last chunk; rows aligned to
pairs of cells and not; halos read from neighbouring boxes of even and odd
widths."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

RTOL = 1e-12  # the per-step parity bar, relative L-infinity per component

WIDTHS = [1, 2, 3, 4, 5, 7, 8, 26, 55, 56, 57, 112, 115, 116, 117, 118, 235, 236, 237, 500]


def _input(D, shape, seed):
    from bamrex_b200 import problems
    u = problems.random_states(D, shape, seed=seed)
    u[:, :, :, shape[2] // 2:] *= 0.35
    return u


@pytest.mark.parametrize("method,limiter,gamma", [(0, 0, 1.4), (0, 2, 5.0 / 3.0), (4, 1, 1.4), (1, 0, 1.4)])
@pytest.mark.parametrize("shift", [0, 1], ids=["paired", "unpaired"])
@pytest.mark.parametrize("D", [1, 2, 3])
def test_flux_and_update_by_width(oracle, D, shift, method, limiter, gamma):
    import torch

    import bamrex_b200 as bx
    dx, dt = [0.01] * D, 0.0005
    po, pg = oracle.Parm(D, adiabatic=gamma, limiter=limiter), bx.Parm(D, adiabatic=gamma, limiter=limiter)
    for w in WIDTHS:
        ny, nz = (3 if D > 1 else 1), (2 if D > 2 else 1)
        g = 2 + shift  # an odd ghost width puts cell lo at an odd element
        u = _input(D, (nz, ny, w + 2 * g), 7 * w + D)
        lo, hi = (0, 0, 0), (w - 1, ny - 1, nz - 1)
        begin = (-g, 0, 0)
        ref = oracle.compute_flux(D, method, 0, lo, hi, u, begin, dx, dt, po)
        ut = torch.tensor(u, device="cuda")
        ft = torch.full(ref.shape, float("nan"), dtype=torch.float64, device="cuda")
        out = torch.full((D + 2, nz, ny, w), float("nan"), dtype=torch.float64, device="cuda")
        bx.sweep_box(method, 0, D, (lo, hi), out, lo, ut, begin, dx, dt, pg, flux=ft, flux_begin=lo)
        got, new = ft.cpu().numpy(), out.cpu().numpy()
        want = u[:, :, :, g:g + w] - dt / dx[0] * (ref[:, :, :, 1:] - ref[:, :, :, :-1])
        for n in range(D + 2):
            assert np.max(np.abs(got[n] - ref[n])) <= RTOL * max(np.max(np.abs(ref[n])), 1e-300), (w, n)
            assert np.max(np.abs(new[n] - want[n])) <= RTOL * np.max(np.abs(want[n])), (w, n)


@pytest.mark.parametrize("precision", [0, 1], ids=["fp64", "fp32_storage"])
@pytest.mark.parametrize("bc", [0, 1, 2])
@pytest.mark.parametrize("cuts", [[0, 64, 97, 128, 131, 200], [0, 2, 5, 66, 130], [0, 30, 60, 90, 120]])
def test_boxes_step_like_one_box(cuts, bc, precision):
    """Boxes of even and odd widths (halos in place where the rows pair up,
    ghost copies elsewhere) step bit for bit like one box."""
    import bamrex_b200 as bx
    from bamrex_b200 import problems
    nx, ny = cuts[-1], 24
    u0 = problems.quadrant_2d(nx, ny=ny)
    whole = [((0, 0, 0), (nx - 1, ny - 1, 0))]
    parts = [((a, y, 0), (b - 1, y + 11, 0)) for y in (0, 12) for a, b in zip(cuts, cuts[1:])]
    outs = []
    for boxes in (whole, parts):
        lev = bx.Level(2, (0, 0, 0), (nx - 1, ny - 1, 0), [0.0, 0.0], [1.0, 1.0], boxes, bx.Parm(2, limiter=1), cfl=0.6,
                       bc_lo=(bc,) * 3, bc_hi=(bc,) * 3, x_mode=bx.XSWEEP_ROWS, staging=bx.STAGING_REGISTERS,
                       precision=precision)
        lev.set_state(u0)
        lev.run(3, use_graph=False)
        outs.append(lev.get_state())
        lev.close()
    np.testing.assert_array_equal(outs[1], outs[0])
