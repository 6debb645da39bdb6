"""The tiled half cycles of the 2D V-cycle against the restatement, bit for
bit: sides that are not multiples of a tile, windows wider than the domain,
every boundary kind and mixtures of them."""
import numpy as np
import pytest

from test_gpu_helmholtz import _device

pytestmark = pytest.mark.gpu

SIZES = [(32, 64), (34, 66), (62, 40), (64, 64), (66, 32), (128, 96), (4, 300), (400, 4), (160, 130), (2, 1026)]
# periodic 0, Dirichlet 1, Neumann 2 (lo, hi of x and y)
BCS = {"periodic": (0, 0, 0, 0), "dirichlet": (1, 1, 1, 1), "neumann": (2, 2, 2, 2), "mixed": (1, 2, 2, 1),
       "x_periodic": (0, 0, 2, 1), "y_periodic": (2, 1, 0, 0)}


def _op(nx, ny, bcs, seed):
    from oracle import helmholtz_oracle as H
    rng = np.random.default_rng(seed)
    kind = {0: H.PERIODIC, 1: H.DIRICHLET, 2: H.NEUMANN}
    faces = [0.5 + rng.uniform(size=(1, ny, nx + 1)), 0.5 + rng.uniform(size=(1, ny + 1, nx))]
    if bcs[0] == 0:
        faces[0][:, :, -1] = faces[0][:, :, 0]
    if bcs[2] == 0:
        faces[1][:, -1, :] = faces[1][:, 0, :]
    return H.Op(2, (nx, ny), [1.0 / nx, 1.0 / ny], tuple(kind[b] for b in (bcs[0], bcs[2], 0)),
                tuple(kind[b] for b in (bcs[1], bcs[3], 0)), 1.1, 0.7, 0.0, 0.3 + rng.uniform(size=(1, ny, nx)), faces)


def _seam_free(nx, ny, bcs):
    """Red and black stay apart across a periodic seam on every level: a level
    with an odd periodic side has neighbours of one colour there, whose update
    order nothing fixes."""
    while nx % 2 == 0 and ny % 2 == 0 and nx >= 4 and ny >= 4:
        nx, ny = nx // 2, ny // 2
    return not ((bcs[0] == 0 and nx % 2 and nx > 1) or (bcs[2] == 0 and ny % 2 and ny > 1))


CASES = [(nx, ny, bc) for nx, ny in SIZES for bc in sorted(BCS) if _seam_free(nx, ny, BCS[bc])]


@pytest.mark.parametrize("nx,ny,bc", CASES)
def test_vcycle_bitwise(nx, ny, bc):
    from oracle import helmholtz_oracle as H
    op = _op(nx, ny, BCS[bc], nx + ny)
    h = _device(op)
    ops = H.hierarchy(op)
    rng = np.random.default_rng(1)
    for _ in range(2):
        rhs = rng.standard_normal((1, ny, nx))
        np.testing.assert_array_equal(h.vcycle(rhs), H.vcycle(ops, rhs))
    h.close()
