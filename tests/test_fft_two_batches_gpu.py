"""FP64 H psi through the two-factor kernels is the same bit for bit whether a launch's
planes fill whole waves of the SMs (plane kernels) or not (line kernels): one and two
blocks per launch sequence on grids of 76 planes, where the first takes lines and the
second planes, with radices up to 16, up to 31 and odd factors above on both axes, on
one of them, and beside a 64- or 128-point axis."""
import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nx,ny", [(72, 70), (34, 51), (34, 48), (48, 34), (86, 40), (40, 86), (62, 60), (45, 52),
                                   (13, 11), (64, 30), (30, 128), (46, 58), (16, 16), (3, 5), (86, 74)])
def test_planes_and_lines(fbse, cuda, nx, ny):
    import torch
    n = nx * ny * 76
    rng = np.random.default_rng(n)
    g = O.Grid(nx, ny, 76, 0.5, 0.5, 0.5, -4.0, -4.0, -4.0, 10.0)
    ctx = fbse.Context(g, rng.normal(size=n), nspin=1, is_complex=True, precision=0)
    x = torch.tensor(rng.normal(size=(2, n)) + 1j * rng.normal(size=(2, n)), device=cuda)
    out = []
    for blocks in (1, 2):
        ctx.set_tuning(fft_chunk_blocks=blocks)
        y = torch.empty_like(x)
        ctx.hpsi(x, y)
        out.append(y)
    assert torch.equal(out[0], out[1])
