"""The mixed path's tensor-core contraction at the edges of its tiles: rows of A beyond
128 and 256, columns beyond 256, odd row lengths (rows that start 8 bytes off), and
lengths that leave 1, 9 and 15 points in the last block of 16."""
import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nh,ne", [(1, 17), (17, 1), (11, 12)])
@pytest.mark.parametrize("dims", [(15, 13, 11), (9, 9, 9), (7, 9, 17)])
def test_contraction_tiles(fbse, cuda, nh, ne, dims):
    import torch
    nx, ny, nz = dims
    n = nx * ny * nz
    g = O.Grid(nx, ny, nz, 0.5, 0.6, 0.7, -0.25 * nx, -0.3 * ny, -0.35 * nz, 10.0)
    rng = np.random.default_rng(n + nh)
    psi = rng.normal(size=(nh + ne, 1, n)) + 1j * rng.normal(size=(nh + ne, 1, n))
    pots = [(rng.normal(size=n) + 1j * rng.normal(size=n)) / n for _ in range(2)]
    ctx = fbse.Context(g, np.zeros(n), nspin=1, is_complex=True, precision=1)
    dev = [torch.tensor(p, device=cuda) for p in pots]
    d, x = ctx.bse_kernel(torch.tensor(psi.reshape(nh + ne, -1), device=cuda), nh, ne, nh, *dev)

    def conv(rho, pot):
        f = np.fft.fftn(rho.reshape(-1, nz, ny, nx), axes=(1, 2, 3)) * pot.reshape(nz, ny, nx) * n
        return np.fft.ifftn(f, axes=(1, 2, 3)).reshape(rho.shape[0], -1)

    rho = lambda i, j: np.sum(psi[i].conj() * psi[j], axis=0)
    el = range(nh, nh + ne)
    p = conv(np.array([rho(a, b) for a in el for b in el]), pots[1])
    q = np.array([rho(j, i) for j in range(nh) for i in range(nh)])
    want = (g.dv * p @ q.T).reshape(ne, ne, nh, nh).transpose(0, 3, 1, 2).reshape(ne * nh, ne * nh)
    assert np.max(np.abs(d.cpu().numpy() - np.tril(want))) <= 3e-5 * np.max(np.abs(want))
    p = conv(np.array([rho(a, i) for a in el for i in range(nh)]), pots[0])
    q = np.array([rho(j, b) for b in el for j in range(nh)])
    want = -g.dv * p @ q.T
    assert np.max(np.abs(x.cpu().numpy() - np.tril(want))) <= 3e-5 * np.max(np.abs(want))
