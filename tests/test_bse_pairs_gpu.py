"""The electron-hole kernels where the pair lists have edges: one state on either
side, odd counts, more rows than an FFT batch of 64, one and two spins."""
import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu

TOL = {0: 1e-10, 1: 3e-5}  # relative to the largest element, as for the other kernel tests


@pytest.mark.parametrize("nh,ne", [(1, 1), (3, 1), (1, 4), (5, 9), (9, 8)])
@pytest.mark.parametrize("nspin", [1, 2])
@pytest.mark.parametrize("precision", [0, 1])
def test_pair_lists(fbse, cuda, nh, ne, nspin, precision):
    import torch
    nx, ny, nz = 14, 12, 15
    n = nx * ny * nz
    g = O.Grid(nx, ny, nz, 0.5, 0.6, 0.7, -3.5, -3.6, -5.25, 10.0)
    rng = np.random.default_rng(nh * 16 + ne)
    psi = rng.normal(size=(nh + ne, nspin, n)) + 1j * rng.normal(size=(nh + ne, nspin, n))
    # any k-space arrays: no symmetry is assumed of them
    pots = [(rng.normal(size=n) + 1j * rng.normal(size=n)) / n for _ in range(2)]
    ctx = fbse.Context(g, np.zeros(n), nspin=nspin, is_complex=True, precision=precision)
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
    got = d.cpu().numpy()
    assert np.max(np.abs(got - np.tril(want))) <= TOL[precision] * np.max(np.abs(want))
    p = conv(np.array([rho(a, i) for a in el for i in range(nh)]), pots[0])
    q = np.array([rho(j, b) for b in el for j in range(nh)])
    want = -g.dv * p @ q.T
    assert np.max(np.abs(x.cpu().numpy() - np.tril(want))) <= TOL[precision] * np.max(np.abs(want))
