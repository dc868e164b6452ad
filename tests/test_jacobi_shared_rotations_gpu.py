"""The Jacobi eigensolver on both sides of the size from which a round's rotations are
formed once for all tiles (n = 320 has a tile for each of 608 CTAs, 322 more): the
complex solve through the exciton stage, the real one through Rayleigh-Ritz."""
import numpy as np
import pytest
import scipy.linalg

from oracle import oracle as O
from tests.test_jacobi_gpu import test_hermitian as hermitian

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [320, 321, 322, 337, 400])
def test_complex(fbse, cuda, n):
    hermitian(fbse, cuda, n, 1.0)


@pytest.mark.parametrize("n", [321, 352])
def test_real(fbse, cuda, n):
    """Ritz values of n random real states against LAPACK's generalised solve on the same
    products: 1e-11 of the largest, for an overlap of condition below 10."""
    import torch
    dims = (20, 21, 22)
    g = O.Grid(*dims, 0.5, 0.5, 0.5, -5.0, -5.25, -5.5, 10.0)
    rng = np.random.default_rng(n)
    ctx = fbse.Context(g, rng.normal(size=int(np.prod(dims))), nspin=1, is_complex=False, precision=0)
    psi = rng.normal(size=(n, int(np.prod(dims))))
    d = torch.tensor(psi, device=cuda)
    h = ctx.residual(d, np.zeros(n)).cpu().numpy()
    over, proj = psi @ psi.T, psi @ h.T
    want = scipy.linalg.eigh((proj + proj.T) / 2, over, eigvals_only=True)
    k, ev, _ = ctx.ortho_diag_sigma(d)
    assert k == n and np.max(np.abs(np.sort(ev) - want)) <= 1e-11 * np.max(np.abs(want))
