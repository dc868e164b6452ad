"""The mixed-radix FFT kernels on axes whose lines have more butterflies than a CTA
has threads (n / R > 256, and > 1024 for whole planes): H psi through them against
the FP64 oracle, on each axis and beside an axis that the two-factor kernels take,
and the Rayleigh-Ritz step, which uses them whatever H psi itself uses."""
import numpy as np
import pytest

from oracle import oracle as O
from tests.systems import random_states, tiny_cluster

pytestmark = pytest.mark.gpu

TOL = {0: 1e-12, 1: 3e-6}  # relative max-norm error of H psi, as for the other FFT kernels

# 512: 256 butterflies of radix 2; 514 = 2 x 257; 780, 900: radices 4 and 3; 1536 has
# no two factors; 2058 = 2 x 3 x 7^3 has more than 1024 butterflies
SHAPES = [s for n in (512, 514, 518, 780, 900, 1050, 1536, 2058) for s in ((n, 3, 2), (3, n, 2), (2, 3, n))] + [
    (18, 2, 810), (17, 1536, 3)]


@pytest.mark.parametrize("shape", SHAPES)
@pytest.mark.parametrize("kernels", [0, 1, 2])
@pytest.mark.parametrize("precision", [0, 1])
def test_hpsi(fbse, cuda, shape, kernels, precision):
    import torch
    sysm = tiny_cluster(*shape, natoms=4, is_complex=True)
    psis = random_states(3, sysm, np.random.default_rng(11))
    ctx = fbse.Context(sysm.grid, sysm.pot, is_complex=True, precision=precision)
    ctx.set_tuning(fft_kernels=kernels)
    x = torch.tensor(psis, dtype=ctx.working_dtype(), device=cuda)
    y = torch.empty_like(x)
    ctx.hpsi(x, y)
    want = np.array([O.hamiltonian(p, sysm) for p in psis])
    assert np.max(np.abs(y.cpu().numpy() - want)) / np.max(np.abs(want)) < TOL[precision]


@pytest.mark.parametrize("shape", [(518, 4, 3), (4, 514, 3), (3, 4, 518), (3, 2, 780)])
def test_ritz(fbse, cuda, shape):
    """Ritz values and sigmas of the FP64 step against the oracle's SVD + eigh."""
    import torch
    sysm = tiny_cluster(*shape, natoms=4, is_complex=True)
    psi = random_states(5, sysm, np.random.default_rng(3))
    u, _ = O.ortho(psi, True, dv=sysm.grid.dv)
    _, vec = O.diag(u, sysm)
    e_or, s_or = O.sigma_e(vec, sysm)
    ctx = fbse.Context(sysm.grid, sysm.pot, is_complex=True, precision=0)
    d = torch.tensor(psi.view(np.float64).reshape(5, -1), device=cuda)
    k, ev, sg = ctx.ortho_diag_sigma(d)
    # as tests/test_ortho_gpu.py: 1e-9 of the energies, 1e-3 of the sigmas
    assert k == 5 and np.allclose(ev, e_or, atol=1e-9 * max(1.0, np.max(np.abs(e_or))))
    assert np.allclose(sg, s_or, rtol=1e-3, atol=1e-8)
