"""The autotuner times the Rayleigh-Ritz step's H psi kernels for themselves: whichever
of H psi and the step comes first, each has its own record where its kernels differ
(the projector gather always, the FFT off the 64 / 128 / 256-point grids)."""
import numpy as np
import pytest

from tests.systems import random_states, tiny_cluster

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ritz_first", [False, True])
@pytest.mark.parametrize("shape,fft", [((16, 18, 20), 2), ((64, 64, 64), 1)])
def test_records(fbse, cuda, shape, fft, ritz_first):
    import torch
    sysm = tiny_cluster(*shape, natoms=6, nspin=2, is_complex=True, so=True)
    ctx = fbse.Context(sysm.grid, sysm.pot, nspin=2, is_complex=True, so=True, proj=sysm.proj)
    psi = random_states(16, sysm, np.random.default_rng(2))
    x = torch.tensor(psi, device=cuda)
    calls = [lambda: ctx.hpsi(x, torch.empty_like(x)),
             lambda: ctx.ortho_diag_sigma(torch.view_as_real(x).reshape(16, -1).clone())]
    for call in calls[::-1] if ritz_first else calls:
        call()
    rep = ctx.tuning_report()
    for kernel, count in (("projector gather", 2), ("fft blocks per launch", fft)):
        probs = [r["problem"] for r in rep if r["kernel"].startswith(kernel)]
        assert len(probs) == count and len(set(probs)) == count, probs
