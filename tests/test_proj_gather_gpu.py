"""The projector gather over clusters of CTAs (few atoms), single CTAs (many
atoms), spheres shorter than a warp's stride and a batch that is no multiple
of a CTA's states, against the FP64 oracle; and the Rayleigh-Ritz step, whose
gather keeps a warp per state, on an odd number of states."""
import numpy as np
import pytest

from oracle import oracle as O
from tests.systems import random_states, tiny_cluster

pytestmark = pytest.mark.gpu

TOL = {0: 1e-12, 1: 3e-6}  # relative max-norm error of H psi, as for the other projector tests


# (atoms, SO, NL, spacing): the spacing sets the points per sphere (about 90 at 1.4, 550 at 0.8)
@pytest.mark.parametrize("natoms,so,nl,d", [(2, True, False, 0.8), (7, True, True, 0.8), (40, True, True, 1.0),
                                            (150, False, True, 1.4), (150, True, True, 1.4)])
@pytest.mark.parametrize("precision", [0, 1])
def test_gather(fbse, cuda, natoms, so, nl, d, precision):
    import torch
    sysm = tiny_cluster(28, 26, 30, d=d, natoms=natoms, nspin=2 if so else 1, is_complex=True, so=so, nl=nl)
    psis = random_states(3, sysm, np.random.default_rng(12))
    ctx = fbse.Context(sysm.grid, sysm.pot, nspin=sysm.nspin, is_complex=True, so=so, nl=nl, proj=sysm.proj,
                       precision=precision)
    x = torch.tensor(psis, dtype=ctx.working_dtype(), device=cuda)
    y = torch.empty_like(x)
    want = np.array([O.hamiltonian(p, sysm) for p in psis])
    for points in (1, 2, 4):
        ctx.set_tuning(gather_points=points)
        ctx.hpsi(x, y)
        got = y.cpu().numpy()
        assert np.max(np.abs(got - want)) / np.max(np.abs(want)) < TOL[precision]
    # the mixed Rayleigh-Ritz step's gather: Rayleigh quotients of five states
    p5 = random_states(5, sysm, np.random.default_rng(13))
    p5 /= np.sqrt(np.sum(np.abs(p5) ** 2, axis=1, keepdims=True) * sysm.grid.dv)
    rows = torch.tensor(p5.view(np.float64), device=cuda)
    k, ev, _ = ctx.ortho_diag_sigma(rows)
    h = np.array([O.hamiltonian(p, sysm) for p in p5])
    g, m = p5.conj() @ p5.T, p5.conj() @ h.T
    lam, v = np.linalg.eigh(g)
    xm = v / np.sqrt(lam)
    ref = np.linalg.eigvalsh(xm.conj().T @ m @ xm)
    assert k == 5 and np.max(np.abs(ev - ref)) / np.max(np.abs(ref)) < TOL[precision]
