"""The two-factor FFT kernels against the FP64 oracle: every radix, odd
factors of 27 to 255, axes whose length has one factor, planes too large for shared memory in either precision,
axes next to one another that the register-resident kernels (64, 128) and the
mixed-radix kernels (a prime factor above 255) take, and tiles with remainders."""
import numpy as np
import pytest

from oracle import oracle as O
from tests.systems import random_states, tiny_cluster

pytestmark = pytest.mark.gpu

TOL = {0: 1e-12, 1: 3e-6}  # relative max-norm error of H psi, as for the other FFT kernels

SHAPES = [
    (2, 3, 4), (5, 6, 7), (9, 10, 12), (14, 15, 16), (13, 11, 8), (17, 19, 23), (29, 31, 18), (20, 21, 24), (25, 50, 36),
    (143, 6, 5), (33, 169, 10), (256, 3, 30), (100, 98, 99), (176, 168, 4), (130, 120, 6), (62, 75, 225),
    (64, 100, 6), (128, 257, 4), (257, 45, 4), (4, 10, 512), (60, 64, 41), (128, 64, 60),
    (27, 37, 41), (74, 86, 10), (43, 9, 106), (16, 148, 53), (111, 8, 254), (176, 166, 7), (130, 134, 5), (1020, 6, 3),
    (4, 6, 2040),
]


@pytest.mark.parametrize("shape", SHAPES)
@pytest.mark.parametrize("precision", [0, 1])
def test_kinetic_and_local(fbse, cuda, shape, precision):
    import torch
    sysm = tiny_cluster(*shape, natoms=4, is_complex=True)
    psis = random_states(3, sysm, np.random.default_rng(11))
    ctx = fbse.Context(sysm.grid, sysm.pot, is_complex=True, precision=precision)
    x = torch.tensor(psis, dtype=ctx.working_dtype(), device=cuda)
    y = torch.empty_like(x)
    ctx.hpsi(x, y)
    want = np.array([O.hamiltonian(p, sysm) for p in psis])
    got = y.cpu().numpy()
    assert np.max(np.abs(got - want)) / np.max(np.abs(want)) < TOL[precision]
