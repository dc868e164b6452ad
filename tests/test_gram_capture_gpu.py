"""fbse_gram between two launches of a captured graph: the graph of a context whose
H psi keeps projector partial sums (hpsi_fused) must still own its buffers after an
overlap that needs far more room, and give the same states."""
import numpy as np
import pytest

from oracle import oracle as O
from tests.systems import tiny_cluster

pytestmark = pytest.mark.gpu


def test_graph_after_gram(fbse, cuda):
    import torch
    sysm = tiny_cluster(128, 128, 12, natoms=6, nspin=2, is_complex=True, so=True)
    ctx = fbse.Context(sysm.grid, sysm.pot, nspin=2, is_complex=True, so=True, proj=sysm.proj, precision=1)
    ctx.set_tuning(hpsi_fused=1)
    emin = float(sysm.pot.min()) - 1.5
    de = float(sysm.pot.max()) + sysm.grid.ke_max + 2.0 - emin
    zn, _, _ = O.samp_points(12)
    an = O.newton_coeff(zn, np.array([emin + 0.2 * de]), emin, de, O.filter_dt(12, de))
    starts, _, _ = O.init_filter_states(-100, 1, sysm.ngrid, 2, True, sysm.grid.dv)
    p0 = torch.tensor(np.ascontiguousarray(starts.view(np.float64).reshape(1, -1)), device=cuda)
    b = fbse.Batch([(ctx, zn, an, emin, de, p0)])
    b.run()
    first = b.out[0].cpu().numpy().copy()
    # 600 x 600 overlaps: 5.8 MB, far more than the partial sums of one state
    rows = torch.randn((600, ctx.stlen), dtype=torch.float64, device=cuda)
    ctx.gram(rows, rows, 0, 2048)
    b.run()
    assert np.array_equal(first, b.out[0].cpu().numpy())
    b.close()
