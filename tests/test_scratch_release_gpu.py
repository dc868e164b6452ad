"""Device memory nearly full, most of what is left in the scratch that an FP64 product
keeps: calls that need room of their own take it from there instead of failing."""
import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("call", ["hpsi", "filter", "energy", "gram"])
def test_scratch_given_back(fbse, cuda, call):
    import torch
    dims, many = (40, 40, 40), 600
    n = int(np.prod(dims))
    g = O.Grid(*dims, 0.5, 0.5, 0.5, -10.0, -10.0, -10.0, 10.0)
    ctx = fbse.Context(g, np.zeros(n), nspin=1, is_complex=True, precision=0)
    rows = torch.ones((256, 2 * n), dtype=torch.float64, device=cuda)
    x = torch.ones((many, n), dtype=torch.complex128, device=cuda)  # 0.6 GB
    y = torch.empty_like(x)
    zn, an = np.zeros(16), np.ones((1, 16), complex)
    out = torch.empty((24, 1, 2 * n), dtype=torch.float64, device=cuda)

    def run(m):
        if call == "hpsi":
            ctx.hpsi(x[:m], y[:m])
        elif call == "filter":  # a ring of 16 x 24 states
            ctx.newton_filter(zn, an, -1.0, 20.0, rows[:max(1, m // 25)], out[:max(1, m // 25)])
        elif call == "energy":
            ctx.energy_all(rows[:max(1, m // 30)])
        else:  # a wider product needs a larger scratch than the kept one
            ctx.gram(rows[:, :2 * n], rows[:max(1, m // 3)])

    run(1)  # its kernels are loaded
    ctx.gram(rows, rows[:128])
    torch.cuda.synchronize()
    free = torch.cuda.mem_get_info()[0]
    hold = torch.empty(free - (24 << 20), dtype=torch.uint8, device=cuda)
    try:
        run(many)
    finally:
        del hold
        torch.cuda.empty_cache()
    run(many)
