"""The exact-slice products over several chunks of K (a small tc_image_bytes: the
sums carried from chunk to chunk, the last one shorter) and for other row counts:
bit for bit the product of one chunk and of all rows."""
import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("cplx", [False, True])
@pytest.mark.parametrize("shape,na,nb", [((16, 16, 16), 3, 5), ((40, 36, 33), 5, 66), ((40, 36, 33), 130, 3)])
def test_chunks_and_row_counts(fbse, cuda, cplx, shape, na, nb):
    import torch
    n = int(np.prod(shape))
    g = O.Grid(*shape, 0.5, 0.5, 0.5, -4.0, -4.0, -4.0, 10.0)
    ctx = fbse.Context(g, np.zeros(n), nspin=1, is_complex=cplx, precision=0)
    rng = np.random.default_rng(5)
    a, b = (torch.tensor(rng.normal(size=(m, n * (2 if cplx else 1))), device=cuda) for m in (na, nb))
    one = ctx.gram(a, b)
    assert np.array_equal(ctx.gram(a[:2].contiguous(), b[:1].contiguous()), one[:2, :1])
    # a split has 32 blocks of 32 values or more, nine slices of each row: 1, 2 and 5 of the
    # smallest splits a chunk
    rows = (na + 127) // 128 * 128 + (nb + 63) // 64 * 64 * (2 if cplx else 1)
    for splits in (1, 2, 5):
        ctx.set_tuning(tc_image_bytes=1.2 * splits * 32 * 32 * 2 * 9 * rows)
        assert np.array_equal(ctx.gram(a, b), one)
