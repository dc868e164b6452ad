"""The FP64 products by exact slices (fbse_gram, the overlap of the Rayleigh-Ritz
step) against extended-precision sums: tile and split remainders, real and
complex rows, slabs at odd offsets, rows of very different size, zero,
denormal and non-finite rows.

Tolerance: a value is rounded to 2^-62 of its row's largest one, the digit
products left out are below 2^-57 of the product of the rows' largest ones, and
each split and the final sum round to 2^-53 of it; so |error| <= K 2^-56
max|a| max|b| + 4 * 2^-53 sum|a||b|, K the number of real terms."""
import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu


def _bound(a, b, sums):
    k = a.shape[1]
    ma, mb = np.max(np.abs(a), axis=1), np.max(np.abs(b), axis=1)
    return k * 2.0 ** -56 * ma[:, None] * mb[None, :] + 4 * 2.0 ** -53 * sums


@pytest.mark.parametrize("cplx", [False, True])
@pytest.mark.parametrize("shape,na,nb,off,cut", [((16, 16, 8), 1, 1, 0, 0), ((17, 13, 11), 3, 64, 1, 2),
                                                 ((20, 17, 19), 64, 65, 0, 0), ((33, 32, 31), 129, 7, 3, 5),
                                                 ((40, 36, 33), 130, 130, 0, 0), ((60, 60, 60), 5, 66, 0, 1)])
def test_gram(fbse, cuda, cplx, shape, na, nb, off, cut):
    import torch
    n = int(np.prod(shape))
    g = O.Grid(*shape, 0.5, 0.5, 0.5, -4.0, -4.0, -4.0, 10.0)
    ctx = fbse.Context(g, np.zeros(n), nspin=1, is_complex=cplx, precision=0)
    rng = np.random.default_rng(21)
    w = 2 if cplx else 1

    def rows(m):
        r = rng.normal(size=(m, n * w)) * np.exp(-rng.uniform(0, 25, size=(m, n * w)))
        return r * 10.0 ** rng.integers(-40, 40, size=(m, 1))

    a, b = rows(na), rows(nb)
    if na > 2:
        a[1] = 0.0
        a[2] *= 1e-290 / np.max(np.abs(a[2]))
    length = n - off - cut
    got = ctx.gram(torch.tensor(a, device=cuda), torch.tensor(b, device=cuda), off, length)
    # checked against extended precision at the edges of the 128 x 64 tiles
    ii, jj = (sorted({v for v in (0, 1, 2, 63, 64, 65, 127, 128, m - 1) if v < m}) for m in (na, nb))
    sl = slice(off * w, (off + length) * w)
    as_, bs_ = a[ii][:, sl], b[jj][:, sl]
    al, bl = as_.astype(np.longdouble), bs_.astype(np.longdouble)
    dv = np.longdouble(g.dx) * g.dy * g.dz
    sums = (np.abs(al) @ np.abs(bl).T * dv).astype(np.float64)
    if cplx:
        ar, ai, br, bi = al[:, 0::2], al[:, 1::2], bl[:, 0::2], bl[:, 1::2]
        re, im = (ar @ br.T + ai @ bi.T) * dv, (ar @ bi.T - ai @ br.T) * dv
        sums = sums + ((np.abs(ar) @ np.abs(bi).T + np.abs(ai) @ np.abs(br).T) * dv).astype(np.float64)
    else:
        re, im = al @ bl.T * dv, np.zeros((len(ii), len(jj)))
    tol = _bound(as_, bs_, sums) + 1e-320
    sub = got[np.ix_(ii, jj)]
    assert np.all(np.abs(sub.real - re) <= tol) and np.all(np.abs(sub.imag - im) <= tol)
    again = ctx.gram(torch.tensor(a, device=cuda), torch.tensor(b, device=cuda), off, length)
    assert np.array_equal(got, again)
    # a row with a NaN or an infinity spoils its own products only
    a[0, off * w + 1] = np.nan
    b[nb - 1, off * w] = np.inf
    bad = ctx.gram(torch.tensor(a, device=cuda), torch.tensor(b, device=cuda), off, length)
    assert np.all(np.isnan(bad[0].real)) and np.all(np.isnan(bad[:, nb - 1].real))
    assert np.array_equal(bad[1:, :nb - 1], got[1:, :nb - 1])
