"""FP64 products by exact slices where the rows' largest values do not meet: every
element against extended precision, relative to sum |a||b| as an FP64 sum has it.

Tolerance, in u = 2^-53 times sum |a||b| (moduli |re| + |im|): 144 from the digits, one
for each split (1760 values or more at these lengths, 1024 assumed) and three for their
conversion and scaling; or, summed in FP64, the terms of one of 256 threads (two
multiply-adds each) and 13 for the tree and the scaling."""
import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu

DIMS = (57, 52, 45)
N = int(np.prod(DIMS))


def _ctx(fbse, cplx):
    g = O.Grid(*DIMS, 0.8, 0.8, 0.8, -22.8, -20.8, -18.0, 10.0)
    return fbse.Context(g, np.zeros(N), nspin=1, is_complex=cplx, precision=0), g


def _packet(x0, width):
    z, y, x = np.meshgrid(*((np.arange(m) - m // 2) * 0.8 for m in DIMS[::-1]), indexing="ij")
    return np.exp(-((x - x0) ** 2 + y ** 2 + z ** 2) / width).reshape(-1)


def _rows(name, rng):
    """(A, B) real rows"""
    if name == "packets":  # up to 36 bohr apart, narrow and wide
        return (np.array([_packet(-s / 2, w) for s in (0, 10, 20, 28, 36) for w in (8.0, 40.0)]),
                np.array([_packet(s / 2, w) for s in (0, 10, 20, 28, 36) for w in (8.0, 40.0)]))
    if name == "steps":  # 1e-9 of the other half's size, every term with the same digits
        a = np.full(N, 1.0 / 3.0)
        a[N // 2:] *= 1e-9
        return np.array([a, a[::-1]]), np.array([a, a[::-1]])
    if name == "graded":  # 40 decades inside each row
        return tuple(rng.normal(size=(m, N)) * 10.0 ** rng.uniform(-40, 0, size=(m, N)) for m in (3, 66))
    if name == "disjoint":  # no point in common: zero exactly
        a = rng.normal(size=(2, N))
        b = rng.normal(size=(3, N))
        a[:, ::2] = 0.0
        b[:, 1::2] = 0.0
        return a, b
    # sizes whose products leave the range of FP64's exponent halfway, and denormal rows
    scale = 10.0 ** np.array([-300, -200, -150, 0, 140])
    a = rng.normal(size=(5, N)) * scale[:, None]
    a[0] *= 1e-12
    return a, rng.normal(size=(5, N)) * scale[::-1, None]


@pytest.mark.parametrize("cplx", [False, True])
@pytest.mark.parametrize("name", ["packets", "steps", "graded", "disjoint", "range"])
def test_componentwise(fbse, cuda, name, cplx):
    import torch
    ctx, g = _ctx(fbse, cplx)
    rng = np.random.default_rng(4)
    a, b = _rows(name, rng)
    if cplx:
        turn = lambda r: np.stack([r * np.cos(0.3 + np.arange(len(r)))[:, None],  # noqa: E731
                                   r * np.sin(0.3 + np.arange(len(r)))[:, None]], axis=2).reshape(len(r), -1)
        a, b = turn(a), turn(b)
    got = ctx.gram(torch.tensor(a, device=cuda), torch.tensor(b, device=cuda))
    al, bl = a.astype(np.longdouble), b.astype(np.longdouble)
    dv = np.longdouble(g.dx) * g.dy * g.dz
    if cplx:
        ar, ai, br, bi = al[:, 0::2], al[:, 1::2], bl[:, 0::2], bl[:, 1::2]
        re, im = (ar @ br.T + ai @ bi.T) * dv, (ar @ bi.T - ai @ br.T) * dv
        sums = (np.abs(ar) + np.abs(ai)) @ (np.abs(br) + np.abs(bi)).T * dv
    else:
        re, im, sums = al @ bl.T * dv, np.zeros((len(a), len(b))), np.abs(al) @ np.abs(bl).T * dv
    splits = -(-(N * (2 if cplx else 1)) // 1024)
    tol = max(144 + splits + 3, 2 * (N // 256 + 1) + 13) * np.longdouble(2.0) ** -53 * sums + 1e-320
    assert np.all(np.abs(got.real - re) <= tol) and np.all(np.abs(got.imag - im) <= tol)
    if name == "disjoint":
        assert not np.any(got)


def test_exciton_kernel_of_a_state_with_an_infinity(fbse, cuda):
    """A hole with an infinity: its own elements are not finite, the others unchanged."""
    import torch
    nh, ne, n = 3, 2, 16 * 15 * 14
    g = O.Grid(16, 15, 14, 0.5, 0.5, 0.5, -4.0, -3.75, -3.5, 10.0)
    ctx = fbse.Context(g, np.zeros(n), nspin=1, is_complex=True, precision=0)
    rng = np.random.default_rng(6)
    psi = rng.normal(size=(nh + ne, n)) + 1j * rng.normal(size=(nh + ne, n))
    pot = [torch.tensor((rng.normal(size=n) + 1j * rng.normal(size=n)) / n, device=cuda) for _ in range(2)]
    clean, _ = ctx.bse_kernel(torch.tensor(psi, device=cuda), nh, ne, nh, *pot)
    psi[1, 77] = np.inf
    bad, _ = ctx.bse_kernel(torch.tensor(psi, device=cuda), nh, ne, nh, *pot)
    clean, bad = clean.cpu().numpy(), bad.cpu().numpy()
    hole = np.arange(nh * ne) % nh
    mine = np.tril((hole[:, None] == 1) | (hole[None, :] == 1))
    assert not np.any(np.isfinite(bad[mine])) and np.array_equal(bad[~mine], clean[~mine])
