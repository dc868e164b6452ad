"""The Jacobi eigensolver through the exciton solve: matrix sizes around the pair
tiles (8 pairs, 32 rows), odd sizes, one state, and a diagonal matrix."""
import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 2, 3, 15, 16, 17, 32, 33, 130, 257])
@pytest.mark.parametrize("scale", [0.0, 1.0])
def test_hermitian(fbse, cuda, n, scale):
    """H = diag(h0) - K^d - K^x against numpy's eigvalsh.  Jacobi is backward stable:
    residuals and orthogonality within n rounding units of the norm (64 covers the
    rotations per element of the ten sweeps)."""
    import torch
    g = O.Grid(8, 8, 8, 0.5, 0.5, 0.5, -2.0, -2.0, -2.0, 10.0)
    ctx = fbse.Context(g, np.zeros(512), nspin=2, is_complex=True, precision=0)
    rng = np.random.default_rng(n)
    d, x = (scale * np.tril(rng.normal(size=(n, n)) + 1j * rng.normal(size=(n, n))) for _ in range(2))
    for m in (d, x):
        m[np.arange(n), np.arange(n)] = m[np.arange(n), np.arange(n)].real
    ev = np.concatenate([[-0.3], rng.uniform(-1, 1, n)])
    full = lambda m: np.tril(m, -1) + np.tril(m, -1).conj().T + np.diag(np.diag(m))
    h = np.diag(ev[1:] - ev[0]) - full(d) - full(x)
    runs = []
    for _ in range(2):
        e, coeff, *_rest = ctx.bse_solve(ev, 1, n, 1, torch.tensor(d, device=cuda), torch.tensor(x, device=cuda))
        runs.append((e, coeff.cpu().numpy()))
    e, c = runs[0]
    assert np.array_equal(e, runs[1][0]) and np.array_equal(c, runs[1][1])
    tol = 64 * max(n, 4) * 2.0 ** -53
    norm = np.linalg.norm(h, 2)
    assert np.max(np.abs(e - np.linalg.eigvalsh(h))) <= tol * norm
    assert np.max(np.abs(c.conj().T @ c - np.eye(n))) <= tol
    assert np.max(np.abs(h @ c - c * e)) <= tol * norm
