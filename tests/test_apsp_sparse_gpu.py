"""Shortest-path steps and walks over the finite entries of a sparse A, bit
for bit against the same steps in numpy (one rounded add per entry, then
minima that ignore NaN) and the oracle's walk. Sizes sit at the edges of the
slices (8 rows), the column blocks (16, 8 and 4 columns: 3500, 7000 rows) and
the vector loads (n a multiple of 4 or not)."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _graph(n, degree, symmetric, odd, seed):
    rng = np.random.default_rng(seed)
    A = np.full((n, n), np.inf, np.float32)
    i, j = rng.integers(0, n, n * degree), rng.integers(0, n, n * degree)
    w = (rng.random(n * degree) * 9 + 0.1).astype(np.float32)
    A[i, j] = w
    if symmetric:
        A[j, i] = A[i, j]
    np.fill_diagonal(A, 0.0)
    if odd and n > 4:  # entries a minimum has to treat with care
        A[0, 1], A[2, 0], A[3, 3], A[1, 4] = np.nan, -0.0, -2.5, -np.inf
    return A


def _jacobi(A, L):
    H = A
    for t in range(L):
        N = np.full_like(A, np.inf)
        for j in range(A.shape[0]):
            for k in np.flatnonzero(~(A[j] == np.inf)):
                with np.errstate(invalid="ignore"):
                    N[:, j] = np.fmin(N[:, j], A[j, k] + H[k, :])
        if np.array_equal(N.view(np.int32), H.view(np.int32)):
            return N, t + 1
        H = N
    return H, L


@pytest.mark.parametrize("n,degree,L", [(1, 1, 2), (7, 2, 9), (8, 2, 3), (9, 3, 12), (31, 4, 40), (129, 3, 5),
                                        (500, 12, 30), (1001, 6, 3), (3500, 2, 2), (3501, 2, 2), (7001, 1, 1)])
@pytest.mark.parametrize("symmetric", [False, True])
def test_sparse_lengths_match_row_steps(n, degree, L, symmetric):
    from netsci_gb300 import device
    A = _graph(n, degree, symmetric, odd=not symmetric and n < 3000, seed=n)
    want, steps = _jacobi(A, L)
    H, got = device.apsp_lengths(torch.from_numpy(A).cuda(), L)
    assert got == steps
    assert np.array_equal(H.cpu().numpy(), want)


@pytest.mark.parametrize("n,L,symmetric", [(13, 1, False), (40, 9, False), (61, 12, True), (130, 6, False)])
def test_sparse_paths_match_oracle(oracle_mod, n, L, symmetric):
    from netsci_gb300 import device
    A = _graph(n, 3, symmetric, odd=False, seed=3 * n)
    Ho, Po = oracle_mod.apsp_paths(A, L, 1e-3)
    H, P = device.apsp_paths(torch.from_numpy(A).cuda(), L, 1e-3)
    assert np.array_equal(H.cpu().numpy(), Ho)
    assert np.array_equal(P.cpu().numpy(), Po)


@pytest.mark.parametrize("n", [2, 65, 600, 1500])
def test_long_chain_ends_in_products(n):
    """A chain of n vertices has hop diameter n - 1: long ones pass the sparse
    steps' share and finish in dense products, with the same count."""
    from netsci_gb300 import device
    w = (np.arange(n - 1) % 7 + 1).astype(np.float32)
    A = np.full((n, n), np.inf, np.float32)
    A[np.arange(n - 1), np.arange(1, n)] = w
    A[np.arange(1, n), np.arange(n - 1)] = w
    np.fill_diagonal(A, 0.0)
    at = np.concatenate([[0.0], np.cumsum(w)]).astype(np.float32)
    dev = torch.from_numpy(A).cuda()
    H, products = device.apsp_lengths(dev, n, H=dev)  # in place
    assert np.array_equal(H.cpu().numpy(), np.abs(at[:, None] - at[None, :]))
    assert products == int(np.ceil(np.log2(max(1, n - 1)))) + 1


@pytest.mark.parametrize("n,L", [(1800, 3), (1801, 4), (2600, 17), (2601, 2601)])
@pytest.mark.parametrize("integer", [False, True])
@pytest.mark.parametrize("alias", [False, True])
def test_relabelled_steps_match_row_steps(n, L, integer, alias):
    """Vertices sorted by degree (degrees from 1 to 160, so that the slices of
    the matrix's own order are mostly padding): every parity of the last step,
    converged or not, and the result over its own input."""
    from netsci_gb300 import device
    rng = np.random.default_rng(n)
    A = np.full((n, n), np.inf, np.float32)
    i = np.arange(1, n)
    j = rng.integers(0, i)                       # a random tree
    A[i, j] = A[j, i] = rng.integers(1, 50, n - 1) if integer else rng.random(n - 1) + np.float32(0.25)
    for hub in rng.choice(n, n // 16, replace=False):
        j = rng.choice(n, 160, replace=False)
        w = rng.integers(1, 50, 160) if integer else rng.random(160) + 0.25
        A[hub, j] = w
        A[j, hub] = w
    np.fill_diagonal(A, 0.0)
    want, steps = _jacobi(A, L)
    a = torch.from_numpy(A).cuda()
    H, got = device.apsp_lengths(a, L, a if alias else None)
    if L < n - 1 or not integer:  # otherwise repeated squaring counts products
        assert got == steps
    assert np.array_equal(H.cpu().numpy(), want)
