"""Solves on either side of each choice between dense steps, steps over the
entries, products and single steps before products: integer weights, whose sums
are exact on every way, against Jacobi steps bit for bit and in the returned
count; few steps on sparse and full matrices against the same steps in numpy."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _graph(n, degree, integer, seed):
    rng = np.random.default_rng(seed)
    pts = rng.random((n, 3))
    r = (degree / (n * 4.0 / 3.0 * np.pi)) ** (1.0 / 3.0)
    w = rng.integers(1, 101, (n, n)).astype(np.float32) if integer else (rng.random((n, n)) * 99 + 1).astype(np.float32)
    w = np.triu(w, 1)
    near = ((pts[:, None, :] - pts[None, :, :]) ** 2).sum(-1) < r * r
    A = np.where(near, w + w.T, np.float32(np.inf)).astype(np.float32)
    np.fill_diagonal(A, 0.0)
    return A


@pytest.mark.parametrize("n", [2, 3, 64, 129, 500, 700, 769, 897, 1025, 1300, 1409])
@pytest.mark.parametrize("degree", [6.0, 16.0])
def test_exact_squaring_matches_steps(n, degree):
    from netsci_gb300 import device
    A = torch.from_numpy(_graph(n, degree, True, n)).cuda()
    device.set_apsp_method(0)
    try:
        want, hops = device.apsp_lengths(A, n)
    finally:
        device.set_apsp_method(-1)
    got, products = device.apsp_lengths(A, n)
    assert torch.equal(got, want)
    assert products == int(np.ceil(np.log2(max(hops, 1)))) + 1
    B = A.clone()
    device.apsp_lengths(B, n, H=B)
    assert torch.equal(B, want)


@pytest.mark.parametrize("n", [5, 64, 130, 257, 385, 600])
@pytest.mark.parametrize("L", [1, 2, 3, 5, 9])
@pytest.mark.parametrize("degree", [6.0, 16.0, 1e9])
def test_few_steps_match_numpy(n, L, degree):
    from netsci_gb300 import device
    A = _graph(n, degree, False, 7 * n)
    H, steps = A, L
    for t in range(L):
        N = np.stack([(A[j][:, None] + H).min(0) for j in range(n)], axis=1)
        same = np.array_equal(N, H)
        H = N
        if same:
            steps = t + 1
            break
    got, count = device.apsp_lengths(torch.from_numpy(A).cuda(), L)
    assert count == steps
    assert np.array_equal(got.cpu().numpy(), H)


@pytest.mark.parametrize("n", [9, 31, 90, 129, 257])
@pytest.mark.parametrize("L", [1, 4, 17])
@pytest.mark.parametrize("degree", [6.0, 1e9])
@pytest.mark.parametrize("symmetric", [True, False])
def test_paths_match_oracle(oracle_mod, n, L, degree, symmetric):
    from netsci_gb300 import device
    A = _graph(n, degree, False, 3 * n)
    if not symmetric:
        A[np.triu_indices(n, 1)] *= np.float32(1.5)
    Ho, Po = oracle_mod.apsp_paths(A, L, 1e-3)
    H, P = device.apsp_paths(torch.from_numpy(A).cuda(), L, 1e-3)
    assert np.array_equal(H.cpu().numpy(), Ho)
    assert np.array_equal(P.cpu().numpy(), Po)
