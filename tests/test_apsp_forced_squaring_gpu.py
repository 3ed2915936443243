"""Squaring on request over graphs large and irregular enough that an automatic
solve would relabel their vertices: lengths against the automatic solve's.

Both sum the same positive weights in another order. A path of h edges has
h - 1 rounded sums on either side, so the two differ by less than
2 h 2^-24 of the length, with h at most the automatic solve's steps."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _geometric(n, degree, seed):
    rng = np.random.default_rng(seed)
    pts = rng.random((n, 3))
    r = (degree / (n * 4.0 / 3.0 * np.pi)) ** (1.0 / 3.0)
    w = np.triu((rng.random((n, n)) * 99 + 1).astype(np.float32), 1)
    near = ((pts[:, None, :] - pts[None, :, :]) ** 2).sum(-1) < r * r
    A = np.where(near, w + w.T, np.float32(np.inf)).astype(np.float32)
    np.fill_diagonal(A, 0.0)
    return A


@pytest.mark.parametrize("n,degree", [(300, 8), (2000, 12), (3000, 8)])
@pytest.mark.parametrize("in_place", [False, True])
def test_requested_squaring_matches_automatic(n, degree, in_place):
    from netsci_gb300 import device
    A = torch.from_numpy(_geometric(n, degree, n)).cuda()
    want, steps = device.apsp_lengths(A, n)
    B = A.clone()
    device.set_apsp_method(1)
    try:
        got, _ = device.apsp_lengths(B, n, H=B if in_place else None)
    finally:
        device.set_apsp_method(-1)
    if not in_place:
        assert torch.equal(B, A)
    assert torch.equal(torch.isinf(got), torch.isinf(want))
    near = torch.isfinite(want)
    assert torch.all((got[near] - want[near]).abs() <= 2 * steps * 2.0 ** -24 * want[near])
