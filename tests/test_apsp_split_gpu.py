"""Dense steps whose tiles are split along k over a cluster, against the
oracle's Jacobi steps bit for bit: sizes on both sides of the split limits
(768 and 1088 padded rows) and of a tile's edge."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,L", [(65, 3), (128, 200), (501, 2), (768, 2), (769, 1), (1025, 1), (1153, 1)])
def test_dense_steps_match_oracle(oracle_mod, n, L):
    from netsci_gb300 import device
    rng = np.random.default_rng(n)
    A = (rng.random((n, n)) * 9 + 0.1).astype(np.float32)  # asymmetric, every entry finite
    np.fill_diagonal(A, 0.0)
    Ho, so, _ = oracle_mod.apsp_lengths(A, L)
    H, steps = device.apsp_lengths(torch.from_numpy(A).cuda(), L)
    assert steps == so
    assert np.array_equal(H.cpu().numpy(), Ho)
