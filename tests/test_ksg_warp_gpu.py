"""Small exhaustive plans, a warp per query, against the oracle bit for bit:
sizes at the edges of a warp's frames (32) and of a CTA's queries (16), the
largest m and k taken, ties and copies of one frame beyond a query's list."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.fixture
def exhaustive():
    from netsci_gb300 import device
    device.set_ksg_search(0)
    yield
    device.set_ksg_search(-1)


@pytest.mark.parametrize("d,k,n,step", [(1, 1, 2, 0), (1, 4, 31, 0), (2, 5, 32, 0), (3, 6, 33, 0), (1, 30, 1000, 0),
                                        (3, 29, 545, 0), (3, 6, 4096, 0), (2, 3, 2049, 0), (1, 4, 1600, 0.5),
                                        (3, 6, 1201, 0.5), (1, 7, 700, 4.0)])
def test_small_plan_matches_oracle(oracle_mod, exhaustive, d, k, n, step):
    from netsci_gb300 import device
    rng = np.random.default_rng(1000 * d + n + k)
    xa = rng.standard_normal(d * n).astype(np.float32)
    xb = (0.7 * xa + 0.7 * rng.standard_normal(d * n)).astype(np.float32)
    if step:
        xa, xb = np.round(xa / step) * np.float32(step), np.round(xb / step) * np.float32(step)
        xa, xb = xa.astype(np.float32), xb.astype(np.float32)
    mi, det = oracle_mod.mi_pair(xa, xb, n, k, d, detail=True)
    X, m = device.pack_trajectory(np.stack([xa, xb]), d)
    out = device.ksg_pair_detail(X[0], X[1], m, k, d)
    for key in ("n_x", "n_y", "eps_x", "eps_y", "kdist"):
        assert np.array_equal(out[key].cpu().numpy(), det[key]), key
    assert float(out["mi"].item()) == mi


def test_small_plan_of_mapped_and_uneven_pairs(oracle_mod, exhaustive):
    """Frame maps are followed; pairs of different m share one launch."""
    from netsci_gb300 import device
    rng = np.random.default_rng(5)
    pairs, expect, keep = [], [], []
    for m, k in ((40, 6), (700, 6), (1300, 6)):
        X = rng.standard_normal((2, 3 * m)).astype(np.float32)
        Xd, _ = device.pack_trajectory(X, 3)
        idx = rng.integers(0, m, m).astype(np.int32)
        fm = torch.from_numpy(idx).cuda()
        keep += [Xd, fm]
        pairs += device.make_pairs(Xd, m, [[0, 1]]) + device.make_pairs(Xd, m, [[0, 1]], fmap=fm, m_samples=m)
        Xr = np.ascontiguousarray(X.reshape(2, 3, m)[:, :, idx]).reshape(2, 3 * m)
        expect += [oracle_mod.mi_pair(X[0], X[1], m, k, 3), oracle_mod.mi_pair(Xr[0], Xr[1], m, k, 3)]
    mi = torch.empty(len(pairs), device="cuda")
    device.ksg_pairs(pairs, 6, 3, mi=mi)
    assert mi.cpu().numpy().tolist() == expect
