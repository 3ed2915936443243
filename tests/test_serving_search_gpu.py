"""Serving on either kernel of node grids: the results of a resident trajectory's
jobs equal a plan's, bit for bit."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _served_equals_plan(N, m, d, k):
    import torch
    from netsci_gb300 import device, serving, synthetic
    rng = np.random.default_rng(N * m + d)
    x = np.cumsum(rng.standard_normal((N, d, m)), axis=2) * 0.05 + rng.standard_normal((N, d, m))
    x = np.ascontiguousarray(x.reshape(N, d * m), np.float32)
    with serving.Server(budget_bytes=1 << 30) as srv:
        t = srv.register_trajectory(x, d)
        jobs = [srv.submit_gc(t, N, k) for _ in range(2)]
        got = [srv.wait(j) for j in jobs]
    Xd, m = device.pack_trajectory(x, d)
    pairs = device.make_pairs(Xd, m, synthetic.all_pairs(N))
    want = torch.empty(len(pairs), device="cuda")
    device.ksg_pairs(pairs, k, d, gc=want)
    for g in got:
        assert np.array_equal(g, want.cpu().numpy())


@pytest.mark.parametrize("d", [1, 2, 3])
@pytest.mark.parametrize("N", [37, 38, 61])  # one kernel for all node grids, and four
def test_registered_node_grids(N, d):
    _served_equals_plan(N, 1001, d, 6)
