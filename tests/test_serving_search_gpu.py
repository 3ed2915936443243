"""Serving on either kernel of node grids and either search: the results of a resident trajectory's
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


# both searches of a tick: low d and k scan the cells, the others take bitmaps;
# m up to 6001 puts jobs over several ticks
@pytest.mark.parametrize("N,m,d,k", [
    (30, 1000, 1, 1), (30, 1027, 1, 3), (40, 1500, 1, 6), (12, 1000, 1, 14), (37, 1001, 2, 1), (38, 1033, 2, 6),
    (39, 1000, 3, 1), (20, 1500, 3, 6), (9, 6001, 1, 2), (9, 6001, 3, 20)])
def test_ticks_match_plans(N, m, d, k):
    _served_equals_plan(N, m, d, k)
