"""The bitmap search on data its radius estimates were not made for: nodes and
coordinates that do not move, frames far from all others, frames on a line,
nodes that repeat each other, drift, mostly equal frames and long tails. Results
against the tiled kernels bit for bit; and where distances do not tie, queries
settle on their bitmaps rather than scan all frames."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

FORMS = ["flat", "still", "all_still", "outlier", "line", "twice", "drift", "mostly_zero", "tails"]
TIED = ("all_still", "mostly_zero")


def _form(form, nodes, d, m):
    rng = np.random.default_rng(m + d)
    x = rng.standard_normal((1, d, m)) * 0.8 + rng.standard_normal((nodes, d, m)) * rng.uniform(0.2, 2.0, (nodes, d, 1))
    if form == "flat":
        x[:, d - 1] = 0.0
    elif form == "still":
        x[::2] = 1.5
    elif form == "all_still":
        x[:] = 1.5
        x[:, :, 3] = 2.0
    elif form == "outlier":
        x[:, :, [7, m - 1]] = 1e6
    elif form == "line":
        x = x[:, :1] * np.ones((1, d, 1))
    elif form == "twice":
        x[1::2] = x[0::2][:x[1::2].shape[0]]
    elif form == "drift":
        x = np.cumsum(x * 0.05, axis=2)
    elif form == "mostly_zero":
        x = x * (rng.random((nodes, 1, m)) < 0.1)
    elif form == "tails":
        x = np.sign(x) * np.abs(x) ** 5
    return np.ascontiguousarray(x, np.float32).reshape(nodes, d * m)


def _run(X, m, k, d, ab, shape=None):
    from netsci_gb300 import device
    mi = torch.empty(len(ab), device="cuda")
    if shape is None:
        device.set_ksg_search(1)
    else:
        device.set_ksg_shape(*shape)
    try:
        plan = device.KsgPlan(device.make_pairs(X, m, ab), k, d, mi=mi)
    finally:
        device.set_ksg_search(-1)
        device.set_ksg_shape()
    plan.run()
    torch.cuda.synchronize()
    plan.check()
    s = plan.shape
    looked = plan.evaluations()[0] / (len(ab) * m)
    plan.close()
    return mi.cpu().numpy().view(np.int32), looked, (s["threads"], s["r"], s["frames"], s["variant"])


@pytest.mark.parametrize("d,k,m", [(1, 4, 3000), (2, 6, 2600), (3, 6, 1200), (3, 6, 2600), (3, 20, 3000), (3, 6, 5300)])
@pytest.mark.parametrize("form", FORMS)
def test_forms_match_tiled_and_settle(d, k, m, form):
    from netsci_gb300 import device
    nodes = 4
    X, _ = device.pack_trajectory(_form(form, nodes, d, m), d)
    ab = [(a, b) for a in range(nodes) for b in range(a + 1, nodes)]
    got, looked, _ = _run(X, m, k, d, ab)
    device.set_ksg_search(0)
    try:
        plan = device.KsgPlan(device.make_pairs(X, m, ab), k, d, mi=torch.empty(len(ab), device="cuda"))
        s = plan.shape
        plan.close()
    finally:
        device.set_ksg_search(-1)
    want, _, _ = _run(X, m, k, d, ab, (s["threads"], s["r"], s["frames"], s["variant"]))
    assert np.array_equal(got, want)
    if form not in TIED and not (form == "flat" and d == 1):
        assert looked < m / 4, looked
