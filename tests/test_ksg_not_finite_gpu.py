"""Coordinates that are not numbers, or infinite, in every coordinate of a
frame: small plans (a warp per query) and the bitmap search, whose queries of
such nodes scan all frames, against the tiled kernels, bit for bit.
With one coordinate per node such a frame's marginal distance is itself not a
number, and the joint distance is the other node's."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

KEYS = ("n_x", "n_y", "eps_x", "eps_y", "kdist", "mi")


def _walk(nodes, d, m, seed, step=0.0):
    rng = np.random.default_rng(seed)
    base = rng.standard_normal((1, d, m)) * 0.8
    x = base + rng.standard_normal((nodes, d, m)) * rng.uniform(0.2, 2.0, (nodes, d, 1))
    if step:
        x = np.round(x / step) * step
    return x.astype(np.float32)


def _spoil(x, form):
    _, d, m = x.shape
    rng = np.random.default_rng(m + d)
    if form == "one_node":
        x[0][:, [5, m // 2, m - 1]] = np.nan
        x[1][:, 17] = np.nan
    elif form == "both_nodes":
        x[:, :, [3, m // 3]] = np.nan
    elif form == "inf":
        x[0][:, 9] = np.inf
        x[1][:, [9, 12]] = -np.inf
    elif form == "many":
        x[0][:, rng.random(m) < 0.4] = np.nan
    elif form == "few":  # four frames left, k of six
        x[:, :, 4:] = np.nan
    elif form == "few_inf":
        x[:, :, 4:] = np.inf
        x[0][:, m // 2:] = -np.inf
    return x


def _tiled_shape(X, m, k, d):
    """A tile shape that is there for d and k: forcing it asks for the tiled kernels."""
    from netsci_gb300 import device
    device.set_ksg_search(0)
    try:
        plan = device.KsgPlan(device.make_pairs(X, m, [(0, 1)]), k, d, mi=torch.empty(1, device="cuda"))
    finally:
        device.set_ksg_search(-1)
    s = plan.shape
    plan.close()
    return s["threads"], s["r"], s["frames"], s["variant"]


def _detail(X, m, k, d):
    """Bits of every output, or what the call was refused with: the replay of a
    tie cannot place neighbours where too many distances are not numbers."""
    from netsci_gb300 import _lib, device
    try:
        out = device.ksg_pair_detail(X[0], X[1], m, k, d)
    except _lib.NsgError as e:
        return str(e)
    return {key: out[key].cpu().numpy().view(np.int32) for key in KEYS}


@pytest.mark.parametrize("d,k", [(1, 4), (1, 30), (2, 6), (3, 6)])
@pytest.mark.parametrize("m", [64, 701, 1500])
@pytest.mark.parametrize("step", [0.0, 0.25])
@pytest.mark.parametrize("form", ["one_node", "both_nodes", "inf", "many", "few", "few_inf"])
def test_small_plans_match_tiled(d, k, m, step, form):
    from netsci_gb300 import device
    if form.startswith("few"):
        m = m // 4 * 4  # whole groups of the tiled kernels' frames
    x = _spoil(_walk(2, d, m, 10 * m + d, step), form)
    X, _ = device.pack_trajectory(x.reshape(2, d * m), d)
    _same_as_tiled(X, m, k, d, -1)


@pytest.mark.parametrize("d,k", [(1, 4), (2, 6), (3, 6), (3, 20)])
@pytest.mark.parametrize("m", [1025, 4301])
@pytest.mark.parametrize("step", [0.0, 0.25])
@pytest.mark.parametrize("form", ["one_node", "both_nodes", "inf", "many", "few", "few_inf"])
def test_bitmap_search_matches_tiled(d, k, m, step, form):
    from netsci_gb300 import device
    if form.startswith("few"):
        m = m // 4 * 4
    x = _spoil(_walk(2, d, m, 10 * m + d, step), form)
    X, _ = device.pack_trajectory(x.reshape(2, d * m), d)
    _same_as_tiled(X, m, k, d, 1)


def _same_as_tiled(X, m, k, d, search):
    from netsci_gb300 import device
    device.set_ksg_search(search)
    try:
        got = _detail(X, m, k, d)
    finally:
        device.set_ksg_search(-1)
    device.set_ksg_shape(*_tiled_shape(X, m, k, d))
    try:
        want = _detail(X, m, k, d)
    finally:
        device.set_ksg_shape()
    if isinstance(want, str):
        assert got == want
        return
    for key in KEYS:
        assert np.array_equal(got[key], want[key]), key
