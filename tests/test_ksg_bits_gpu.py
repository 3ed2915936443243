"""Bitmap search and the counts that follow it, against the exhaustive kernels
bit for bit: sizes on both sides of every change of the search's words per
lane, bins per row, warps per CTA and list length, and past the largest m whose
rows fit; counts in groups of one to seven variables and by rank; ties around
the longest row kept in shared memory; coordinates that are not finite."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

KEYS = ("n_x", "n_y", "eps_x", "eps_y", "kdist", "mi")


def _both(f):
    """f() with the cell-grid search and with the exhaustive one."""
    from netsci_gb300 import device
    out = []
    try:
        for mode in (1, 0):
            device.set_ksg_search(mode)
            out.append(f())
    finally:
        device.set_ksg_search(-1)
    return out


def _bits(t):
    return t.cpu().numpy().view(np.int32)


def _same_detail(x, m, k, d):
    from netsci_gb300 import device
    X, _ = device.pack_trajectory(x, d)
    got, want = _both(lambda: device.ksg_pair_detail(X[0], X[1], m, k, d))
    for key in KEYS:
        assert np.array_equal(_bits(got[key]), _bits(want[key])), key


def _walk(nodes, d, m, seed, step=0.0):
    rng = np.random.default_rng(seed)
    base = rng.standard_normal((1, d, m)) * 0.8
    x = base + rng.standard_normal((nodes, d, m)) * rng.uniform(0.2, 2.0, (nodes, d, 1))
    if step:
        x = np.round(x / step) * step
    return x.reshape(nodes, d * m).astype(np.float32)


# (d, k, m): the last m before a change of configuration, and the first after
@pytest.mark.parametrize("d,k,m", [
    (1, 6, 14051), (1, 6, 14053), (1, 12, 11650), (1, 13, 11355), (1, 30, 21637), (1, 6, 19361),
    (2, 6, 3210), (2, 6, 3212), (2, 6, 7726), (2, 12, 2648), (2, 13, 2589), (2, 6, 8353), (2, 6, 15777), (2, 62, 17001),
    (3, 6, 1858), (3, 6, 1860), (3, 6, 4208), (3, 6, 4210), (3, 12, 1640), (3, 13, 1615), (3, 6, 401), (3, 6, 5025),
    (3, 6, 9377), (3, 6, 10657), (3, 6, 18081), (3, 30, 21409), (3, 6, 25021), (3, 6, 25057), (3, 13, 23713)])
def test_every_configuration_matches_exhaustive(d, k, m):
    _same_detail(_walk(2, d, m, 100 * d + k + m), m, k, d)


@pytest.mark.parametrize("d,k,m", [(1, 4, 1300), (2, 12, 1500), (3, 6, 2700), (3, 20, 4300)])
@pytest.mark.parametrize("form", ["rounded", "coarse", "constant", "copies", "heavy"])
def test_distributions_match_exhaustive(d, k, m, form):
    x = _walk(2, d, m, m, {"rounded": 0.125, "coarse": 2.0}.get(form, 0.0)).reshape(2, d, m)
    if form == "constant":
        x[0, 0] = 3.25
        x[1, d - 1] = -1.0
    elif form == "copies":  # each frame about 50 times
        x = x[:, :, np.random.default_rng(3).integers(0, m // 50, m)]
    elif form == "heavy":
        x = np.sign(x) * np.abs(x) ** 9
    _same_detail(np.ascontiguousarray(x).reshape(2, d * m), m, k, d)


@pytest.mark.parametrize("d,m", [(2, 1200), (3, 1500), (3, 4300)])
@pytest.mark.parametrize("form", ["inf", "nan", "overflow"])
def test_not_finite_matches_exhaustive(d, m, form):
    """Infinite and NaN coordinates in a few frames, and finite ones whose
    differences overflow; the pair's and a star's counts."""
    from netsci_gb300 import device
    x = _walk(10, d, m, 7 * m + d).reshape(10, d, m)
    if form == "inf":
        x[0, 1, 5] = x[0, 1, 77] = x[3, 0, 9] = np.inf
        x[1, 0, 300] = -np.inf
    elif form == "nan":
        x[0, 0, 11] = x[4, 1, 500] = x[1, 1, 11] = np.nan
    else:
        x[0] *= np.float32(3e38) / np.abs(x[0]).max()
        x[2, 0] *= np.float32(3e38) / np.abs(x[2, 0]).max()
    x = x.reshape(10, d * m)
    _same_detail(x[:2], m, 6, d)
    _same_pairs(x, m, 6, d, [(0, b) for b in range(1, 10)] + [(2, 5), (3, 4)])


def _same_pairs(x, m, k, d, ab, fmap=None):
    from netsci_gb300 import device
    X, _ = device.pack_trajectory(x, d)
    f = None if fmap is None else torch.from_numpy(fmap).cuda()
    pairs = device.make_pairs(X, m, ab, fmap=f, m_samples=m)

    def run():
        mi = torch.empty(len(pairs), device="cuda")
        device.ksg_pairs(pairs, k, d, mi=mi)
        return mi

    got, want = _both(run)
    assert np.array_equal(_bits(got), _bits(want))


@pytest.mark.parametrize("d", [1, 2, 3])
@pytest.mark.parametrize("partners", [1, 2, 3, 4, 5, 6, 7, 8, 9, 13, 32, 33, 255, 256, 257, 261])
@pytest.mark.parametrize("orders", [0, 1])
def test_counts_of_a_star_match_exhaustive(d, partners, orders):
    """One node in `partners` pairs: groups up to seven; with query orders
    ranks from eight on, in passes of 256 whose last one may hold one to four
    variables; without, direct comparisons of up to four in small batches."""
    from netsci_gb300 import device
    m = 1025
    try:
        device.set_ksg_orders(orders)
        _same_pairs(_walk(partners + 1, d, m, partners, 0.03125 if partners % 2 else 0.0), m, 4, d,
                    [(0, b) if b % 3 else (b, 0) for b in range(1, partners + 1)])
    finally:
        device.set_ksg_orders(-1)


@pytest.mark.parametrize("d,k,m,nodes", [(1, 1, 500, 12), (1, 6, 4001, 9), (1, 9, 1000, 40), (1, 20, 1000, 40),
                                         (2, 1, 2200, 18), (2, 6, 700, 18), (2, 6, 2200, 18), (3, 1, 1400, 18),
                                         (3, 6, 700, 38), (3, 6, 1025, 39), (3, 30, 500, 20)])
@pytest.mark.parametrize("step", [0.0, 0.25])
@pytest.mark.parametrize("mapped", [False, True])
def test_lists_on_either_side_of_the_scan(d, k, m, nodes, step, mapped):
    """All pairs of a few nodes, where the estimates choose between the scan of
    cells and the bitmaps; also resampled (copies of frames)."""
    fmap = np.random.default_rng(m).integers(0, m, m).astype(np.int32) if mapped else None
    _same_pairs(_walk(nodes, d, m, nodes + m, step), m, k, d,
                [(a, b) for a in range(nodes) for b in range(a + 1, nodes)], fmap)


def test_chain_of_many_nodes():
    """More than a wave of nodes with two variables each."""
    _same_pairs(_walk(200, 3, 601, 9), 601, 6, 3, [(a, a + 1) for a in range(199)])


@pytest.mark.parametrize("m", [3399, 3400, 3401])
@pytest.mark.parametrize("d", [1, 3])
def test_ties_around_the_longest_shared_row(oracle_mod, m, d):
    from netsci_gb300 import device
    x = _walk(2, d, m, m, 0.25)
    mi, det = oracle_mod.mi_pair(x[0], x[1], m, 6, d, detail=True)
    assert det["ties"] > 0
    X, _ = device.pack_trajectory(x, d)
    out = device.ksg_pair_detail(X[0], X[1], m, 6, d)
    for key in KEYS[:5]:
        assert np.array_equal(out[key].cpu().numpy(), det[key]), key
    assert float(out["mi"].item()) == mi


@pytest.mark.parametrize("m", [17, 401, 2450, 2500, 5150, 5200, 20480])
@pytest.mark.parametrize("d,k", [(1, 3), (3, 40)])
def test_ties_match_the_kernel_for_long_rows(m, d, k):
    """A pair of longer rows in the plan sends every tie to that kernel."""
    from netsci_gb300 import device
    if k >= m:
        k = m - 2
    X, _ = device.pack_trajectory(_walk(2, d, m, m + d, 0.5), d)
    L, _ = device.pack_trajectory(_walk(2, d, 20481, 1, 1.0), d)
    own = device.make_pairs(X, m, [(0, 1)])
    mi = torch.empty(3, device="cuda")
    device.ksg_pairs(own, k, d, mi=mi[:1])
    device.ksg_pairs(own + device.make_pairs(L, 20481, [(0, 1)]), k, d, mi=mi[1:])
    assert _bits(mi[0:1]) == _bits(mi[1:2])


@pytest.mark.parametrize("m", [7, 8, 9, 511, 512, 513, 1023, 1024, 1025, 2049, 4100])
def test_sums_at_chunk_edges(oracle_mod, m):
    """The serial sum over the samples, in its chunks of 512."""
    from netsci_gb300 import device
    x = _walk(2, 1, m, m)
    X, _ = device.pack_trajectory(x, 1)
    mi = torch.empty(1, device="cuda")
    device.ksg_pairs(device.make_pairs(X, m, [(0, 1)]), 3, 1, mi=mi)
    assert float(mi.item()) == oracle_mod.mi_pair(x[0], x[1], m, 3, 1)
