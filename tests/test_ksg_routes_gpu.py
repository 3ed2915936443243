"""Every route of a plan named and checked: bitmaps and the scan of cells against
the tiled kernels bit for bit, at both sides of each change of the bitmap
search's layout (words a lane, bins a row, warps and CTAs), for every list
length of the scan, with and without query orders, ties resolved by the scan's
record and by its second scan; and which route plans take by themselves past the
largest m whose bitmaps fit."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _walk(nodes, d, m, seed, step=0.0):
    rng = np.random.default_rng(seed)
    base = rng.standard_normal((1, d, m)) * 0.8
    x = base + rng.standard_normal((nodes, d, m)) * rng.uniform(0.2, 2.0, (nodes, d, 1))
    if step:
        x = np.round(x / step) * step
    return x.reshape(nodes, d * m).astype(np.float32)


def _run(pairs, k, d, route):
    from netsci_gb300 import device
    mi = torch.empty(len(pairs), device="cuda")
    plan = device.KsgPlan(pairs, k, d, mi=mi, route=route)
    took = plan.route
    plan.run()
    torch.cuda.synchronize()
    plan.check()
    ties = plan.tied_samples()
    plan.close()
    return mi.cpu().numpy().view(np.int32), took, ties


def _compare(x, m, k, d, routes, ab=((0, 1),)):
    from netsci_gb300 import device
    X, _ = device.pack_trajectory(x, d)
    pairs = device.make_pairs(X, m, list(ab))
    want, took, _ = _run(pairs, k, d, "tiled")
    assert took == "tiled"
    for route in routes:
        got, took, _ = _run(pairs, k, d, route)
        assert took == route
        assert np.array_equal(got, want), route


# last m of a layout and the first of the next, for rows of 54 bins
EDGES = {(1, 6): [2433, 5249, 11137, 14052, 22657], (1, 13): [9601, 19841], (2, 6): [897, 1921, 3211, 4225, 7725, 8577, 15745],
         (2, 13): [641, 2589, 6282], (3, 6): [385, 1153, 1859, 2689, 4209, 5505, 10369, 10625, 10977, 17793, 18305, 19017],
         (3, 13): [1615, 2177, 3664, 4737, 9089, 9601], (3, 30): [1385, 3147]}


@pytest.mark.parametrize("d,k,m", [(d, k, m + s) for (d, k), ms in EDGES.items() for m in ms for s in (-1, 0)])
def test_bitmap_layouts(d, k, m):
    _compare(_walk(2, d, m, 100 * d + k + m), m, k, d, ["bitmaps"])


@pytest.mark.parametrize("d,k,m,route", [(3, 6, 24448, "bitmaps"), (3, 6, 25425, "bitmaps"), (3, 6, 26240, "bitmaps"),
                                         (3, 6, 26241, "scan"), (3, 13, 24704, "bitmaps"), (3, 13, 24705, "scan"),
                                         (2, 6, 37040, "bitmaps"), (2, 6, 37041, "scan")])
def test_largest_bitmaps(d, k, m, route):
    from netsci_gb300 import device
    from netsci_gb300._lib import NsgError
    x = _walk(2, d, m, m)
    X, _ = device.pack_trajectory(x, d)
    pairs = device.make_pairs(X, m, [(0, 1)])
    plan = device.KsgPlan(pairs, k, d, mi=torch.empty(1, device="cuda"))
    assert plan.route == route
    plan.close()
    if route == "scan":
        with pytest.raises(NsgError):
            device.KsgPlan(pairs, k, d, mi=torch.empty(1, device="cuda"), route="bitmaps")
    _compare(x, m, k, d, [route])


@pytest.mark.parametrize("d,k,m", [(1, 4, 2500), (2, 6, 3001), (3, 6, 4096), (3, 1, 2100), (3, 14, 2600), (3, 17, 2600),
                                   (2, 31, 2200), (3, 62, 2300), (3, 6, 50), (1, 3, 9), (3, 6, 24000)])
@pytest.mark.parametrize("step", [0.0, 0.125])
@pytest.mark.parametrize("orders", [0, 1])
def test_scan_of_cells(d, k, m, step, orders):
    from netsci_gb300 import device
    if m > 20000 and step:
        pytest.skip("thousands of long replays")
    device.set_ksg_orders(orders)
    try:
        _compare(_walk(4, d, m, m + k, step), m, k, d, ["scan", "bitmaps"], [(0, 1), (2, 1), (0, 3)])
    finally:
        device.set_ksg_orders(-1)


@pytest.mark.parametrize("k", [1, 6, 17])
def test_scan_tie_record_matches_second_scan(oracle_mod, k):
    """Frame-mapped pairs keep a record of ties while they scan; the same rows
    copied out by hand scan the cells again. Both list the same samples."""
    from netsci_gb300 import device, synthetic
    N, m = 5, 2300
    X, _ = synthetic.protein_trajectory(N, m, seed=11)
    idx = np.random.default_rng(12).integers(0, m, size=m).astype(np.int32)
    fmap = torch.from_numpy(idx).cuda()
    Xd, mm = device.pack_trajectory(X, 3)
    Xr = np.ascontiguousarray(X.reshape(N, 3, m)[:, :, idx].reshape(N, 3 * m))
    Xrd, _ = device.pack_trajectory(Xr, 3)
    ab = synthetic.all_pairs(N)
    want = np.asarray(oracle_mod.pairs(Xr, m, 3, ab, k, gc=False, threads=8), np.float32).view(np.int32)
    ties = []
    for pairs in (device.make_pairs(Xd, mm, ab, fmap=fmap, m_samples=m), device.make_pairs(Xrd, mm, ab)):
        got, took, n = _run(pairs, k, 3, "scan")
        assert took == "scan"
        assert np.array_equal(got, want)
        ties.append(n)
    assert ties[0] == ties[1]


@pytest.mark.parametrize("d,k,m", [(1, 1, 2), (1, 30, 31), (2, 5, 33), (3, 6, 1201), (3, 30, 500)])
@pytest.mark.parametrize("step", [0.0, 0.5])
def test_warp_route(d, k, m, step):
    _compare(_walk(3, d, m, m + k, step), m, k, d, ["warp"], [(0, 1), (2, 0)])


@pytest.mark.parametrize("m", [20479, 20480, 20481])
def test_ties_around_the_longest_shared_row(oracle_mod, m):
    """A CTA replays a tied sample in shared memory up to 20480 frames."""
    from netsci_gb300 import device
    x = _walk(2, 1, m, m).reshape(2, m)
    x[:, :4000] = np.round(x[:, :4000] * 512) / 512
    X, _ = device.pack_trajectory(x, 1)
    got, _, ties = _run(device.make_pairs(X, m, [(0, 1)]), 6, 1, None)
    assert ties > 0
    assert got.view(np.float32)[0] == oracle_mod.mi_pair(x[0], x[1], m, 6, 1)


def test_routes_that_do_not_take_the_pairs():
    from netsci_gb300 import device
    from netsci_gb300._lib import NsgError
    X, _ = device.pack_trajectory(_walk(2, 3, 200, 1), 3)
    with pytest.raises(NsgError):  # lists of the warp kernel end at k = 30
        device.KsgPlan(device.make_pairs(X, 200, [(0, 1)]), 31, 3, mi=torch.empty(1, device="cuda"), route="warp")


@pytest.mark.parametrize("n", [1023, 1024, 1025])
def test_dense_steps_around_the_split(oracle_mod, n):
    """Dense shortest-path steps share a tile between two CTAs up to n = 1024."""
    from netsci_gb300 import device
    A = (np.random.default_rng(n).random((n, n)) * 9 + 0.1).astype(np.float32)
    np.fill_diagonal(A, 0.0)
    Ho, so, _ = oracle_mod.apsp_lengths(A, 1)
    H, steps = device.apsp_lengths(torch.from_numpy(A).cuda(), 1)
    assert steps == so
    assert np.array_equal(H.cpu().numpy(), Ho)
