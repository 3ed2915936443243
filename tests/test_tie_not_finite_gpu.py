"""Ties among frames of which some are not numbers in both nodes: their joint
distance is neither smaller nor larger than any other, and the replayed sort
(sort_prefix.h) leaves them wherever its steps do. The tie kernels, a CTA per
sample up to 20480 frames and a warp per sample beyond, against that routine
run serially on the host."""
import ctypes
import shutil
import subprocess
from pathlib import Path

import numpy as np
import pytest

ROOT = Path(__file__).resolve().parent.parent


@pytest.fixture(scope="module")
def replay(tmp_path_factory):
    cxx = shutil.which("g++")
    if cxx is None:
        pytest.skip("no g++")
    so = tmp_path_factory.mktemp("sort") / "rows.so"
    subprocess.run([cxx, "-O2", "-std=c++17", "-shared", "-fPIC", "-I", str(ROOT / "netsci_gb300" / "csrc"),
                    str(ROOT / "tests" / "native" / "sort_prefix_rows.cpp"), "-o", str(so)], check=True)
    f = ctypes.CDLL(str(so)).sort_prefix_row

    def order(key, T):
        key = np.ascontiguousarray(key, np.float32)
        idx = np.empty(len(key), np.int32)
        assert f(key.ctypes.data_as(ctypes.c_void_p), idx.ctypes.data_as(ctypes.c_void_p), len(key), T)
        return idx[:T]
    return order


def _case(d, m, seed):
    rng = np.random.default_rng(seed)
    xa = np.round(rng.standard_normal((d, m)) * 4) / 4
    xb = np.round((0.6 * xa + rng.standard_normal((d, m))) * 4) / 4
    lost = rng.choice(m, 6, replace=False)
    xa[:, lost] = xb[:, lost] = np.nan
    return xa.astype(np.float32), xb.astype(np.float32), lost


def _expected(xa, xb, k, replay, queries):
    """{query: (n_x, n_y, eps_x, eps_y)} of the queries whose neighbours the sort's order decides."""
    out = {}
    for q in queries:
        da = np.abs(xa - xa[:, q:q + 1]).max(0)
        db = np.abs(xb - xb[:, q:q + 1]).max(0)
        dz = np.maximum(da, db)
        near = np.sort(dz[~np.isnan(dz)])
        u = near[k]
        at = dz == u
        if u == 0 or (near <= u).sum() <= k + 1:
            continue
        if len(set(zip(da[at], db[at]))) == 1:
            continue
        idx = replay(dz, k + 1)[1:]
        ex, ey = np.nanmax(np.append(da[idx], 0)), np.nanmax(np.append(db[idx], 0))
        out[q] = ((da <= ex).sum() - 1, (db <= ey).sum() - 1, ex, ey)
    return out


@pytest.mark.gpu
@pytest.mark.parametrize("d,m,k", [(1, 40, 4), (1, 701, 6), (3, 700, 6), (2, 4097, 20), (3, 9000, 6), (3, 20483, 6)])
def test_ties_with_lost_frames_follow_the_sort(replay, d, m, k):
    from netsci_gb300 import device
    xa, xb, lost = _case(d, m, m)
    queries = np.setdiff1d(np.arange(m), lost)[:1500]
    want = _expected(xa, xb, k, replay, queries)
    assert len(want) >= 5
    X, _ = device.pack_trajectory(np.stack([xa, xb]).reshape(2, d * m), d)
    out = device.ksg_pair_detail(X[0], X[1], m, k, d)
    got = [out[key].cpu().numpy() for key in ("n_x", "n_y", "eps_x", "eps_y")]
    for q, w in want.items():
        assert tuple(g[q] for g in got) == w, q
