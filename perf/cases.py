"""The workloads this library's speed is judged on, through its public entry points.

A case is a dict with a ``kind``:

* ``pair``      one call of ``netcalc.mutualInformationGpu`` or ``generalizedCorrelationGpu``
                on two host arrays: the reference's own unit of work, and the smallest call.
* ``list``      ``netcalc.mutualInformation`` / ``generalizedCorrelation`` over all node pairs
                of a host trajectory: upload, plan, kernels and read-back in one call.
* ``plan``      a reusable ``device.KsgPlan`` over consecutive pairs of the all-pairs list of a
                resident trajectory: the large single system, batch by batch.
* ``uneven``    one plan over all pairs of several resident trajectories of unequal N and m.
* ``bootstrap`` one plan over all pairs of a node subset for several frame resamples.
* ``lengths``   ``device.apsp_lengths`` on a resident random geometric graph.
* ``dense``     ``netcalc.correlationToAdjacency`` and ``hedetniemiAllShortestPathLengths`` on a
                full correlation matrix, host arrays in and out.
* ``paths``     ``netcalc.hedetniemiAllShortestPaths`` (lengths and node sequences) on a contact
                graph, host arrays in and out.

Trajectories are those of the repository's synthetic generator in distribution: a random
walk of 3.8 A steps as the mean structure, five collective modes and isotropic 0.5 A noise.
``motion`` "thermal" takes the modes as random unit vectors over all coordinates (small
per-node amplitudes, nearly independent nodes); "collective" gives every node mode
amplitudes of the order of the noise, so that nodes correlate strongly.
"""
import math

import numpy as np
import torch

import netsci_gb300.cuarray as cuarray
import netsci_gb300.device as device
import netsci_gb300.netcalc as netcalc

MODE_SIGMAS = (2.0, 1.5, 1.0, 0.7, 0.5)


def listed():
    return [
        # Two scalar variables, 2000 samples: the tutorial's Gaussian example, one blocking call.
        dict(name="pair_gauss_2000", kind="pair", gc=False, m=2000, d=1, k=4, rho=0.8),
        # One node pair of a long trajectory, as a program that loops over pairs itself calls it.
        dict(name="pair_gc_10000", kind="pair", gc=True, m=10000, d=3, k=6, rho=0.6),
        # A 56-residue protein, 1000 frames, all pairs: an ordinary small analysis.
        dict(name="list_protein_56", kind="list", gc=True, N=56, m=1000, d=3, k=6, motion="thermal"),
        # An odd-sized system with strongly correlated nodes: an ordinary medium analysis.
        dict(name="list_odd_101", kind="list", gc=True, N=101, m=3001, d=3, k=6, motion="collective"),
        # Two-dimensional variables (dihedral pairs, say) and a larger k, mutual information.
        dict(name="list_planar_k20", kind="list", gc=False, N=40, m=2500, d=2, k=20, motion="collective"),
        # The large system: 8192 pairs of 2000 nodes at 10000 frames, a plan run batch by batch.
        dict(name="plan_2000x10000", kind="plan", N=2000, m=10000, d=3, k=6, pairs=8192, first=0.37,
             motion="thermal"),
        # Many trajectories of unequal length and size in one plan.
        dict(name="uneven_16", kind="uneven", T=16, N_lo=50, N_hi=110, m_lo=500, m_hi=5000, d=3, k=6,
             motion="thermal"),
        # Bootstrap resamples (frames drawn with replacement) of a 100-node subset.
        dict(name="bootstrap_100x2", kind="bootstrap", N=100, m=10000, resamples=2, d=3, k=6,
             motion="thermal"),
        # Shortest paths of a sparse 2000-node graph: integer weights, then real weights.
        dict(name="lengths_int_2000", kind="lengths", N=2000, degree=12.0, integer=True),
        dict(name="lengths_float_2000", kind="lengths", N=2000, degree=12.0, integer=False),
        # Every pair of 500 nodes connected by 1/r of its correlation.
        dict(name="dense_500", kind="dense", N=500),
        # Node sequences of the shortest paths on a 300-residue contact graph.
        dict(name="paths_300", kind="paths", N=300, L=20, tolerance=1e-4),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["pair", "list", "list", "plan", "uneven", "bootstrap", "lengths", "dense", "paths"])
    motion = rng.choice(["thermal", "collective"])
    d = rng.choice([1, 2, 3, 3])
    k = rng.choice([1, 3, 4, 6, 6, 6, 10, 20, 30])
    if kind == "pair":
        return dict(kind=kind, gc=rng.random() < 0.5, m=_log(rng, 500, 20000), d=d, k=k, rho=rng.uniform(0.0, 0.95))
    if kind == "list":
        m = _log(rng, 500, 5000)
        return dict(kind=kind, gc=rng.random() < 0.7, N=_log(rng, 10, 120), m=m, d=d, k=k, motion=motion)
    if kind == "plan":
        m = _log(rng, 1000, 10000)
        most = max(256, min(8192, int(6e11 / m / m)))
        return dict(kind=kind, N=_log(rng, 150, 2000), m=m, d=3, k=6, pairs=_log(rng, 256, most),
                    first=rng.random(), motion=motion)
    if kind == "uneven":
        return dict(kind=kind, T=rng.randint(4, 16), N_lo=20, N_hi=rng.randint(40, 110), m_lo=500,
                    m_hi=rng.randint(1000, 5000), d=3, k=6, motion=motion)
    if kind == "bootstrap":
        return dict(kind=kind, N=rng.randint(20, 90), m=_log(rng, 1000, 10000), resamples=rng.randint(1, 3), d=3, k=6,
                    motion=motion)
    if kind == "lengths":
        return dict(kind=kind, N=_log(rng, 100, 2000), degree=rng.uniform(6.0, 16.0), integer=rng.random() < 0.4)
    if kind == "dense":
        return dict(kind=kind, N=_log(rng, 50, 1000))
    return dict(kind=kind, N=_log(rng, 30, 400), L=rng.randint(5, 30), tolerance=1e-4)


# -- inputs -----------------------------------------------------------------------
def _sizes(c):
    """(N, m) of every trajectory of an "uneven" case, the same for every seed."""
    rng = np.random.default_rng(1000 + c["T"])
    return [(int(rng.integers(c["N_lo"], c["N_hi"] + 1)), int(rng.integers(c["m_lo"], c["m_hi"] + 1)))
            for _ in range(c["T"])]


def _trajectory(N, m, d, motion, seed):
    """(N, d, m) float32 coordinates on the GPU and the (N, d) mean structure."""
    g = torch.Generator(device="cuda").manual_seed(seed)
    step = torch.randn(N, d, generator=g, device="cuda", dtype=torch.float64)
    step *= 3.8 / step.norm(dim=1, keepdim=True)
    mean = step.cumsum(0)
    sig = torch.tensor(MODE_SIGMAS, device="cuda", dtype=torch.float64)
    modes = torch.randn(N * d, len(MODE_SIGMAS), generator=g, device="cuda", dtype=torch.float64)
    if motion == "thermal":
        modes /= modes.norm(dim=0, keepdim=True)
    else:
        modes *= 0.3
    amp = torch.randn(len(MODE_SIGMAS), m, generator=g, device="cuda", dtype=torch.float64) * sig[:, None]
    x = (modes @ amp).reshape(N, d, m) + mean[:, :, None]
    x += 0.5 * torch.randn(N, d, m, generator=g, device="cuda", dtype=torch.float32)
    return x.float(), mean.cpu().numpy()


def _packed(x):
    """Resident layout of ``device``: planes padded to a multiple of 64 samples."""
    N, d, m = x.shape
    out = torch.full((N, d, (m + 63) // 64 * 64), float("inf"), device="cuda")
    out[:, :, :m] = x
    return out


def _all_pairs(N):
    a, b = np.triu_indices(N, 1)
    return np.stack([a, b], axis=1).astype(np.int32)


def _slice(c):
    ab = _all_pairs(c["N"])
    n = min(c["pairs"], len(ab))
    first = int(c["first"] * (len(ab) - n))
    return ab[first:first + n]


def _geometric_graph(N, degree, integer, seed):
    rng = np.random.default_rng(seed)
    pts = rng.random((N, 3))
    r = (degree / (max(N - 1, 1) * 4.0 / 3.0 * np.pi)) ** (1.0 / 3.0)
    near = ((pts[:, None, :] - pts[None, :, :]) ** 2).sum(-1) < r * r
    w = rng.integers(1, 101, size=(N, N)).astype(np.float32) if integer else \
        (rng.random((N, N)) * 99 + 1).astype(np.float32)
    w = np.triu(w, 1)
    A = np.where(near, w + w.T, np.float32(np.inf)).astype(np.float32)
    np.fill_diagonal(A, 0.0)
    return A


def _contact_graph(N, seed):
    """-ln of a correlation on the contacts (closer than 8 A) of a compact chain."""
    rng = np.random.default_rng(seed)
    step = rng.standard_normal((N, 3))
    step *= 3.8 / np.linalg.norm(step, axis=1, keepdims=True)
    pos = np.cumsum(step, axis=0)
    dist = np.linalg.norm(pos[:, None, :] - pos[None, :, :], axis=-1)
    r = np.triu(rng.uniform(0.05, 0.95, (N, N)), 1)
    w = -np.log(r + r.T + np.eye(N))
    A = np.where(dist < 8.0, w, np.inf).astype(np.float32)
    np.fill_diagonal(A, 0.0)
    return A


def _correlations(N, seed):
    rng = np.random.default_rng(seed)
    r = np.triu(rng.beta(2.0, 4.0, (N, N)) * 0.98 + 0.01, 1)
    C = (r + r.T).astype(np.float32)
    np.fill_diagonal(C, 1.0)
    return C


def _float_array(a):
    f = cuarray.FloatCuArray()
    f.fromNumpy2D(np.ascontiguousarray(a, np.float32))
    return f


def _pair_inputs(c, seed):
    rng = np.random.default_rng(seed)
    a = rng.standard_normal((c["d"], c["m"]))
    b = c["rho"] * a + math.sqrt(1.0 - c["rho"] ** 2) * rng.standard_normal((c["d"], c["m"]))
    return a.astype(np.float32), b.astype(np.float32)


def _resamples(c, seed):
    rng = np.random.default_rng(seed + 77)
    return [rng.integers(0, c["m"], c["m"]).astype(np.int32) for _ in range(c["resamples"])]


def prepare(case, seed):
    c, kind = case, case["kind"]
    s = dict(case=c)
    if kind == "pair":
        a, b = _pair_inputs(c, seed)
        s.update(a=_float_array(a), b=_float_array(b))
    elif kind == "list":
        x, _ = _trajectory(c["N"], c["m"], c["d"], c["motion"], seed)
        ab = cuarray.IntCuArray()
        ab.fromNumpy2D(_all_pairs(c["N"]))
        s.update(X=_float_array(x.reshape(c["N"], -1).cpu().numpy()), ab=ab, R=cuarray.FloatCuArray())
    elif kind in ("plan", "uneven", "bootstrap"):
        if kind == "plan":
            x, _ = _trajectory(c["N"], c["m"], c["d"], c["motion"], seed)
            s["keep"] = [_packed(x)]
            pairs = device.make_pairs(s["keep"][0], c["m"], _slice(c))
        elif kind == "uneven":
            s["keep"], pairs = [], []
            for t, (N, m) in enumerate(_sizes(c)):
                x, _ = _trajectory(N, m, c["d"], c["motion"], seed * 1000 + t)
                s["keep"].append(_packed(x))
                pairs += device.make_pairs(s["keep"][-1], m, _all_pairs(N))
        else:
            x, _ = _trajectory(c["N"], c["m"], c["d"], c["motion"], seed)
            s["keep"], pairs = [_packed(x)], []
            for f in _resamples(c, seed):
                s["keep"].append(torch.from_numpy(f).cuda())
                pairs += device.make_pairs(s["keep"][0], c["m"], _all_pairs(c["N"]), fmap=s["keep"][-1])
        s["out"] = [torch.empty(len(pairs), device="cuda") for _ in range(3)]
        s["plan"] = device.KsgPlan(pairs, c["k"], c["d"], mi=s["out"][0], gc=s["out"][1], w=s["out"][2])
        s["plan"].prepare()
    elif kind == "lengths":
        s["A"] = torch.from_numpy(_geometric_graph(c["N"], c["degree"], c["integer"], seed)).cuda()
    elif kind == "dense":
        s.update(C=_float_array(_correlations(c["N"], seed)), A=cuarray.FloatCuArray(), H=cuarray.FloatCuArray())
    else:
        s.update(A=_float_array(_contact_graph(c["N"], seed)), H=cuarray.FloatCuArray(), P=cuarray.IntCuArray())
    return s


# -- one pass ---------------------------------------------------------------------
def run(state):
    c, kind = state["case"], state["case"]["kind"]
    if kind == "pair":
        f = netcalc.generalizedCorrelationGpu if c["gc"] else netcalc.mutualInformationGpu
        return f(state["a"], state["b"], c["k"], c["m"], 2, c["d"])
    if kind == "list":
        f = netcalc.generalizedCorrelation if c["gc"] else netcalc.mutualInformation
        f(state["X"], state["R"], state["ab"], c["k"], c["m"], 2, c["d"])
        return state["R"].toNumpy1D()
    if kind in ("plan", "uneven", "bootstrap"):
        state["plan"].run()
        return state["out"]
    if kind == "lengths":
        return device.apsp_lengths(state["A"], c["N"])
    if kind == "dense":
        netcalc.correlationToAdjacency(state["A"], state["C"], c["N"])
        netcalc.hedetniemiAllShortestPathLengths(state["A"], state["H"], c["N"])
        return [state["A"].toNumpy2D(), state["H"].toNumpy2D()]
    netcalc.hedetniemiAllShortestPaths(state["A"], state["H"], state["P"], c["L"], c["tolerance"])
    return [state["H"].toNumpy2D(), state["P"].toNumpy1D()]


# -- what a pass cannot do without ------------------------------------------------
def _ksg_work(pairs, m, d, k):
    """Per sample of a pair: the distances to its k neighbours (2d differences and maxima)
    and two marginal counts, each at least a binary search per coordinate."""
    return pairs * m * (4.0 * d * k + 2.0 * d * math.ceil(math.log2(m)))


def work(case):
    c, kind = case, case["kind"]
    if kind == "pair":
        return dict(bytes=8.0 * c["d"] * c["m"] + 4, flops=_ksg_work(1, c["m"], c["d"], c["k"]))
    if kind == "list":
        pairs = c["N"] * (c["N"] - 1) // 2
        return dict(bytes=4.0 * c["d"] * c["m"] * c["N"] + 12.0 * pairs, flops=_ksg_work(pairs, c["m"], c["d"], c["k"]))
    if kind == "plan":
        ab = _slice(c)
        return dict(bytes=4.0 * c["d"] * c["m"] * len(np.unique(ab)) + 12.0 * len(ab),
                    flops=_ksg_work(len(ab), c["m"], c["d"], c["k"]))
    if kind == "uneven":
        b = f = 0.0
        for N, m in _sizes(c):
            b += 4.0 * c["d"] * m * N + 6.0 * N * (N - 1)
            f += _ksg_work(N * (N - 1) // 2, m, c["d"], c["k"])
        return dict(bytes=b, flops=f)
    if kind == "bootstrap":
        pairs = c["resamples"] * c["N"] * (c["N"] - 1) // 2
        return dict(bytes=4.0 * c["d"] * c["m"] * c["N"] + 4.0 * c["m"] * c["resamples"] + 12.0 * pairs,
                    flops=_ksg_work(pairs, c["m"], c["d"], c["k"]))
    n2 = float(c["N"]) ** 2
    if kind == "lengths":  # every edge relaxed once for every source, an add and a minimum
        return dict(bytes=8.0 * n2, flops=2.0 * n2 * (c["degree"] + 1))
    if kind == "dense":
        return dict(bytes=12.0 * n2, flops=2.0 * n2 * c["N"])
    return dict(bytes=(8.0 + 4.0 * c["L"]) * n2, flops=2.0 * n2 * c["L"])


# -- the same values in 64 bits ---------------------------------------------------
_EXACT_MOST = 6e9  # sample-sample distances a case may need


def _mi64(a, b, k):
    """KSG estimate (second algorithm) of rows a, b: (d, m) float64 tensors."""
    m = a.shape[1]
    total = torch.zeros((), dtype=torch.float64, device=a.device)
    step = max(1, min(m, (1 << 26) // m))
    for q in range(0, m, step):
        da = (a[:, q:q + step, None] - a[:, None, :]).abs().amax(0)
        db = (b[:, q:q + step, None] - b[:, None, :]).abs().amax(0)
        near = torch.maximum(da, db).topk(k + 1, dim=1, largest=False).indices
        ea = da.gather(1, near).amax(1, keepdim=True)
        eb = db.gather(1, near).amax(1, keepdim=True)
        nx = (da <= ea).sum(1) - 1
        ny = (db <= eb).sum(1) - 1
        total += (torch.digamma(nx.double()) + torch.digamma(ny.double())).sum()
    psi = torch.digamma(torch.tensor([m, k], dtype=torch.float64))
    return float(psi[0] + psi[1]) - 1.0 / k - float(total) / m


def _gc64(mi, d):
    return math.sqrt(1.0 - math.exp(-2.0 * mi / d)) if mi > 0 else 0.0


def _relaxed(A, steps):
    """Shortest walks of at most steps + 1 edges from a 64-bit symmetric weight matrix."""
    H = A.clone()
    for _ in range(steps):
        N = torch.stack([(A[j][:, None] + H).amin(0) for j in range(A.shape[0])], dim=1)
        if torch.equal(N, H):
            break
        H = N
    return H


def _closure(A):
    H = A.clone()
    for v in range(A.shape[0]):
        H = torch.minimum(H, H[:, v:v + 1] + H[v:v + 1, :])
    return H


def exact(case, seed):
    c, kind = case, case["kind"]
    if kind == "pair":
        a, b = (torch.from_numpy(v).cuda().double() for v in _pair_inputs(c, seed))
        mi = _mi64(a, b, c["k"])
        return _gc64(mi, c["d"]) if c["gc"] else mi
    if kind == "list":
        if c["N"] * (c["N"] - 1) / 2 * c["m"] ** 2 > _EXACT_MOST:
            return None
        x = _trajectory(c["N"], c["m"], c["d"], c["motion"], seed)[0].double()
        mi = [_mi64(x[a], x[b], c["k"]) for a, b in _all_pairs(c["N"])]
        return np.array([_gc64(v, c["d"]) for v in mi] if c["gc"] else mi)
    if kind in ("plan", "uneven", "bootstrap"):
        return None
    if kind == "lengths":
        A = torch.from_numpy(_geometric_graph(c["N"], c["degree"], c["integer"], seed)).cuda().double()
        return (_closure(A), None)
    if kind == "dense":
        C = torch.from_numpy(_correlations(c["N"], seed)).cuda().double()
        A = 1.0 / C
        A.fill_diagonal_(0.0)
        return [A, _closure(A)]
    A = torch.from_numpy(_contact_graph(c["N"], seed)).cuda().double()
    return [_relaxed(A, c["L"]), None]
