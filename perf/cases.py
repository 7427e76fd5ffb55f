"""The measured workloads: what a user of this package has it compute.

A user holds the mean-centred coordinates of a trajectory (synth_traj stands
in for MD data) and asks for the matrix of one estimator: KSG, Gaussian,
Gaussian-copula (GCMI) or transfer entropy (TE).  Analysis scripts call the
functions that take and return numpy arrays; programs that keep trajectories
on the GPU use the plans (KsgPlan, TePlan).  The sizes are the package's own
configurations (64 x 500, 247 x 2000, 5000-frame trajectories, uneven batches)
and odd sizes around them.

listed() names twelve cases, draw() gives more of the same ranges, prepare()
makes inputs and plans, run() is one pass, work() the bytes and operations a
pass cannot do without, exact() the result in plain float64 torch.
"""

import math

import numpy as np
import torch

import gmx_correlation_b200 as gc
from gmx_correlation_b200.synth import synth_traj

# One stream for everything a program with device-resident plans enqueues.
_STREAM = None
_SCREEN = None

# (natoms, nframes, k) ranges of each kind; lags of the TE kinds.  The upper
# ends are the listed cases' sizes or their cost (pairs x frames^2).
_KINDS = ("ksg", "wrap", "plan", "long", "noalloc", "batch", "gauss", "gcmi", "te", "teplan", "screened")


def listed():
    return [
        # the small configuration, arrays in and out: one matrix of a short trajectory in a script
        {"name": "ksg 64x500 k10", "kind": "ksg", "natoms": 64, "nframes": 500, "k": 10},
        # one pair of already normalised rows: the smallest call, where latency and launches count
        {"name": "ksg pair 2000 k100", "kind": "wrap", "natoms": 2, "nframes": 2000, "k": 100},
        # the headline matrix with coordinates resident on the GPU
        {"name": "ksg 247x2000 k100", "kind": "plan", "natoms": 247, "nframes": 2000, "k": 100},
        # a long production run of a smaller protein: 5000-frame rows, odd sizes
        {"name": "ksg 151x4999 k100", "kind": "plan", "natoms": 151, "nframes": 4999, "k": 100},
        # a few residues over a very long trajectory (more frames than the row sort takes)
        {"name": "ksg 8x20001 k50", "kind": "long", "natoms": 8, "nframes": 20001, "k": 50},
        # a plugin that may not allocate device memory
        {"name": "ksg noalloc 48x901 k20", "kind": "noalloc", "natoms": 48, "nframes": 901, "k": 20},
        # replicas of a small peptide analysed together, each with its own length
        {"name": "ksg batch 24", "kind": "batch", "count": 24, "natoms": 60, "nframes": 900, "k": 10},
        # -linear of a large protein, arrays in and out
        {"name": "gauss 600x4000", "kind": "gauss", "natoms": 600, "nframes": 4000, "k": 0},
        # the copula estimator on the reference protein, arrays in and out
        {"name": "gcmi 247x2000", "kind": "gcmi", "natoms": 247, "nframes": 2000, "k": 0},
        # information flow between a few residues in a script
        {"name": "te 40x700 k10 lag5", "kind": "te", "natoms": 40, "nframes": 700, "k": 10, "lag": 5},
        # transfer entropy of the headline trajectory, resident on the GPU
        {"name": "te 247x2000 k100 lag1", "kind": "teplan", "natoms": 247, "nframes": 2000, "k": 100, "lag": 1},
        # the learned screen keeping its predictions, exact KSG on the audit sample
        {"name": "screened 247x2000 k100", "kind": "screened", "natoms": 247, "nframes": 2000, "k": 100},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(_KINDS)
    c = {"kind": kind}
    if kind == "ksg":
        c.update(natoms=_log_int(rng, 8, 120), nframes=rng.randint(200, 1600), k=rng.choice([4, 6, 10, 20]))
    elif kind == "wrap":
        c.update(natoms=2, nframes=_log_int(rng, 300, 5000), k=rng.choice([6, 10, 50, 100]))
    elif kind == "plan":
        T = _log_int(rng, 800, 5200)
        most = int(math.sqrt(2 * 2.4e11) / T)
        c.update(natoms=rng.randint(60, max(61, min(300, most))), nframes=T, k=rng.choice([10, 30, 50, 100]))
    elif kind == "long":
        c.update(natoms=rng.randint(4, 7), nframes=rng.randint(16400, 21000), k=rng.choice([10, 50, 100]))
    elif kind == "noalloc":
        c.update(natoms=_log_int(rng, 6, 64), nframes=rng.randint(150, 1024), k=rng.choice([5, 10, 20, 50]))
    elif kind == "batch":
        c.update(count=rng.randint(4, 32), natoms=rng.randint(24, 64), nframes=rng.randint(400, 900),
                 k=rng.choice([10, 50]))
    elif kind in ("gauss", "gcmi"):
        hi = 600 if kind == "gauss" else 300
        c.update(natoms=_log_int(rng, 20, hi), nframes=_log_int(rng, 300, 4000), k=0)
    elif kind == "te":
        c.update(natoms=_log_int(rng, 6, 60), nframes=rng.randint(200, 1200), k=rng.choice([5, 10, 20]),
                 lag=rng.choice([1, 5, 10]))
    elif kind == "teplan":
        T = _log_int(rng, 800, 4200)
        most = int(math.sqrt(2.3e11) / T)
        c.update(natoms=rng.randint(40, max(41, min(260, most))), nframes=T, k=rng.choice([10, 50, 100]),
                 lag=rng.choice([1, 5, 10]))
    else:
        c.update(natoms=rng.randint(60, 240), nframes=rng.randint(800, 2000), k=rng.choice([10, 50, 100]))
    return c


def _traj(case, seed):
    """Coordinates of one trajectory; the plan-sized ones are float32-rounded like stored MD positions."""
    n, T = case["natoms"], case["nframes"]
    if case["kind"] in ("ksg", "wrap", "te"):
        return synth_traj(n, T, 8, 0.05, seed=seed)
    return synth_traj(n, T, 16, 0.08, seed=seed, fp32=True)


def _batch(case, seed):
    """Uneven replicas: atoms and frames between half of the case's sizes and
    the sizes (the case's own, so a program that repeats the analysis on new
    data of the same set-up repeats its shapes)."""
    rng = np.random.Generator(np.random.Philox(case["count"] + 100 * case["natoms"] + 10000 * case["nframes"]))
    out = []
    for i in range(case["count"]):
        n = int(rng.integers(max(2, case["natoms"] // 2), case["natoms"] + 1))
        T = int(rng.integers(max(case["k"] + 1, case["nframes"] // 2), case["nframes"] + 1))
        out.append(synth_traj(n, T, 16, 0.08, seed=1000 * seed + i, fp32=True))
    return out


def _stream():
    global _STREAM
    if _STREAM is None:
        _STREAM = torch.cuda.Stream()
    return _STREAM


def prepare(case, seed):
    kind, k = case["kind"], case["k"]
    if kind == "batch":
        return {"kind": kind, "trajs": _batch(case, seed), "k": k}
    x = _traj(case, seed)
    n, T = x.shape[0], x.shape[1]
    s = {"kind": kind, "x": x, "k": k, "lag": case.get("lag", 0)}
    if kind == "wrap":
        s["X"], s["psi"], _ = gc.kraskov_prepare(x)
    elif kind in ("plan", "noalloc"):
        s["d_x"] = torch.from_numpy(x).cuda()
        s["d_out"] = torch.zeros(n * (n - 1) // 2, dtype=torch.float64, device="cuda")
        if kind == "plan":
            s["plan"] = gc.KsgPlan(n, T, k)
    elif kind == "teplan":
        s["d_x"] = torch.from_numpy(x).cuda()
        s["d_out"] = torch.zeros(n, n, dtype=torch.float64, device="cuda")
        s["plan"] = gc.TePlan(n, T, k, s["lag"])
    elif kind == "screened":
        global _SCREEN
        if _SCREEN is None:
            from gmx_correlation_b200.screen import TrainedScreen
            _SCREEN = TrainedScreen.load()
        s["model"] = _SCREEN.model
    return s


def run(s):
    kind = s["kind"]
    if kind in ("ksg", "long"):
        return gc.kraskov_corrmatrix(s["x"], s["k"])
    if kind == "wrap":
        return gc.kraskov_wrap(s["X"], s["psi"], 1, 0, s["k"])
    if kind in ("plan", "teplan"):
        s["plan"].run(s["d_x"].data_ptr(), s["d_out"].data_ptr(), _stream().cuda_stream)
        return s["d_out"]
    if kind == "noalloc":
        n, T = s["x"].shape[0], s["x"].shape[1]
        gc.ksg_pair_mi_noalloc(s["d_x"].data_ptr(), n, T, s["k"], s["d_out"].data_ptr(), _stream().cuda_stream)
        return s["d_out"]
    if kind == "batch":
        return gc.ksg_batch(s["trajs"], s["k"])
    if kind == "gauss":
        return gc.gauss_corrmatrix(s["x"])
    if kind == "gcmi":
        return gc.gcmi_corrmatrix(s["x"])
    if kind == "te":
        return gc.te_matrix(s["x"], s["k"], s["lag"])
    r, rep = gc.ksg_screened(s["x"], s["k"], s["model"], sigma_max=float("inf"), margin=0.0)
    return {"r": r, "flagged": int(rep["flagged"]), "audited": int(rep["audited"]), "exact": int(rep["exact"])}


def work(case):
    """Coordinates read and results written once.  KSG and TE need every
    atom's marginal distances (5 operations each) and at least k joint
    maxima per pair and query; the linear estimators 9 products and sums per
    frame of every atom pair."""
    n, T, k = case["natoms"], case["nframes"], case["k"]
    kind = case["kind"]
    if kind == "batch":  # mean atoms and frames of the uneven replicas
        n, T = int(0.75 * n), int(0.75 * T)
    pairs = n * (n - 1) // 2
    io = 24.0 * n * T
    if kind in ("gauss", "gcmi"):
        return {"bytes": io + 8.0 * n * n, "flops": 18.0 * pairs * T}
    if kind in ("te", "teplan"):
        return {"bytes": io + 8.0 * n * n, "flops": 11.0 * n * T * T + 2.0 * pairs * T * 2 * k}
    if kind == "screened":  # exact KSG on a twentieth of the pairs
        pairs = pairs // 20 + 1
    one = {"bytes": io + 8.0 * n * n, "flops": 5.0 * n * T * T + 1.0 * pairs * T * k}
    if kind == "batch":
        one = {q: v * case["count"] for q, v in one.items()}
    return one


def _digamma(n):
    psi = np.zeros(n + 2)
    psi[1] = -0.57721566490153
    for i in range(1, n + 1):
        psi[i + 1] = psi[i] + 1.0 / i
    return torch.from_numpy(psi).cuda()


def _maxdist(c, i0, i1):
    """Max-norm distances of queries i0 .. i1 - 1 to all frames; c: [..., T, 3]."""
    d = (c[..., i0:i1, None, 0] - c[..., None, :, 0]).abs()
    for a in (1, 2):
        d = torch.maximum(d, (c[..., i0:i1, None, a] - c[..., None, :, a]).abs())
    return d


def _ksg_exact(x, k):
    """Kraskov's second estimator over all pairs: [n, n] with diagonal 2000."""
    z = torch.from_numpy(x).cuda()
    z = (z - z.mean(1, keepdim=True)) / z.std(1, keepdim=True)
    n, T = z.shape[0], z.shape[1]
    psi = _digamma(T)
    a1, a2 = torch.tril_indices(n, n, -1, device="cuda")
    total = torch.zeros(len(a1), dtype=torch.float64, device="cuda")
    step = max(1, int(6e7 // (len(a1) * T)))
    chunk = max(1, int(6e7 // T))
    for i0 in range(0, T, step):
        i1 = min(T, i0 + step)
        D = _maxdist(z, i0, i1)  # [n, q, T]
        q = torch.arange(i1 - i0, device="cuda")
        D[:, q, i0 + q] = float("inf")
        for p0 in range(0, len(a1), chunk):
            p, r = a1[p0:p0 + chunk], a2[p0:p0 + chunk]
            near = torch.topk(torch.maximum(D[p], D[r]), k, dim=-1, largest=False).indices
            for m in (p, r):
                eps = torch.gather(D[m], -1, near).amax(-1, keepdim=True)
                total[p0:p0 + chunk] += psi[(D[m] <= eps).sum(-1)].sum(-1)
    mi = psi[T] + psi[k] - 1.0 / k - total / T
    out = torch.full((n, n), 2000.0, dtype=torch.float64, device="cuda")
    out[a1, a2] = mi
    out[a2, a1] = mi
    return out, mi


def _te_exact(x, k, lag):
    """TE(a2 -> a1) in row a1, column a2: strict counts of the subspaces within the k-th 9-D distance."""
    z = torch.from_numpy(x).cuda()
    n, T = z.shape[0], z.shape[1]
    Nv = T - lag
    past, fut = z[:, :Nv], z[:, lag:]
    psi = _digamma(Nv + 1)
    a1, a2 = (torch.ones(n, n, device="cuda") - torch.eye(n, device="cuda")).nonzero(as_tuple=True)
    total = torch.zeros(len(a1), dtype=torch.float64, device="cuda")
    step = max(1, int(6e7 // (len(a1) * Nv)))
    chunk = max(1, int(6e7 // Nv))
    for i0 in range(0, Nv, step):
        i1 = min(Nv, i0 + step)
        P = _maxdist(past, i0, i1)
        G = torch.maximum(P, _maxdist(fut, i0, i1))
        q = torch.arange(i1 - i0, device="cuda")
        P[:, q, i0 + q] = float("inf")
        G[:, q, i0 + q] = float("inf")
        for p0 in range(0, len(a1), chunk):
            p, r = a1[p0:p0 + chunk], a2[p0:p0 + chunk]
            eps = torch.topk(torch.maximum(G[p], P[r]), k, dim=-1, largest=False).values[..., -1:]
            term = psi[(P[p] < eps).sum(-1) + 1] - psi[(G[p] < eps).sum(-1) + 1]
            term -= psi[(torch.maximum(P[p], P[r]) < eps).sum(-1) + 1]
            total[p0:p0 + chunk] += (psi[k] + term).sum(-1)
    out = torch.zeros(n, n, dtype=torch.float64, device="cuda")
    out[a1, a2] = total / Nv
    return out


def _logdet_mi(v):
    """0.5 (log det C_a + log det C_b - log det C_ab) of the uncentred second moments; v: [n, T, 3]."""
    n, T = v.shape[0], v.shape[1]
    f = v.permute(1, 0, 2).reshape(T, 3 * n)
    C = (f.T @ f / T).reshape(n, 3, n, 3).permute(0, 2, 1, 3)
    a1, a2 = torch.tril_indices(n, n, -1, device="cuda")
    d = torch.arange(n, device="cuda")
    own = torch.logdet(C[d, d])
    J = torch.cat([torch.cat([C[a1, a1], C[a1, a2]], 2), torch.cat([C[a2, a1], C[a2, a2]], 2)], 1)
    mi = 0.5 * (own[a1] + own[a2] - torch.logdet(J))
    out = torch.full((n, n), 2000.0, dtype=torch.float64, device="cuda")
    out[a1, a2] = mi
    out[a2, a1] = mi
    return out


def _copula(x):
    """Normal scores of the midranks; frames of equal value share the mean score."""
    n, T = x.shape[0], x.shape[1]
    score = torch.special.ndtri((torch.arange(T, dtype=torch.float64, device="cuda") + 0.5) / T)
    v = torch.from_numpy(x).cuda().permute(0, 2, 1).reshape(3 * n, T)
    z = torch.empty_like(v)
    for c in range(3 * n):
        _, inv, cnt = torch.unique(v[c], return_inverse=True, return_counts=True)
        end = cnt.cumsum(0)
        cum = torch.cat([score.new_zeros(1), score.cumsum(0)])
        mean = torch.where(cnt == 1, score[end - 1], (cum[end] - cum[end - cnt]) / cnt)
        z[c] = mean[inv]
    return z.reshape(n, 3, T).permute(0, 2, 1)


def exact(case, seed):
    kind, k = case["kind"], case["k"]
    n, T = case["natoms"], case["nframes"]
    if kind == "screened":
        return None  # predictions of a trained network
    evals = n * (n - 1) // 2 * float(T) * T * case.get("count", 1) * (2 if kind in ("te", "teplan") else 1)
    if kind not in ("gauss", "gcmi") and evals > 1.3e10:
        return None  # over about 20 seconds in plain torch
    if kind == "batch":
        return [_ksg_exact(x, k)[0] for x in _batch(case, seed)]
    x = _traj(case, seed)
    if kind in ("ksg", "long"):
        return _ksg_exact(x, k)[0]
    if kind == "wrap":
        return float(_ksg_exact(x, k)[1][0])
    if kind in ("plan", "noalloc"):  # pairs in the order (1, 0), (2, 0), (2, 1), ...
        return _ksg_exact(x, k)[1]
    if kind in ("te", "teplan"):
        return _te_exact(x, k, case["lag"])
    v = torch.from_numpy(x).cuda() if kind == "gauss" else _copula(x)
    return _logdet_mi(v)
