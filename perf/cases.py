"""Cases by which the speed of the self-join framework is judged.

Each case is one call a user's program makes through the public entry points
(the package's functions over the C ABI of include/knnsj.h): joins of points
that are resident on the device, a join of host arrays, a batch of uneven
joins, outlier scores of a result table, and a training step of the learned
starting radius.  Sizes come from the benchmark configurations (datasets.py,
bench.py), from the tests, or are generic; the values follow the same
distributions as datasets.py, drawn on the device where the data live there.
"""
from __future__ import annotations

import ctypes
import math

import numpy as np
import torch

import hybrid_k_nearest_neighbor_self_join_gb300 as kj
from hybrid_k_nearest_neighbor_self_join_gb300 import _lib, datasets

LEARNED = kj.RADIUS_LEARNED
PLAIN = kj.RADIUS_PLAIN


def listed() -> list[dict]:
    return [
        # the smallest set of the batched configuration joined by itself:
        # launches, synchronisations and host work are all there is
        dict(name="join2d_2k", kind="join", dist="gmm", n=2_000, d=2, k=8, di=2, beta=0.05, dtype="float32",
             mode="plain", comps=8, ufrac=0.2),
        # the small benchmark configuration: uniform points, BETA = 0
        dict(name="uniform2d_100k", kind="join", dist="uniform", n=100_000, d=2, k=8, di=2, beta=0.0,
             dtype="float32", mode="plain"),
        # the headline workload: a sky catalogue's positions, learned radii
        dict(name="sky2d_25m", kind="join", dist="sky", n=25_000_000, d=2, k=64, di=2, beta=0.025, dtype="float32",
             mode="learned"),
        # a catalogue of ordinary, odd size under the reference's own BETA
        # schedule (what the drop-in wrapper runs)
        dict(name="sky2d_3m_plain", kind="join", dist="sky", n=3_000_017, d=2, k=64, di=2, beta=0.025,
             dtype="float32", mode="plain"),
        # an ordinary three-dimensional point cloud of odd size, defaults
        dict(name="cloud3d_1m", kind="join", dist="gmm", n=1_000_003, d=3, k=32, di=3, beta=0.05, dtype="float32",
             mode="plain", comps=20, ufrac=0.2),
        # the four-dimensional configuration with long rows
        dict(name="gmm4d_5m", kind="join", dist="gmm", n=5_000_000, d=4, k=128, di=4, beta=0.05, dtype="float32",
             mode="learned", comps=50, ufrac=0.2),
        # the double-precision configuration: the largest call
        dict(name="gmm6d_10m_f64", kind="join", dist="gmm", n=10_000_000, d=6, k=16, di=6, beta=0.05,
             dtype="float64", mode="learned", comps=100, ufrac=0.1),
        # feature vectors with more dimensions than the grid indexes, of a
        # size that is a multiple of nothing
        dict(name="wide12d_60k", kind="join", dist="gmm", n=60_013, d=12, k=15, di=6, beta=0.05, dtype="float32",
             mode="plain", comps=20, ufrac=0.05),
        # the call with NumPy arrays in and out, as the wrapper makes it
        dict(name="host2d_500k", kind="host", dist="sky", n=500_009, d=2, k=16, di=2, beta=0.05, dtype="float32",
             mode="learned"),
        # a sample of the batched configuration: independent uneven sets
        dict(name="batched_30", kind="batched", sets=30, shapes=4, n_lo=2_000, n_hi=500_000, beta=0.05,
             dtype="float32", mode="learned"),
        # outlier scores of a device-resident result table
        dict(name="outlier_2m", kind="outlier", dist="sky", n=2_000_003, d=2, k=16, dtype="float32"),
        # one step of training the learned radius: loss and gradient of the
        # network on features and exact k-th distances
        dict(name="radius_grad_200k", kind="grad", n=200_003, quantile=0.9),
    ]


# the largest drawn size per dimension count: more dimensions search wider
# rings per query
_DRAW_N = {2: 8_000_000, 3: 3_000_000, 4: 1_000_000, 5: 500_000, 6: 300_000, 8: 100_000, 12: 50_000}


def _log_uniform(rng, lo: float, hi: float) -> int:
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng) -> dict:
    kind = rng.choices(["join", "host", "batched", "outlier", "grad"], [14, 2, 2, 1, 1])[0]
    if kind == "grad":
        return dict(kind=kind, n=_log_uniform(rng, 1_000, 500_000), quantile=round(rng.uniform(0.5, 0.95), 3))
    if kind == "batched":
        return dict(kind=kind, sets=rng.randint(2, 30), shapes=rng.randrange(1 << 20), n_lo=2_000,
                    n_hi=_log_uniform(rng, 5_000, 300_000), beta=0.05, dtype=rng.choice(["float32", "float32", "float64"]), mode=rng.choice(["plain", "learned"]))
    if kind == "outlier":
        return dict(kind=kind, dist="sky", n=_log_uniform(rng, 5_000, 4_000_000), d=2,
                    k=_log_uniform(rng, 4, 64), dtype=rng.choice(["float32", "float64"]))
    d = rng.choice([2, 2, 2, 3, 3, 4, 4, 5, 6, 8, 12])
    dtype = rng.choice(["float32", "float32", "float64"])
    k = _log_uniform(rng, 4, 128)
    hi = _DRAW_N[d] // (2 if dtype == "float64" else 1) // (2 if kind == "host" else 1)
    n = max(_log_uniform(rng, 2_000, hi), 2 * (k + 1))
    dist = rng.choice(["sky", "sky", "uniform", "gmm"]) if d == 2 else rng.choice(["gmm", "gmm", "uniform"])
    if d > 6:
        dist = "gmm"
    di = min(d, 6) if rng.random() < 0.8 else rng.randint(2, min(d, 6))
    if d <= 3:
        di = d
    di = max(di, min(d, 4))
    return dict(kind=kind, dist=dist, n=n, d=d, k=k, di=di, beta=rng.choice([0.0, 0.025, 0.05]), dtype=dtype,
                mode=rng.choice(["plain", "learned"]), comps=rng.randint(1, 60),
                ufrac=round(rng.uniform(0.05, 0.3), 3))


# ---- inputs ----------------------------------------------------------------

def _sky_base(g, m: int) -> torch.Tensor:
    dev = g.device
    x = torch.rand(m, generator=g, device=dev, dtype=torch.float64) * 360.0
    band = torch.rand(m, generator=g, device=dev) < 0.7
    y = torch.where(band, (torch.randn(m, generator=g, device=dev, dtype=torch.float64) * 8.0).clamp_(-90.0, 90.0),
                    torch.rand(m, generator=g, device=dev, dtype=torch.float64) * 180.0 - 90.0)
    return torch.stack([x, y], 1)


def _sky(g, n: int) -> torch.Tensor:
    """Equatorial band plus background plus 200 dense clumps, rows shuffled."""
    per = int(round(n * 0.001))
    m = 200 * per
    base = _sky_base(g, n - m)
    centres = _sky_base(g, 200)
    clumps = centres.repeat_interleave(per, 0)
    clumps = clumps + 0.2 * torch.randn(m, 2, generator=g, device=g.device, dtype=torch.float64)
    clumps[:, 1].clamp_(-90.0, 90.0)
    return torch.cat([base, clumps])[torch.randperm(n, generator=g, device=g.device)]


def _gmm(g, n: int, d: int, comps: int, ufrac: float) -> torch.Tensor:
    """Anisotropic Gaussians (axis sd log-uniform in [0.005, 0.1]) plus a
    uniform background, rows shuffled."""
    dev = g.device
    n_g = n - int(round(n * ufrac))
    centres = torch.rand(comps, d, generator=g, device=dev, dtype=torch.float64)
    span = math.log(0.1) - math.log(0.005)
    sds = torch.exp(math.log(0.005) + span * torch.rand(comps, d, generator=g, device=dev, dtype=torch.float64))
    lab = torch.randint(0, comps, (n_g,), generator=g, device=dev)
    pts = torch.rand(n, d, generator=g, device=dev, dtype=torch.float64)
    pts[:n_g] = centres[lab] + sds[lab] * torch.randn(n_g, d, generator=g, device=dev, dtype=torch.float64)
    return pts[torch.randperm(n, generator=g, device=dev)]


def _points(case: dict, seed: int) -> torch.Tensor:
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    n, d = case["n"], case["d"]
    if case["dist"] == "sky":
        x = _sky(g, n)
    elif case["dist"] == "gmm":
        x = _gmm(g, n, d, case["comps"], case["ufrac"])
    else:
        x = torch.rand(n, d, generator=g, device="cuda", dtype=torch.float64)
    return x.to(getattr(torch, case["dtype"])).contiguous()


def _batch_shapes(case: dict) -> list[tuple]:
    """(n, d, components, uniform share, k) of each set, as
    datasets.batched_sets draws them; the case fixes them."""
    rng = np.random.default_rng(case["shapes"])
    m = case["sets"]
    sizes = np.exp(rng.uniform(np.log(case["n_lo"]), np.log(case["n_hi"]), m)).astype(np.int64)
    return list(zip(sizes.tolist(), rng.choice([2, 3, 4, 6, 8], m).tolist(), rng.integers(1, 21, m).tolist(),
                    rng.uniform(0.05, 0.30, m).tolist(), rng.choice([8, 32], m).tolist()))


def _batch(case: dict, seed: int):
    shapes = _batch_shapes(case)
    xs = [datasets.gmm(n, d, comps, ufrac, seed * 1000 + i, dtype=np.dtype(case["dtype"]))
          for i, (n, d, comps, ufrac, _) in enumerate(shapes)]
    return xs, [s[4] for s in shapes]


def _grad_inputs(case: dict, seed: int):
    """A trained model, and samples as training sees them: features of the
    model's own input distribution, targets around its output."""
    rng = np.random.default_rng(seed)
    model = kj.get_radius_model()
    n = case["n"]
    mean, istd = model[:24], model[24:48]
    std = np.where(istd > 0, 1.0 / np.where(istd > 0, istd, 1.0), 0.0)
    feats = (mean + std * rng.standard_normal((n, 24))).astype(np.float32)
    targets = rng.normal(0.2, 0.5, n).astype(np.float32)
    return model, feats, targets


def _mode(case: dict) -> int:
    return LEARNED if case["mode"] == "learned" else PLAIN


def prepare(case: dict, seed: int) -> dict:
    kind = case["kind"]
    if kind == "grad":
        model, feats, targets = _grad_inputs(case, seed)
        return dict(case=case, model=model, feats=feats, targets=targets)
    if kind == "batched":
        xs, ks = _batch(case, seed)
        return dict(case=case, xs=xs, ks=ks)
    x = _points(case, seed)
    n, K = case["n"], case["k"] + 1
    if kind == "host":
        return dict(case=case, x=x.cpu().numpy())
    ids = torch.empty(n, K, dtype=torch.int32, device="cuda")
    dists = torch.empty(n, K, dtype=x.dtype, device="cuda")
    state = dict(case=case, x=x, ids=ids, dists=dists)
    torch.cuda.synchronize()  # the join runs on the library's own stream
    if kind == "outlier":
        kj.selfjoin_device(x.data_ptr(), np.dtype(case["dtype"]), n, case["d"], case["k"], ids.data_ptr(),
                           dists.data_ptr(), radius_mode=LEARNED)
        state.update(mean=torch.empty(n, dtype=torch.float64, device="cuda"),
                     dist_rank=torch.empty(n, dtype=torch.int32, device="cuda"),
                     in_degree=torch.empty(n, dtype=torch.int64, device="cuda"),
                     degree_rank=torch.empty(n, dtype=torch.int32, device="cuda"))
    torch.cuda.synchronize()
    return state


# ---- one pass --------------------------------------------------------------

def run(state: dict):
    case = state["case"]
    kind = case["kind"]
    if kind == "join":
        kj.selfjoin_device(state["x"].data_ptr(), np.dtype(case["dtype"]), case["n"], case["d"], case["k"],
                           state["ids"].data_ptr(), state["dists"].data_ptr(), num_indexed_dims=case["di"],
                           beta=case["beta"], radius_mode=_mode(case))
        return dict(ids=state["ids"], dists=state["dists"])
    if kind == "host":
        ids, dists = kj.selfjoin(state["x"], case["k"], num_indexed_dims=case["di"], beta=case["beta"],
                                 radius_mode=_mode(case))
        return dict(ids=ids, dists=dists)
    if kind == "batched":
        out = kj.selfjoin_batched(state["xs"], state["ks"], beta=case["beta"], radius_mode=_mode(case))
        return [a for pair in out for a in pair]
    if kind == "outlier":
        kj.outlier_scores_device(state["ids"].data_ptr(), state["dists"].data_ptr(), np.dtype(case["dtype"]),
                                 case["n"], case["k"] + 1, state["mean"].data_ptr(), state["dist_rank"].data_ptr(),
                                 state["in_degree"].data_ptr(), state["degree_rank"].data_ptr())
        return {key: state[key] for key in ("mean", "dist_rank", "in_degree", "degree_rank")}
    model, feats, targets = state["model"], state["feats"], state["targets"]
    grad = np.empty(_lib.RADIUS_MODEL_FLOATS - 48, np.float32)
    loss = ctypes.c_double(0.0)
    _lib.check(_lib.load().knnsj_radius_grad(model.ctypes.data, feats.ctypes.data, targets.ctypes.data, case["n"],
                                             case["quantile"], grad.ctypes.data, ctypes.byref(loss)),
               "knnsj_radius_grad")
    return dict(grad=grad, loss=loss.value)


# ---- what a pass cannot do without ----------------------------------------

def _join_work(n: int, d: int, k: int, s: int) -> tuple[float, float]:
    # the points in, the rows out; one distance per returned neighbour
    return n * d * s + n * (k + 1) * (4.0 + s), n * (k + 1) * 3.0 * d


def work(case: dict) -> dict:
    kind = case["kind"]
    s = 8 if case.get("dtype") == "float64" else 4
    if kind in ("join", "host"):
        b, f = _join_work(case["n"], case["d"], case["k"], s)
    elif kind == "batched":
        pairs = [_join_work(n, d, k, s) for n, d, _, _, k in _batch_shapes(case)]
        b, f = sum(p[0] for p in pairs), sum(p[1] for p in pairs)
    elif kind == "outlier":
        n, K = case["n"], case["k"] + 1
        b, f = n * K * (4.0 + s) + n * (8 + 4 + 8 + 4), n * K
    else:  # forward, and twice that backward
        macs = 24 * 64 + 64 * 64 + 64
        b, f = case["n"] * 25 * 4.0 + 2 * _lib.RADIUS_MODEL_FLOATS * 4, case["n"] * macs * 2.0 * 3
    return {"bytes": float(b), "flops": float(f)}


# ---- 64-bit values ---------------------------------------------------------

_EXACT_MAX_N = 130_000


def _exact_rows(x: torch.Tensor, K: int) -> torch.Tensor:
    """Distances of the K nearest points of every point, in 64 bits."""
    p = x.double()
    n, d = p.shape
    out = torch.empty(n, K, dtype=torch.float64, device=p.device)
    step = max(1, 100_000_000 // n)
    for i in range(0, n, step):
        q = p[i:i + step]
        acc = torch.zeros(q.shape[0], n, dtype=torch.float64, device=p.device)
        for j in range(d):
            t = q[:, j, None] - p[None, :, j]
            acc.addcmul_(t, t)
        out[i:i + step] = acc.topk(K, 1, largest=False, sorted=True).values.sqrt_()
    return out


def _exact_grad(case: dict, seed: int):
    model, feats, targets = _grad_inputs(case, seed)
    m = torch.from_numpy(model).cuda().double()
    sizes = [24, 24, 24 * 64, 64, 64 * 64, 64, 64, 1]
    mean, istd, w1, b1, w2, b2, w3, b3 = torch.split(m, sizes)
    params = [w1.reshape(24, 64), b1, w2.reshape(64, 64), b2, w3, b3]
    params = [p.clone().requires_grad_(True) for p in params]
    x = (torch.from_numpy(feats).cuda().double() - mean) * istd
    h = torch.relu(torch.relu(x @ params[0] + params[1]) @ params[2] + params[3])
    e = torch.from_numpy(targets).cuda().double() - (h @ params[4] + params[5])
    q = case["quantile"]
    loss = torch.where(e > 0, q * e, (q - 1.0) * e).mean()
    grads = torch.autograd.grad(loss, params)
    return dict(grad=torch.cat([g.reshape(-1) for g in grads]).cpu().numpy(), loss=float(loss))


def exact(case: dict, seed: int):
    kind = case["kind"]
    if kind == "grad":
        return _exact_grad(case, seed)
    if kind == "batched":
        out = []
        xs, ks = _batch(case, seed)
        if sum(float(x.shape[0]) ** 2 for x in xs if x.shape[0] <= _EXACT_MAX_N) > 4e10:
            return None
        for x, k in zip(xs, ks):
            small = x.shape[0] <= _EXACT_MAX_N
            out += [None, _exact_rows(torch.from_numpy(x).cuda(), k + 1).cpu().numpy() if small else None]
        return out
    if kind == "outlier":
        state = prepare(case, seed)
        return dict(mean=state["dists"].double().sum(1) / case["k"], dist_rank=None, in_degree=None,
                    degree_rank=None)
    if case["n"] > _EXACT_MAX_N:
        return None
    dists = _exact_rows(_points(case, seed), case["k"] + 1)
    return dict(ids=None, dists=dists.cpu().numpy() if kind == "host" else dists)
