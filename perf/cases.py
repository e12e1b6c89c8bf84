"""The joins that a user of this library runs, for measuring it.

Every case is one epsilon self-join through a public entry point:

    device   gsj_join on points in device memory, numNeighbors and neighborTable
             copied into the caller's device buffers (gsj_result_counts,
             gsj_result_table): the join inside a GPU program, through the C ABI
    host     SelfJoin.run_host between pinned host buffers: the batched pipeline
    gdsjoin  GDSJoinPy_f32 and copyResultIntoPythonArray64 on host arrays: the
             two calls of the reference's Python users

The caller's buffers have room for more than the expected number of pairs, and
every output is a whole buffer (zeros behind the last pair).

The point distributions are those of gpu_self_join_b200/synth.py, generated on
the GPU: the distribution's parameters (centres, scales, factors) are fixed, the
points come from the seed.  eps is chosen for a mean number of neighbours: the
mean is 1 + (N - 1) p(eps) with p the probability that two points of the
distribution lie within eps, and PAIR_EPS holds eps at fixed p for each
distribution (measured on 2,048 x 400,000 sampled pairs).
"""

import ctypes
import functools
import math

import numpy as np
import torch

from gpu_self_join_b200 import JoinConfig, SelfJoin, _native

# log10 p -> eps, p the probability that a pair of points lies within eps
PAIR_P = (-6.0, -5.5, -5.0, -4.5, -4.0, -3.5, -3.0, -2.5, -2.0)
PAIR_EPS = {
    "gmm2d": (0.2009, 0.3597, 0.6368, 1.132, 2.023, 3.622, 6.561, 12.3, 25.29),
    "gmm6d": (1.352, 1.656, 2.028, 2.495, 3.112, 3.926, 5.058, 6.761, 9.705),
    "derived18d": (0.3162, 0.3681, 0.4325, 0.5117, 0.6138, 0.7516, 0.9462, 1.259, 1.82),
    "heavy8": (1.309, 1.521, 1.77, 2.065, 2.404, 2.812, 3.311, 3.926, 4.699),
    "heavy16": (5.408, 5.943, 6.516, 7.194, 7.98, 8.892, 9.977, 11.3, 12.91),
    "heavy32": (6.653, 7.145, 7.674, 8.279, 8.995, 9.84, 10.81, 12.02, 13.55),
    "heavy90": (11.09, 11.75, 12.5, 13.34, 14.29, 15.38, 16.71, 18.28, 20.23),
}
UNIFORM_SIDE = 100.0


def eps_for(dist, n, N, mean):
    """eps for `mean` neighbours a point (itself included) among N points."""
    p = max(mean - 1.0, 0.5) / (N - 1)
    if dist == "uniform":
        ball = math.pi ** (n / 2) / math.gamma(n / 2 + 1)
        return UNIFORM_SIDE * (p / ball) ** (1.0 / n)
    y = np.log10(np.array(PAIR_EPS[dist if dist != "heavy" else "heavy%d" % n]))
    x = np.array(PAIR_P)
    t = math.log10(p)
    # log-log interpolation, the end segments continued
    i = int(np.clip(np.searchsorted(x, t) - 1, 0, x.size - 2))
    return float(10.0 ** (y[i] + (y[i + 1] - y[i]) * (t - x[i]) / (x[i + 1] - x[i])))


# ------------------------------------------------------------------ points
@functools.lru_cache(maxsize=None)
def parameters(dist, n):
    """The distribution's fixed parameters, as gpu_self_join_b200/synth.py draws them."""
    rng = np.random.default_rng(20261203 + {"gmm2d": 1, "gmm6d": 2, "derived18d": 3}.get(dist, 4 + n))
    if dist == "gmm2d":
        K = 64
        return {"centres": rng.uniform(0.0, 1000.0, (K, 2)), "sigma": np.repeat(rng.uniform(5.0, 40.0, (K, 1)), 2, 1),
                "w": rng.dirichlet(np.ones(K))}
    if dist == "gmm6d":
        K = 32
        return {"centres": rng.uniform(0.0, 100.0, (K, 6)), "sigma": rng.uniform(1.0, 6.0, (K, 6)),
                "w": np.full(K, 1.0 / K)}
    if dist == "derived18d":
        K = 16
        return {"centres": rng.uniform(-4.0, 4.0, (K, 8)), "sigma": np.exp(rng.standard_normal((K, 8))),
                "w": np.full(K, 1.0 / K)}
    if dist == "heavy":
        ng = min(12, n)
        m = n - ng
        return {"sigma": np.sqrt(np.exp(rng.uniform(math.log(1.0), math.log(100.0), ng))),
                "F": rng.standard_normal((m, min(8, m))) * 0.6, "diag": np.sqrt(rng.uniform(0.3, 1.0, m))}
    return {}


def points(dist, n, N, dtype, seed, device):
    """N x n points of the distribution."""
    g = torch.Generator(device=device).manual_seed(seed)
    P = {k: torch.tensor(v, dtype=torch.float32, device=device) for k, v in parameters(dist, n).items()}

    def normal(*shape):
        return torch.randn(*shape, generator=g, device=device)

    def uniform(*shape):
        return torch.rand(*shape, generator=g, device=device)

    def mixture(count):
        edges = torch.cumsum(P["w"], 0)
        comp = torch.searchsorted(edges, uniform(count) * edges[-1]).clamp_(max=edges.numel() - 1)
        return P["centres"][comp] + normal(count, P["centres"].shape[1]) * P["sigma"][comp]

    if dist == "uniform":
        x = uniform(N, n) * UNIFORM_SIDE
    elif dist == "gmm2d":  # a tenth of the points is uniform background
        x = mixture(N)
        back = uniform(N) < 0.1
        x = torch.where(back[:, None], uniform(N, 2) * 1000.0, x)
    elif dist == "gmm6d":
        x = mixture(N)
    elif dist == "derived18d":
        b = mixture(N)
        d = [b[:, 0] * b[:, 1], b[:, 2] * b[:, 3], b[:, 4] / (1 + b[:, 5].abs()), b[:, 6] / (1 + b[:, 7].abs()),
             (b[:, 0] ** 2 + b[:, 2] ** 2).sqrt(), (b[:, 1] ** 2 + b[:, 3] ** 2 + b[:, 5] ** 2).sqrt(),
             (b[:, 4:8] ** 2).sum(1).sqrt(), b[:, 0] * b[:, 7], b[:, 2].tanh() * b[:, 6], b[:, 1] / (1 + b[:, 3] ** 2)]
        d = torch.stack(d, 1)
        x = torch.cat([b, d + 0.05 * normal(N, 10)], 1)
        x = (x - x.mean(0)) / x.std(0)
    elif dist == "heavy":  # Gaussian dims, then multivariate Student-t (nu = 3) with a factor correlation
        x = normal(N, min(12, n)) * P["sigma"]
        m = n - x.shape[1]
        if m:
            z = normal(N, P["F"].shape[1]) @ P["F"].T + normal(N, m) * P["diag"]
            chi = (normal(N, 3) ** 2).sum(1, keepdim=True)
            x = torch.cat([x, z / (chi / 3.0).sqrt()], 1)
    else:
        raise ValueError(dist)
    return x.to(torch.float64 if dtype == "float64" else torch.float32).contiguous()


# ------------------------------------------------------------------ cases
# The switches each kind of data is joined with (synth.WORKLOADS): the unicomp
# traversal on low-dimensional data, REORDER + ILP 8 + SHORTCIRCUIT +
# QUERYREORDER on high-dimensional data.
SWITCHES = ("stamp", "reorder", "ilp", "shortcircuit", "query_reorder")
LOW = {"stamp": True, "reorder": False, "ilp": 0, "shortcircuit": False, "query_reorder": False}
HIGH = {"stamp": False, "reorder": True, "ilp": 8, "shortcircuit": True, "query_reorder": True}


def make(dist, n, N, mean, k=None, dtype="float32", via="device"):
    c = {"dist": dist, "n": n, "N": N, "mean": mean, "k": min(n, 6) if k is None else k, "dtype": dtype, "via": via}
    c.update(HIGH if dist in ("derived18d", "heavy") else LOW)
    c["eps"] = eps_for(dist, n, N, mean)
    return c


def listed():
    return [
        # the smallest join: a program that joins a few thousand points, where launches and host round trips count
        dict(make("uniform", 2, 2_003, 32.0), name="uniform2d_2k"),
        # the reference's own example size and shape (100,000 x 2, test_dat.txt) through its Python call, host to host
        dict(make("uniform", 2, 100_000, 32.4, via="gdsjoin"), name="gdsjoin2d_100k"),
        # double precision data in 3-D (DTYPE double), an odd size
        dict(make("uniform", 3, 250_007, 32.0, dtype="float64"), name="uniform3d_f64_250k"),
        # clustered 2-D data whose lists go to pinned host buffers in batches while they are produced
        dict(make("gmm2d", 2, 2_000_000, 32.0, via="host"), name="gmm2d_host_2M"),
        # the 2-D headline workload: 20M points, mean 32 neighbours
        dict(make("gmm2d", 2, 20_000_000, 32.0), name="gmm2d_20M"),
        # a small six-dimensional join: every dimension indexed, few points a cell
        dict(make("gmm6d", 6, 30_011, 24.0), name="gmm6d_30k"),
        # the 6-D workload: 5M points, mean 64 neighbours
        dict(make("gmm6d", 6, 5_000_000, 64.0), name="gmm6d_5M"),
        # requests of the request stream (N log-uniform in [10k, 500k], n of 8, 16, 32, 90, mean 10 to 100)
        dict(make("heavy", 8, 142_016, 17.0), name="heavy8d_142k"),
        dict(make("heavy", 32, 45_047, 91.0), name="heavy32d_45k"),
        # fewer indexed dimensions than data dimensions (NUMINDEXEDDIM 3 of 8): populated cells, no tensor-core screen
        dict(make("heavy", 8, 120_011, 50.0, k=3), name="heavy8d_k3_120k"),
        # the 90-D workload: 515,345 points, mean 50 neighbours
        dict(make("heavy", 90, 515_345, 50.0), name="heavy90d_515k"),
        # the 18-D workload: 5M points, mean 100 neighbours
        dict(make("derived18d", 18, 5_000_000, 100.0), name="derived18d_5M"),
    ]


def draw(rng):
    def size(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind = rng.choice(["uniform", "gmm2d", "gmm2d", "gmm6d", "gmm6d", "derived18d", "heavy", "heavy", "heavy", "host", "gdsjoin"])
    if kind == "uniform":
        n = rng.choice([2, 3])
        return make("uniform", n, size(2_000, 2_000_000), rng.uniform(8.0, 64.0), dtype=rng.choice(["float32", "float64"]))
    if kind == "gmm2d":
        return make("gmm2d", 2, size(50_000, 16_000_000), rng.uniform(8.0, 48.0))
    if kind == "gmm6d":
        return make("gmm6d", 6, size(20_000, 4_000_000), rng.uniform(8.0, 64.0), dtype="float32")
    if kind == "derived18d":
        return make("derived18d", 18, size(30_000, 3_000_000), rng.uniform(10.0, 100.0))
    if kind == "heavy":
        n = rng.choice([8, 16, 32, 90])
        return make("heavy", n, size(10_000, 300_000 if n == 8 else 500_000), rng.uniform(10.0, 100.0), k=rng.choice([3, 6, 6, 6]))
    if kind == "host":
        return make("gmm2d", 2, size(100_000, 3_000_000), rng.uniform(8.0, 48.0), via="host")
    return make("uniform", 2, size(10_000, 200_000), rng.uniform(8.0, 48.0), via="gdsjoin")


@functools.lru_cache(maxsize=None)
def session(via):
    """The program's one join handle: made once, it joins whatever comes."""
    if via == "host":
        return SelfJoin(0)
    handle = ctypes.c_void_p()
    _native.check(_native.lib().gsj_create(ctypes.byref(handle), 0))
    return handle


def prepare(case, seed):
    x = points(case["dist"], case["n"], case["N"], case["dtype"], seed, "cuda")
    N, n, via = case["N"], case["n"], case["via"]
    room = int(1.5 * N * case["mean"])  # entries of the caller's neighborTable
    state = {"via": via, "eps": case["eps"], "N": N, "n": n, "room": room}
    if via == "gdsjoin":
        state["points"] = x.cpu().numpy().reshape(-1)
        state["counts"], state["table"] = np.zeros(N, np.uint32), np.zeros(room, np.uint32)
        return state
    state["join"] = session(via)
    if via == "host":
        p, c, t = (torch.zeros(m, dtype=d, pin_memory=True)
                   for m, d in ((N * n, x.dtype), (N, torch.int32), (room, torch.int32)))
        p.copy_(x.reshape(-1))
        state["points"] = p.numpy().reshape(N, n)
        state["counts"], state["table"] = c.numpy().view(np.uint32), t.numpy().view(np.uint32)
        state["config"] = JoinConfig(**{f: case[f] for f in SWITCHES}, indexed_dims=case["k"])
        return state
    config = _native.default_config()
    config.dim, config.indexed_dims = n, case["k"]
    config.dtype = _native.GSJ_FLOAT64 if case["dtype"] == "float64" else _native.GSJ_FLOAT32
    for f in SWITCHES:
        setattr(config, f, int(case[f]))
    state["points"], state["config"] = x, config
    state["counts"] = torch.zeros(N, dtype=torch.int32, device="cuda")
    state["table"] = torch.zeros(room, dtype=torch.int32, device="cuda")
    return state


def run(state):
    L, check = _native.lib(), _native.check
    counts, table = state["counts"], state["table"]
    if state["via"] == "gdsjoin":
        check(L.GDSJoinPy_f32(state["points"].ctypes.data, state["N"], state["eps"], state["n"], 0, counts.ctypes.data))
        check(L.copyResultIntoPythonArray64(table.ctypes.data, int(counts.sum(dtype=np.uint64))))
    elif state["via"] == "host":
        state["join"].run_host(state["points"], state["eps"], state["config"], counts=counts, table=table)
    else:
        join = state["join"]
        check(L.gsj_join(join, state["points"].data_ptr(), state["N"], state["eps"], ctypes.byref(state["config"]), 1,
                         None), join)
        check(L.gsj_result_counts(join, counts.data_ptr(), 1), join)
        check(L.gsj_result_table(join, table.data_ptr(), state["room"], 1), join)
    return counts, table


def work(case):
    """The points read once, counts and lists written once; the
    distance of every reported pair (a subtraction and a fused multiply-add a
    dimension)."""
    size = 8 if case["dtype"] == "float64" else 4
    N, n, pairs = case["N"], case["n"], case["N"] * case["mean"]
    return {"bytes": N * n * size + 4 * N + 4 * pairs, "flops": 3 * n * pairs}
