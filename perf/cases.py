"""What the engine's speed is measured on: the work a user has it do, through its public entry points.

A case is a plain dict.  Its kinds:

* count: one count of a pattern in a resident graph (`Executor.count`), the engine's main call; exact or
  reference-compatible mode, default configuration unless `tile` says otherwise.
* batch: many (pattern, graph) jobs in one prepared launch (`Batch.run` + `Batch.counts`).
* ingest: a graph from host CSR arrays (`Graph.from_csr(device=True)` + `upload`), then the 4-clique and 4-cycle.
* train, gradient, predict: the learned cost model's network (`costmodel.MLP`) in training, its gradient, and ranking.

Graphs are the repository's own generators: R-MAT (a, b, c = .57, .19, .19), Erdos-Renyi and Barabasi-Albert.
"""
from __future__ import annotations

import math

import numpy as np
import torch

import graphautotune_b200 as g
from graphautotune_b200 import costmodel

WEDGE, TRIANGLE = "001001110", "011101110"
K4, C4 = "0111101111011110", "0101101001011010"
STAR4, PATH4, PAW, DIAMOND = ("0001000100011110", "0001001001011010", "0001001101011110",
                              "0011001111011110")
HOUSE = "0100110110010110110010100"
CYCLE5 = "0001100101010101010011000"
K5 = "0111110111110111110111110"


def _adj(n: int, edges: list[tuple[int, int]]) -> str:
    s = ["0"] * (n * n)
    for u, v in edges:
        s[u * n + v] = s[v * n + u] = "1"
    return "".join(s)


K6 = _adj(6, [(i, j) for i in range(6) for j in range(i)])
K7 = _adj(7, [(i, j) for i in range(7) for j in range(i)])
CYCLE6_CHORD = _adj(6, [(0, 1), (1, 2), (2, 3), (3, 4), (4, 5), (5, 0), (0, 3)])
FIVE = [p for p in g.enumerate_patterns(5) if p != K5]  # 20 plan-interpreted patterns


def listed() -> list[dict]:
    return [
        # the smallest benchmark configuration: a triangle count on a sparse uniform graph; latency counts
        dict(name="triangle_er10k", kind="count", mode="exact", pattern=TRIANGLE, tile=32,
             graph="er", n=10000, degree=16.0),
        # the headline configuration's two counts: power-law graph of 2^20 vertices, 16M edges
        dict(name="k4_rmat20", kind="count", mode="exact", pattern=K4, tile=32,
             graph="rmat", scale=20, samples=1 << 24),
        dict(name="c4_rmat20", kind="count", mode="exact", pattern=C4, tile=32,
             graph="rmat", scale=20, samples=1 << 24),
        # a larger clique on a denser power-law graph (average degree about 32)
        dict(name="k5_rmat18", kind="count", mode="exact", pattern=K5, tile=32,
             graph="rmat", scale=18, samples=(1 << 22) - 5),
        # the 6-cycle with a chord: six vertices, the deepest nest that is enumerated here
        dict(name="cycle6chord_rmat10", kind="count", mode="exact", pattern=CYCLE6_CHORD, tile=32,
             graph="rmat", scale=10, samples=1 << 13),
        # the five-vertex house, exact and by the reference's own rules
        dict(name="house_rmat14", kind="count", mode="exact", pattern=HOUSE, tile=32,
             graph="rmat", scale=14, samples=1 << 17),
        dict(name="house_ref_rmat12", kind="count", mode="ref", pattern=HOUSE, tile=32,
             graph="rmat", scale=12, samples=1 << 15),
        # a 5-cycle on a preferential-attachment graph of odd size
        dict(name="cycle5_ba20011", kind="count", mode="exact", pattern=CYCLE5, tile=32,
             graph="ba", n=20011, m=9),
        # all 20 plan-interpreted five-vertex patterns over uneven graphs in one launch
        dict(name="batch20x6", kind="batch", graphs=6, max_log2=12),
        # from host arrays to two counts: what a user with a new graph waits for
        dict(name="ingest_rmat18", kind="ingest", graph="rmat", scale=18, samples=1 << 22),
        # the cost model: training on collected timings, and ranking a set of candidates
        dict(name="mlp_train_4k", kind="train", rows=4001, features=38, epochs=10, batch=256),
        dict(name="mlp_predict_64", kind="predict", rows=64, features=38),
    ]


def _log_uniform(rng, lo: float, hi: float) -> int:
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _draw_graph(rng, max_scale: int) -> dict:
    """A graph of up to 2^max_scale vertices, average degree about 16."""
    kind = rng.choice(["rmat", "rmat", "er", "ba"])
    if kind == "rmat":
        scale = rng.randint(10, max_scale)
        return dict(graph="rmat", scale=scale, samples=_log_uniform(rng, 4 << scale, 8 << scale))
    n = _log_uniform(rng, 1 << 10, 1 << min(max_scale, 16))
    if kind == "er":
        return dict(graph="er", n=n, degree=round(rng.uniform(6.0, 24.0), 2))
    return dict(graph="ba", n=n, m=rng.randint(4, 9))


def draw(rng) -> dict:
    """One more case of the same ranges."""
    what = rng.choice(["small", "small", "wedge4", "clique", "clique", "five", "five", "six", "ref",
                       "batch", "ingest", "train", "gradient", "predict"])
    if what == "small":  # three- and four-vertex plan patterns
        return dict(kind="count", mode="exact", tile=32,
                    pattern=rng.choice([WEDGE, TRIANGLE, STAR4, PATH4, PAW, DIAMOND]),
                    **_draw_graph(rng, 17))
    if what == "wedge4":
        return dict(kind="count", mode="exact", pattern=rng.choice([K4, C4]), tile=32,
                    **_draw_graph(rng, 20))
    if what == "clique":
        pattern, top = rng.choice([(K4, 18), (K5, 16), (K6, 12), (K7, 10)])
        return dict(kind="count", mode="exact", pattern=pattern, tile=32, **_draw_graph(rng, top))
    if what == "six":
        graph = rng.choice([dict(graph="rmat", scale=10, samples=_log_uniform(rng, 1 << 12, 1 << 13)),
                            dict(graph="er", n=_log_uniform(rng, 1000, 8000),
                                 degree=round(rng.uniform(6.0, 16.0), 2))])
        return dict(kind="count", mode="exact", pattern=CYCLE6_CHORD, tile=32, **graph)
    if what == "five":
        return dict(kind="count", mode="exact", pattern=rng.choice(FIVE),
                    tile=rng.choice([32, 32, 16, 8]), **_draw_graph(rng, 12))
    if what == "ref":
        return dict(kind="count", mode="ref", tile=32,
                    pattern=rng.choice([TRIANGLE, K4, C4, PATH4, DIAMOND, HOUSE]),
                    **_draw_graph(rng, 12))
    if what == "batch":
        return dict(kind="batch", graphs=rng.randint(1, 8), max_log2=rng.randint(10, 12))
    if what == "ingest":
        return dict(kind="ingest", **_draw_graph(rng, 18))
    if what == "train":
        return dict(kind="train", rows=_log_uniform(rng, 200, 4001), features=rng.randint(8, 64),
                    epochs=rng.randint(1, 10), batch=rng.choice([64, 100, 256]))
    rows = _log_uniform(rng, 3, 20000)
    return dict(kind=what, rows=rows, features=rng.randint(8, 64))


def _graph(case: dict, seed: int) -> "g.Graph":
    seed = seed & 0xFFFFFFFF
    if case["graph"] == "rmat":
        return g.Graph.rmat(case["scale"], case["samples"], seed=seed, device=True)
    if case["graph"] == "er":
        return g.Graph.erdos_renyi(case["n"], case["degree"], seed)
    return g.Graph.barabasi_albert(case["n"], case["m"], seed, device=True)


def _batch_graphs(case: dict, seed: int) -> list["g.Graph"]:
    """Uneven graphs, alternately R-MAT and Barabasi-Albert: the first of the largest size, the others' vertex
    counts log-uniform below it."""
    rng = np.random.default_rng(seed)
    out = []
    for i in range(case["graphs"]):
        n = int(2 ** (case["max_log2"] if i == 0 else rng.uniform(9, case["max_log2"])))
        s = int(rng.integers(1 << 31))
        if i % 2 == 0:
            scale = max(1, round(math.log2(n)))
            out.append(g.Graph.rmat(scale, 8 << scale, seed=s, device=True))
        else:
            out.append(g.Graph.barabasi_albert(n, int(rng.integers(4, 10)), s, device=True))
    return out


def _mlp_inputs(case: dict, seed: int):
    """Standardised features, log-time-like targets and He-uniform weights."""
    rng = np.random.default_rng(seed)
    n, f = case["rows"], case["features"]
    X = rng.standard_normal((n, f)).astype(np.float32)
    T = (X[:, : min(f, 8)].sum(1) * 0.3 + np.abs(X[:, 0]) + 0.1 * rng.standard_normal(n)).astype(np.float32)
    p = [rng.uniform(-1, 1, (i, o)) * math.sqrt(6.0 / i) for i, o in ((f, 64), (64, 64), (64, 1))]
    params = np.concatenate([p[0].ravel(), np.zeros(64), p[1].ravel(), np.zeros(64), p[2].ravel(),
                             np.zeros(1)]).astype(np.float32)
    return X, T, params, int(rng.integers(1 << 31))


def prepare(case: dict, seed: int) -> dict:
    kind = case["kind"]
    if kind == "count":
        gr = _graph(case, seed)
        exact = case["mode"] == "exact"
        gr.upload(degree_order=exact)
        cfg = g.Config.engine_default()
        cfg.threads_per_warp = case["tile"]
        sched = g.Schedule(case["pattern"], case["mode"], gr if exact else None)
        return dict(kind=kind, graph=gr, schedule=sched, executor=g.Executor(cfg))
    if kind == "batch":
        graphs = _batch_graphs(case, seed)
        b = g.Batch()
        for gr in graphs:
            gr.upload()
            for p in FIVE:
                b.add(gr, g.Schedule(p, "exact"))
        b.prepare(g.Config.engine_default(), cuda_graph=True)
        return dict(kind=kind, batch=b)
    if kind == "ingest":
        off, adj = _graph(case, seed).csr()
        off, adj = torch.from_numpy(off).pin_memory(), torch.from_numpy(adj).pin_memory()
        return dict(kind=kind, off=off, adj=adj, executor=g.Executor(),
                    schedules=[g.Schedule(p, "exact") for p in (K4, C4)])
    X, T, params, shuffle = _mlp_inputs(case, seed)
    net = costmodel.MLP(case["features"], 0)
    net.set_params(params)
    return dict(kind=kind, case=case, net=net, X=X, T=T, params=params, shuffle=shuffle)


def run(state: dict):
    kind = state["kind"]
    if kind == "count":
        return state["executor"].count(state["graph"], state["schedule"]).count
    if kind == "batch":
        state["batch"].run()
        return np.array(state["batch"].counts(), dtype=np.int64)
    if kind == "ingest":
        gr = g.Graph.from_csr(state["off"].numpy(), state["adj"].numpy(), check_symmetry=False,
                              device=True)
        gr.upload()
        return [state["executor"].count(gr, s).count for s in state["schedules"]]
    net = state["net"]
    if kind == "predict":
        return net.predict(state["X"])
    if kind == "gradient":
        grad, loss = net.gradient(state["X"], state["T"])
        return dict(grad=grad, loss=loss)
    c = state["case"]
    net.set_params(state["params"])
    loss = net.train(state["X"], state["T"], epochs=c["epochs"], batch=c["batch"], lr=1e-3,
                     seed=state["shuffle"])
    return dict(params=net.params(), loss=loss)


def work(case: dict) -> dict:
    """Counts: the graph's CSR once.  Network: rows and parameters once per pass over them, 2 flops per
    parameter and row forward, 4 backward."""
    kind = case["kind"]
    if kind == "count" or kind == "ingest":
        V, E, _ = _graph(case, 1).info()
        return dict(bytes=8 * (V + 1) + 4 * E + 8, flops=0)
    if kind == "batch":
        infos = [gr.info() for gr in _batch_graphs(case, 1)]
        return dict(bytes=sum(8 * (v + 1) + 4 * e for v, e, _ in infos) + 8 * len(infos) * len(FIVE), flops=0)
    n, f = case["rows"], case["features"]
    p = f * 64 + 64 + 64 * 64 + 64 + 64 + 1
    if kind == "predict":
        return dict(bytes=4 * (n * f + n + p), flops=2 * n * p)
    if kind == "gradient":
        return dict(bytes=4 * (n * (f + 1) + 2 * p + 1), flops=6 * n * p)
    return dict(bytes=4 * case["epochs"] * n * (f + 1) + 8 * p, flops=6 * case["epochs"] * n * p)


# ------------------------------------------------------------------ the network in 64 bits


class _MT64:
    """mt19937_64, the generator the training shuffles draw from."""

    def __init__(self, seed: int):
        m = (1 << 64) - 1
        s = [seed & m]
        for i in range(1, 312):
            s.append((6364136223846793005 * (s[-1] ^ (s[-1] >> 62)) + i) & m)
        self.s, self.i = np.array(s, np.uint64), 312

    def _twist(self):
        s, up, low = self.s, np.uint64(0xFFFFFFFF80000000), np.uint64(0x7FFFFFFF)
        a, one = np.uint64(0xB5026F5AA96619E9), np.uint64(1)

        def mix(hi, lo, far):
            x = (hi & up) | (lo & low)
            return far ^ (x >> one) ^ np.where(x & one, a, np.uint64(0))

        s[:156] = mix(s[:156], s[1:157], s[156:312])
        s[156:311] = mix(s[156:311], s[157:312], s[:155])
        s[311:] = mix(s[311:], s[:1], s[155:156])
        x = s ^ ((s >> np.uint64(29)) & np.uint64(0x5555555555555555))
        x = x ^ ((x << np.uint64(17)) & np.uint64(0x71D67FFFEDA60000))
        x = x ^ ((x << np.uint64(37)) & np.uint64(0xFFF7EEE000000000))
        self.out, self.i = [int(v) for v in x ^ (x >> np.uint64(43))], 0

    def below(self, n: int) -> int:
        """Uniform in [0, n): the high word of a 64x64-bit product, rejecting the biased low words."""
        while True:
            if self.i >= 312:
                self._twist()
            p = self.out[self.i] * n
            self.i += 1
            low = p & ((1 << 64) - 1)
            if low >= n or low >= ((1 << 64) - n) % n:
                return p >> 64


def _shuffle(order: list, rng: _MT64) -> None:
    """std::shuffle as GNU libstdc++ does it: two positions from each draw."""
    n, i = len(order), 1
    if n % 2 == 0 and n > 0:
        j = rng.below(2)
        order[1], order[j] = order[j], order[1]
        i = 2
    while i < n:
        x, y = divmod(rng.below((i + 1) * (i + 2)), i + 2)
        order[i], order[x] = order[x], order[i]
        order[i + 1], order[y] = order[y], order[i + 1]
        i += 2


def _split(p: np.ndarray, f: int):
    at = np.cumsum([f * 64, 64, 64 * 64, 64, 64])
    w1, b1, w2, b2, w3, b3 = np.split(p, at)
    return w1.reshape(f, 64), b1, w2.reshape(64, 64), b2, w3, b3


def _forward(p, X):
    w1, b1, w2, b2, w3, b3 = _split(p, X.shape[1])
    h1 = np.maximum(X @ w1 + b1, 0)
    h2 = np.maximum(h1 @ w2 + b2, 0)
    return h1, h2, h2 @ w3 + b3[0]


def _gradient(p, X, T):
    _, _, w2, _, w3, _ = _split(p, X.shape[1])
    h1, h2, y = _forward(p, X)
    dy = 2 * (y - T) / len(T)
    d2 = np.outer(dy, w3) * (h2 > 0)
    d1 = (d2 @ w2.T) * (h1 > 0)
    parts = [X.T @ d1, d1.sum(0), h1.T @ d2, d2.sum(0), h2.T @ dy, [dy.sum()]]
    return np.concatenate([np.ravel(v) for v in parts]), float(np.mean((y - T) ** 2))


def exact(case: dict, seed: int):
    kind = case["kind"]
    if kind not in ("train", "gradient", "predict"):
        return None  # counts are whole numbers
    X, T, p, shuffle = _mlp_inputs(case, seed)
    X, T, p = X.astype(np.float64), T.astype(np.float64), p.astype(np.float64)
    if kind == "predict":
        return _forward(p, X)[2]
    if kind == "gradient":
        grad, loss = _gradient(p, X, T)
        return dict(grad=grad, loss=loss)
    rng, order = _MT64(shuffle), list(range(len(T)))
    m, v, step = np.zeros_like(p), np.zeros_like(p), 0
    lr, b1, b2, eps = (float(np.float32(x)) for x in (1e-3, 0.9, 0.999, 1e-8))
    for _ in range(case["epochs"]):
        _shuffle(order, rng)
        for b in range(0, len(order), case["batch"]):
            rows = order[b:b + case["batch"]]
            grad, _ = _gradient(p, X[rows], T[rows])
            step += 1
            m = b1 * m + (1 - b1) * grad
            v = b2 * v + (1 - b2) * grad * grad
            p = p - lr * (m / (1 - b1 ** step)) / (np.sqrt(v / (1 - b2 ** step)) + eps)
    return dict(params=p, loss=float(np.mean((_forward(p, X)[2] - T) ** 2)))
