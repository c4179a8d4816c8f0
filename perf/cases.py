"""The calls this library is measured on.

Each case is one pass through the public Python API, with the engine (and the
generator object, where a program keeps one) made beforehand and carried from
pass to pass, as a program that samples repeatedly does.  Two ways of holding
an engine are in use: one ``Vmt19937_64`` (the reference's own programs and
benchmark, bit-exact with the single stream) and 608 of them in one handle (the
one-engine-per-thread use, which fills the GPU).

``exact`` restates the fixed-draw kinds in 64-bit arithmetic with plain torch:
MT19937-64, the bit-to-uniform conversion in the output's own type, then the
transform in float64.
"""
import math

import numpy as np
import torch

import eigenrand_gb300 as er

DT = {"f32": torch.float32, "f64": torch.float64, "i32": torch.int32}
SIZE = {"f32": 4, "f64": 8, "i32": 4}
M64 = (1 << 64) - 1

# The univariate sweep of the library's benchmark: (kind, a, b, trials).
SWEEP_REAL = [("uniformReal", 0, 0, 0), ("balanced", 0, 0, 0), ("exponential", 1, 0, 0), ("normal", 0, 1, 0),
              ("lognormal", 0, 1, 0), ("cauchy", 0, 1, 0), ("weibull", 1.5, 1, 0), ("gamma", 0.5, 1, 0),
              ("gamma", 1, 1, 0), ("gamma", 5, 1, 0), ("beta", 0.5, 2, 0)]
SWEEP_INT = [("poisson", 4, 0, 0), ("poisson", 100, 0, 0), ("binomial", 0.3, 0, 20), ("discrete", 0, 0, 16)]
CLOSED = ("uniformReal", "balanced", "exponential", "normal", "lognormal", "cauchy", "weibull")


def _uni(name, kind, dtype, rows, cols, streams, a=0.0, b=0.0, trials=0):
    c = {"op": "univariate", "kind": kind, "dtype": dtype, "rows": rows, "cols": cols, "streams": streams,
         "a": float(a), "b": float(b), "trials": trials}
    return dict(c, name=name) if name else c


def listed():
    return [
        # one small vector from one engine: noise for a step of a control loop or a unit test
        _uni("normal_f32_32x32_one", "normal", "f32", 32, 32, 1, 0, 1),
        # the reference benchmark's array size give or take one, a size that is no whole number of packets
        _uni("uniform_f32_1001x999_one", "uniformReal", "f32", 1001, 999, 1),
        # filling a large buffer with uniforms: Monte Carlo input, dropout masks
        _uni("uniform_f32_8192x8192_608", "uniformReal", "f32", 8192, 8192, 608),
        # double-precision Monte Carlo paths
        _uni("normal_f64_3001x2000_608", "normal", "f64", 3001, 2000, 608, 0, 1),
        # the reference benchmark's gamma call (rejection) at its 1000 x 1000, in double
        _uni("gamma05_f64_1000x1000_one", "gamma", "f64", 1000, 1000, 1, 0.5, 1),
        # A/B-test posterior draws: a beta call on one engine
        _uni("beta_f32_1000x1000_one", "beta", "f32", 1000, 1000, 1, 0.5, 2),
        # the whole univariate sweep at 1024 x 1024 on one engine, as the reference benchmark runs it
        {"name": "sweep_1024_one", "op": "sweep", "rows": 1024, "cols": 1024, "streams": 1},
        # the same sweep at 4096 x 4096 on 608 engines: the library's headline workload
        {"name": "sweep_4096_608", "op": "sweep", "rows": 4096, "cols": 4096, "streams": 608},
        # correlated normals: a million draws of a 64-dimensional Gaussian
        {"name": "mvnormal_d64_1e6", "op": "mvnormal", "dim": 64, "samples": 1000000, "streams": 608},
        # random covariance matrices for Bayesian models
        {"name": "wishart_d32_1e5", "op": "wishart", "dim": 32, "df": 40, "samples": 100000, "streams": 608},
        # topic-model style mixture weights
        {"name": "dirichlet_k64_1e6", "op": "dirichlet", "dim": 64, "samples": 1000000, "streams": 608},
        # many gamma parameter sets with uneven counts in one call
        {"name": "batched_gamma_2e5", "op": "batched", "sets": 200000, "most": 4096},
    ]


def _log(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def draw(rng):
    op = rng.choice(["univariate"] * 6 + ["sweep", "mvnormal", "wishart", "dirichlet", "batched"])
    if op == "univariate":
        kind = rng.choice(["uniformReal", "balanced", "exponential", "normal", "lognormal", "cauchy", "weibull",
                           "gamma", "gamma", "beta", "poisson", "binomial", "discrete"])
        dtype = "i32" if kind in ("poisson", "binomial", "discrete") else rng.choice(["f32", "f64"])
        streams = rng.choice([1, 1, 608])
        most = 1 << 26
        if dtype != "f32" or kind not in ("uniformReal", "balanced", "exponential", "normal"):
            most = 1 << 24
        if kind == "beta":  # the costliest sampler on one engine
            most = 1000000 if streams == 1 else 1 << 22
        n = _log(rng, 1024, most)
        cols = max(8, 8 * int(math.sqrt(n) / 8))
        rows = max(1, int(n / cols))
        if kind in ("uniformReal", "balanced") and rng.random() < 0.5:
            cols += rng.randrange(8)  # a partial last packet, which only these kinds take
        a, b, trials = 0.0, 1.0, 0
        if kind in ("gamma", "beta"):
            a = rng.choice([0.5, 1.0, 2.0, 5.0, round(_log(rng, 0.1, 20), 3)])
            b = 1.0 if kind == "gamma" else rng.choice([0.5, 2.0, round(_log(rng, 0.5, 8), 3)])
        elif kind == "exponential":
            a = rng.choice([1.0, round(_log(rng, 0.1, 10), 3)])
        elif kind == "weibull":
            a = round(_log(rng, 0.5, 5), 3)
        elif kind == "poisson":
            a = round(_log(rng, 0.5, 200), 3)
        elif kind == "binomial":
            a, trials = round(rng.uniform(0.05, 0.95), 3), int(_log(rng, 4, 500))
        elif kind == "discrete":
            trials = int(_log(rng, 3, 200))
        return _uni(None, kind, dtype, rows, cols, streams, a, b, trials)
    if op == "sweep":
        streams = rng.choice([1, 608])
        side = 8 * int(_log(rng, 16, 128 if streams == 1 else 500))
        return {"op": op, "rows": side, "cols": side, "streams": streams}
    if op == "mvnormal":
        dim = int(_log(rng, 2, 256))
        return {"op": op, "dim": dim, "samples": 8 * int(_log(rng, 100, min(125000, 8000000 // dim))),
                "streams": rng.choice([1, 608])}
    if op == "wishart":
        dim = int(_log(rng, 2, 64))
        return {"op": op, "dim": dim, "df": dim + rng.randrange(1, 20),
                "samples": 8 * int(_log(rng, 100, min(12500, 12800000 // (dim * dim)))), "streams": 608}
    if op == "dirichlet":
        dim = int(_log(rng, 2, 128))
        return {"op": op, "dim": dim, "samples": 8 * int(_log(rng, 100, min(125000, 8000000 // dim))),
                "streams": 608}
    return {"op": op, "sets": int(_log(rng, 1000, 200000)), "most": int(_log(rng, 64, 4096))}


# ---------------------------------------------------------------- one call
def _weights(n, seed):
    return np.random.default_rng(seed).uniform(0, 1, n).tolist()


def _call(kind, dtype, rows, cols, urng, a, b, trials, weights=None):
    dt = DT[dtype]
    if kind in ("uniformReal", "balanced"):
        return getattr(er, kind)(rows, cols, urng, dtype=dt)
    if kind == "normal":
        return er.normal(rows, cols, urng, dtype=dt)
    if kind == "exponential":
        return er.exponential(rows, cols, urng, a, dtype=dt)
    if kind in ("lognormal", "cauchy", "weibull", "gamma", "beta"):
        return getattr(er, kind)(rows, cols, urng, a, b, dtype=dt)
    if kind == "poisson":
        return er.poisson(rows, cols, urng, a)
    if kind == "binomial":
        return er.binomial(rows, cols, urng, trials, a)
    return er.discrete(rows, cols, urng, weights)


def _covariance(dim, seed):
    rng = np.random.default_rng(seed)
    x = rng.standard_normal((dim, dim))
    return rng.standard_normal(dim), x @ x.T + dim * np.eye(dim)


def _engine_seed(seed):
    return (1234 + 8191 * seed) & M64


def prepare(case, seed):
    s = {"case": case}
    if case["op"] == "batched":
        rng = np.random.default_rng(seed)
        n = case["sets"]
        # the same counts in another order for another seed, so that the total stays the same
        counts = np.random.default_rng(n).integers(1, case["most"] + 1, n).astype(np.int32)
        counts = torch.from_numpy(rng.permutation(counts)).cuda()
        s["counts"] = counts
        s["a"] = torch.from_numpy((10.0 ** rng.uniform(-1, 2, n)).astype(np.float32)).cuda()
        s["b"] = torch.ones(n, dtype=torch.float32, device="cuda")
        ends = torch.cumsum(counts.to(torch.int64), 0)
        s["offsets"] = ends - counts
        s["out"] = torch.empty(int(ends[-1]), dtype=torch.float32, device="cuda")
        s["seed"] = _engine_seed(seed)
        return s
    s["urng"] = er.Vmt19937_64(_engine_seed(seed), streams=case["streams"])
    if case["op"] == "univariate" and case["kind"] == "discrete":
        s["weights"] = _weights(case["trials"], seed)
    elif case["op"] == "sweep":
        s["weights"] = _weights(16, seed)
    elif case["op"] == "mvnormal":
        s["gen"] = er.MvNormalGen(*_covariance(case["dim"], seed))
    elif case["op"] == "wishart":
        s["gen"] = er.WishartGen(case["df"], _covariance(case["dim"], seed)[1])
    elif case["op"] == "dirichlet":
        s["gen"] = er.DirichletGen(np.random.default_rng(seed).uniform(0.1, 2.0, case["dim"]))
    return s


def run(s):
    c = s["case"]
    if c["op"] == "univariate":
        return _call(c["kind"], c["dtype"], c["rows"], c["cols"], s["urng"], c["a"], c["b"], c["trials"],
                     s.get("weights"))
    if c["op"] == "sweep":
        r, k, u = c["rows"], c["cols"], s["urng"]
        out = []
        for kind, a, b, t in SWEEP_REAL:
            out += [_call(kind, d, r, k, u, a, b, t) for d in ("f32", "f64")]
        return out + [_call(kind, "i32", r, k, u, a, b, t, s["weights"]) for kind, a, b, t in SWEEP_INT]
    if c["op"] == "batched":
        return er.sample_batched("GAMMA", s["counts"], s["a"], s["b"], seed=s["seed"], out=s["out"],
                                 offsets=s["offsets"])[0]
    return s["gen"].generate(s["urng"], c["samples"])


def work(case):
    """The output, written once, and for the matrix kinds the products (the
    lower triangle counted as half).  Sampling reads nothing but engine state;
    its integer and bit operations are not counted as flops."""
    if case["op"] == "univariate":
        return {"bytes": case["rows"] * case["cols"] * SIZE[case["dtype"]], "flops": 0}
    if case["op"] == "sweep":
        n = case["rows"] * case["cols"]
        return {"bytes": n * (len(SWEEP_REAL) * 12 + len(SWEEP_INT) * 4), "flops": 0}
    if case["op"] == "batched":
        return {"bytes": case["sets"] * (20 + 4 * (case["most"] + 1) // 2), "flops": 0}
    d, n = case["dim"], case["samples"]
    if case["op"] == "mvnormal":
        return {"bytes": 4 * d * n, "flops": d * (d + 1) * n}
    if case["op"] == "wishart":
        return {"bytes": 4 * d * d * n, "flops": (d ** 3 // 3 + d ** 3 // 3 + d * d) * n}
    return {"bytes": 4 * d * n, "flops": 2 * d * n}


# ---------------------------------------------------------------- 64-bit values
def _i64(x):
    return x - (1 << 64) if x >= 1 << 63 else x


def _srl(x, n):
    return (x >> n) & ((1 << (64 - n)) - 1)


class _Words:
    """K Vmt19937_64 engines (lanes seeded seed + 4k + l) as int64 bit patterns."""

    def __init__(self, seed, streams):
        w = np.empty((312, 4 * streams), np.uint64)
        w[0] = np.uint64(seed) + np.arange(4 * streams, dtype=np.uint64)
        f = np.uint64(6364136223846793005)
        for i in range(1, 312):
            w[i] = (w[i - 1] ^ (w[i - 1] >> np.uint64(62))) * f + np.uint64(i)
        self.mt = torch.from_numpy(w.view(np.int64)).cuda()
        self.streams = streams
        self.left = torch.empty((0, 4 * streams), dtype=torch.int64, device="cuda")

    @staticmethod
    def _twist(a, b, c):
        t = (a & _i64(M64 ^ ((1 << 31) - 1))) | (b & ((1 << 31) - 1))
        return _srl(t, 1) ^ (-(t & 1) & _i64(0xb5026f5aa96619e9)) ^ c

    def packets(self, n):
        """The next n packets of every engine, (streams, n, 4)."""
        got = [self.left]
        have = self.left.shape[0]
        while have < n:
            o = self.mt
            lo = self._twist(o[:156], o[1:157], o[156:312])
            hi = self._twist(o[156:312], torch.cat([o[157:312], lo[:1]]), lo)
            r = self.mt = torch.cat([lo, hi])
            r = r ^ (_srl(r, 29) & 0x5555555555555555)
            r = r ^ ((r << 17) & 0x71d67fffeda60000)
            r = r ^ ((r << 37) & _i64(0xfff7eee000000000))
            got.append(r ^ _srl(r, 43))
            have += 312
        w = torch.cat(got)
        self.left = w[n:].clone()
        return w[:n].reshape(n, self.streams, 4).transpose(0, 1)


def _halves(w):
    """The 32-bit words of 64-bit lanes, low first, as non-negative int64."""
    return torch.stack([w & 0xffffffff, _srl(w, 32)], -1).flatten(-2)


def _uniform(w, dtype):
    """bit_to_ur of packet words: exact in the output's type, as float64."""
    if dtype == "f32":
        return (_halves(w) & 0x7fffff).double() / (1 << 23)
    return (w & ((1 << 52) - 1)).double() / (1 << 52)


def _fixed_draws(words, kind, dtype, n, a, b):
    """n values of a fixed-draw kind from `words`, split over its engines.
    None for Cauchy in float: its norm is that of the few values next to the
    pole, where the rounding of pi (u - 1/2) to float decides the value."""
    width = 8 if dtype == "f32" else 4
    tail = n % width
    each, more = divmod(n // width, words.streams)
    most = each + (1 if more else 0)
    if tail and words.streams > 1 and more:
        return None  # the tail's engine stops one packet before the others do
    use = most
    if kind in ("normal", "lognormal"):
        use += most % 2
    if kind == "balanced" and dtype == "f64":
        use = (most + 1) // 2
    w = words.packets(use)
    tailw = words.packets(tail)[-1, :, 0] if tail else None
    if kind in ("normal", "lognormal"):
        u = _uniform(w, dtype).reshape(words.streams, use // 2, 2, width)
        radius = torch.sqrt(-2.0 * torch.log1p(-u[:, :, 0]))
        theta = 2.0 * math.pi * u[:, :, 1]
        v = torch.stack([radius * torch.sin(theta), radius * torch.cos(theta)], 2)
        if kind == "lognormal":
            v = torch.exp(v * b + a)
    elif kind == "balanced":
        scale = float(1 << 31) if dtype == "f32" else float((1 << 31) - 1)
        v = (_halves(w) & 0x7fffffff).double() / scale * 2.0 - 1.0
    else:
        u = _uniform(w, dtype)
        if kind == "uniformReal":
            v = u
        elif kind == "exponential":
            v = -torch.log1p(-u) / a
        elif kind == "cauchy":
            v = a + b * torch.tan(math.pi * (u - 0.5))
        else:
            v = torch.exp(torch.log(-torch.log1p(-u)) / a) * b
    if kind == "cauchy" and dtype == "f32":
        return None
    v = v.reshape(words.streams, -1)
    parts = [v[:more, :(each + 1) * width].flatten(), v[more:, :each * width].flatten()]
    if tail:
        if kind == "uniformReal":
            parts.append(_uniform(tailw[:, None], dtype)[:, 0] if dtype == "f64" else
                         _uniform(tailw, dtype)[::2])
        else:
            parts.append((tailw & 0x7fffffff).double() / float((1 << 31) - (dtype == "f64")) * 2.0 - 1.0)
    return torch.cat(parts)


def _shaped(v, rows, cols):
    return None if v is None else v.reshape(cols, rows).t()


def exact(case, seed):
    """float64 values of the kinds with a fixed number of draws per value.
    None for the rejection kinds (which candidates they keep hangs on their
    comparisons' rounding), for the sweep calls after the first of those, and
    for the full-size sweep (too long)."""
    if case["op"] == "univariate" and case["kind"] in CLOSED:
        words = _Words(_engine_seed(seed), case["streams"])
        v = _fixed_draws(words, case["kind"], case["dtype"], case["rows"] * case["cols"], case["a"], case["b"])
        return _shaped(v, case["rows"], case["cols"])
    if case["op"] == "sweep" and case["streams"] == 1:
        words = _Words(_engine_seed(seed), 1)
        n = case["rows"] * case["cols"]
        out = []
        for kind, a, b, _ in SWEEP_REAL:
            for d in ("f32", "f64"):
                v = _fixed_draws(words, kind, d, n, a, b) if kind in CLOSED else None
                out.append(_shaped(v, case["rows"], case["cols"]))
        return out + [None] * len(SWEEP_INT)
    if case["op"] == "mvnormal":
        d, n = case["dim"], case["samples"]
        mean, cov = (torch.from_numpy(x).cuda() for x in _covariance(d, seed))
        z = _fixed_draws(_Words(_engine_seed(seed), case["streams"]), "normal", "f32", d * n, 0, 1)
        return (z.reshape(n, d) @ torch.linalg.cholesky(cov).t() + mean).t()
    return None
