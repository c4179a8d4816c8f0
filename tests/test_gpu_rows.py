"""Rows of gamma draws in one launch (Dirichlet and Wishart calls on 128 engines and
more: generate_gamma_rows, k_trials over several rows) against the oracle: rows of
every kind of shape beside each other, each stream's words and carried lanes taken
on from row to row and from call to call, uneven and empty slices, another engine
count in between, captured calls, and the words left afterwards.  Dirichlet bit for
bit (column sums in category order); Wishart within the products' rounding."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

if not torch.cuda.is_available():
    pytest.skip("needs a CUDA GPU", allow_module_level=True)

NPDT = {torch.float32: np.float32, torch.float64: np.float64}
ALPHA = np.array([0.03, 1.0, 19.0, 1.5, 0.5, 2.0, 30.5, 1e-4, 5.0, 0.999, 20.0, 1.0001])


class Stream:
    """One stream of the object: its engine and a generator state per row."""

    def __init__(self, oracle, seed, k, nrows):
        self.e = oracle.Engine(seed + 4 * k)
        self.gens = [oracle.Gen() for _ in range(nrows)]


def slice_of(k, K, packets):
    per, rem = divmod(packets, K)
    first = k * per + min(k, rem)
    return first, per + (1 if k < rem else 0)


def check_words(er, u, K, streams):
    u.sync()
    raw = er.raw_u64(u, 64 * K).cpu().numpy().view(np.uint64)
    for k, s in streams.items():
        assert np.array_equal(raw[64 * k:64 * (k + 1)], s.e.raw(16)), f"words after the calls, stream {k}"


def expect_dirichlet(oracle, streams, K, x, packets, tdt):
    P = 8 if tdt == torch.float32 else 4
    x = x.t().contiguous().cpu().numpy()  # samples x dim
    for k, s in streams.items():
        first, cnt = slice_of(k, K, packets)
        if not cnt:
            continue
        rows = [oracle.generate(s.e, s.gens[i], "GAMMA", cnt * P, NPDT[tdt], float(a), 1.0) for i, a in enumerate(ALPHA)]
        tot = rows[0]
        for r in rows[1:]:
            tot = tot + r
        ref = np.stack([r / tot for r in rows], axis=1)
        got = x[first * P:(first + cnt) * P]
        assert np.array_equal(got.view(np.uint8), np.ascontiguousarray(ref).view(np.uint8)), f"packets={packets} stream {k}"


@pytest.mark.parametrize("tdt", [torch.float32, torch.float64])
@pytest.mark.parametrize("K", [128, 300])
def test_dirichlet(gpulib, oracle, K, tdt):
    er = gpulib
    P = 8 if tdt == torch.float32 else 4
    g = er.DirichletGen(ALPHA, dtype=tdt)
    which = (0, 1, 57, K - 1)
    u = er.Vmt19937_64(70, streams=K)
    streams = {k: Stream(oracle, 70, k, len(ALPHA)) for k in which}
    for packets in (3 * K + 58, K, 5, 41 * K + 1, K - 1, 400 * K + 2):
        expect_dirichlet(oracle, streams, K, g.generate(u, packets * P), packets, tdt)
    check_words(er, u, K, streams)


def test_dirichlet_engine_counts_in_turn(gpulib, oracle):
    """Another engine count starts the generators' carried lanes anew (and takes the
    rows one by one below 128 engines); the same engines go on with their words."""
    er = gpulib
    g = er.DirichletGen(ALPHA)
    engines = {}
    for K, packets in ((128, 300), (200, 511), (128, 129), (64, 200), (128, 1000), (128, 77), (200, 200)):
        if K not in engines:
            engines[K] = (er.Vmt19937_64(9 * K, streams=K), {k: Stream(oracle, 9 * K, k, len(ALPHA)) for k in (0, K // 2, K - 1)})
        u, streams = engines[K]
        if engines.get("last") != K:
            for s in streams.values():
                s.gens = [oracle.Gen() for _ in ALPHA]
        engines["last"] = K
        expect_dirichlet(oracle, streams, K, g.generate(u, 8 * packets), packets, torch.float32)
    for K in (64, 128, 200):
        check_words(er, engines[K][0], K, engines[K][1])


def test_dirichlet_captured(gpulib, oracle):
    er = gpulib
    K, packets = 150, 700
    g = er.DirichletGen(ALPHA)
    u = er.Vmt19937_64(31, streams=K)
    streams = {k: Stream(oracle, 31, k, len(ALPHA)) for k in (0, 99, K - 1)}
    s = torch.cuda.Stream()
    with torch.cuda.stream(s):
        first = g.generate(u, 8 * packets, stream=s)  # grows the scratch, makes the rows' table
        s.synchronize()
        out = torch.empty_strided(first.shape, first.stride(), dtype=first.dtype, device="cuda")
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=s):
            g.generate(u, 8 * packets, out=out, stream=s)
        for x in (first, None, None):
            if x is None:
                graph.replay()
                s.synchronize()
                x = out
            expect_dirichlet(oracle, streams, K, x, packets, torch.float32)
    check_words(er, u, K, streams)


@pytest.mark.parametrize("d,df,tdt,tol", [(3, 4, torch.float32, 1e-5), (6, 21, torch.float32, 1e-5), (5, 24, torch.float64, 1e-12)])
def test_wishart(gpulib, oracle, d, df, tdt, tol):
    """chi-squared rows of df, df - 1, ...: GS, integral and tan shapes beside each other."""
    er = gpulib
    K, P = 130, 8 if tdt == torch.float32 else 4
    a = np.random.default_rng(2).standard_normal((d, d))
    scale = a @ a.T + d * np.eye(d)
    g = er.WishartGen(df, scale, dtype=tdt)
    u = er.Vmt19937_64(41, streams=K)
    es = [oracle.Engine(41 + 4 * k) for k in range(K)]
    norm = [oracle.Gen() for _ in range(K)]
    chi = [[oracle.Gen() for _ in range(d)] for _ in range(K)]
    L = oracle.get_lt(scale)
    for packets in (2 * K + 11, 3 * K, 44):
        n = packets * P
        W = g.generate(u, n).cpu().numpy().astype(np.float64)
        nn = n * d * (d - 1) // 2
        z = [oracle.generate(es[k], norm[k], "NORMAL_STD", slice_of(k, K, nn // P)[1] * P, NPDT[tdt])
             if slice_of(k, K, nn // P)[1] else np.empty(0, NPDT[tdt]) for k in range(K)]
        chis = np.empty((d, n), NPDT[tdt])
        for k in range(K):
            first, cnt = slice_of(k, K, packets)
            for i in range(d):
                if cnt:
                    chis[i, first * P:(first + cnt) * P] = oracle.generate(es[k], chi[k][i], "CHI_SQUARED", cnt * P, NPDT[tdt],
                                                                           float(df - i))
        ref = oracle.wishart_f64(L, np.concatenate(z), chis, d, n)
        assert np.max(np.abs(W - ref)) <= tol * np.max(np.abs(ref)), f"packets={packets}"
    u.sync()
    raw = er.raw_u64(u, 64 * K).cpu().numpy().view(np.uint64)
    for k in range(K):
        assert np.array_equal(raw[64 * k:64 * (k + 1)], es[k].raw(16)), f"words after the calls, stream {k}"
