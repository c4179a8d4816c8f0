"""BetaGen's general branch through words in memory (gr_chain.cu) against the
oracle, bit for bit, over consecutive calls of one generator object (lanes
carried from call to call): sizes around the rule that takes a call there,
around one and several segments, composition groups, several engines, a plan
too short for the call (the one-CTA walk goes on), and a call of more than one
scratch buffer.  Both components closed form, either or both rejecting."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

if not torch.cuda.is_available():
    pytest.skip("needs a CUDA GPU", allow_module_level=True)


def bits(x):
    return x.view(np.uint64 if x.itemsize == 8 else np.uint32)


def check(er, oracle, kind, tdt, a, b, streams, packets, seed=4711):
    npdt = {torch.float32: np.float32, torch.float64: np.float64}[tdt]
    P = 8 if tdt == torch.float32 else 4
    u = er.Vmt19937_64(seed, streams=streams)
    g = er._Gen(tdt, a, b, kind=kind)
    es = [oracle.Engine(seed + 4 * k) for k in range(streams)]
    ogs = [oracle.Gen() for _ in range(streams)]
    look = sorted({0, streams // 2, streams - 1})
    for pk in packets:
        n = pk * P
        out = g.generate(n * streams, 1, u).reshape(-1).cpu().numpy()
        for k in look:
            ref = oracle.generate(es[k], ogs[k], kind, n, npdt, a, b)
            assert np.array_equal(bits(out[k * n:(k + 1) * n]), bits(ref)), f"packets={pk} stream {k}"
    u.sync()
    raw = er.raw_u64(u, 64 * streams).cpu().numpy().view(np.uint64)
    for k in look:
        assert np.array_equal(raw[64 * k:64 * (k + 1)], es[k].raw(16)), "engine after the calls"


@pytest.mark.parametrize("tdt", [torch.float32, torch.float64])
@pytest.mark.parametrize("a,b", [(0.5, 2.0), (2.0, 0.5), (1.0, 3.0), (2.5, 4.0), (0.3, 1.0), (22.0, 1.5), (0.2, 0.9 + 1),
                                 (1.0, 0.6), (0.05, 19.0), (3.0, 7.0)])
def test_one_engine(gpulib, oracle, tdt, a, b):
    check(gpulib, oracle, "BETA", tdt, a, b, 1, (191, 192, 193, 1000, 1701, 7, 20000, 3, 60001))


@pytest.mark.parametrize("streams", [3, 70, 300])
@pytest.mark.parametrize("tdt", [torch.float32, torch.float64])
@pytest.mark.parametrize("a,b", [(0.5, 2.0), (3.0, 0.4), (2.5, 1.5)])
def test_several_engines(gpulib, oracle, tdt, a, b, streams):
    check(gpulib, oracle, "BETA", tdt, a, b, streams, (200, 2500, 191, 400))


def test_fisher_f(gpulib, oracle):
    check(gpulib, oracle, "FISHER_F", torch.float32, 5.0, 2.0, 1, (300, 5000))
    check(gpulib, oracle, "FISHER_F", torch.float64, 1.0, 6.0, 1, (300, 5000))


@pytest.mark.parametrize("scale", ["0.4", "0.01"])
def test_short_plan(gpulib, oracle, monkeypatch, scale):
    monkeypatch.setenv("GR_WALK_PLAN_SCALE", scale)
    check(gpulib, oracle, "BETA", torch.float32, 0.5, 2.0, 1, (5000, 300, 20000))
    check(gpulib, oracle, "BETA", torch.float64, 2.5, 1.5, 3, (5000, 300))


def test_more_than_one_buffer(gpulib, oracle):
    check(gpulib, oracle, "BETA", torch.float32, 0.5, 2.0, 1, (1500000, 192))


@pytest.mark.parametrize("kind,a,t", [("POISSON", 4.0, 0), ("POISSON", 11.9, 0), ("POISSON", 0.05, 0),
                                      ("BINOMIAL", 0.004, 100), ("BINOMIAL", 0.996, 200)])
@pytest.mark.parametrize("streams", [1, 3])
def test_poisson_walk(gpulib, oracle, kind, a, t, streams):
    """PoissonGen (mean < 12) and BinomialGen (mean < 1): the same chain over
    half packets, with and without a cached half packet at the start."""
    er = gpulib
    u = er.Vmt19937_64(31, streams=streams)
    g = er._Gen(torch.int32, a, 0.0, trials=t, kind=kind)
    es = [oracle.Engine(31 + 4 * k) for k in range(streams)]
    ogs = [oracle.Gen() for _ in range(streams)]
    er.randBits(4 * streams, 1, u)
    for e in es:
        oracle.generate(e, oracle.Gen(), "RANDBITS", 4, np.int32)
    for pk in (511, 512, 513, 1300, 3, 9001, 60000):
        n = 4 * pk
        out = g.generate(n * streams, 1, u).reshape(-1).cpu().numpy()
        for k in range(streams):
            ref = oracle.generate(es[k], ogs[k], kind, n, np.int32, a, 0.0, t)
            assert np.array_equal(out[k * n:(k + 1) * n], ref), f"packets={pk} stream {k}"
    u.sync()
    raw = er.raw_u64(u, 64 * streams).cpu().numpy().view(np.uint64)
    for k in range(streams):
        assert np.array_equal(raw[64 * k:64 * (k + 1)], es[k].raw(16)), "engine after the calls"


def test_poisson_more_than_one_buffer(gpulib, oracle):
    er = gpulib
    u = er.Vmt19937_64(8)
    e, og = oracle.Engine(8), oracle.Gen()
    for n in (4 * 1400000, 4 * 600):
        out = er.poisson(n, 1, u, 4.0).reshape(-1).cpu().numpy()
        assert np.array_equal(out, oracle.generate(e, og, "POISSON", n, np.int32, 4.0))
    u.sync()
