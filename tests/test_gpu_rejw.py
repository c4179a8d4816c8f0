"""CompressMask rejection samplers over words in memory (gr_rejw.cu) against
the oracle, bit for bit, over consecutive calls of one generator object: sizes
around the rule that takes a call there and around tiles of trials, carried
lanes and (int32 kinds) the engine's half packet from call to call, several
engines, a plan too short for the call, more than one scratch buffer."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

if not torch.cuda.is_available():
    pytest.skip("needs a CUDA GPU", allow_module_level=True)

CASES = [("GAMMA", torch.float32, 0.5, 1.0, 0), ("GAMMA", torch.float64, 0.3, 2.0, 0),
         ("GAMMA", torch.float32, 0.97, 1.5, 0), ("GAMMA", torch.float64, 0.03, 1.0, 0),
         ("GAMMA", torch.float32, 1.5, 1.0, 0), ("GAMMA", torch.float64, 25.0, 0.5, 0),
         ("CHI_SQUARED", torch.float32, 7.0, 0.0, 0), ("BETA", torch.float32, 0.4, 0.7, 0),
         ("BETA", torch.float64, 0.9, 0.2, 0), ("FISHER_F", torch.float64, 1.0, 1.5, 0),
         ("POISSON", torch.int32, 100.0, 0.0, 0), ("BINOMIAL", torch.int32, 0.3, 0.0, 100),
         ("BINOMIAL", torch.int32, 0.8, 0.0, 60)]
NPDT = {torch.float32: np.float32, torch.float64: np.float64, torch.int32: np.int32}


def bits(x):
    return x.view(np.uint64 if x.itemsize == 8 else np.uint32)


def check(er, oracle, case, streams, packets, half=False):
    kind, tdt, a, b, t = case
    P = 8 if tdt == torch.float32 else 4
    u = er.Vmt19937_64(90, streams=streams)
    g = er._Gen(tdt, a, b, trials=t, kind=kind)
    es = [oracle.Engine(90 + 4 * k) for k in range(streams)]
    ogs = [oracle.Gen() for _ in range(streams)]
    if half:  # leaves half a packet in every engine's cache
        er.randBits(4 * streams, 1, u)
        for e in es:
            oracle.generate(e, oracle.Gen(), "RANDBITS", 4, np.int32)
    for pk in packets:
        n = pk * P
        out = g.generate(n * streams, 1, u).reshape(-1).cpu().numpy()
        for k in range(streams):
            ref = oracle.generate(es[k], ogs[k], kind, n, NPDT[tdt], a, b, t)
            assert np.array_equal(bits(out[k * n:(k + 1) * n]), bits(ref)), f"{case} packets={pk} stream {k}"
    u.sync()
    raw = er.raw_u64(u, 64 * streams).cpu().numpy().view(np.uint64)
    for k in range(streams):
        assert np.array_equal(raw[64 * k:64 * (k + 1)], es[k].raw(16)), "engine after the calls"


@pytest.mark.parametrize("case", CASES)
def test_sizes(gpulib, oracle, case):
    check(gpulib, oracle, case, 1, (511, 512, 513, 1024, 3, 4097, 1, 50000))


@pytest.mark.parametrize("case", CASES[-3:] + CASES[:2])
def test_half_packets_and_streams(gpulib, oracle, case):
    check(gpulib, oracle, case, 1, (512, 2049, 2), half=True)
    check(gpulib, oracle, case, 3, (600, 7, 1500), half=True)


@pytest.mark.parametrize("scale", ["0.3", "0.9"])
def test_short_plan(gpulib, oracle, monkeypatch, scale):
    monkeypatch.setenv("GR_REJECT_PLAN_SCALE", scale)
    for case in (CASES[0], CASES[1], CASES[4], CASES[-3]):
        check(gpulib, oracle, case, 1, (3000, 600), half=True)


def test_more_than_one_buffer(gpulib, oracle):
    check(gpulib, oracle, CASES[0], 1, (2300000, 512))


def test_filter_band_covers_the_errors():
    """The accept pre-test's band 2^-18 (1 + 40/alpha) against the spread
    between float32 and float64 evaluations of the bound qx."""
    rng = np.random.default_rng(3)
    for alpha in (0.01, 0.1, 0.5, 0.9, 0.999):
        vx = (rng.integers(0, 1 << 23, 200000) / (1 << 23) + 2.0 ** -26).astype(np.float32)
        lv32, lv64 = np.log(vx), np.log(vx.astype(np.float64))
        ia, am1 = np.float32(1) / np.float32(alpha), np.float32(alpha) - np.float32(1)
        q1 = np.exp(-np.exp(ia * lv32))
        q1x = np.exp(-np.exp(float(ia) * lv64))
        q2 = np.exp(np.log(np.float32(1) - lv32) * am1)
        q2x = np.exp(np.log(1 - lv64) * float(am1))
        band = 2.0 ** -18 * (1 + 40 / alpha)
        assert np.max(np.abs(q1 / q1x - 1)) < band / 19
        assert np.max(np.abs(q2 / q2x - 1)) < band / 19


@pytest.mark.parametrize("tdt", [torch.float32, torch.float64])
@pytest.mark.parametrize("alpha", [1.0001, 1.05, 1.5, 3.3, 19.5, 200.0, 30000.0])
def test_tan_filter_decides_as_the_reference(gpulib, oracle, tdt, alpha):
    """10^6 trials per shape: one accept flag that differs would shift every
    later value."""
    er = gpulib
    u, e = er.Vmt19937_64(5), oracle.Engine(5)
    npdt = np.float32 if tdt == torch.float32 else np.float64
    n = 1 << 20 if tdt == torch.float32 else 1 << 19
    out = er.gamma(n, 1, u, alpha, 1.0, dtype=tdt).reshape(-1).cpu().numpy()
    assert np.array_equal(bits(out), bits(oracle.generate(e, oracle.Gen(), "GAMMA", n, npdt, alpha, 1.0)))
