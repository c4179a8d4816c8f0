"""BetaGen with one rejection component on many engines (k_beta's look-up of
whole visits, gr_samplers.cu) against the oracle, bit for bit: each pair of
sampler types and order, records at the edges of a block's positions, calls of
one packet and of many blocks, lanes carried from call to call."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

if not torch.cuda.is_available():
    pytest.skip("needs a CUDA GPU", allow_module_level=True)

# GS / tan with integral (1 to 19 packets) and exponential, both orders
PAIRS = [(0.5, 2.0), (2.0, 0.5), (0.5, 1.0), (1.0, 0.3), (1.5, 2.0), (2.0, 25.5), (0.03, 19.0), (19.0, 0.97),
         (1.0, 300.0), (20.0, 1.0), (1.01, 19.0)]
NPDT = {torch.float32: np.float32, torch.float64: np.float64}


@pytest.mark.parametrize("tdt", [torch.float32, torch.float64])
@pytest.mark.parametrize("kind,a,b", [("BETA", a, b) for a, b in PAIRS] + [("FISHER_F", 1.0, 4.0), ("FISHER_F", 6.0, 3.0)])
def test_many_engines(gpulib, oracle, kind, a, b, tdt):
    er = gpulib
    K, P = 300, 8 if tdt == torch.float32 else 4
    u = er.Vmt19937_64(17, streams=K)
    g = er._Gen(tdt, a, b, trials=0, kind=kind)
    which = (0, 1, 151, 299)
    es = {k: (oracle.Engine(17 + 4 * k), oracle.Gen()) for k in which}
    for pk in (1, 30, 47, 160, 161, 1500, 2):
        n = pk * P
        out = g.generate(n * K, 1, u).reshape(-1).cpu().numpy()
        for k in which:
            ref = oracle.generate(*es[k], kind, n, NPDT[tdt], a, b, 0)
            got = out[k * n:(k + 1) * n]
            bad = np.nonzero(got.view(np.uint8) != ref.view(np.uint8))[0]
            assert bad.size == 0, f"{pk} packets, stream {k}: {bad[:3]}"
    u.sync()
    raw = er.raw_u64(u, 64 * K).cpu().numpy().view(np.uint64)
    for k in which:
        assert np.array_equal(raw[64 * k:64 * (k + 1)], es[k][0].raw(16)), "engine after the calls"


@pytest.mark.parametrize("tdt", [torch.float32, torch.float64])
@pytest.mark.parametrize("a,b", PAIRS[:8])
def test_one_engine_small_calls(gpulib, oracle, a, b, tdt):
    er = gpulib
    P = 8 if tdt == torch.float32 else 4
    u, e = er.Vmt19937_64(5), oracle.Engine(5)
    g, og = er._Gen(tdt, a, b, trials=0, kind="BETA"), oracle.Gen()
    for pk in (1, 2, 60, 191, 5, 104):
        out = g.generate(pk * P, 1, u).reshape(-1).cpu().numpy()
        ref = oracle.generate(e, og, "BETA", pk * P, NPDT[tdt], a, b, 0)
        assert np.array_equal(out.view(np.uint8), ref.view(np.uint8)), pk
