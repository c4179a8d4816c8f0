"""Calls captured in a CUDA graph after a smaller warm-up call of the same
generator object, on sizes that take other paths than the warm-up: replayed once,
the output and the raw words afterwards against the oracle.  A longer call
between capture and replay leaves the graph's memory alone."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

if not torch.cuda.is_available():
    pytest.skip("needs a CUDA GPU", allow_module_level=True)

NPDT = {torch.float32: np.float32, torch.float64: np.float64, torch.int32: np.int32}
# kind, type, a, b, trials, engines, packets of the warm-up, of the captured call
CASES = [("NORMAL_STD", torch.float64, 0.0, 0.0, 0, 1, 100, 200), ("UNIFORM_REAL", torch.float32, 0.0, 0.0, 0, 1, 64, 3000),
         ("RANDBITS", torch.int32, 0.0, 0.0, 0, 1, 64, 600001), ("NORMAL_STD", torch.float32, 0.0, 0.0, 0, 100, 64, 700),
         ("GAMMA", torch.float32, 0.5, 1.0, 0, 1, 400, 70000), ("GAMMA", torch.float64, 2.5, 1.0, 0, 64, 64, 600),
         ("BETA", torch.float32, 0.5, 2.0, 0, 32, 64, 500), ("BETA", torch.float64, 0.5, 2.0, 0, 1, 64, 20000),
         ("POISSON", torch.int32, 4.0, 0.0, 0, 32, 64, 700), ("POISSON", torch.int32, 100.0, 0.0, 0, 16, 64, 700),
         ("BINOMIAL", torch.int32, 0.3, 0.0, 20, 100, 16, 100)]


@pytest.mark.parametrize("case", CASES)
def test_capture_after_a_smaller_call(gpulib, oracle, case):
    er = gpulib
    kind, tdt, a, b, t, K, warm, packets = case
    P = 8 if tdt == torch.float32 else 4
    u = er.Vmt19937_64(61, streams=K)
    g = er._Gen(tdt, a, b, trials=t, kind=kind)
    which = sorted({0, K // 2, K - 1})
    es = {k: (oracle.Engine(61 + 4 * k), oracle.Gen()) for k in which}

    def expect(x, pk):
        x = x.reshape(-1).cpu().numpy()
        n = pk * P
        for k in which:
            ref = oracle.generate(*es[k], kind, n, NPDT[tdt], a, b, t)
            assert np.array_equal(x[k * n:(k + 1) * n].view(np.uint8), ref.view(np.uint8)), f"{case} stream {k}"

    s = torch.cuda.Stream()
    with torch.cuda.stream(s):
        first = g.generate(warm * P * K, 1, u, stream=s)
        s.synchronize()
        expect(first, warm)
        out = torch.zeros(packets * P * K, 1, dtype=tdt, device="cuda")
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=s):
            g.generate(packets * P * K, 1, u, out=out, stream=s)
        # a longer call on the same engine, then on from its end with the graph
        longer = g.generate(2 * packets * P * K, 1, u, stream=s)
        graph.replay()
        s.synchronize()
    expect(longer, 2 * packets)
    expect(out, packets)
    u.sync()
    raw = er.raw_u64(u, 64 * K).cpu().numpy().view(np.uint64)
    for k in which:
        assert np.array_equal(raw[64 * k:64 * (k + 1)], es[k][0].raw(16)), f"words after the calls, stream {k}"
