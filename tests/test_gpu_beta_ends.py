"""Where short beta calls end (k_beta, gr_samplers.cu: the last outputs of a call
trial by trial, masks decided by the filters and then one open position after the
other): sizes around an engine block's worth of packets, in consecutive calls of
one generator object, against the oracle, bit for bit."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

if not torch.cuda.is_available():
    pytest.skip("needs a CUDA GPU", allow_module_level=True)

NPDT = {torch.float32: np.float32, torch.float64: np.float64}


@pytest.mark.parametrize("tdt", [torch.float32, torch.float64])
@pytest.mark.parametrize("a,b", [(0.5, 2.0), (3.0, 2.5), (2.5, 1.0), (2.5, 1.5), (0.05, 19.0), (0.5, 1.5), (1e-4, 2.0),
                                 (1.0, 3.0)])
@pytest.mark.parametrize("streams", [1, 300])
def test_short_calls(gpulib, oracle, a, b, tdt, streams):
    er = gpulib
    P = 8 if tdt == torch.float32 else 4
    u = er.Vmt19937_64(801, streams=streams)
    g = er._Gen(tdt, a, b, kind="BETA")
    which = sorted({0, streams // 2, streams - 1})
    es = {k: (oracle.Engine(801 + 4 * k), oracle.Gen()) for k in which}
    for pk in (1, 2, 5, 15, 16, 17, 18, 33, 47, 48, 49, 50, 51, 52, 64, 95, 96, 97, 101, 102, 103, 160, 161, 177):
        n = pk * P
        out = g.generate(n * streams, 1, u).reshape(-1).cpu().numpy()
        for k in which:
            ref = oracle.generate(*es[k], "BETA", n, NPDT[tdt], a, b)
            assert np.array_equal(out[k * n:(k + 1) * n].view(np.uint8), ref.view(np.uint8)), f"packets={pk} stream {k}"
    u.sync()
    raw = er.raw_u64(u, 64 * streams).cpu().numpy().view(np.uint64)
    for k in which:
        assert np.array_equal(raw[64 * k:64 * (k + 1)], es[k][0].raw(16)), f"words after the calls, stream {k}"
