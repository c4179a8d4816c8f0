"""Shapes whose trials nearly all are fully accepted, so that the carried lanes
come from trials far back (gr_rejw.cu: fifo_lane, gr_chain.cu: carried_lane):
against the oracle, bit for bit (0 / 0 of two underflowed draws: NaN for NaN, its
sign is the host's), over consecutive calls, and no slower than an ordinary
shape."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

if not torch.cuda.is_available():
    pytest.skip("needs a CUDA GPU", allow_module_level=True)

NPDT = {torch.float32: np.float32, torch.float64: np.float64}
U = {torch.float32: np.uint32, torch.float64: np.uint64}
SHAPES = [("GAMMA", 1e-6, 1.0), ("GAMMA", 1e-4, 1.0), ("GAMMA", 2e-3, 1.0), ("BETA", 1e-4, 1e-4), ("BETA", 1e-3, 0.9),
          ("BETA", 1e-5, 2.0), ("BETA", 1e-3, 2.0), ("BETA", 3.0, 1e-4), ("BETA", 1e-4, 2.5), ("BETA", 1.0, 2e-3)]


@pytest.mark.parametrize("tdt", [torch.float32, torch.float64])
@pytest.mark.parametrize("kind,a,b", SHAPES)
@pytest.mark.parametrize("streams,calls", [(1, (20000, 513, 60001, 7)), (70, (700, 3000, 5))])
def test_values(gpulib, oracle, kind, a, b, tdt, streams, calls):
    er = gpulib
    P = 8 if tdt == torch.float32 else 4
    u = er.Vmt19937_64(15, streams=streams)
    g = er._Gen(tdt, a, b, kind=kind)
    which = sorted({0, streams - 1})
    es = {k: (oracle.Engine(15 + 4 * k), oracle.Gen()) for k in which}
    for pk in calls:
        n = pk * P
        out = g.generate(n * streams, 1, u).reshape(-1).cpu().numpy()
        for k in which:
            ref = oracle.generate(*es[k], kind, n, NPDT[tdt], a, b)
            got = out[k * n:(k + 1) * n]
            same = (got.view(U[tdt]) == ref.view(U[tdt])) | (np.isnan(got) & np.isnan(ref))
            assert same.all(), f"packets={pk} stream {k}: {np.nonzero(~same)[0][:5]}"
    u.sync()
    raw = er.raw_u64(u, 64 * streams).cpu().numpy().view(np.uint64)
    for k in which:
        assert np.array_equal(raw[64 * k:64 * (k + 1)], es[k][0].raw(16)), "engine after the calls"


def _ms(er, kind, a, b, n):
    u = er.Vmt19937_64(3)
    g = er._Gen(torch.float32, a, b, kind=kind)
    out = torch.empty(n, 1, dtype=torch.float32, device="cuda")
    times = []
    for _ in range(4):
        e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        e0.record()
        g.generate(n, 1, u, out=out)
        e1.record()
        torch.cuda.synchronize()
        times.append(e0.elapsed_time(e1))
    return min(times[1:])


@pytest.mark.parametrize("kind,a,b,a0,b0", [("GAMMA", 1e-6, 1.0, 0.5, 1.0), ("GAMMA", 1e-4, 1.0, 0.5, 1.0),
                                            ("BETA", 1e-4, 1e-4, 0.4, 0.7), ("BETA", 1e-5, 2.0, 0.5, 2.0),
                                            ("BETA", 1e-3, 2.0, 0.5, 2.0)])
def test_time(gpulib, kind, a, b, a0, b0):
    """One call of 2^21 floats on one engine against an ordinary shape's, whose
    trials are more."""
    assert _ms(gpulib, kind, a, b, 1 << 21) < 3 * _ms(gpulib, kind, a0, b0, 1 << 21)
