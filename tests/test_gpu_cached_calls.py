"""Calls that the cached half packet (engine) or half unit (generator object)
serves whole, so that k_direct makes no packet: many of them in turn with calls
that leave a half, on one engine and on many, outputs and the raw words
afterwards against the oracle."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

if not torch.cuda.is_available():
    pytest.skip("needs a CUDA GPU", allow_module_level=True)

# kind, type, values that a whole packet (unit) gives beyond the call's
CASES = [("BALANCED", torch.float64, 4), ("RANDBITS", torch.int32, 4), ("UNIFORM_INT", torch.int32, 4),
         ("GEOMETRIC", torch.int32, 4), ("NORMAL_STD", torch.float32, 8), ("NORMAL_STD", torch.float64, 4)]
NPDT = {torch.float32: np.float32, torch.float64: np.float64, torch.int32: np.int32}
ARGS = {"UNIFORM_INT": (0.0, 1023.0), "GEOMETRIC": (0.25, 0.0)}


@pytest.mark.parametrize("streams", [1, 608])
@pytest.mark.parametrize("kind,tdt,n", CASES)
def test_served_from_the_cache(gpulib, oracle, kind, tdt, n, streams):
    er = gpulib
    a, b = ARGS.get(kind, (0.0, 0.0))
    u = er.Vmt19937_64(52, streams=streams)
    g = er._Gen(tdt, a, b, kind=kind)
    which = sorted({0, streams // 3, streams - 1})
    es = {k: (oracle.Engine(52 + 4 * k), oracle.Gen()) for k in which}
    for call in range(200):
        out = g.generate(n * streams, 1, u).reshape(-1)
        if call % 20 < 2:
            got = out.cpu().numpy()
        for k in which:
            ref = oracle.generate(*es[k], kind, n, NPDT[tdt], a, b)
            if call % 20 < 2:
                assert np.array_equal(got[k * n:(k + 1) * n].view(np.uint8), ref.view(np.uint8)), f"call {call} stream {k}"
    raw = er.raw_u64(u, 64 * streams).cpu().numpy().view(np.uint64)
    for k in which:
        assert np.array_equal(raw[64 * k:64 * (k + 1)], es[k][0].raw(16)), f"words after the calls, stream {k}"
