"""Calls on few engines take one scratch allocation, before their first launch;
where there is none to be had they take the path that needs none.  Sequences of
calls of which one, each in turn, finds no scratch (GR_SCRATCH_FAIL), and one in
which none does: outputs and the raw words afterwards against the oracle."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

if not torch.cuda.is_available():
    pytest.skip("needs a CUDA GPU", allow_module_level=True)

NPDT = {torch.float32: np.float32, torch.float64: np.float64, torch.int32: np.int32}
CASES = [("UNIFORM_REAL", torch.float32, 0.0, 0.0, 0), ("NORMAL_STD", torch.float64, 0.0, 0.0, 0),
         ("BALANCED", torch.float64, 0.0, 0.0, 0), ("GAMMA", torch.float32, 5.0, 1.0, 0),
         ("BINOMIAL", torch.int32, 0.3, 0.0, 20), ("GAMMA", torch.float64, 0.5, 1.0, 0),
         ("POISSON", torch.int32, 100.0, 0.0, 0), ("POISSON", torch.int32, 4.0, 0.0, 0),
         ("BETA", torch.float32, 0.5, 2.0, 0), ("BETA", torch.float64, 2.5, 1.5, 0)]
CALLS = {1: (3001, 640, 140001, 2600), 20: (3001, 640, 2601)}  # packets per engine


@pytest.mark.parametrize("streams", [1, 20])
@pytest.mark.parametrize("case", CASES)
def test_no_scratch_for_one_call(gpulib, oracle, monkeypatch, case, streams):
    er = gpulib
    kind, tdt, a, b, t = case
    P = 8 if tdt == torch.float32 else 4
    calls = CALLS[streams]
    which = sorted({0, streams - 1})
    es = {k: (oracle.Engine(70 + 4 * k), oracle.Gen()) for k in which}
    refs = [{k: oracle.generate(*es[k], kind, pk * P, NPDT[tdt], a, b, t) for k in which} for pk in calls]
    words = {k: es[k][0].raw(16) for k in which}
    for bad in list(range(len(calls))) + [None]:
        u = er.Vmt19937_64(70, streams=streams)
        g = er._Gen(tdt, a, b, trials=t, kind=kind)
        for i, pk in enumerate(calls):
            if i == bad or bad is None:
                monkeypatch.setenv("GR_SCRATCH_FAIL", "1")
            else:
                monkeypatch.delenv("GR_SCRATCH_FAIL", raising=False)
            n = pk * P
            out = g.generate(n * streams, 1, u).reshape(-1).cpu().numpy()
            for k in which:
                assert np.array_equal(out[k * n:(k + 1) * n].view(np.uint8), refs[i][k].view(np.uint8)), \
                    f"{case} call {i} (no scratch: {bad}) stream {k}"
        monkeypatch.delenv("GR_SCRATCH_FAIL", raising=False)
        u.sync()
        raw = er.raw_u64(u, 64 * streams).cpu().numpy().view(np.uint64)
        for k in which:
            assert np.array_equal(raw[64 * k:64 * (k + 1)], words[k]), f"words after the calls, stream {k}"
