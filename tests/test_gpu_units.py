"""Fixed-unit kinds on many engines (k_units, gr_trials.cu) against the oracle,
bit for bit, over consecutive calls: units of one to nineteen packets and of odd
and even numbers of half packets, calls that end next to a block's last word, the
engine's cached half packet carried in and out."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

if not torch.cuda.is_available():
    pytest.skip("needs a CUDA GPU", allow_module_level=True)

CASES = [("GAMMA", torch.float32, 2.0, 1.5, 0), ("GAMMA", torch.float64, 5.0, 1.0, 0), ("GAMMA", torch.float32, 19.0, 1.0, 0),
         ("GAMMA", torch.float64, 19.0, 2.0, 0), ("STUDENT_T", torch.float32, 3.0, 0.0, 0),
         ("STUDENT_T", torch.float64, 4.5, 0.0, 0), ("BINOMIAL", torch.int32, 0.3, 0.0, 1),
         ("BINOMIAL", torch.int32, 0.7, 0.0, 2), ("BINOMIAL", torch.int32, 0.01, 0.0, 7),
         ("BINOMIAL", torch.int32, 0.5, 0.0, 20), ("BINOMIAL", torch.int32, 1.0, 0.0, 24),
         ("BINOMIAL", torch.int32, 0.0, 0.0, 3)]
NPDT = {torch.float32: np.float32, torch.float64: np.float64, torch.int32: np.int32}


@pytest.mark.parametrize("half", [False, True])
@pytest.mark.parametrize("case", CASES)
def test_many_engines(gpulib, oracle, case, half):
    er = gpulib
    kind, tdt, a, b, t = case
    K, P = 200, 8 if tdt == torch.float32 else 4
    U = t if kind == "BINOMIAL" else 2 if kind == "STUDENT_T" else int(a)
    block = 624 // U if kind == "BINOMIAL" else 312 // U  # units of a block
    u = er.Vmt19937_64(40, streams=K)
    g = er._Gen(tdt, a, b, trials=t, kind=kind)
    which = (0, 77, 199)
    es = {k: (oracle.Engine(40 + 4 * k), oracle.Gen()) for k in which}
    if half:
        er.randBits(4 * K, 1, u)
        for e, _ in es.values():
            oracle.generate(e, oracle.Gen(), "RANDBITS", 4, np.int32)
    for pk in (1, block - 1, 1, block, block + 1, 3, 5 * block + 2):
        if pk < 1:
            continue
        n = pk * P
        out = g.generate(n * K, 1, u).reshape(-1).cpu().numpy()
        for k in which:
            ref = oracle.generate(*es[k], kind, n, NPDT[tdt], a, b, t)
            bad = np.nonzero(out[k * n:(k + 1) * n].view(np.uint8) != ref.view(np.uint8))[0]
            assert bad.size == 0, f"{case} {pk} units, stream {k}: {bad[:3]}"
    u.sync()
    raw = er.raw_u64(u, 64 * K).cpu().numpy().view(np.uint64)
    for k in which:
        assert np.array_equal(raw[64 * k:64 * (k + 1)], es[k][0].raw(16)), "engine after the calls"
