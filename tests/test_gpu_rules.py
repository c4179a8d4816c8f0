"""Calls just below, at and above the sizes from which a kind goes through words
in memory (gr_api.cu: words_from, units_from, reject_from, poisson_from,
chain_from), in consecutive calls of one generator object, on one engine and on
engine counts next to where a rule ends: against the oracle, bit for bit."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

if not torch.cuda.is_available():
    pytest.skip("needs a CUDA GPU", allow_module_level=True)

f32, f64, i32 = torch.float32, torch.float64, torch.int32
NPDT = {f32: np.float32, f64: np.float64, i32: np.int32}
# kind, type, a, b, trials, {engines: the largest size that the one-CTA path takes, output packets}
CASES = [
    ("UNIFORM_REAL", f32, 0, 0, 0, {1: 5180, 64: 16520}), ("UNIFORM_REAL", f64, 0, 0, 0, {1: 3664}),
    ("BALANCED", f64, 0, 0, 0, {1: 2 * 1516}), ("RANDBITS", i32, 0, 0, 0, {1: 2 * 5180}),
    ("NORMAL_STD", f32, 0, 0, 0, {1: 1516, 127: 3532}), ("NORMAL_STD", f64, 0, 0, 0, {1: 452, 127: 767}),
    ("GAMMA", f32, 2, 1, 0, {1: 525, 128: 1600}), ("GAMMA", f64, 5, 1, 0, {1: 220, 128: 400}),
    ("STUDENT_T", f64, 4, 0, 0, {1: 165}), ("BINOMIAL", i32, 0.3, 0, 20, {1: 320, 96: 690}),
    ("BINOMIAL", i32, 0.3, 0, 1, {1: 2760}), ("GAMMA", f32, 0.5, 1, 0, {1: 1000, 192: 4072}),
    ("GAMMA", f64, 0.5, 1, 0, {1: 600, 256: 1910}), ("GAMMA", f64, 2.5, 1, 0, {1: 430}),
    ("BETA", f32, 0.4, 0.7, 0, {1: 1300}), ("POISSON", i32, 100, 0, 0, {1: 1000}), ("BINOMIAL", i32, 0.3, 0, 100, {1: 560}),
    ("POISSON", i32, 4, 0, 0, {1: 710, 256: 1065}), ("POISSON", i32, 0.5, 0, 0, {1: 3406}),
    ("BETA", f32, 0.5, 2, 0, {1: 520, 192: 1780}), ("BETA", f64, 0.5, 2, 0, {1: 452}), ("BETA", f32, 0.5, 1, 0, {1: 405}),
    ("BETA", f32, 2.5, 1.5, 0, {1: 53, 256: 125}), ("BETA", f64, 2.5, 1.5, 0, {1: 53}), ("BETA", f32, 3, 2.5, 0, {1: 145}),
    ("BETA", f32, 1, 3, 0, {1: 75})]


@pytest.mark.parametrize("kind,tdt,a,b,t,at", CASES)
def test_around_the_rule(gpulib, oracle, kind, tdt, a, b, t, at):
    er = gpulib
    P = 8 if tdt == f32 else 4
    for streams, edge in at.items():
        u = er.Vmt19937_64(23, streams=streams)
        g = er._Gen(tdt, a, b, trials=t, kind=kind)
        which = sorted({0, streams - 1})
        es = {k: (oracle.Engine(23 + 4 * k), oracle.Gen()) for k in which}
        for pk in (edge, edge + 1, edge - 1, edge + 2, 1, edge * 9 // 10, edge * 11 // 10, edge * 21 // 20, edge * 19 // 20):
            n = pk * P
            out = g.generate(n * streams, 1, u).reshape(-1).cpu().numpy()
            for k in which:
                ref = oracle.generate(*es[k], kind, n, NPDT[tdt], a, b, t)
                assert np.array_equal(out[k * n:(k + 1) * n].view(np.uint8), ref.view(np.uint8)), \
                    f"{streams} engines, packets={pk}, stream {k}"
        u.sync()
        raw = er.raw_u64(u, 64 * streams).cpu().numpy().view(np.uint64)
        for k in which:
            assert np.array_equal(raw[64 * k:64 * (k + 1)], es[k][0].raw(16)), "words after the calls"
