"""Calls on few engines whose raw words go through memory (k_words_wide /
k_words_warp, k_xform): lengths around the thresholds, around the 156-word
phases, the 48-phase exchanges and the jump-ahead segments, odd packet counts
with caches carried to the next call, several engines, and a call longer than
one scratch buffer, all bit for bit against the oracle."""
import ctypes

import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

if not torch.cuda.is_available():
    pytest.skip("needs a CUDA GPU", allow_module_level=True)


def bits(x):
    return x.view(np.uint64 if x.itemsize == 8 else np.uint32)


@pytest.mark.parametrize("streams", [1, 3])
@pytest.mark.parametrize("kind,tdt", [("NORMAL_STD", torch.float32), ("NORMAL_STD", torch.float64),
                                      ("BALANCED", torch.float64), ("UNIFORM_REAL", torch.float32),
                                      ("RANDBITS", torch.int32), ("EXPONENTIAL", torch.float64)])
def test_lengths_and_caches(gpulib, oracle, kind, tdt, streams):
    er = gpulib
    npdt = {torch.float32: np.float32, torch.float64: np.float64, torch.int32: np.int32}[tdt]
    P = 8 if tdt == torch.float32 else 4
    u = er.Vmt19937_64(321, streams=streams)
    g = er._Gen(tdt, kind=kind)
    es = [oracle.Engine(321 + 4 * k) for k in range(streams)]
    ogs = [oracle.Gen() for _ in range(streams)]
    for pk in (157, 311, 625, 2561, 48 * 156 + 1, 48 * 156 * 2 + 155, 7, 40001, 131072 + 3):
        n = pk * P
        out = g.generate(n * streams, 1, u).reshape(-1).cpu().numpy()
        for k in range(streams):
            ref = oracle.generate(es[k], ogs[k], kind, n, npdt)
            assert np.array_equal(bits(out[k * n:(k + 1) * n]), bits(ref)), f"{kind} {tdt} packets={pk} stream {k}"


@pytest.mark.parametrize("streams", [1, 5, 127])
def test_raw_segments(gpulib, oracle, streams):
    """Jump-ahead segments of several lengths, the last one short, and enough
    engines for the warp form of the word kernel."""
    er = gpulib
    u = er.Vmt19937_64(9, streams=streams)
    es = [oracle.Engine(9 + 4 * k) for k in range(streams)]
    for pk in (1 << 19, (1 << 18) + 1) if streams == 1 else (20001, 30002):
        got = er.raw_u64(u, 4 * pk * streams).cpu().numpy().view(np.uint64)
        for k in range(streams):
            ref = es[k].raw(pk)
            if k in (0, streams // 2, streams - 1):
                assert np.array_equal(got[4 * pk * k:4 * pk * (k + 1)], ref), f"packets={pk} stream {k}"


def test_more_than_one_buffer(gpulib, oracle):
    er = gpulib
    u = er.Vmt19937_64(77)
    e = oracle.Engine(77)
    pk = (1 << 22) + 12345
    got = er.raw_u64(u, 4 * pk).cpu().numpy().view(np.uint64)
    assert np.array_equal(got, e.raw(pk))
    assert np.array_equal(er.raw_u64(u, 64).cpu().numpy().view(np.uint64), e.raw(16))


@pytest.mark.parametrize("kind,tdt,a,t", [("GAMMA", torch.float32, 5.0, 0), ("GAMMA", torch.float64, 19.0, 0),
                                          ("STUDENT_T", torch.float32, 4.0, 0), ("STUDENT_T", torch.float64, 2.5, 0),
                                          ("BINOMIAL", torch.int32, 0.3, 20), ("BINOMIAL", torch.int32, 0.3, 1),
                                          ("BINOMIAL", torch.int32, 0.9, 7)])
@pytest.mark.parametrize("streams", [1, 3])
def test_units_of_packets(gpulib, oracle, kind, tdt, a, t, streams):
    """Kinds whose output takes a fixed run of packets (k_staged_words): around
    the threshold, with half packets carried (binomial), and in several
    scratch buffers."""
    er = gpulib
    npdt = {torch.float32: np.float32, torch.float64: np.float64, torch.int32: np.int32}[tdt]
    P = 8 if tdt == torch.float32 else 4
    u = er.Vmt19937_64(12, streams=streams)
    g = er._Gen(tdt, a, 1.0 if kind == "GAMMA" else 0.0, trials=t, kind=kind)
    es = [oracle.Engine(12 + 4 * k) for k in range(streams)]
    og = oracle.Gen()
    U = {"GAMMA": int(a), "STUDENT_T": 2, "BINOMIAL": max(1, (t + 1) // 2)}[kind]
    for un in (624 // U, 624 // U + 1, 701, 3, 20001) + ((1 << 22) // U + 77,) * (streams == 1):
        n = un * P
        out = g.generate(n * streams, 1, u).reshape(-1).cpu().numpy()
        for k in range(streams):
            ref = oracle.generate(es[k], og, kind, n, npdt, a, 1.0 if kind == "GAMMA" else 0.0, t)
            assert np.array_equal(bits(out[k * n:(k + 1) * n]), bits(ref)), f"{kind} units={un} stream {k}"
    raw = er.raw_u64(u, 64 * streams).cpu().numpy().view(np.uint64)
    for k in range(streams):
        assert np.array_equal(raw[64 * k:64 * (k + 1)], es[k].raw(16)), "engine after the calls"
