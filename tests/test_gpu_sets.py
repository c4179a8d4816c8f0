"""GammaGen<float> parameter sets (k_gamma_sets, gr_trials.cu) against the
oracle, bit for bit: more sets than the resident grid takes at once, sets of
several engine blocks and batches, counts around a packet, empty sets, every
branch of the shape."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

if not torch.cuda.is_available():
    pytest.skip("needs a CUDA GPU", allow_module_level=True)

# GS, exponential, product of uniforms (1 to 19 packets a trial), tan
SHAPES = [0.5, 1.0, 2.0, 19.0, 1.5, 20.0, 0.02, 0.99, 5.0, 300.0]


def check(er, oracle, counts, a, seed, which):
    b = np.linspace(0.5, 2.0, len(counts)).astype(np.float32)
    out, off = er.sample_batched("GAMMA", torch.from_numpy(counts), torch.from_numpy(a), torch.from_numpy(b), None, seed=seed)
    torch.cuda.synchronize()
    out, off = out.cpu().numpy(), off.cpu().numpy()
    for i in which:
        ref = oracle.vop_set(seed + 4 * int(i), "GAMMA", int(counts[i]), float(a[i]), float(b[i]), 0)
        got = out[off[i]:off[i] + counts[i]]
        bad = np.nonzero(got.view(np.uint32) != ref.view(np.uint32))[0]
        assert bad.size == 0, f"set {i} (alpha {a[i]}, {counts[i]} values): {bad[:5]}"


@pytest.mark.parametrize("shape", SHAPES)
def test_sizes(gpulib, oracle, shape):
    counts = np.array([1, 7, 8, 9, 2495, 2496, 2497, 1280, 1281, 0, 20000, 3], np.int32)
    check(gpulib, oracle, counts, np.full(len(counts), shape, np.float32), 31, [i for i in range(len(counts)) if counts[i]])


def test_more_sets_than_the_grid(gpulib, oracle):
    n = 1500
    counts = (np.arange(n) % 97 * 9).astype(np.int32)
    a = np.array(SHAPES, np.float32)[np.arange(n) % len(SHAPES)]
    check(gpulib, oracle, counts, a, 5, [i for i in range(0, n, 7) if counts[i]])
