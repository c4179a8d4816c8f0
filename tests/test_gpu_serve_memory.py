"""The serving loop's device memory: results and the scratch of the calls come from
the server's pool and stay within its budget, also where one request's scratch
alone would not fit, and nothing outside the pool grows with the requests; the
results are those of plain calls."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

if not torch.cuda.is_available():
    pytest.skip("needs a CUDA GPU", allow_module_level=True)

MB = 1 << 20
KINDS = [("BETA", torch.float64, 0.5, 2.0, 0), ("GAMMA", torch.float32, 0.5, 1.0, 0), ("NORMAL", torch.float32, 0.0, 1.0, 0),
         ("POISSON", torch.int32, 4.0, 0.0, 0), ("GAMMA", torch.float64, 5.0, 1.0, 0), ("BINOMIAL", torch.int32, 0.3, 0.0, 100),
         ("BETA", torch.float32, 2.5, 1.5, 0), ("NORMAL", torch.float64, 1.0, 2.0, 0)]


@pytest.mark.parametrize("budget", [4 * MB, 12 * MB, 64 * MB])
def test_within_the_budget(gpulib, budget):
    er = gpulib
    from eigenrand_gb300.serving import Server
    slots, seeds = 6, list(range(300, 308))
    plain = [er.Vmt19937_64(s) for s in seeds]
    refs = {}
    for i in range(3):
        for c, (kind, dt, a, b, t) in enumerate(KINDS):
            n = 100000 + 40000 * i
            refs[c, i] = er._sample(kind, n, 1, plain[c], dt, a, b, t).reshape(-1).cpu().numpy()
    del plain
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    srv = Server(len(seeds), seeds, budget, slots=slots)
    free = torch.cuda.mem_get_info()[0]
    tickets = {srv.submit(c, kind, dt, 100000 + 40000 * i, a, b, t): (c, i)
               for i in range(3) for c, (kind, dt, a, b, t) in enumerate(KINDS)}
    done = 0
    while done < len(tickets):
        for x in srv.progress():
            assert x["status"] == 0
            got = srv.read(x["ticket"], x["count"])
            ref = refs[tickets[x["ticket"]]]
            assert np.array_equal(got.view(np.uint8), ref.view(np.uint8)), tickets[x["ticket"]]
            srv.release(x["ticket"])
            done += 1
        assert srv.pending()[2] <= budget
    assert srv.pending() == (0, 0, 0)
    # the pool rounds every allocation up (512 bytes); a request has two
    assert 0 < srv.memory() <= budget + 2 * slots * 512
    # what the pool keeps: its blocks are of 32 MiB, and fragments count
    assert free - torch.cuda.mem_get_info()[0] <= budget + 64 * MB


def test_large_requests_do_not_grow_the_library(gpulib):
    """Eight large requests at a time: their scratch, some 100 MB each if it may be had,
    is inside the budget."""
    er = gpulib
    from eigenrand_gb300.serving import Server
    torch.cuda.empty_cache()
    budget = 200 * MB
    srv = Server(8, list(range(8)), budget, slots=8)
    free = torch.cuda.mem_get_info()[0]
    for c in range(8):
        srv.submit(c, "BETA", torch.float64, 1 << 20, 0.5, 2.0)
    done = 0
    while done < 8:
        for x in srv.progress():
            assert x["status"] == 0
            srv.release(x["ticket"])
            done += 1
    assert srv.memory() <= budget + 16 * 512
    assert free - torch.cuda.mem_get_info()[0] <= budget + 64 * MB
