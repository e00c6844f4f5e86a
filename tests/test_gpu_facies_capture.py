"""crava_facies_prob under stream capture: the first facies call of a context, captured, replays to the direct call's
probabilities bit by bit (one volume has no host table to wait for, so the call does not synchronise)."""
import numpy as np
import pytest

from crava_b200 import api

pytestmark = pytest.mark.gpu


def test_first_call_of_a_context_can_be_captured():
    import torch
    nx, ny, nz, nb, nf = 45, 7, 12, (12, 10, 6), 3
    rng = np.random.default_rng(5)
    mean = torch.from_numpy(rng.uniform(0.05, 0.95, (3, nz, ny, 2 * (nx // 2 + 1))).astype(np.float32)).cuda()
    dens = torch.from_numpy(rng.uniform(0.0, 1.0, (nf, nb[2], nb[1], nb[0])).astype(np.float32)).cuda()
    fd, keep = api.facies_desc(np.array([0.2, 0.3, 0.5], np.float32), nb, [0.0] * 3, [1.0 / n for n in nb], 0.02)
    prob = torch.zeros((nf + 1, nz, ny, 2 * (nx // 2 + 1)), device="cuda")
    ctx = api.Context(0)

    def call(stream):
        api.facies_prob(ctx, fd, dens.data_ptr(), nb[0], [t.data_ptr() for t in mean], nx, ny, nz, nx, ny,
                        [t.data_ptr() for t in prob], stream=stream)

    s = torch.cuda.Stream()
    s.wait_stream(torch.cuda.current_stream())
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=s):
        call(s.cuda_stream)
    for _ in range(2):
        prob.fill_(7.0)
        torch.cuda.synchronize()
        graph.replay()
        torch.cuda.synchronize()
        got = prob.clone()
    prob.fill_(3.0)
    call(torch.cuda.current_stream().cuda_stream)
    torch.cuda.synchronize()
    assert torch.equal(got, prob)
    assert float(got[:nf].max()) > 0.0
    del graph
    ctx.close()
