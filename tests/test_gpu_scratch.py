"""The scratch that a context keeps between facies calls: bounded, and given back when an allocation finds no memory
(injected on the host: nothing is exhausted) and with the context."""
import numpy as np
import pytest

from crava_b200 import api, synth

pytestmark = pytest.mark.gpu


def facies_call(ctx, torch):
    nb, dims = (100, 100, 50), (64, 64, 32)
    fd, _k = api.facies_desc([0.5, 0.5], nb, (7.9, 7.0, 7.7), (0.007, 0.012, 0.01), 0.05)
    dens = torch.rand((2, nb[2], nb[1], 2 * (nb[0] // 2 + 1)), device="cuda")
    mean = torch.full((3, dims[2], dims[1], 2 * (dims[0] // 2 + 1)), 8.0, device="cuda")
    out = torch.empty((3,) + mean.shape[1:], device="cuda")
    api.facies_prob(ctx, fd, dens.data_ptr(), dens.shape[3], [m.data_ptr() for m in mean], *dims, dims[0], dims[1],
                    [o.data_ptr() for o in out])
    torch.cuda.synchronize()


def test_kept_scratch_gives_way():
    import torch
    ctx = api.Context(0)
    facies_call(ctx, torch)
    facies_call(ctx, torch)
    kept = torch.cuda.mem_get_info()[0]
    api._check(api.lib().crava_ctx_fail_next_allocs(ctx.handle, 1))
    blk = synth.make_block_fast(synth.BlockSpec(nx=8, ny=8, nz=16, theta_deg=(10.0,), peak_hz=(30.0,), sn=(5.0,), nsim=0))
    with pytest.raises(api.CravaError):
        api.Job(ctx, blk, api.PRIOR_SEPARABLE)
    # 500 000 bins of 16 bytes at least were kept, and are free again
    assert torch.cuda.mem_get_info()[0] - kept >= 16 * 500_000
    facies_call(ctx, torch)                   # and the scratch comes back
    ctx.close()
