"""crava_invert_noalloc on input grids that start one float off an 8-byte boundary: odd nxp asks for no more than
a float's alignment of its real inputs.  The same results as from aligned inputs, which are only read."""
import ctypes

import numpy as np
import pytest

from crava_b200 import api, synth
from tests.test_zz_no_alloc import _noalloc_fn

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dims", [(21, 8, 20), (35, 5, 24)])
def test_odd_rows_at_any_float(dims):
    import torch
    nx, ny, nz = dims
    blk = synth.make_block_fast(synth.BlockSpec(nx=nx, ny=ny, nz=nz, theta_deg=(10.0, 30.0), peak_hz=(30.0,) * 2,
                                                sn=(5.0,) * 2, nsim=1, seed=nx))
    desc, _k = api.make_desc(blk, api.PRIOR_SEPARABLE, 0, seed=7)
    grids = [np.ascontiguousarray(g) for g in (*blk.data, *blk.mean)]
    f, results = _noalloc_fn(), []
    for off in (0, 1, 3):
        d_in = []
        for g in grids:
            t = torch.zeros(g.size + 4, dtype=torch.float32, device="cuda")
            t[off:off + g.size] = torch.from_numpy(g.reshape(-1)).cuda()
            d_in.append(t)
        d_out = [torch.zeros(grids[0].shape, dtype=torch.float32, device="cuda") for _ in range(12)]
        ins = (ctypes.c_void_p * len(d_in))(*[t.data_ptr() + 4 * off for t in d_in])
        outs = (ctypes.c_void_p * len(d_out))(*[t.data_ptr() for t in d_out])
        st = f(ctypes.byref(desc), ins, outs, torch.cuda.current_stream().cuda_stream)
        assert st == api.OK, api.lib().crava_last_error()
        torch.cuda.synchronize()
        results.append([t.cpu().numpy() for t in d_out])
        for t, g in zip(d_in, grids):
            assert np.array_equal(t.cpu().numpy()[off:off + g.size], g.reshape(-1))
    for r in results[1:]:
        for a, b in zip(results[0], r):
            assert np.array_equal(a, b)
