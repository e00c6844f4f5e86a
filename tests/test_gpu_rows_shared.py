"""Rows of odd length share a complex line with their neighbour: a zero or tiny row beside a large one is
told apart from it to the transforms' rounding of the large one (TOL_FFT of test_gpu_rows.py, row by row)."""
import math

import numpy as np
import pytest

from crava_b200 import api
from tests.test_gpu_rows import TOL_FFT

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    c = api.Context(0)
    yield c
    c.close()


# splits with and without a factor above 24, an odd and an even number of rows; the large rows first or second of
# their pair
@pytest.mark.parametrize("nxp", [21, 105, 125, 243, 729])
@pytest.mark.parametrize("dims", [(2, 2), (4, 2), (5, 3)])
@pytest.mark.parametrize("small", [0.0, 1e-6])
@pytest.mark.parametrize("first", [0, 1])
def test_small_row_beside_a_large_one(ctx, nxp, dims, small, first):
    import torch
    nyp, nzp = dims
    rng = np.random.default_rng(nxp + nyp)
    amp = np.where((np.arange(nyp * nzp) + first) % 2 == 0, 1e3, small).reshape(nzp, nyp, 1)
    x = (rng.standard_normal((nzp, nyp, nxp)) * amp).astype(np.float32)
    g = torch.zeros((nzp, nyp, nxp + 1), dtype=torch.float32, device="cuda")
    g[..., :nxp] = torch.from_numpy(x).cuda()
    api.fft_r2c(ctx, g.data_ptr(), nxp, nyp, nzp, False)
    torch.cuda.synchronize()
    spec = g.cpu().numpy().view(np.complex64)
    ref = np.fft.rfftn(x.astype(np.float64)) / math.sqrt(x.size)
    assert np.linalg.norm(spec - ref) < TOL_FFT * np.linalg.norm(ref)
    api.fft_c2r(ctx, g.data_ptr(), nxp, nyp, nzp, False)
    torch.cuda.synchronize()
    err = np.linalg.norm(g.cpu().numpy()[..., :nxp].astype(np.float64) - x, axis=-1)
    assert err.max() < TOL_FFT * np.linalg.norm(x, axis=-1).max()
