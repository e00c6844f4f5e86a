"""Columns on both sides of the rule that sends them to the paired or the scalar form (line4 in fft4.cuh: the length, the
scalar split's larger factor, the direction, up to or above 64 x-points) and with the threads of a length whose three
stages need a warp more: 3D r2c / c2r against numpy float64 at the tolerance of the other transform tests."""
import math

import numpy as np
import pytest

from crava_b200 import api
from tests.test_gpu_rows import TOL_FFT, crel

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    c = api.Context(0)
    yield c
    c.close()


# 64 and 65 x-points of the half spectrum (and the widths of odd rows next to them)
@pytest.mark.parametrize("nxp", [126, 125, 128, 135])
@pytest.mark.parametrize("nyp", [180, 189, 192, 240, 250, 252, 256, 270, 280])
def test_columns_match_numpy(ctx, nxp, nyp):
    import torch
    nzp = 3
    rng = np.random.default_rng(nxp + 3 * nyp)
    x = rng.standard_normal((nzp, nyp, nxp)).astype(np.float32)
    g = torch.zeros((nzp, nyp, 2 * (nxp // 2 + 1)), dtype=torch.float32, device="cuda")
    g[..., :nxp] = torch.from_numpy(x).cuda()
    api.fft_r2c(ctx, g.data_ptr(), nxp, nyp, nzp, False)
    torch.cuda.synchronize()
    ref = np.fft.rfftn(x.astype(np.float64)) / math.sqrt(x.size)
    assert crel(g.cpu().numpy().view(np.complex64), ref) < TOL_FFT
    api.fft_c2r(ctx, g.data_ptr(), nxp, nyp, nzp, False)
    torch.cuda.synchronize()
    assert crel(g.cpu().numpy()[..., :nxp], x) < TOL_FFT


@pytest.mark.parametrize("nzp", [192, 250, 252, 256, 270])
def test_lines_in_depth_match_numpy(ctx, nzp):
    import torch
    nxp, nyp = 128, 4
    rng = np.random.default_rng(nzp)
    x = rng.standard_normal((nzp, nyp, nxp)).astype(np.float32)
    g = torch.zeros((nzp, nyp, nxp + 2), dtype=torch.float32, device="cuda")
    g[..., :nxp] = torch.from_numpy(x).cuda()
    api.fft_r2c(ctx, g.data_ptr(), nxp, nyp, nzp, False)
    torch.cuda.synchronize()
    ref = np.fft.rfftn(x.astype(np.float64)) / math.sqrt(x.size)
    assert crel(g.cpu().numpy().view(np.complex64), ref) < TOL_FFT
    api.fft_c2r(ctx, g.data_ptr(), nxp, nyp, nzp, False)
    torch.cuda.synchronize()
    assert crel(g.cpu().numpy()[..., :nxp], x) < TOL_FFT
