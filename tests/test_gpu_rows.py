"""The x transforms of staged row chunks at the sizes where they can go wrong: odd lengths (two
rows per complex line) with an odd number of rows, a single short last chunk, and grids that start
off a 16-byte boundary (8-byte copies instead of 16-byte ones and the bulk copy); 3D r2c / c2r
against numpy float64 at the tolerance of the other transform tests, and the words around the
grid untouched."""
import math

import numpy as np
import pytest

from crava_b200 import api

pytestmark = pytest.mark.gpu

TOL_FFT = 2e-6


def crel(x, ref):
    x = np.asarray(x, dtype=np.complex128)
    ref = np.asarray(ref, dtype=np.complex128)
    return float(np.linalg.norm(x - ref) / max(np.linalg.norm(ref), 1e-300))


@pytest.fixture(scope="module")
def ctx():
    c = api.Context(0)
    yield c
    c.close()


# odd lengths of the smallest, short-factor, square and largest splits; even ones (half length
# 125 = 25 x 5, 16 = 4 x 4, 135, 512); 15 or 35 rows and rows that fill no whole chunk
@pytest.mark.parametrize("dims", [(21, 5, 3), (25, 3, 5), (105, 5, 7), (125, 7, 5), (225, 9, 25), (243, 5, 3),
                                  (729, 3, 5), (250, 5, 3), (32, 27, 5), (270, 7, 5), (1024, 3, 3)])
@pytest.mark.parametrize("off", [0, 2])
def test_rows_match_numpy(ctx, dims, off):
    import torch
    nxp, nyp, nzp = dims
    rnxp = 2 * (nxp // 2 + 1)
    n = nzp * nyp * rnxp
    rng = np.random.default_rng(nxp + 5 * nyp + 11 * nzp + off)
    x = rng.standard_normal((nzp, nyp, nxp)).astype(np.float32)
    buf = torch.full((n + off + 6,), 7.0, dtype=torch.float32, device="cuda")
    g = buf[off:off + n].view(nzp, nyp, rnxp)
    g[..., :nxp] = torch.from_numpy(x).cuda()
    api.fft_r2c(ctx, g.data_ptr(), nxp, nyp, nzp, False)
    torch.cuda.synchronize()
    spec = g.cpu().numpy().view(np.complex64)
    ref = np.fft.rfftn(x.astype(np.float64)) / math.sqrt(nxp * nyp * nzp)
    assert crel(spec, ref) < TOL_FFT
    api.fft_c2r(ctx, g.data_ptr(), nxp, nyp, nzp, False)
    torch.cuda.synchronize()
    out = g.cpu().numpy()
    assert crel(out[..., :nxp], x) < TOL_FFT
    assert np.all(out[..., nxp:] == 0.0)
    edge = buf.cpu().numpy()
    assert np.all(edge[:off] == 7.0) and np.all(edge[off + n:] == 7.0)
