"""The smoother of the facies histograms: the reference normalises it by a float sum in bin order, which
loses the tails; a unit histogram smoothed gives the smoother itself, against that sum restated with
numpy's sequential float32 accumulation.  Bin counts below one chunk of the device's sum (8192), a whole
number of chunks, and others; narrow and wide Gaussians (few bins that count, all of them).

Tolerance: the FP32 transforms of up to 500k bins give 1e-6 norm-wise, a differently rounded
exponential moves the float sum by about 1e-6 more; 2e-5 still tells the float sum from the exact
one where that is asked (they differ by more than 1e-4)."""
import numpy as np
import pytest

from crava_b200 import api

pytestmark = pytest.mark.gpu

TOL = 2e-5


def smoother32(nb, dv, S):
    cyc = lambda n: np.where(np.arange(n) <= n // 2, np.arange(n), np.arange(n) - n).astype(np.float64)
    j, k, l = cyc(nb[0])[None, None, :], cyc(nb[1])[None, :, None], cyc(nb[2])[:, None, None]
    f = j * dv[0] * j * dv[0] * S[0, 0] + k * dv[1] * k * dv[1] * S[1, 1] + l * dv[2] * l * dv[2] * S[2, 2] \
        + 2 * j * dv[0] * k * dv[1] * S[1, 0] + 2 * j * dv[0] * l * dv[2] * S[2, 0] + 2 * k * dv[1] * l * dv[2] * S[2, 1]
    v = np.exp((np.float32(-0.5) * f.astype(np.float32)).astype(np.float64)).astype(np.float32)
    return v, np.cumsum(v.reshape(-1), dtype=np.float32)[-1]


@pytest.mark.parametrize("nb,width,tails", [((100, 100, 50), 1.0, True), ((20, 16, 10), 1.0, False), ((15, 12, 9), 0.3, False),
                                            ((128, 64, 48), 2.0, False), ((81, 63, 35), 0.6, False)])
def test_smoother_keeps_the_float_sum(nb, width, tails):
    import torch
    dv = (0.7 / nb[0], 1.2 / nb[1], 0.5 / nb[2])
    sig = width * np.array([[0.003, 0.001, 0.0005], [0.001, 0.004, 0.0002], [0.0005, 0.0002, 0.001]])
    S = np.linalg.inv(sig)
    ctx = api.Context(0)
    rna = 2 * (nb[0] // 2 + 1)
    d = torch.zeros((2, nb[2], nb[1], rna), device="cuda")
    d[:, 0, 0, 0] = torch.tensor([1.0, 3.0], device="cuda")
    fd, _k = api.facies_desc([0.4, 0.6], nb, (7.9, 7.0, 7.7), dv, 0.05)
    api.facies_smooth(ctx, fd, S, d.data_ptr())
    torch.cuda.synchronize()
    got = d.cpu().numpy()[..., :nb[0]].astype(np.float64)
    v, total = smoother32(nb, dv, S)
    ref = v.astype(np.float64) / float(total)
    for f, scale in enumerate((1.0, 3.0)):
        assert np.linalg.norm(got[f] - scale * ref) / np.linalg.norm(scale * ref) < TOL
    if tails:
        assert abs(v.sum(dtype=np.float64) / float(total) - 1) > 1e-4
    ctx.close()
