"""Density volumes are packed in pairs of cells while they then take 8 to 256 MB, and one by one below and beyond: a large
volume and its crops, all with the bins that the parameters reach, lie in different layouts and give the same bits, in
both kernels (up to four facies, more) and with corner volumes, from below the first bin centre on."""
import numpy as np
import pytest

from crava_b200 import api

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nf", [1, 3, 4, 6])
@pytest.mark.parametrize("nang", [0, 1])
def test_layouts_agree(nf, nang):
    import torch
    ctx = api.Context(0)
    nx, ny, nz = 45, 12, 10
    row = 2 * (nx // 2 + 1)
    rng = np.random.default_rng(nf + 10 * nang)
    big, mid, crop = (300, 200, 150), (128, 64, 64), (31, 20, 9)   # 288 MB, 17 to 67 MB and 0.2 to 0.7 MB in pairs
    d_big = [torch.rand((nf, big[2], big[1], big[0]), device="cuda") for _ in range(1 << nang)]
    d_mid, d_crop = [[d[:, :n[2], :n[1]].contiguous() for d in d_big] for n in (mid, crop)]
    post = torch.from_numpy(np.stack([rng.uniform(-1.0, n - 1.0, (nz, ny, row)) for n in crop]).astype(np.float32)).cuda()
    scale = rng.uniform(1.0, 2.0, (nang, ny, nx)).astype(np.float32) if nang else np.zeros(0, np.float32)
    res = []
    for nb, dens in ((big, d_big), (mid, d_mid), (crop, d_crop)):
        fds = [api.facies_desc([1.0 / nf] * nf, nb, (0.0, 0.0, 0.0), (1.0, 1.0, 1.0), 0.0) for _ in dens]
        out = torch.zeros((nf + 2, nz, ny, row), device="cuda")
        api.facies_prob_local_noise(ctx, [f[0] for f in fds], [d.data_ptr() for d in dens], big[0], scale,
                                    [x.data_ptr() for x in post], nx, ny, nz, nx, ny,
                                    [o.data_ptr() for o in out[:nf + 1]], out[nf + 1].data_ptr())
        torch.cuda.synchronize()
        res.append(out.cpu().numpy())
    assert np.array_equal(res[0], res[1]) and np.array_equal(res[0], res[2])
    assert np.all(res[0][nf + 1, ..., :nx] > 0)
    ctx.close()
