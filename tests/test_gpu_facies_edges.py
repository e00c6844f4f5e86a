"""Facies probabilities at the edges of their arithmetic, in both kernels (up to four facies in registers, more in
the general form): quotients below the normal range rounded as IEEE division rounds them, voxels exactly on
a bin centre beside a cell that must not count, parameters that are not finite, axes of one bin, and shapes
of few long or many short rows."""
import numpy as np
import pytest

from crava_b200 import api

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    c = api.Context(0)
    yield c
    c.close()


def prob(ctx, dens, vmin, dv, prior, undef, post):
    """dens (nf, nb2, nb1, nb0), post (3, nz, ny, nx) -> probabilities (nf + 1, nz, ny, nx), likelihood."""
    import torch
    nf, nb = dens.shape[0], dens.shape[:0:-1]
    _, nz, ny, nx = post.shape
    row = 2 * (nx // 2 + 1)
    fd, _k = api.facies_desc(list(prior), nb, vmin, dv, undef)
    d = torch.from_numpy(np.ascontiguousarray(dens, dtype=np.float32)).cuda()
    g = torch.zeros((3, nz, ny, row), device="cuda")
    g[..., :nx] = torch.from_numpy(np.ascontiguousarray(post, dtype=np.float32)).cuda()
    out = torch.zeros((nf + 2, nz, ny, row), device="cuda")
    api.facies_prob_local_noise(ctx, [fd], [d.data_ptr()], nb[0], np.zeros(0, np.float32),
                                [x.data_ptr() for x in g], nx, ny, nz, nx, ny, [o.data_ptr() for o in out[:nf + 1]],
                                out[nf + 1].data_ptr())
    torch.cuda.synchronize()
    o = out.cpu().numpy()
    assert np.all(o[..., nx:] == np.float32(-99999.0))
    return o[:nf + 1, ..., :nx], o[nf + 1, ..., :nx]


UNIT = ((0.0, 0.0, 0.0), (1.0, 1.0, 1.0))       # bin i has its centre at i + 1/2, exactly


@pytest.mark.parametrize("nf", [3, 6])
def test_tiny_probabilities_are_divided(ctx, nf):
    """Densities of 1e-45 to 1e-37 beside one of order one: the probabilities val / sum equal numpy's, bit for bit."""
    rng = np.random.default_rng(nf)
    nb = (16, 16, 16)
    dens = np.exp2(rng.uniform(-149, -125, (nf,) + nb)).astype(np.float32)
    dens[0] = rng.uniform(0.5, 3.0, nb).astype(np.float32)
    k, j, i = np.meshgrid(*[np.arange(16)] * 3, indexing="ij")
    post = np.stack([i, j, k]).astype(np.float32) + np.float32(0.5)
    prior = np.ones(nf, dtype=np.float32)
    p, lh = prob(ctx, dens, *UNIT, prior, 0.02, post)
    assert np.all(lh > 0.5)
    for f in range(nf):
        assert np.array_equal(p[f], dens[f] / lh), f


def test_bin_centre_beside_an_infinite_cell(ctx):
    """A bin width whose reciprocal is rounded: where (v - vmin) / dv is exactly a centre, the pair of cells begins at
    that centre with weight zero for the next one; the cell before it, infinite here, must not enter."""
    dv = np.float64(0.7) / 100
    i = np.arange(2, 100)
    # parameters whose distance over the width is exactly i + 1/2, but whose product with the reciprocal is less
    v = ((i + 0.5) * dv).astype(np.float32)
    vmin = v.astype(np.float64) - (i + 0.5) * dv        # one volume per value: vmin makes the distance exact
    bad = [(a, b, n) for a, b, n in zip(v, vmin, i)
           if (np.float64(a) - b) / dv - 0.5 == n and np.floor((np.float64(a) - b) * (1.0 / dv) - 0.5) == n - 1]
    assert bad
    for a, b, n in bad[:4]:
        dens = np.ones((2, 1, 1, 100), dtype=np.float32)
        dens[0, 0, 0, n] = 0.25
        dens[0, 0, 0, n - 1] = np.inf
        post = np.zeros((3, 1, 1, 5), dtype=np.float32)
        post[0] = a
        p, lh = prob(ctx, dens, (float(b), 0.0, 0.0), (float(dv), 1.0, 1.0), [0.5, 0.5], 0.02, post)
        assert np.all(np.isfinite(lh)) and np.all(p[0] == np.float32(0.125) / lh), (a, b, n)


@pytest.mark.parametrize("nf", [2, 5])
@pytest.mark.parametrize("nb", [(1, 8, 4), (8, 1, 4), (8, 8, 1), (1, 1, 1)])
def test_one_bin_axes_and_values_that_are_not_finite(ctx, nf, nb):
    """One-bin axes use their bin everywhere; infinite parameters the edge bins; a NaN parameter the first."""
    rng = np.random.default_rng(sum(nb) + nf)
    dens = rng.uniform(0.1, 1.0, (nf, nb[2], nb[1], nb[0])).astype(np.float32)
    vals = np.array([-np.inf, -3.0, 0.5, 1.25, 3.5, 100.0, np.inf, np.nan], dtype=np.float32)
    a, b, c = np.meshgrid(vals, vals, vals, indexing="ij")
    post = np.stack([a, b, c])
    prior = rng.uniform(0.2, 1.0, nf).astype(np.float32)
    p, lh = prob(ctx, dens, *UNIT, prior, 0.02, post)

    def axis(v, n):
        f = v.astype(np.float64) - 0.5
        i = np.where(np.isnan(f), -1, np.floor(np.clip(f, -2, n + 2))).astype(int)
        edge = (i < 0) | (i >= n - 1)
        lo = np.where(i < 0, 0, np.where(i >= n - 1, n - 1, i))
        return lo, np.where(edge, lo, lo + 1), np.where(edge, 0.0, np.nan_to_num(f, posinf=0, neginf=0) - i)

    ax = [axis(post[d], nb[d]) for d in range(3)]
    val = []
    for f in range(nf):
        s = 0.0
        for x in (0, 1):
            for y in (0, 1):
                for z in (0, 1):
                    w = 1.0
                    for d, h in enumerate((x, y, z)):
                        w = w * (ax[d][2] if h else 1.0 - ax[d][2])
                    s = s + w * dens[f][ax[2][z], ax[1][y], ax[0][x]].astype(np.float64)
        val.append(float(prior[f]) * s)
    tot = 0.02 / float(np.prod(nb)) + sum(val)
    # float32 products and sums of eight terms: 1e-6
    assert np.max(np.abs(lh - tot) / tot) < 2e-6
    for f in range(nf):
        assert np.max(np.abs(p[f] - val[f] / tot)) < 2e-6, f


@pytest.mark.parametrize("nf", [3, 6])
@pytest.mark.parametrize("dims", [(1000, 2, 3), (301, 1, 1), (2, 70, 90), (31, 9, 1), (33, 1, 300)])
def test_rows_of_every_length(ctx, dims, nf):
    """Few long rows are shared by warps, short ones leave lanes idle: every voxel once, none beyond."""
    nx, ny, nz = dims
    rng = np.random.default_rng(nx + nf)
    dens = rng.uniform(0.1, 1.0, (nf, 4, 4, 4)).astype(np.float32)
    cell = rng.integers(0, 4, (3, nz, ny, nx))
    p, lh = prob(ctx, dens, *UNIT, np.ones(nf, np.float32), 0.0, cell.astype(np.float32) + np.float32(0.5))
    at = dens[:, cell[2], cell[1], cell[0]]
    tot = at.astype(np.float64).sum(axis=0)
    assert np.max(np.abs(lh - tot) / tot) < 2e-6
    assert np.max(np.abs(p[:nf] - at / tot)) < 2e-6
