"""The pencil pass where test_gpu_pencil_shapes.py does not reach, against the FP64 oracle at that file's
tolerances."""
import numpy as np
import pytest

from crava_b200 import api, synth
from oracle import bindings as ob
from oracle import ref64
from tests.test_gpu_pencil_shapes import TOL_COV, TOL_MEAN, TOL_SIM, crel

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    c = api.Context(0)
    yield c
    c.close()


def block(nx, ny, nz, nth, nsim, seed=0):
    return synth.make_block(synth.BlockSpec(nx=nx, ny=ny, nz=nz, theta_deg=tuple(np.linspace(5.0, 45.0, nth)),
                                            peak_hz=(30.0,) * nth, sn=(5.0,) * nth, nsim=nsim, seed=seed or nz + nth))


def check_against_oracle(ctx, blk, prior=api.PRIOR_SEPARABLE, tol_sim=TOL_SIM, **more):
    nx, ny, nz, nsim = blk.nx, blk.ny, blk.nz, blk.nsim
    post = ref64.posterior(blk)
    noise = ob.sim_noise(5, nsim, blk.nxp, blk.nyp, blk.nzp) if nsim else None
    out = api.invert_block(ctx, blk, prior, noise=noise, **more)
    assert out["counters"]["inverted_bins"] == post.n_inverted
    for a in range(3):
        assert crel(out["mean"][a][..., :nx], post.mean[a][..., :nx]) < TOL_MEAN, ("mean", a)
    for q in range(6):
        assert crel(out["cov"][q][..., :nx], post.cov[q][..., :nx]) < TOL_COV, ("cov", q)
    for s in range(nsim):
        sim = ref64.simulate(blk, post, noise[s])
        for a in range(3):
            assert crel(out["sims"][s, a][..., :nx], sim[a][..., :nx]) < tol_sim, ("sim", s, a)
    return out


# tiles that fill the shared memory of an SM to within its last kilobyte
@pytest.mark.parametrize("case", [(6, 5, 640, 2, 1), (5, 4, 640, 6, 0), (7, 4, 525, 3, 2), (20, 4, 375, 5, 0)])
def test_tiles_at_the_cap(ctx, case):
    check_against_oracle(ctx, block(*case))


# The Cholesky forms (prior grids, FP64 re-factorisation of some and of all bins, the separable prior without
# its eigen tables), where their tiles, orders and splits can go wrong: odd rows with 8-byte accesses, a tile one
# bin early, ragged last tiles and batches, every inlined split and general ones, 1 to 8 angles.  Realisations
# on prior grids: a bin whose prior spectrum is zero carries the grids' rounding, 1e-7 of the spectrum, and the
# realisations its square root, 3e-4; three times that.
CHOL_SHAPES = [(9, 7, 20, 2, 3), (9, 8, 125, 3, 5), (14, 6, 96, 4, 0), (30, 6, 128, 5, 4), (16, 6, 200, 4, 4),
               (36, 9, 256, 6, 3), (24, 7, 320, 7, 1), (12, 4, 343, 8, 2), (35, 40, 36, 1, 1)]


@pytest.mark.parametrize("case", CHOL_SHAPES)
def test_prior_grids(ctx, case):
    blk = block(*case)
    covs, _ = ref64.prior_cov_grids(blk)
    ec = ref64.fill_err_corr_zero_grad(blk.corr_xy, blk.nxp, blk.nyp, blk.nzp)
    for t in (0.0, 1.0):
        check_against_oracle(ctx, blk, api.PRIOR_GRIDS, tol_sim=1e-3, cov_grids=covs, err_corr=ec, fp64_threshold=t)


@pytest.mark.parametrize("case", CHOL_SHAPES)
@pytest.mark.parametrize("threshold", [0.0, 1.0, 100.0])
def test_separable_prior_by_cholesky(ctx, case, threshold):
    blk = block(*case)
    pk = api.pencil_key(blk.nzp, blk.ntheta)
    saved = api.tuning_get("pencil_kernel", pk)
    try:
        api.tuning_set("pencil_kernel", pk, 1)
        out = check_against_oracle(ctx, blk, fp64_threshold=threshold)
    finally:
        api.tuning_set("pencil_kernel", pk, saved)
    n = out["counters"]["fp64_bins"]
    assert n == 0 if threshold == 0.0 else n > 0 if threshold == 1.0 else n >= 0


# Tile widths, realisation batches and threads change the order of the work, not its results.
@pytest.mark.parametrize("dims", [(36, 9, 256), (21, 8, 90)])
@pytest.mark.parametrize("kernel", [1, 2])
def test_every_tile_gives_the_same(ctx, dims, kernel):
    nx, ny, nz = dims
    blk = block(nx, ny, nz, 3, 5)
    pk = api.pencil_key(nz, 3)
    keys = ("pencil_kernel", "pencil_w", "pencil_sb", "pencil_threads")
    saved = [api.tuning_get(k, pk) for k in keys]
    outs = []
    try:
        for w, sb, t in [(w, sb, 256) for w in (2, 4, 8) for sb in (1, 2, 3, 4)] + [(4, 2, 64), (4, 2, 192), (8, 1, 512)]:
            for k, v in zip(keys, (kernel, w, sb, t)):
                api.tuning_set(k, pk, v)
            outs.append(api.invert_block(ctx, blk, api.PRIOR_SEPARABLE, seed=17))
    finally:
        for k, v in zip(keys, saved):
            api.tuning_set(k, pk, v)
    for o in outs[1:]:
        for key in ("mean", "cov", "sims"):
            assert np.array_equal(outs[0][key], o[key]), key
