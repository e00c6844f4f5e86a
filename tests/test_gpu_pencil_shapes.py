"""The pencil pass at the edges of its tiles and plans, against the FP64 oracle: z lengths of one to
four stages and of every inlined split, the widest and narrowest tiles, rows that start on odd bins
(16-byte pairs, the tile one bin early) and z strides that allow 8-byte accesses only, ragged
last tiles and realisation batches, no realisations, 1 to 8 angle stacks.

Tolerances (norm-wise per grid): FP32 rounding, 6e-8, through about 100 operations per value in the
three transforms and the per-bin step gives some 1e-6; ten times that for the mean, and a
hundred for the covariance, whose per-bin differences S - ... cancel up to a factor of ten more; the
realisations as in the parity tests (the bins whose prior spectrum is zeroed carry rounding
residue, which the realisations take the square root of)."""
import numpy as np
import pytest

from crava_b200 import api, synth
from oracle import bindings as ob
from oracle import ref64

pytestmark = pytest.mark.gpu

TOL_MEAN, TOL_COV, TOL_SIM = 1e-5, 1e-4, 1e-4


def crel(x, ref):
    x = np.asarray(x, dtype=np.complex128)
    ref = np.asarray(ref, dtype=np.complex128)
    return float(np.linalg.norm(x - ref) / max(np.linalg.norm(ref), 1e-300))


@pytest.fixture(scope="module")
def ctx():
    c = api.Context(0)
    yield c
    c.close()


# (nx, ny, nz, angles, realisations, keep residuals)
@pytest.mark.parametrize("case", [
    (6, 5, 16, 1, 1, True),       # one stage; 20 bins a plane
    (9, 7, 20, 2, 3, False),      # one stage; 35 bins a plane: 8-byte accesses; ragged batch
    (9, 8, 125, 3, 5, False),     # three stages (5 x 5 x 5); odd rows one bin early
    (14, 6, 96, 4, 0, True),      # no realisations
    (30, 6, 128, 5, 4, False),    # 16 x 8
    (16, 6, 200, 4, 4, False),    # 20 x 10
    (20, 5, 243, 6, 2, False),    # 9 x 9 x 3
    (36, 9, 256, 6, 3, True),     # 16 x 16; a tile of one early bin, a last one of three
    (24, 7, 320, 7, 1, False),    # 20 x 16; 91 bins a plane
    (12, 4, 343, 8, 2, False),    # 7 x 7 x 7
    (10, 4, 625, 2, 1, False),    # four stages
    (7, 4, 1024, 8, 1, False),    # the longest line: two-bin tiles
    (5, 3, 1000, 3, 16, False),   # 9 bins a plane, 16 realisations
])
def test_pencil_shapes_match_oracle(ctx, case):
    nx, ny, nz, nth, nsim, resid = case
    blk = synth.make_block(synth.BlockSpec(nx=nx, ny=ny, nz=nz, theta_deg=tuple(np.linspace(5.0, 45.0, nth)),
                                           peak_hz=(30.0,) * nth, sn=(5.0,) * nth, nsim=nsim, seed=nz + nth))
    post = ref64.posterior(blk)
    noise = ob.sim_noise(5, nsim, nx, ny, nz) if nsim else None
    out = api.invert_block(ctx, blk, api.PRIOR_SEPARABLE, noise=noise, keep_residual=resid)
    assert out["counters"]["inverted_bins"] == post.n_inverted
    for a in range(3):
        assert crel(out["mean"][a][..., :nx], post.mean[a][..., :nx]) < TOL_MEAN, ("mean", a)
    for q in range(6):
        assert crel(out["cov"][q][..., :nx], post.cov[q][..., :nx]) < TOL_COV, ("cov", q)
    for s in range(nsim):
        sim = ref64.simulate(blk, post, noise[s])
        for a in range(3):
            assert crel(out["sims"][s, a][..., :nx], sim[a][..., :nx]) < TOL_SIM, ("sim", s, a)
    if resid:
        for l in range(nth):
            assert crel(out["resid_spec"][l], post.resid_spec[l]) < 1e-3, ("resid", l)


@pytest.mark.parametrize("dims", [(9, 8, 50), (9, 7, 45), (36, 5, 256)])
def test_product_noise_is_the_same_in_every_tile(ctx, dims):
    """Product-mode realisations do not depend on the tile (width, batch) that computes them: the bins'
    draws come from their own index, on the self-mirrored planes too."""
    nx, ny, nz = dims
    blk = synth.make_block_fast(synth.BlockSpec(nx=nx, ny=ny, nz=nz, theta_deg=(10.0, 30.0), peak_hz=(30.0, 30.0),
                                                sn=(5.0, 5.0), nsim=3, seed=3))
    pk = api.pencil_key(nz, 2)
    outs = []
    for w, sb in ((8, 2), (4, 1), (2, 3)):
        saved = [(k, api.tuning_get(k, pk)) for k in ("pencil_w", "pencil_sb")]
        try:
            api.tuning_set("pencil_w", pk, w)
            api.tuning_set("pencil_sb", pk, sb)
            outs.append(api.invert_block(ctx, blk, api.PRIOR_SEPARABLE, seed=41))
        finally:
            for k, v in saved:
                api.tuning_set(k, pk, v)
    for o in outs[1:]:
        for key in ("mean", "cov", "sims"):
            assert np.array_equal(outs[0][key], o[key]), key
