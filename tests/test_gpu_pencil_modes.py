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


def check_against_oracle(ctx, blk, prior=api.PRIOR_SEPARABLE, **more):
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
            assert crel(out["sims"][s, a][..., :nx], sim[a][..., :nx]) < TOL_SIM, ("sim", s, a)
    return out


# tiles that fill the shared memory of an SM to within its last kilobyte
@pytest.mark.parametrize("case", [(6, 5, 640, 2, 1), (5, 4, 640, 6, 0), (7, 4, 525, 3, 2), (20, 4, 375, 5, 0)])
def test_tiles_at_the_cap(ctx, case):
    check_against_oracle(ctx, block(*case))
