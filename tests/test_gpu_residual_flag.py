"""Outputs of a job that keeps its residual spectra against those of the same job without: they differ in the
order of roundings only (tolerances of test_gpu_pencil_shapes.py, each side being that near to the oracle),
at a z length whose split is inlined and at others, with odd and even rows and columns."""
import numpy as np
import pytest

from crava_b200 import api, synth
from tests.test_gpu_pencil_shapes import TOL_COV, TOL_MEAN, TOL_SIM, crel

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    c = api.Context(0)
    yield c
    c.close()


def block(nx, ny, nz, nsim=2):
    return synth.make_block_fast(synth.BlockSpec(nx=nx, ny=ny, nz=nz, theta_deg=(8.0, 20.0, 32.0), peak_hz=(30.0,) * 3,
                                                 sn=(5.0,) * 3, nsim=nsim, seed=nx + nz))


@pytest.mark.parametrize("dims", [(20, 36, 128), (21, 25, 256), (20, 25, 200), (21, 36, 63)])
def test_outputs_with_and_without(ctx, dims):
    blk = block(*dims)
    a = api.invert_block(ctx, blk, api.PRIOR_SEPARABLE, seed=5)
    b = api.invert_block(ctx, blk, api.PRIOR_SEPARABLE, seed=5, keep_residual=True)
    for key, tol in (("mean", TOL_MEAN), ("cov", TOL_COV), ("sims", TOL_SIM)):
        for q in range(len(a[key])):
            assert crel(a[key][q], b[key][q]) < 2 * tol, (key, q)
