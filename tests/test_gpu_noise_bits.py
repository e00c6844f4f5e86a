"""Both pencil passes make the same draw for a bin: pair_noise (two bins at once) and device_noise3 (one) give
the same bits, on the planes that are their own mirror too, at even and odd sizes and for pairs that start
on an even or odd bin or one before the grid."""
import os
import subprocess

import pytest

from crava_b200 import build as cbuild

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def exe(tmp_path_factory):
    out = str(tmp_path_factory.mktemp("noise") / "noise_check")
    subprocess.run([cbuild.NVCC] + cbuild.ARCH + cbuild.FLAGS + ["-I" + cbuild.CSRC, "-o", out,
                    os.path.join(ROOT, "tests", "native", "noise_check.cu")], check=True)
    return out


@pytest.mark.parametrize("dims", [(35, 24, 20), (36, 25, 21), (8, 2, 2)])
@pytest.mark.parametrize("first", [0, -1])
def test_pair_draws_are_the_scalar_ones(exe, dims, first):
    r = subprocess.run([exe, *map(str, dims), str(first)], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, r
    bins, differing = (int(v) for v in r.stdout.split())
    nxp, nyp, nzp = dims
    assert bins == 2 * (nxp // 2 + 1) * nyp * nzp and differing == 0
