"""The tile of the pencil pass (pencil_shape) for every z length up to the longest a job may have, 1 to 8
angles and 0 to 16 realisations: a shape comes back, and one that the kernel takes; on small blocks one
that uses the SMs.  Runs the built library's own function, without a device."""
import os
import subprocess

import pytest

from crava_b200 import build as cbuild

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.fixture(scope="module")
def check(tmp_path_factory):
    exe = str(tmp_path_factory.mktemp("shape") / "pencil_shape_check")
    subprocess.run([cbuild.NVCC, "-std=c++17", "-O2", "-I" + cbuild.CSRC, "-o", exe,
                    os.path.join(ROOT, "tests", "native", "pencil_shape_check.cu"), cbuild.build(),
                    "-Xlinker", "-rpath," + cbuild.HERE], check=True)

    def run(*args):
        r = subprocess.run([exe, *map(str, args)], capture_output=True, text=True, timeout=600)
        assert r.returncode == 0, (r.returncode, r.stderr)
        return [int(v) for v in r.stdout.split()], r.stderr

    return run


def test_every_job_has_a_shape(check):
    (shapes, bad), err = check()
    assert shapes > 70000 and bad == 0, err


@pytest.mark.parametrize("dims", [(20, 20, 40), (24, 36, 42), (32, 30, 40), (32, 24, 54), (24, 24, 128), (36, 9, 256)])
@pytest.mark.parametrize("nth,nsim", [(2, 1), (4, 8), (3, 16)])
@pytest.mark.parametrize("eig", [0, 1])
def test_small_blocks_fill_the_sms(check, dims, nth, nsim, eig):
    """Fewer tiles than SMs: narrow ones, and the threads of a whole SM as far as there are pairs (bins without the
    eigen form) to take."""
    (W, SB, T, tiles), _ = check(*dims, nth, nsim, eig)
    assert W <= 4 and tiles <= 2 * 148 and SB >= min(nsim, 2)
    units = dims[2] * W // (2 if eig else 1)
    per_sm = -(-tiles // 148)
    assert T >= min(512 // per_sm // 32 * 32, units)
