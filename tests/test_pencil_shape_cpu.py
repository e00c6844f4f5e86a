"""The tile of the pencil pass (pencil_shape) for every z length up to the longest a job may have, 1 to 8
angles and 0 to 16 realisations: a shape comes back, and one that the kernel takes.  Runs the built
library's own function, without a device."""
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
        shapes, bad = (int(v) for v in r.stdout.split())
        assert shapes > 70000 and bad == 0, r.stderr

    return run


def test_every_job_has_a_shape(check):
    check()
