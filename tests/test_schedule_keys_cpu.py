"""Every schedule key that the tuner sweeps, or that the shipped table sets, is read by the library: a key that
no code reads would be tuned and stored for nothing."""
import os
import re

import crava_b200
from crava_b200 import build as cbuild

HERE = os.path.dirname(crava_b200.__file__)


def test_keys_are_read():
    src = "".join(open(os.path.join(cbuild.CSRC, f)).read() for f in sorted(os.listdir(cbuild.CSRC)))
    # tuned("key", ...) and tuned(cond ? "a" : "b", ...)
    read = set()
    for m in re.finditer(r"tuned\(([^;]*?),\s*[\w.]", src):
        read.update(re.findall(r'"(\w+)"', m.group(1)))
    tuner = open(os.path.join(HERE, "autotune.py")).read().split("def tune_workload")[1]
    swept = set(re.findall(r'"((?:pencil|line4|x4)_\w+)"', tuner))
    table = {l.split()[0] for l in open(os.path.join(HERE, "schedules.txt")) if l.strip() and not l.startswith("#")}
    assert swept and table and read
    assert swept - read == set() and table - read == set()
