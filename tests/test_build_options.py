"""The kernels' shapes are constants: no macro given to the compiler makes a
library other than the one that is tested (a level-0 emit at another register
budget ended with a device fault)."""
import os
import re
import shutil
import subprocess

import pytest

from rtgb import build

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "tesina-rt_gb300", "csrc")


def test_no_macro_changes_a_kernel():
    for f in sorted(os.listdir(CSRC)):
        if not f.endswith((".cu", ".cuh", ".h")):
            continue
        src = open(os.path.join(CSRC, f)).read()
        assert not re.findall(r"#\s*if(?:n?def|\s+!?\s*defined).*\bRT_\w+", src), f


@pytest.mark.skipif(shutil.which(build.NVCC) is None, reason="no nvcc")
def test_no_value_is_read_before_it_is_set(tmp_path):
    """The operands of & are evaluated in any order: a hit test that sets t and
    the comparison of t are no operands of one."""
    r = subprocess.run([build.NVCC] + build.FLAGS + ["-ptx", os.path.join(CSRC, "trace.cu"), "-o",
                                                     str(tmp_path / "trace.ptx")], capture_output=True, text=True)
    assert r.returncode == 0 and "used before its value" not in r.stderr, r.stderr[:2000]
