"""The kernels' shapes are constants: no macro given to the compiler makes a
library other than the one that is tested (a level-0 emit at another register
budget ended with a device fault)."""
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "tesina-rt_gb300", "csrc")


def test_no_macro_changes_a_kernel():
    for f in sorted(os.listdir(CSRC)):
        if not f.endswith((".cu", ".cuh", ".h")):
            continue
        src = open(os.path.join(CSRC, f)).read()
        assert not re.findall(r"#\s*if(?:n?def|\s+!?\s*defined).*\bRT_\w+", src), f
