"""TMA loads stay within one CTA's shared memory: no load names several CTAs of
a cluster as its destination, so a kernel may run on any rank of a job."""
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.abspath(__file__)), "..", "automs_gb300", "csrc")


def test_loads_have_one_destination():
    files = [f for f in sorted(os.listdir(CSRC)) if f.endswith((".cu", ".cuh", ".h", ".cpp"))]
    assert files
    for name in files:
        with open(os.path.join(CSRC, name)) as f:
            # the pieces of one inline instruction joined
            text = re.sub(r'"\s*"', "", f.read())
        for op in re.findall(r"cp\.async\.bulk[\w.:]*", text):
            assert "multi" not in op, f"{name}: {op}"
