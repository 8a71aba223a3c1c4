"""The code that a wait leaves in the status word when it runs out names the kernel: no two source files share one."""
import glob
import os
import re

from tests.conftest import ROOT


def test_codes_name_one_kernel():
    of = {}
    for path in sorted(glob.glob(os.path.join(ROOT, "smallframework_b200", "csrc", "*.cu"))):
        with open(path) as f:
            for code in re.findall(r"\bstatus, (\d+)\b", f.read()):
                of.setdefault(int(code), set()).add(os.path.basename(path))
    assert len(of) > 50 and all(len(files) == 1 for files in of.values()), {c: f for c, f in of.items() if len(f) > 1}
