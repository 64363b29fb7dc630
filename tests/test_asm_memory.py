"""Every inline PTX statement of the kernels that reads, writes or orders memory
tells the compiler so (a "memory" clobber)."""
import glob
import os
import re

from conftest import ROOT


def test_memory_statements_clobber_memory():
    seen = 0
    for path in sorted(glob.glob(os.path.join(ROOT, "goldbach-l0_gb300", "csrc", "*.cu*"))):
        text = open(path).read()
        for m in re.finditer(r"\basm\b[^;]*?\((.*?)\);\s", text, re.S):
            if re.search(r'"[^"]*\b(red|atom|ld|st|cp|mbarrier|fence)\.', m.group(1)):
                seen += 1
                assert '"memory"' in m.group(1), (os.path.basename(path), m.group(1)[:80])
    assert seen >= 8
