"""The library's sources have one form: no macro given to the compiler changes
what they do (a switch of the tile widths had been left in once)."""
import os
import re

from conftest import ROOT


def test_no_conditional_compilation():
    for folder in ("jenhine_b200/csrc", "jenhine_b200/host", "include"):
        for d, _, names in os.walk(os.path.join(ROOT, folder)):
            for name in names:
                if not name.endswith((".cu", ".cuh", ".cpp", ".h")):
                    continue
                with open(os.path.join(d, name)) as f:
                    found = re.findall(r"^[ \t]*#[ \t]*(?:el)?if.*", f.read(), re.M)
                assert all(re.search(r"ifndef \w+_H\b|__cplusplus", line) for line in found), (name, found)
