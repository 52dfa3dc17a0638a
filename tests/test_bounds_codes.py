"""The checked build's failure codes (GLOBE_BOUNDS) name one check each, whichever file it is in."""
import collections
import glob
import os
import re

from helpers import ROOT


def test_codes_are_unique():
    codes = collections.Counter()
    for path in glob.glob(os.path.join(ROOT, "globe_gb300", "csrc", "*.cu*")):
        with open(path) as f:
            codes.update(re.findall(r"\b(0x[0-9A-Fa-f]{4}u)\)", f.read()))
    assert len(codes) >= 10
    assert not [c for c, n in codes.items() if n > 1]
