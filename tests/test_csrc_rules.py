"""Rules of the kernels' sources that a run cannot show, read from the text (no device)."""
import glob
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "mma_gb300", "csrc")


def _code(path):
    return re.sub(r"//[^\n]*|/\*.*?\*/", "", open(path).read(), flags=re.S)


def test_shuffles_name_their_lanes():
    """__activemask() names the lanes that happen to be converged and converges none: a sum that shuffles
    under it can miss lanes.  Every shuffle and vote names the lanes that take part."""
    for path in glob.glob(os.path.join(CSRC, "*.cu*")):
        assert "__activemask" not in _code(path), os.path.basename(path)
