"""Rules that the kernels' sources keep and no run can check."""
import glob
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "bevy_eulerian_fluid_b200", "csrc")


def test_warp_exchanges_name_their_lanes():
    """The lanes that happen to run together (__activemask) need not include the partner of a shuffle: after a branch
    per lane the value exchanged is then undefined, whatever a compiler makes of it today."""
    sources = glob.glob(os.path.join(CSRC, "*.cu*"))
    assert len(sources) > 5
    for path in sources:
        code = re.sub(r"//[^\n]*", "", open(path).read())
        assert "__activemask" not in code, os.path.basename(path)
