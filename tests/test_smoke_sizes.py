"""smoke() reaches the kernels that large calls take: its sizes lie on the right sides of the library's limits."""
import os
import re

import __graft_entry__ as entry

CSRC = os.path.join(entry.ROOT, "ebgeometry_b200", "csrc", "capi_mesh.cu")


def test_smoke_takes_packets_and_points():
    with open(CSRC) as fh:
        src = fh.read()
    call = int(re.search(r"POINT_CALL = (\d+);", src).group(1))
    triangles = int(re.search(r"num_triangles >= (\d+)", src).group(1))
    assert entry.SMOKE_FEW <= call < entry.SMOKE_POINTS
    assert 20 * 4 ** entry.SMOKE_LEVEL >= triangles
