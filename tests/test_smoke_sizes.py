"""smoke() reaches the kernels that large calls take: its sizes lie on the right sides of the library's limits."""
import os
import re

import __graft_entry__ as entry

CSRC = os.path.join(entry.ROOT, "ebgeometry_b200", "csrc")


def _constant(name):
    for file in ("capi_mesh.cu", "capi_internal.h"):
        with open(os.path.join(CSRC, file)) as fh:
            found = re.search(rf"{name}\s*= (\d+);", fh.read())
        if found:
            return int(found.group(1))
    raise KeyError(name)


def test_smoke_takes_packets_and_points():
    call, triangles = _constant("POINT_CALL"), _constant("PACKET_TRIANGLES")
    assert entry.SMOKE_FEW <= call < entry.SMOKE_POINTS
    assert 20 * 4 ** entry.SMOKE_LEVEL >= triangles
