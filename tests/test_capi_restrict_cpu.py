"""mgp_restrict refuses centrings that are neither node (0) nor cell (1) before it looks at
the arrays' memory: the nodal kernel writes a point more than an array of such a centring
has, and device arrays are written where they lie."""
from __future__ import annotations

import ctypes as C

import numpy as np
import pytest

from mgpoisson2d_b200.types import Box, BoxData


@pytest.mark.parametrize("offi,offj", [(2, 1), (1, 2), (2, 2), (-1, 0), (0, 7)])
def test_unknown_centrings_are_refused(offi, offj):
    import mgpoisson2d_b200.api as api
    f = Box.of_size(16, 12)
    c = f.coarsened(2, 2)
    fine, crse = BoxData(f), BoxData(c, fill=3.0)
    rc = api._lib.mgp_restrict(C.byref(f.c()), C.byref(fine.c()), C.byref(c.c()), C.byref(crse.c()), offi, offj)
    assert rc == _einval() and b"offi" in api._lib.mgp_last_error()
    assert np.all(crse.data == 3.0)


def _einval():
    import os
    import re
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    src = open(os.path.join(root, "include", "mgp2d.h")).read()
    return int(re.search(r"MGP_EINVAL\s*=?\s*\(?(-?\d+)", src).group(1))
