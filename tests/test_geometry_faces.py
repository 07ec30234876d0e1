"""CPU: no strip of the advance kernel ends with a vertical NTFF face's column.  The face's
sample averages Ez of its column and the one to the right, and a strip has the last time
level of its owned columns alone."""
from __future__ import annotations

import pytest

from test_geometry import _items


@pytest.mark.parametrize("T,cols", [(1, 1), (2, 1), (2, 2), (2, 4), (3, 1), (3, 2), (4, 1), (4, 2), (6, 1), (8, 1)])
def test_no_strip_ends_at_a_face(tomo, T, cols):
    lib = tomo.library()
    for nx in list(range(40, 130)) + [195, 200, 333, 400, 401, 600, 1024, 2048]:
        for nc in (0, 8, 12, 16, 32):
            for d in range(nc + 1, min(nc + 36, nx // 2 - 2)):
                cover = [x for x0, x1, *_ in _items(lib, nx, nc, d, T, cols) for x in range(x0, x1)]
                assert sorted(cover) == list(range(nx + 1)), (nx, nc, d)
                for x0, x1, *_ in _items(lib, nx, nc, d, T, cols):
                    assert x1 - 1 not in (d, nx - d - 1), (nx, nc, d, x0, x1)
                    assert x1 - x0 >= 1
