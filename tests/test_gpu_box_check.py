"""`is_dealiased` in both its forms (a mode per thread; whole rows per warp from
4096 rows of 64 points in float32, 128 in float64): the first and the last modes
inside the 2/3 box are not seen, one mode outside is, wherever it stands."""
import math

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("f64", [False, True])
@pytest.mark.parametrize("dims", [(4, 4, 4), (8, 16, 1024), (64, 64, 32), (32, 64, 128), (64, 64, 64), (64, 64, 128),
                                  (1024, 4, 256), (32, 128, 512)])
def test_one_mode(h3, dims, f64):
    g = h3.make_grid(*dims, dtype=torch.float64 if f64 else torch.float32)
    u = torch.zeros(3, dims[0], dims[1], dims[2] // 2 + 1, dtype=g.cdtype, device="cuda")
    cx, cy, cz = (n // 3 for n in dims)
    inside = [(0, 0, 0), (cx, cy, cz), (-cx, -cy, 0), (0, cy, cz), (-cx, 0, cz)]
    outside = [(cx + 1, 0, 0), (-cx - 1, 0, cz), (0, cy + 1, 0), (0, -cy - 1, 0), (0, 0, cz + 1), (-1, -1, dims[2] // 2),
               (cx, cy, cz + 1), (-1, -1, cz + 1), (dims[0] // 2, dims[1] // 2, dims[2] // 2)]
    for c in range(3):
        for at in inside:
            u[(c,) + at] = 1.0
    assert h3.is_dealiased(u, g)
    for n, at in enumerate(outside):
        u[(n % 3,) + at] = (1e-30, 1e-30j, math.nan)[n // 3]
        assert not h3.is_dealiased(u, g)
        u[(n % 3,) + at] = 0.0
    assert h3.is_dealiased(u, g)
