"""Device memory that a destroyed plan gives back."""
import gc

import pytest
import torch

pytestmark = pytest.mark.gpu


def _free():
    torch.cuda.synchronize()
    return torch.cuda.mem_get_info()[0]


def test_destroyed_plan_gives_back_the_force_buffer(h3):
    """Ten plans that ran a forced step, one after another: nothing stays
    allocated (one force buffer is three compact components, 8 MB on the 2/3 box
    of 128^3)."""
    def forced_step():
        g = h3.make_grid(128)
        h3.rk4_step(h3.make_ns_rhs(g), u, p, 1e-3, 0.0, assume_dealiased=True, f_ext=f)
        torch.cuda.synchronize()
        del g
        gc.collect()

    u = h3.hit_initial_field(0, h3.make_grid(128))
    f = torch.zeros_like(u)
    p = h3.NSParams(nu=0.01)
    forced_step()  # module loads and the caching allocator's blocks
    before = _free()
    for _ in range(10):
        forced_step()
    assert before - _free() < 8 << 20
