"""A cotangent that is not finite at a mode outside the 2/3 box, with a state
inside it: the viscosity's cotangent -sum k^2 Re(conj(v) u) meets 0 * NaN (or
0 * Inf) there and is NaN, as the sum over all modes gives; the state's cotangent
is not finite at that mode alone, and the linear forcing's coefficient (whose
sum runs over the box) stays finite."""
import math

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("bad", [math.nan, math.inf, None])
@pytest.mark.parametrize("f64", [False, True])
@pytest.mark.parametrize("dims", [(16, 8, 16), (64, 16, 64)])
def test_nonfinite_cotangent_outside_the_box(h3, dims, f64, bad):
    g = h3.make_grid(*dims, dtype=torch.float64 if f64 else torch.float32)
    u = h3.hit_initial_field(3, g)
    gen = torch.Generator(device="cuda").manual_seed(5)
    v = torch.randn(u.shape, generator=gen, dtype=u.dtype, device="cuda")
    if bad is not None:
        v[1, dims[0] // 2, 1, 1] = complex(bad, 0.0)  # |kx| > Nx / 3
    rhs, p = h3.make_ns_rhs(g), h3.NSParams(nu=0.02, forcing=h3.LinearForcing(A=0.3))
    for ub, pb in (h3.rhs_vjp(rhs, u, p, v), h3.rk4_step_vjp(rhs, u, p, 1e-3, v),
                   h3.rollout_vjp(rhs, u, p, 1e-3, 3, v, checkpoint_every=2)):
        assert torch.equal(torch.isfinite(ub), torch.isfinite(v))
        assert math.isfinite(pb["nu"]) if bad is None else math.isnan(pb["nu"])
        assert math.isfinite(pb["A"])
