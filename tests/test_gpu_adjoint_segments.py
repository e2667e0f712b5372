"""The segment store of the rollout's transpose: its size against a segment of
full states, and segments in which only some steps' stage inputs are kept."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _free():
    torch.cuda.synchronize()
    return torch.cuda.mem_get_info()[0]


def test_rollout_vjp_segment_store(h3):
    """One segment of 100 steps at 128^3.  The workspace of the whole call stays
    within the checkpoint, the K = 100 states of the segment and 26 states (what
    the transposes in the reference layout hold beside them: 8.4 of the general
    path, 3 + 1.5 + 2 transform inputs, fields and products, 3.2 of the 3-D
    transforms, 8 stage inputs and cotangents): 127 states of 25.6 MB.  All 400
    stage inputs as compact states are 131 by themselves."""
    g0 = h3.make_grid(128)
    u = h3.hit_initial_field(0, g0) * 0.1
    v = torch.randn(u.shape, generator=torch.Generator(device="cuda").manual_seed(1), dtype=u.dtype, device="cuda")
    p = h3.NSParams(nu=0.01, forcing=h3.BandForcing(eps=0.1, kmin=1.0, kmax=2.0))
    ref, pref = h3.rollout_vjp(h3.make_ns_rhs(g0), u, p, 1e-3, 100, v, checkpoint_every=10)
    g = h3.make_grid(128)
    g.plan  # tables and diagnostics scratch
    before = _free()
    ub, pb = h3.rollout_vjp(h3.make_ns_rhs(g), u, p, 1e-3, 100, v, checkpoint_every=100)
    used = before - _free()
    state = u.numel() * u.element_size()
    assert used <= 127 * state
    _close((ub, pb), (ref, pref), 1e-5)


def _close(got, ref, tol):
    """Rounding of a rollout: states and cotangents of 100 steps within 1e-5 in
    float32 and 1e-12 in float64, as everywhere in the suite; a parameter's
    cotangent is a sum of random signs over the modes: a hundred times that."""
    assert float((got[0] - ref[0]).norm() / ref[0].norm()) <= tol
    for k in ref[1]:
        assert got[1][k] == pytest.approx(ref[1][k], rel=100 * tol, abs=1e-300)


@pytest.mark.parametrize("kind", ["linear", "band", "hold"])
@pytest.mark.parametrize("dims,f64", [((32, 8, 16), True), ((16, 16, 16), False), ((8, 8, 4), True)])
def test_rollout_vjp_long_segments(h3, dims, f64, kind):
    """Segments longer than the store of stage inputs (33 steps; rows of four
    points, whose padded box is larger than the full rows, keep full states)
    against segments of one step."""
    g = h3.make_grid(*dims, dtype=torch.float64 if f64 else torch.float32)
    u = h3.hit_initial_field(2, g) * 0.1
    v = torch.randn(u.shape, generator=torch.Generator(device="cuda").manual_seed(1), dtype=u.dtype, device="cuda")
    forcing = {"linear": h3.LinearForcing(A=0.3), "band": h3.BandForcing(eps=0.1, kmin=1.0, kmax=2.0),
               "hold": h3.HoldEnergyForcing(0.02, 0.02, tau=0.7)}[kind]
    rhs, p = h3.make_ns_rhs(g), h3.NSParams(nu=0.02, forcing=forcing)
    ref, pref = h3.rollout_vjp(rhs, u, p, 1e-3, 40, v, checkpoint_every=1)
    for K in (33, 40):
        _close(h3.rollout_vjp(rhs, u, p, 1e-3, 40, v, checkpoint_every=K), (ref, pref), 1e-12 if f64 else 1e-5)
