"""Which transposes ask whether the state lies in the 2/3 box, and, at every
fused column length along x and row length along z, the RHS transpose on the box
against the general layout.  Tolerances: rounding of one transpose, 1e-12 in
float64 and 1e-5 in float32, as for one RHS."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _case(h3, dims, f64):
    g = h3.make_grid(*dims, dtype=torch.float64 if f64 else torch.float32)
    u = h3.hit_initial_field(1, g)
    v = torch.randn(u.shape, generator=torch.Generator(device="cuda").manual_seed(2), dtype=u.dtype, device="cuda")
    return h3.make_ns_rhs(g), u, v, h3.NSParams(nu=0.02, forcing=h3.BandForcing(eps=0.1, kmin=1.0, kmax=2.0))


# one RHS transpose: from 2^19 modes of fused columns; a step or a rollout: fused columns
@pytest.mark.parametrize("dims,f64,rhs_checks,step_checks", [
    ((32, 32, 32), False, 0, 1), ((64, 64, 256), False, 1, 1), ((64, 64, 128), True, 0, 1),
    ((256, 8, 16), False, 0, 1), ((256, 8, 16), True, 0, 0), ((512, 8, 8), False, 0, 0),
    ((256, 64, 64), True, 0, 0)])
def test_box_checks(h3, monkeypatch, dims, f64, rhs_checks, step_checks):
    import importlib
    adj = importlib.import_module("3dhit_b200.adjoint")
    asked = []
    flags = adj.resolve_flags
    monkeypatch.setattr(adj, "resolve_flags", lambda *a: asked.append(1) or flags(*a))
    rhs, u, v, p = _case(h3, dims, f64)
    h3.rhs_vjp(rhs, u, p, v)
    assert len(asked) == rhs_checks
    h3.rk4_step_vjp(rhs, u, p, 1e-3, v)
    assert len(asked) == rhs_checks + step_checks
    h3.rollout_vjp(rhs, u, p, 1e-3, 2, v)
    assert len(asked) == rhs_checks + 2 * step_checks


@pytest.mark.parametrize("f64", [False, True])
@pytest.mark.parametrize("dims", [(4, 8, 16), (8, 16, 4), (16, 4, 32), (32, 8, 64), (64, 4, 128), (128, 8, 8),
                                  (256, 4, 16), (16, 8, 256), (8, 4, 512), (4, 4, 1024), (16, 128, 8), (8, 256, 8),
                                  (4, 512, 8), (4, 1024, 8)])
def test_rhs_vjp_box_against_general(h3, monkeypatch, dims, f64):
    import importlib
    adj = importlib.import_module("3dhit_b200.adjoint")
    rhs, u, v, p = _case(h3, dims, f64)
    out = []
    for line in (0, 1 << 62):
        monkeypatch.setattr(adj, "_BOX_CHECK_MODES", line)
        out.append(h3.rhs_vjp(rhs, u, p, v))
    h3.check_device("rhs_vjp")
    tol = 1e-12 if f64 else 1e-5
    (ub, pb), (ub0, pb0) = out
    assert float((ub - ub0).norm() / ub0.norm()) <= tol
    for k in pb:
        assert pb[k] == pytest.approx(pb0[k], rel=100 * tol, abs=1e-300)
