"""The fused RHS transpose (field-parallel x passes, fused z pass) at every
column length it serves along x and every row length along z, on the
dealiased layout (a state inside the 2/3 box) and on the general one, against
the oracle's transpose; the RK4 step's and the rollout's transposes (segments
with and without a remainder) on ragged grids.  Tolerances as in
test_gpu_adjoint.py: 1e-10 in float64, 2e-4 in float32."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _rel(a, b):
    return float(np.linalg.norm(a - b) / np.linalg.norm(b))


def _case(h3, orc, dims, f64, dealiased, kind="band"):
    rng = np.random.default_rng(sum(dims) + f64)
    og = orc.make_grid(*dims, dtype=np.float64)
    u = orc.to_spectral(rng.standard_normal((3,) + dims), og)
    if dealiased:
        u = orc.project(orc.dealias(u, og), og)
    u = np.ascontiguousarray(u)
    v = rng.standard_normal(u.shape) + 1j * rng.standard_normal(u.shape)
    g = h3.make_grid(*dims, dtype=torch.float64 if f64 else torch.float32)
    forc = {"band": lambda m: m.BandForcing(0.1, 1.0, 2.0), "hold": lambda m: m.HoldEnergyForcing(1.5, 0.02, tau=0.7),
            "linear": lambda m: m.LinearForcing(0.3)}[kind]
    ct = torch.complex128 if f64 else torch.complex64
    dev = [torch.as_tensor(np.ascontiguousarray(x), dtype=ct, device="cuda") for x in (u, v)]
    return og, u, v, g, h3.NSParams(0.02, forc(h3)), orc.NSParams(0.02, forc(orc)), dev


@pytest.mark.parametrize("dealiased", [True, False])
@pytest.mark.parametrize("f64", [False, True])
@pytest.mark.parametrize("dims", [(4, 8, 16), (8, 16, 4), (16, 4, 32), (32, 8, 64), (64, 4, 128), (128, 8, 8),
                                  (256, 4, 16), (16, 8, 256), (8, 4, 512), (4, 4, 1024)])
def test_rhs_vjp_at_every_length(h3, orc, dims, f64, dealiased):
    og, u, v, g, p, po, (ud, vd) = _case(h3, orc, dims, f64, dealiased)
    ub, pb = h3.rhs_vjp(h3.make_ns_rhs(g), ud, p, vd)
    h3.check_device("rhs_vjp")
    ubo, pbo = orc.rhs_vjp(og, u, po, v)
    tol = 1e-10 if f64 else 2e-4
    assert _rel(ub.cpu().numpy(), ubo) < tol
    scale = max(abs(pbo.get(k, 0.0)) for k in ("nu", "A", "eps"))
    for k in ("nu", "A", "eps"):
        assert abs(pb[k] - pbo.get(k, 0.0)) <= tol * max(1.0, scale)


@pytest.mark.parametrize("dealiased", [True, False])
@pytest.mark.parametrize("kind", ["linear", "band", "hold"])
def test_step_and_rollout_vjp_ragged(h3, orc, kind, dealiased):
    og, u, v, g, p, po, (ud, vd) = _case(h3, orc, (32, 8, 16), True, dealiased, kind)
    rhs, dt = h3.make_ns_rhs(g), 1e-3
    scale = np.sqrt((np.abs(u) ** 2).mean())
    ud, u = ud / scale, u / scale
    ub, _ = h3.rk4_step_vjp(rhs, ud, p, dt, vd)
    assert _rel(ub.cpu().numpy(), orc.rk4_step_vjp(og, u, po, dt, v)[0]) < 1e-10
    us, orhs = [u], orc.make_ns_rhs(og)
    for _ in range(4):
        us.append(orc.rk4_step(orhs, us[-1], po, dt, 0.0))
    ref = v
    for x in reversed(us):
        ref = orc.rk4_step_vjp(og, x, po, dt, ref)[0]
    for K in (1, 2, 5, 20):  # five steps: segments of one, with a remainder, and one short segment
        ub, _ = h3.rollout_vjp(rhs, ud, p, dt, 5, vd, checkpoint_every=K)
        assert _rel(ub.cpu().numpy(), ref) < 1e-10
