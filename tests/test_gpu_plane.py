"""The plane kernel of small grids (y-inverse, z pass and y-forward of one x
plane in shared memory): every pair of row lengths it serves, against the
oracle's RHS and RK4 step on a dealiased state.  Tolerances as for every other
length (test_gpu_lengths.py): 1e-5 in float32, 1e-12 in float64."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("f64", [False, True])
@pytest.mark.parametrize("ny", [8, 16, 32, 64])
@pytest.mark.parametrize("nz", [8, 16, 32, 64])
def test_plane_pass(h3, orc, ny, nz, f64):
    dims, dtype = (8, ny, nz), np.float64 if f64 else np.float32
    og = orc.make_grid(*dims, dtype=dtype)
    rng = np.random.default_rng(ny + 3 * nz)
    u0 = orc.to_spectral(rng.standard_normal((3,) + dims).astype(dtype), og)
    u0 = orc.project(orc.dealias(u0, og), og).astype(og.cdtype)
    g = h3.make_grid(*dims, dtype=torch.float64 if f64 else torch.float32)
    p = h3.NSParams(nu=0.01, forcing=h3.LinearForcing(A=0.2))
    po = orc.NSParams(nu=0.01, forcing=orc.LinearForcing(A=0.2))
    rhs, orhs = h3.make_ns_rhs(g), orc.make_ns_rhs(og)
    tol = 1e-12 if f64 else 1e-5
    du, du0 = rhs(u0, p, 0.0, assume_dealiased=True).cpu().numpy(), orhs(u0, po, 0.0)
    assert np.linalg.norm(du - du0) <= tol * np.linalg.norm(du0)
    u1, u10 = h3.rollout(rhs, u0, p, 1e-3, 3, assume_dealiased=True).cpu().numpy(), u0
    for _ in range(3):
        u10 = orc.rk4_step(orhs, u10, po, 1e-3, 0.0)
    assert np.linalg.norm(u1 - u10) <= tol * np.linalg.norm(u10)
