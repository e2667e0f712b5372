"""The RHS through the plane kernel where its planes are not staged (more than 148
of them), and through every kernel of the RHS with a state that is not finite: one
bad mode reaches all modes of the 2/3 box and none outside."""
import math

import pytest
import torch

from test_gpu_cufft import cufft_rhs

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("f64", [False, True])
@pytest.mark.parametrize("dims", [(256, 8, 8), (256, 8, 64), (256, 64, 8), (256, 32, 16), (256, 64, 64), (512, 16, 32)])
def test_unstaged_planes(h3, dims, f64):
    g = h3.make_grid(*dims, dtype=torch.float64 if f64 else torch.float32)
    gen = torch.Generator(device="cuda").manual_seed(sum(dims))
    u = h3.to_spectral(torch.randn((3,) + dims, generator=gen, dtype=g.dtype, device="cuda"), g)
    u = h3.project(h3.dealias(u, g), g) / (dims[0] * dims[1] * dims[2]) ** 0.5
    du = h3.make_ns_rhs(g)(u, h3.NSParams(nu=0.01, forcing=h3.LinearForcing(A=0.2)), 0.0, assume_dealiased=True)
    ref = cufft_rhs(u, g, 0.01, 0.2)
    assert float((du - ref).norm() / ref.norm()) < (1e-12 if f64 else 1e-5)


@pytest.mark.parametrize("bad", [math.nan, math.inf])
@pytest.mark.parametrize("dims,f64", [((32, 32, 32), False), ((32, 32, 32), True), ((256, 16, 16), False),  # k_plane, k_p3f
                                      ((8, 128, 128), False), ((8, 8, 256), False), ((8, 256, 512), False),
                                      ((512, 8, 8), False), ((8, 512, 8), False), ((16, 8, 128), True),
                                      ((8, 256, 16), True)])
def test_nonfinite_state(h3, dims, f64, bad):
    g = h3.make_grid(*dims, dtype=torch.float64 if f64 else torch.float32)
    u = h3.hit_initial_field(0, g)
    u[1, 1, 1, 1] = complex(bad, 0.0)
    box = g.dealias.expand(3, *g.dealias.shape[-3:])
    for assume in (True, False):
        du = h3.make_ns_rhs(g)(u, h3.NSParams(nu=0.01), 0.0, assume_dealiased=assume)
        assert not torch.isfinite(du[box]).any()
        assert not du[~box].any()  # zero: the mean mode and everything outside the box
