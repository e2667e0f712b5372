"""The column passes on both sides of the sizes where another kernel takes over:
the y passes of the 3-D transforms (three components, general layout) through
k_axis2 below and k_axis above its limit (512 MB at 128 points, 128 MB at 256 and
512), and the RHS on the 2/3 box of 512 x 128 x 256, whose y-forward (138 MB) is
the 128-point k_axis2.  Against cuFFT in float64; tolerances as for every other
length: 1e-5 in float32, 1e-12 in float64."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _rel(a, b):
    return float((a - b).abs().pow(2).sum().sqrt() / b.abs().pow(2).sum().sqrt())


@pytest.mark.parametrize("dims,f64", [((512, 128, 256), False), ((1024, 128, 512), False),  # 213, 830 MB
                                      ((64, 256, 128), False), ((256, 256, 256), False),    # 28, 214
                                      ((128, 512, 64), False), ((128, 512, 256), False),    # 63, 214
                                      ((32, 256, 64), True), ((256, 256, 128), True)])      # 16, 226
def test_transforms(h3, dims, f64):
    g = h3.make_grid(*dims, dtype=torch.float64 if f64 else torch.float32)
    gen = torch.Generator(device="cuda").manual_seed(sum(dims))
    x = torch.randn((3,) + dims, generator=gen, dtype=g.dtype, device="cuda")
    tol = 1e-12 if f64 else 1e-5
    xh = h3.to_spectral(x, g)
    for c in range(3):
        assert _rel(xh[c], torch.fft.rfftn(x[c].double())) < tol
    y = h3.to_physical(xh, g)
    for c in range(3):
        assert _rel(y[c], x[c].double()) < tol


def test_box_forward_of_128_points_beyond_l2(h3):
    from test_gpu_cufft import cufft_rhs
    g = h3.make_grid(512, 128, 256)
    gen = torch.Generator(device="cuda").manual_seed(1)
    u = h3.to_spectral(torch.randn(3, 512, 128, 256, generator=gen, device="cuda"), g)
    u = h3.project(h3.dealias(u, g), g) / (512 * 128 * 256) ** 0.5
    du = h3.make_ns_rhs(g)(u, h3.NSParams(nu=0.01, forcing=h3.LinearForcing(A=0.2)), 0.0, assume_dealiased=True)
    assert _rel(du, cufft_rhs(u, g, 0.01, 0.2)) < 1e-5
