"""Every kernel that stages its input by TMA gives up its bounded wait, reports
it and leaves the device usable: with the limit at 0 polls the wait for a tile
ends at once (the CTA drains its copies with the default limit and returns),
`check_device` raises, and with the default limit restored the same call is
bit-identical to the one before.  Each shape has one staged kernel: the flag is that
kernel's."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _gives_up(h3, call):
    nat = h3._native
    ref = call()
    h3.check_device()  # starts clear
    nat.call("hit_set_wait_limit", 0)
    try:
        call()
        with pytest.raises(h3.DeviceWaitError):
            h3.check_device("give-up test")
    finally:
        nat.call("hit_set_wait_limit", -1)
    h3.check_device()  # read and cleared
    assert torch.equal(call(), ref)
    h3.check_device()


# The y passes of the 3-D transforms, the only staged ones there (rows of 64
# points in float32 and of 16 in float64 take no TMA, nor do columns of 4):
# k_axis2 at 128 .. 512 points (256 in float64), k_axis above.  (Forward passes of
# 128 points within L2 stage nothing.)
@pytest.mark.parametrize("n,f64,forward", [(128, False, False), (256, False, False), (256, False, True),
                                           (512, False, False), (512, False, True), (1024, False, False),
                                           (1024, False, True), (256, True, False), (256, True, True),
                                           (512, True, False), (512, True, True)])
def test_column_pass(h3, n, f64, forward):
    g = h3.make_grid(4, n, 16 if f64 else 64, dtype=torch.float64 if f64 else torch.float32)
    gen = torch.Generator(device="cuda").manual_seed(n)
    if forward:
        x = torch.randn(3, 4, n, g.Nz, generator=gen, dtype=g.dtype, device="cuda")
        _gives_up(h3, lambda: h3.to_spectral(x, g))
    else:
        x = torch.randn(3, 4, n, g.Nz // 2 + 1, generator=gen, dtype=g.cdtype, device="cuda")
        _gives_up(h3, lambda: h3.to_physical(x, g))


# The z pass, the plane kernel and the 512-point x pass of the RHS, each the only
# staged kernel of its shape (columns of at most 64 points stage nothing, the
# plane kernel nothing beyond 148 planes).
@pytest.mark.parametrize("dims,f64,box", [
    ((8, 8, 128), False, True), ((8, 8, 128), False, False),  # k_zwarp
    ((8, 8, 256), False, True), ((8, 8, 512), False, True),   # k_zw16
    ((8, 8, 1024), False, True),                              # k_zpair
    ((8, 8, 128), True, True), ((8, 8, 16), False, False),    # k_zcross
    ((8, 32, 32), False, True),                               # k_plane
    ((512, 8, 8), False, True),                               # k_p3m
])
def test_rhs_kernel(h3, dims, f64, box):
    g = h3.make_grid(*dims, dtype=torch.float64 if f64 else torch.float32)
    u = h3.hit_initial_field(0, g)
    rhs, p = h3.make_ns_rhs(g), h3.NSParams(nu=0.01)
    _gives_up(h3, lambda: rhs(u, p, 0.0, assume_dealiased=box))


# the transpose's z pass: rows of 16 points and float64 k_zadj, 128 points k_zadjw
@pytest.mark.parametrize("nz,f64", [(16, False), (128, False), (128, True)])
def test_transpose_z_pass(h3, nz, f64):
    g = h3.make_grid(8, 8, nz, dtype=torch.float64 if f64 else torch.float32)
    u = h3.hit_initial_field(0, g)
    v = torch.randn(u.shape, generator=torch.Generator(device="cuda").manual_seed(1), dtype=u.dtype, device="cuda")
    rhs, p = h3.make_ns_rhs(g), h3.NSParams(nu=0.01, forcing=h3.LinearForcing(A=0.2))
    _gives_up(h3, lambda: h3.rhs_vjp(rhs, u, p, v)[0])
