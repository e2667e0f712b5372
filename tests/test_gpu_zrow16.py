"""The z pass with 16 values per lane (rows of 256 and 512 points on the
dealiased layout): fewer row groups than warps, one row group per warp, and a
last wave that is partly empty, against the oracle's RHS.  Tolerance as for
every other length in float32 (test_gpu_lengths.py): 1e-5."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dims", [(8, 8, 256), (128, 32, 256), (64, 128, 256), (8, 8, 512), (32, 64, 512), (64, 64, 512)])
def test_z_pass(h3, orc, dims):
    og = orc.make_grid(*dims, dtype=np.float32)
    rng = np.random.default_rng(sum(dims))
    u0 = orc.to_spectral(rng.standard_normal((3,) + dims).astype(np.float32), og)
    u0 = orc.project(orc.dealias(u0, og), og).astype(og.cdtype)
    rhs = h3.make_ns_rhs(h3.make_grid(*dims, dtype=torch.float32))
    du = rhs(u0, h3.NSParams(nu=0.01), 0.0, assume_dealiased=True).cpu().numpy()
    du0 = orc.make_ns_rhs(og)(u0, orc.NSParams(nu=0.01), 0.0)
    assert np.linalg.norm(du - du0) <= 1e-5 * np.linalg.norm(du0)
