"""The TMA-staged two-stage column pass (columns of 128, 256 and, in float32, 512
points): tiles at the end of a row that are only partly valid, fewer tiles than
CTAs and several per CTA, both layouts, against the oracle's RHS.  Tolerances as
for every other length (test_gpu_lengths.py): 1e-5 in float32, 1e-12 in float64."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("box", [True, False])
@pytest.mark.parametrize("dims,f64", [((8, 128, 8), False), ((8, 128, 64), False), ((64, 128, 128), False),
                                      ((8, 256, 8), False), ((32, 256, 128), False), ((8, 512, 8), False),
                                      ((8, 512, 32), False), ((16, 512, 128), False), ((8, 256, 8), True),
                                      ((16, 256, 64), True)])
def test_column_pass(h3, orc, dims, f64, box):
    dtype = np.float64 if f64 else np.float32
    og = orc.make_grid(*dims, dtype=dtype)
    rng = np.random.default_rng(sum(dims))
    u0 = orc.to_spectral(rng.standard_normal((3,) + dims).astype(dtype), og)
    u0 = (orc.project(orc.dealias(u0, og), og) if box else orc.project(u0, og)).astype(og.cdtype)
    rhs = h3.make_ns_rhs(h3.make_grid(*dims, dtype=torch.float64 if f64 else torch.float32))
    du = rhs(u0, h3.NSParams(nu=0.01), 0.0, assume_dealiased=box).cpu().numpy()
    du0 = orc.make_ns_rhs(og)(u0, orc.NSParams(nu=0.01), 0.0)
    assert np.linalg.norm(du - du0) <= (1e-12 if f64 else 1e-5) * np.linalg.norm(du0)
