"""Strided inputs give the bits of contiguous ones: coefficients as two slices of one
tensor, grid keys, indices and gradients as every other element of a wider one."""
import pytest
import torch

from refutil import SceneTensors
from sv_raster_b200 import _C as mC
from sv_raster_b200 import synthetic
from test_gpu_batched import _raster

pytestmark = pytest.mark.gpu


def _every_other(t):
    wide = torch.zeros(*t.shape[:-1], 2 * t.shape[-1], dtype=t.dtype, device=t.device)
    wide[..., ::2] = t
    return wide[..., ::2]


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_coefficients_as_slices_of_one_tensor(dtype):
    C = SceneTensors(synthetic.config_scene("c1"))
    r, _ = _raster(C)
    gen = torch.Generator(device="cuda").manual_seed(2)
    # as wide as the scene's own (16 terms), and so narrow that both copies are of a size
    for M, deg in ((16, 3), (2, 0)):
        both = torch.randn(len(C.centers), M, 3, device="cuda", generator=gen).to(dtype)
        r.prepare(both[:, 0].contiguous(), both[:, 1:].contiguous(), deg)
        want = r.arrays()["rgbs"].clone()
        r.arrays()["rgbs"].zero_()
        r.prepare(both[:, 0], both[:, 1:], deg)
        seen = r.arrays()["ndup"] > 0
        assert torch.equal(r.arrays()["rgbs"][seen], want[seen])


@pytest.mark.parametrize("dim", [1, 3])
def test_strided_grid_gathers(dim):
    gen = torch.Generator(device="cuda").manual_seed(dim)
    n, m = 3000, 5000
    key = torch.randint(0, m, (n, 8), device="cuda", generator=gen)
    care = torch.randperm(n, device="cuda", generator=gen)
    pts = torch.randn(m, dim, device="cuda", generator=gen)
    d = torch.randint(-8, 9, (n, 8) if dim == 1 else (n, 8, 3), device="cuda", generator=gen).float()  # exact sums
    fwd = mC.gather_triinterp_geo_params if dim == 1 else mC.gather_triinterp_feat_params
    bwd = mC.gather_triinterp_geo_params_bw if dim == 1 else mC.gather_triinterp_feat_params_bw
    assert torch.equal(fwd(_every_other(key), _every_other(care), _every_other(pts)), fwd(key, care, pts))
    assert torch.equal(bwd(_every_other(key), _every_other(care), m, _every_other(d)), bwd(key, care, m, d))
