"""Densities outside the ordinary range in the batched path: infinities, the types'
lowest and highest values, and corners masked with them one by one.

With the fast arithmetic a voxel with a corner at minus infinity (or one so low that
the interpolant is far below zero everywhere else) is empty and one with a corner at
plus infinity opaque: the same bits as voxels that are so by finite densities equal
in all corners, where the interpolant is exact."""
import numpy as np
import pytest
import torch

from refutil import rel_err
from sv_raster_b200 import synthetic
from sv_raster_b200.batched import BatchedRasterizer

pytestmark = pytest.mark.gpu

LOW32, LOW16 = torch.finfo(torch.float32).min, torch.finfo(torch.bfloat16).min
EMPTY, OPAQUE = -1e4, 1e6  # in all corners: no alpha; an optical depth past any exponent


class _Cam:
    def __init__(self, c):
        self.__dict__.update({k: getattr(c, k) for k in ("width", "height", "tanfovx", "tanfovy", "cx", "cy", "near")})
        self.w2c, self.c2w = (torch.from_numpy(m).cuda() for m in (c.w2c, c.c2w))


class _Scene:
    def __init__(self, n=1500):
        sc = synthetic.config_scene("c1")
        keep = np.sort(np.argsort(sc.lengths.reshape(-1), kind="stable")[-n:])
        t = lambda a, dt=torch.float32: torch.from_numpy(np.ascontiguousarray(a)).cuda().to(dt)
        self.n = n
        self.d = [t(sc.octpath[keep].reshape(-1, 1), torch.int64), t(sc.centers[keep]), t(sc.lengths[keep])]
        self.max_level = sc.max_level
        self.geos = t(sc.geos[keep])
        self.sh0 = t(np.random.default_rng(0).uniform(-1, 1, (n, 3)))
        self.shs = torch.zeros(n, 15, 3).cuda()


@pytest.fixture(scope="module")
def scene():
    return _Scene()


def _run(s, geos, ns, ppt, grid, size=(120, 88)):
    cam = _Cam(synthetic.make_camera(*size, 50.0, (0.1, -0.2, -1.4)))
    r = BatchedRasterizer([cam], *s.d, max_level=s.max_level, n_samp_per_vox=ns, tile_size=8)
    r.set_staging(32)
    r.set_pixels_per_thread(ppt)
    r.fit_capacity(s.sh0, s.shs, 0)
    r.prepare(s.sh0, s.shs, 0)
    gen = torch.Generator(device="cuda").manual_seed(1)
    dC = torch.randn(3 * r.n_pixels, device="cuda", generator=gen)
    dT = torch.randn(r.n_pixels, device="cuda", generator=gen)
    if grid:  # every voxel its own eight grid points
        key = torch.arange(8 * s.n, device="cuda").view(-1, 8)
        color, T = r.render_grid(key, geos.reshape(-1))
        g = torch.zeros(8 * s.n, device="cuda")
        r.backward_render_grid(key, geos.reshape(-1), T, dC, dT, g)
        g = g.view(-1, 8)
    else:
        color, T = r.render(geos)
        g = torch.zeros(s.n, 8, device="cuda")
        r.backward_render(geos, T, dC, dT, g)
    assert r.header()[1] == 0
    return color, T, g


CORNERS = [[0, 1, 2, 3, 4, 5, 6, 7], [0], [7], [0, 3, 5, 6], [1, 2, 4, 6, 7]]


@pytest.mark.parametrize("ns,ppt,grid,dtype", [(1, 1, False, torch.float32), (1, 1, True, torch.float32),
                                               (1, 1, False, torch.bfloat16), (1, 1, True, torch.bfloat16),
                                               (3, 1, False, torch.float32), (1, 2, False, torch.float32),
                                               (2, 2, True, torch.float32)])
@pytest.mark.parametrize("corners", CORNERS)
@pytest.mark.parametrize("value", [-float("inf"), LOW32, LOW16, -1e30, -1e12, float("inf")])
def test_masked_voxels(scene, value, corners, ns, ppt, grid, dtype):
    s = scene
    if dtype == torch.bfloat16 and value == LOW32:
        pytest.skip("rounds to minus infinity, which is covered")
    masked = torch.arange(s.n, device="cuda") % 3 == 0
    geos, want = s.geos.clone(), s.geos.clone()
    for c in corners:
        geos[masked, c] = value
    want[masked] = EMPTY if value < 0 else OPAQUE
    c0, t0, g0 = _run(s, want.to(dtype), ns, ppt, grid)
    c1, t1, g1 = _run(s, geos.to(dtype), ns, ppt, grid)
    assert torch.equal(c0, c1) and torch.equal(t0, t1)
    assert torch.isfinite(g1).all() and not g1[masked].any()
    assert rel_err(g1, g0) < 1e-5  # up to the order of the additions


@pytest.mark.parametrize("ns", [1, 3])
def test_highest_and_lowest_corners_together(scene, ns):
    """Corners whose differences pass the largest float: as the same pattern 2^28
    times smaller (whose interpolant has the same sign everywhere but within rounding
    of its zeros: under one pixel in a hundred)."""
    s = scene
    sign = torch.tensor([1, -1, -1, 1, -1, 1, 1, -1], device="cuda", dtype=torch.float32)
    big = (-LOW32) * sign.expand(s.n, 8).contiguous()
    c0, t0, g0 = _run(s, big * 2.0 ** -28, ns, 1, False)
    c1, t1, g1 = _run(s, big, ns, 1, False)
    assert torch.isfinite(g1).all()
    assert ((t0 - t1).abs() > 1e-6).float().mean() < 0.01
