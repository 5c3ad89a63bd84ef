"""Batched exact arithmetic: the backward recovers each pixel's transmittance by dividing
by 1 - alpha record by record, so its rays and alphas have to be the forward's bit for
bit: for small voxels one unit in the last place of a ray moves alpha by 1e-3."""
import numpy as np
import pytest
import torch

from sv_raster_b200 import synthetic
from sv_raster_b200.batched import BatchedRasterizer

pytestmark = pytest.mark.gpu

LEVEL, SIZE = 12, 24


class _Cam:
    def __init__(self, c):
        self.__dict__.update({k: getattr(c, k) for k in ("width", "height", "tanfovx", "tanfovy", "cx", "cy", "near")})
        self.w2c, self.c2w = (torch.from_numpy(m).cuda() for m in (c.w2c, c.c2w))


@pytest.fixture(scope="module")
def block():
    """8 x 8 x 6 cells of 1/4096 at the centre, an optical depth of one or two each, seen
    from 1.6 away by 24 x 24 pixels 35 degrees off the optical axis (where both of the
    two products summed in a ray's direction count)."""
    ijk = np.stack(np.meshgrid(np.arange(8), np.arange(8), np.arange(6), indexing="ij"), -1).reshape(-1, 3) + 2045
    path = synthetic.ijk_to_octpath(ijk, np.full(len(ijk), LEVEL))
    centers, lengths = synthetic.decode_voxels(path, np.full(len(ijk), LEVEL))[:2]
    rng = np.random.default_rng(0)
    t = lambda a, dt=torch.float32: torch.from_numpy(np.ascontiguousarray(a)).cuda().to(dt)
    mid = centers.mean(0).astype(np.float64)
    cam = synthetic.make_camera(SIZE, SIZE, float(2 * np.degrees(np.arctan(5.5 / 2 ** LEVEL / 1.6))),
                                tuple(mid + np.array([0.13, -0.21, -1.58])),
                                target=tuple(mid + np.array([-0.8, 0.75, 0.0])))
    x, y, z = (cam.w2c.astype(np.float64) @ np.append(mid, 1.0))[:3]
    focal = 0.5 * SIZE / cam.tanfovx
    cam.cx, cam.cy = SIZE / 2 - focal * x / z, SIZE / 2 - focal * y / z
    return dict(d=[t(path.reshape(-1, 1), torch.int64), t(centers), t(lengths).reshape(-1, 1)], n=len(ijk), cam=cam,
                geos=t(rng.uniform(20.0, 90.0, (len(ijk), 8))))


@pytest.mark.parametrize("grid", [False, True])
@pytest.mark.parametrize("ns,tile,ppt", [(1, 8, 1), (2, 8, 1), (3, 16, 1), (1, 16, 1), (1, 8, 2), (3, 16, 2)])
def test_weights_of_a_pixel_add_up(block, ns, tile, ppt, grid):
    """With the gradient of one pixel's red alone, the voxels' colour gradients are the
    records' weights, which add up to 1 - T.  A record's recovered T takes a division
    (2 ulp), a subtraction and the forward's product, 4 * 2^-24 in all, and a pixel
    has under 20 records: 20 * 4 * 2^-24 = 5e-6; the sum's own rounding as much again."""
    b = block
    r = BatchedRasterizer([_Cam(b["cam"])], *b["d"], max_level=LEVEL, n_samp_per_vox=ns, tile_size=tile, exact=True)
    r.set_pixels_per_thread(ppt)
    sh0, shs = torch.zeros(b["n"], 3).cuda(), torch.zeros(b["n"], 15, 3).cuda()
    r.fit_capacity(sh0, shs, 0)
    r.prepare(sh0, shs, 0)
    key = torch.arange(8 * b["n"], device="cuda").view(-1, 8)
    color, T = r.render_grid(key, b["geos"].reshape(-1)) if grid else r.render(b["geos"])
    contrib = r.arrays()["n_contrib"]
    opaque = torch.nonzero((T < 0.2) & (contrib > 0)).reshape(-1)
    assert len(opaque) > 200
    worst = 0.0
    for p in opaque[:: len(opaque) // 40].tolist():
        dC = torch.zeros(3 * r.n_pixels, device="cuda")
        dC[p] = 1.0
        if grid:
            r.backward_render_grid(key, b["geos"].reshape(-1), T, dC, torch.zeros_like(T),
                                   torch.zeros(8 * b["n"], device="cuda"))
        else:
            r.backward_render(b["geos"], T, dC, torch.zeros_like(T), torch.zeros(b["n"], 8, device="cuda"))
        weights = r.arrays()["drgbs"][0, :, 0].double()
        worst = max(worst, abs(weights.sum().item() - (1.0 - T[p].double().item())))
    assert r.header()[1] == 0
    assert worst < 1e-5
