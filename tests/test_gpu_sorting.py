"""Orders made on the GPU where their pieces can go wrong: segment lengths around
the sizes at which the sorts change form, against a stable sort on the CPU."""
import numpy as np
import pytest
import torch

from sv_raster_b200 import _C as mC
from sv_raster_b200 import synthetic
from sv_raster_b200.batched import BatchedRasterizer
from sv_raster_b200.levels21 import _C as dC

pytestmark = pytest.mark.gpu


class _Cam:
    def __init__(self, c):
        self.__dict__.update({k: getattr(c, k) for k in ("width", "height", "tanfovx", "tanfovy", "cx", "cy", "near")})
        self.w2c, self.c2w = (torch.from_numpy(m).cuda() for m in (c.w2c, c.c2w))


def _cuda(a, dt=torch.float32):
    return torch.from_numpy(np.ascontiguousarray(a)).cuda().to(dt)


def _instances(ndup, bbox, quad, width, height, tile):
    """(tile, voxel, quadrant) of every instance in generation order: voxels, their
    quadrants ascending, their tiles row by row."""
    gx, gy = -(-width // tile), -(-height // tile)
    out = []
    bb = bbox.view(np.uint32).astype(np.int64)
    for v in np.nonzero(ndup)[0]:
        x0, y0, x1, y1 = bb[v, 0] >> 16, bb[v, 0] & 0xFFFF, bb[v, 1] >> 16, bb[v, 1] & 0xFFFF
        x0, x1 = (min(gx - 1, int(x) // tile) for x in (x0, x1))
        y0, y1 = (min(gy - 1, int(y) // tile) for y in (y0, y1))
        for q in range(8):
            if quad[v] >> q & 1:
                out += [(y * gx + x, v, q) for y in range(y0, y1 + 1) for x in range(x0, x1 + 1)]
    return np.array(out, np.int64).reshape(-1, 3)


def _repeat(q, levels):
    r = 0
    for _ in range(levels):
        r = r << 3 | q
    return r


def _sorted(inst, path, levels):
    rank = np.array([int(path[v]) ^ _repeat(int(q), levels) for _, v, q in inst], np.uint64)
    order = np.lexsort((rank, inst[:, 0]))  # stable: generation order breaks ties
    return inst[order], rank[order]


@pytest.mark.parametrize("n,size", [(1, (8, 8)), (31, (8, 8)), (33, (24, 8)), (300, (8, 8)), (700, (8, 8)),
                                    (1500, (16, 8)), (5000, (8, 8)), (9000, (16, 16)), (3000, (96, 80))])
def test_batched_tile_lists_are_the_stable_sort(n, size):
    """One to several thousand instances in a tile: every register width, one and
    several runs, and their merge; two views, one of them from inside."""
    sc = synthetic.config_scene("c1", seed=n, n_voxels=max(n, 200))
    keep = np.sort(np.random.default_rng(n).permutation(len(sc.octpath))[:n])
    path, centers, lengths = sc.octpath[keep], sc.centers[keep], sc.lengths[keep]
    cams = [_Cam(synthetic.make_camera(*size, 50.0, (0.1, -0.2, -1.6))),
            _Cam(synthetic.make_camera(*size, 70.0, (0.03, -0.02, 0.01), target=(0.4, 0.1, 0.3)))]
    r = BatchedRasterizer(cams, _cuda(path, torch.int64), _cuda(centers), _cuda(lengths), max_level=8, tile_size=8)
    sh0, shs = torch.zeros(n, 3).cuda(), torch.zeros(n, 15, 3).cuda()
    total = r.fit_capacity(sh0, shs, 3)
    r.prepare(sh0, shs, 3)
    count, err = r.header()
    assert err == 0 and count == total
    a = r.arrays()
    ranges, vals = a["ranges"].cpu().numpy(), a["sorted_vals"].cpu().numpy().view(np.uint32)
    ndup, bbox = a["ndup"].cpu().numpy(), a["bbox"].cpu().numpy()
    tile0 = 0
    for k, c in enumerate(cams):
        nt = -(-c.width // 8) * -(-c.height // 8)
        # the quadrant bits: those of the corners in front of the camera
        w2c, eye = c.w2c.cpu().numpy().astype(np.float32), c.c2w.cpu().numpy()[:3, 3]
        sg = np.array([[2 * (i >> 2 & 1) - 1, 2 * (i >> 1 & 1) - 1, 2 * (i & 1) - 1] for i in range(8)], np.float32)
        corners = centers[:, None] + 0.5 * lengths[:, None] * sg[None]
        front = corners @ w2c[2, :3] + w2c[2, 3] >= c.near
        neg = (corners < eye).astype(np.int64)
        bits = np.where(front, 1 << (neg[..., 0] * 4 + neg[..., 1] * 2 + neg[..., 2]), 0)
        quad = np.bitwise_or.reduce(bits, 1)
        inst, _ = _sorted(_instances(ndup[k], bbox[k], quad, c.width, c.height, 8), path, 16)
        for t in range(nt):
            a0, a1 = ranges[tile0 + t]
            want = inst[inst[:, 0] == t]
            assert a1 - a0 == len(want)
            assert np.array_equal(vals[a0:a1], (want[:, 2] << 29 | want[:, 1]).astype(np.uint32))
        tile0 += nt


@pytest.mark.parametrize("n_chains,size", [(1, (16, 16)), (40, (48, 32)), (64, (200, 136)), (300, (16, 16))])
def test_deep_keys_are_the_stable_sort(n_chains, size):
    """21-level binning: (tile, 63-bit rank) keys and their values, from one tile
    (its lowest bit shares a word with the rank) to many, short and long."""
    sc = synthetic.deep_scene(n_voxels=2000, n_chains=n_chains, seed=n_chains)
    cam = _Cam(synthetic.make_camera(*size, 60.0, (0.05, -0.1, -1.2)))
    centers, lengths, path = _cuda(sc.centers), _cuda(sc.lengths), _cuda(sc.octpath.reshape(-1, 1), torch.int64)
    n = len(sc.octpath)
    ndup, geom = dC.rasterize_preprocess(cam.width, cam.height, cam.tanfovx, cam.tanfovy, cam.cx, cam.cy, cam.w2c,
                                         cam.c2w, cam.near, path, centers, lengths)
    R, binning, *_ = dC.rasterize_voxels(1, cam.width, cam.height, cam.tanfovx, cam.tanfovy, cam.cx, cam.cy, cam.w2c,
                                         cam.c2w, 0.0, False, False, False, False, path, centers, lengths,
                                         _cuda(sc.geos), torch.zeros(n, 3).cuda(), geom)
    hi, lo, vals = dC.unpack_sorted_list(binning, R, cam.width, cam.height)
    _, _, bbox, quad = mC.unpack_geom_state(geom, n)
    inst, rank = _sorted(_instances(ndup.cpu().numpy(), bbox.cpu().numpy(), quad.cpu().numpy(), cam.width, cam.height,
                                    16), sc.octpath, 21)
    tile = inst[:, 0].astype(np.uint64)
    assert R == len(inst)
    assert np.array_equal(lo.cpu().numpy().view(np.uint64), tile << np.uint64(63) | rank)
    assert np.array_equal(hi.cpu().numpy().view(np.uint64), tile >> np.uint64(1))
    assert np.array_equal(vals.cpu().numpy().view(np.uint32), (inst[:, 2] << 29 | inst[:, 1]).astype(np.uint32))


@pytest.mark.parametrize("n,views", [(262_144, 64), (262_145, 64), (600_000, 40)])
def test_scan_of_many_pairs(n, views):
    """The radix binning's scan over (view, voxel) pairs on both sides of the 16.7M from
    which its CTAs' sums are scanned first, and past them: its total is the counts', and
    the lists are the counting sort's."""
    gen = torch.Generator(device="cuda").manual_seed(n)
    k = torch.randperm(1 << 21, device="cuda", generator=gen)[:n]
    ijk = torch.stack([k >> 14, (k >> 7) & 127, k & 127], 1)
    path = torch.zeros_like(k)
    for b in range(7):
        o = (ijk >> b) & 1
        path |= (o[:, 0] * 4 + o[:, 1] * 2 + o[:, 2]) << (3 * b)
    centers = ((ijk.float() + 0.5) / 128 - 0.5).contiguous()
    cams = [_Cam(synthetic.make_camera(40, 24, 40.0, (0.05 * v, -0.2, -2.0))) for v in range(views)]
    sh0, shs = torch.zeros(n, 3).cuda(), torch.zeros(n, 0, 3).cuda()
    got = []
    for binning in (0, 1):
        r = BatchedRasterizer(cams, path << 27, centers, torch.full((n, 1), 1 / 128, device="cuda"), max_level=7,
                              tile_size=8)
        r.set_binning(binning)
        total = r.fit_capacity(sh0, shs, 0)
        r.prepare(sh0, shs, 0)
        assert r.header() == (total, 0)
        a = r.arrays()
        assert total == int(a["ndup"].long().sum())
        got.append((a["ranges"].clone(), a["sorted_vals"][:total].clone()))
        del r
    assert torch.equal(got[0][0], got[1][0]) and torch.equal(got[0][1], got[1][1])
