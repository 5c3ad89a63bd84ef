"""Tile lists of so many instances that their sorted runs are merged by windows: against
a stable sort, for the counting sort's rank positions, for keys with values (radix
binning, 16 levels) and for 21-level keys, with equal keys among them."""
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


def _level(n):
    """The coarsest grid, 128^3 and up, with n cells."""
    return next(lv for lv in range(7, 16) if n <= 1 << (3 * lv))


def _cells(n, seed):
    """n cells of that grid in random order: (octree path of 16 levels, of 21, centres,
    lengths)."""
    gen, lv = torch.Generator(device="cuda").manual_seed(seed), _level(n)
    k = torch.randperm(1 << (3 * lv), device="cuda", generator=gen)[:n]
    ijk = torch.stack([k >> (2 * lv), (k >> lv) & ((1 << lv) - 1), k & ((1 << lv) - 1)], 1)
    path = torch.zeros_like(k)
    for b in range(lv):
        oct_ = ((ijk >> b) & 1)
        path |= (oct_[:, 0] * 4 + oct_[:, 1] * 2 + oct_[:, 2]) << (3 * b)
    centers = ((ijk.float() + 0.5) / (1 << lv) - 0.5).contiguous()
    return (path << (3 * (16 - lv)), path << (3 * (21 - lv)), centers,
            torch.full((n, 1), 1.0 / (1 << lv), device="cuda"))


def _sorted_by(tile, rank):
    """Stable order by (tile, rank): two stable sorts."""
    order = torch.sort(rank, stable=True).indices
    return order[torch.sort(tile[order], stable=True).indices]


def _ranks(path, vals, levels):
    """Morton rank of each instance (quadrant | voxel in vals): the path with every
    octant flipped by the quadrant."""
    vals = vals.long() & 0xFFFFFFFF
    q, v = vals >> 29, vals & ((1 << 29) - 1)
    rep = torch.zeros_like(q)
    for _ in range(levels):
        rep = rep << 3 | q
    return path[v] ^ rep


# around the number of runs (16 of 2,048 positions; 16 of 4,096 keys, or of 2,048) from
# which windows merge, whole and partial last runs, hundreds of runs, and more (2,816 of
# positions, 2,432 of 2,048 keys) than a window keeps track of
SIZES = [18_432, 32_768, 32_769, 40_000, 65_536, 65_537, 400_000, 1_500_000, 6_500_000]


@pytest.mark.parametrize("n", SIZES)
def test_one_tile_of_all_voxels(n):
    """A view of one 8x8 tile that sees every voxel from outside: the counting sort's and
    the radix binning's lists, both against the stable order of the (voxel, quadrant)
    pairs."""
    path, _, centers, lengths = _cells(n, n)
    cam = _Cam(synthetic.make_camera(8, 8, 40.0, (0.3, -0.2, -3.0)))
    sh0, shs = torch.zeros(n, 3).cuda(), torch.zeros(n, 0, 3).cuda()
    lists = []
    for binning, buckets in ((1, (512, 4096)), (0, (512, 4096)), (0, (512, 2048))):
        r = BatchedRasterizer([cam], path, centers, lengths, max_level=_level(n), tile_size=8)
        r.set_culling(0)
        r.set_binning(binning)
        r.set_sort_buckets(*buckets)
        total = r.fit_capacity(sh0, shs, 0)
        assert total >= n
        r.prepare(sh0, shs, 0)
        assert r.header() == (total, 0)
        assert r.arrays()["ranges"].tolist() == [[0, total]]
        lists.append(r.arrays()["sorted_vals"][:total].clone())
    assert torch.equal(lists[0], lists[1]) and torch.equal(lists[0], lists[2])
    vals = lists[0].long() & 0xFFFFFFFF
    rank = _ranks(path, lists[0], 16)
    assert (rank[1:] >= rank[:-1]).all()
    # every voxel once per quadrant of its corners; equal ranks in order of voxel, then quadrant
    pair = (vals & ((1 << 29) - 1)) * 8 + (vals >> 29)
    assert torch.unique(pair).numel() == total
    assert (torch.unique(pair >> 3) == torch.arange(n, device="cuda")).all()
    same = rank[1:] == rank[:-1]
    assert (pair[1:][same] > pair[:-1][same]).all()


@pytest.mark.parametrize("levels", [16, 21])
@pytest.mark.parametrize("n,size,dist,twice", [
    (25_000, (16, 16), 3.0, True), (32_700, (16, 16), 3.0, False), (65_536, (16, 16), 3.0, False),
    (70_000, (16, 16), 3.0, True), (400_000, (16, 16), 3.0, False), (300_000, (32, 16), 3.0, True),
    (150_000, (512, 16), 60.0, False), (200_000, (512, 16), 60.0, True),
    (21_500_000, (16, 16), 3.0, True)])  # more runs (5,152 of 4,096 keys) than a window keeps track of
def test_keys_with_values_are_the_stable_sort(levels, n, size, dist, twice):
    """Single views of one and two 16x16 tiles, and of 32 of which two hold everything.
    `twice`: half of the voxels have another's path, so equal keys must keep the order in
    which they were generated.  21 levels: by tile first and (from 32,768 instances per
    tile on average) by rank first."""
    path16, path21, centers, lengths = _cells(n, n + 1)
    path = path16 if levels == 16 else path21
    if twice:
        path = path[torch.arange(n, device="cuda") // 2 * 2].contiguous()
    C = mC if levels == 16 else dC
    cam = _Cam(synthetic.make_camera(*size, 40.0, (0.3, -0.2, -dist)))
    a = (cam.width, cam.height, cam.tanfovx, cam.tanfovy, cam.cx, cam.cy, cam.w2c, cam.c2w)
    p = path.reshape(-1, 1)
    ndup, geom = C.rasterize_preprocess(*a, cam.near, p, centers, lengths)
    R, binning, *_ = C.rasterize_voxels(1, *a, 0.0, False, False, False, False, p, centers, lengths,
                                        torch.full((n, 8), 5.0, device="cuda"), torch.zeros(n, 3).cuda(), geom)
    got = C.unpack_sorted_list(binning, R, cam.width, cam.height)[-1].long() & 0xFFFFFFFF
    # the instances in generation order: voxels, quadrants, tiles row by row
    _, _, bbox, quad = mC.unpack_geom_state(geom, n)
    bb = bbox.long() & 0xFFFFFFFF
    gx = -(-cam.width // 16)
    x0, x1 = ((bb[:, k] >> 16) // 16 for k in (0, 1))
    x1 = x1.clamp(max=gx - 1)
    v = torch.arange(n, device="cuda")
    cand = [(v, q, t) for q in range(8) for t in range(gx)]
    vox = torch.cat([c[0] for c in cand])
    q = torch.cat([torch.full_like(v, c[1]) for c in cand])
    t = torch.cat([torch.full_like(v, c[2]) for c in cand])
    on = ((quad.long()[vox] >> q) & 1 > 0) & (x0[vox] <= t) & (t <= x1[vox]) & (ndup.long()[vox] > 0)
    vox, q, t = vox[on], q[on], t[on]
    gen = torch.sort((vox * 8 + q) * gx + t).indices
    vox, q, t = vox[gen], q[gen], t[gen]
    vals = q << 29 | vox
    assert R == vals.numel()
    assert torch.equal(got, vals[_sorted_by(t, _ranks(path.reshape(-1), vals, levels))])


@pytest.mark.parametrize("capacity", [None, 50_000])
@pytest.mark.parametrize("sizes,n", [([(24, 16)], 65_535), ([(24, 16)], 65_536), ([(320, 160)], 204_799),
                                     ([(320, 160)], 204_800), ([(24, 16), (8, 8), (40, 24)], 70_000),
                                     ([(24, 16), (40, 24)], 300_000), ([(256, 256)], 600_000),
                                     ([(720, 360)], 1_100_000), ([(8, 8), (360, 200)], 150_000)])
def test_copies_of_the_counts(sizes, n, capacity):
    """On both sides of 65,536 voxels and of 256 per tile, from where the counting sort's
    counts and cursors are kept in copies: the lists of the radix binning, and within a
    capacity that is too small lists that keep to it, with the error word set."""
    path, _, centers, lengths = _cells(n, n + 2)
    cams = [_Cam(synthetic.make_camera(*s, 30.0, (0.3 - 0.2 * k, -0.2, -2.0))) for k, s in enumerate(sizes)]
    sh0, shs = torch.zeros(n, 3).cuda(), torch.zeros(n, 0, 3).cuda()
    got = []
    for binning in (1, 0):
        r = BatchedRasterizer(cams, path, centers, lengths, max_level=_level(n), tile_size=8, capacity=capacity)
        r.set_culling(0)
        r.set_binning(binning)
        if capacity is None:
            r.fit_capacity(sh0, shs, 0)
        r.prepare(sh0, shs, 0)
        total, err = r.header()
        a = r.arrays()
        if capacity is not None and total > capacity:
            assert err == 4  # capacity
            if binning:
                rg = a["ranges"].long()
                assert (rg[:, 1] <= capacity).all() and (rg[:, 1] - rg[:, 0]).sum() == capacity
            continue
        assert err == 0
        got.append((a["ranges"].clone(), a["sorted_vals"][:total].clone()))
    if got:
        assert torch.equal(got[0][0], got[1][0]) and torch.equal(got[0][1], got[1][1])
