"""Kernels at the sizes where they change form: lists around a staging round and
longer than the gradient rows' room, boxes under a pixel, the limits between the
backward's forms, remainders and misaligned starts of the vector kernels."""
import math

import numpy as np
import pytest
import torch

import oracle as O
from refutil import rel_err
from sv_raster_b200 import _C as mC
from sv_raster_b200 import synthetic
from sv_raster_b200.batched import BatchedRasterizer

pytestmark = pytest.mark.gpu


class _Cam:
    def __init__(self, c):
        self.__dict__.update({k: getattr(c, k) for k in ("width", "height", "tanfovx", "tanfovy", "cx", "cy", "near")})
        self.w2c, self.c2w = (torch.from_numpy(m).cuda() for m in (c.w2c, c.c2w))


class _Scene:
    """The n largest (or smallest) voxels of the small scene, in octree order."""

    def __init__(self, n, large, seed=0):
        sc = synthetic.config_scene("c1")
        by_size = np.argsort(sc.lengths.reshape(-1), kind="stable")
        keep = np.sort(by_size[-n:] if large else by_size[:n])
        r = np.random.default_rng(seed)
        t = lambda a, dt=torch.float32: torch.from_numpy(np.ascontiguousarray(a)).cuda().to(dt)
        self.n, self.max_level = n, sc.max_level
        self.path, self.centers, self.lengths, self.geos = (
            a[keep] for a in (sc.octpath, sc.centers, sc.lengths, sc.geos))
        self.sh0 = r.uniform(-1.0, 1.0, (n, 3)).astype(np.float32)
        self.rgbs = (0.28209479177387814 * self.sh0.astype(np.float64) + 0.5).astype(np.float32)
        self.d = [t(self.path.reshape(-1, 1), torch.int64), t(self.centers), t(self.lengths)]
        self.d_geos, self.d_sh0, self.d_shs = t(self.geos), t(self.sh0), torch.zeros(n, 15, 3).cuda()


def _raster(s, cams, ns=1, **kw):
    r = BatchedRasterizer([_Cam(c) for c in cams], *s.d, max_level=s.max_level, n_samp_per_vox=ns, **kw)
    r.fit_capacity(s.d_sh0, s.d_shs, 0)
    return r


def _forward_backward(r, s, dC, dT):
    r.prepare(s.d_sh0, s.d_shs, 0)
    color, T = r.render(s.d_geos)
    g = r.backward(s.d_geos, T, dC, dT, 0, 16)
    total, err = r.header()
    assert err == 0
    return color, T, g, total


# Against 64 bits.  A ray enters and leaves a voxel at t ~ 2 known to 2^-23 * 2, so
# the path through one of 1/256 is off by up to 2.4e-7 * 256 = 6e-5 of itself, both
# ways at random: the images' norm stays within 1e-4, the gradients', which also
# hold the place in the voxel (another 6e-5 for each of up to three samples), 5e-4.
@pytest.mark.parametrize("exact", [False, True])
@pytest.mark.parametrize("n,large,size,dist,ns,tile", [
    (1, True, (8, 8), 1.6, 1, 8), (63, True, (8, 8), 1.6, 1, 8), (64, True, (17, 9), 1.6, 2, 8),
    (65, True, (8, 8), 1.6, 1, 8), (129, False, (8, 8), 1.6, 1, 8), (1000, False, (8, 8), 2.0, 1, 8),
    (3000, True, (24, 8), 0.6, 3, 8), (3000, True, (40, 33), 1.2, 1, 16), (4000, False, (16, 16), 6.0, 1, 16)])
def test_batched_compositing_matches_oracle(n, large, size, dist, ns, tile, exact):
    s = _Scene(n, large, seed=n)
    cam = synthetic.make_camera(*size, 50.0, (0.1, -0.2, -dist))
    r = _raster(s, [cam], ns=ns, tile_size=tile, exact=exact)
    rng = np.random.default_rng(7)
    dC = rng.standard_normal((3, size[1], size[0])).astype(np.float32)
    dT = rng.standard_normal((1, size[1], size[0])).astype(np.float32)
    color, T, g, _ = _forward_backward(r, s, torch.from_numpy(dC).cuda().reshape(-1),
                                       torch.from_numpy(dT).cuda().reshape(-1))
    o = O.render_view(cam, s.path, s.centers, s.lengths, s.geos, s.rgbs, n_samp=ns, mode="f64")
    b = O.render_bwd(cam, o["ranges"], o["tile_last"], o["vals"], o["bbox"], s.centers, s.lengths, s.geos, s.rgbs,
                     o["n_contrib"], o["T"], dC, dT, n_samp=ns, mode="f64")
    ref = lambda a: torch.from_numpy(np.asarray(a)).cuda().reshape(-1)
    assert rel_err(color, ref(o["color"])) < 1e-4
    assert rel_err(T, ref(o["T"])) < 1e-4
    assert rel_err(g[0].reshape(-1), ref(b["dL_dgeos"])) < 5e-4
    assert rel_err(g[1].reshape(-1), ref(b["subdiv"])) < 5e-4
    assert rel_err(g[2].reshape(-1), ref(0.28209479177387814 * b["dL_drgbs"])) < 5e-4


@pytest.mark.parametrize("size,n,large,dist,broad", [
    ((600, 480), 2000, True, 1.6, True), ((600, 488), 2000, True, 1.6, True),  # 4,500 and 4,575 tiles
    ((2048, 2040), 500, True, 1.6, True), ((2048, 2048), 500, True, 1.6, True),  # 65,280 and 65,536
    ((2048, 2056), 5000, False, 6.0, False), ((2049, 2049), 3000, True, 0.7, True)])
def test_backward_forms_agree(size, n, large, dist, broad):
    """On both sides of each limit the backward with its own choice of form and
    staging adds up the same terms as the one-pixel form with rounds of 128: equal
    up to the order of the additions (1e-5, as between any two schedules)."""
    s = _Scene(n, large, seed=n)
    cam = synthetic.make_camera(*size, 50.0, (0.1, -0.2, -dist))
    gen = torch.Generator(device="cuda").manual_seed(5)
    dC = torch.randn(3 * size[0] * size[1], device="cuda", generator=gen)
    dT = torch.randn(size[0] * size[1], device="cuda", generator=gen)
    r0 = _raster(s, [cam], tile_size=8)
    r0.set_staging(32)
    r0.set_backward_staging(128)
    c0, t0, base, _ = _forward_backward(r0, s, dC, dT)
    r = _raster(s, [cam], tile_size=8)
    r.set_staging(32)
    r.set_backward_pixels_per_thread(2)
    c1, t1, got, total = _forward_backward(r, s, dC, dT)
    bb = r.arrays()["bbox"].reshape(-1, 2).long()[r.arrays()["ndup"].reshape(-1) > 0] & 0xFFFFFFFF
    px = (((bb[:, 1] >> 16) - (bb[:, 0] >> 16) + 1) * ((bb[:, 1] & 0xFFFF) - (bb[:, 0] & 0xFFFF) + 1)).sum().item()
    assert (px >= 16 * total) == broad  # the rule that picks the form on the device
    assert torch.equal(c0, c1) and torch.equal(t0, t1)
    for a, b in zip(got[:3], base[:3]):
        assert rel_err(a, b) < 1e-5


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("deg", [0, 1, 2, 3])
@pytest.mark.parametrize("n_views", [1, 2, 64])
def test_batched_colours_and_their_gradients(n_views, deg, dtype):
    """Colours of one view (coefficients read in place) and of several (held in
    registers), and the gradients' rows, against 64 bits on the stored values.  A
    colour is at most 16 terms of up to four factors, 16 * 4 * 2^-24 = 4e-6; a
    gradient sums up to 64 views of such terms, 64 * 4 * 2^-24 = 1.5e-5 at worst.
    bf16 gradients are the fp32 ones rounded once."""
    n = 1001  # not a multiple of a block, a warp or a row group
    s = _Scene(n, False, seed=3)
    rng = np.random.default_rng(deg)
    shs = torch.from_numpy(rng.standard_normal((n, 15, 3)).astype(np.float32)).cuda().to(dtype)
    sh0 = s.d_sh0.to(dtype)
    pos = [(math.cos(a) * 2.0, -0.3, math.sin(a) * 2.0) for a in np.linspace(0.1, 6.1, n_views)]
    cams = [synthetic.make_camera(24, 16, 50.0, p) for p in pos]
    r = BatchedRasterizer([_Cam(c) for c in cams], *s.d, max_level=s.max_level)
    r.fit_capacity(sh0, shs, deg)
    r.prepare(sh0, shs, deg)
    a = r.arrays()
    rgbs, ndup = a["rgbs"].reshape(n_views, n, 3).clone(), a["ndup"].reshape(n_views, n).cpu().numpy()
    n0, ns_ = sh0.float().cpu().numpy(), shs.float().cpu().numpy()
    color, T = r.render(s.d_geos)
    dC = torch.from_numpy(rng.standard_normal(color.numel()).astype(np.float32)).cuda()
    g = r.backward(s.d_geos, T, dC, torch.zeros_like(T), deg, 16)
    d_rgb = r.arrays()["drgbs"][..., :3].cpu().numpy()
    want0, wants = np.zeros((n, 3)), np.zeros((n, 15, 3))
    for v, c in enumerate(cams):
        vis = np.nonzero(ndup[v])[0]
        eye = c.c2w[:3, 3]
        o = O.sh_fwd(deg, vis, s.centers, eye, n0, ns_, mode="f64")
        assert rel_err(rgbs[v][vis], torch.from_numpy(o[vis]).cuda()) < 1e-5
        d0, ds = O.sh_bwd(deg, 16, vis, s.centers, eye, d_rgb[v], mode="f64")
        want0 += d0
        wants += ds
    assert rel_err(g[2], torch.from_numpy(want0).cuda()) < 2e-5
    assert rel_err(g[3].reshape(-1), torch.from_numpy(wants).cuda().reshape(-1)) < 2e-5
    b0, bs = torch.empty_like(g[2], dtype=torch.bfloat16), torch.empty_like(g[3], dtype=torch.bfloat16)
    r.backward_sh(deg, 16, b0, bs)
    f0, fs = torch.empty_like(g[2]), torch.empty_like(g[3])
    r.backward_sh(deg, 16, f0, fs)
    assert torch.equal(b0, f0.bfloat16()) and torch.equal(bs, fs.bfloat16())


@pytest.mark.parametrize("deg,M", [(0, 1), (1, 4), (2, 16), (3, 16)])
@pytest.mark.parametrize("n_idx", [1, 31, 33, 129, 1000])
def test_plain_sh_on_unsorted_part(n_idx, deg, M):
    """Rows of the colours and of their gradients for an unsorted part of the
    voxels: 16 terms of up to four factors against 64 bits (4e-6, bound 1e-5);
    rows outside stay zero."""
    P = 1000
    rng = np.random.default_rng(n_idx + deg)
    centers = rng.uniform(-0.5, 0.5, (P, 3)).astype(np.float32)
    sh0, shs = (rng.standard_normal(sh).astype(np.float32) for sh in ((P, 3), (P, M - 1, 3)))
    eye, d = np.array([0.3, -0.2, -1.7], np.float32), rng.standard_normal((P, 3)).astype(np.float32)
    idx = rng.permutation(P)[:n_idx]
    t = lambda a: torch.from_numpy(a).cuda()
    rgb = mC.sh_compute(deg, t(idx), t(centers), t(eye), t(sh0), t(shs))
    o = O.sh_fwd(deg, idx, centers, eye, sh0, shs, mode="f64")
    assert rel_err(rgb, t(o)) < 1e-5
    g0, gs = mC.sh_compute_bw(deg, M, t(idx), t(centers), t(eye), rgb, t(d))
    d0, ds = O.sh_bwd(deg, M, idx, centers, eye, d, mode="f64")
    assert rel_err(g0, t(d0)) < 1e-5
    assert rel_err(gs.reshape(-1), t(ds).reshape(-1)) < 1e-5
    out = np.setdiff1d(np.arange(P), idx)
    assert not rgb[out].any() and not g0[out].any() and not gs[out].any()


@pytest.mark.parametrize("sparse,biased", [(False, False), (True, False), (True, True)])
@pytest.mark.parametrize("n,offset", [(1, 0), (3, 0), (4, 0), (5, 0), (1023, 0), (4097, 0), (5, 1), (4096, 1), (4097, 3)])
def test_adam_remainders_and_misaligned_starts(n, offset, sparse, biased):
    """Whole groups of four, remainders, and tensors that start off a 16-byte
    boundary give one result, that of 64 bits within a few roundings of the
    parameter (|p| < 6: 6 * 4 * 2^-24 < 2e-6), and leave their neighbours alone."""
    rng = np.random.default_rng(n)
    host = [rng.standard_normal(n).astype(np.float32) for _ in range(3)] + [rng.uniform(0.1, 1.0, n).astype(np.float32)]
    host[1][::3] = 0.0
    run = mC.biased_adam_step if biased else mC.unbiased_adam_step
    step = () if biased else (5,)

    def go(off):
        whole = [torch.full((n + 8,), 7.0, device="cuda") for _ in host]
        parts = [w[off:off + n] for w in whole]
        for p, h in zip(parts, host):
            p.copy_(torch.from_numpy(h))
        run(sparse, *parts, *step, 0.02, 0.9, 0.99, 1e-8)
        assert all((w[:off] == 7.0).all() and (w[off + n:] == 7.0).all() for w in whole)
        return [parts[i].clone() for i in (0, 2, 3)]

    got, aligned = go(offset), go(0)
    assert all(torch.equal(a, b) for a, b in zip(got, aligned))
    want = O.adam(host[0], host[1], host[2], host[3], 5, 0.02, 0.9, 0.99, 1e-8, biased=biased, sparse=sparse, mode="f64")
    for a, w in zip(got, want):
        assert np.abs(a.cpu().numpy() - w).max() < 2e-6


@pytest.mark.parametrize("sparse", [False, True])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("sizes", [(1, 7, 4096), (8 << 20,), ((8 << 20) - 2, 3), ((8 << 20) + 2051, 5, 1023)])
def test_fused_adam_equals_single_groups(sizes, dtype, sparse):
    """Several groups in one launch, kept in the cache or streamed past it, with
    remainders: the same bits as each group by itself (bf16: on the stored values,
    rounded once)."""
    from sv_raster_b200.sparse_adam import FusedSparseAdam, SparseAdam
    gen = torch.Generator(device="cuda").manual_seed(sum(sizes))
    draw = lambda n: torch.randn(n, device="cuda", generator=gen)
    one = [draw(n).to(dtype).requires_grad_(True) for n in sizes]
    ref = [p.detach().float().requires_grad_(True) for p in one]
    for p, q in zip(one, ref):
        g = draw(p.numel())
        g[::3] = 0.0
        g[: p.numel() // 2] = 0.0  # whole groups of four without a gradient
        p.grad_dtype = torch.float32  # parameters in 16 bits keep their gradients in 32
        p.grad, q.grad = g, g.clone()
    a = FusedSparseAdam([{"params": [p], "lr": 0.01 * (k + 1)} for k, p in enumerate(one)], sparse=sparse)
    b = SparseAdam([{"params": [q], "lr": 0.01 * (k + 1)} for k, q in enumerate(ref)], sparse=sparse)
    a.step()
    b.step()
    for p, q in zip(one, ref):
        assert torch.equal(p.detach(), q.detach().to(dtype))
        assert torch.equal(a.state[p]["exp_avg"], b.state[q]["exp_avg"])
        assert torch.equal(a.state[p]["exp_avg_sq"], b.state[q]["exp_avg_sq"])
