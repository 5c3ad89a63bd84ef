"""Workloads of the rasterizer whose speed is measured, each one pass through
its public entry points: multi-view training and evaluation steps
(``batched``), single-view drop-in renders (``view``), the grid-point
parameters of the reference's training loop (``gridpoints``) and the optimizer
step (``adam``).

``listed()`` gives the fixed cases, ``draw(rng)`` more of the same ranges,
``prepare(case, seed)`` what a program holds before the call (seeded scenes on
the GPU with the distributions of ``sv_raster_b200.synthetic``), ``run(state)``
one pass, ``work(case)`` the bytes and operations it cannot do without and
``exact(case, seed)`` the outputs of that pass evaluated in 64 bits by plain
torch.
"""
import math
from types import SimpleNamespace

import numpy as np
import torch

DEV = "cuda"
NEAR = 0.02
BG_LEVELS = (5, 7)


# ---------------------------------------------------------------------------
# cases
# ---------------------------------------------------------------------------
def _batched(name, **kw):
    c = dict(kind="batched", scene="mixed", l0=8, l1=12, voxels=2_000_000, views=1, width=1297, height=840,
             uneven=False, rmin=1.6, rmax=1.6, dtype="bf16", n_samp=1, sh_degree=3, backward=True, grid=False)
    c.update(kw)
    return dict(c, name=name) if name else c


def _view(name, **kw):
    c = dict(kind="view", scene="mixed", l0=8, l1=12, voxels=2_000_000, width=1297, height=840, rmin=1.6, rmax=1.6,
             levels=16, n_samp=1, sh_degree=3, backward=True, depth=False, normal=False, max_w=False, dist=0.0,
             concen=0.0, ascending=0.0, bg=0.0)
    c.update(kw)
    return dict(c, name=name) if name else c


def _gridpoints(name, **kw):
    c = dict(kind="gridpoints", scene="mixed", l0=8, l1=12, voxels=2_000_000, channels=1, tv_sparse=False)
    c.update(kw)
    return dict(c, name=name) if name else c


def _adam(name, **kw):
    c = dict(kind="adam", voxels=2_000_000, fused=False, dtype="fp32", sparse=True, touched=0.4, sh_degree=3)
    c.update(kw)
    return dict(c, name=name) if name else c


def listed():
    return [
        # a training step on a small object, three thumbnails: launches and latency
        _batched("step-tiny", scene="sphere", l0=6, l1=8, voxels=20_000, views=3, width=256, height=200, rmin=1.5,
                 rmax=1.5, dtype="fp32"),
        # the ordinary single-view training step of a 2M-voxel scene
        _batched("step-one-view"),
        # one step over many cameras of uneven resolution, seen from farther away
        _batched("step-uneven-views", views=16, width=1600, height=1200, uneven=True, rmin=2.0, rmax=4.0),
        # the largest scene with eight full-HD views per step
        _batched("step-full-hd", l0=8, l1=14, voxels=8_000_000, views=8, width=1920, height=1080, rmin=1.5, rmax=2.0),
        # training the reference's own parametrisation, densities on grid points, four views per step
        _batched("step-grid-points", l0=8, l1=12, voxels=1_000_000, views=4, width=1007, height=755, rmin=1.5,
                 rmax=2.5, dtype="fp32", grid=True),
        # evaluation renders of a trained scene at three samples per voxel, no gradients
        _batched("eval-views", voxels=1_500_000, views=6, width=1280, height=720, rmin=1.5, rmax=2.0, dtype="fp32",
                 n_samp=3, backward=False),
        # the drop-in training iteration: one view per call, colour concentration on
        _view("view-train", concen=0.01),
        # the same from inside the scene with every regulariser and output, octrees 21 levels deep
        _view("view-regularised", l0=10, l1=15, levels=21, voxels=300_000, width=801, height=601, rmin=0.3, rmax=0.3,
              n_samp=2, depth=True, normal=True, dist=0.1, concen=0.01, ascending=0.01, bg=1.0),
        # an interactive viewer's frame: depth and normal maps, per-voxel maximum weight, no gradients
        _view("view-frame", voxels=700_000, width=960, height=540, rmin=1.5, rmax=1.5, backward=False, depth=True,
              normal=True, max_w=True),
        # a thumbnail of a small object, forward and backward: latency of the drop-in calls
        _view("view-tiny", scene="sphere", l0=6, l1=8, voxels=20_000, width=200, height=136, rmin=1.5, rmax=1.5),
        # the grid-point part of a training iteration: gather, its backward and the total-variation gradient
        _gridpoints("grid-gather-tv"),
        # the optimizer's step over all parameters of a 2M-voxel scene, untouched voxels skipped
        _adam("adam-sparse"),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["batched", "batched", "batched", "view", "view", "gridpoints", "adam"])
    n = _log(rng, 20_000, 4_000_000)
    l0, l1 = (6, 8) if n < 60_000 else rng.choice([(8, 12), (8, 12), (8, 14), (9, 13)])
    scene = "sphere" if n < 60_000 else "mixed"
    rmin = round(rng.uniform(1.2, 2.5), 2)
    geo = dict(scene=scene, l0=l0, l1=l1, voxels=n)
    deg = rng.choice([3, 3, 3, 2, 1, 0])
    if kind == "batched":
        views = _log(rng, 1, 12)
        width = _log(rng, 120, min(1920, int(math.sqrt(6e6 / views * 1.5))))
        back = rng.random() < 0.8
        return _batched(None, **geo, views=views, width=width, height=max(48, int(width * rng.uniform(0.5, 0.9))),
                        uneven=rng.random() < 0.3, rmin=rmin, rmax=round(rmin + rng.uniform(0.0, 1.0), 2),
                        dtype=rng.choice(["bf16", "fp32"]), n_samp=rng.choice([1, 1, 1, 2, 3]), sh_degree=deg,
                        backward=back, grid=back and n <= 2_000_000 and rng.random() < 0.3)
    if kind == "view":
        width = _log(rng, 120, 1600)
        extra = rng.random() < 0.5
        return _view(None, **geo, width=width, height=max(48, int(width * rng.uniform(0.5, 0.9))), rmin=rmin, rmax=rmin,
                     levels=rng.choice([16, 16, 16, 21]), n_samp=rng.choice([1, 1, 2, 3]), sh_degree=deg,
                     backward=rng.random() < 0.7, depth=extra, normal=extra and rng.random() < 0.7,
                     max_w=rng.random() < 0.3, dist=rng.choice([0.0, 0.1]) if extra else 0.0,
                     concen=rng.choice([0.0, 0.01]), ascending=rng.choice([0.0, 0.0, 0.01]), bg=rng.choice([0.0, 1.0]))
    if kind == "gridpoints":
        return _gridpoints(None, **geo, channels=rng.choice([1, 1, 3]), tv_sparse=rng.random() < 0.5)
    fused = rng.random() < 0.5
    return _adam(None, voxels=n, fused=fused, dtype=rng.choice(["fp32", "bf16"]) if fused else "fp32",
                 sparse=rng.random() < 0.7, touched=round(rng.uniform(0.1, 1.0), 2), sh_degree=deg)


# ---------------------------------------------------------------------------
# seeded scenes on the GPU (the distributions of sv_raster_b200.synthetic)
# ---------------------------------------------------------------------------
class _Rand:
    def __init__(self, seed):
        self.g = torch.Generator(device=DEV).manual_seed(int(seed))

    def uniform(self, *shape, lo=0.0, hi=1.0, dtype=torch.float32):
        return torch.rand(*shape, device=DEV, generator=self.g, dtype=dtype) * (hi - lo) + lo

    def normal(self, *shape, dtype=torch.float32):
        return torch.randn(*shape, device=DEV, generator=self.g, dtype=dtype)

    def perm(self, n):
        return torch.randperm(n, device=DEV, generator=self.g)


def _unit(v):
    return v / v.norm(dim=-1, keepdim=True)


def _points(r, what, m, surf):
    f64 = torch.float64
    if what == "sphere":
        return _unit(r.normal(m, 3, dtype=f64)) * (0.4 + 0.02 * r.normal(m, 1, dtype=f64))
    if what == "surf":
        k = (r.uniform(m) * 3).long().clamp(max=2)
        return surf[0][k] + _unit(r.normal(m, 3, dtype=f64)) * (surf[1][k][:, None] + 0.01 * r.normal(m, 1, dtype=f64))
    p = r.uniform(3 * m, 3, lo=-0.5, hi=0.5, dtype=f64)  # the cube shell 0.36 < |p|_inf < 0.5
    return p[p.abs().amax(1) > 0.36][:m]


def _region_level(p, l0, l1, salt):
    side = 1 << l0
    c = ((p + 0.5) * side).floor().long().clamp(0, side - 1)
    h = (c[:, 0] * 73856093) ^ (c[:, 1] * 19349663) ^ (c[:, 2] * 83492791) ^ salt
    h = (h ^ (h >> 13)) * 0x5BD1E995
    return l0 + ((h ^ (h >> 15)) & 0x7FFFFFFF) % (l1 - l0 + 1)


def _cells(r, what, want, l0, l1, salt, surf):
    """`want` distinct octree cells (i, j, k, level) around the sampled points (fewer where the levels hold fewer)."""
    keys = torch.zeros(0, dtype=torch.int64, device=DEV)
    m = max(4096, int(1.3 * want))
    for _ in range(8):
        p = _points(r, what, m, surf).clamp(-0.5 + 1e-7, 0.5 - 1e-7)
        lv = _region_level(p, l0, l1, salt)
        side = torch.ones_like(lv) << lv
        c = ((p + 0.5) * side[:, None]).floor().long()
        before = keys.numel()
        keys = torch.unique(torch.cat([keys, (lv << 52) | (c[:, 0] * side * side + c[:, 1] * side + c[:, 2])]))
        if keys.numel() >= want or keys.numel() < 1.02 * before:
            break
    keys = keys[r.perm(keys.numel())[:want]]
    lv = keys >> 52
    idx = keys & ((1 << 52) - 1)
    side = torch.ones_like(lv) << lv
    return torch.stack([idx // (side * side), (idx // side) % side, idx % side], 1), lv


def _scene(case, r, levels=16):
    """Octree voxels and their parameters: a jittered sphere, or three surfaces and a background shell."""
    n = case["voxels"]
    params = r
    if case["kind"] == "gridpoints" or case.get("grid"):
        r = _Rand(n)  # one octree per case: the number of its grid points is the size of the outputs
    surf = (r.uniform(3, 3, lo=-0.08, hi=0.08, dtype=torch.float64), r.uniform(3, lo=0.1, hi=0.18, dtype=torch.float64))
    if case["scene"] == "sphere":
        ijk, lv = _cells(r, "sphere", n, case["l0"], case["l1"], 7, surf)
    else:
        bi, bl = _cells(r, "bg", int(0.3 * n), *BG_LEVELS, 11, surf)
        si, sl = _cells(r, "surf", n - bi.shape[0], case["l0"], case["l1"], 13, surf)
        ijk, lv = torch.cat([bi, si]), torch.cat([bl, sl])
    p = r.perm(lv.numel())
    ijk, lv = ijk[p], lv[p]
    path = torch.zeros_like(lv)
    for b in range(levels):
        path |= ((((ijk[:, 0] >> b) & 1) << 2) | (((ijk[:, 1] >> b) & 1) << 1) | ((ijk[:, 2] >> b) & 1)) << (3 * b)
    path = path << (3 * (levels - lv))
    size = torch.ldexp(torch.ones_like(lv, dtype=torch.float64), -lv)[:, None]
    s = SimpleNamespace(ijk=ijk, lv=lv, path=path.reshape(-1, 1).contiguous(), lengths=size.float().contiguous(),
                        centers=(-0.5 + (ijk + 0.5) * size).float().contiguous(), P=lv.numel(), r=params)
    s.mu, s.sd = (-1.0, 1.0) if case["scene"] == "sphere" else (-2.0, 1.5)
    return s


def _params(case, s, dtype=torch.float32):
    m = (case["sh_degree"] + 1) ** 2
    s.geos = (s.mu + s.sd * s.r.normal(s.P, 8)).to(dtype)
    s.sh0 = (0.2 * s.r.normal(s.P, 3)).to(dtype)
    s.shs = (0.2 * s.r.normal(s.P, m - 1, 3)).to(dtype)


def _grid_keys(s, levels=16):
    """Corner-point indices [P,8] into the deduplicated grid points of the voxels, and their number."""
    shift = levels - s.lv
    code = torch.zeros(s.P, 8, dtype=torch.int64, device=DEV)
    for a in range(3):
        off = torch.tensor([(c >> (2 - a)) & 1 for c in range(8)], device=DEV)
        code = (code << 17) | ((s.ijk[:, a:a + 1] + off) << shift[:, None])
    uniq, inv = torch.unique(code.reshape(-1), return_inverse=True)
    return inv.reshape(-1, 8).contiguous(), uniq.numel()


class _Cam:
    """A pinhole camera as the entry points take it (float values as 32 bits hold them)."""

    def __init__(self, w, h, fov, pos, target):
        f32 = lambda x: float(np.float32(x))  # noqa: E731
        self.width, self.height, self.near = int(w), int(h), NEAR
        self.tanfovx = f32(math.tan(math.radians(fov) * 0.5))
        self.tanfovy = f32(self.tanfovx * h / w)
        self.cx, self.cy = w * 0.5, h * 0.5
        fwd = target - pos
        fwd = fwd / np.linalg.norm(fwd)
        right = np.cross(fwd, np.array([0.0, -1.0, 0.0]))
        right /= np.linalg.norm(right)
        c2w = np.eye(4)
        c2w[:3, 0], c2w[:3, 1], c2w[:3, 2], c2w[:3, 3] = right, np.cross(fwd, right), fwd, pos
        self.c2w = torch.from_numpy(c2w.astype(np.float32)).to(DEV)
        self.w2c = torch.from_numpy(np.linalg.inv(c2w).astype(np.float32)).to(DEV)


def _cameras(case, seed):
    rng = np.random.default_rng(seed + 1)
    size = np.random.default_rng(17)  # a rig's resolutions belong to the case
    cams = []
    for _ in range(case.get("views", 1)):
        d = rng.standard_normal(3)
        d[1] = np.clip(d[1], -0.9 * np.linalg.norm(d[[0, 2]]), 0.9 * np.linalg.norm(d[[0, 2]]))
        k = size.uniform(0.4, 1.0) if case.get("uneven") else 1.0
        w, h = int(case["width"] * k), int(case["height"] * k)
        target = rng.uniform(-0.05, 0.05, 3)
        cams.append(_Cam(w, h, 50.0, d / np.linalg.norm(d) * rng.uniform(case["rmin"], case["rmax"]), target))
    return cams


# ---------------------------------------------------------------------------
# what a program has in hand, and one pass
# ---------------------------------------------------------------------------
def _batched_inputs(case, seed):
    r = _Rand(seed)
    s = _scene(case, r)
    dtype = torch.bfloat16 if case["dtype"] == "bf16" else torch.float32
    _params(case, s, dtype)
    if case["grid"]:
        s.key, m = _grid_keys(s)
        s.grid = (s.mu + s.sd * r.normal(m)).to(dtype)
    s.cams = _cameras(case, seed)
    pix = sum(c.width * c.height for c in s.cams)
    # the gradient of a mean squared error against a target image
    s.dC = r.uniform(3 * pix, lo=-1.0, hi=1.0) * (2.0 / (3 * pix))
    return s


def _prepare_batched(case, seed):
    from sv_raster_b200.batched import BatchedRasterizer
    s = _batched_inputs(case, seed)
    level = int(s.lv.max())
    raster = BatchedRasterizer(s.cams, s.path, s.centers, s.lengths, max_level=level, n_samp_per_vox=case["n_samp"],
                               tile_size=8)
    # the launch parameters that the autotuner arrives at for these scenes
    raster.set_staging(64)
    raster.set_backward_staging(32)
    raster.set_backward_pixels_per_thread(2)
    raster.fit_capacity(s.sh0, s.shs, case["sh_degree"])
    dens = s.grid if case["grid"] else s.geos
    st = SimpleNamespace(case=case, raster=raster, key=s.key if case["grid"] else None, dens=dens, sh0=s.sh0,
                         shs=s.shs, dC=s.dC)
    if case["backward"]:
        for t in (st.dens, st.sh0, st.shs):
            t.requires_grad_(True)
    return st


def _run_batched(st):
    from sv_raster_b200.batched import BatchedRender, GridBatchedRender
    c = st.case
    if not c["backward"]:
        with torch.no_grad():
            return dict(zip(("color", "T"), BatchedRender.apply(st.raster, c["sh_degree"], st.dens, st.sh0, st.shs)))
    if c["grid"]:
        color, T = GridBatchedRender.apply(st.raster, c["sh_degree"], st.key, st.dens, st.sh0, st.shs)
    else:
        color, T = BatchedRender.apply(st.raster, c["sh_degree"], st.dens, st.sh0, st.shs)
    g = torch.autograd.grad(color, (st.dens, st.sh0, st.shs), st.dC)
    return {"color": color.detach(), "T": T.detach(), "ddens": g[0], "dsh0": g[1], "dshs": g[2]}


def _view_inputs(case, seed):
    r = _Rand(seed)
    s = _scene(case, r, case["levels"])
    _params(case, s)
    s.cams = _cameras(case, seed)
    h, w = s.cams[0].height, s.cams[0].width
    s.gt = r.uniform(3, h, w)
    s.dC = r.uniform(3, h, w, lo=-1.0, hi=1.0) * (2.0 / (3 * h * w))
    s.dD = r.uniform(3, h, w, lo=-1.0, hi=1.0) * (0.1 / (h * w))
    s.dD[1:] = 0.0  # a loss on the mean depth (the distortion and median channels carry none)
    s.dN = r.uniform(3, h, w, lo=-1.0, hi=1.0) * (0.1 / (h * w))
    return s


def _prepare_view(case, seed):
    s = _view_inputs(case, seed)
    if case["levels"] == 21:
        from sv_raster_b200.levels21 import renderer
    else:
        from sv_raster_b200 import renderer
    cam = s.cams[0]
    settings = renderer.RasterSettings(
        color_mode="sh", n_samp_per_vox=case["n_samp"], image_width=cam.width, image_height=cam.height,
        tanfovx=cam.tanfovx, tanfovy=cam.tanfovy, cx=cam.cx, cy=cam.cy, w2c_matrix=cam.w2c, c2w_matrix=cam.c2w,
        bg_color=case["bg"], near=NEAR, need_depth=case["depth"], need_normal=case["normal"],
        track_max_w=case["max_w"], lambda_R_concen=case["concen"], lambda_ascending=case["ascending"],
        lambda_dist=case["dist"], gt_color=s.gt)
    s.subdiv = torch.ones(s.P, 1, device=DEV)
    if case["backward"]:
        for t in (s.geos, s.sh0, s.shs, s.subdiv):
            t.requires_grad_(True)
    return SimpleNamespace(case=case, s=s, settings=settings, renderer=renderer)


def _run_view(st):
    c, s, renderer = st.case, st.s, st.renderer

    def vox_fn(idx, cam_pos, color_mode):
        rgbs = renderer.SH_eval.apply(c["sh_degree"], idx, s.centers, cam_pos, None, s.sh0, s.shs)
        return {"geos": s.geos, "rgbs": rgbs, "subdiv_p": s.subdiv}

    def call():
        return renderer.rasterize_voxels(st.settings, s.path, s.centers, s.lengths, vox_fn)

    if not c["backward"]:
        with torch.no_grad():
            color, depth, normal, T, max_w = call()
    else:
        color, depth, normal, T, max_w = call()
    out = {"color": color, "T": T}
    outs, ups = [color], [s.dC]
    if c["depth"] or c["dist"] > 0:
        out["depth"] = depth
    if c["depth"]:
        outs.append(depth)
        ups.append(s.dD)
    if c["normal"]:
        out["normal"] = normal
        outs.append(normal)
        ups.append(s.dN)
    if c["max_w"]:
        out["max_w"] = max_w
    if c["backward"]:
        g = torch.autograd.grad(outs, (s.geos, s.sh0, s.shs, s.subdiv), ups)
        out.update(zip(("dgeos", "dsh0", "dshs", "dsubdiv"), g))
    return {k: v.detach() for k, v in out.items()}


def _gridpoint_inputs(case, seed):
    r = _Rand(seed)
    s = _scene(case, r)
    s.key, m = _grid_keys(s)
    c = case["channels"]
    s.pts = s.mu + s.sd * r.normal(m, c)
    s.care = torch.arange(s.P, device=DEV)
    s.dvox = r.normal(s.P, 8) * 1e-6 if c == 1 else r.normal(s.P, 8, c) * 1e-6
    # a view touches part of the voxels: the others bring no gradient
    seen = r.uniform(s.P) < 0.4
    s.dvox = torch.where(seen[(...,) + (None,) * (s.dvox.dim() - 1)], s.dvox, torch.zeros_like(s.dvox))
    s.size_inv = 1.0 / s.lengths
    s.weight = 1e-7
    return s


def _prepare_gridpoints(case, seed):
    s = _gridpoint_inputs(case, seed)
    s.case = case
    s.pts.requires_grad_(True)
    return s


def _run_gridpoints(s):
    from sv_raster_b200.grid_loss_bw import total_variation
    from sv_raster_b200.renderer import GatherFeatParams, GatherGeoParams
    fn = GatherGeoParams if s.case["channels"] == 1 else GatherFeatParams
    vox = fn.apply(s.key, s.care, s.pts)
    (grad,) = torch.autograd.grad(vox, (s.pts,), s.dvox)
    total_variation(s.pts.detach(), s.key, s.weight, s.size_inv, False, s.case["tv_sparse"], grad)
    return {"vox": vox.detach(), "grad": grad}


ADAM = dict(betas=(0.9, 0.99), eps=1e-15)
ADAM_LR = (0.025, 0.01, 0.00025)


def _adam_inputs(case, seed):
    r = _Rand(seed)
    n, m = case["voxels"], (case["sh_degree"] + 1) ** 2
    dtype = torch.bfloat16 if case["dtype"] == "bf16" else torch.float32
    shapes = [(n, 8), (n, 3)] + ([(n, m - 1, 3)] if m > 1 else [])
    seen = r.uniform(n) < case["touched"]
    out = []
    for k, sh in enumerate(shapes):
        p = (r.normal(*sh) * 0.2).to(dtype)
        g = r.normal(*sh) * 1e-5
        g *= seen.view(-1, *[1] * (len(sh) - 1))
        avg = r.normal(*sh) * 1e-6
        sq = r.uniform(*sh, lo=0.1, hi=1.0) * 1e-10
        out.append((p, g, avg, sq, ADAM_LR[k]))
    return out


def _prepare_adam(case, seed):
    from sv_raster_b200.sparse_adam import FusedSparseAdam, SparseAdam
    items = _adam_inputs(case, seed)
    params = [torch.nn.Parameter(p) for p, *_ in items]
    cls = FusedSparseAdam if case["fused"] else SparseAdam
    opt = cls([{"params": [p], "lr": it[4]} for p, it in zip(params, items)], sparse=case["sparse"], **ADAM)
    for p, (_, g, avg, sq, _) in zip(params, items):
        p.grad_dtype = torch.float32  # parameters in 16 bits keep their gradients in 32
        p.grad = g
        opt.state[p].update(step=10, exp_avg=avg, exp_avg_sq=sq)
    return SimpleNamespace(case=case, opt=opt, params=params, grads=[it[1] for it in items])


def _run_adam(st):
    st.opt.step()
    return [[p.detach(), st.opt.state[p]["exp_avg"], st.opt.state[p]["exp_avg_sq"]] for p in st.params]


_KINDS = {"batched": (_prepare_batched, _run_batched), "view": (_prepare_view, _run_view),
          "gridpoints": (_prepare_gridpoints, _run_gridpoints), "adam": (_prepare_adam, _run_adam)}


def prepare(case, seed):
    st = _KINDS[case["kind"]][0](case, seed)
    torch.cuda.synchronize()
    return st


def run(state):
    return _KINDS[state.case["kind"]][1](state)


# ---------------------------------------------------------------------------
# what a pass cannot do without
# ---------------------------------------------------------------------------
# (pixel, voxel) pairs in which the ray meets the voxel and has not stopped yet, per pixel of an image, counted by
# exact(): the mixed scenes' rays cross three surfaces many voxels thick (16 to 46, by distance and level).
PAIRS_PER_PIXEL = {"sphere": 2.0, "mixed": 30.0}
FLOPS_FORWARD, FLOPS_SAMPLE, FLOPS_BACKWARD = 30, 35, 60  # per such pair; each sample; the gradient terms


def work(case):
    n = case["voxels"]
    if case["kind"] == "adam":
        m = (case["sh_degree"] + 1) ** 2
        e = n * (8 + 3 * m)
        on = case["touched"] if case["sparse"] else 1.0
        pb = 2 if case["dtype"] == "bf16" else 4
        return {"bytes": e * (4 + on * (2 * pb + 16)), "flops": 14.0 * e * on}
    if case["kind"] == "gridpoints":
        c = case["channels"]
        pts = 5 * n  # grid points of the scenes, shared corners counted once
        return {"bytes": n * 8 * (8 + 3 * 4 * c) + 4 * c * pts * 3, "flops": 16.0 * n * c}
    m = (case["sh_degree"] + 1) ** 2
    views = case.get("views", 1)
    pix = views * case["width"] * case["height"] * (0.52 if case.get("uneven") else 1.0)
    pb = 2 if case.get("dtype") == "bf16" else 4
    per_vox = 8 + 16 + pb * (8 + 3 * m)
    per_pix = 16 + (4 * case.get("depth", 0) + 4 * case.get("normal", 0)) * 3
    flops = (FLOPS_FORWARD + FLOPS_SAMPLE * case["n_samp"])
    if case["backward"]:
        per_vox += pb * (8 + 3 * m)
        per_pix += 12
        flops += FLOPS_FORWARD + FLOPS_SAMPLE * case["n_samp"] + FLOPS_BACKWARD
    pairs = pix * PAIRS_PER_PIXEL[case["scene"]]
    return {"bytes": n * per_vox + pix * per_pix, "flops": pairs * flops + 60.0 * n * views}


# ---------------------------------------------------------------------------
# the same outputs in 64 bits
# ---------------------------------------------------------------------------
F64 = torch.float64
MAX_ALPHA, MIN_ALPHA, STOP_T, STEP_SCALE = 0.99999, 0.00001, 0.0001, 100.0
C0, C1 = 0.28209479177387814, 0.4886025119029199
C2 = (1.0925484305920792, -1.0925484305920792, 0.31539156525252005, -1.0925484305920792, 0.5462742152960396)
C3 = (-0.5900435899266435, 2.890611442640554, -0.4570457994644658, 0.3731763325901154, -0.4570457994644658,
      1.445305721320277, -0.5900435899266435)


def _sh_basis(d, deg):
    x, y, z = d.unbind(-1)
    b = []
    if deg > 0:
        b += [-C1 * y, C1 * z, -C1 * x]
    if deg > 1:
        xx, yy, zz, xy, yz, xz = x * x, y * y, z * z, x * y, y * z, x * z
        b += [C2[0] * xy, C2[1] * yz, C2[2] * (2 * zz - xx - yy), C2[3] * xz, C2[4] * (xx - yy)]
    if deg > 2:
        b += [C3[0] * y * (3 * xx - yy), C3[1] * xy * z, C3[2] * y * (4 * zz - xx - yy),
              C3[3] * z * (2 * zz - 3 * xx - 3 * yy), C3[4] * x * (4 * zz - xx - yy), C3[5] * z * (xx - yy),
              C3[6] * x * (xx - 3 * yy)]
    return torch.stack(b, -1) if b else d.new_zeros(d.shape[0], 0)


def _corner_weights(q):
    x, y, z = q.unbind(-1)
    w = [(a * b * c) for a in (1 - x, x) for b in (1 - y, y) for c in (1 - z, z)]
    return torch.stack(w, -1)


def _act(d):
    e = torch.exp(0.909090909091 * d - 0.904689820196)
    return torch.where(d > 1.1, d, e), torch.where(d > 1.1, torch.ones_like(d), 0.909090909091 * e)


def _contract(x):
    return torch.where(x < 1, x, 2 - 1 / x)


def _scan_mul(x, pos, longest):
    """Product of x over its segment up to each element (pos: place in the segment)."""
    d = 1
    while d < longest:
        y = torch.cat([torch.ones_like(x[:d]), x[:-d]])
        x = torch.where(pos >= d, x * y, x)
        d *= 2
    return x


def _scan_add(x, pos, longest):
    d = 1
    while d < longest:
        y = torch.cat([torch.zeros_like(x[:d]), x[:-d]])
        x = torch.where(pos >= d, x + y, x)
        d *= 2
    return x


class _Exact:
    """One view composited in 64 bits, and its backward."""

    def __init__(self, s, cam, geos, sh0, shs, deg, ns, bg, levels=16):
        self.s, self.cam, self.ns, self.bg, self.deg = s, cam, ns, bg, deg
        W, H = self.W, self.H = cam.width, cam.height
        c2w, w2c = cam.c2w.to(F64), cam.w2c.to(F64)
        self.o = c2w[:3, 3]
        self.ctr, self.len = s.centers.to(F64), s.lengths.to(F64).reshape(-1)
        self.geos = geos
        # rays
        ys, xs = torch.meshgrid(torch.arange(H, device=DEV, dtype=F64), torch.arange(W, device=DEV, dtype=F64),
                                indexing="ij")
        cd = torch.stack([(xs + 0.5 - cam.cx) * 2 * cam.tanfovx / W, (ys + 0.5 - cam.cy) * 2 * cam.tanfovy / H,
                          torch.ones_like(xs)], -1).reshape(-1, 3)
        self.rninv = 1 / cd.norm(dim=1)
        self.dir = (cd @ c2w[:3, :3].T) * self.rninv[:, None]
        neg = (self.dir < 0).long()
        quad = neg[:, 0] * 4 + neg[:, 1] * 2 + neg[:, 2]
        # pixel boxes and quadrants of the voxels
        u0 = torch.full((s.P,), 1e9, device=DEV, dtype=F64)
        v0, u1, v1 = u0.clone(), -u0, -u0
        bits = torch.zeros(s.P, dtype=torch.int64, device=DEV)
        for c in range(8):
            sg = torch.tensor([2 * ((c >> 2) & 1) - 1, 2 * ((c >> 1) & 1) - 1, 2 * (c & 1) - 1], device=DEV, dtype=F64)
            wp = self.ctr + 0.5 * self.len[:, None] * sg
            p = wp @ w2c[:3, :3].T + w2c[:3, 3]
            front = p[:, 2] >= np.float32(NEAR)
            u, v = p[:, 0] / p[:, 2], p[:, 1] / p[:, 2]
            u0, u1 = torch.where(front, torch.minimum(u0, u), u0), torch.where(front, torch.maximum(u1, u), u1)
            v0, v1 = torch.where(front, torch.minimum(v0, v), v0), torch.where(front, torch.maximum(v1, v), v1)
            n = (wp < self.o).long()
            bits |= torch.where(front, torch.ones_like(bits) << (n[:, 0] * 4 + n[:, 1] * 2 + n[:, 2]),
                                torch.zeros_like(bits))
        fx, fy = 0.5 * W / cam.tanfovx, 0.5 * H / cam.tanfovy
        x0, x1 = (fx * u0 + cam.cx - 0.5).clamp(min=0), (fx * u1 + cam.cx - 0.5).clamp(max=W)
        y0, y1 = (fy * v0 + cam.cy - 0.5).clamp(min=0), (fy * v1 + cam.cy - 0.5).clamp(max=H)
        rel = self.ctr - self.o
        seen = (rel.square().sum(1) >= NEAR * NEAR) & (x0 <= x1) & (y0 <= y1) & (bits != 0)
        ix0, iy0 = x0.round().long(), y0.round().long()
        ix1, iy1 = x1.round().long().clamp(max=W - 1), y1.round().long().clamp(max=H - 1)
        seen &= (ix0 <= ix1) & (iy0 <= iy1)
        self.seen = seen
        # colours of the voxels from here
        d = rel / rel.norm(dim=1, keepdim=True)
        self.basis = _sh_basis(d, deg)
        rgb = C0 * sh0.to(F64) + 0.5
        for k in range(self.basis.shape[1]):
            rgb = rgb + self.basis[:, k:k + 1] * shs[:, k].to(F64)
        self.rgb = rgb.clamp(min=0)
        # front-to-back place of each voxel for each ray quadrant
        present = torch.unique(quad).tolist()
        place = {}
        flat = s.path.reshape(-1)
        for q in present:
            rep = 0
            for _ in range(levels):
                rep = (rep << 3) | q
            o = torch.argsort(flat ^ rep)
            place[q] = torch.empty_like(o)
            place[q][o] = torch.arange(s.P, device=DEV)
        ids = torch.nonzero(seen).reshape(-1)
        w, h = (ix1 - ix0 + 1)[ids], (iy1 - iy0 + 1)[ids]
        cnt = w * h
        end = torch.cumsum(cnt, 0)
        total = int(end[-1]) if ids.numel() else 0
        keep = []
        i = 0
        limit = 24_000_000
        while i < ids.numel():
            base = int(end[i - 1]) if i else 0
            j = max(i + 1, int(torch.searchsorted(end, base + limit, right=True)))
            sub = torch.arange(i, j, device=DEV).repeat_interleave(cnt[i:j])
            loc = torch.arange(sub.numel(), device=DEV) - (end[sub] - cnt[sub] - base)
            vid = ids[sub]
            pix = (iy0[vid] + loc // w[sub]) * W + ix0[vid] + loc % w[sub]
            ok = (bits[vid] >> quad[pix]) & 1 == 1
            vid, pix = vid[ok], pix[ok]
            a, b = self._slab(vid, pix)
            ok = a <= b
            vid, pix, a, b = vid[ok], pix[ok], a[ok], b[ok]
            vol = self._samples(vid, pix, a, b)[0]
            ok = (1 - torch.exp(-vol)).clamp(max=MAX_ALPHA) >= MIN_ALPHA
            vid, pix, vol = vid[ok], pix[ok], vol[ok]
            key = pix * s.P
            qd = quad[pix]
            for q in present:
                m = qd == q
                key[m] += place[q][vid[m]]
            keep.append((key, vid.int(), vol))
            i = j
        del place
        self.pairs_tested = total
        key, vid, vol = (torch.cat([k[t] for k in keep]) for t in range(3))
        del keep
        key, order = torch.sort(key)
        vid, vol = vid[order].long(), vol[order]
        pix = key // s.P
        del key, order
        n = pix.numel()
        at = torch.arange(n, device=DEV)
        first = torch.ones(n, dtype=torch.bool, device=DEV)
        first[1:] = pix[1:] != pix[:-1]
        start = torch.cummax(torch.where(first, at, torch.zeros_like(at)), 0).values
        pos = at - start
        longest = int(pos.max()) + 1 if n else 1
        alpha = (1 - torch.exp(-vol)).clamp(max=MAX_ALPHA)
        T = _scan_mul(torch.cat([torch.ones(1, device=DEV, dtype=F64), 1 - alpha[:-1]]).masked_fill(first, 1.0), pos,
                      longest)  # before each pair
        ok = T >= STOP_T
        self.pix, self.vid, self.vol, self.alpha, self.T = pix[ok], vid[ok], vol[ok], alpha[ok], T[ok]
        self.pos, self.longest = pos[ok], longest
        self.n = self.pix.numel()
        self.w = self.T * self.alpha
        self.Tfin = torch.ones(H * W, device=DEV, dtype=F64)
        last = torch.ones(self.n, dtype=torch.bool, device=DEV)
        last[:-1] = self.pix[1:] != self.pix[:-1]
        self.Tfin[self.pix[last]] = (self.T * (1 - self.alpha))[last]

    def _slab(self, vid, pix):
        inv = 1 / self.dir[pix]
        r = 0.5 * self.len[vid][:, None]
        rel = self.ctr[vid] - self.o
        t0, t1 = (rel - r) * inv, (rel + r) * inv
        return torch.minimum(t0, t1).amax(1), torch.maximum(t0, t1).amin(1)

    def _samples(self, vid, pix, a, b):
        """Optical depth, and per sample its share, d(share)/d(corner density) scale and place in the voxel."""
        step = (b - a) / self.ns
        geo = self.geos[vid].to(F64)
        vol, each = 0.0, []
        for k in range(self.ns):
            t = a + (k + 0.5) * step
            q = (self.o + t[:, None] * self.dir[pix] - self.ctr[vid]) / self.len[vid][:, None] + 0.5
            w = _corner_weights(q)
            act, grad = _act((geo * w).sum(1))
            v = STEP_SCALE * step * act
            vol = vol + v
            each.append((v, STEP_SCALE * step * grad, w))
        return vol, each

    def _add(self, values, idx=None, size=None):
        out = torch.zeros((size or self.W * self.H,) + values.shape[1:], device=DEV, dtype=F64)
        return out.index_add_(0, self.pix if idx is None else idx, values)

    def color(self):
        c = torch.stack([self._add(self.w * self.rgb[self.vid, k]) for k in range(3)])
        return c + (self.Tfin * self.bg)[None]

    def _dval(self, a, b, each):
        """A pair's expected depth per unit of transmittance, and its derivative by each sample's optical depth."""
        al = [(1 - torch.exp(-e[0])).clamp(max=MAX_ALPHA) for e in each]
        ss = (b - a) / self.ns
        t = [a + (k + 0.5) * ss for k in range(self.ns)]
        if self.ns == 1:
            return al[0] * t[0], [t[0] * (1 - al[0])]
        if self.ns == 2:
            return (al[0] * t[0] + (1 - al[0]) * al[1] * t[1],
                    [(t[0] - al[1] * t[1]) * (1 - al[0]), (t[1] - al[0] * t[1]) * (1 - al[1])])
        a0, a1, a2 = al
        return (a0 * t[0] + (1 - a0) * a1 * t[1] + (1 - a0) * (1 - a1) * a2 * t[2],
                [(t[0] + a1 * a2 * t[2] - a1 * t[1] - a2 * t[2]) * (1 - a0),
                 (t[1] + a0 * a2 * t[2] - a0 * t[1] - a2 * t[2]) * (1 - a1),
                 (t[2] + a0 * a1 * t[2] - a0 * t[2] - a1 * t[2]) * (1 - a2)])

    def _normal(self, geo):
        g = geo.view(-1, 2, 2, 2)
        n = torch.stack([(g[:, 1] - g[:, 0]).sum((1, 2)), (g[:, :, 1] - g[:, :, 0]).sum((1, 2)),
                         (g[:, :, :, 1] - g[:, :, :, 0]).sum((1, 2))], -1)
        return n, 1 / torch.sqrt(n.square().sum(1) + 1e-15)

    def _chunks(self, limit=8_000_000):
        for i in range(0, self.n, limit):
            yield slice(i, min(self.n, i + limit))

    def maps(self, depth, dist, normal):
        """(depth [3,HW], normal [3,HW]) as the entry point lays them out."""
        HW = self.W * self.H
        D, N = torch.zeros(3, HW, device=DEV, dtype=F64), torch.zeros(3, HW, device=DEV, dtype=F64)
        for c in self._chunks():
            pix, vid = self.pix[c], self.vid[c]
            a, b = self._slab(vid, pix)
            if depth:
                each = self._samples(vid, pix, a, b)[1]
                D[0].index_add_(0, pix, self.T[c] * self._dval(a, b, each)[0])
            if dist:
                D[1].index_add_(0, pix, self.w[c] * 0.5 * (_contract(a) + _contract(b)))
            if normal:
                n, rl = self._normal(self.geos[vid].to(F64))
                N.index_add_(1, pix, (self.w[c] * rl)[None] * n.T)
        if depth:
            D[0] *= self.rninv
            # the voxel in which the transmittance falls to a half, and the first of 16 samples past that
            at = torch.full((HW,), -1, dtype=torch.int64, device=DEV)
            m = self.T > 0.5
            at.scatter_reduce_(0, self.pix[m], torch.nonzero(m).reshape(-1), "amax")
            px = torch.nonzero(at >= 0).reshape(-1)
            vid, T = self.vid[at[px]], self.T[at[px]]
            a, b = self._slab(vid, px)
            step = (b - a) / 16
            geo = self.geos[vid].to(F64)
            med = a - 0.5 * step
            for k in range(16):
                go = T > 0.5
                med = torch.where(go, med + step, med)
                t = a + (k + 0.5) * step
                q = (self.o + t[:, None] * self.dir[px] - self.ctr[vid]) / self.len[vid][:, None] + 0.5
                act = _act((geo * _corner_weights(q)).sum(1))[0]
                T = torch.where(go, T * torch.exp(-STEP_SCALE * step * act), T)
            D[2][px] = med * self.rninv[px]
        return D, N

    def max_w(self):
        out = torch.zeros(self.s.P, device=DEV, dtype=F64)
        return out.scatter_reduce_(0, self.vid, self.w, "amax").reshape(-1, 1)

    def backward(self, dC, dgeos, dsh0, dshs, subdiv=None, dD=None, dN=None, dist=0.0, concen=0.0, ascending=0.0,
                 gt=None, ddist=None):
        """Adds one view's gradients; dC [3,HW], dD [HW] of the mean depth, dN [3,HW]."""
        HW = self.W * self.H
        lam = 1.0 / HW
        dW = torch.empty(self.n, device=DEV, dtype=F64)
        behind_extra = torch.zeros(self.n, device=DEV, dtype=F64)  # T * depth share, for the pairs in front
        if dist:
            m = torch.empty(self.n, device=DEV, dtype=F64)
            ext = torch.empty(self.n, device=DEV, dtype=F64)
            for c in self._chunks():
                a, b = self._slab(self.vid[c], self.pix[c])
                ca, cb = _contract(a), _contract(b)
                m[c], ext[c] = 0.5 * (ca + cb), cb - ca
            wm = self.w * m
            pre_w, pre_wm = _scan_add(self.w, self.pos, self.longest), _scan_add(wm, self.pos, self.longest)
            suf_w, suf_wm = self._add(self.w)[self.pix] - pre_w, self._add(wm)[self.pix] - pre_wm
            pre_w, pre_wm = pre_w - self.w, pre_wm - wm
        for c in self._chunks():
            pix, vid = self.pix[c], self.vid[c]
            v = (dC[:, pix] * self.rgb[vid].T).sum(0)
            if dist:
                v = v + dist * lam * (2.0 / 3.0 * self.w[c] * ext[c] +
                                      2 * (m[c] * (pre_w[c] - suf_w[c]) - (pre_wm[c] - suf_wm[c])))
            if dN is not None:
                n, rl = self._normal(self.geos[vid].to(F64))
                v = v + (dN[:, pix] * (rl[None] * n.T)).sum(0)
            dW[c] = v
            if dD is not None:
                a, b = self._slab(vid, pix)
                behind_extra[c] = (dD * self.rninv)[pix] * self._dval(a, b, self._samples(vid, pix, a, b)[1])[0]
        # what lies behind each pair, per unit of the transmittance left behind it
        R_last = (self.bg * dC.sum(0))[self.pix]
        share = (self.w * dW + self.T * behind_extra).flip(0)
        rpos = self._count_from_back()
        behind = _scan_add(share, rpos, self.longest).flip(0) - share.flip(0)
        R = (behind + self.Tfin[self.pix] * R_last) / (self.T * (1 - self.alpha))
        dA = self.T * (dW - R)
        drgb = torch.zeros(self.s.P, 3, device=DEV, dtype=F64)
        for c in self._chunks():
            pix, vid = self.pix[c], self.vid[c]
            a, b = self._slab(vid, pix)
            geo = self.geos[vid].to(F64)
            vol, each = self._samples(vid, pix, a, b)
            dI = dA[c] * torch.exp(-vol)
            extra = [0.0] * self.ns
            if dD is not None:
                up = (dD * self.rninv)[pix] * self.T[c]
                extra = [up * x for x in self._dval(a, b, each)[1]]
            g = 0.0
            for (v, s, w), x in zip(each, extra):
                g = g + ((dI + x) * s)[:, None] * w
            if dN is not None:
                n, rl = self._normal(geo)
                up = self.w[c][:, None] * dN[:, pix].T
                ln = rl[:, None] * (up - (up * n).sum(1, keepdim=True) * rl[:, None] ** 2 * n)
                sg = torch.tensor([[2 * ((k >> (2 - ax)) & 1) - 1 for ax in range(3)] for k in range(8)], device=DEV,
                                  dtype=F64)
                g = g + ln @ sg.T
            if ascending:
                ends = [_corner_weights((self.o + t[:, None] * self.dir[pix] - self.ctr[vid]) /
                                        self.len[vid][:, None] + 0.5) for t in (a, b)]
                falls = (geo * ends[0]).sum(1) > (geo * ends[1]).sum(1)
                g = g + (ascending * lam * self.w[c] * falls)[:, None] * (ends[0] - ends[1])
            dgeos.index_add_(0, vid, g)
            r = self.w[c][:, None] * dC[:, pix].T
            if concen:
                r = r + (2 * concen * lam * self.w[c])[:, None] * (self.rgb[vid] - gt[:, pix].T)
            drgb.index_add_(0, vid, r)
            if subdiv is not None:
                subdiv.index_add_(0, vid, (dA[c] * self.alpha[c]).abs()[:, None])
        dsh0 += C0 * drgb
        for k in range(self.basis.shape[1]):
            dshs[:, k] += self.basis[:, k:k + 1] * drgb

    def _count_from_back(self):
        n = self.n
        p = self.pix.flip(0)
        at = torch.arange(n, device=DEV)
        first = torch.ones(n, dtype=torch.bool, device=DEV)
        first[1:] = p[1:] != p[:-1]
        return at - torch.cummax(torch.where(first, at, torch.zeros_like(at)), 0).values


def _exact_batched(case, seed):
    s = _batched_inputs(case, seed)
    dens = s.grid[s.key] if case["grid"] else s.geos
    grads = [torch.zeros(s.P, 8, device=DEV, dtype=F64), torch.zeros(s.P, 3, device=DEV, dtype=F64),
             torch.zeros(s.shs.shape, device=DEV, dtype=F64)]
    colors, Ts, at = [], [], 0
    for cam in s.cams:
        e = _Exact(s, cam, dens, s.sh0, s.shs, case["sh_degree"], case["n_samp"], 0.0)
        hw = cam.width * cam.height
        colors.append(e.color().reshape(-1))
        Ts.append(e.Tfin)
        if case["backward"]:
            e.backward(s.dC[3 * at:3 * (at + hw)].view(3, hw).to(F64), *grads)
        at += hw
        del e
    out = {"color": torch.cat(colors), "T": torch.cat(Ts)}
    if case["backward"]:
        if case["grid"]:
            d = torch.zeros(s.grid.numel(), device=DEV, dtype=F64)
            grads[0] = d.index_add_(0, s.key.reshape(-1), grads[0].reshape(-1))
        out.update(ddens=grads[0], dsh0=grads[1], dshs=grads[2])
    return out


def _exact_view(case, seed):
    s = _view_inputs(case, seed)
    cam = s.cams[0]
    h, w = cam.height, cam.width
    e = _Exact(s, cam, s.geos, s.sh0, s.shs, case["sh_degree"], case["n_samp"], case["bg"], case["levels"])
    out = {"color": e.color().view(3, h, w), "T": e.Tfin.view(1, h, w)}
    D, N = e.maps(case["depth"], case["dist"] > 0, case["normal"])
    if case["depth"] or case["dist"] > 0:
        out["depth"] = D.view(3, h, w)
    if case["normal"]:
        out["normal"] = N.view(3, h, w)
    if case["max_w"]:
        out["max_w"] = e.max_w()
    if case["backward"]:
        g = [torch.zeros(s.P, 8, device=DEV, dtype=F64), torch.zeros(s.P, 3, device=DEV, dtype=F64),
             torch.zeros(s.shs.shape, device=DEV, dtype=F64), torch.zeros(s.P, 1, device=DEV, dtype=F64)]
        flat = lambda t: t.reshape(3, -1).to(F64)  # noqa: E731
        e.backward(flat(s.dC), *g, dD=flat(s.dD)[0] if case["depth"] else None,
                   dN=flat(s.dN) if case["normal"] else None, dist=case["dist"], concen=case["concen"],
                   ascending=case["ascending"], gt=flat(s.gt))
        out.update(zip(("dgeos", "dsh0", "dshs", "dsubdiv"), g))
    return out


def _exact_gridpoints(case, seed):
    s = _gridpoint_inputs(case, seed)
    pts = s.pts.to(F64)
    vox = pts[s.key]  # [P,8,C]
    key = s.key.reshape(-1)
    grad = torch.zeros_like(pts).index_add_(0, key, s.dvox.to(F64).reshape(key.numel(), -1))
    # the side of each edge neighbour of a corner inside its voxel
    n = torch.arange(8, device=DEV)
    tv = sum(((vox > vox[:, n ^ b]) * 2 - 1) for b in (1, 2, 4)).to(F64)
    tv = tv * (s.weight * 0.01 * s.size_inv.to(F64))[:, :, None]
    if case["tv_sparse"]:
        tv = tv * (grad[s.key] != 0).any(1, keepdim=True)
    grad.index_add_(0, key, tv.reshape(key.numel(), -1))
    return {"vox": vox[:, :, 0] if case["channels"] == 1 else vox, "grad": grad}


def _exact_adam(case, seed):
    b1, b2 = ADAM["betas"]
    step = 11
    out = []
    for p, g, avg, sq, lr in _adam_inputs(case, seed):
        p, g, avg, sq = (t.to(F64) for t in (p, g, avg, sq))
        a2 = b1 * avg + (1 - b1) * g
        s2 = b2 * sq + (1 - b2) * g * g
        p2 = p - lr / (1 - b1 ** step) * a2 / (s2.sqrt() / math.sqrt(1 - b2 ** step) + ADAM["eps"])
        if case["sparse"]:
            on = g != 0
            a2, s2, p2 = torch.where(on, a2, avg), torch.where(on, s2, sq), torch.where(on, p2, p)
        out.append([p2, a2, s2])
    return out


def exact(case, seed):
    return {"batched": _exact_batched, "view": _exact_view, "gridpoints": _exact_gridpoints,
            "adam": _exact_adam}[case["kind"]](case, seed)
