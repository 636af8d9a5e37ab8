"""Performance cases of the framework: what its users have it do, through its public calls.

A case names a family (what is run) and a scene (block edge, block grid, point clusters,
storage type).  Scenes are the seeded clouds of the surface workloads: spheres on 16^3
blocks (the 512^3 workload and its small versions) or rotated ellipsoids on 32^3 blocks
(crops of the 4096^3 three-level workload), made on the GPU from the seed.

  pipeline  points on the device -> refinement map, splat, finalise, sweeps: the whole
            reconstruction of one frame
  sweep     applyChannelPdeFast on a field resident in HBM
  splat     splat + finalise of a frame's particles on an existing layout
  g2p       trilinear interpolation of the field at particles in random order
  restrict  downsampleFloatChannelNew of the value blocks
  halo      fillHaloBlock_ of every value block, with a coarser level beside it
  solve     multigrid-preconditioned CG to a relative residual of 1e-6, FP32 or mixed
  warmnet   loss and gradients of the learned warm start (a training step's work)
  render    the ray-marched view of the surface from the demo's camera
"""
import ctypes as C
import math

import torch

from msbg_gb300 import gpu as G

DEV = "cuda" if torch.cuda.is_available() else "cpu"
STORAGE = {"f32": G.F32, "f16": G.F16, "u16": G.U16}
TORCH = {"f32": torch.float32, "f16": torch.float16, "u16": torch.int16}
TYPESTR = {"f32": "<f4", "f16": "<f2", "u16": "<i2"}  # uint16 bytes, seen as int16
R, NB = 2.0, 2.0  # particle radius and narrow-band distance of the demo, in voxels
LAPL = {"mcf": 4, "jacobi": 17}
CH_X, CH_B, CH_COEF = 1, 2, 3  # solver channels; 3..6: cx, cy, cz, diagonal


def _case(name, family, bs, nb, objects, pts, storage, **more):
    return dict(name=name, family=family, bs=bs, nx=nb[0], ny=nb[1], nz=nb[2], objects=objects, pts=pts,
                storage=storage, **more)


def listed():
    return [
        # the tests' and the smoke run's size: a preview frame, bound by launches and latency
        _case("pipeline_64", "pipeline", 16, (4, 4, 4), 2, 1500, "u16", iters=20, variant="exact"),
        # the 512^3 surface workload: an ordinary frame on one GPU
        _case("pipeline_512", "pipeline", 16, (32, 32, 32), 64, 32000, "f32", iters=20, variant="exact"),
        # the headline metric, curvature flow at FP16 storage, on a crop of the 4096^3 workload
        _case("mcf_f16", "sweep", 32, (128, 128, 128), 24, 32000, "f16", kind="mcf", iters=10, variant="fast"),
        # the same with the diffusion kernel on the crop that kernels are profiled on
        _case("jacobi_f16", "sweep", 32, (128, 128, 128), 96, 32000, "f16", kind="jacobi", iters=10, variant="fast"),
        # a time step's splat on a kept layout
        _case("splat_f16", "splat", 32, (128, 128, 128), 24, 32000, "f16"),
        # particles read the field back (advection, level-set correction)
        _case("g2p_f16", "g2p", 32, (128, 128, 128), 48, 32000, "f16"),
        # a coarser copy of the density for display or for the next grid level
        _case("restrict_f16", "restrict", 32, (128, 128, 128), 48, 32000, "f16"),
        # halo boxes for a caller's own stencil
        _case("halo_f16", "halo", 32, (128, 128, 128), 16, 32000, "f16"),
        # pressure solve on the 512^3 layout
        _case("solve_f32", "solve", 16, (32, 32, 32), 64, 32000, "f32", method="plain"),
        # pressure solve with FP16-storage corrections on the profiling crop of the 4096^3 layout
        _case("solve_mixed", "solve", 32, (128, 128, 128), 12, 32000, "f32", method="mixed"),
        # one training pair of the warm start's trainer (its default: one cluster)
        _case("warmnet_grad", "warmnet", 32, (128, 128, 128), 1, 32000, "f32"),
        # the demo's picture of the reconstructed surface
        _case("render_f16", "render", 32, (128, 128, 128), 48, 32000, "f16", width=1280, height=720),
    ]


def draw(rng):
    def spread(lo, hi):  # a whole number, even over the logarithm
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    family = rng.choice(["pipeline", "sweep", "splat", "g2p", "restrict", "halo", "solve", "warmnet", "render"])
    storage = rng.choice(["f32", "f16", "u16"])
    bs = 16 if family == "pipeline" else 32 if family in ("warmnet", "render") else rng.choice([16, 32])
    if bs == 16:  # frames from 64^3 to the 512^3 workload, not always cubes
        n = spread(4, 32)
        nb = tuple(max(4, min(32, n + rng.randint(-n // 4, n // 4))) for _ in range(3))
        objects = max(1, min(64, int(64 * (n / 32) ** 2)))
        pts = spread(1000, 32000)
    else:  # crops of the 4096^3 workload
        nb = tuple(rng.randint(96, 128) for _ in range(3))
        objects = {"sweep": spread(2, 48), "splat": spread(1, 24), "g2p": spread(1, 48), "restrict": spread(1, 48),
                   "halo": spread(1, 16), "solve": spread(1, 8), "warmnet": 1, "render": spread(4, 48)}[family]
        pts = spread(8000, 32000)
    more = {}
    if family == "pipeline":
        more = dict(iters=2 * rng.randint(1, 10), variant="exact")
    elif family == "sweep":
        # uint16 fields go through the reference's own operation order, whose bytes are the reference's
        more = dict(kind=rng.choice(["mcf", "jacobi"]), iters=2 * rng.randint(1, 5),
                    variant="exact" if storage == "u16" else rng.choice(["fast", "exact"]))
    elif family == "solve":
        storage, more = "f32", dict(method=rng.choice(["plain", "mixed"]))
    elif family == "warmnet":
        storage = "f32"
    elif family == "render":
        more = dict(width=spread(240, 1280), height=spread(135, 720))
    c = _case("", family, bs, nb, objects, pts, storage, **more)
    del c["name"]
    return c


# ---- scenes ---------------------------------------------------------------------------------

def _cloud(case, seed, dev):
    """Points [n, 3] (FP32, voxels) on the scene's spheres or ellipsoids, a little moved by the seed: a
    point stays where the move would touch other blocks, so that every seed has the case's layout."""
    k, n = case["objects"], case["pts"]
    g = torch.Generator(device=dev).manual_seed(k * 7919 + n * 17 + case["nx"])
    res = torch.tensor([case["nx"], case["ny"], case["nz"]], device=dev, dtype=torch.float32) * case["bs"]
    small = float(res.min())
    c = (0.1 + 0.8 * torch.rand(k, 3, generator=g, device=dev)) * res
    u = torch.randn(k, n, 3, generator=g, device=dev)
    u /= u.norm(dim=2, keepdim=True)
    if case["bs"] == 16:
        p = c[:, None] + (0.02 + 0.04 * torch.rand(k, 1, 1, generator=g, device=dev)) * small * u
    else:
        ax = (0.005 + 0.025 * torch.rand(k, 1, 3, generator=g, device=dev)) * small
        q = torch.randn(k, 4, generator=g, device=dev)
        w, x, y, z = (q / q.norm(dim=1, keepdim=True)).unbind(1)
        rot = torch.stack([1 - 2 * (y * y + z * z), 2 * (x * y - z * w), 2 * (x * z + y * w),
                           2 * (x * y + z * w), 1 - 2 * (x * x + z * z), 2 * (y * z - x * w),
                           2 * (x * z - y * w), 2 * (y * z + x * w), 1 - 2 * (x * x + y * y)], 1).reshape(k, 3, 3)
        p = c[:, None] + torch.einsum("knj,kij->kni", ax * u, rot)
    p = torch.minimum((p + 0.1 * torch.randn(k, n, 3, generator=g, device=dev)).clamp_min(1.0), res - 1.01).reshape(-1, 3)
    g.manual_seed(int(seed) * 7919 + 17)
    moved = torch.minimum((p + 0.5 * torch.randn(k * n, 3, generator=g, device=dev)).clamp_min(1.0), res - 1.01)
    same = torch.ones(k * n, 1, dtype=torch.bool, device=dev)
    for r in (0.0, *(_bands(case) or (R + NB,))):
        for a, b in zip(_box(case, p, r), _box(case, moved, r)):
            same &= (a == b).all(1, keepdim=True)
    return torch.where(same, moved, p).contiguous()


def _box(case, pts, r):
    """First and last block of the points' boxes of radius r, per axis."""
    nb = torch.tensor([case["nx"], case["ny"], case["nz"]], device=pts.device)
    b = pts * (1.0 / case["bs"])
    return (b - r / case["bs"]).to(torch.int32).clamp_min(0), torch.minimum((b + r / case["bs"]).to(torch.int32), nb - 1)


def _bands(case):
    return None if case["bs"] == 16 else (8.0, 16.0)


def _blocks(case, pts):
    """Ids of the scene's value blocks, ascending: the blocks of every point's band box."""
    lo, hi = _box(case, pts, (_bands(case) or (R + NB,))[0])
    keys = []
    for k in range(8):
        x, y, z = (torch.where(torch.tensor(bool((k >> i) & 1), device=pts.device), hi[:, i], lo[:, i]) for i in range(3))
        keys.append(torch.unique((z.long() * case["ny"] + y) * case["nx"] + x))
    return torch.unique(torch.cat(keys))


class _View:
    """Device memory of the library as a tensor's source."""

    def __init__(self, ptr, shape, typestr, keep):
        self.__cuda_array_interface__ = dict(shape=tuple(shape), typestr=typestr, data=(int(ptr), False), version=2)
        self.keep = keep


def _view(ptr, shape, typestr, keep=None):
    return torch.as_tensor(_View(ptr, shape, typestr, keep), device="cuda")


def _device(n, typestr):
    """A device buffer of the library's and a tensor on it."""
    buf = G.DeviceBuffer.alloc(n * int(typestr[2:]))
    return buf, _view(buf.ptr, (n,), typestr, buf)


def _payload(g, case, chan=0, storage=None):
    return _view(g.payload_ptr(chan), (case["n"], case["bs"] ** 3), TYPESTR[storage or case["storage"]], g)


def _scene(case, seed, field):
    """A grid with the scene's layout (and its splatted field), and the points on the device."""
    pts = _cloud(case, seed, "cuda")
    buf, t = _device(pts.numel(), "<f4")
    t.copy_(pts.reshape(-1))
    bs = case["bs"]
    g = G.MultiresSparseGrid(case["nx"] * bs, case["ny"] * bs, case["nz"] * bs, bs, 3, STORAGE[case["storage"]])
    torch.cuda.synchronize()
    s = dict(case, g=g, buf=buf, points=pts.shape[0])
    _layout(s)
    if field:
        g.splat(buf, s["points"], R, NB)
        g.splat_finalize(R, NB)
    s["n"] = int(g.info().nActive)
    return s


def _layout(s):
    g, buf, n = s["g"], s["buf"], s["points"]
    if _bands(s) is None:
        g.mark_points(buf, n, R + NB)
        g.levels_from_marks()
    else:
        g.levels_from_bands(buf, n, _bands(s))
    g.regularizeRefinementMap()
    g.setRefinementMap(1.0)


def _system(case, seed, bids):
    """Face coefficients U[0.5, 2] and the diagonal (FP32) on the blocks `bids`; the right-hand side
    N(0, 1) of zero mean, or (warm start) a smooth solution with its own right-hand side; the
    neighbour table [6][cells] (-1: none)."""
    bs, nx, ny, nz = case["bs"], case["nx"], case["ny"], case["nz"]
    n, v = bids.numel(), bs ** 3
    gen = torch.Generator(device=DEV).manual_seed(int(seed) * 104729 + 5)
    nbr = _neighbours(case, bids)
    low = [0.5 + 1.5 * torch.rand(n * v, generator=gen, device=DEV) for _ in range(3)]
    diag = torch.zeros(n * v, device=DEV)
    for a in range(3):
        up = nbr[2 * a + 1]
        rim = 0.5 + 1.5 * torch.rand(n * v, generator=gen, device=DEV)
        diag += low[a] + torch.where(up >= 0, low[a][up.clamp_min(0).long()], rim)
    if case["family"] == "warmnet":
        i = torch.arange(bs, device=DEV)
        z, y, x = torch.meshgrid(i, i, i, indexing="ij")
        bx, by, bz = bids % nx, (bids // nx) % ny, bids // (nx * ny)
        at = [(b[:, None] * bs + c.reshape(1, -1)).float() for b, c in ((bx, x), (by, y), (bz, z))]
        xs = 0.1 * torch.randn(n, v, generator=gen, device=DEV)
        for _ in range(6):
            k = torch.randn(4, generator=gen, device=DEV) * 0.15
            xs += torch.sin(k[0] * at[0] + k[1] * at[1] + k[2] * at[2] + 40 * k[3])
        xs = xs.reshape(-1)
        b = _operator(low, diag, nbr, xs)
        return low, diag, b, xs, nbr
    b = torch.randn(n * v, generator=gen, device=DEV)
    return low, diag, b - b.mean(), None, nbr


def _neighbours(case, bids):
    """Cell indices of the six neighbours of every cell of the blocks, -1 outside them (int32)."""
    bs, nx, ny, nz = case["bs"], case["nx"], case["ny"], case["nz"]
    slot = torch.full((nz + 2, ny + 2, nx + 2), -1, device=bids.device, dtype=torch.int32)
    bx, by, bz = bids % nx + 1, (bids // nx) % ny + 1, bids // (nx * ny) + 1
    own = torch.arange(bids.numel(), device=bids.device, dtype=torch.int32)
    slot[bz, by, bx] = own
    cell = torch.arange(bs ** 3, device=bids.device, dtype=torch.int32).reshape(1, bs, bs, bs)
    out = []
    for a in range(3):
        st, dim = bs ** a, 3 - a
        for d in (-1, 1):
            nb = slot[bz + (d if a == 2 else 0), by + (d if a == 1 else 0), bx + (d if a == 0 else 0)]
            idx = own.reshape(-1, 1, 1, 1) * bs ** 3 + cell + d * st
            edge = bs - 1 if d > 0 else 0
            far = nb.reshape(-1, 1, 1, 1) * bs ** 3 + cell + d * st - d * st * bs
            far = torch.where(nb.reshape(-1, 1, 1, 1) >= 0, far, torch.full_like(far, -1))
            idx.select(dim, edge).copy_(far.expand_as(idx).select(dim, edge))
            out.append(idx.reshape(-1))
    return out


def _operator(low, diag, nbr, x):
    """A x: diagonal minus the face-weighted neighbours."""
    y = diag * x
    for a in range(3):
        lo, up = nbr[2 * a], nbr[2 * a + 1]
        y -= torch.where(lo >= 0, low[a] * x[lo.clamp_min(0)], 0)
        i = up.clamp_min(0)
        y -= torch.where(up >= 0, low[a][i] * x[i], 0)
    return y


def _channels(s, arrays):
    """FP32 channels of the solver filled from tensors."""
    for ch, t in arrays.items():
        s["g"].channel_create(ch, G.F32)
        if t is not None:
            _payload(s["g"], s, ch, "f32").copy_(t.reshape(s["n"], -1))


def _weights(seed):
    """He-normal start of the network (2-16-16-16-2 channels, 27 taps)."""
    ch, gen = (2, 16, 16, 16, 2), torch.Generator().manual_seed(int(seed) + 3)
    w = [torch.randn(27, ch[i], ch[i + 1], generator=gen) * math.sqrt(2 / (27 * ch[i])) * (0.5 if i == 3 else 1.0)
         for i in range(4)]
    return w, [0.05 * torch.randn(ch[i + 1], generator=gen) for i in range(4)]


# ---- the cases ------------------------------------------------------------------------------

def prepare(case, seed):
    f = case["family"]
    s = _scene(case, seed, f in ("sweep", "g2p", "restrict", "halo", "render"))
    g, v, bs = s["g"], s["n"] * case["bs"] ** 3, case["bs"]
    if f == "g2p":
        gen = torch.Generator(device="cuda").manual_seed(int(seed) + 11)
        at = _view(s["buf"].ptr, (s["points"], 3), "<f4", s["buf"])
        at.copy_(at[torch.randperm(s["points"], generator=gen, device="cuda")])
        s["out"], s["res"] = _device(s["points"], "<f4")
    elif f == "restrict":
        s["out"], s["res"] = _device(v // 8, "<f4")
    elif f == "halo":
        lv, slot = g.levels(), g.slots()
        st0 = torch.tensor(slot).where(torch.tensor(lv) == 0, torch.tensor(G.LBLK_NONE, dtype=torch.int32))
        one = torch.tensor(lv) == 1
        st1 = torch.where(one, torch.cumsum(one, 0) - 1, G.LBLK_NONE).to(torch.int32)
        n1 = int(one.sum())
        gen = torch.Generator(device="cuda").manual_seed(int(seed) + 13)
        pay1 = torch.rand(max(n1, 1) * (bs // 2) ** 3, generator=gen, device="cuda")
        pay1 = pay1.to(TORCH[s["storage"]]) if s["storage"] != "u16" else (pay1 * 32767).to(torch.int16)
        s["level"] = [(g.to_device(st0.numpy()), g.payload_ptr(0)), (g.to_device(st1.numpy()), pay1.data_ptr()), pay1]
        for l in range(2):
            g.level_grid_bind(0, l, STORAGE[s["storage"]], s["level"][l][0].ptr, s["level"][l][1], 0.0, 1.0)
        s["bids"] = g.to_device(g.active_blocks())
        s["out"], s["res"] = _device(s["n"] * (bs + 2) ** 3, "<f4")
    elif f in ("solve", "warmnet"):
        low, diag, b, xs, _ = _system(case, seed, torch.tensor(g.active_blocks(), device="cuda").long())
        _channels(s, {CH_X: xs, CH_B: b, CH_COEF: low[0], CH_COEF + 1: low[1], CH_COEF + 2: low[2], CH_COEF + 3: diag})
        torch.cuda.synchronize()
        g.poisson_set_coefficients(CH_COEF, CH_COEF + 1, CH_COEF + 2, CH_COEF + 3)
        if f == "warmnet":
            w, c = _weights(seed)
            g.warmnet_set([x.numpy() for x in w], [x.numpy() for x in c])
    elif f == "render":
        s["out"], s["res"] = _device(case["width"] * case["height"] * 3, "|u1")
    return s


def _sweeps(s, kind, iters):
    s["g"].applyChannelPdeFast(0, laplTyp=-(LAPL[kind] + G.OPT_8_COLOR_SCHEME), doConstrZeroOne=1, numIter=iters,
                               timeStep=0.1, variant=G.SWEEP_FAST if s["variant"] == "fast" else G.SWEEP_EXACT)


def run(s):
    f, g = s["family"], s["g"]
    if f == "pipeline":
        _layout(s)
        g.splat(s["buf"], s["points"], R, NB)
        g.splat_finalize(R, NB)
        _sweeps(s, "mcf", s["iters"])
        return _payload(g, s)
    if f == "sweep":
        _sweeps(s, s["kind"], s["iters"])
        return _payload(g, s)
    if f == "splat":
        if s["storage"] == "f32":  # the FP32 splat takes the minimum with what the channel holds
            g.fill(1.0, 0)
        g.splat(s["buf"], s["points"], R, NB)
        g.splat_finalize(R, NB)
        return _payload(g, s)
    if f == "g2p":
        g.interpolate_device(0, s["buf"], s["points"], s["out"], G.IP_RENDER_DENS if s["storage"] == "u16" else 0)
    elif f == "restrict":
        g._check(g.L.msbg_gpu_downsample_channel(g.h, 0, C.c_void_p(s["out"].ptr), 0))
    elif f == "halo":
        g.fill_halo_blocks_device(0, 0, s["bids"], s["n"], 1, G.BC_COARSE_LEVEL, s["out"])
    elif f == "solve":
        g.fill(0.0, CH_X)
        if s["method"] == "plain":
            g.mgpcg_solve(CH_X, CH_B, tol=1e-6, max_iter=200)
        else:
            g.mgpcg_solve_mixed(CH_X, CH_B, tol=1e-6, max_outer=12, inner_tol=3e-2, max_inner=60)
        return _payload(g, s, CH_X, "f32")
    elif f == "warmnet":
        loss, w, c = g.warmnet_loss_grad(CH_B, CH_X)
        return {"loss": loss, "w": w, "c": c}
    elif f == "render":
        g.render_device(0, s["width"], s["height"], G.DEMO_CAMERA, s["out"])
    return s["res"]


def work(case):
    """Bytes: inputs read once, outputs written once (a sweep reads and writes its field in every
    iteration, as the field is larger than what a chip keeps).  Operations: those of the arithmetic."""
    f, bs = case["family"], case["bs"]
    n = case["objects"] * case["pts"]
    blocks = int(_blocks(case, _cloud(case, 0, DEV)).numel())
    v, e = blocks * bs ** 3, 4 if case["storage"] == "f32" else 2
    sphere = 268 * 6  # voxels of a particle's sphere, operations each
    if f == "pipeline":
        return {"bytes": 12 * n + v * e * (1 + 2 * case["iters"]), "flops": n * sphere + 62 * v * case["iters"]}
    if f == "sweep":
        return {"bytes": 2 * e * v * case["iters"], "flops": (62 if case["kind"] == "mcf" else 9) * v * case["iters"]}
    if f == "splat":
        return {"bytes": 12 * n + v * e, "flops": n * sphere}
    if f == "g2p":
        return {"bytes": 16 * n + min(v, 8 * n) * e, "flops": 27 * n}
    if f == "restrict":
        return {"bytes": v * e + v // 8 * 4, "flops": v // 8 * 128}
    if f == "halo":
        return {"bytes": blocks * (bs ** 3 * e + (bs + 2) ** 3 * 4), "flops": 0}
    if f == "solve":  # about 6 iterations, each an operator and 8 smoothing sweeps with 14 operations a cell
        return {"bytes": 6 * 4 * v, "flops": 6 * 12 * 14 * v}
    if f == "warmnet":
        macs = 27 * (2 * 16 + 16 * 16 + 16 * 16 + 16 * 2) * v // 8
        return {"bytes": 3 * 4 * v, "flops": 2 * 3 * macs}
    return {"bytes": 3 * case["width"] * case["height"] + v * e, "flops": 9 * case["width"] * case["height"] * 0.5 * max(
        case["nx"], case["ny"], case["nz"]) * bs}


# ---- the same in 64 bits ------------------------------------------------------------------------

class _Field64:
    """A field on the scene's blocks and its gathers, in FP64 (slot grid with one empty rim)."""

    def __init__(self, case, bids):
        self.bs, self.bids = case["bs"], bids
        self.nb = (case["nx"], case["ny"], case["nz"])
        nx, ny, nz = self.nb
        self.slot = torch.full((nz * ny * nx,), -1, device=bids.device, dtype=torch.int64)
        self.slot[bids] = torch.arange(bids.numel(), device=bids.device)

    def coords(self, which):
        nx, ny, _ = self.nb
        b = self.bids[which]
        return b % nx, (b // nx) % ny, b // (nx * ny)

    def read(self, f, x, y, z):
        """Values at voxel coordinates inside the domain (broadcast), 0 in blocks without payload."""
        bs, (nx, ny, _) = self.bs, self.nb
        s = self.slot[(z // bs * ny + y // bs) * nx + x // bs]
        at = ((s.clamp_min(0) * bs + z % bs) * bs + y % bs) * bs + x % bs
        return torch.where(s >= 0, f.reshape(-1)[at], 0.0)

    def boxes(self, f, which, own):
        """Halo-1 boxes of the blocks; outside the domain: the own block's nearest voxel (own), else
        the voxel at the clamped position."""
        bs = self.bs
        r = torch.arange(-1, bs + 1, device=f.device)
        g, lim, inside = [], [], []
        for b, n in zip(self.coords(which), self.nb):
            p = b[:, None] * bs + r
            inside.append((p >= 0) & (p < n * bs))
            lim.append(torch.minimum(torch.maximum(p, b[:, None] * bs), b[:, None] * bs + bs - 1))
            g.append(p.clamp(0, n * bs - 1))

        def full(a):
            return a[0][:, None, None, :], a[1][:, None, :, None], a[2][:, :, None, None]

        v = self.read(f, *full(g))
        if own:
            ix, iy, iz = full(inside)
            v = torch.where(ix & iy & iz, v, self.read(f, *full(lim)))
        return v

    def sweeps(self, f, kind, iters, dt=0.1):
        f = f.clone()
        bx, by, bz = self.coords(slice(None))
        color = (bx & 1) + 2 * (by & 1) + 4 * (bz & 1)
        for _ in range(iters):
            for c in range(8):
                for part in torch.nonzero(color == c)[:, 0].split(2048):
                    if not part.numel():
                        continue
                    b = self.boxes(f, part, True)
                    i = slice(1, -1)

                    def F(dx, dy, dz):
                        e = self.bs + 1
                        return b[:, 1 + dz:e + dz, 1 + dy:e + dy, 1 + dx:e + dx]

                    f0 = b[:, i, i, i]
                    if kind == "jacobi":
                        s6 = F(-1, 0, 0) + F(1, 0, 0) + F(0, -1, 0) + F(0, 1, 0) + F(0, 0, -1) + F(0, 0, 1)
                        v = (f0 + dt * s6) / (1 + 6 * dt)
                    else:
                        fx, fy, fz = (0.5 * (F(*p) - F(*(-q for q in p))) for p in ((1, 0, 0), (0, 1, 0), (0, 0, 1)))
                        fxx, fyy, fzz = (F(*p) + F(*(-q for q in p)) - 2 * f0 for p in ((1, 0, 0), (0, 1, 0), (0, 0, 1)))

                        def mixed(a, d):
                            def at(i, j):
                                p = [0, 0, 0]
                                p[a], p[d] = i, j
                                return F(*p)
                            return 0.25 * (at(1, 1) - at(1, -1) - at(-1, 1) + at(-1, -1))

                        xx, yy, zz = fx * fx, fy * fy, fz * fz
                        h = (yy + zz) * fxx + (xx + zz) * fyy + (xx + yy) * fzz
                        h -= 2 * (fx * fy * mixed(0, 1) + fx * fz * mixed(0, 2) + fy * fz * mixed(1, 2))
                        g2 = xx + yy + zz
                        h = torch.where(g2 > float(torch.tensor(1e-7)), h / g2, 0.0)
                        v = f0 + (dt * h).clamp(-0.1, 0.1)
                    f[part] = v.clamp(0, 1).reshape(part.numel(), -1)
        return f


def _field(case, pts, field):
    """The splatted and finalised field: distances and density in the FP32 steps that define it."""
    bs, storage = case["bs"], case["storage"]
    dev = pts.device
    m = torch.ones(field.bids.numel() * bs ** 3, device=dev)
    r, hi = R + NB, torch.tensor([case["nx"], case["ny"], case["nz"]], device=dev) * bs - 1
    o = torch.arange(9, device=dev, dtype=torch.int32)
    nx, ny, _ = field.nb
    for p in pts.split(65536):
        lo = torch.ceil(p - r - 0.5).to(torch.int32).clamp_min(0)
        up = torch.minimum(torch.floor(p + r - 0.5).to(torch.int32), hi)
        i = lo[:, :, None] + o
        ok = i <= up[:, :, None]
        d = i.float() - (p - 0.5)[:, :, None]
        d = d * d
        d2 = (d[:, 2, :, None, None] + d[:, 1, None, :, None]) + d[:, 0, None, None, :]
        ok = ok[:, 2, :, None, None] & ok[:, 1, None, :, None] & ok[:, 0, None, None, :] & (d2 <= r * r)
        k, c, b, a = torch.nonzero(ok).unbind(1)
        x, y, z = i[k, 0, a].long(), i[k, 1, b].long(), i[k, 2, c].long()
        s = field.slot[(z // bs * ny + y // bs) * nx + x // bs]
        at = ((s * bs + z % bs) * bs + y % bs) * bs + x % bs
        m.scatter_reduce_(0, at, d2[k, c, b, a] * (1.0 / (r * r)), "amin")
    if storage == "u16":
        m = torch.floor(m * 65535.0 + 0.5) * torch.tensor(1 / 65535.0, device=dev)
    elif storage == "f16":
        m = m.half().float()
    dist = torch.sqrt(m * (r * r)) - R
    lin = ((dist + R) * torch.tensor(1.0 / (2 * R + NB), device=dev)).masked_fill(dist < -R, 0.0).masked_fill(dist >= R + NB, 1.0)
    f = torch.where(m < 0.999, 1.0 - lin, 0.0)
    if storage == "u16":
        return (torch.floor(f * 65535.0 + 0.5).double() / 65535.0).reshape(-1, bs ** 3)
    return (f.half() if storage == "f16" else f).double().reshape(-1, bs ** 3)


def _conjugate_gradients(low, diag, nbr, b, tol=1e-11):
    w = []
    for a in range(3):
        lo, up = nbr[2 * a], nbr[2 * a + 1]
        w += [torch.where(lo >= 0, low[a], 0), torch.where(up >= 0, low[a][up.clamp_min(0)], 0)]
    idx = [i.clamp_min(0) for i in nbr]
    x, r = torch.zeros_like(b), b.clone()
    z = r / diag
    p, rz, stop = z.clone(), torch.dot(r, z), float(torch.dot(b, b)) * tol * tol
    for it in range(4000):
        q = diag * p
        for wi, i in zip(w, idx):
            q -= wi * p[i]
        alpha = rz / torch.dot(p, q)
        x += alpha * p
        r -= alpha * q
        if it % 25 == 24 and float(torch.dot(r, r)) <= stop:
            break
        z = r / diag
        new = torch.dot(r, z)
        p = z + (new / rz) * p
        rz = new
    return x


def _gradients(case, seed, bids):
    """The network's loss and gradients: weights and the convolutions' inputs rounded to BF16 going
    forward, as the network is defined; all else in FP64."""
    low, diag, b, xs, nbr = _system(case, seed, bids)
    del nbr
    bs, h = case["bs"], case["bs"] // 2
    n = bids.numel()

    def children(t):
        return t.double().reshape(n, h, 2, h, 2, h, 2).permute(0, 1, 3, 5, 2, 4, 6).reshape(n * h ** 3, 8)

    b1, xbar = children(b).sum(1), children(xs).mean(1)
    # level-1 diagonal of P^T A P / 2: the children's diagonals less twice the faces inside the cell
    inner = children(diag).sum(1)
    for a in range(3):
        c = children(low[a])
        inner -= 2 * sum(c[:, k] for k in range(8) if (k >> a) & 1)
    d1 = 0.5 * inner
    S = b1.square().mean().sqrt()
    net = dict(case, bs=h)
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    slot = torch.full((nz + 2, ny + 2, nx + 2), -1, device=bids.device, dtype=torch.int64)
    bx, by, bz = bids % nx + 1, (bids // nx) % ny + 1, bids // (nx * ny) + 1
    slot[bz, by, bx] = torch.arange(n, device=bids.device)
    i = torch.arange(h, device=bids.device)

    def tap(t):  # cell index of the tap's neighbour, n h^3 (a zero row) where there is none
        p = [i + t % 3 - 1, i + (t // 3) % 3 - 1, i + t // 9 - 1]
        q = [torch.div(v, h, rounding_mode="floor") for v in p]
        s = slot[bz[:, None, None, None] + q[2][:, None, None], by[:, None, None, None] + q[1][:, None],
                 bx[:, None, None, None] + q[0]]
        at = ((s * h + (p[2] % h)[:, None, None]) * h + (p[1] % h)[:, None]) * h + p[0] % h
        return torch.where(s >= 0, at, n * net["bs"] ** 3).reshape(-1)

    taps = [tap(t) for t in range(27)]

    def bf(t):
        return t.float().bfloat16().double()

    w, c = _weights(seed)
    W, c = [bf(x.to(bids.device)) for x in w], [x.double().to(bids.device) for x in c]
    acts = [torch.stack([b1 / S, d1 / d1.mean() - 1], 1)]
    for l in range(4):
        a = torch.cat([bf(acts[-1]), torch.zeros(1, acts[-1].shape[1], device=bids.device, dtype=torch.float64)])
        y = c[l] + sum(a[taps[t]] @ W[l][t] for t in range(27))
        acts.append(y.relu() if l < 3 else y)

    def mean2(t):  # mean over the 2x2x2 cells of a parent, on each of them
        m = t.reshape(n, h // 2, 2, h // 2, 2, h // 2, 2).mean((2, 4, 6), keepdim=True)
        return m.expand(n, h // 2, 2, h // 2, 2, h // 2, 2).reshape(-1)

    x1 = S * (acts[4][:, 0] + mean2(acts[4][:, 1]))
    den = xbar.square().sum()
    loss = (x1 - xbar).square().sum() / den
    gx = 2 * (x1 - xbar) / den
    g = torch.stack([S * gx, S * mean2(gx)], 1)
    gw, gc = [None] * 4, [None] * 4
    for l in (3, 2, 1, 0):
        if l < 3:
            g = g * (acts[l + 1] > 0)
        a = torch.cat([acts[l], torch.zeros(1, acts[l].shape[1], device=bids.device, dtype=torch.float64)])
        gw[l] = torch.stack([a[taps[t]].T @ g for t in range(27)])
        gc[l] = g.sum(0)
        if l:
            gp = torch.cat([g, torch.zeros(1, g.shape[1], device=bids.device, dtype=torch.float64)])
            g = sum(gp[taps[26 - t]] @ W[l][t].T for t in range(27))  # tap 26 - t looks the other way
    return {"loss": float(loss), "w": gw, "c": gc}


def exact(case, seed):
    f, bs = case["family"], case["bs"]
    if f in ("halo", "render"):
        return None  # copies of stored values, and bytes
    if case["storage"] == "u16" and f in ("pipeline", "sweep", "splat"):
        return None  # whole numbers
    pts = _cloud(case, seed, DEV)
    bids = _blocks(case, pts)
    if f == "solve":
        low, diag, b, _, nbr = _system(case, seed, bids)
        return _conjugate_gradients([x.double() for x in low], diag.double(), nbr, b.double()).reshape(-1, bs ** 3)
    if f == "warmnet":
        return _gradients(case, seed, bids)
    field = _Field64(case, bids)
    phi = _field(case, pts, field)
    if f == "splat":
        return phi
    if f == "pipeline":
        return field.sweeps(phi, "mcf", case["iters"])
    if f == "sweep":
        return field.sweeps(phi, case["kind"], case["iters"])
    if f == "g2p":
        gen = torch.Generator(device=DEV).manual_seed(int(seed) + 11)
        p = pts[torch.randperm(pts.shape[0], generator=gen, device=DEV)].double() - 0.5
        i = torch.floor(p)
        t = p - i
        hi = torch.tensor([case["nx"], case["ny"], case["nz"]], device=DEV) * bs - 1
        out = 0.0
        for k in range(8):
            o = torch.tensor([k & 1, (k >> 1) & 1, k >> 2], device=DEV)
            q = torch.minimum((i.long() + o).clamp_min(0), hi)
            out = out + torch.where(o == 1, t, 1 - t).prod(1) * field.read(phi, q[:, 0], q[:, 1], q[:, 2])
        return out
    k = torch.tensor([1.0, 3.0, 3.0, 1.0], device=DEV, dtype=torch.float64) / 8
    res = []
    for part in torch.arange(bids.numel(), device=DEV).split(1024):
        b = field.boxes(phi, part, False)
        for dim in (1, 2, 3):
            b = (b.unfold(dim, 4, 2) * k).sum(-1)
        res.append(b.reshape(part.numel(), -1))
    return torch.cat(res).reshape(-1)
