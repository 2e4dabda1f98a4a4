"""The work that programs built on mirorr_b200 have it do, as cases to be timed.

A case is a dict of plain values.  `prepare` makes what a program holds before
the call (volumes, masks, point pairs, the matcher or batch handle), `run` is
one pass through the public entry points, `work` the bytes and operations the
pass cannot do without, and `exact` its result in 64 bits from plain torch.

Kinds:
  match      one GetOffsets call of the C interface on device volumes, into the
             program's own arrays: the call a registration makes once or twice
             per iteration, and the one a program makes that keeps its own
             optimiser.
  register   a whole registration, from host arrays or device volumes.
  batch      several registrations of uneven sizes through one Batch.
  resample   one image + mask pass onto another grid, device to device.
  lts        one trimmed least-squares fit on device point pairs.
  final      the last resampling of a registration, host array to host array.
"""
import ctypes
import math
import random

import numpy as np
import torch

import mirorr_b200 as mb

_DEV = "cuda:0"
_CTX = []


def _context():
    """The program's one context (a device, a stream and its scratch memory)."""
    if not _CTX:
        _CTX.append(mb.Context(0))
    return _CTX[0]


# ---- the cases ----------------------------------------------------------------

def _match(name, size, storage="f32", bw=4, nw=7, gap=3, keep=1.0, masks=False, scores=False):
    return {"name": name, "kind": "match", "nx": size[0], "ny": size[1], "nz": size[2],
            "storage": storage, "bw": bw, "nw": nw, "gap": gap, "keep": keep, "masks": masks,
            "scores": scores}


def _register(name, size, symmetric, affine, levels, nw, gap, keep, host, gaussians):
    return {"name": name, "kind": "register", "nx": size[0], "ny": size[1], "nz": size[2],
            "symmetric": symmetric, "affine": affine, "levels": levels, "nw": nw, "gap": gap,
            "keep": keep, "host": host, "gaussians": gaussians}


def listed():
    return [
        # The coarsest level of a classic rigid registration of 128 x 128 x 64:
        # 1,920 blocks, the top half by variance, called ten times a level.
        # Launches and latency decide.  The scores are read back too.
        _match("match_coarse_level", (64, 64, 32), nw=7, gap=4, keep=0.5, scores=True),
        # The matcher as it comes (block 4, window 5, spacing 2), on a volume
        # with odd axes: what a program gets that sets the images and nothing else.
        _match("match_default_params", (131, 117, 61), nw=5, gap=2, scores=True),
        # The finest level of the symmetric affine registration below: 300
        # thousand blocks of 729 candidates, the most frequent large call.
        _match("match_finest_level", (256, 256, 128), nw=9, gap=3),
        # The command line's window and spacing, ragged axes, a field of view on
        # both images: blocks and windows across the mask edges.
        _match("match_masked_ragged", (219, 203, 107), nw=7, gap=3, masks=True),
        # A pair of the batched configuration's mean size, stored as BF16; the
        # scores are read back as weights.
        _match("match_bf16", (208, 208, 104), storage="bf16", nw=7, gap=3, scores=True),
        # The finest level of the large configuration: 512 x 512 x 256 stored as
        # FP16, block 5, radius 5, the top 30 % of 2.4 million blocks.
        _match("match_f16_block5_large", (512, 512, 256), storage="f16", bw=5, nw=11, gap=3,
               keep=0.3),
        # One classic rigid registration from host arrays, two levels: the small job.
        _register("register_classic_rigid", (128, 128, 64), False, False, 2, 7, 4, 0.5, True, 40),
        # One symmetric affine registration of device volumes, three levels: the
        # headline job.
        _register("register_symmetric_affine", (256, 256, 128), True, True, 3, 9, 3, 1.0, False,
                  80),
        # Eight pairs of uneven sizes, rigid and affine, stored as BF16, from
        # host arrays through one batch.
        {"name": "batch_bf16_uneven", "kind": "batch", "pairs": 8, "sizes": 2, "storage": "bf16",
         "nw": 7, "gap": 3, "levels": 3, "symmetric": False},
        # An image and its mask into the middle space at the finest level.
        {"name": "resample_finest_level", "kind": "resample", "nx": 256, "ny": 256, "nz": 128,
         "ox": 256, "oy": 256, "oz": 128, "nearest": False},
        # The fit of the finest level's pairs, a third of them outliers.
        {"name": "lts_affine", "kind": "lts", "points": 240000, "affine": True, "keep": 0.5},
        # What the command line does last, with its default interpolator.
        {"name": "final_bspline", "kind": "final", "nx": 256, "ny": 256, "nz": 128, "ox": 256,
         "oy": 256, "oz": 128, "interpolator": "bspline"},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _size(rng, lo, hi):
    """A volume of lo to hi voxels whose axes are within a factor of about two
    of each other, with the shorter z of most scans; odd and even."""
    n = math.exp(rng.uniform(math.log(lo), math.log(hi)))
    fx, fy, fz = rng.uniform(0.8, 1.25), rng.uniform(0.8, 1.25), rng.uniform(0.4, 0.9)
    s = (n / (fx * fy * fz)) ** (1.0 / 3.0)
    return [max(20, int(round(s * f))) for f in (fx, fy, fz)]


def draw(rng):
    kind = rng.choice(["match", "match", "match", "match16", "match16", "register", "batch",
                       "resample", "lts", "final"])
    if kind == "match":
        nx, ny, nz = _size(rng, 60e3, 9e6)
        return _nameless(_match("", (nx, ny, nz), nw=rng.choice([5, 7, 9]),
                                gap=rng.choice([2, 3, 4]), keep=rng.choice([0.5, 1.0, 1.0]),
                                masks=rng.random() < 0.4))
    if kind == "match16":
        bw, nw, keep = rng.choice([(4, 7, 1.0), (4, 7, 0.5), (5, 11, 0.3)])
        nx, ny, nz = _size(rng, 60e3, 12e6)
        return _nameless(_match("", (nx, ny, nz), storage=rng.choice(["bf16", "f16"]), bw=bw, nw=nw,
                                gap=rng.choice([3, 4]), keep=keep, masks=rng.random() < 0.4,
                                scores=True))
    if kind == "register":
        nx, ny, nz = _size(rng, 300e3, 6e6)
        return _nameless(_register("", (nx, ny, nz), rng.random() < 0.5, rng.random() < 0.5,
                                   rng.choice([2, 3]), rng.choice([7, 9]), rng.choice([3, 4]),
                                   rng.choice([0.5, 1.0]), rng.random() < 0.5, 60))
    if kind == "batch":
        return {"kind": "batch", "pairs": rng.randint(2, 8), "sizes": rng.randint(10, 10 ** 6),
                "storage": rng.choice(["bf16", "f16"]), "nw": 7, "gap": 3,
                "levels": rng.choice([2, 3]), "symmetric": rng.random() < 0.5}
    if kind == "resample":
        nx, ny, nz = _size(rng, 60e3, 16e6)
        ox, oy, oz = [max(8, int(round(v * rng.uniform(0.7, 1.2)))) for v in (nx, ny, nz)]
        return {"kind": "resample", "nx": nx, "ny": ny, "nz": nz, "ox": ox, "oy": oy, "oz": oz,
                "nearest": rng.random() < 0.25}
    if kind == "lts":
        return {"kind": "lts", "points": _log_int(rng, 1500, 500000),
                "affine": rng.random() < 0.7, "keep": rng.choice([0.5, 0.5, 0.8])}
    nx, ny, nz = _size(rng, 60e3, 9e6)
    ox, oy, oz = [max(8, int(round(v * rng.uniform(0.8, 1.1)))) for v in (nx, ny, nz)]
    return {"kind": "final", "nx": nx, "ny": ny, "nz": nz, "ox": ox, "oy": oy, "oz": oz,
            "interpolator": rng.choice(["bspline", "bspline", "sinc"])}


def _nameless(case):
    return {k: v for k, v in case.items() if k != "name"}


# ---- inputs ---------------------------------------------------------------------

def _rotation(rng, degrees):
    axis = rng.normal(size=3)
    axis /= np.linalg.norm(axis)
    a = math.radians(rng.uniform(0.0, degrees))
    k = np.array([[0, -axis[2], axis[1]], [axis[2], 0, -axis[0]], [-axis[1], axis[0], 0]])
    return np.eye(3) + math.sin(a) * k + (1 - math.cos(a)) * (k @ k)


def _phantom(nx, ny, nz, gaussians, seed, degrees, shift, affine):
    """(fixed, moving) float32 device volumes (z, y, x): a sum of anisotropic
    Gaussians in [0, 1] with N(0, 0.1) noise; the moving image is a second
    modality (a non-monotone map) of the fixed one through a small transform."""
    rng = np.random.default_rng(seed)
    ax = [torch.arange(n, device=_DEV, dtype=torch.float32) for n in (nx, ny, nz)]
    x, y, z = ax[0].view(1, 1, -1), ax[1].view(1, -1, 1), ax[2].view(-1, 1, 1)
    vol = torch.zeros((nz, ny, nx), device=_DEV)
    for _ in range(gaussians):
        c = rng.uniform([0, 0, 0], [nx - 1, ny - 1, nz - 1])
        sig = rng.uniform(4.0, 16.0, size=3)
        r, _ = np.linalg.qr(rng.normal(size=(3, 3)))
        q = r @ np.diag(1.0 / sig ** 2) @ r.T
        amp = float(rng.uniform(0.0, 1.0))
        reach = 4.0 * sig.max()
        lo = np.maximum(np.floor(c - reach), 0).astype(int)
        hi = np.minimum(np.ceil(c + reach) + 1, [nx, ny, nz]).astype(int)
        dx, dy, dz = (v - float(m) for v, m in
                      zip((x[..., lo[0]:hi[0]], y[:, lo[1]:hi[1]], z[lo[2]:hi[2]]), c))
        e = (q[0, 0] * dx * dx + q[1, 1] * dy * dy + 2 * q[0, 1] * dx * dy) \
            + (q[2, 2] * dz * dz + 2 * q[0, 2] * dx * dz + 2 * q[1, 2] * dy * dz)
        vol[lo[2]:hi[2], lo[1]:hi[1], lo[0]:hi[0]] += amp * torch.exp(-0.5 * e)
    clean = (vol - vol.min()) / (vol.max() - vol.min()).clamp(min=1e-12)
    gen = torch.Generator(device=_DEV)
    gen.manual_seed(int(rng.integers(2 ** 62)))
    fixed = clean + 0.1 * torch.randn(clean.shape, generator=gen, device=_DEV)
    m = _rotation(rng, degrees)
    if affine:
        m = m @ np.diag(rng.uniform(0.9, 1.1, size=3))
    centre = (np.array([nx, ny, nz]) - 1.0) / 2.0
    off = centre + rng.uniform(-shift, shift, size=3) - m @ centre
    mapped = 0.6 * torch.sin(3.0 * clean) + 0.4 * clean * clean
    moving = torch.empty_like(mapped)
    scale = [2.0 / max(n - 1, 1) for n in (nx, ny, nz)]
    for k0 in range(0, nz, 64):
        zz = z[k0:k0 + 64]
        g = [(m[r, 0] * x + m[r, 1] * y + (m[r, 2] * zz + float(off[r]))) * scale[r] - 1.0
             for r in range(3)]
        g = torch.stack(torch.broadcast_tensors(*g), dim=-1).unsqueeze(0)
        moving[k0:k0 + 64] = torch.nn.functional.grid_sample(
            mapped[None, None], g, mode="bilinear", padding_mode="zeros", align_corners=True)[0, 0]
    moving += 0.1 * torch.randn(clean.shape, generator=gen, device=_DEV)
    return fixed, moving


def _field_of_view(nx, ny, nz, rng):
    """An ellipsoid field of view (uint8, 255 inside) with an offset centre."""
    c = [(n - 1) / 2 + rng.uniform(-0.06, 0.06) * n for n in (nx, ny, nz)]
    r = [rng.uniform(0.42, 0.56) * n for n in (nx, ny, nz)]
    v = [((torch.arange(n, device=_DEV, dtype=torch.float32) - m) / s) ** 2
         for n, m, s in zip((nx, ny, nz), c, r)]
    inside = v[0].view(1, 1, -1) + v[1].view(1, -1, 1) + v[2].view(-1, 1, 1) <= 1.0
    return (inside.to(torch.uint8) * 255).contiguous()


def _match_inputs(case, seed):
    """(base, search, base mask, search mask): a pair in the middle of a
    registration, within about a degree and two voxels of each other."""
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    fixed, moving = _phantom(nx, ny, nz, 60, seed, 1.0, 2.0, False)
    if case["storage"] != "f32":
        t = torch.bfloat16 if case["storage"] == "bf16" else torch.float16
        fixed, moving = fixed.to(t), moving.to(t)
    bm = sm = None
    if case["masks"]:
        rng = np.random.default_rng(seed + 17)
        bm, sm = _field_of_view(nx, ny, nz, rng), _field_of_view(nx, ny, nz, rng)
    return moving.contiguous(), fixed.contiguous(), bm, sm


def _resample_inputs(case, seed):
    rng = np.random.default_rng(seed)
    img, _ = _phantom(case["nx"], case["ny"], case["nz"], 30, seed, 1.0, 1.0, False)
    mask = _field_of_view(case["nx"], case["ny"], case["nz"], rng)
    gi = mb.Geometry.make((case["nx"], case["ny"], case["nz"]))
    go = mb.Geometry.make((case["ox"], case["oy"], case["oz"]))
    m = _rotation(rng, 4.0) @ np.diag(rng.uniform(0.97, 1.03, size=3))
    ci = (np.array([case["nx"], case["ny"], case["nz"]]) - 1.0) / 2.0
    co = (np.array([case["ox"], case["oy"], case["oz"]]) - 1.0) / 2.0
    C, e = mb.resample_map(go, gi, m, ci - m @ co + rng.uniform(-3, 3, size=3))
    return img, mask, C, e


def _lts_inputs(case, seed):
    """Matches as the matcher emits them: block positions on the grid, match
    positions on the voxel lattice near a small transform of them, a third of
    them anywhere in the window."""
    rng = np.random.default_rng(seed)
    n = case["points"]
    side = max(8.0, (27.0 * n) ** (1.0 / 3.0))
    p = 3.0 * np.floor(rng.uniform(0, side / 3.0, size=(n, 3))) + 2.0
    m = _rotation(rng, 2.0)
    if case["affine"]:
        m = m @ np.diag(rng.uniform(0.98, 1.02, size=3))
    c = np.full(3, side / 2)
    q = np.rint((p - c) @ m.T + c + rng.uniform(-1.5, 1.5, size=3) + rng.normal(0, 0.4, (n, 3)))
    out = rng.random(n) < 0.33
    q[out] = p[out] + rng.integers(-4, 5, size=(int(out.sum()), 3))
    return torch.from_numpy(p).to(_DEV), torch.from_numpy(q).to(_DEV)


def _batch_sizes(case):
    r = random.Random(case["sizes"])
    return [(r.randint(96, 320), r.randint(96, 320), r.randint(48, 160))
            for _ in range(case["pairs"])]


# ---- prepare and run --------------------------------------------------------------

def prepare(case, seed):
    ctx = _context()
    s = {"case": case, "ctx": ctx}
    kind = case["kind"]
    if kind == "match":
        base, search, bm, sm = _match_inputs(case, seed)
        g = mb.Geometry.make((case["nx"], case["ny"], case["nz"]))
        m = mb.BlockMatcher(ctx)
        m.SetBlockWidth(case["bw"])
        m.SetNhoodWidth(case["nw"])
        m.SetNhoodGap(case["gap"])
        m.SetBlockKeep(case["keep"])
        m.SetStorage(case["storage"])
        if case["storage"] == "f32":
            m.SetBaseImageDevice(g, base.data_ptr())
            m.SetSearchImageDevice(g, search.data_ptr())
        else:
            m.SetBaseImageDevice16(g, base.data_ptr())
            m.SetSearchImageDevice16(g, search.data_ptr())
        if bm is not None:
            m.SetBaseMaskDevice(bm.data_ptr())
            m.SetSearchMaskDevice(sm.data_ptr())
        nb = int(np.prod(m.Grid()[0]))
        s.update(matcher=m, hold=(base, search, bm, sm), capacity=nb,
                 blocks=np.zeros((nb, 3)), matches=np.zeros((nb, 3)),
                 best=np.zeros(nb, np.float32), second=np.zeros(nb, np.float32),
                 status=np.zeros(nb, np.uint8))
    elif kind == "register":
        nx, ny, nz = case["nx"], case["ny"], case["nz"]
        degrees, shift = (8.0, 12.0) if case["affine"] else (5.0, 8.0)
        fixed, moving = _phantom(nx, ny, nz, case["gaussians"], seed, degrees, shift,
                                 case["affine"])
        if case["host"]:
            fixed, moving = fixed.cpu().numpy(), moving.cpu().numpy()
        s.update(fixed=fixed, moving=moving, geom=mb.Geometry.make((nx, ny, nz)),
                 params=mb.reg_params(symmetric=case["symmetric"],
                                      kind="affine" if case["affine"] else "rigid",
                                      levels=case["levels"], iterations=10, nhood_gap=case["gap"],
                                      nhood_width=case["nw"], block_keep=case["keep"]))
    elif kind == "batch":
        pairs = []
        for i, size in enumerate(_batch_sizes(case)):
            affine = i % 2 == 1
            f, m = _phantom(*size, 40, seed * 1009 + i, 5.0, 8.0, affine)
            p = mb.reg_params(symmetric=case["symmetric"], kind="affine" if affine else "rigid",
                              levels=case["levels"], iterations=10, nhood_gap=case["gap"],
                              nhood_width=case["nw"], storage=case["storage"])
            pairs.append((mb.to_storage(f.cpu().numpy(), case["storage"]),
                          mb.to_storage(m.cpu().numpy(), case["storage"]), p))
        s.update(pairs=pairs, batch=mb.Batch(ctx, max_slots=case["pairs"]))
    elif kind == "resample":
        img, mask, C, e = _resample_inputs(case, seed)
        out = torch.empty((case["oz"], case["oy"], case["ox"]), device=_DEV)
        s.update(img=img, mask=mask, C=C, e=e, out=out,
                 outm=torch.empty(out.shape, dtype=torch.uint8, device=_DEV))
    elif kind == "lts":
        p, q = _lts_inputs(case, seed)
        s.update(p=p, q=q)
    else:
        img, _, C, e = _resample_inputs(case, seed)
        s.update(img=img.cpu().numpy(), C=C, e=e)
    torch.cuda.synchronize()  # the library works on a stream of its own
    return s


def _transform(t):
    return {"matrix": t.M, "offset": t.off, "center": np.array(t.center),
            "params": t.param_vector()}


def run(s):
    case, ctx = s["case"], s["ctx"]
    kind = case["kind"]
    if kind == "match":
        h, n, lib = s["matcher"]._h, ctypes.c_size_t(0), mb.lib()
        st = lib.mirorr_bm_get_offsets(h, s["capacity"], s["blocks"].ctypes.data,
                                       s["matches"].ctypes.data, ctypes.byref(n))
        out = {"kept": n.value, "blocks": s["blocks"], "matches": s["matches"]}
        if st == 0 and case["scores"]:
            st = lib.mirorr_bm_block_results(h, s["capacity"], None, s["best"].ctypes.data,
                                             s["second"].ctypes.data, s["status"].ctypes.data,
                                             ctypes.byref(n))
            out.update(best=s["best"], second=s["second"], status=s["status"])
        if st != 0:
            raise mb.MirorrError(st, lib.mirorr_last_error().decode())
        return out
    if kind == "register":
        if case["host"]:
            t, st = mb.register(ctx, s["fixed"], s["moving"], s["params"], s["geom"], s["geom"])
        else:
            t, st = mb.register_device(ctx, s["fixed"].data_ptr(), s["geom"],
                                       s["moving"].data_ptr(), s["geom"], s["params"])
        return dict(_transform(t), iterations=np.array(st.iterations_run[:st.levels_run]),
                    evaluated=int(st.block_ncc_evaluated))
    if kind == "batch":
        b = s["batch"]
        ids = [b.submit(f, m, p) for f, m, p in s["pairs"]]
        b.run()
        return [_transform(b.result(i)[0]) for i in ids]
    if kind == "resample":
        mb.resample_device(ctx, s["img"].data_ptr(), s["mask"].data_ptr(),
                           (case["nx"], case["ny"], case["nz"]),
                           (case["ox"], case["oy"], case["oz"]), s["C"], s["e"],
                           s["out"].data_ptr(), s["outm"].data_ptr(), nearest=case["nearest"])
        return {"image": s["out"], "mask": s["outm"]}
    if kind == "lts":
        t = mb.Transform.make(mb.AFFINE if case["affine"] else mb.RIGID,
                              [1.0, 0, 0, 0, 1.0, 0, 0, 0, 1.0, 0, 0, 0] if case["affine"]
                              else [0.0] * 6)
        n = mb.lts_noalloc(ctx, t, case["points"], s["p"].data_ptr(), s["q"].data_ptr(),
                           case["keep"])
        return dict(_transform(t), iterations=n)
    return {"image": mb.resample_final(ctx, s["img"], (case["ox"], case["oy"], case["oz"]),
                                       s["C"], s["e"], case["interpolator"])}


# ---- the work of one pass -------------------------------------------------------------

def _grid(n, bw, gap):
    k = (n - bw) // gap + 1
    return k, (n - gap * (k - 1) - bw) // 2


def _candidates(n, bw, gap, nw):
    """Candidate positions along one axis, summed over its blocks."""
    k, start = _grid(n, bw, gap)
    r, total = nw // 2, 0
    for b in range(k):
        o = start + b * gap
        total += min(o - r + nw, n - bw + 1) - max(o - r, 0)
    return total


def _match_work(size, bw, gap, nw, keep, elem, masks):
    n = size[0] * size[1] * size[2]
    blocks = cands = 1
    for v in size:
        blocks *= _grid(v, bw, gap)[0]
        cands *= _candidates(v, bw, gap, nw)
    keep = min(keep, 1.0)
    # two volumes (and masks) read, two points of three doubles written per kept
    # block, taken as half of the searched ones; 2 B flops a candidate
    return {"bytes": n * (2 * elem + (2 if masks else 0)) + 24.0 * blocks * keep,
            "flops": 2.0 * bw ** 3 * cands * keep}


def _register_work(size, levels, symmetric, bw, gap, nw, keep, elem):
    """The matcher calls of five iterations a level (a registration stops when
    its parameters do) and the images and masks resampled for them."""
    total = {"bytes": 2.0 * elem * size[0] * size[1] * size[2], "flops": 0.0}
    for lev in range(levels):
        s = [max(bw, v >> lev) for v in size]
        w = _match_work(s, bw, gap, nw, keep, elem, True)
        calls = 5 * (2 if symmetric else 1)
        total["bytes"] += calls * (w["bytes"] + (2 * elem + 2) * s[0] * s[1] * s[2])
        total["flops"] += calls * w["flops"]
    return total


def work(case):
    kind = case["kind"]
    if kind == "match":
        return _match_work((case["nx"], case["ny"], case["nz"]), case["bw"], case["gap"],
                           case["nw"], case["keep"], 4 if case["storage"] == "f32" else 2,
                           case["masks"])
    if kind == "register":
        return _register_work((case["nx"], case["ny"], case["nz"]), case["levels"],
                              case["symmetric"], 4, case["gap"], case["nw"], case["keep"], 4)
    if kind == "batch":
        w = [_register_work(s, case["levels"], case["symmetric"], 4, case["gap"], case["nw"], 1.0,
                            2) for s in _batch_sizes(case)]
        return {k: sum(v[k] for v in w) for k in ("bytes", "flops")}
    if kind == "lts":
        # six doubles a pair; the moments of a pair are some sixty operations
        return {"bytes": 48.0 * case["points"], "flops": 100.0 * case["points"]}
    nin, nout = case["nx"] * case["ny"] * case["nz"], case["ox"] * case["oy"] * case["oz"]
    if kind == "resample":
        return {"bytes": 5.0 * (nin + nout), "flops": 25.0 * nout}
    taps = 64 if case["interpolator"] == "bspline" else 1000
    return {"bytes": 4.0 * (nin + nout), "flops": 2.0 * taps * nout}


# ---- 64-bit results ------------------------------------------------------------------

def _exact_match(case, seed):
    """Every block against every candidate of its window: means over the block,
    sums over the voxels inside both masks, the squared correlation, the best
    and second best (the first in raster order among equals)."""
    base, search, bm, sm = _match_inputs(case, seed)
    size = (case["nx"], case["ny"], case["nz"])
    nx, ny, nz = size
    bw, nw, gap = case["bw"], case["nw"], case["gap"]
    grid = [_grid(n, bw, gap) for n in size]
    ax = [torch.arange(k, device=_DEV) * gap + s for k, s in grid]
    oz, oy, ox = (v.reshape(-1) for v in torch.meshgrid(ax[2], ax[1], ax[0], indexing="ij"))
    dv = torch.arange(bw, device=_DEV)
    vox = ((dv.view(-1, 1, 1) * ny + dv.view(1, -1, 1)) * nx + dv.view(1, 1, -1)).reshape(-1)
    org = (oz * ny + oy) * nx + ox
    nb = org.numel()
    bflat, sflat = base.reshape(-1), search.reshape(-1)
    keep = torch.ones(nb, dtype=torch.bool, device=_DEV)
    chunk = 1 << 17
    if case["keep"] < 1.0:
        var = torch.empty(nb, dtype=torch.float64, device=_DEV)
        for i in range(0, nb, chunk):
            x = bflat[org[i:i + chunk, None] + vox].float()
            var[i:i + chunk] = (x * x).double().mean(1) - x.double().mean(1) ** 2
        k = min(int((1.0 - case["keep"]) * nb), nb - 1)
        keep = var > torch.sort(var).values[k]
    best = torch.full((nb,), -3.0, dtype=torch.float64, device=_DEV)
    second = best.clone()
    arg = org.clone()
    r = nw // 2
    todo = torch.nonzero(keep).reshape(-1)
    for i in range(0, todo.numel(), chunk):
        t = todo[i:i + chunk]
        at = org[t, None] + vox
        x = bflat[at].double()
        xd = x - x.mean(1, keepdim=True)
        mb_ = (bm.reshape(-1)[at] != 0) if bm is not None else None
        if mb_ is not None:
            xd = xd * mb_
        sxx = (xd * xd).sum(1)
        f1, f2 = best[t], second[t]
        pos = torch.full_like(t, -1)
        cx, cy, cz = ox[t], oy[t], oz[t]
        for dz in range(-r, -r + nw):
            for dy in range(-r, -r + nw):
                for dx in range(-r, -r + nw):
                    ok = ((cx + dx >= 0) & (cx + dx <= nx - bw) & (cy + dy >= 0)
                          & (cy + dy <= ny - bw) & (cz + dz >= 0) & (cz + dz <= nz - bw))
                    p = torch.where(ok, org[t] + (dz * ny + dy) * nx + dx, org[t])
                    y = sflat[p[:, None] + vox].double()
                    yd = y - y.mean(1, keepdim=True)
                    if mb_ is None:
                        sxy, sx, sy = (xd * yd).sum(1), sxx, (yd * yd).sum(1)
                    else:
                        ms = sm.reshape(-1)[p[:, None] + vox] != 0
                        yd = yd * ms
                        sxy, sx = (xd * yd).sum(1), (xd * xd * ms).sum(1)
                        sy = (yd * yd * mb_).sum(1)
                    s = torch.where((sx <= 0) | (sy <= 0), -2.0, sxy * sxy / sx / sy)
                    s = torch.where(ok, s, -4.0)
                    up = s > f1
                    f2 = torch.where(up, f1, torch.maximum(f2, s))
                    pos = torch.where(up, p, pos)
                    f1 = torch.where(up, s, f1)
        best[t], second[t] = f1, f2
        arg[t] = torch.where(pos < 0, org[t], pos)
    fb, fs = best.float().double(), second.float().double()
    kept = keep & (fb > 1e-7) & ((fb - fs).abs() > 1e-4)

    def points(lin):
        p = torch.zeros((nb, 3), dtype=torch.float64, device=_DEV)
        p[:lin.numel()] = torch.stack([lin % nx, (lin // nx) % ny, lin // (nx * ny)], 1) + bw / 2
        return p

    out = {"kept": None, "blocks": None, "matches": None}
    if case["storage"] == "f32":  # 16-bit storage: a score at the threshold moves every later row
        out.update(blocks=points(org[kept]), matches=points(arg[kept]))
    if case["scores"]:
        out.update(best=best, second=second, status=None)
    return out


def _continuous(case, C, e):
    o = [torch.arange(case[a], device=_DEV, dtype=torch.float64) for a in ("ox", "oy", "oz")]
    x, y, z = o[0].view(1, 1, -1), o[1].view(1, -1, 1), o[2].view(-1, 1, 1)
    return [float(e[r]) + float(C[r, 0]) * x + float(C[r, 1]) * y + float(C[r, 2]) * z
            for r in range(3)]


def _inside(c, size):
    ok = torch.ones_like(c[0], dtype=torch.bool)
    for v, n in zip(c, size):
        ok &= (v >= -0.5) & (v < n - 0.5)
    return ok


def _exact_resample(case, seed):
    img, mask, C, e = _resample_inputs(case, seed)
    size = (case["nx"], case["ny"], case["nz"])
    c = _continuous(case, C, e)
    ok = _inside(c, size)
    if case["nearest"]:
        i = [torch.floor(v + 0.5).long().clamp(0, n - 1) for v, n in zip(c, size)]
        at = (i[2] * size[1] + i[1]) * size[0] + i[0]
        return {"image": torch.where(ok, img.reshape(-1)[at].double(), 0.0), "mask": None}
    lo = [torch.floor(v).long().clamp(0, n - 1) for v, n in zip(c, size)]
    w = [(v - b).clamp(min=0.0) for v, b in zip(c, lo)]
    hi = [(b + 1).clamp(max=n - 1) for b, n in zip(lo, size)]
    flat = img.reshape(-1)
    val = torch.zeros_like(c[0])
    for kz in (0, 1):
        for ky in (0, 1):
            for kx in (0, 1):
                at = ((hi, lo)[kz == 0][2] * size[1] + (hi, lo)[ky == 0][1]) * size[0] \
                    + (hi, lo)[kx == 0][0]
                f = (w[0] if kx else 1 - w[0]) * (w[1] if ky else 1 - w[1]) \
                    * (w[2] if kz else 1 - w[2])
                val += f * flat[at].double()
    return {"image": torch.where(ok, val, 0.0), "mask": None}


def _bspline_coefficients(v):
    """Cubic B-spline coefficients along the last axis (mirror boundaries)."""
    n = v.shape[-1]
    if n == 1:
        return v
    z = math.sqrt(3.0) - 2.0
    c = list((v * 6.0).unbind(-1))
    k = torch.arange(2 * n - 2, device=v.device, dtype=torch.float64)
    ring = torch.cat([v, v.flip(-1)[..., 1:-1]], -1) * 6.0
    c[0] = (ring * (z ** k)).sum(-1) / (1.0 - z ** (2 * n - 2))
    for i in range(1, n):
        c[i] = c[i] + z * c[i - 1]
    c[n - 1] = z / (z * z - 1.0) * (z * c[n - 2] + c[n - 1])
    for i in range(n - 2, -1, -1):
        c[i] = z * (c[i + 1] - c[i])
    return torch.stack(c, -1)


def _exact_final(case, seed):
    img, _, C, e = _resample_inputs(case, seed)
    size = (case["nx"], case["ny"], case["nz"])
    c = _continuous(case, C, e)
    ok = _inside(c, size)
    low = [torch.floor(v).long() for v in c]
    if case["interpolator"] == "bspline":
        v = img.double()
        for axis in (2, 1, 0):
            v = _bspline_coefficients(v.transpose(axis, 2)).transpose(axis, 2).contiguous()
        taps, first = 4, -1

        def weight(d, k):
            t = (d - (k - 1)).abs()
            return torch.where(t < 1, 2.0 / 3.0 - t * t + t ** 3 / 2, (2 - t).clamp(min=0) ** 3 / 6)

        def index(b, n):
            m = b.abs() % (2 * n - 2) if n > 1 else b * 0
            return torch.where(m >= n, 2 * n - 2 - m, m)
    else:
        v = img.double()
        taps, first = 10, -4

        def weight(d, k):
            t = d - (k - 4)
            return (1 - t * t / 25.0) * torch.sinc(t)

        def index(b, n):
            return b.clamp(0, n - 1)
    flat = v.reshape(-1)
    d = [a - b for a, b in zip(c, low)]
    out = torch.zeros_like(c[0])
    for kz in range(taps):
        for ky in range(taps):
            row = (index(low[2] + first + kz, size[2]) * size[1]
                   + index(low[1] + first + ky, size[1])) * size[0]
            wzy = weight(d[2], kz) * weight(d[1], ky)
            for kx in range(taps):
                out += wzy * weight(d[0], kx) * flat[row + index(low[0] + first + kx, size[0])]
    return {"image": torch.where(ok, out, 0.0)}


def _exact_lts(case, seed):
    """The trimmed affine fit: the residuals' cut-off value, the subset's
    moments, least squares, until the parameters settle.  The translation is
    taken about the previous centre and the centre then moves to the subset's
    mean, as the reference does."""
    p, q = _lts_inputs(case, seed)
    n = case["points"]
    M = torch.eye(3, dtype=torch.float64, device=_DEV)
    off = torch.zeros(3, dtype=torch.float64, device=_DEV)
    rc = torch.zeros_like(off)
    last = torch.cat([M.reshape(-1), off])
    share, delta, it = 1.0, 1.0, 0
    while True:
        r = ((p @ M.T + off - q) ** 2).sum(1)
        cut = r.max() if share > 0.99999 else torch.sort(r).values[min(int(share * n), n - 1)]
        a, b = p[r <= cut], q[r <= cut]
        ma, mq = a.mean(0), b.mean(0)
        rot = ((b - mq).T @ (a - ma)) @ torch.linalg.inv((a - ma).T @ (a - ma))
        tr = (mq - rc) - rot @ (ma - rc)
        now = torch.cat([rot.reshape(-1), tr])
        before, delta = delta, float(((last - now) ** 2).sum())
        # the loop compares with the parameters of the identity throughout
        rc = ma
        M, off = rot, tr + ma - rot @ ma
        share, it = case["keep"], it + 1
        if not (delta > 1e-3 and it - 1 < 100 and abs(delta - before) > 1e-3):
            break
    return {"matrix": M, "offset": off, "center": torch.zeros_like(off),
            "params": torch.cat([M.reshape(-1), off]), "iterations": None}


def exact(case, seed):
    kind = case["kind"]
    if kind == "match":
        blocks = 1
        for a in ("nx", "ny", "nz"):
            blocks *= _grid(case[a], case["bw"], case["gap"])[0]
        if blocks * min(case["keep"], 1.0) * case["nw"] ** 3 * case["bw"] ** 3 > 2.5e10:
            return None  # about 20 seconds and more
        return _exact_match(case, seed)
    if kind == "resample":
        return _exact_resample(case, seed)
    if kind == "final":
        return _exact_final(case, seed)
    if kind == "lts" and case["affine"]:
        return _exact_lts(case, seed)
    # a registration is tens of dependent matcher calls: minutes in 64 bits; the
    # rigid fit ends in Euler angles of a quaternion whose sign is a convention
    return None
