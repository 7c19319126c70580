"""The work this library is used for, as cases that can be timed and compared.

A case is one call (or, for a request, the few calls) of a program that
registers an ultrasound with an MR/CT: an optimizer step of one transform, a
batch of candidate transforms, a 2D-to-3D frame stack, normalised mutual
information, and a whole registration request from host images to the
optimum. Images are the synthetic MR/ultrasound pairs of the benchmark
(ellipsoid phantom with noise; 0.7 MR + 0.5 |Sobel MR| + 0.05 under a seeded
affine with unit-mean Rayleigh speckle), made on the GPU from the seed.

    listed()             the cases
    draw(rng)            another case of the same ranges
    prepare(case, seed)  images uploaded, transforms in host memory
    run(state)           one pass through the public API
    work(case)           bytes and operations one pass cannot do without
    exact(case, seed)    the values in 64 bits, from the formulas
"""
import math
import random

import numpy as np
import torch

from lc2registration_gb300 import capi
from lc2registration_gb300.geometry import Geometry

DTYPES = {"f32": torch.float32, "f16": torch.float16, "bf16": torch.bfloat16}
ELEM = {"f32": 4, "f16": 2, "bf16": 2}


def _case(name, kind, mode, hr_moving, storage, r, m, f, count, ms=1.0, fs=1.0, vs=1.0, blocks=False,
          frames=0, layout=0, maxeval=0):
    """kind: 'evaluate' (count transforms in one call), 'stack', 'request'.
    m, f: moving and fixed image size; ms, fs, vs: their spacing and the
    virtual grid's in mm."""
    c = {"kind": kind, "mode": mode, "hr_moving": hr_moving, "storage": storage, "r": r,
         "mx": m[0], "my": m[1], "mz": m[2], "fx": f[0], "fy": f[1], "fz": f[2],
         "ms": ms, "fs": fs, "vs": vs, "count": count, "blocks": blocks, "frames": frames,
         "layout": layout, "maxeval": maxeval}
    if name:
        c["name"] = name
    return c


def listed():
    cube = lambda n: (n, n, n)
    return [
        # one BOBYQA step of a 2D registration: a single transform, all latency
        _case("step_2d_256_r3_f32", "evaluate", "2D", True, "f32", 3, (256, 256, 1), (256, 256, 1), 1),
        # a population of candidate 2D affines in one launch
        _case("batch_2d_256_r3_f32", "evaluate", "2D", True, "f32", 3, (256, 256, 1), (256, 256, 1),
              512),
        # one BOBYQA step of a 3D registration, MR 128^3 into ultrasound 96^3
        _case("step_3d_96_r3_f32", "evaluate", "3D", True, "f32", 3, cube(128), cube(96), 1),
        # DIRECT / population batches of the same registration
        _case("batch_3d_96_r3_f32", "evaluate", "3D", True, "f32", 3, cube(128), cube(96), 100),
        # one step of a full-size registration in 16-bit storage, 9^3 patches
        _case("step_3d_256_r4_f16", "evaluate", "3D", True, "f16", 4, cube(256), cube(256), 1,
              blocks=True),
        # the headline: candidate affines at 256^3 in a batch, 10 % constant blocks
        _case("batch_3d_256_r4_f16", "evaluate", "3D", True, "f16", 4, cube(256), cube(256), 128,
              blocks=True),
        # clinical sizes: ragged, anisotropic extents, resampled spacing, bf16
        _case("batch_3d_ragged_r2_bf16", "evaluate", "3D", True, "bf16", 2, (181, 217, 163),
              (165, 133, 149), 25, ms=1.0, fs=0.9, vs=1.1),
        # HighResolutionModality: Fixed, the reference's 3D setting: the ultrasound is resampled
        _case("fixed_3d_160_r3_f32", "evaluate", "3D", False, "f32", 3, cube(128), cube(160), 50),
        # the same in 2D, frame-grabber size
        _case("fixed_2d_400x300_r4_f32", "evaluate", "2D", False, "f32", 4, (400, 300, 1),
              (400, 300, 1), 100),
        # 2D-to-3D: 64 frames of uneven sizes, 16 poses each, in one launch
        _case("stack_64x16_r3_f32", "stack", "2DTo3D", True, "f32", 3, cube(256), (0, 0, 1), 16,
              fs=0.5, vs=0.5, frames=64, layout=1),
        # PatchSize 0: normalised mutual information
        _case("mi_3d_128_f32", "evaluate", "3D", True, "f32", 0, cube(128), cube(128), 50),
        # a whole request: create, upload host images, rigid BOBYQA, result
        _case("request_3d_96_r3_f32", "request", "3D", True, "f32", 3, cube(128), cube(96), 1,
              maxeval=80),
    ]


def _log_int(rng, lo, hi):
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    what = rng.choice(["batch3", "batch3", "step3", "batch2", "step2", "fixed3", "fixed2", "stack",
                       "mi", "request3", "request2"])
    storage = rng.choice(["f32", "f32", "f16", "bf16"])
    budget = 60 * 256 ** 3  # voxel evaluations of a batch: under half the largest listed case
    if what in ("batch3", "step3", "fixed3", "mi"):
        f = [_log_int(rng, 48, 256) for _ in range(3)]
        m = [max(40, min(256, int(v * rng.uniform(0.8, 1.35)))) for v in f]
        most = max(1, min(256, budget // (f[0] * f[1] * f[2])))
        count = 1 if what == "step3" else _log_int(rng, 2, max(2, most))
        r = 0 if what == "mi" else rng.choice([2, 3, 4])
        vs = rng.choice([1.0, 1.0, 0.9, 1.2])
        if vs < 1.0:
            f = [min(v, 230) for v in f]
        return _case(None, "evaluate", "3D", what != "fixed3", storage, r, m, f, count, vs=vs,
                     blocks=rng.random() < 0.3)
    if what in ("batch2", "step2", "fixed2"):
        f = [_log_int(rng, 64, 768) for _ in range(2)] + [1]
        m = [max(64, int(v * rng.uniform(0.8, 1.35))) for v in f[:2]] + [1]
        count = 1 if what == "step2" else _log_int(rng, 2, 512)
        return _case(None, "evaluate", "2D", what != "fixed2", storage, rng.choice([2, 3, 4, 5]), m,
                     f, count)
    if what == "stack":
        n = _log_int(rng, 96, 256)
        return _case(None, "stack", "2DTo3D", True, storage, rng.choice([2, 3, 4]), (n, n, n),
                     (0, 0, 1), _log_int(rng, 1, 32), fs=0.5, vs=0.5, frames=rng.randint(3, 48),
                     layout=rng.randint(2, 10 ** 6))
    if what == "request2":
        f = [_log_int(rng, 96, 512) for _ in range(2)] + [1]
        return _case(None, "request", "2D", rng.random() < 0.5, storage, rng.choice([3, 4]), f, f, 1,
                     maxeval=rng.randint(30, 120))
    f = [_log_int(rng, 48, 160) for _ in range(3)]
    m = [int(v * rng.uniform(1.0, 1.3)) for v in f]
    return _case(None, "request", "3D", rng.random() < 0.5, storage, rng.choice([2, 3, 4]), m, f, 1,
                 maxeval=rng.randint(30, 80))


# ---------------------------------------------------------------------------
# Inputs
# ---------------------------------------------------------------------------

def _sides(case):
    """Pixels per side of each frame: the benchmark's five sizes (layout 1),
    any size between 97 and 512 otherwise."""
    rng = random.Random(case["layout"])
    if case["layout"] == 1:
        return [rng.choice((128, 192, 256, 384, 512)) for _ in range(case["frames"])]
    return [rng.randint(97, 512) for _ in range(case["frames"])]


def _geoms(case):
    """(fixed, moving) geometries; both centred at the same point."""
    nd = 2 if case["mode"] == "2D" else 3
    md, fd = [case["mx"], case["my"], case["mz"]], [case["fx"], case["fy"], case["fz"]]
    ms, fs = [case["ms"]] * nd + [1.0] * (3 - nd), [case["fs"]] * nd + [1.0] * (3 - nd)
    org = [(md[a] * ms[a] - fd[a] * fs[a]) / 2 if a < nd else 0.0 for a in range(3)]
    return Geometry(tuple(fd), tuple(fs), tuple(org)), Geometry(tuple(md), tuple(ms), (0.0, 0.0, 0.0))


def _matrix(nd, rot, trans, scale, shear, center):
    """Row-major float32 virtual->moving mm matrix, x_m = L (x - C) + C + T."""
    d = math.pi / 180.0
    if nd == 2:
        c, s = math.cos(rot[0] * d), math.sin(rot[0] * d)
        L = np.array([[c, -s], [s, c]]) @ np.array([[1.0, shear[0]], [0.0, 1.0]]) @ np.diag(scale[:2])
    else:
        R = np.eye(3)
        for a, (i, j) in enumerate(((1, 2), (2, 0), (0, 1))):
            c, s = math.cos(rot[a] * d), math.sin(rot[a] * d)
            Q = np.eye(3)
            Q[i, i] = Q[j, j] = c
            Q[i, j], Q[j, i] = -s, s
            R = Q @ R
        L = R @ np.array([[1.0, shear[0], shear[1]], [0.0, 1.0, shear[2]], [0.0, 0.0, 1.0]]) \
            @ np.diag(scale)
    C = np.array(center[:nd])
    M = np.eye(nd + 1)
    M[:nd, :nd] = L
    M[:nd, nd] = C - L @ C + np.array(trans[:nd])
    return M.astype(np.float32)


def _random_matrix(rng, nd, center, extent, wide=1.0):
    """An affine of the benchmark's ranges: rotation to 8 degrees (5 in 2D),
    translation to a tenth of the extent, scale 0.95-1.05, shear 0.03."""
    a = 8.0 if nd == 3 else 5.0
    rot = [rng.uniform(-a, a) * wide for _ in range(3)]
    trans = [rng.uniform(-0.08, 0.08) * extent * wide for _ in range(3)]
    scale = [1.0 + rng.uniform(-0.05, 0.05) * wide for _ in range(3)]
    shear = [rng.uniform(-0.03, 0.03) * wide for _ in range(3)]
    return _matrix(nd, rot, trans, scale, shear, center)


def _phantom(dim, blobs, gen, rng):
    """Smooth-edged ellipsoids with intensities U[0, 1] on 0.1, plus noise."""
    ax = [torch.arange(n, device="cuda", dtype=torch.float32) for n in dim]
    img = torch.full((dim[2], dim[1], dim[0]), 0.1, device="cuda")
    small = min(n for n in dim if n > 1)
    for _ in range(blobs):
        q = torch.zeros((1, 1, 1), device="cuda")
        for a in range(3):
            if dim[a] == 1:
                continue
            c, rad = rng.uniform(0.2, 0.8) * dim[a], rng.uniform(0.08, 0.25) * small
            sh = [1, 1, 1]
            sh[2 - a] = dim[a]
            q = q + (((ax[a] - c) / rad) ** 2).reshape(sh)
        w = torch.sigmoid((1.0 - q) * (small * 0.04))
        img = img + (rng.uniform(0.0, 1.0) - img) * w
    noise = torch.randn(img.shape, device="cuda", generator=gen) * 0.01
    return img + noise


def _sobel(v, nd):
    """Sobel magnitude with zero padding (sum of |taps| 8 in 2D, 32 in 3D)."""
    def smooth(t, d):
        p = _pad1(t, d)
        n = t.shape[d]
        return p.narrow(d, 0, n) + 2 * t + p.narrow(d, 2, n)

    def diff(t, d):
        p = _pad1(t, d)
        n = t.shape[d]
        return p.narrow(d, 2, n) - p.narrow(d, 0, n)

    if nd == 2:
        gx, gy = smooth(diff(v, 2), 1), smooth(diff(v, 1), 2)
        return torch.sqrt(gx * gx + gy * gy)
    sz = smooth(v, 0)
    gx, gy = smooth(diff(sz, 2), 1), smooth(diff(sz, 1), 2)
    gz = smooth(smooth(diff(v, 0), 1), 2)
    return torch.sqrt(gx * gx + gy * gy + gz * gz)


def _pad1(t, d):
    z = torch.zeros_like(t.narrow(d, 0, 1))
    return torch.cat([z, t, z], d)


def _sample(img, ig, grid_dim, grid_sp, grid_org, mat, nd, dtype):
    """img (z, y, x) sampled linearly on a grid mapped by mat (grid mm -> image
    mm); 0 outside [0, dim - 1]."""
    M = np.asarray(mat, dtype=np.float64).reshape(nd + 1, nd + 1)
    idx = [torch.arange(n, device="cuda", dtype=dtype).reshape([-1 if 2 - a == k else 1 for k in range(3)])
           for a, n in enumerate(grid_dim)]
    ok, lo, fr = None, [], []
    for a in range(nd):
        p = float(M[a, nd] - ig.origin[a] + sum(M[a, b] * grid_org[b] for b in range(nd))) / ig.spacing[a]
        for b in range(nd):
            p = p + idx[b] * float(M[a, b] * grid_sp[b] / ig.spacing[a])
        p = p.expand(grid_dim[2], grid_dim[1], grid_dim[0])
        inside = (p >= 0) & (p <= ig.dim[a] - 1)
        ok = inside if ok is None else ok & inside
        f = p.floor().clamp(0, max(0, ig.dim[a] - 2))
        lo.append(f.long())
        fr.append((p - f).clamp(0, 1))
    flat = img.reshape(-1)
    dims = ig.dim
    out = 0
    for corner in range(1 << nd):
        w, o = 1.0, 0
        for a in range(nd):
            b = corner >> a & 1
            w = w * (fr[a] if b else 1 - fr[a])
            step = 1 if a == 0 else dims[0] if a == 1 else dims[0] * dims[1]
            o = o + (lo[a] + (b if dims[a] > 1 else 0)) * step
        out = out + w * flat[o].to(dtype)
    return torch.where(ok, out, torch.zeros_like(out))


def _speckle(shape, gen):
    u = torch.rand(shape, device="cuda", generator=gen)
    return torch.sqrt(-2.0 * torch.log(1.0 - u)) / math.sqrt(math.pi / 2)


def _constant_blocks(us, rng, frac=0.1, b=16):
    """A tenth of the ultrasound replaced by constant 16^3 blocks."""
    nb = [max(1, s // b) for s in us.shape]
    total = nb[0] * nb[1] * nb[2]
    for p in rng.sample(range(total), int(round(frac * total))):
        z, y, x = p // (nb[1] * nb[2]), p // nb[2] % nb[1], p % nb[2]
        us[z * b:(z + 1) * b, y * b:(y + 1) * b, x * b:(x + 1) * b] = 0.05 + 0.4 * rng.random()
    return us


def _inputs(case, seed):
    """Device images and host matrices of a case, from the seed alone."""
    rng = random.Random(seed * 7919 + 17)
    gen = torch.Generator(device="cuda")
    gen.manual_seed(seed)
    nd = 2 if case["mode"] == "2D" else 3
    pd = 3 if case["mode"] == "3D" else 2
    if case["kind"] == "stack":
        _, mg = _geoms(dict(case, fx=1, fy=1))
        mr = _phantom(mg.dim, 12, gen, rng)
        base = 0.7 * mr + 0.5 * _sobel(mr, 3) + 0.05
        c = mg.center()
        frames = []
        for s in _sides(case):
            sp = case["fs"]
            fg = Geometry((s, s, 1), (sp, sp, sp), (c[0] - s * sp / 2, c[1] - s * sp / 2, c[2]))
            ext = 0.3 * min(mg.dim)
            truth = _random_matrix(rng, 3, fg.center(), ext)
            us = _sample(base, mg, fg.dim, fg.spacing, fg.origin, truth, 3, torch.float32)
            us = us * _speckle(us.shape, gen)
            mats = [_random_matrix(rng, 3, fg.center(), ext) for _ in range(case["count"])]
            frames.append((fg, us, np.stack(mats)))
        return mg, mr, frames
    fg, mg = _geoms(case)
    hg, ug = (mg, fg) if case["hr_moving"] else (fg, mg)
    mr = _phantom(hg.dim, 12 if nd == 3 else 6, gen, rng)
    base = 0.7 * mr + 0.5 * _sobel(mr, pd) + 0.05
    ext = min(case["fx"] * case["fs"], case["fy"] * case["fs"])
    center = fg.center()
    truth = _random_matrix(rng, nd, center, ext, 0.5)
    to_mr = truth if case["hr_moving"] else np.linalg.inv(truth.astype(np.float64))
    us = _sample(base, hg, ug.dim, ug.spacing, ug.origin, to_mr, nd, torch.float32)
    us = us * _speckle(us.shape, gen)
    if case["blocks"]:
        us = _constant_blocks(us, rng)
    mats = np.stack([_random_matrix(rng, nd, center, ext) for _ in range(case["count"])])
    fixed, moving = (us, mr) if case["hr_moving"] else (mr, us)
    return fg, fixed.contiguous(), mg, moving.contiguous(), mats


def prepare(case, seed):
    if case["kind"] == "stack":
        mg, mr, frames = _inputs(case, seed)
        st = capi.Stack(mg, case["r"], case["storage"])
        st.set_moving(mr.cpu().numpy())
        ids, mats = [], []
        for fg, us, m in frames:
            fid = st.add_frame(fg, [case["vs"]] * 3, us.cpu().numpy())
            ids += [fid] * len(m)
            mats.append(m)
        return {"stack": st, "ids": ids, "mats": np.concatenate(mats)}
    fg, fixed, mg, moving, mats = _inputs(case, seed)
    if case["kind"] == "request":
        nr = 3 if case["mode"] == "2D" else 6
        init = np.concatenate([np.zeros(nr), np.ones(2 if nr == 3 else 3), np.zeros(1 if nr == 3 else 3)])
        lo, hi = init.copy(), init.copy()
        lo[:nr], hi[:nr] = -12.0, 12.0
        return {"case": case, "fg": fg, "mg": mg, "fixed": fixed.cpu().numpy(),
                "moving": moving.cpu().numpy(), "init": init, "lo": lo, "hi": hi}
    ctx = capi.Context(case["mode"], fg, mg, [case["vs"]] * 3, case["r"], case["hr_moving"],
                       case["storage"])
    torch.cuda.synchronize()
    ctx.set_images_device(fixed.data_ptr(), moving.data_ptr())
    return {"ctx": ctx, "mats": mats, "count": case["count"]}


def run(state):
    if "stack" in state:
        return state["stack"].evaluate(state["ids"], state["mats"])
    if "ctx" in state:
        if state["count"] == 1:
            return state["ctx"].evaluate(state["mats"])
        return state["ctx"].evaluate_batch(state["mats"])
    case = state["case"]
    with capi.Context(case["mode"], state["fg"], state["mg"], [case["vs"]] * 3, case["r"],
                      case["hr_moving"], case["storage"]) as ctx:
        ctx.set_images(state["fixed"], state["moving"])
        out = capi.register(ctx, state["init"], state["lo"], state["hi"], state["fg"].center(),
                            rounds=[(["translation", "rotation"], 1e-6)],
                            round_maxeval=case["maxeval"])
    return {"params": out["params"], "lc2": out["lc2"], "evaluations": out["evaluations"]}


# ---------------------------------------------------------------------------
# What a pass cannot do without
# ---------------------------------------------------------------------------

def _virtual_dim(case):
    if case["mode"] == "2D":
        return [int(math.ceil(case[k] * case["fs"] / case["vs"])) for k in ("fx", "fy")] + [1]
    return [int(math.ceil(round(case[k] * case["fs"] / case["vs"], 4))) for k in ("fx", "fy", "fz")]


def work(case):
    """Bytes: the moving image once per pass, the static image and its
    weighting factors once, matrices and values. Operations per voxel and
    transform: the linear sample, the Sobel magnitude, the patch sums' five
    products and running windows, and the 2x2 solve (mutual information: the
    sample, the bin and one count)."""
    nd = 2 if case["mode"] == "2D" else 3
    e = ELEM[case["storage"]]
    nm = case["mx"] * case["my"] * case["mz"]
    if case["kind"] == "stack":
        px = sum(s * s for s in _sides(case))
        evals, voxels = case["frames"] * case["count"], px * case["count"]
        static = px
    else:
        d = _virtual_dim(case)
        static = d[0] * d[1] * d[2]
        evals = case["maxeval"] if case["kind"] == "request" else case["count"]
        voxels = static * evals
    if case["r"] == 0:
        return {"bytes": float(nm * e + static + evals * 72), "flops": float(voxels * 26)}
    fields = 7 if case["hr_moving"] else 5
    per = (7 * 3 if nd == 3 else 3 * 3) + (10 if case["mode"] != "3D" else 26) * case["hr_moving"] \
        + 5 + fields * 2 * (3 if case["mode"] == "3D" else 2) + 30
    return {"bytes": float(nm * e + static * (e + 4) + evals * 72), "flops": float(voxels * per)}


# ---------------------------------------------------------------------------
# The values in 64 bits
# ---------------------------------------------------------------------------

def _stored(t, storage):
    """The image as the library holds it: rounded to the storage type."""
    return t.to(DTYPES[storage]).double()


def _box(t, r, dims):
    """Sums over (2r+1)-wide windows along dims, full windows only."""
    w = 2 * r + 1
    for d in dims:
        acc, have, size, at = None, t, 1, 0
        n = t.shape[d] - w + 1
        while True:
            if w & size:
                part = have.narrow(d, at, n)
                acc = part if acc is None else acc + part
                at += size
            size *= 2
            if size > w:
                break
            half = size // 2
            have = have.narrow(d, 0, have.shape[d] - half) + have.narrow(d, half, have.shape[d] - half)
        t = acc
    return t


def _lc2(U, M, G, r, pd):
    """Variance-weighted LC2 of one evaluation: per full patch with every
    ultrasound value above 1e-6 and sample variance above 1e-6, sigma times
    the explained share of the least-squares fit U ~ a M + b G + c."""
    dims = (2, 1, 0) if pd == 3 else (2, 1)
    w = 2 * r + 1
    if any(U.shape[d] < w for d in dims):
        return 0.0
    n = float(w ** pd)
    good = _box((U > 1e-6).double(), r, dims) > n - 0.5
    u, m, g = U - U.mean(), M - M.mean(), G - G.mean()
    su, sm, sg = (_box(t, r, dims) for t in (u, m, g))

    def centred(a, b, sa, sb):
        return _box(a * b, r, dims) - sa * sb / n

    duu, dmm, dgg = centred(u, u, su, su), centred(m, m, sm, sm), centred(g, g, sg, sg)
    dum, dug, dmg = centred(u, m, su, sm), centred(u, g, su, sg), centred(m, g, sm, sg)
    var = duu / (n - 1)
    good = good & (var > 1e-6)
    sigma = torch.where(good, var.clamp_min(0).sqrt(), torch.zeros_like(var))
    km, kg = dmm / (n - 1) > 1e-12, dgg / (n - 1) > 1e-12
    one = torch.ones_like(dmm)
    em, eg = dum * dum / torch.where(km, dmm, one), dug * dug / torch.where(kg, dgg, one)
    det = dmm * dgg - dmg * dmg
    full = km & kg & (det > 1e-10 * dmm * dgg)
    e2 = (dgg * dum * dum - 2 * dmg * dum * dug + dmm * dug * dug) / torch.where(full, det, one)
    e = torch.where(full, e2, torch.where(km, em, torch.where(kg, eg, torch.zeros_like(em))))
    meas = sigma * e / torch.where(good, duu, one)
    meas = torch.where(good & (meas > 0) & torch.isfinite(meas), meas, torch.zeros_like(meas))
    v = meas.sum() / sigma.sum()
    return float(v) if bool(torch.isfinite(v)) else 0.0


def _entropy(counts, n):
    c = counts[counts > 0].double()
    return math.log(n) - float((c * c.log()).sum()) / n


def _bins(t):
    lo, hi = t.min(), t.max()
    s = 255.0 / (hi - lo) if bool(hi > lo) else 0.0
    return ((t - lo) * s + 0.5).floor().long()


def _nmi(static_bins, warped):
    n = static_bins.numel()
    b = _bins(warped)
    joint = torch.bincount((static_bins + 256 * b).reshape(-1), minlength=65536)
    hs, hw = (_entropy(torch.bincount(t.reshape(-1), minlength=256), n) for t in (static_bins, b))
    return (hs + hw) / _entropy(joint, n)


def exact(case, seed):
    if case["kind"] == "request":
        return None  # an optimizer's path, not a value
    with torch.no_grad():
        if case["kind"] == "stack":
            mg, mr, frames = _inputs(case, seed)
            mov = _stored(mr, case["storage"])
            out = []
            for fg, us, mats in frames:
                U = _stored(us, case["storage"])
                for m in mats:
                    M = _sample(mov, mg, fg.dim, fg.spacing, fg.origin, m, 3, torch.float64)
                    out.append(_lc2(U, M, _sobel(M, 2), case["r"], 2))
            return np.array(out)
        fg, fixed, mg, moving, mats = _inputs(case, seed)
        nd = 2 if case["mode"] == "2D" else 3
        pd = 3 if case["mode"] == "3D" else 2
        vs32 = float(np.float32(case["vs"]))
        vs = [vs32] * nd + [1.0] * (3 - nd)
        vd = [int(math.ceil(float(np.float32(fg.dim[a]) * np.float32(fg.spacing[a]) / np.float32(vs32))))
              if a < nd else 1 for a in range(3)]
        static = _sample(fixed.double(), fg, vd, vs, fg.origin, np.eye(nd + 1), nd, torch.float64)
        if case["hr_moving"]:
            static = _stored(static, case["storage"])
        mov = _stored(moving, case["storage"])
        Gs = _sobel(static, pd) if not case["hr_moving"] else None
        sb = _bins(static) if case["r"] == 0 else None
        out = []
        for m in mats:
            W = _sample(mov, mg, vd, vs, fg.origin, m, nd, torch.float64)
            if case["r"] == 0:
                out.append(_nmi(sb, W))
            elif case["hr_moving"]:
                out.append(_lc2(static, W, _sobel(W, pd), case["r"], pd))
            else:
                out.append(_lc2(W, static, Gs, case["r"], pd))
        return out[0] if case["count"] == 1 else np.array(out)
