"""The work that users of the bake path have it do, as cases to measure.

Every case goes through the package's public Python API (fornos_b200.api), on
seeded synthetic meshes and maps.  `op` names the kind of call:

  maps     the cheap maps of one low- / high-poly pair: UV rasterisation, mesh
           mapping, height, position and tangent-space normal maps
  sample   one hemisphere pass (AO, bent normals, thickness, or AO + bent
           normals from one traversal) over a mapped texture
  import   what happens once per asset: normals, tangents and welded directions
           computed on the device, texel map, BVH and scene built on the device,
           then the normal map
  bake     the one-shot bake from host arrays to host arrays, all six bakers
  batch    a queue of small AO jobs, replayed as a CUDA graph
  export   the image of a finished map, with dilation for 8-bit images
  denoise  the feature image and the denoiser network over a 16-sample bake
  train    a few optimiser steps of the denoiser's training loop, its loss and
           the updated weights

Sizes are those of the repository's bench and tests and the range around them.
"""
import math

import numpy as np
import torch

from fornos_b200 import api
from fornos_b200 import workloads as W
from fornos_b200.denoise_train import DEFAULT_OUT as TRAINED_WEIGHTS
from fornos_b200.denoise_train import init_params

PERMS = api.PERMS
KINDS = {"ao": api.AO, "bn": api.BN, "thickness": api.THICK, "ao_bn": api.AO_BN}
MODES = {"float_rgb8": api.EXPORT_FLOAT_RGB8, "float_f32": api.EXPORT_FLOAT_F32,
         "normal_rgb8": api.EXPORT_NORMAL_RGB8, "vector_f32": api.EXPORT_VECTOR_F32}


def listed():
    return [
        # a preview of the cheap maps while the artist moves sliders: latency and launches count
        dict(name="maps_preview", op="maps", shape="sphere", hi=96, tex=128, mapping="smooth"),
        # the same maps of a finished asset: a heightfield of 2.1M triangles at 2048 x 2048
        dict(name="maps_full", op="maps", shape="plane", hi=1024, tex=2048, mapping="smooth"),
        # interactive AO of a small prop at a few samples
        dict(name="ao_preview", op="sample", kind="ao", shape="sphere", hi=64, tex=96, spp=16, max_d=0.5),
        # AO of a prop at 512 x 512 with 64 samples
        dict(name="ao_512", op="sample", kind="ao", shape="sphere", hi=512, tex=512, spp=64, max_d=0.5),
        # AO and bent normals of the heightfield, 256 samples: the bulk of a production bake
        dict(name="ao_bn_1024", op="sample", kind="ao_bn", shape="plane", hi=1024, tex=1024, spp=256, max_d=0.3),
        # thickness at a size and sample count that are multiples of nothing
        dict(name="thickness_777", op="sample", kind="thickness", shape="sphere", hi=1001, tex=777, spp=100, max_d=0.5),
        # opening an asset of 2.1M triangles up to its normal map
        dict(name="import_2m", op="import", shape="plane", hi=1024, tex=1024),
        # a whole bake from a host program's arrays, as an application embeds it
        dict(name="bake_512", op="bake", shape="plane", hi=512, tex=512, spp=128, max_d=0.3),
        # a queue of sixteen props of different sizes and sample counts
        dict(name="batch_16", op="batch", jobs=16, tex=128, spp=64),
        # the 8-bit AO image of a 2048 x 2048 atlas, dilated by the reference's default of 16
        dict(name="export_2048", op="export", tex=2048, mode="float_rgb8", dilate=16),
        # denoising a 1024 x 1024 AO + bent-normal map
        dict(name="denoise_1024", op="denoise", tex=1024),
        # training at the batch size that the repository's weights were trained with
        dict(name="train_16k", op="train", batch=16384, steps=4, dataset=131072),
    ]


def draw(rng):
    def log_int(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    op = rng.choice(["maps", "sample", "sample", "sample", "import", "bake", "batch", "export", "denoise", "train"])
    shape = rng.choice(["sphere", "plane"])
    max_d = round(rng.uniform(0.2, 0.5), 3)
    if op == "maps":
        return dict(op=op, shape=shape, hi=log_int(32, 1000), tex=log_int(64, 2000),
                    mapping=rng.choice(["smooth", "lowpoly", "hybrid"]))
    if op == "sample":
        tex = log_int(64, 1000)
        spp = min(log_int(8, 512), max(8, (1 << 28) // (tex * tex)))
        return dict(op=op, kind=rng.choice(sorted(KINDS)), shape=shape, hi=log_int(32, 1000), tex=tex, spp=spp,
                    max_d=max_d)
    if op == "import":
        return dict(op=op, shape=shape, hi=log_int(48, 1000), tex=log_int(64, 1000))
    if op == "bake":
        return dict(op=op, shape=shape, hi=log_int(32, 500), tex=log_int(64, 500), spp=log_int(16, 128), max_d=max_d)
    if op == "batch":
        return dict(op=op, jobs=rng.randint(2, 24), tex=log_int(48, 192), spp=rng.choice([16, 32, 50, 64, 128]))
    if op == "export":
        mode = rng.choice(sorted(MODES))
        return dict(op=op, tex=log_int(100, 2000), mode=mode,
                    dilate=rng.randint(0, 24) if mode.endswith("rgb8") else 0)
    if op == "denoise":
        return dict(op=op, tex=log_int(64, 1020))
    return dict(op=op, batch=128 * log_int(2, 128), steps=rng.randint(1, 6), dataset=log_int(20000, 130000))


# ------------------------------------------------------------------ device buffers as tensors
_CONTEXT = []


def context():
    """One context per process, as a program keeps it."""
    if not _CONTEXT:
        _CONTEXT.append(api.Context(0))
    return _CONTEXT[0]


class _Memory:
    def __init__(self, buf, shape, typestr):
        self.buf = buf  # a tensor made from this keeps the buffer alive
        self.__cuda_array_interface__ = dict(shape=tuple(shape), typestr=typestr, data=(buf.device_ptr, False),
                                             version=3)


def tensor(buf, shape, typestr="<f4"):
    """The buffer's memory as a tensor (no copy; the buffer owns it)."""
    return torch.as_tensor(_Memory(buf, shape, typestr), device="cuda")


# ------------------------------------------------------------------ meshes
def heights(quads, seed):
    """Heightfield over [0, 1]^2 as W.plane_pair shapes it: four octaves of
    value noise and 200 hemispherical bumps, computed on the GPU."""
    rng = np.random.default_rng(seed)
    n = quads + 1
    c = torch.arange(n, dtype=torch.float64, device="cuda") / quads
    y, x = torch.meshgrid(c, c, indexing="ij")
    z = torch.zeros_like(x)
    amp, freq = 0.05, 4
    for _ in range(4):
        lat = torch.from_numpy(rng.uniform(-1.0, 1.0, size=(freq + 2, freq + 2))).cuda()
        fx, fy = x * freq, y * freq
        ix, iy = fx.floor().clamp(max=freq).long(), fy.floor().clamp(max=freq).long()
        tx, ty = fx - ix, fy - iy
        sx, sy = tx * tx * (3 - 2 * tx), ty * ty * (3 - 2 * ty)
        z += amp * ((lat[iy, ix] * (1 - sx) + lat[iy, ix + 1] * sx) * (1 - sy) +
                    (lat[iy + 1, ix] * (1 - sx) + lat[iy + 1, ix + 1] * sx) * sy)
        amp, freq = amp * 0.5, freq * 2
    cx, cy = rng.uniform(0, 1, 200), rng.uniform(0, 1, 200)
    rad = rng.uniform(0.01, 0.05, 200)
    for k in range(200):
        i0, i1 = max(0, int((cx[k] - rad[k]) * quads)), min(n, int((cx[k] + rad[k]) * quads) + 2)
        j0, j1 = max(0, int((cy[k] - rad[k]) * quads)), min(n, int((cy[k] + rad[k]) * quads) + 2)
        d2 = (c[i0:i1][None, :] - cx[k]) ** 2 + (c[j0:j1][:, None] - cy[k]) ** 2
        z[j0:j1, i0:i1] += (rad[k] ** 2 - d2).clamp(min=0).sqrt()
    return z.cpu().numpy()


def meshes(shape, hi, seed):
    """(low-poly, high-poly) arrays: `hi` is the high-poly's quads per side of
    the plane, or its segments round the sphere."""
    if shape == "plane":
        return W.grid_plane(64), W.grid_plane(hi, heights=heights(hi, seed))
    return W.sphere_pair(seed=seed, hi_seg=(hi, max(8, hi // 2)))


class Pair:
    """A low- / high-poly pair as a program holds it before the bake."""

    def __init__(self, shape, hi, seed, mapping="smooth"):
        ctx = context()
        lo, high = meshes(shape, hi, seed)
        self.triangles = high.triangle_count
        self.high = api.Mesh(high)
        self.high.compute_normals_device(ctx, api.NORMALS_VERTEX)
        self.low = api.Mesh(lo)
        self.low.compute_tangent_space()
        self.dirs = self.low.copy()
        self.dirs.compute_vertex_normals_aggressive()
        self.scene = api.Scene.build(ctx, self.high)
        self.mapping = mapping

    def texel_map(self, tex):
        if self.mapping == "lowpoly":
            return api.TexelMap.from_mesh(context(), self.low, tex, tex)
        if self.mapping == "hybrid":
            return api.TexelMap.from_meshes_hybrid(context(), self.low, self.dirs, tex, tex, 0.05)
        return api.TexelMap.from_meshes(context(), self.low, self.dirs, tex, tex)


def mapped(pair, tex, max_dist=api.FLT_MAX):
    ctx = context()
    tmap = pair.texel_map(tex)
    coords, tidx = ctx.buffer(16 * max(tmap.count, 1)), ctx.buffer(4 * max(tmap.count, 1))
    api.meshmap(ctx, pair.scene, tmap, True, coords, tidx, max_dist=max_dist)
    return tmap, coords, tidx


def sample_table(spp, seed):
    return context().upload(api.samples_cosine(spp, PERMS, seed & 0x7FFFFFFF))


# ------------------------------------------------------------------ synthetic maps
def covered(tex):
    """Row-major indices of an atlas' covered pixels: charts of different
    sizes with gaps between them, about three quarters of the image."""
    g = torch.Generator(device="cuda").manual_seed(1)
    cells = 4
    y, x = torch.meshgrid(torch.arange(tex, device="cuda"), torch.arange(tex, device="cuda"), indexing="ij")
    cy, cx = (y * cells // tex), (x * cells // tex)
    fy, fx = (y * cells % tex) / tex - 0.5, (x * cells % tex) / tex - 0.5
    size = 0.38 + 0.11 * torch.rand(cells, cells, generator=g, device="cuda")
    round_ = torch.rand(cells, cells, generator=g, device="cuda") < 0.3
    s, r = size[cy, cx], round_[cy, cx]
    inside = torch.where(r, (fx * fx + fy * fy).sqrt() < s, torch.maximum(fx.abs(), fy.abs()) < s)
    return inside.reshape(-1).nonzero().reshape(-1)


def smooth_noise(tex, seed, octaves=5):
    """A smooth field in about [-1, 1] over tex x tex pixels."""
    g = torch.Generator(device="cuda").manual_seed(seed)
    out = torch.zeros(tex, tex, device="cuda", dtype=torch.float64)
    for k in range(octaves):
        lat = torch.rand(1, 1, (2 << k) + 2, (2 << k) + 2, generator=g, device="cuda", dtype=torch.float64) * 2 - 1
        out += torch.nn.functional.interpolate(lat, (tex, tex), mode="bicubic", align_corners=True)[0, 0] * 0.5 ** k
    return out / 2


def low_sample_bake(tex, seed):
    """A 16-sample AO + bent-normal bake of a heightfield over the unit square,
    one texel per pixel of a covered atlas: float32 / int32 tensors."""
    g = torch.Generator(device="cuda").manual_seed(seed + 1)
    idx = covered(tex)
    n = idx.numel()
    z = 0.08 * smooth_noise(tex, seed + 2)
    dzx, dzy = torch.zeros_like(z), torch.zeros_like(z)
    dzx[:, 1:] = (z[:, 1:] - z[:, :-1]) * tex
    dzy[1:, :] = (z[1:, :] - z[:-1, :]) * tex
    nrm = torch.stack([-dzx, -dzy, torch.ones_like(z)], -1).reshape(-1, 3)[idx]
    nrm = nrm / nrm.norm(dim=1, keepdim=True)
    xy = torch.stack([(idx % tex + 0.5) / tex, (torch.div(idx, tex, rounding_mode="floor") + 0.5) / tex], -1)
    pos = torch.cat([xy, z.reshape(-1)[idx][:, None]], 1)
    ao = (0.75 + 0.3 * smooth_noise(tex, seed + 3).reshape(-1)[idx]).clamp(0, 1)
    ao = torch.floor(ao * 16 + torch.rand(n, generator=g, device="cuda", dtype=torch.float64)).clamp(0, 16) / 16
    bn = nrm + 0.25 * torch.randn(n, 3, generator=g, device="cuda", dtype=torch.float64)
    bn = bn / bn.norm(dim=1, keepdim=True)
    miss = torch.rand(n, generator=g, device="cuda") < 0.01
    tidx = torch.where(miss, torch.full((n,), -1, device="cuda"), 3 * torch.arange(n, device="cuda")).int()
    dist = 0.02 + 0.01 * torch.rand(n, generator=g, device="cuda", dtype=torch.float64)
    coords = torch.stack([dist, torch.full_like(dist, 0.25), torch.full_like(dist, 0.25), torch.full_like(dist, 0.5)], 1)
    f = lambda t: t.float().contiguous()  # noqa: E731
    return dict(idx=idx.int(), tidx=tidx, coords=f(coords), ao=f(ao), bn=f(bn), pos=f(pos), nrm=f(nrm))


def octahedral(v):
    s = v.abs().sum(1)
    p = v[:, :2] / s[:, None]
    sign = torch.where(p >= 0, 1.0, -1.0).to(v.dtype)
    return torch.where(v[:, 2:3] < 0, (1 - p.abs().flip(1)) * sign, p)


def feature_image(b, tex, max_d):
    """The network's feature image in 64 bits: 3 planes of tex x tex x 4."""
    f = torch.zeros(3, tex * tex, 4, dtype=torch.float64, device="cuda")
    hit = b["tidx"] != -1
    p = b["idx"].long()[hit]
    d = lambda k: b[k].double()[hit]  # noqa: E731
    f[0, p] = torch.cat([d("ao")[:, None], octahedral(d("bn")), torch.ones(p.numel(), 1, device="cuda")], 1)
    f[1, p] = torch.cat([d("pos") / max_d, d("coords")[:, :1] / max_d], 1)
    f[2, p, :2] = octahedral(d("nrm"))
    x, y = p % tex, torch.div(p, tex, rounding_mode="floor")
    total, k = torch.zeros(p.numel(), dtype=torch.float64, device="cuda"), torch.zeros(p.numel(), device="cuda")
    for dx, dy in ((1, 0), (-1, 0), (0, 1), (0, -1)):
        ok = (x + dx >= 0) & (y + dy >= 0) & (x + dx < tex) & (y + dy < tex)
        q = torch.where(ok, p + dx + dy * tex, 0)
        ok &= f[0, q, 3] > 0
        total += torch.where(ok, (f[1, q, :3] - f[1, p, :3]).norm(dim=1), 0.0)
        k += ok
    f[2, p, 2] = torch.where(k > 0, total / k.clamp(min=1), 0.0)
    return f


def input_rows(f, tex, pixels):
    """The network's 250 inputs for the given pixels, padded to 256 columns."""
    x, y = pixels % tex, torch.div(pixels, tex, rounding_mode="floor")
    c, sp = f[1, pixels, :3], f[2, pixels, 2]
    out = torch.zeros(pixels.numel(), 256, dtype=f.dtype, device=f.device)
    for j in range(25):
        dx, dy = j % 5 - 2, j // 5 - 2
        ok = (x + dx >= 0) & (y + dy >= 0) & (x + dx < tex) & (y + dy < tex)
        q = torch.where(ok, pixels + dx + dy * tex, 0)
        ok &= f[0, q, 3] > 0
        rel = torch.where((sp > 0)[:, None], ((f[1, q, :3] - c) / sp.clamp(min=1e-30)[:, None]).clamp(-4, 4), 0.0)
        v = torch.cat([f[0, q, :3], rel, f[2, q, :2], f[1, q, 3:4], torch.ones_like(sp)[:, None]], 1)
        out[:, 10 * j:10 * j + 10] = torch.where(ok[:, None], v, 0.0)
    return out


def network(params, x):
    """The denoiser's network in the precision of `x`."""
    q = {k: params[o:o + int(np.prod(s))].reshape(s) for k, (o, s) in api.DN_LAYOUT.items()}
    h = torch.nn.functional.gelu(x @ q["w1"].T + q["b1"], approximate="tanh")
    h = torch.nn.functional.gelu(h @ q["w2"].T + q["b2"], approximate="tanh")
    return h @ q["w3"].T + q["b3"]


def training_set(case, seed):
    """(bf16 input rows, float32 targets, row order) of a training run."""
    tex = 384
    n = case["dataset"]
    b = low_sample_bake(tex, seed)
    f = feature_image(b, tex, 0.3)
    g = torch.Generator(device="cuda").manual_seed(seed + 9)
    pixels = b["idx"].long()[torch.randint(0, b["idx"].numel(), (n,), generator=g, device="cuda")]
    rows = torch.cat([input_rows(f, tex, p) for p in pixels.split(32768)]).to(torch.bfloat16)
    targets = torch.randn(n, 4, generator=g, device="cuda") * 0.08 + rows[:, :1].float() * 0.02
    order = torch.cat([torch.randperm(n, generator=g, device="cuda") for _ in range(1 + case["batch"] * case["steps"] // n)])
    return rows, targets, order[:case["batch"] * case["steps"]].int()


# ------------------------------------------------------------------ prepare
def prepare(case, seed):
    return _PREPARE[case["op"]](case, seed)


def _prepare_maps(case, seed):
    ctx = context()
    pair = Pair(case["shape"], case["hi"], seed, case["mapping"])
    n = pair.texel_map(case["tex"]).count
    bufs = {"coords": ctx.buffer(16 * n), "tidx": ctx.buffer(4 * n), "height": ctx.buffer(4 * n),
            "position": ctx.buffer(12 * n), "normals": ctx.buffer(12 * n)}
    out = [tensor(bufs["coords"], (n, 4)), tensor(bufs["tidx"], (n,), "<i4"), tensor(bufs["height"], (n,)),
           tensor(bufs["position"], (n, 3)), tensor(bufs["normals"], (n, 3))]
    return dict(op="maps", pair=pair, tex=case["tex"], bufs=bufs, out=out)


def _prepare_sample(case, seed):
    ctx = context()
    pair = Pair(case["shape"], case["hi"], seed)
    tmap, coords, tidx = mapped(pair, case["tex"])
    n, both = tmap.count, case["kind"] == "ao_bn"
    w0 = 3 if case["kind"] == "bn" else 1
    bufs = [ctx.buffer(4 * w0 * n), ctx.buffer(12 * n) if both else None, ctx.buffer(4 * n),
            ctx.buffer(4 * n) if both else None]
    out = [tensor(bufs[0], (n, 3) if w0 == 3 else (n,)), tensor(bufs[2], (n,), "<i4")]
    if both:
        out += [tensor(bufs[1], (n, 3)), tensor(bufs[3], (n,), "<i4")]
    return dict(op="sample", pair=pair, tmap=tmap, coords=coords, tidx=tidx, table=sample_table(case["spp"], seed),
                kind=KINDS[case["kind"]], spp=case["spp"], max_d=case["max_d"], bufs=bufs, out=out)


def _prepare_import(case, seed):
    lo, high = meshes(case["shape"], case["hi"], seed)
    low = api.Mesh(lo)
    low.compute_tangent_space()
    dirs = low.copy()
    dirs.compute_vertex_normals_aggressive()
    ctx = context()
    n = api.TexelMap.from_meshes(ctx, low, dirs, case["tex"], case["tex"]).count
    bufs = {"coords": ctx.buffer(16 * n), "tidx": ctx.buffer(4 * n), "normals": ctx.buffer(12 * n)}
    out = [tensor(bufs["coords"], (n, 4)), tensor(bufs["tidx"], (n,), "<i4"), tensor(bufs["normals"], (n, 3))]
    return dict(op="import", low=api.Mesh(lo), high=api.Mesh(high), tex=case["tex"], bufs=bufs, out=out)


def _prepare_bake(case, seed):
    ctx = context()
    pair = Pair(case["shape"], case["hi"], seed)
    tmap = pair.texel_map(case["tex"])
    t = tmap.download()
    n = tmap.count
    nodes, pos4, nrm4 = api.BVH.build_flat_device(ctx, pair.high)
    pix8, pixt12 = np.zeros((n, 8), np.float32), np.zeros((n, 12), np.float32)
    pix8[:, 0:3], pix8[:, 4:7] = t["positions"], t["directions"]
    pixt12[:, 0:3], pixt12[:, 4:7], pixt12[:, 8:11] = t["normals"], t["tangents"], t["bitangents"]

    def pinned(a):
        p = torch.empty(a.nbytes, dtype=torch.uint8, pin_memory=True).numpy().view(a.dtype).reshape(a.shape)
        p[...] = a
        return p

    f = lambda *s: pinned(np.zeros(s, np.float32))  # noqa: E731
    out = dict(coords4=f(n, 4), tidx=pinned(np.zeros(n, np.uint32)), height=f(n), position3=f(n, 3),
               normals3=f(n, 3), ao=f(n), bent_normals3=f(n, 3), thickness=f(n))
    sampler = dict(sample_count=case["spp"], min_distance=0.001, max_distance=case["max_d"], seed=seed & 0x7FFFFFFF)
    return dict(op="bake", nodes=pinned(nodes), pos4=pinned(pos4), nrm4=pinned(nrm4), tex=case["tex"],
                pix8=pinned(pix8), pixt12=pinned(pixt12), idx=pinned(t["indices"]), sampler=sampler, outputs=out,
                out=[out[k].view(np.int32) if k == "tidx" else out[k] for k in sorted(out)])


def _batch_jobs(case):
    """Sizes of the queue's props: (shape, high-poly size, texture, samples)."""
    scale = (0.5, 1.0, 0.75, 1.5, 0.6, 1.25)
    return [("sphere" if i % 3 else "plane", 32 + 24 * (i * 7 % 8), max(16, int(case["tex"] * scale[i % 6])),
             case["spp"] if i % 2 else max(8, case["spp"] // 2)) for i in range(case["jobs"])]


def _prepare_batch(case, seed):
    ctx = context()
    jobs, keep, out, tables = [], [], [], {}
    for i, (shape, hi, tex, spp) in enumerate(_batch_jobs(case)):
        pair = Pair(shape, hi, seed + 17 * i)
        tmap, coords, tidx = mapped(pair, tex)
        if spp not in tables:
            tables[spp] = sample_table(spp, seed)
        jobs.append(dict(scene=pair.scene, coords=coords, tidx=tidx, texel_count=tmap.count, spp=spp,
                         min_distance=0.001, max_distance=0.4, samples=tables[spp], out0=ctx.buffer(4 * tmap.count),
                         hits0=ctx.buffer(4 * tmap.count)))
        out += [tensor(jobs[-1]["out0"], (tmap.count,)), tensor(jobs[-1]["hits0"], (tmap.count,), "<i4")]
        keep.append((pair, tmap))
    batch = api.Batch(ctx, jobs, api.AO)
    batch.run()
    batch.capture()
    return dict(op="batch", batch=batch, jobs=jobs, keep=keep, out=out)


def _export_values(case, seed):
    idx = covered(case["tex"])
    v = 0.6 + 0.5 * smooth_noise(case["tex"], seed + 3).reshape(-1)[idx]
    if not case["mode"].startswith("float"):
        x, y = (smooth_noise(case["tex"], seed + k).reshape(-1)[idx] for k in (4, 5))
        v = torch.stack([x, y, 1 + 0 * x], 1)
        v = v / v.norm(dim=1, keepdim=True)
    return idx, v.float()


def _texel_map(tex, idx):
    n = idx.numel()
    return api.TexelMap.from_host(context(), tex, tex, np.zeros((n, 8), np.float32), np.zeros((n, 12), np.float32),
                                  idx.cpu().numpy().astype(np.uint32))


def _prepare_export(case, seed):
    idx, v = _export_values(case, seed)
    return dict(op="export", tmap=_texel_map(case["tex"], idx), data=context().upload(v.cpu().numpy()),
                mode=MODES[case["mode"]], dilate=case["dilate"])


def _prepare_denoise(case, seed):
    ctx, tex = context(), case["tex"]
    b = low_sample_bake(tex, seed)
    n = b["ao"].numel()
    up = {k: ctx.upload(b[k].cpu().numpy()) for k in ("tidx", "coords", "ao", "bn", "pos", "nrm")}
    params = np.load(TRAINED_WEIGHTS)["params"]
    image, ao, bn = ctx.buffer(48 * tex * tex), ctx.buffer(4 * n), ctx.buffer(12 * n)
    return dict(op="denoise", tmap=_texel_map(tex, b["idx"]), up=up, net=api.Denoiser(ctx, params), image=image, ao=ao,
                bn=bn, out=[tensor(image, (3, tex * tex, 4)), tensor(ao, (n,)), tensor(bn, (n, 3))])


def _prepare_train(case, seed):
    ctx = context()
    rows, targets, order = training_set(case, seed)
    return dict(op="train", net=api.Denoiser(ctx, init_params(seed)),
                rows=ctx.upload(rows.view(torch.int16).cpu().numpy()), targets=ctx.upload(targets.cpu().numpy()),
                order=ctx.upload(order.cpu().numpy()), n=case["dataset"], batch=case["batch"], steps=case["steps"])


_PREPARE = dict(maps=_prepare_maps, sample=_prepare_sample, bake=_prepare_bake, batch=_prepare_batch,
                export=_prepare_export, denoise=_prepare_denoise, train=_prepare_train)
_PREPARE["import"] = _prepare_import


# ------------------------------------------------------------------ run
def run(s):
    return _RUN[s["op"]](s)


def _normal_map(ctx, scene, tmap, b):
    api.gather(ctx, scene, api.GATHER_NORMAL, b["coords"], b["tidx"], b["normals"], 0, tmap.count)
    api.tangent_space(ctx, tmap, b["normals"])


def _run_maps(s):
    ctx, b, scene = context(), s["bufs"], s["pair"].scene
    tmap = s["pair"].texel_map(s["tex"])
    api.meshmap(ctx, scene, tmap, True, b["coords"], b["tidx"])
    api.gather(ctx, scene, api.GATHER_HEIGHT, b["coords"], b["tidx"], b["height"], 0, tmap.count)
    api.gather(ctx, scene, api.GATHER_POSITION, b["coords"], b["tidx"], b["position"], 0, tmap.count)
    _normal_map(ctx, scene, tmap, b)
    return s["out"]


def _run_sample(s):
    b = s["bufs"]
    api.hemisphere(context(), s["pair"].scene, s["coords"], s["tidx"], s["kind"], s["spp"], 0.001, s["max_d"],
                   s["table"], b[0], b[1], b[2], b[3], 0, s["tmap"].count)
    return s["out"]


def _run_import(s):
    ctx, b = context(), s["bufs"]
    s["high"].compute_normals_device(ctx, api.NORMALS_VERTEX)
    s["low"].compute_tangent_space_device(ctx)
    dirs = s["low"].copy()
    dirs.compute_normals_device(ctx, api.NORMALS_WELDED)
    tmap = api.TexelMap.from_meshes(ctx, s["low"], dirs, s["tex"], s["tex"])
    scene = api.Scene.build(ctx, s["high"])
    api.meshmap(ctx, scene, tmap, True, b["coords"], b["tidx"])
    _normal_map(ctx, scene, tmap, b)
    info = scene.info()
    return s["out"] + [info["node_count"], info["leaf_count"], info["depth"]]


def _run_bake(s):
    k = s["sampler"]
    api.bake(context(), s["nodes"], s["pos4"], s["nrm4"], s["tex"], s["tex"], s["pix8"], s["pixt12"], s["idx"],
             s["outputs"], height_map=True, position_map=True, normals_map=True, ao=k,
             bent_normals=dict(k, tangent_space=True), thickness=k)
    return s["out"]


def _run_batch(s):
    s["batch"].replay()
    return s["out"]


def _run_export(s):
    image, (lo, hi) = api.export_image(context(), s["tmap"], s["data"], s["mode"], dilate=s["dilate"])
    return [image, lo, hi]


def _run_denoise(s):
    u = s["up"]
    api.denoise_features(context(), s["tmap"], u["coords"], u["tidx"], u["ao"], u["bn"], u["pos"], u["nrm"], 0.3,
                         s["image"])
    s["net"].apply(s["tmap"], s["image"], u["tidx"], u["ao"], u["bn"], s["ao"], s["bn"])
    return s["out"]


def _run_train(s):
    for k in range(s["steps"]):
        s["net"].train_step(s["rows"], s["targets"], s["n"], s["batch"], s["order"], k * s["batch"], lr=3e-3)
    return [s["net"].last_loss(), s["net"].get_params()]


_RUN = dict(maps=_run_maps, sample=_run_sample, bake=_run_bake, batch=_run_batch, export=_run_export,
            denoise=_run_denoise, train=_run_train)
_RUN["import"] = _run_import


# ------------------------------------------------------------------ work
def _triangles(shape, hi):
    return 2 * hi * hi if shape == "plane" else 2 * hi * (max(8, hi // 2) - 1)


def _ray_flops(triangles):
    """One ray that goes straight to the triangle it hits: two boxes a level
    of a binary tree over leaves of eight (six subtractions and products, eight
    compares each), then one triangle."""
    return 2 * 20 * max(1.0, math.log2(max(2, triangles / 8))) + 60


def work(case):
    op = case["op"]
    if op in ("maps", "sample", "import", "bake"):
        tris, texels = _triangles(case["shape"], case["hi"]), case["tex"] ** 2
        scene = tris * (3 * 32 + 36 * 2 / 8)  # corners (position, normal) and nodes
        if op == "maps":
            return dict(bytes=scene + texels * (16 + 4 + 4 + 12 + 12), flops=2 * texels * _ray_flops(tris))
        if op == "import":
            # mesh in, scene out, maps out; a comparison and a move per triangle and level
            return dict(bytes=tris * 48 + scene + texels * (16 + 4 + 12),
                        flops=2 * texels * _ray_flops(tris) + 20 * tris * math.log2(max(2, tris / 8)))
        passes = 1 if op == "sample" else 2
        out = 20 if op == "sample" else 16 + 4 + 4 + 12 + 12 + 4 + 12 + 4
        return dict(bytes=scene + PERMS * case["spp"] * 16 + texels * (20 + out),
                    flops=passes * texels * case["spp"] * _ray_flops(tris))
    if op == "batch":
        jobs = _batch_jobs(case)
        return dict(bytes=sum(_triangles(s, h) * 105 + t * t * 28 for s, h, t, _ in jobs),
                    flops=sum(t * t * k * _ray_flops(_triangles(s, h)) for s, h, t, k in jobs))
    if op == "export":
        px = case["tex"] ** 2
        floats = 1 if case["mode"].startswith("float") else 3
        return dict(bytes=0.75 * px * 4 * (1 + floats) + px * (3 if case["mode"].endswith("rgb8") else 4 * floats),
                    flops=px * 4)
    flops = 2 * (250 * 64 + 64 * 64 + 64 * 4)
    if op == "denoise":
        px = case["tex"] ** 2
        return dict(bytes=px * (48 + 0.75 * (4 + 4 + 16 + 16 + 24 + 16)), flops=0.75 * px * flops)
    rows = case["batch"] * case["steps"]
    return dict(bytes=rows * (512 + 16 + 4) + api.DN_PARAMS * 12, flops=3 * rows * flops)


# ------------------------------------------------------------------ tolerance
def tolerance(case):
    op = case["op"]
    if op in ("maps", "import"):
        # the mapping is defined bit for bit; a ray on an edge shared by two triangles may take either
        return {"rel": 1e-5, "max": 0.5, "differ": 1e-5}
    if op in ("sample", "bake", "batch"):
        # 32-bit sums over a texel's samples; a grazing ray may change one sample of a texel
        return {"rel": 2e-5, "max": 0.25, "differ": 1e-4}
    if op == "export":
        return {"rel": 1e-6, "max": 1e-5, "differ": 0.0}
    if op == "denoise":
        # bf16 network: a value at a rounding boundary may round either way
        return {"rel": 1e-3, "max": 0.1}
    # bf16 activations and gradients; Adam divides by the gradient's own size, so that a small gradient's rounding
    # shows in its weight's step
    return {"rel": 1e-2, "max": 0.5}


# ------------------------------------------------------------------ exact
def exact(case, seed):
    f = _EXACT.get(case["op"])
    return f(case, seed) if f else None


def _unit(v):
    return v / v.norm(dim=-1, keepdim=True)


def _exact_low(lo, mapping):
    """Low-poly corners in 64 bits: positions, normals, directions, texcoords,
    tangents and bitangents of every triangle, (triangles, 3, .)."""
    d = lambda a: torch.from_numpy(a.astype(np.float64)).cuda()  # noqa: E731
    verts, tris = torch.from_numpy(lo.vertices.astype(np.int64)).cuda(), torch.from_numpy(lo.triangles.astype(np.int64)).cuda()
    pos, uv, nrm = d(lo.positions), d(lo.texcoords), d(lo.normals)
    p, u, n = pos[verts[tris, 0]], uv[verts[tris, 1]], nrm[verts[tris, 2]]
    face = _unit(torch.linalg.cross(p[:, 1] - p[:, 0], p[:, 2] - p[:, 0]))
    # directions: face normals summed over equal positions
    _, slot = torch.unique(pos[verts[tris, 0]].reshape(-1, 3), dim=0, return_inverse=True)
    acc = torch.zeros(int(slot.max()) + 1, 3, dtype=torch.float64, device="cuda")
    acc.index_add_(0, slot, face.repeat_interleave(3, 0))
    dirs = _unit(acc)[slot].reshape(-1, 3, 3) if mapping != "lowpoly" else n
    # tangents: per vertex
    e0, e1, t0, t1 = p[:, 1] - p[:, 0], p[:, 2] - p[:, 0], u[:, 1] - u[:, 0], u[:, 2] - u[:, 0]
    sdir = (e0 * t1[:, 1:] - e1 * t0[:, 1:]) / (t0[:, :1] * t1[:, 1:] - t1[:, :1] * t0[:, 1:])
    tacc = torch.zeros(verts.shape[0], 3, dtype=torch.float64, device="cuda")
    tacc.index_add_(0, tris.reshape(-1), sdir.repeat_interleave(3, 0))
    vn = nrm[verts[:, 2]]
    t = _unit(tacc - vn * (vn * tacc).sum(1, keepdim=True))
    b = torch.linalg.cross(vn, t)
    return p, n, dirs, u, t[tris], b[tris]


def _exact_texels(case, lo):
    """Texel rows of the low-poly's UV raster, in 64 bits; later triangles win."""
    p, n, d, u, t, b = _exact_low(lo, case["mapping"])
    tex = case["tex"]
    owner = torch.full((tex * tex,), -1, dtype=torch.int64, device="cuda")
    bary = torch.zeros(tex * tex, 3, dtype=torch.float64, device="cuda")
    uc = u.cpu().numpy()
    for f in range(uc.shape[0]):
        s = (uc[f] - 0.5 / tex) * tex
        # rounded half away from zero; a box that starts below zero is left out, as in the reference's unsigned loops
        x0, y0 = (int(math.copysign(math.floor(abs(v) + 0.5), v)) for v in s.min(0))
        x1, y1 = (int(min(tex - 1, math.floor(v + 0.5))) for v in s.max(0))
        if x0 < 0 or y0 < 0 or x1 < x0 or y1 < y0:
            continue
        ys, xs = np.mgrid[y0:y1 + 1, x0:x1 + 1]
        q = np.stack([(xs + 0.5) / tex, (ys + 0.5) / tex], -1).reshape(-1, 2) - uc[f, 0]
        a, c = uc[f, 1] - uc[f, 0], uc[f, 2] - uc[f, 0]
        det = a[0] * c[1] - c[0] * a[1]
        if det == 0:
            continue
        i, j = (q[:, 0] * c[1] - c[0] * q[:, 1]) / det, (a[0] * q[:, 1] - q[:, 0] * a[1]) / det
        w = np.stack([1 - i - j, i, j], -1)
        ok = ((w >= -0.001) & (w <= 1)).all(1)
        at = torch.from_numpy((ys * tex + xs).reshape(-1)[ok]).cuda()
        owner[at] = f
        bary[at] = torch.from_numpy(w[ok]).cuda()
    at = (owner >= 0).nonzero().reshape(-1)
    f, w = owner[at], bary[at][:, :, None]
    mix = lambda v: (v[f] * w).sum(1)  # noqa: E731
    return mix(p), _unit(mix(d)), _unit(mix(n)), _unit(mix(t)), _unit(mix(b))


def _exact_high(high):
    """High-poly triangles in 64 bits: corners, smooth corner normals, and the
    plane and barycentric terms of the ray tests."""
    pos = torch.from_numpy(high.positions.astype(np.float64)).cuda()
    verts = torch.from_numpy(high.vertices.astype(np.int64)[:, 0]).cuda()
    vi = verts[torch.from_numpy(high.triangles.astype(np.int64)).cuda()]
    p = pos[vi]
    v0, v1 = p[:, 1] - p[:, 0], p[:, 2] - p[:, 0]
    face = _unit(torch.linalg.cross(v0, v1))
    acc = torch.zeros_like(pos)
    acc.index_add_(0, vi.reshape(-1), face.repeat_interleave(3, 0))
    return p, _unit(acc)[vi], v0, v1, face


def _exact_hits(tri, o, d, slack):
    """Distances of rays against every triangle (infinite where missed) and
    the barycentrics, (rays, triangles), in chunks of rays: yields
    (first ray, one past the last, distance, cosine, x, y, z)."""
    p, _, v0, v1, face = tri
    d00, d01, d11 = (v0 * v0).sum(1), (v0 * v1).sum(1), (v1 * v1).sum(1)
    den = d00 * d11 - d01 * d01
    step = max(1, int(2e7 // p.shape[0]))
    for r0 in range(0, o.shape[0], step):
        r1 = min(r0 + step, o.shape[0])
        nd = d[r0:r1] @ face.T
        dist = ((p[:, 0] * face).sum(1)[None] - o[r0:r1] @ face.T) / nd
        along = lambda v: o[r0:r1] @ v.T + dist * (d[r0:r1] @ v.T) - (p[:, 0] * v).sum(1)[None]  # noqa: E731
        d20, d21 = along(v0), along(v1)
        y, z = (d11 * d20 - d01 * d21) / den, (d00 * d21 - d01 * d20) / den
        x = 1 - y - z
        ok = (x >= -slack) & (y >= -slack) & (z >= -slack) & (y <= 1) & (z <= 1)
        yield r0, r1, torch.where(ok, dist, math.inf), nd, x, y, z


def _exact_mapping(case, seed, rays=1):
    """The texels' rows and their mapping in 64 bits, by testing every
    triangle, or None for a case where that takes too long.  On the plane the
    rays run along the axes, and one that lies in a box face misses the box
    by the reference's rule, so only the sphere has a value of its own."""
    if case.get("mapping") == "hybrid" or case["shape"] == "plane" or case["tex"] ** 2 * _triangles(case["shape"], case["hi"]) * rays > 2e9:
        return None
    lo, high = meshes(case["shape"], case["hi"], seed)
    rows = _exact_texels(dict(mapping="smooth", **case) if "mapping" not in case else case, lo)
    tri = _exact_high(high)
    o, d = rows[:2]
    best = torch.full((o.shape[0],), math.inf, dtype=torch.float64, device="cuda")
    found = torch.zeros(o.shape[0], dtype=torch.int64, device="cuda")
    w = torch.zeros(o.shape[0], 3, dtype=torch.float64, device="cuda")
    # the nearest triangle facing along the direction, on either side of the texel
    for r0, r1, dist, nd, x, y, z in _exact_hits(tri, o, d, 1e-5):
        best[r0:r1], k = torch.where(nd > 0, dist.abs(), math.inf).min(1)
        found[r0:r1] = k
        w[r0:r1] = torch.stack([v.gather(1, k[:, None])[:, 0] for v in (x, y, z)], 1)
    hit = best < math.inf
    return rows, tri, hit, best, found, torch.where(hit[:, None], w, 0.0)


def _exact_maps(case, seed):
    m = _exact_mapping(case, seed)
    if m is None:
        return None
    (_, _, n, t, b), tri, hit, best, k, w = m
    coords = torch.cat([torch.where(hit, best, api.FLT_MAX)[:, None], w], 1)
    position = torch.where(hit[:, None], (tri[0][k] * w[:, :, None]).sum(1), 0.0)
    ts = _tangent_space(_unit((tri[1][k] * w[:, :, None]).sum(1)), n, t, b)
    return [coords, None, torch.where(hit, best, 0.0), position, torch.where(hit[:, None], ts, math.nan)]


def _exact_sample(case, seed):
    """AO by testing every triangle; the other kinds also count hits past the
    maximum distance in a leaf that starts before it, so they have no value
    without the package's own tree."""
    m = _exact_mapping(case, seed, case["spp"]) if case["kind"] == "ao" else None
    if m is None:
        return None
    _, tri, hit, _, k, w = m
    o = (tri[0][k] * w[:, :, None]).sum(1)
    d = _unit((tri[1][k] * w[:, :, None]).sum(1))
    zero = torch.zeros_like(d[:, 0])
    wide = d[:, 0].abs() > d[:, 1].abs()
    ty = _unit(torch.where(wide[:, None], torch.stack([d[:, 2], zero, -d[:, 0]], 1),
                           torch.stack([zero, d[:, 2], -d[:, 1]], 1)))
    tx = torch.linalg.cross(d, ty)
    spp = case["spp"]
    table = torch.from_numpy(api.samples_cosine(spp, PERMS, seed & 0x7FFFFFFF)).cuda().double().reshape(PERMS, spp, 4)
    occluded = torch.zeros(o.shape[0], dtype=torch.float64, device="cuda")
    for s in range(spp):
        rs = table[torch.arange(o.shape[0], device="cuda") % PERMS, s]
        ray = _unit(tx * rs[:, 0:1] + ty * rs[:, 1:2] + d * rs[:, 2:3])
        for r0, r1, dist, _, _, _, _ in _exact_hits(tri, o, ray, 0.0):
            occluded[r0:r1] += ((dist >= 0.001) & (dist < case["max_d"])).any(1)
    return [torch.where(hit, 1 - occluded / spp, 1.0), None]


def _tangent_space(v, n, t, b):
    """v against the rows of the adjugate of (n, t, b), as the tangent-space pass orders them."""
    rows = torch.stack([torch.linalg.cross(b, n), torch.linalg.cross(n, t), torch.linalg.cross(t, b)], 1)
    return _unit((rows * v[:, None, :]).sum(2))


def _exact_export(case, seed):
    if case["mode"].endswith("rgb8"):
        return None
    idx, v = _export_values(case, seed)
    tex = case["tex"]
    v = v.double()
    flip = (tex - 1 - torch.div(idx, tex, rounding_mode="floor")) * tex + idx % tex
    if case["mode"] == "float_f32":
        lo, hi = v.min(), v.max()
        image = torch.zeros(tex * tex, dtype=torch.float64, device="cuda")
        image[flip] = (v - lo) / (hi - lo)
        return [image.reshape(tex, tex), float(lo), float(hi)]
    image = torch.zeros(3, tex * tex, dtype=torch.float64, device="cuda")
    image[:, flip] = v.T.flip(0)
    return [image.reshape(3, tex, tex), None, None]


def _exact_denoise(case, seed):
    tex = case["tex"]
    b = low_sample_bake(tex, seed)
    f = feature_image(b, tex, 0.3)
    params = torch.from_numpy(np.load(TRAINED_WEIGHTS)["params"].astype(np.float64)).cuda()
    y = torch.cat([network(params, input_rows(f, tex, p)) for p in b["idx"].long().split(65536)])
    ao = (b["ao"].double() + y[:, 0]).clamp(0, 1)
    bn = _unit(b["bn"].double() + y[:, 1:])
    miss = b["tidx"] == -1
    return [f, torch.where(miss, 1.0, ao), torch.where(miss[:, None], 0.0, bn)]


def _exact_train(case, seed):
    rows, targets, order = training_set(case, seed)
    p = torch.from_numpy(init_params(seed).astype(np.float64)).cuda()
    m, v, loss = torch.zeros_like(p), torch.zeros_like(p), None
    for k in range(case["steps"]):
        at = order[k * case["batch"]:(k + 1) * case["batch"]].long()
        q = p.clone().requires_grad_(True)
        loss = ((network(q, rows[at].double()) - targets[at].double()) ** 2).mean()
        loss.backward()
        m = 0.9 * m + 0.1 * q.grad
        v = 0.999 * v + 0.001 * q.grad ** 2
        p = p - 3e-3 * (m / (1 - 0.9 ** (k + 1))) / ((v / (1 - 0.999 ** (k + 1))).sqrt() + 1e-8)
    return [float(loss), p]


_EXACT = dict(maps=_exact_maps, sample=_exact_sample, export=_exact_export, denoise=_exact_denoise, train=_exact_train)
