"""Performance cases of the voxel-lighting path, each one call (or one frame)
that a program using the library makes through its public entry points.

A case's "kind" names the path; its other fields are sizes and options. Grids,
models and images are seeded synthetic ones of the same make as the benchmark's
(noise grids with boxes, fbm terrain, Vox models of random palette blocks,
pinhole G-buffers). One library context serves the whole process, as in an
engine.
"""
import math

import numpy as np
import torch

import voxelengine_gb300 as V
from voxelengine_gb300 import scenes as S

F32, F64, DEV = torch.float32, torch.float64, "cuda"
OUTS = ("shadow", "ao", "ao_vis", "spec", "spec_t")


def listed():
    return [
        # smallest call: a thumbnail / probe-sized view of a 128^3 prop scene, odd image size; launches and latency count
        dict(name="occl_small", kind="occl", n=128, boxes=20, W=161, H=91, n_ao=8, n_spec=1, ao_len=32.0),
        # the headline frame: 512^3 world at 1080p, 1 shadow + 8 AO + 1 specular ray a pixel
        dict(name="occl_1080p", kind="occl", n=512, boxes=2000, W=1920, H=1080, n_ao=8, n_spec=1, ao_len=32.0),
        # open-world view: 1024^3 terrain with placed models, 18 long rays a pixel (the wide trace layout)
        dict(name="occl_terrain", kind="terrain", n=1024, inst=1500, W=1920, H=1080, n_ao=16, n_spec=1, ao_len=64.0),
        # many views of grids of mixed sizes in one launch (thumbnails, probes, split screens)
        dict(name="batch_mixed", kind="batch", count=24, e0=64, e1=320, r0=65536, r1=1048576, n_ao=8, n_spec=1),
        # one optimisation step of the differentiable variant: forward, loss gradient, adjoint
        dict(name="soft_step", kind="soft", nx=128, ny=128, nz=128, W=512, H=512, n_ao=16, length=24.0),
        # the G-buffer producer: 4096 Vox instances (the engine's per-frame cap) at 1080p
        dict(name="primary_1080p", kind="primary", n=512, inst=4096, W=1920, H=1080),
        # the engine's own light passes of a frame: sun + ambient, reflection, and 64 point / spot lights
        dict(name="lights_1080p", kind="lights", n=512, boxes=500, W=1920, H=1080, nlights=64),
        # temporal accumulation of the lighting under a panning camera
        dict(name="taa_1080p", kind="taa", n=512, W=1920, H=1080),
        # per-frame grid update: 64 moved entities in an engine-sized ShadowVox grid (524 x 188 x 524 bytes)
        dict(name="update_engine", kind="update", nx=1048, ny=376, nz=1048, ents=64, e0=8, e1=48),
        # level load: a saved world read from the engine's R8 layout, then 2048 placed models set in it
        dict(name="load_world", kind="load", nx=512, ny=512, nz=512, inst=2048, e0=8, e1=64),
        # gameplay and baking queries: independent rays with full records, exact and marched
        dict(name="rays_1m", kind="rays", n=384, boxes=200, rays=1000003),
        # a whole small frame: move entities, draw, trace, 16 lights, accumulate (640x360, a preview window)
        dict(name="frame_360p", kind="frame", n=256, inst=256, ents=12, W=640, H=360, nlights=16),
    ]


def _log(rng, a, b):
    return int(round(math.exp(rng.uniform(math.log(a), math.log(b)))))


def _image(rng, lo, hi):
    npix = _log(rng, lo, hi)
    w = max(9, int(round(math.sqrt(npix * rng.uniform(1.0, 2.2)))))
    return dict(W=w, H=max(7, npix // w))


def draw(rng):
    kind = rng.choice(["occl", "occl", "terrain", "batch", "soft", "soft", "primary", "lights", "taa", "update", "load",
                       "rays", "frame"])
    even = lambda a, b: 2 * _log(rng, a // 2, b // 2)  # noqa: E731
    if kind == "occl":
        n = even(64, 640)
        return dict(kind=kind, n=n, boxes=rng.randint(0, n), n_ao=rng.choice([1, 4, 8, 13, 16]),
                    n_spec=rng.choice([0, 1, 2]), ao_len=rng.choice([16.0, 32.0, 48.0]), **_image(rng, 8000, 2000000))
    if kind == "terrain":
        return dict(kind=kind, n=even(1020, 1100), inst=rng.randint(0, 1500), n_ao=rng.choice([4, 8, 16]),
                    n_spec=rng.choice([0, 1]), ao_len=rng.choice([32.0, 64.0]), **_image(rng, 100000, 2000000))
    if kind == "batch":
        return dict(kind=kind, count=rng.randint(3, 24), e0=64, e1=rng.randint(96, 320), r0=65536,
                    r1=_log(rng, 131072, 1048576), n_ao=rng.choice([4, 8]), n_spec=rng.choice([0, 1]))
    if kind == "soft":
        return dict(kind=kind, nx=even(32, 160), ny=even(32, 128), nz=even(32, 160), n_ao=rng.randint(1, 16),
                    length=rng.choice([8.0, 16.0, 24.0]), **_image(rng, 2000, 260000))
    if kind == "primary":
        return dict(kind=kind, n=even(128, 640), inst=_log(rng, 30, 4096), **_image(rng, 30000, 2000000))
    if kind == "lights":
        n = even(96, 576)
        return dict(kind=kind, n=n, boxes=rng.randint(0, n), nlights=_log(rng, 1, 64), **_image(rng, 20000, 2000000))
    if kind == "taa":
        return dict(kind=kind, n=even(96, 512), **_image(rng, 5000, 2000000))
    if kind == "update":
        return dict(kind=kind, nx=even(128, 1048), ny=even(64, 376), nz=even(128, 1048), ents=_log(rng, 1, 64), e0=8,
                    e1=rng.randint(12, 48))
    if kind == "load":
        return dict(kind=kind, nx=even(64, 640), ny=even(64, 400), nz=even(64, 640), inst=_log(rng, 1, 2048), e0=8,
                    e1=rng.randint(12, 64))
    if kind == "rays":
        n = even(64, 512)
        return dict(kind=kind, n=n, boxes=rng.randint(0, n), rays=_log(rng, 500, 1000000))
    return dict(kind=kind, n=even(128, 384), inst=_log(rng, 16, 512), ents=rng.randint(1, 16), nlights=rng.randint(1, 32),
                **_image(rng, 20000, 500000))


# ------------------------------------------------------------------ inputs
_CTX = []


def _ctx():
    if not _CTX:
        _CTX.append(V.Context(0))
    return _CTX[0]


class _Mem:
    """Device memory of a grid, for torch.as_tensor; the tensor keeps this object, and it the grid."""

    def __init__(self, grid, ptr, nbytes, width):
        self.grid = grid
        self.__cuda_array_interface__ = dict(shape=(nbytes // width,), typestr="<i%d" % width, data=(ptr, False), version=3)


def _grid_buffers(G):
    """The grid's own words, tile map and trace layout, as tensors over its memory."""
    d = G.describe()
    bufs = {"words": torch.as_tensor(_Mem(G, d.words, d.words_bytes, 8), device=DEV),
            "tile_mask": torch.as_tensor(_Mem(G, d.tile_mask, d.tile_mask_bytes, 4), device=DEV)}
    if d.trace_words:
        bufs["trace_words"] = torch.as_tensor(_Mem(G, d.trace_words, d.trace_words_bytes, 8), device=DEV)
    return bufs


def _empty(npix, ch=1, dtype=F32):
    return torch.empty(npix * ch, dtype=dtype, device=DEV)


def _gen(seed):
    return torch.Generator(device=DEV).manual_seed(seed)


def _rand(g, *shape):
    return torch.rand(*shape, dtype=F32, device=DEV, generator=g)


def _noise_grid(n, boxes, seed):
    G = V.Grid(_ctx(), n, n, n)
    G.scene_noise(seed, 0.55, 1.0 / 32.0, 8)
    if boxes:
        G.scene_boxes(seed, boxes, 4, max(5, min(48, n // 4)))
    return G


def _gbuffer(G, cam, tgt, W, H, seed):
    pos, nrm, rough = _empty(W * H, 3), _empty(W * H, 3), _empty(W * H)
    V.scene_gbuffer(_ctx(), G, cam, tgt, W, H, seed, pos, nrm, rough)
    return dict(pos=pos, nrm=nrm, rough=rough)


def _placement(rng, dims, shape, R=None, centre=None):
    """Column-major world matrix of a model whose centre lies inside the grid."""
    R = S.rotation_matrix(rng) if R is None else R
    centre = rng.uniform(0.0, np.asarray(dims) / 10.0) if centre is None else centre
    m = np.eye(4)
    m[:3, :3] = R
    m[:3, 3] = centre - R @ (0.05 * np.array(shape[::-1]))
    return np.ascontiguousarray(m.T.astype(np.float32)).reshape(16), R, centre


def _models(seed, count, e0, e1):
    ms = S.vox_models(seed, count, e0, e1, fill=0.4)
    dev = [torch.from_numpy(m).cuda() for m in ms]
    return ms, dev, [(d.data_ptr(),) + m.shape[::-1] for m, d in zip(ms, dev)]


def _moves(rng, dims, models, n):
    """Entities that move a little and turn: (pose A, pose B, pivot, model)."""
    out = []
    for _ in range(n):
        mi = int(rng.integers(0, len(models)))
        a, R, c = _placement(rng, dims, models[mi].shape)
        t = rng.uniform(-0.1, 0.1)
        turn = np.array([[math.cos(t), 0, math.sin(t)], [0, 1, 0], [-math.sin(t), 0, math.cos(t)]])
        b, _, _ = _placement(rng, dims, models[mi].shape, turn @ R, c + rng.uniform(-0.5, 0.5, 3))
        out.append((a, b, rng.uniform(0.0, 0.5, 3).astype(np.float32), mi))
    return out


def _both_ways(moves):
    return [[(a, b, p, m) for a, b, p, m in moves], [(b, a, p, m) for a, b, p, m in moves]]


def _lights(rng, n, count):
    return [(rng.uniform(0.0, n / 10.0, 3).astype(np.float32), float(rng.uniform(4.0, 12.0)), i % 3 == 2) for i in range(count)]


def prepare(case, seed):
    c, k, ctx = case, case["kind"], _ctx()
    st = dict(case=case, ctx=ctx)
    rng, g = np.random.default_rng(seed), _gen(seed)
    npix = c.get("W", 0) * c.get("H", 0)
    st["npix"] = npix
    if k in ("occl", "terrain"):
        if k == "occl":
            cam, tgt = S.camera(c["n"])
            G, shadow_len = _noise_grid(c["n"], c["boxes"], seed), 100.0
        else:
            G, shadow_len = V.Grid(ctx, c["n"], c["n"], c["n"]), 256.0
            G.scene_terrain(seed, c["n"] / 16.0, c["n"] / 4.0, 4.0 / c["n"], 6)
            ms, dev, desc = _models(seed + 1, 16, 16, 96)
            ins = []
            for _ in range(c["inst"]):
                mi = int(rng.integers(0, len(ms)))
                centre = rng.uniform(0.0, np.array([c["n"], c["n"] * 0.35, c["n"]]) / 10.0)
                ins.append((_placement(rng, None, ms[mi].shape, None, centre)[0], mi, V.OP_SET))
            V.voxelize(ctx, G, desc, ins)
            torch.cuda.synchronize()
            cam, tgt = S.terrain_camera(c["n"], c["n"] * 0.3)
        st.update(grid=G, **_gbuffer(G, cam, tgt, c["W"], c["H"], seed))
        st["params"] = V.make_params(light_dir=S.light_dir(seed), cam_pos=cam, shadow_len=shadow_len, ao_len=c["ao_len"],
                                     n_ao=c["n_ao"], n_spec=c["n_spec"], seed=seed & 0x7FFFFFFF)
        st["out"] = {o: _empty(npix) for o in OUTS}
    elif k == "batch":
        R = 1 + c["n_ao"] + c["n_spec"]
        items, sizes, mix = [], [], np.random.default_rng(c["count"])  # the sizes belong to the case
        for i in range(c["count"]):
            n = 2 * int(round(math.exp(mix.uniform(math.log(c["e0"]), math.log(c["e1"]))) / 2))
            W, H = S.image_for_pixels(math.exp(mix.uniform(math.log(c["r0"]), math.log(c["r1"]))) / R)
            sizes.append((n, W, H))
        start = np.concatenate([[0], np.cumsum([W * H for _, W, H in sizes])])
        st["out"] = {o: _empty(int(start[-1])) for o in OUTS}  # the views' outputs one after another
        for i, (n, W, H) in enumerate(sizes):
            s = (seed * 1009 + i) & 0x7FFFFFFF
            cam, tgt = S.camera(n)
            G = V.Grid(ctx, n, n, n)
            G.scene_noise(s, float(rng.uniform(0.45, 0.65)), 1.0 / 32.0, 8)
            P = V.make_params(light_dir=S.light_dir(s), cam_pos=cam, ao_len=32.0, n_ao=c["n_ao"], n_spec=c["n_spec"], seed=s)
            items.append(dict(grid=G, npix=W * H, width=W, height=H, params=P, **_gbuffer(G, cam, tgt, W, H, s),
                              **{o: t[start[i]:start[i + 1]] for o, t in st["out"].items()}))
        st.update(items=items, batch=V.Batch(ctx, items))
    elif k == "soft":
        dims = (c["nz"], c["ny"], c["nx"], 4)
        n = min(c["nx"], c["ny"], c["nz"])
        G = V.Grid(ctx, c["nx"], c["ny"], c["nz"])
        G.scene_noise(seed, 0.55, 1.0 / 32.0, 8)
        cam = np.array([0.5 * c["nx"], 1.15 * c["ny"] + 0.2 * n, -0.1 * c["nz"]], np.float32)
        tgt = np.array([0.5 * c["nx"], 0.5 * c["ny"], 0.5 * c["nz"]], np.float32)
        st.update(_gbuffer(G, cam, tgt, c["W"], c["H"], seed))
        st["soft"] = torch.empty(dims, dtype=F32, device=DEV)
        V.scene_soft(ctx, st["soft"], seed, albedo_seed=seed + 1)
        st["params"] = V.make_soft_params(light_dir=S.light_dir(seed), length=c["length"], n_ao=c["n_ao"], seed=seed & 0x7FFFFFFF)
        st["target"] = _rand(g, npix, 3)
        for b in ("image", "light", "gimg"):
            st[b] = torch.empty((npix, 3), dtype=F32, device=DEV)
        st["grad"] = torch.zeros_like(st["soft"])
    elif k in ("primary", "frame"):
        n = c["n"]
        ms, dev, desc = _models(seed, 48 if k == "primary" else 12, 16, min(64, n // 4))
        vol = rng.integers(0, len(ms), c["inst"]).astype(np.int32)
        worlds = np.array([_placement(rng, (n, n, n), ms[v].shape)[0] for v in vol], np.float32).reshape(-1, 16)
        cam, tgt = S.camera(n)
        st.update(vols=V.VolumeSet(ctx, ms), cam=cam * np.float32(0.1), tgt=tgt * np.float32(0.1),
                  pos=_empty(npix, 3), nrm=_empty(npix, 3), depth=_empty(npix), material=_empty(npix, 1, torch.int32),
                  instance=_empty(npix, 1, torch.int32))
        st["cmds"] = [V.voxcmds(worlds, vol)] * 2
        if k == "frame":
            moves = _moves(rng, (n, n, n), ms, c["ents"])
            pivots = lambda m, p: (m.reshape(4, 4).T @ np.array([[1, 0, 0, -p[0]], [0, 1, 0, -p[1]], [0, 0, 1, -p[2]], [0, 0, 0, 1]])).T  # noqa: E731
            G = V.Grid(ctx, n, n, n)
            V.voxelize(ctx, G, desc, [(w, int(v), V.OP_SET) for w, v in zip(worlds, vol)])
            after = [np.array([pivots(e[1 - s], e[2]).reshape(16) for e in moves], np.float32) for s in (0, 1)]
            mvol = np.array([e[3] for e in moves], np.int32)
            st["cmds"] = [V.voxcmds(np.concatenate([worlds, after[s]]), np.concatenate([vol, mvol])) for s in (0, 1)]
            st.update(grid=G, dev=dev, desc=desc, ents=_both_ways(moves), turn=0, noise=_rand(g, npix * 4), wpos=_empty(npix, 3),
                      lights=_lights(rng, n, c["nlights"]), lit=_empty(npix, 1, torch.int64), color=torch.full((npix * 3,), 0.5, device=DEV),
                      mat=torch.zeros(npix * 4, device=DEV), motion=(_rand(g, npix * 2) - 0.5) * 2e-3, light=torch.zeros((npix, 4), device=DEV),
                      last=_rand(g, npix * 4), taa=_empty(npix, 4), bufs=_grid_buffers(G))
            st["out"] = {o: _empty(npix) for o in OUTS}
            st["params"] = V.make_params(light_dir=S.light_dir(seed), cam_pos=cam, ao_len=32.0, n_ao=8, n_spec=1, seed=seed & 0x7FFFFFFF)
    elif k == "lights":
        n = c["n"]
        cam, tgt = S.camera(n)
        G = _noise_grid(n, c["boxes"], seed)
        gb = _gbuffer(G, cam, tgt, c["W"], c["H"], seed)
        p3, n3 = gb["pos"].view(-1, 3), gb["nrm"].view(-1, 3)
        view = p3 - torch.from_numpy(cam).cuda()
        st.update(grid=G, **gb, wpos=gb["pos"] * 0.1, noise=_rand(g, npix * 4), lights=_lights(rng, n, c["nlights"]),
                  depth=view.norm(dim=1) / 40960.0, refl=(view - 2.0 * (view * n3).sum(1, keepdim=True) * n3).contiguous(),
                  shadow=_empty(npix), irr=_empty(npix), refl_t=_empty(npix), lit=_empty(npix, 1, torch.int64),
                  in_range=_empty(npix, 1, torch.int64))
    elif k == "taa":
        n = c["n"]
        cam, tgt = S.camera(n)
        gb = _gbuffer(_noise_grid(n, n, seed), cam, tgt, c["W"], c["H"], seed)
        p3, n3 = gb["pos"].view(-1, 3), gb["nrm"].view(-1, 3)
        sky = (n3 == 0).all(1)
        # materials and albedo in blocks of 16^3 voxels out of a small palette; lighting smooth with one ray's noise
        block = (p3 / 16.0).floor().to(torch.int64)
        mi = ((block[:, 0] * 7 + block[:, 1] * 13 + block[:, 2] * 29) % 8).abs()
        pal, mats = _rand(g, 8, 3), _rand(g, 8, 4) * 0.1
        depth = (p3 - torch.from_numpy(cam).cuda()).norm(dim=1) / 40960.0
        light = torch.rand(npix, 4, device=DEV, generator=g) * 0.3 + 0.2 + 0.4 * ((p3[:, :1] * 0.05).sin() + 1.0) * 0.5
        st.update(nrm=gb["nrm"], color=pal[mi].contiguous(), mat=mats[mi].contiguous(), depth=torch.where(sky, torch.ones_like(depth), depth),
                  light=light, last=(light + 0.1 * torch.randn(npix, 4, device=DEV, generator=g)).clamp(0, 1).contiguous(),
                  # the sky carries no motion
                  motion=((~sky)[:, None] * (torch.tensor([0.006, 0.004], device=DEV) + (_rand(g, npix, 2) - 0.5) * 1e-3)).contiguous(), noise=_rand(g, npix * 4), taa=_empty(npix, 4))
    elif k in ("update", "load"):
        dims = (c["nx"], c["ny"], c["nz"])
        ms, dev, desc = _models(seed, 16, c["e0"], c["e1"])
        G = V.Grid(ctx, *dims)
        G.scene_noise(seed, 0.6, 1.0 / 32.0, 8)
        st.update(grid=G, dev=dev, desc=desc, turn=0, bufs=_grid_buffers(G))
        if k == "update":
            moves = _moves(rng, dims, ms, c["ents"])
            st["ents"] = _both_ways(moves)
        else:
            st["saved"] = _empty(dims[0] * dims[1] * dims[2] // 8, 1, torch.uint8)
            G.export_r8(st["saved"])
            G.clear()
            st["ins"] = [(_placement(rng, dims, ms[i % len(ms)].shape)[0], i % len(ms), V.OP_SET) for i in range(c["inst"])]
            st["aabb"] = torch.empty((c["inst"], 6), dtype=torch.int32, device=DEV)
    else:  # rays: origins in the open half of the volume, directions over the sphere, lengths as the passes use
        n, r = c["n"], c["rays"]
        st["grid"] = _noise_grid(n, c["boxes"], seed)
        d = torch.nn.functional.normalize(torch.randn(r, 3, device=DEV, generator=g), dim=1)
        o = _rand(g, r, 3) * float(n)
        st["rays"] = torch.cat([o, d, 16.0 + 240.0 * _rand(g, r, 1)], 1).contiguous()
        st["exact"], st["march"] = (torch.empty((r, 6), dtype=torch.int32, device=DEV) for _ in range(2))
    return st


# --------------------------------------------------------------------- run
def run(st):
    c, ctx, k, npix = st["case"], st["ctx"], st["case"]["kind"], st["npix"]
    if k in ("occl", "terrain"):
        V.trace_occlusion(ctx, st["grid"], st["pos"], st["nrm"], st["rough"], npix, st["params"], width=c["W"], height=c["H"], **st["out"])
        return st["out"]
    if k == "batch":
        st["batch"].run()
        return st["out"]
    if k == "soft":
        V.trace_soft_fwd(ctx, st["soft"], st["pos"], st["nrm"], npix, st["params"], st["image"], st["light"])
        torch.sub(st["image"], st["target"], out=st["gimg"])
        st["gimg"].mul_(2.0 / st["image"].numel())
        st["grad"].zero_()
        V.trace_soft_bwd(ctx, st["soft"], st["pos"], st["nrm"], npix, st["params"], st["gimg"], st["light"], st["grad"])
        return {"image": st["image"], "light": st["light"], "grad": st["grad"]}
    if k == "primary":
        V.trace_primary(ctx, st["vols"], None, None, st["cam"], st["tgt"], c["W"], c["H"], st["pos"], st["nrm"], st["depth"],
                        st["material"], st["instance"], cmds=st["cmds"][0])
        return {o: st[o] for o in ("pos", "nrm", "depth", "material", "instance")}
    if k == "lights":
        V.light_ambient(ctx, st["grid"], st["pos"], st["nrm"], st["depth"], st["noise"], npix, st["shadow"], st["irr"])
        V.light_reflection(ctx, st["grid"], st["pos"], st["nrm"], st["refl"], st["rough"], st["noise"], npix, st["refl_t"])
        V.light_points(ctx, st["grid"], st["wpos"], st["nrm"], st["noise"], npix, st["lights"], st["lit"], st["in_range"])
        return {o: st[o] for o in ("shadow", "irr", "refl_t", "lit", "in_range")}
    if k == "taa":
        V.light_taa(ctx, st["light"], st["last"], st["color"], st["nrm"], st["mat"], st["depth"], st["motion"], st["noise"],
                    c["W"], c["H"], st["taa"])
        return st["taa"]
    if k == "update":
        reg = V.shadowvox_update(ctx, st["grid"], st["desc"], st["ents"][st["turn"]])
        st["turn"] ^= 1
        return {"regions": reg, **st["bufs"]}
    if k == "load":
        st["aabb"][:, :3] = 1 << 20
        st["aabb"][:, 3:] = 0
        st["grid"].import_r8(st["saved"])
        V.voxelize(ctx, st["grid"], st["desc"], st["ins"], st["aabb"])
        return {"aabb": st["aabb"], **st["bufs"]}
    if k == "rays":
        V.trace_rays(ctx, st["grid"], st["rays"], c["rays"], V.MODE_DDA, st["exact"])
        V.trace_rays(ctx, st["grid"], st["rays"], c["rays"], V.MODE_SPARSE, st["march"])
        return {"exact": st["exact"], "march": st["march"]}
    reg = V.shadowvox_update(ctx, st["grid"], st["desc"], st["ents"][st["turn"]])
    V.trace_primary(ctx, st["vols"], None, None, st["cam"], st["tgt"], c["W"], c["H"], st["pos"], st["nrm"], st["depth"],
                    st["material"], st["instance"], cmds=st["cmds"][st["turn"]])
    V.trace_occlusion(ctx, st["grid"], st["pos"], st["nrm"], None, npix, st["params"], width=c["W"], height=c["H"], **st["out"])
    torch.mul(st["pos"], 0.1, out=st["wpos"])
    V.light_points(ctx, st["grid"], st["wpos"], st["nrm"], st["noise"], npix, st["lights"], st["lit"])
    st["light"][:, 0].copy_(st["out"]["shadow"])
    st["light"][:, 1].copy_(st["out"]["ao"])
    st["light"][:, 2].copy_(st["out"]["spec"])
    V.light_taa(ctx, st["light"], st["last"], st["color"], st["nrm"], st["mat"], st["depth"].div_(4096.0), st["motion"], st["noise"],
                c["W"], c["H"], st["taa"])
    st["turn"] ^= 1
    return {"regions": reg, "words": st["bufs"]["words"], "pos": st["pos"], "instance": st["instance"], "lit": st["lit"],
            "taa": st["taa"], **st["out"]}


# -------------------------------------------------------------------- work
def work(case):
    """Bytes: every input and output once. Operations: the steps of rays of
    about half their length (most end at a hit), nine a step, and a hundred to
    set up each ray; forty for a bilinear tap of sixteen values."""
    c, k = case, case["kind"]
    npix = c.get("W", 0) * c.get("H", 0)

    def occl(n3, px, n_ao, n_spec, ao_len, shadow_len):
        rays = px * (1 + n_ao + n_spec)
        steps = px * 0.75 * (shadow_len * 0.5 + n_ao * ao_len + n_spec * 64.0)
        return dict(bytes=n3 / 8 + px * 48, flops=rays * 100 + steps * 9)

    if k in ("occl", "terrain"):
        return occl(c["n"] ** 3, npix, c["n_ao"], c["n_spec"], c["ao_len"], 100.0 if k == "occl" else 256.0)
    if k == "batch":
        R = 1 + c["n_ao"] + c["n_spec"]
        mean = lambda a, b: (b - a) / math.log(b / a) if b > a else a  # noqa: E731
        n3 = (c["e1"] ** 3 - c["e0"] ** 3) / (3 * math.log(c["e1"] / c["e0"])) if c["e1"] > c["e0"] else c["e0"] ** 3
        w = occl(n3, mean(c["r0"], c["r1"]) / R, c["n_ao"], c["n_spec"], 32.0, 100.0)
        return {q: v * c["count"] for q, v in w.items()}
    if k == "soft":
        vox, rays = c["nx"] * c["ny"] * c["nz"], npix * (1 + c["n_ao"])
        return dict(bytes=vox * 16 * 3 + npix * (48 + 48 + 36), flops=rays * 200 + rays * c["length"] * 0.75 * 60)
    if k == "primary":
        return dict(bytes=npix * 36 + c["inst"] * 72 + 48 * 40 ** 3, flops=npix * 600.0)
    if k == "lights":
        return dict(bytes=c["n"] ** 3 / 8 + npix * (48 + 12 + 56 + 4 + 52), flops=npix * 3000.0)
    if k == "taa":
        return dict(bytes=npix * (68 + 16 + 16 + 16), flops=npix * 12 * 16 * 8.0)
    if k == "update":
        v = c["ents"] * ((c["e0"] + c["e1"]) / 2) ** 3
        return dict(bytes=v * 2 * 1.4, flops=v * 2 * 24)
    if k == "load":
        v, n3 = c["inst"] * ((c["e0"] + c["e1"]) / 2) ** 3, c["nx"] * c["ny"] * c["nz"]
        return dict(bytes=16 * ((c["e0"] + c["e1"]) / 2) ** 3 + n3 * 3 / 8, flops=v * 24)
    if k == "rays":
        return dict(bytes=c["n"] ** 3 / 8 + c["rays"] * 2 * 52, flops=c["rays"] * (100 + 40 * 9 + 100 + 30 * 12))
    w = occl(c["n"] ** 3, npix, 8, 1, 32.0, 100.0)
    return dict(bytes=w["bytes"] + npix * (36 + 40 + 116), flops=w["flops"] + npix * (600 + 1500 + 1536))


# ------------------------------------------------------- the values, in 64 bits
def _pcg(v):
    m = 0xFFFFFFFF
    s = (v * 747796405 + 2891336453) & m
    w = (((s >> ((s >> 28) + 4)) ^ s) * 277803737) & m
    return (w >> 22) ^ w


def _u01(seed, pix, sample):
    """The sample's uniform number for each pixel (PCG of seed, pixel, sample)."""
    h = _pcg((_pcg((int(_pcg(torch.tensor([seed & 0xFFFFFFFF]))[0]) + pix) & 0xFFFFFFFF) + sample) & 0xFFFFFFFF)
    return (h >> 8).to(F64) / 16777216.0


def _occupancy(G):
    """bool[nz, ny, nx] from the grid's 4^3-brick words."""
    d = G.describe()
    w = torch.as_tensor(_Mem(G, d.words, d.words_bytes, 8), device=DEV).view(d.bz, d.by, d.bx)
    occ = torch.empty((d.bz * 4, d.by * 4, d.bx * 4), dtype=torch.bool, device=DEV)
    for b in range(64):
        occ[b >> 4::4, (b >> 2) & 3::4, b & 3::4] = ((w >> b) & 1).bool()
    return occ


def _unit(v):
    return v / v.norm(dim=1, keepdim=True)


def _frame(nrm):
    x, y, z = nrm.unbind(1)
    o = torch.zeros_like(x)
    t = torch.where((z.abs() > 0.5)[:, None], torch.stack([o, -z, y], 1), torch.stack([-y, x, o], 1))
    return t, torch.linalg.cross(nrm, t)


def _local(t, b, n, l):
    return t * l[:, :1] + b * l[:, 1:2] + n * l[:, 2:]


def _cosine(u1, u2):
    r, th = u1.sqrt(), 6.283 * u2
    return torch.stack([r * th.cos(), r * th.sin(), (1.0 - u1).clamp_min(0).sqrt()], 1)


def _walk(o, d, maxt, dims, visit):
    """The cells of the exact DDA of each ray, at most 256, up to maxt:
    visit(ids, cells, t) says which rays end there."""
    ids = torch.arange(o.shape[0], device=DEV)
    s = torch.where(d > 0, 1, -1)
    cell = o.floor().to(torch.int64)
    td = 1.0 / d.abs()
    tm = torch.where(d == 0, torch.full_like(d, math.inf), (cell + (s > 0) - o) / d)
    hi = torch.tensor(dims, device=DEV) + 1
    for n in range(256):
        m = tm.min(dim=1, keepdim=True).values
        inside = ((cell >= 0) & (cell <= hi)).all(1)
        stop = visit(ids, cell, m[:, 0], inside) | ~inside | (m[:, 0] >= maxt)
        sel = tm == m
        cell, tm = cell + s * sel, tm + torch.where(sel, td, torch.zeros_like(td))
        live = torch.nonzero(~stop).view(-1)
        if live.numel() == 0:
            return
        if live.numel() < stop.numel():
            ids, s, cell, td, tm = ids[live], s[live], cell[live], td[live], tm[live]


def _first_hit(occ, o, d, maxt, dims):
    """(hit, t of the hit cell's far side) of each ray."""
    hit = torch.zeros(o.shape[0], dtype=torch.bool, device=DEV)
    t = torch.zeros(o.shape[0], dtype=F64, device=DEV)
    top = torch.tensor([s - 1 for s in reversed(occ.shape)], device=DEV)

    def visit(ids, cell, m, inside):
        q = torch.minimum(cell.clamp_min(0), top)
        h = occ[q[:, 2], q[:, 1], q[:, 0]] & inside
        hit[ids[h]] = True
        t[ids[h]] = m[h]
        return h

    _walk(o, d, maxt, dims, visit)
    return hit, t


def _f(x):
    return torch.tensor(list(x), dtype=F64, device=DEV)


def _exact_occlusion(st):
    G, P, npix = st["grid"], st["params"], st["npix"]
    occ, dims = _occupancy(G), (G.nx, G.ny, G.nz)
    n_all = st["nrm"].view(-1, 3).to(F64)
    pix = torch.nonzero((n_all != 0).any(1)).view(-1)
    p, n, ro = st["pos"].view(-1, 3).to(F64)[pix], n_all[pix], st["rough"].to(F64)[pix]
    o, (t, b) = p + n * P.bias, _frame(n)
    out = {q: torch.ones(npix, dtype=F64, device=DEV) for q in OUTS}
    out["spec_t"].fill_(P.spec_len)
    out["shadow"][pix] = (~_first_hit(occ, o, _f(P.light_dir).expand_as(o), P.shadow_len, dims)[0]).to(F64)
    ao, vis = torch.zeros_like(ro), torch.zeros_like(ro)
    for k in range(P.n_ao):
        l = _cosine(_u01(P.seed, pix, 64 + 2 * k), _u01(P.seed, pix, 65 + 2 * k))
        hit, tt = _first_hit(occ, o, _local(t, b, n, l), P.ao_len, dims)
        ao += (torch.where(hit, tt.clamp_max(P.ao_len), torch.full_like(tt, P.ao_len)) / P.ao_len) ** 2
        vis += (~hit).to(F64)
    out["ao"][pix], out["ao_vis"][pix] = ao / P.n_ao, vis / P.n_ao
    sp, sd = torch.zeros_like(ro), torch.zeros_like(ro)
    v = _unit(_f(P.cam_pos) - p)
    for j in range(P.n_spec):
        u1, u2 = _u01(P.seed, pix, 2 * j), _u01(P.seed, pix, 2 * j + 1)
        ct = ((1 - u1) / (1 + (ro ** 4 - 1) * u1)).sqrt()
        sn, ph = (1 - ct * ct).clamp_min(0).sqrt(), 6.2831855 * u2
        h = _local(t, b, n, torch.stack([sn * ph.cos(), sn * ph.sin(), ct], 1))
        hit, tt = _first_hit(occ, o, _unit(2 * (v * h).sum(1, keepdim=True) * h - v), P.spec_len, dims)
        sp += (~hit).to(F64)
        sd += torch.where(hit, tt, torch.full_like(tt, P.spec_len))
    if P.n_spec:
        out["spec"][pix], out["spec_t"][pix] = sp / P.n_spec, sd / P.n_spec
    return out


def _exact_soft(st):
    P, npix, soft = st["params"], st["npix"], st["soft"].to(F64)
    nz, ny, nx, _ = soft.shape
    vox, amax = soft.view(-1, 4), 1.0 - 1.0 / 4096.0
    p, n = st["pos"].view(-1, 3).to(F64), st["nrm"].view(-1, 3).to(F64)
    sc = (p - 0.5 * n).floor().to(torch.int64)
    ok = (n != 0).any(1) & (sc >= 0).all(1) & (sc < torch.tensor([nx, ny, nz], device=DEV)).all(1)
    pix = torch.nonzero(ok).view(-1)
    p, n, sc = p[pix], n[pix], sc[pix]
    surf = sc[:, 0] + nx * (sc[:, 1] + ny * sc[:, 2])
    o, (t, b) = p + n * P.bias, _frame(n)
    ka = P.k_amb / P.n_ao if P.n_ao else 0.0
    light = torch.zeros_like(p)
    paths = []
    for k in range(P.n_shadow + P.n_ao):
        j = k - P.n_shadow
        d = _f(P.light_dir).expand_as(o) if j < 0 else _local(t, b, n, _cosine(_u01(P.seed, pix, 64 + 2 * j), _u01(P.seed, pix, 65 + 2 * j)))
        T, C, cells = torch.ones(len(pix), dtype=F64, device=DEV), torch.zeros_like(p), []

        def visit(ids, cell, m, inside):
            data = inside & (cell < torch.tensor([nx, ny, nz], device=DEV)).all(1)
            r, q = ids[data], cell[data]
            q = q[:, 0] + nx * (q[:, 1] + ny * q[:, 2])
            a = vox[q, 0].clamp(0.0, amax)
            cells.append((r, q, T[r].clone()))
            C[r] += (T[r] * a)[:, None] * vox[q, 1:]
            T[r] *= 1.0 - a
            stop = torch.zeros_like(data)
            stop[data] = T[r] < 2.0 ** -40
            return stop

        _walk(o, d.contiguous(), P.len, (nx, ny, nz), visit)
        light += P.k_sun * T[:, None] if j < 0 else ka * (T[:, None] + C)
        paths.append((j < 0, cells))
    image, lit = torch.zeros((npix, 3), dtype=F64, device=DEV), torch.zeros((npix, 3), dtype=F64, device=DEV)
    image[pix], lit[pix] = vox[surf, 1:] * light, light
    g = (image - st["target"].to(F64)) * (2.0 / image.numel())
    g = g[pix]
    grad = torch.zeros_like(vox)
    grad[:, 1:].index_add_(0, surf, g * light)
    w_all = g * vox[surf, 1:]
    for sun, cells in paths:
        w = w_all * (P.k_sun if sun else ka)
        suf, back = torch.ones(len(pix), dtype=F64, device=DEV), torch.zeros_like(w)
        for r, q, pre in reversed(cells):
            raw, alb = vox[q, 0], vox[q, 1:]
            a = raw.clamp(0.0, amax)
            free = ((raw >= 0) & (raw <= amax)).to(F64)
            da = -w[r].sum(1) * pre * suf[r]
            if not sun:
                da = da + (w[r] * pre[:, None] * (alb - back[r])).sum(1)
                grad[:, 1:].index_add_(0, q, w[r] * (pre * a)[:, None])
                back[r] = a[:, None] * alb + (1 - a)[:, None] * back[r]
            grad[:, 0].index_add_(0, q, da * free)
            suf[r] *= 1 - a
    return {"image": image, "light": lit, "grad": grad.view(nz, ny, nx, 4)}


def _march(occ, dims, o, d, dist, step):
    """Distance of the fixed-step marcher (fine phase to 16, 2^3 blocks after); dist where nothing is met."""
    t = torch.full((o.shape[0],), float(dist), dtype=F64, device=DEV)
    half = torch.tensor([s // 2 for s in dims], device=DEV)
    coarse = torch.zeros([s // 2 for s in reversed(dims)], dtype=torch.bool, device=DEV)
    for b in range(8):
        coarse |= occ[(b >> 2) & 1:dims[2]:2, (b >> 1) & 1:dims[1]:2, b & 1:dims[0]:2]
    ids, pos, at = torch.arange(o.shape[0], device=DEV), o, step
    d = d * step
    for fine in (True, False):
        while at < (16.0 if fine else min(dist, 164.0)) and ids.numel():
            blk = (pos * 0.5).trunc().to(torch.int64) if fine else pos.trunc().to(torch.int64).div(2, rounding_mode="trunc")
            ok = ((blk >= 0) & (blk < half)).all(1)
            q = torch.minimum(blk.clamp_min(0), half - 1)
            if fine:
                q = 2 * q + (pos - 0.5 * (2 * pos).floor() > 0.25)
                ok &= (q < torch.tensor(dims, device=DEV)).all(1)
                q = torch.minimum(q, torch.tensor(dims, device=DEV) - 1)
            h = ok & (occ if fine else coarse)[q[:, 2], q[:, 1], q[:, 0]]
            t[ids[h]] = at
            pos = pos + d
            at += step
            live = torch.nonzero(~h).view(-1)
            ids, pos, d = ids[live], pos[live], d[live]
        step, d = 2 * step, 2 * d
    return t


def _exact_lights(st):
    G = st["grid"]
    occ, dims = _occupancy(G), (G.nx, G.ny, G.nz)
    p, n = st["pos"].view(-1, 3).to(F64), st["nrm"].view(-1, 3).to(F64)
    u = st["noise"].view(-1, 4).to(F64)
    flip = torch.stack([torch.ones_like(u[:, 0])] * 2 + [torch.sign(u[:, 2] - 0.5)], 1)
    l = _cosine(u[:, 0], u[:, 1])
    jit = l * 0.1 * flip
    sun = _unit(torch.tensor([[0.3, 0.4, 0.5]], dtype=F64, device=DEV))
    wd = _unit(0.5 * sun + 0.5 * jit)
    s = (st["depth"].to(F64) / 0.2).clamp(0, 1)
    o = p + wd * u[:, 3:] + jit * 2.5 + n * (s * s * (3 - 2 * s) * 50.0 + 1.5)[:, None]
    shadow = (_march(occ, dims, o, wd, 128.0, 0.5) == 128.0).to(F64)
    t, b = _frame(n)
    dd = _march(occ, dims, o, _local(t, b, n, l), 128.0, 2.5) / 128.0
    rg = (st["rough"].to(F64) * 0.1)[:, None]
    d = (_unit(st["refl"].to(F64)) * (1 - rg) + l * flip * rg) * (1 + 0.5 * u[:, 3:])
    # a sky pixel's reflection has no direction: the pass leaves it at the end of the ray
    d, o = d.nan_to_num(0.0), p + n * u[:, 3:] + n
    return {"shadow": shadow, "irr": dd * dd * 0.05, "refl_t": _march(occ, dims, o, d, 256.0, 0.5), "lit": None, "in_range": None}


def _exact_taa(st):
    c = st["case"]
    W, H = c["W"], c["H"]
    img = {q: st[q].view(H, W, -1).to(F64) for q in ("light", "last", "color", "nrm", "mat", "depth", "motion")}
    every = torch.cat([img[q] for q in ("nrm", "color", "mat", "depth", "motion", "light")], 2)

    def tex(a, u, v):
        x, y = u * W - 0.5, v * H - 0.5
        x0, y0 = x.floor(), y.floor()
        ax, ay = (x - x0)[:, None], (y - y0)[:, None]
        xs = [(x0 + i).clamp(0, W - 1).to(torch.int64) for i in (0, 1)]
        ys = [(y0 + i).clamp(0, H - 1).to(torch.int64) for i in (0, 1)]
        return (a[ys[0], xs[0]] * (1 - ax) + a[ys[0], xs[1]] * ax) * (1 - ay) + (a[ys[1], xs[0]] * (1 - ax) + a[ys[1], xs[1]] * ax) * ay

    def split(q):
        return q[:, :3], q[:, 3:6], q[:, 6:10], q[:, 10], q[:, 11:13], q[:, 13:16]

    i = torch.arange(W * H, device=DEV)
    uv = torch.stack([((i % W) + 0.5) / W, ((i // W) + 0.5) / H], 1).to(F64)
    out = img["light"].view(-1, 4).clone()
    cu, cv = uv.unbind(1)
    mid = tex(every, cu, cv)
    old = uv + mid[:, 11:13]
    # a pixel is sky where the sampled depth is 1 in the pass's own fp32
    d32 = st["depth"].view(H, W)
    size = torch.tensor([[W, H]], dtype=F32, device=DEV).expand(W * H, 2)  # a tensor: torch multiplies by a number's reciprocal
    u32, v32 = (torch.stack([(i % W).to(F32) + 0.5, (i // W).to(F32) + 0.5], 1) / size).unbind(1)
    sky = tex(d32[:, :, None], u32, v32)[:, 0] == 1.0
    off = ((old < 0) | (old > 1)).any(1)

    def factor(me, it, scale):
        n, col, m, de, mo, _ = split(me)
        n2, col2, m2, de2, mo2, li = split(it)
        f = (1.0 - (m - m2).norm(dim=1) >= 0.8).to(F64) * (n * n2).sum(1).clamp_min(0)
        f = f * (1 - ((de - de2).abs() * 4096.0).clamp(0, 1)) * (1 - ((col - col2).norm(dim=1) * scale).clamp(0, 1))
        return torch.where((mo - mo2).norm(dim=1) > 0.1, torch.zeros_like(f), f), li

    # what the last frame did not see: the 19 x 19 neighbours of this one
    s = torch.nonzero(off & ~sky).view(-1)
    acc, count = torch.zeros((len(s), 3), dtype=F64, device=DEV), torch.zeros(len(s), dtype=F64, device=DEV)
    for x in range(-9, 10):
        for y in range(-9, 10):
            f, li = factor(mid[s], tex(every, (cu[s] + x / W).clamp(0.001, 0.999), (cv[s] + y / H).clamp(0.001, 0.999)), 1.0)
            acc, count = acc + f[:, None] * li, count + f
    count = torch.where(count < 1e-4, torch.full_like(count, math.nan), count)  # no neighbour alike: the pass divides by zero
    out[s] = torch.cat([acc / count[:, None], torch.ones_like(f)[:, None]], 1)
    # the rest: a 12-tap spiral, the history clipped to its range
    s = torch.nonzero(~off & ~sky).view(-1)
    me, here, last = mid[s], out[s, :3], tex(img["last"], old[s, 0], old[s, 1])
    hist, var, de = last[:, :3], last[:, 3], me[:, 10]
    scale = torch.minimum(torch.full_like(de, 0.5), 1 / de)
    lo, hi = torch.full_like(hist, 1e4), torch.zeros_like(hist)
    col, count, diff = torch.zeros_like(hist), torch.zeros_like(de), torch.ones_like(de)
    angle, radius = st["noise"].view(-1, 4)[s, 0].to(F64) * 3.1415 * 2.118033988749895, 1.0
    while radius <= 12.0:
        radius += 1.0
        rv = radius * (var + 1) * scale
        f, li = factor(me, tex(every, (cu[s] + angle.cos() / W * rv).clamp(0.001, 0.999), (cv[s] + angle.sin() / H * rv).clamp(0.001, 0.999)), 1e4)
        f = f * (1.212 - radius / 12.0)
        lo, hi = torch.minimum(lo, li), torch.maximum(hi, li)
        col, count, diff = col + f[:, None] * li, count + f, diff + (li - here).norm(dim=1) * f
        angle = angle + 2.39
    here = (here + col) / (count + 1)[:, None]
    hist = torch.minimum(torch.maximum(hist, lo), hi)
    lum = ((here - hist).abs() * torch.tensor([0.2125, 0.7154, 0.0721], dtype=F64, device=DEV)).sum(1)
    var = var + (lum * 5.5).clamp(0, 1) - diff / radius * 0.08 + me[:, 11:13].norm(dim=1) * 20.0
    t = (1 - var).clamp(0.3, 0.9)[:, None]
    out[s] = torch.cat([here * (1 - t) + hist * t, (var * 0.7).clamp(0, 1)[:, None]], 1)
    return out.view(-1)


def exact(case, seed):
    """Ray records, bit masks, grids and command frames are discrete or follow
    the shader's fp32 walk of the mips: no 64-bit value."""
    k = case["kind"]
    if k not in ("occl", "terrain", "batch", "soft", "lights", "taa"):
        return None
    st = prepare(case, seed)
    if k == "batch":
        views = [_exact_occlusion(it) for it in st["items"]]
        return {o: torch.cat([v[o] for v in views]) for o in OUTS}
    if k in ("occl", "terrain"):
        return _exact_occlusion(st)
    if k == "soft":  # laid out as run() returns it
        return _exact_soft(st)
    return _exact_lights(st) if k == "lights" else _exact_taa(st)
