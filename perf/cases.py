"""The work this library's users have it do, as timed cases.

Every case goes through a public entry point: the C-ABI of include/ubr.h with
the frame's buffers in device memory (ubr_render, ubr_render_batch,
ubr_adjoint, the segment queries), or the Python ``render`` call with host
arrays.  Contexts carry the library's default settings.  Scenes are the
seeded synthetic molecules of ``umbreon_gb300.scenes``.
"""
import copy
import ctypes as C
import math

import numpy as np
import torch

from umbreon_gb300 import abi, api, scenes
from umbreon_gb300.api import Context, make_render_desc


def listed():
    return [
        # A small molecule redrawn while it is turned: the smallest call
        # (primary rays and shading only), where launches and latency count.
        dict(name="preview_spheres_640x480", kind="frame", model="spheres", n=2000, w=640, h=480),
        # The figure a user exports: 20k atoms and their bonds, full HD,
        # supersampled, ambient occlusion, two shadowed lights, fog.
        dict(name="figure_ball_and_stick_1920x1080_ss2", kind="frame", model="ball_and_stick", n=20000, w=1920, h=1080,
             ss=2, ao=16),
        # A half-transparent molecular surface over its atoms: triangles,
        # several transparency rounds, many AO rays, an odd frame size.
        dict(name="surface_transparent_1023x769", kind="frame", model="surface", n=1500, w=1023, h=769, ao=32),
        # Quality output of an opaque surface: enhanced AO with its AOVs and
        # the a-trous denoiser that uses them as guides.
        dict(name="surface_aov_denoised_800x600", kind="frame", model="surface", n=800, w=800, h=600, ao=16,
             opaque=True, aov=True, denoise=True),
        # Adaptive antialiasing of the figure at a smaller, ragged size.
        dict(name="adaptive_aa_ball_and_stick_1277x717_ss2", kind="frame", model="ball_and_stick", n=12000, w=1277,
             h=717, ss=2, ao=8, adaptive=True),
        # Path-traced global illumination with every option at its default
        # (integrator 2: gather grid, denoise, upsample, edge patch).
        dict(name="gi_pt2_ball_and_stick_1920x1080_ss2", kind="frame", model="ball_and_stick", n=20000, w=1920, h=1080,
             ss=2, gi=2),
        # The first integrator on the render grid of a small frame, without
        # the filters: the gather itself.
        dict(name="gi_pt1_spheres_640x480", kind="frame", model="spheres", n=2000, w=640, h=480, gi=1, full=True),
        # A turntable movie: many frames of several molecules in one call.
        dict(name="turntable_batch_24_frames", kind="batch", frames=24, models=4, most=200000, big=1024, ao=8),
        # One iteration of fitting a scene to an image: gradients of the
        # sphere frame with enhanced AO, a shadowed light and fog.
        dict(name="adjoint_100k_spheres_1024x1024", kind="adjoint", n=100000, w=1024, h=1024, ao=16, falloff=1.0),
        # Visibility of the edge pass's strokes: a million segments through
        # atoms and bonds, and a mesh query that skips each edge's own faces.
        dict(name="segments_ball_and_stick_1m", kind="segments", model="ball_and_stick", n=20000, segs=1000000),
        dict(name="segments_filtered_surface_200k", kind="segments", model="surface", n=800, segs=200001, filtered=True),
        # The whole Python call at the default frame size, host arrays in and
        # out: flatten, upload, tree build, render, read back.
        dict(name="render_call_host_1024x768", kind="call", n=3000, w=1024, h=768, ao=16),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["frame", "frame", "frame", "frame", "gi", "batch", "adjoint", "segments", "call"])
    if kind == "frame":
        model = rng.choice(["spheres", "ball_and_stick", "surface"])
        if model == "surface":
            c = dict(kind="frame", model=model, n=_log(rng, 100, 1500), w=_log(rng, 150, 1024), h=_log(rng, 150, 1024),
                     ao=rng.choice([4, 8, 16, 32]))
            if rng.random() < 0.5:
                c["opaque"] = True
                if rng.random() < 0.5:
                    c["aov"] = True
                    c["denoise"] = rng.random() < 0.5
        else:
            c = dict(kind="frame", model=model, n=_log(rng, 300, 20000 if model == "ball_and_stick" else 100000),
                     w=_log(rng, 200, 1920), h=_log(rng, 150, 1080), ss=rng.choice([1, 1, 2, 3]),
                     ao=rng.choice([0, 0, 8, 13, 16, 24]))
            if c["ss"] > 1 and rng.random() < 0.3:
                c["adaptive"] = True
        return c
    if kind == "gi":
        full = rng.random() < 0.4
        return dict(kind="frame", model=rng.choice(["spheres", "ball_and_stick"]), n=_log(rng, 300, 20000),
                    w=_log(rng, 160, 960 if full else 1600), h=_log(rng, 120, 540 if full else 900),
                    ss=1 if full else rng.choice([1, 2]), gi=rng.choice([1, 2, 2]), full=full,
                    bounces=rng.choice([1, 1, 2]))
    if kind == "batch":
        return dict(kind="batch", frames=rng.randint(2, 24), models=rng.randint(1, 4), most=_log(rng, 6000, 200000),
                    big=rng.choice([256, 512, 1024]), ao=rng.choice([0, 8]))
    if kind == "adjoint":
        return dict(kind="adjoint", n=_log(rng, 1000, 100000), w=_log(rng, 100, 1024), h=_log(rng, 100, 1024),
                    ao=rng.choice([0, 4, 8, 16]), falloff=rng.choice([0.0, 1.0, 1.0, 2.0]))
    if kind == "segments":
        model = rng.choice(["spheres", "ball_and_stick", "surface"])
        return dict(kind="segments", model=model, n=_log(rng, 300, 1000 if model == "surface" else 20000),
                    segs=_log(rng, 500, 1000000), filtered=model == "surface" and rng.random() < 0.6)
    return dict(kind="call", n=_log(rng, 300, 5000), w=_log(rng, 160, 1024), h=_log(rng, 120, 768),
                ao=rng.choice([0, 8, 16]))


# --- scenes -----------------------------------------------------------------

def _surface_box(n):
    return 60.0 * (n / 10000.0) ** (1.0 / 3.0)


def _scene(case, seed):
    """(Scene, RenderOptions) of a single-frame case."""
    w, h, model = case.get("w", 640), case.get("h", 480), case["model"]
    s = scenes.BASE_SEED + 1009 * (seed + 1)
    if model == "spheres":
        n = case["n"]
        box = 40.0 * (n / 2000.0) ** (1.0 / 3.0)
        sc, opt = scenes.space_filling(seed=s, n=n, width=w, height=h)
        cr, col, mats = scenes.random_spheres(n, box, s)
        sc.sphere_center_radius, sc.sphere_color, sc.sphere_material = cr, col, mats
        sc.camera.position = (0.5 * box, 0.5 * box, 3.0 * box)
        sc.camera.height = 1.2 * box * max(1.0, h / w)
        opt.supersample = case.get("ss", 1)
    elif model == "ball_and_stick":
        sc, opt = scenes.ball_and_stick(seed=s, n=case["n"], width=w, height=h, supersample=case.get("ss", 1))
    else:
        sc, opt = scenes.molecular_surface(seed=s, n_atoms=case["n"], box=_surface_box(case["n"]),
                                           n_spheres=case["n"] // 2, width=w, height=h)
        if case.get("opaque"):
            sc.mesh_colors[:, 3] = 1.0
    if "ao" in case:
        opt.aoSamples = case["ao"]
        opt.shadows = case["ao"] > 0
        opt.aoDistance = min(opt.aoDistance, 6.0)
    if case.get("gi"):
        opt.gi, opt.giIntegrator, opt.aoSamples = True, case["gi"], 0
        opt.shadows = model == "ball_and_stick"
        opt.giBounces = case.get("bounces", 1)
        if case.get("full"):
            opt.pt1GatherDiv, opt.pt1Denoise = 1, False
    if case.get("aov"):
        opt.aoWriteAov, opt.aoFalloffPower = True, 1.0
    if case.get("denoise"):
        opt.denoiser = 1
    if case.get("adaptive"):
        opt.aaMode = 1
    return sc, opt


def _differentiable(case, seed):
    sc, opt = scenes.differentiable(seed=scenes.BASE_SEED + 1009 * (seed + 1), n=case["n"], res=case["w"],
                                    ao_samples=case["ao"])
    opt.height = case["h"]
    opt.aoFalloffPower = case["falloff"]
    sc.camera.height *= max(1.0, case["h"] / case["w"])
    return sc, opt


def _segments(sc, case, seed):
    """Segments between points near the model, as an edge pass asks: from a
    stroke point on or beside the geometry toward the viewer or to another
    point; a filtered query lists each segment's own faces."""
    r = np.random.default_rng(1000 + seed)
    n = case["segs"]
    if sc.mesh_positions is not None:
        tri = np.asarray(sc.mesh_index).reshape(-1, 3)
        f = r.integers(0, len(tri), n)
        p = sc.mesh_positions[tri[f]].mean(1)
        span = sc.mesh_positions.max(0) - sc.mesh_positions.min(0)
    else:
        cr = sc.sphere_center_radius
        f = r.integers(0, len(cr), n)
        d = r.normal(size=(n, 3))
        p = cr[f, :3] + d / np.linalg.norm(d, axis=1, keepdims=True) * (cr[f, 3:] * 1.01)
        span = cr[:, :3].max(0) - cr[:, :3].min(0)
    q = p + np.array([0.0, 0.0, 2.0]) * span.max()
    near = r.random(n) < 0.5
    q[near] = p[near] + r.normal(size=(int(near.sum()), 3)) * 0.1 * span.max()
    segs = np.concatenate([p, q], 1).astype(np.float32)
    k = r.integers(0, 3, n)  # own faces per segment: none, one or two
    offs = np.zeros(n + 1, np.uint32)
    np.cumsum(k, out=offs[1:])
    faces = np.repeat(f, k).astype(np.int32)
    if len(faces) == 0:
        faces = np.zeros(1, np.int32)
    return segs, offs, faces


# --- prepare ----------------------------------------------------------------

_PLANES = (("color", torch.float32, 4), ("depth", torch.float32, 1), ("view_z", torch.float32, 1),
           ("hit_geom", torch.int32, 1), ("hit_prim", torch.int32, 1))


def _device_frame(opt):
    """A ubr_frame with every plane in device memory, and its tensors."""
    frames, out = _device_frames([opt])
    ss = max(1, opt.supersample)
    for name, _, ch in _PLANES:
        size = (opt.height, opt.width, ch) if name == "color" else (opt.height * ss, opt.width * ss)
        out[name] = out[name].view(size)
    fr = frames[0]
    if opt.aoWriteAov:
        for _, name, ch in api.AOV_FIELDS:
            out[name] = torch.empty((opt.height, opt.width, ch), dtype=torch.float32, device="cuda")
            setattr(fr, name, C.cast(C.c_void_p(out[name].data_ptr()), abi.f32p))
    return fr, out


def _device_frames(opts):
    """A ubr_frame per options, the frames' planes of one kind in one device
    allocation (as a movie's frames are kept), and these allocations."""
    frames = []
    for _ in opts:
        frames.append(abi.Frame())
        frames[-1].memory = abi.MEMORY_DEVICE
    out = {}
    for name, dt, ch in _PLANES:
        counts = [o.width * o.height * (ch if name == "color" else max(1, o.supersample) ** 2) for o in opts]
        out[name] = t = torch.empty(sum(counts), dtype=dt, device="cuda")
        at = t.data_ptr()
        for fr, k in zip(frames, counts):
            setattr(fr, name, C.cast(C.c_void_p(at), abi.u32p if dt == torch.int32 else abi.f32p))
            at += 4 * k
    return frames, out


class _State:
    """Holds what a program keeps between calls; closes it in order."""

    def __init__(self, **kw):
        self.__dict__.update(kw)

    def __del__(self):
        for b in self.__dict__.get("built", ()):
            b.release()
        ctx = self.__dict__.get("ctx")
        if ctx is not None:
            ctx.close()


def prepare(case, seed):
    kind = case["kind"]
    if kind == "call":
        sc, opt = scenes.ball_and_stick(seed=scenes.BASE_SEED + 1009 * (seed + 1), n=case["n"], width=case["w"],
                                        height=case["h"], supersample=1, ao_samples=case["ao"])
        return _State(kind=kind, scene=sc, opt=opt)
    ctx = Context(torch.cuda.current_device())
    if kind == "frame":
        sc, opt = _scene(case, seed)
        built = ctx.build(sc)
        desc, keep = make_render_desc(sc, opt)
        fr, out = _device_frame(opt)
        st = _State(kind=kind, ctx=ctx, built=[built], desc=desc, keep=keep, frame=fr, out=out)
    elif kind == "batch":
        sizes = [r for r in (256, 512, 1024) if r <= case["big"]]
        bases, items = scenes.turntable_batch(seed=scenes.BASE_SEED + 1009 * (seed + 1), n_items=case["frames"],
                                              n_scenes=case["models"], ao_samples=case["ao"],
                                              max_spheres=case["most"], min_spheres=5000)
        built = [ctx.build(b) for b in bases]
        arr = (abi.BatchItem * len(items))()
        for i, (_, _, opt) in enumerate(items):  # every size in turn
            opt.width = opt.height = sizes[i % len(sizes)]
        frames, out = _device_frames([opt for _, _, opt in items])
        keep = [frames]
        for i, (si, sc, opt) in enumerate(items):
            desc, k = make_render_desc(sc, opt)
            keep += [desc, k]
            arr[i].scene = built[si].handle
            arr[i].desc = C.pointer(desc)
            arr[i].frame = C.pointer(frames[i])
        st = _State(kind=kind, ctx=ctx, built=built, items=arr, count=len(items), keep=keep, out=out)
    elif kind == "adjoint":
        sc, opt = _differentiable(case, seed)
        target, topt = scenes.differentiable_target(sc, opt, seed=scenes.BASE_SEED + 7 * seed)
        pics = []
        for a, o in ((target, topt), (sc, opt)):
            b = ctx.build(a)
            d, keep = make_render_desc(a, o)
            fr, out = _device_frame(o)
            ctx._check(ctx._L.ubr_render(ctx.handle, b.handle, C.byref(d), C.byref(fr), None, None))
            pics.append(out["color"])
            if a is not sc:
                b.release()
        # dL/d(colour) of the mean squared difference of the two pictures
        dcol = ((pics[1] - pics[0]) * (2.0 / pics[0].numel())).contiguous()
        n = sc.sphere_count()
        out = dict(sphere_color=torch.empty((n, 3), device="cuda"), sphere_center=torch.empty((n, 3), device="cuda"),
                   sphere_radius=torch.empty(n, device="cuda"))
        g = abi.Grads()
        g.memory = abi.MEMORY_DEVICE
        for k, t in out.items():
            setattr(g, k, C.cast(C.c_void_p(t.data_ptr()), abi.f32p))
        st = _State(kind=kind, ctx=ctx, built=[b], desc=d, keep=keep, dcol=dcol, grads=g, out=out)
    else:
        sc, _ = _scene(case, seed)
        built = ctx.build(sc)
        segs, offs, faces = _segments(sc, case, seed)
        n = len(segs)
        dev = [torch.from_numpy(a).cuda() for a in (segs, offs.view(np.int32), faces)]
        out = torch.empty(n, dtype=torch.uint8, device="cuda")
        st = _State(kind=kind, ctx=ctx, built=[built], n=n, segs=dev[0], offs=dev[1], faces=dev[2], out=out,
                    filtered=bool(case.get("filtered")))
    torch.cuda.synchronize()
    return st


# --- one pass ---------------------------------------------------------------

def run(st):
    if st.kind == "call":
        f = api.render(st.scene, st.opt)
        return dict(color=f.color, depth=f.depth, view_z=f.viewZ, hit_geom=f.hit_geom, hit_prim=f.hit_prim)
    ctx, L = st.ctx, st.ctx._L
    if st.kind == "frame":
        ctx._check(L.ubr_render(ctx.handle, st.built[0].handle, C.byref(st.desc), C.byref(st.frame), None, None))
    elif st.kind == "batch":
        ctx._check(L.ubr_render_batch(ctx.handle, st.count, st.items, None))
    elif st.kind == "adjoint":
        g = st.grads
        ctx._check(L.ubr_adjoint(ctx.handle, st.built[0].handle, C.byref(st.desc), C.c_void_p(st.dcol.data_ptr()),
                                 C.byref(g)))
        f32 = lambda a: np.array(list(a), np.float32)
        return dict(st.out, material=f32(g.material), light_direction=f32(g.light_direction[0]),
                    light_color=f32(g.light_color[0]), ambient_color=f32(g.ambient_color),
                    background=f32(g.background), fog_range=f32([g.fog_start, g.fog_end]),
                    fog_color=f32(g.fog_color), ao=f32([g.ao_distance, g.ao_intensity]))
    elif st.filtered:
        ctx._check(L.ubr_occluded_filtered_batch(ctx.handle, st.built[0].handle, st.segs.data_ptr(), st.n, 1e-4, 1e-3,
                                                 0.0, st.offs.data_ptr(), st.faces.data_ptr(), st.out.data_ptr(),
                                                 abi.MEMORY_DEVICE))
    else:
        ctx._check(L.ubr_occluded_batch(ctx.handle, st.built[0].handle, st.segs.data_ptr(), st.n, 1e-4,
                                        st.out.data_ptr(), abi.MEMORY_DEVICE))
    return st.out


# --- what a pass cannot do without --------------------------------------------

# share of a frame's samples whose primary ray meets the model, as rendered
_COVER = {"spheres": 0.58, "ball_and_stick": 0.25, "surface": 0.8}
_BYTES = {"spheres": 36, "ball_and_stick": 36 + 52, "surface": 200 * 24}  # input arrays per atom
_PRIMS = {"spheres": 1, "ball_and_stick": 2, "surface": 200}              # primitives per atom


def _ray_flops(prims):
    """A ray's least work: the boxes of the 8 children on one root-to-leaf
    path (6 multiply-adds each) and one primitive test."""
    return max(1.0, math.log(max(2, prims), 8)) * 8 * 12 + 40


def _frame_work(model, n, w, h, ss, ao, lights, layers=1, gi_rays=0.0):
    hi, out = w * h * ss * ss, w * h
    hits = _COVER[model] * hi * layers
    rays = hi + hits * (ao + (lights if ao else 0)) + gi_rays
    return dict(bytes=int(n * _BYTES[model] + 16 * out + 16 * hi), flops=int(rays * _ray_flops(n * _PRIMS[model]) + hits * 100))


def work(case):
    k = case["kind"]
    if k == "call":
        return _frame_work("ball_and_stick", case["n"], case["w"], case["h"], 1, case["ao"], 2)
    if k == "frame":
        m, ss = case["model"], case.get("ss", 1)
        gi = 0.0
        if case.get("gi"):  # 8 gather rays per covered grid point, one shadow ray per gather hit
            gi = _COVER[m] * case["w"] * case["h"] * 8 * 1.5 * case.get("bounces", 1)
        layers = 2 if m == "surface" and not case.get("opaque") else 1
        w = _frame_work(m, case["n"], case["w"], case["h"], 1 if case.get("adaptive") else ss, case.get("ao", 0), 2,
                        layers, gi)
        if case.get("aov"):
            w["bytes"] += 48 * case["w"] * case["h"]
        return w
    if k == "batch":
        px = sum(r * r for r in (256, 512, 1024) if r <= case["big"]) / sum(1 for r in (256, 512, 1024) if r <= case["big"])
        one = _frame_work("spheres", int(math.sqrt(5000.0 * case["most"])), int(math.sqrt(px)), int(math.sqrt(px)), 1,
                          case["ao"], 2)
        return {a: int(v * case["frames"]) for a, v in one.items()}
    if k == "adjoint":
        px = case["w"] * case["h"]
        one = _frame_work("spheres", case["n"], case["w"], case["h"], 1, case["ao"], 1)
        return dict(bytes=int(16 * px + case["n"] * (36 + 28)), flops=one["flops"] + 300 * px)
    m = case["model"]
    return dict(bytes=int(25 * case["segs"] + case["n"] * _BYTES[m] + (8 * case["segs"] if case.get("filtered") else 0)),
                flops=int(case["segs"] * _ray_flops(case["n"] * _PRIMS[m])))


# --- the same answers in 64 bits ------------------------------------------------

def exact(case, seed):
    """The frame of an unoccluded sphere model (nearest sphere of every pixel,
    the POV finish under one distant light) in float64.  Frames with AO,
    shadow or gather rays take far longer than 20 s by brute force: None."""
    if case["kind"] != "frame" or case["model"] != "spheres" or case.get("gi") or case.get("ao"):
        return None
    ss = case.get("ss", 1)
    if ss != 1 or case.get("adaptive") or case["n"] * case["w"] * case["h"] > 2e10:
        return None
    sc, opt = _scene(case, seed)
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    T = lambda a: torch.as_tensor(np.asarray(a), dtype=torch.float64, device=dev)
    cr, col = T(sc.sphere_center_radius), T(sc.sphere_color)[:, :3]
    cx, cy, cz = sc.camera.position
    W, H = opt.width, opt.height
    half_h = 0.5 * sc.camera.height
    half_w = half_h * W / H
    x = cx + (2.0 * (torch.arange(W, device=dev, dtype=torch.float64) + 0.5) / W - 1.0) * half_w
    y = cy + (1.0 - 2.0 * (torch.arange(H, device=dev, dtype=torch.float64) + 0.5) / H) * half_h
    light = -T(sc.lights[0].direction)
    light = light / light.norm()
    m = sc.sphere_material[0]
    half = light + T([0.0, 0.0, 1.0])
    half = half / half.norm()
    rows = max(1, int(3e7 / (W * len(cr))))
    out = {k: [] for k in ("color", "depth")}
    for r0 in range(0, H, rows):
        yy = y[r0:r0 + rows]
        dx2 = (x[:, None] - cr[None, :, 0]) ** 2
        d2 = (yy[:, None] - cr[None, :, 1]) ** 2
        q = (cr[:, 3] ** 2)[None, None, :] - (d2[:, None, :] + dx2[None, :, :])
        top = torch.where(q >= 0, cr[:, 2] + torch.sqrt(torch.clamp(q, min=0.0)), torch.full_like(q, -1e300))
        z, k = top.max(-1)
        hit = z > -1e299
        p = torch.stack([x[None, :].expand_as(z), yy[:, None].expand_as(z), z], -1)
        n = (p - cr[k, :3]) / cr[k, 3:4]
        ndl, nh = (n * light).sum(-1), (n * half).sum(-1)
        c = col[k]
        amb = float(m["ambient"]) * T(sc.ambientColor)
        rgb = c * amb
        lit = ndl > 0
        li = sc.lights[0].intensity * T(sc.lights[0].color)
        diff = float(m["diffuse"]) * ndl[..., None] * c * li
        spec = float(m["specular"]) * torch.clamp(nh, min=0.0)[..., None] ** (1.0 / float(m["roughness"])) * li
        rgb = rgb + torch.where(lit[..., None], diff + spec, torch.zeros_like(rgb))
        rgb = torch.where(hit[..., None], rgb, T(sc.background).expand_as(rgb))
        out["color"].append(torch.cat([rgb, torch.ones_like(z)[..., None]], -1))
        out["depth"].append(torch.where(hit, cz - z, torch.zeros_like(z)))
    color, depth = torch.cat(out["color"]), torch.cat(out["depth"])
    return dict(color=color, depth=depth, view_z=depth, hit_geom=None, hit_prim=None)
