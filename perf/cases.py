"""The work a user of this framework has it do, as cases to be timed and compared.

Seven kinds of pass, each through the public entry points:

  update      one tick of a probe field (ProbeField.tick) with the dirty lanes a moving
              scene needs, and its atlases read back to page-locked memory, as a host
              program that owns the renderer's textures does every frame;
  facade      installSpeedballGI(...).update() with the facade's defaults: two cascades,
              the ray budget's partial updates, both cascades' atlases read back;
  batch       one frame of several fields as a replayed CUDA graph (GraphFrame);
  adjoint     one gradient: GIAdjoint.forward and backward;
  gather      the receiver gather over a G-buffer (sb_gather_irradiance);
  reflect     the combined receiver with the reflection lobes (sb_gather_reflections);
  rays        a path tracer's bounce: closest hits and shadow queries on device arrays
              (sb_raycast_device, sb_occluded_device);
  build       BLAS builds of resident meshes (sb_build_blas_device).

listed() holds one representative of each range, draw() any other. Sizes come from the
repository's scenes (speedball_b200.synth) and benchmark; scenes, inputs and frames are
functions of the seed. Passes are only enqueued where the entry points allow it, all on
one stream, as one renderer's frames are.
"""
from __future__ import annotations

import ctypes as C
import math

import numpy as np
import torch

from speedball_b200 import _abi, synth
from speedball_b200.adjoint import GIAdjoint
from speedball_b200.batch import BatchedFrame, GraphFrame, Lane
from speedball_b200.field import ProbeField, installSpeedballGI

ATRIUM = synth.ATRIUM_TRIS
FRAMES = 4  # distinct motion frames a state cycles through


# ------------------------------------------------------------------ the cases
def listed():
    return [
        # the smallest field: 512 probes x 64 rays in the 82k-triangle room, nothing moving;
        # launches and latency count
        dict(name="room_update", kind="update", scene="room", tris=81932, res=8, rays=64, jitter="gated",
             reflection="off", emitters=False, motion=False),
        # every option of the update at once: both reflection lobes on every texel, a sphere
        # and two point emitters, a new ray basis each solve
        dict(name="room_ultra_emitters", kind="update", scene="room", tris=81932, res=13, rays=96,
             jitter="montecarlo", reflection="ultra", emitters=True, motion=False),
        # the headline workload: Sponza-scale atrium, 33 clustered lights, 3 movers and one
        # deforming mesh every frame, 4,096 probes x 64 rays
        dict(name="atrium_frame", kind="update", scene="atrium", tris=ATRIUM, res=16, rays=64, jitter="gated",
             reflection="off", emitters=False, motion=True),
        # the largest batch scene at the highest of its ray counts
        dict(name="atrium_500k_128rays", kind="update", scene="atrium", tris=500_000, res=16, rays=128,
             jitter="montecarlo", reflection="off", emitters=False, motion=True),
        # what a program that keeps every default gets: two cascades in turn, 1,536 probes a tick
        dict(name="atrium_facade_defaults", kind="facade", tris=ATRIUM, divisions=16, rays=64, motion=True),
        # several small fields a frame, refit lanes and solves in one graph
        dict(name="batch_4_fields", kind="batch", tris=120_000, fields=4, res=11, rays=80),
        # the differentiated workload: 416 parameters, two feedback solves
        dict(name="adjoint_room", kind="adjoint", res=8, rays=64, materials=64, lights=32, solves=2),
        # the default receiver on a full-HD G-buffer
        dict(name="gather_1080p", kind="gather", width=1920, height=1080, res=16, cascades=1, cheby=0.0, dual=False),
        # the receiver with visibility weights inside a fine cascade, an odd screen size
        dict(name="gather_cheby_cascades_1366", kind="gather", width=1366, height=768, res=16, cascades=2, cheby=1.0,
             dual=False),
        # irradiance and reflection layer of a full-HD G-buffer
        dict(name="reflect_high_1080p", kind="reflect", width=1920, height=1080, res=12, tier="high", cheby=0.0),
        # a diffuse bounce of a full-HD path tracer with one shadow ray per vertex
        dict(name="rays_bounce_1080p", kind="rays", tris=ATRIUM, width=1920, height=1080, bounce=True),
        # every mesh of the atrium built where it lies
        dict(name="build_atrium_meshes", kind="build", tris=ATRIUM, meshes=30),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _screen(rng):
    w = _log(rng, 61, 1920)
    return w, max(1, min(1080, int(w * rng.uniform(0.4, 0.7))))


def draw(rng):
    kind = rng.choice(["update", "update", "update", "facade", "batch", "adjoint", "gather", "gather", "reflect",
                       "rays", "build", "build"])
    rays = rng.randrange(32, 129, 16)
    if kind == "update":
        room = rng.random() < 0.4
        return dict(kind=kind, scene="room" if room else "atrium", tris=81932 if room else _log(rng, 20_000, 500_000),
                    res=rng.randint(2, 16), rays=rays, jitter=rng.choice(["gated", "montecarlo"]),
                    reflection=rng.choice(["off", "off", "rough", "high", "ultra"]),
                    emitters=room and rng.random() < 0.5, motion=not room and rng.random() < 0.7)
    if kind == "facade":
        return dict(kind=kind, tris=_log(rng, 20_000, 500_000), divisions=rng.randint(6, 24), rays=rays,
                    motion=rng.random() < 0.5)
    if kind == "batch":
        return dict(kind=kind, tris=_log(rng, 20_000, 200_000), fields=rng.randint(2, 4), res=rng.randint(4, 12),
                    rays=rays)
    if kind == "adjoint":
        return dict(kind=kind, res=rng.randint(3, 10), rays=rays, materials=rng.randint(4, 64),
                    lights=rng.randint(1, 32), solves=rng.randint(1, 3))
    if kind == "gather":
        w, h = _screen(rng)
        cascades = rng.randint(1, 2)
        return dict(kind=kind, width=w, height=h, res=rng.randint(2, 24), cascades=cascades,
                    cheby=rng.choice([0.0, 0.0, 0.6, 1.0]), dual=cascades == 1 and rng.random() < 0.3)
    if kind == "reflect":
        w, h = _screen(rng)
        return dict(kind=kind, width=w, height=h, res=rng.randint(4, 14), tier=rng.choice(["rough", "high", "ultra"]),
                    cheby=rng.choice([0.0, 1.0]))
    if kind == "rays":
        w, h = _screen(rng)
        return dict(kind=kind, tris=_log(rng, 20_000, 500_000), width=w, height=h, bounce=rng.random() < 0.6)
    return dict(kind=kind, tris=_log(rng, 300, 600_000), meshes=rng.choice([1, 1, rng.randint(2, 30)]))


# ------------------------------------------------------------------ preparing
_stream_of_frames = None


def _stream():
    """The one stream every state's work runs on."""
    global _stream_of_frames
    if _stream_of_frames is None:
        _stream_of_frames = torch.cuda.Stream()
    return _stream_of_frames


def _on_stream(field):
    field.synchronize()
    _abi.check(field._lib.sb_set_stream(field.ctx, C.c_void_p(_stream().cuda_stream)), field.ctx)


def _atrium(seed, tris, res=None, rays=64):
    scene = synth.atrium(seed=seed % 100_003, total_tris=max(20_000, tris))
    if res:
        scene.meta["grid"] = dict(scene.meta["grid"], res=(res,) * 3, rays=rays)
    return scene


def _field(scene, rays, jitter="gated", reflection="off", clustered=True):
    """A field whose tick updates every probe, over the scene's own grid."""
    g = scene.meta["grid"]
    f = ProbeField(scene, volumes=dict(gridMin=g["gridMin"], gridSize=g["gridSize"], res=g["res"]), cascades=1,
                   rays=rays, clusteredLighting=clustered, hysteresis=scene.meta["hysteresis"], jitterMode=jitter,
                   reflectionQuality=reflection)
    f.setHysteresisNormalization(False)
    f.setRayBudget(1 << 24, maxProbesPerTick=1 << 20)
    return f


def _readable(field, cascades=1, room=0):
    """(buffer id, values, page-locked tensor) of every atlas a renderer takes from the field;
    `room`: values of a staging buffer that holds any fitted grid's atlas."""
    out = []
    for ci in range(cascades):
        g = field.cascadeGrid(ci)
        n = int(g.res[0] * g.res[1] * g.res[2]) * 64 * 4
        names = ["IRRADIANCE_ATLAS", "DEPTH_ATLAS"]
        if field.getReflectionQuality() != "off":
            names.append("ROUGH_ATLAS")
        sizes = [n] * len(names)
        lay = field.reflectionLayout(ci)
        if lay["glossyAtlasW"]:
            names.append("GLOSSY_ATLAS")
            sizes.append(lay["glossyAtlasW"] * lay["glossyAtlasH"] * 4)
        # the atlases' texels are binary16
        out += [(_abi.BUF[k] | (ci << 8), s, torch.zeros(max(s, room), dtype=torch.float16, pin_memory=True))
                for k, s in zip(names, sizes)]
    return out


def _read(field, readable):
    """Queues the reads behind the field's work."""
    for which, n, a in readable:
        _abi.check(field._lib.sb_read_buffer_async(field.ctx, which, 0, n, _dev(a)), field.ctx)
    return [a for _, _, a in readable]


def _motion(scene, seed):
    return [synth.atrium_motion(scene, seed % 1009 + k) for k in range(FRAMES)]


def _move(state):
    """The next motion frame into the scene, and its dirty marks."""
    mats, pos = state["frames"][state["at"] % FRAMES]
    state["at"] += 1
    scene, gi = state["scene"], state["gi"]
    scene.meshes[scene.meta["deformer"]].positions = pos
    for i, m in mats.items():
        scene.instances[i].world = m
    gi.markDeformsDirty()
    gi.markTransformsDirty(list(mats))


def _prepare_update(c, seed):
    if c["scene"] == "room":
        scene = synth.room_spheres(seed % 100_003)
        if c["emitters"]:
            scene = synth.add_emitters(scene, seed=seed % 9973)
        scene.meta["grid"] = dict(scene.meta["grid"], res=(c["res"],) * 3)
    else:
        scene = _atrium(seed, c["tris"], c["res"])
    f = _field(scene, c["rays"], c["jitter"], c["reflection"], clustered=c["scene"] != "room")
    _on_stream(f)
    s = dict(scene=scene, gi=f, field=f, at=0, frames=_motion(scene, seed) if c["motion"] else None)
    return _warm(s, 1)


def _prepare_facade(c, seed):
    scene = _atrium(seed, c["tris"])

    def failed(e):
        raise e
    gi = installSpeedballGI(scene, divisions=c["divisions"], rays=c["rays"], onError=failed)
    f = gi.advanced["field"]
    _on_stream(f)
    s = dict(scene=scene, gi=gi, field=f, at=0, frames=_motion(scene, seed) if c["motion"] else None)
    # C0 has at most divisions + 1 probes an axis, C1 at most twice C0's
    return _warm(s, 2 if f.hasFineCascade() else 1, 2 * (c["divisions"] + 1) ** 3 * 64 * 4)


def _warm(s, cascades, room=0):
    """A field that is up: its trees are built and it has been updated."""
    s["read"] = _readable(s["field"], cascades, room)
    for _ in range(2):
        _tick(s)
    s["field"].synchronize()
    return s


def _tick(s):
    if s["frames"]:
        _move(s)
    if s["gi"] is s["field"]:
        s["field"].tick()
    else:
        s["gi"].update()
    return _read(s["field"], s["read"])


def _prepare_batch(c, seed):
    scenes = [_atrium(seed + 31 * k, int(c["tris"] * (0.4 + 0.4 * k)), max(2, c["res"] - k), c["rays"])
              for k in range(c["fields"])]
    fields = [_field(s, c["rays"], "montecarlo") for s in scenes]
    for f in fields:
        _on_stream(f)
    lanes = []
    for s, f in zip(scenes, fields):
        d = s.meta["deformer"]
        lanes.append(Lane(f, [(int(f.pool.blas_root[d]), int(f.pool.blas_end[d]))]))
    s = dict(fields=fields, graph=GraphFrame(BatchedFrame(fields), lanes), read=[_readable(f) for f in fields])
    for _ in range(2):
        _batch(s)
    fields[0].synchronize()
    return s


def _batch(s):
    s["graph"].tick()
    return [_read(f, r) for f, r in zip(s["fields"], s["read"])]


def _prepare_adjoint(c, seed):
    scene = synth.room_spheres(seed % 100_003, n_materials=c["materials"], n_point=c["lights"], n_dir=0)
    scene.meta["grid"] = dict(scene.meta["grid"], res=(c["res"],) * 3)
    f = _field(scene, c["rays"], clustered=False)
    _on_stream(f)
    adj = GIAdjoint(f, solves=c["solves"])
    rng = np.random.default_rng(seed)
    base = adj.parameters()
    adj.setParameters(albedo=base["albedo"] * rng.uniform(0.8, 1.2, base["albedo"].shape),
                      lightScale=rng.uniform(0.5, 2.0, c["lights"]))
    target = adj.forward()
    adj.setParameters(albedo=base["albedo"], lightScale=np.ones(c["lights"]))
    return dict(field=f, adj=adj, target=target)


def _run_adjoint(s):
    loss = s["adj"].forward(s["target"])
    grads = s["adj"].backward()
    return dict(loss=np.float32(loss), irradiance=s["adj"].readE(), **grads)


def _gbuffer(c, seed, box_min, box_size):
    """A pinhole camera's G-buffer of a box interior with spheres in it: positions, normals,
    normal-mapped normals, the camera's mirror direction with a roughness; float4 rows."""
    dev = "cuda"
    g = torch.Generator(device=dev).manual_seed(seed)
    w, h = c["width"], c["height"]
    lo = torch.tensor(box_min, device=dev, dtype=torch.float64)
    size = torch.tensor(box_size, device=dev, dtype=torch.float64)
    hi = lo + size
    cam = lo + size * (0.3 + 0.4 * torch.rand(3, generator=g, device=dev, dtype=torch.float64))
    x = (torch.arange(w, device=dev, dtype=torch.float64) + 0.5) / w * 2 - 1
    y = ((torch.arange(h, device=dev, dtype=torch.float64) + 0.5) / h * 2 - 1) * h / w
    Y, X = torch.meshgrid(y, x, indexing="ij")
    d = torch.stack([torch.ones_like(X), -Y, X], -1).reshape(-1, 3)
    turn = float(torch.rand(1, generator=g, device=dev)) * 2 * math.pi
    d = torch.stack([d[:, 0] * math.cos(turn) - d[:, 2] * math.sin(turn), d[:, 1],
                     d[:, 0] * math.sin(turn) + d[:, 2] * math.cos(turn)], -1)
    d = d / d.norm(dim=1, keepdim=True)
    to = torch.where(d > 0, hi, lo)
    ta = (to - cam) / torch.where(d.abs() < 1e-9, torch.full_like(d, 1e-9), d)
    t, axis = ta.min(dim=1)
    n = torch.zeros_like(d)
    n.scatter_(1, axis[:, None], -torch.sign(d.gather(1, axis[:, None])))
    centres = lo + size * torch.rand(12, 3, generator=g, device=dev, dtype=torch.float64)
    radii = float(size.min()) * (0.03 + 0.1 * torch.rand(12, generator=g, device=dev, dtype=torch.float64))
    for k in range(12):
        oc = cam - centres[k]
        b = d @ oc
        disc = b * b - (oc @ oc - radii[k] ** 2)
        ts = -b - disc.clamp_min(0).sqrt()
        hit = (disc > 0) & (ts > 1e-3) & (ts < t)
        t = torch.where(hit, ts, t)
        ns = (cam + d * ts[:, None] - centres[k]) / radii[k]
        n = torch.where(hit[:, None], ns, n)
    p = cam + d * t[:, None]
    det = n + 0.15 * torch.randn(n.shape, generator=g, device=dev, dtype=torch.float64)
    det = det / det.norm(dim=1, keepdim=True)
    r = d - 2 * (d * n).sum(1, keepdim=True) * n
    rough = torch.rand(p.shape[0], 1, generator=g, device=dev, dtype=torch.float64)
    zero = torch.zeros(p.shape[0], 1, device=dev, dtype=torch.float64)
    return [torch.cat(v, 1).float().contiguous() for v in ((p, zero), (n, zero), (det, zero), (r, rough))]


def _gutter():
    """The texel of a 6 x 6 octahedral tile that each texel of the 8 x 8 tile mirrors."""
    src = np.zeros((8, 8, 2), np.int64)
    for y in range(8):
        for x in range(8):
            ex, ey = x in (0, 7), y in (0, 7)
            if ex and ey:
                sx, sy = (6 if x == 0 else 1), (6 if y == 0 else 1)
            elif ey:
                sx, sy = 7 - x, (1 if y == 0 else 6)
            elif ex:
                sx, sy = (1 if x == 0 else 6), 7 - y
            else:
                sx, sy = x, y
            src[y, x] = sy - 1, sx - 1
    return src


def _atlases(seed, res, cell):
    """Irradiance and depth-moment atlases of a res^3 field: smooth over directions, every
    probe its own, binary16 RGBA tiles with the mirrored gutter."""
    rng = np.random.default_rng(seed)
    P = res ** 3
    u = (np.arange(6) + 0.5) / 6 * 2 - 1
    fx, fy = np.meshgrid(u, u)
    z = 1 - np.abs(fx) - np.abs(fy)
    t = np.maximum(-z, 0)
    d = np.stack([fx + np.where(fx >= 0, -t, t), fy + np.where(fy >= 0, -t, t), z], -1)
    d /= np.linalg.norm(d, axis=-1, keepdims=True)
    a = rng.uniform(0.1, 3.0, (P, 1, 1, 3))
    b = rng.uniform(-0.3, 0.3, (P, 3, 3))
    e = a * (1 + np.einsum("pck,yxk->pyxc", b, d)) * rng.uniform(0.9, 1.1, (P, 6, 6, 1))
    m = cell * rng.uniform(0.2, 2.5, (P, 1, 1)) * rng.uniform(0.8, 1.2, (P, 6, 6))
    m2 = m * m * rng.uniform(1.0, 1.3, (P, 6, 6))
    one, zero = np.ones((P, 6, 6)), np.zeros((P, 6, 6))
    g = _gutter()
    out = []
    for tile in (np.concatenate([e, one[..., None]], -1), np.stack([m, m2, zero, one], -1)):
        full = tile[:, g[..., 0], g[..., 1]]  # P, 8, 8, 4
        atlas = full.reshape(res, res, res, 8, 8, 4).transpose(0, 1, 3, 2, 4, 5).reshape(res * res * 8, res * 8, 4)
        out.append(np.ascontiguousarray(atlas.astype(np.float16)))
    return out


GATHER_BOXES = (((0.5, 0.5, 0.5), (9.0, 9.0, 9.0)), ((2.5, 2.0, 2.25), (4.5, 5.0, 4.75)))  # field, fine cascade


def _gather_inputs(c, seed):
    boxes = GATHER_BOXES[:c["cascades"]]
    atlases = [_atlases(seed * 2 + k, c["res"], min(size) / max(1, c["res"] - 1)) for k, (_, size) in enumerate(boxes)]
    return atlases, _gbuffer(c, seed, *GATHER_BOXES[0])


def _gather_params(c, cell_min):
    lib = _abi.load()
    prm = _abi.sb_gather_params()
    lib.sb_gather_params_defaults(C.byref(prm))
    prm.normalBias[0] = max(1e-4, cell_min * 0.04)
    prm.chebyStrength = c["cheby"]
    prm.cascades = c.get("cascades", 1)
    if c.get("dual"):
        prm.dualDetail, prm.detailStrength = 1, 0.7
    return prm


def _small_room(res, seed, tier="off", rays=32):
    scene = synth.room_spheres(seed % 100_003)
    scene.meta["grid"] = dict(scene.meta["grid"], gridMin=GATHER_BOXES[0][0], gridSize=GATHER_BOXES[0][1],
                              res=(res,) * 3)
    f = _field(scene, rays, reflection=tier, clustered=False)
    _on_stream(f)
    return f


def _dev(t):
    """A tensor's memory, on either side."""
    return C.c_void_p(t.data_ptr())


def _prepare_gather(c, seed):
    atlases, gbuf = _gather_inputs(c, seed)
    f = _small_room(c["res"], seed)
    if c["cascades"] == 2:
        f.configureCascade(1, *GATHER_BOXES[1], (c["res"],) * 3)
    for ci, pair in enumerate(atlases):
        for key, a in zip(("IRRADIANCE_ATLAS", "DEPTH_ATLAS"), pair):
            _abi.check(f._lib.sb_upload_range(f.ctx, _abi.BUF[key] | (ci << 8), 0, a.size, _abi.ptr(a)), f.ctx)
    f.synchronize()
    n = gbuf[0].shape[0]
    return dict(field=f, prm=_gather_params(c, f.grid.cellMin), gbuf=gbuf[:3], n=n,
                out=torch.zeros(n, 4, device="cuda"))


def _run_gather(s):
    f, g = s["field"], s["gbuf"]
    _abi.check(f._lib.sb_gather_irradiance(f.ctx, C.byref(s["prm"]), _dev(g[0]), _dev(g[1]), _dev(g[2]), s["n"],
                                           _dev(s["out"])), f.ctx)
    return s["out"]


def _prepare_reflect(c, seed):
    f = _small_room(c["res"], seed, c["tier"], rays=64)
    for _ in range(2):
        f.tick()
    f.synchronize()
    gbuf = _gbuffer(c, seed, *GATHER_BOXES[0])
    n = gbuf[0].shape[0]
    return dict(field=f, prm=_gather_params(c, f.grid.cellMin), gbuf=gbuf, n=n, out=torch.zeros(n, 4, device="cuda"),
                refl=torch.zeros(n, 4, device="cuda"))


def _run_reflect(s):
    f, g = s["field"], s["gbuf"]
    _abi.check(f._lib.sb_gather_reflections(f.ctx, C.byref(s["prm"]), *[_dev(t) for t in g], s["n"], _dev(s["out"]),
                                            _dev(s["refl"])), f.ctx)
    return dict(irradiance=s["out"], reflection=s["refl"])


def _raycast(s):
    f = s["field"]
    _abi.check(f._lib.sb_raycast_device(f.ctx, _dev(s["ro"]), _dev(s["rd"]), s["n"], _dev(s["t"]), _dev(s["tri"]),
                                        _dev(s["inst"])), f.ctx)


def _prepare_rays(c, seed):
    """Camera rays of a pinhole camera in the atrium, or the cosine-distributed bounce off
    what they hit; shadow rays from the same points toward a point light each."""
    scene = _atrium(seed, c["tris"], 8)
    f = _field(scene, 32)
    _on_stream(f)
    f.tick()
    f.synchronize()
    dev = "cuda"
    gen = torch.Generator(device=dev).manual_seed(seed)
    g = scene.meta["grid"]
    lo, size = (torch.tensor(v, device=dev, dtype=torch.float32) for v in (g["gridMin"], g["gridSize"]))
    cam = lo + size * (0.35 + 0.3 * torch.rand(3, generator=gen, device=dev))
    w, h = c["width"], c["height"]
    x = (torch.arange(w, device=dev) + 0.5) / w * 2 - 1
    y = ((torch.arange(h, device=dev) + 0.5) / h * 2 - 1) * h / w
    Y, X = torch.meshgrid(y, x, indexing="ij")
    rd = torch.stack([torch.ones_like(X), -Y, X], -1).reshape(-1, 3)
    rd = (rd / rd.norm(dim=1, keepdim=True)).contiguous()
    n = rd.shape[0]
    s = dict(field=f, n=n, ro=cam.expand(n, 3).contiguous(), rd=rd, t=torch.zeros(n, device=dev),
             tri=torch.zeros(n, device=dev, dtype=torch.int32), inst=torch.zeros(n, device=dev, dtype=torch.int32),
             blocked=torch.zeros(n, device=dev, dtype=torch.uint8))
    torch.cuda.synchronize()
    _raycast(s)
    torch.cuda.synchronize()
    hit = s["tri"] >= 0
    p = torch.where(hit[:, None], s["ro"] + s["rd"] * (s["t"] * 0.999)[:, None],
                    lo + size * torch.rand(n, 3, generator=gen, device=dev))
    if c["bounce"]:
        # a hemisphere about the reversed view ray stands in for the surface normal's
        v = torch.randn(n, 3, generator=gen, device=dev)
        v = v / v.norm(dim=1, keepdim=True) - s["rd"]
        s["ro"], s["rd"] = p.contiguous(), (v / v.norm(dim=1, keepdim=True).clamp_min(1e-6)).contiguous()
    lights = torch.tensor(np.asarray(scene.lights)[1:, 1:4], device=dev, dtype=torch.float32)
    to = lights[torch.randint(lights.shape[0], (n,), generator=gen, device=dev)] - p
    dist = to.norm(dim=1).clamp_min(1e-3)
    s.update(so=p.contiguous(), sd=(to / dist[:, None]).contiguous(), dist=dist.contiguous())
    torch.cuda.synchronize()
    return s


def _run_rays(s):
    _raycast(s)
    f = s["field"]
    _abi.check(f._lib.sb_occluded_device(f.ctx, _dev(s["so"]), _dev(s["sd"]), _dev(s["dist"]), s["n"],
                                         _dev(s["blocked"])), f.ctx)
    return dict(t=s["t"], tri=s["tri"], inst=s["inst"], blocked=s["blocked"])


class _Context:
    """A bare context: BLAS builds need no field."""

    def __init__(self):
        self.lib, self.ctx = _abi.load(), C.c_void_p()
        _abi.check(self.lib.sb_create(C.byref(_abi.sb_device_opts(0, 0)), C.byref(self.ctx)))
        _abi.check(self.lib.sb_set_stream(self.ctx, C.c_void_p(_stream().cuda_stream)), self.ctx)

    def __del__(self):
        try:
            self.lib.sb_destroy(self.ctx)
        except Exception:
            pass


def _prepare_build(c, seed):
    rng = np.random.default_rng(seed)
    if c["meshes"] == 1:
        make = (synth.column_prism, synth.arched_panel, synth.floor_slab)[seed % 3]
        meshes = [make(c["tris"], rng)]
    else:
        # the scene's mesh sizes, the same for every seed
        raw = np.exp(np.random.default_rng(c["meshes"]).uniform(math.log(500), math.log(60_000), c["meshes"]))
        counts = np.maximum(2, np.round(raw * c["tris"] / raw.sum())).astype(int)
        meshes = [(synth.column_prism, synth.arched_panel, synth.floor_slab)[k % 3](int(n), rng)
                  for k, n in enumerate(counts)]
    # the pool the trees are built into: one array each, a slice per mesh
    T = [int(idx.shape[0]) for _, idx in meshes]
    at = np.concatenate([[0], np.cumsum(T)])
    nodes = torch.zeros(2 * int(at[-1]), 8, dtype=torch.int32, device="cuda")
    order = torch.zeros(int(at[-1]), dtype=torch.int32, device="cuda")
    count = torch.zeros(len(meshes), dtype=torch.int32, device="cuda")
    dev = [(torch.from_numpy(np.ascontiguousarray(pos, np.float32)).cuda(),
            torch.from_numpy(np.ascontiguousarray(idx).astype(np.int32)).cuda(), T[k],
            nodes[2 * at[k]:2 * at[k + 1]], order[at[k]:at[k + 1]], count[k:k + 1])
           for k, (pos, idx) in enumerate(meshes)]
    return dict(ctx=_Context(), meshes=dev, nodes=nodes, order=order, count=count)


def _run_build(s):
    lib, ctx = s["ctx"].lib, s["ctx"].ctx
    for pos, idx, tris, nodes, order, count in s["meshes"]:
        _abi.check(lib.sb_build_blas_device(ctx, _dev(pos), pos.shape[0], _dev(idx), tris, 8, _dev(nodes),
                                            _dev(order), _dev(count)), ctx)
    return dict(nodes=s["nodes"], order=s["order"], count=s["count"])


PREPARE = dict(update=_prepare_update, facade=_prepare_facade, batch=_prepare_batch, adjoint=_prepare_adjoint,
               gather=_prepare_gather, reflect=_prepare_reflect, rays=_prepare_rays, build=_prepare_build)
RUN = dict(update=_tick, facade=_tick, batch=_batch, adjoint=_run_adjoint, gather=_run_gather, reflect=_run_reflect,
           rays=_run_rays, build=_run_build)


def prepare(case, seed):
    state = PREPARE[case["kind"]](case, int(seed))
    torch.cuda.synchronize()
    state["kind"] = case["kind"]
    return state


def run(state):
    return RUN[state["kind"]](state)


# ------------------------------------------------------------------ the least work
RAY_FLOPS = 7 * 8 * 20 + 2 * 45     # an 8-wide walk: 7 nodes of 8 box tests, 2 triangle tests
SHADOW_FLOPS = 12 * 2 * 20 + 45     # an any-hit walk


def _update_work(probes, rays, tris, lights, glossy=0, rough=False):
    n = probes * rays
    shade = 400 * n                                     # frame, gates, one-bounce read of 8 taps
    blend = n * 36 * 2 * (9 + (4 if rough else 0)) + n * glossy * 10
    flops = n * RAY_FLOPS + n * lights * SHADOW_FLOPS + shade + blend
    bytes_ = tris * 48 + probes * (36 * 24 * 2 + 64 * 24 + (64 * 40 if rough else 0) + glossy * 48)
    return dict(bytes=bytes_, flops=flops)


def work(case):
    k = case["kind"]
    if k == "update":
        glossy = {"high": 50, "ultra": 324}.get(case["reflection"], 0)
        return _update_work(case["res"] ** 3, case["rays"], case["tris"], 3 if case["scene"] == "room" else 1.6,
                            glossy, case["reflection"] != "off")
    if k == "facade":
        return _update_work(98_304 // case["rays"], case["rays"], case["tris"], 1.6)
    if k == "batch":
        w = [_update_work(max(2, case["res"] - i) ** 3, case["rays"], int(case["tris"] * (0.4 + 0.4 * i)), 1.6)
             for i in range(case["fields"])]
        return dict(bytes=sum(x["bytes"] for x in w), flops=sum(x["flops"] for x in w))
    if k == "adjoint":
        w = _update_work(case["res"] ** 3, case["rays"], 81932, 0.5 * case["lights"])
        # the reverse pass re-shades each ray and undoes the blend and the shading
        back = case["res"] ** 3 * case["rays"] * (400 * 3 + 36 * 2 * 16)
        return dict(bytes=2 * case["solves"] * w["bytes"], flops=case["solves"] * (w["flops"] + back))
    if k in ("gather", "reflect"):
        n = case["width"] * case["height"]
        casc = case.get("cascades", 1)
        taps = 8 * (1 + (case["cheby"] > 0)) + (8 * 3 if k == "reflect" else 0) + (8 if case.get("dual") else 0)
        return dict(bytes=n * (64 if k == "gather" else 96) + casc * case["res"] ** 3 * 1024,
                    flops=n * casc * (100 + taps * 40))
    if k == "rays":
        n = case["width"] * case["height"]
        return dict(bytes=n * (24 + 12 + 28 + 1) + case["tris"] * 48, flops=n * (RAY_FLOPS + SHADOW_FLOPS))
    return dict(bytes=case["tris"] * (12 + 6 + 4 + 10), flops=case["tris"] * 300)


# ------------------------------------------------------------------ in 64 bits
def _oct(n):
    n = n / n.abs().sum(1, keepdim=True).clamp_min(1e-20)
    f = (1 - n[:, [1, 0]].abs()) * torch.where(n[:, :2] >= 0, 1.0, -1.0)
    return torch.where(n[:, 2:] < 0, f, n[:, :2]) * 0.5 + 0.5


def _fetch(atlas, tile_y, tile_x, uv):
    """Bilinear, inside an 8 x 8 tile with its 6 x 6 interior."""
    x, y = tile_x * 8 + 0.5 + uv[:, 0] * 6, tile_y * 8 + 0.5 + uv[:, 1] * 6
    x0, y0 = x.floor(), y.floor()
    fx, fy = (x - x0)[:, None], (y - y0)[:, None]
    x0, y0 = x0.long(), y0.long()
    return (atlas[y0, x0] * (1 - fx) + atlas[y0, x0 + 1] * fx) * (1 - fy) + \
           (atlas[y0 + 1, x0] * (1 - fx) + atlas[y0 + 1, x0 + 1] * fx) * fy


def _exact_cascade(c, box, atlases, cage, P, Nvis, Ndir, dual):
    f64 = dict(device=P.device, dtype=torch.float64)
    res = c["res"]
    lo, size = (torch.tensor(np.float32(v), **f64) for v in box)
    rm1 = max(res - 1, 1)
    gf = (cage - lo) / (size / rm1)
    base = gf.floor().clamp(0, max(res - 2, 0))
    frac = (gf - base).clamp(0, 1)
    Nn = Nvis / Nvis.norm(dim=1, keepdim=True)
    oN, oS = _oct(Ndir / Ndir.norm(dim=1, keepdim=True)), _oct(Nn)
    irr, dep = (torch.tensor(a.astype(np.float64), **f64) for a in atlases)
    cs = float(np.float32(c["cheby"]))
    acc, wsum = torch.zeros(P.shape[0], 3, **f64), torch.zeros(P.shape[0], **f64)
    for i in range(8):
        d = torch.tensor([i & 1, (i >> 1) & 1, (i >> 2) & 1], **f64)
        p = base + d
        w = torch.where(d > 0, frac, 1 - frac).prod(1) + 1e-4
        ty, tx = p[:, 2] * res + p[:, 1], p[:, 0]
        if cs:
            pos = lo + p / rm1 * size
            to = P - pos
            dist = to.norm(dim=1)
            inv = 1 / dist.clamp_min(1e-6)
            m = _fetch(dep, ty, tx, _oct(to * inv[:, None]))
            var = (m[:, 1] - m[:, 0] ** 2).abs()
            dm = (dist - m[:, 0]).clamp_min(0)
            ch = torch.where(dist <= m[:, 0], torch.ones_like(dist), var / (var + dm * dm).clamp_min(1e-6))
            vis = (1 - cs) + (ch ** 3).clamp_min(0.05) * cs
            wrap = (-to * inv[:, None] * Nn).sum(1) * 0.5 + 0.5
            w = w * ((1 - cs) + (wrap * wrap).clamp_min(0.05) * cs) * vis
        e = _fetch(irr, ty, tx, oN)[:, :3]
        if dual:
            t = float(np.float32(0.7))
            e = _fetch(irr, ty, tx, oS)[:, :3] * (1 - t) + e * t
        acc += e * w[:, None]
        wsum += w
    return acc / wsum.clamp_min(1e-4)[:, None]


def exact(case, seed):
    """The gather in 64 bits. The updates, gradients and ray queries have none here: a
    restatement of the trace without a tree takes minutes at these sizes; trees and hit
    records are whole numbers."""
    if case["kind"] != "gather":
        return None
    atlases, (pos, nrm, det, _) = _gather_inputs(case, int(seed))
    cell = min(GATHER_BOXES[0][1]) / max(1, case["res"] - 1)
    bias = float(np.float32(max(1e-4, float(np.float32(cell)) * 0.04)))
    out = []
    for a in range(0, pos.shape[0], 1 << 19):
        p, n, d = (t[a:a + (1 << 19), :3].double() for t in (pos, nrm, det))
        P = p + n * bias
        if case["cascades"] == 1:
            E = _exact_cascade(case, GATHER_BOXES[0], atlases[0], P, P, n, d, case["dual"])
        else:
            E0, E1 = (_exact_cascade(case, GATHER_BOXES[k], atlases[k], p, P, n, d, False) for k in (0, 1))
            lo, size = (torch.tensor(np.float32(v), device=P.device, dtype=torch.float64) for v in GATHER_BOXES[1])
            f = (P - lo) / size
            edge = torch.minimum(f, 1 - f).amin(1)
            w = (edge / float(np.float32(0.15))).clamp(0, 1)[:, None]
            E = E0 * (1 - w) + E1 * w
        out.append(torch.cat([E.clamp_min(0), torch.ones_like(E[:, :1])], 1))
    return torch.cat(out)
