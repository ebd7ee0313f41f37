"""The work that programs give this framework, as cases that can be timed.

Every case goes through the package's public entry points: path-traced stills
(vs_render and the film download), ray batches, real-time ReSTIR frames with
and without the denoiser, cache-terminated frames, the radiance-cache network
by itself and the render-job server.  Scenes are the package's own procedural
ones; a seed moves the camera and the sampler's streams (and makes the rays,
features, targets and weights), so that another seed is another input of the
same cost.
"""
import math

import numpy as np
import torch

import vision_b200 as vb
from vision_b200 import scenes

LR, BETA1, BETA2, EPS = 1e-3, 0.9, 0.999, 1e-8

ROOMS = dict(box=scenes.box_room, material=scenes.material_room, principled=scenes.principled_room,
             substrate=scenes.substrate_room, plastic=scenes.plastic_room, metallic=scenes.metallic_room,
             mix=scenes.mix_room, point=scenes.point_light_room)

_ctx = None


def context():
    """A program has one context for all of its scenes."""
    global _ctx
    if _ctx is None:
        _ctx = vb.Context(0)
    return _ctx


def listed():
    return [
        # An interactive viewer's preview: a few thousand paths, a display
        # image; launches and latency are what counts.
        dict(name="preview_64", kind="room", room="box", width=64, height=64, spp=1, depth=8, dim=4, sampler="pcg",
             film="rgba8"),
        # The plain tracer's own small workload (bench: box_room).
        dict(name="box_room_256", kind="room", room="box", width=256, height=256, spp=16, depth=8, dim=4,
             sampler="pcg", film="fp32"),
        # Layered glossy materials at an odd size, three wavelengths, the
        # schema's default sampler and the FP64 film of convergence studies.
        dict(name="principled_393x221", kind="room", room="principled", width=393, height=221, spp=8, depth=8, dim=3,
             sampler="independent", film="fp64"),
        # The headline scene (2.3 M triangles, glass, gold and principled
        # materials, HDR sky) at its resolution, a few samples of a still.
        dict(name="large_scene_1024", kind="large", width=1024, height=1024, spp=8, depth=16, subdivisions=7, grid=1000,
             sky=2048),
        # Many instances of two meshes: two-level traversal.
        dict(name="instanced_640x360", kind="instanced", width=640, height=360, spp=4, depth=16, copies=16),
        # A batch of incoherent rays from another renderer or a tool (visibility, baking).
        dict(name="rays_1048573", kind="rays", n=1048573, subdivisions=6, grid=500),
        # A frame of the real-time many-light workload (bench: many_lights), shown on a display.
        dict(name="realtime_1080", kind="realtime", width=1920, height=1080, emitters=10000, lights=32, denoise=False),
        # A smaller real-time view with the denoiser, odd size.
        dict(name="denoised_633x357", kind="realtime", width=633, height=357, emitters=1000, lights=16, denoise=True),
        # Cache-terminated frames that train as they render (bench: radiance_cache).
        dict(name="cached_1080", kind="cached", width=1920, height=1080, frames=2, train=65536),
        # The network at the queries of a whole 1080p frame.
        dict(name="infer_2073600", kind="infer", n=2073600),
        # Four training steps of the frame's size.
        dict(name="train_65536", kind="train", n=65536, steps=4),
        # Mixed jobs on two resident scenes, submitted together.
        dict(name="server_jobs", kind="server", jobs=12, scale=1.0),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["room", "room", "large", "instanced", "rays", "realtime", "cached", "infer", "train", "server"])
    if kind == "room":
        return dict(kind=kind, room=rng.choice(sorted(ROOMS)), width=_log_int(rng, 32, 640),
                    height=_log_int(rng, 32, 400), spp=_log_int(rng, 1, 16), depth=rng.randint(2, 16),
                    dim=rng.choice([3, 4]), sampler=rng.choice(["pcg", "independent"]),
                    film=rng.choice(["rgba8", "fp32", "fp64"]))
    if kind == "large":
        return dict(kind=kind, width=_log_int(rng, 64, 1024), height=_log_int(rng, 64, 1024), spp=_log_int(rng, 1, 8),
                    depth=rng.randint(4, 16), subdivisions=rng.randint(4, 6), grid=10 * rng.randint(10, 60),
                    sky=rng.choice([512, 1024]))
    if kind == "instanced":
        return dict(kind=kind, width=_log_int(rng, 64, 640), height=_log_int(rng, 64, 360), spp=_log_int(rng, 1, 4),
                    depth=rng.randint(4, 16), copies=rng.randint(9, 16))
    if kind == "rays":
        return dict(kind=kind, n=_log_int(rng, 100, 1048573), subdivisions=rng.randint(3, 6),
                    grid=10 * rng.randint(5, 50))
    if kind == "realtime":
        return dict(kind=kind, width=_log_int(rng, 160, 1920), height=_log_int(rng, 90, 1080),
                    emitters=_log_int(rng, 30, 3000), lights=rng.choice([8, 16, 32]), denoise=rng.random() < 0.5)
    if kind == "cached":
        return dict(kind=kind, width=_log_int(rng, 160, 1920), height=_log_int(rng, 90, 1080), frames=rng.randint(1, 2),
                    train=rng.choice([0, 4096, 16000, 65536]))
    if kind == "infer":
        return dict(kind=kind, n=_log_int(rng, 100, 2073600))
    if kind == "train":
        return dict(kind=kind, n=_log_int(rng, 100, 65536), steps=rng.randint(1, 4))
    return dict(kind=kind, jobs=rng.randint(3, 12), scale=rng.uniform(0.4, 1.0))


def _move(sc, seed, spread):
    """The scene's camera shifted by the seed, and its sampler's streams."""
    r = np.random.default_rng(seed)
    p = sc["camera"]["param"]["transform"]["param"]
    p["position"] = [float(x + spread * d) for x, d in zip(p["position"], r.uniform(-1.0, 1.0, 3))]
    sc["sampler"]["param"]["seed"] = int(seed) % 65521
    return sc


def _room(c, seed):
    kw = dict(width=c["width"], height=c["height"], dimension=c["dim"], sampler=c["sampler"], max_depth=c["depth"])
    return _move(ROOMS[c["room"]](**kw), seed, 0.05)


def _outdoors(c, seed, **kw):
    return _move(scenes.large_scene(width=c.get("width", 64), height=c.get("height", 64), max_depth=c.get("depth", 16),
                                    subdivisions=c["subdivisions"], grid=c["grid"], sky_width=c.get("sky", 256),
                                    sky_height=c.get("sky", 256) // 2), seed, 0.1)


def _scene(doc):
    return vb.Scene(context(), doc).build_accel()


def _server_jobs(c):
    """(scene, width, height, spp) of each job."""
    sizes = [(256, 256), (480, 270), (191, 107), (640, 360)]
    s = c["scale"]
    return [(i % 2, max(16, int(sizes[i % 4][0] * s)), max(16, int(sizes[i % 4][1] * s)), (1, 16, 4)[i % 3])
            for i in range(c["jobs"])]


def _generator(seed):
    return torch.Generator("cuda").manual_seed(int(seed))


def _weights(seed):
    """Master weights W[l][in][out] as the network is initialised: uniform in +-sqrt(6 / 64)."""
    r = np.random.default_rng(seed)
    return r.uniform(-1.0, 1.0, vb.CACHE_PARAMS).astype(np.float32) * np.float32(math.sqrt(6.0 / 64.0))


def _features(n, seed):
    g = _generator(seed)
    return torch.empty(n, 64, device="cuda").uniform_(0.0, 1.0, generator=g).to(torch.bfloat16)


def _targets(n, seed):
    return torch.empty(n, 4, device="cuda").exponential_(1.0, generator=_generator(seed + 1))


def _cache(seed):
    cache = vb.RadianceCache(context(), seed=seed % 1000 + 1)
    cache.set_weights(_weights(seed))
    cache.set_optimizer(LR, BETA1, BETA2, EPS)
    return cache


def prepare(case, seed):
    c = case
    st = dict(case=c)
    if c["kind"] == "room":
        st["scene"] = _scene(_room(c, seed))
    elif c["kind"] == "large":
        st["scene"] = _scene(_outdoors(c, seed))
    elif c["kind"] == "instanced":
        st["scene"] = _scene(_move(scenes.instanced_scene(width=c["width"], height=c["height"], copies=c["copies"],
                                                          max_depth=c["depth"]), seed, 0.5))
    elif c["kind"] == "rays":
        st["scene"] = _scene(_outdoors(c, seed))
        g, n = _generator(seed), c["n"]
        rays = torch.empty(n, 8, device="cuda")
        rays[:, 0:3] = torch.rand(n, 3, device="cuda", generator=g) * torch.tensor([20.0, 2.5, 20.0], device="cuda") + \
            torch.tensor([-10.0, 0.02, -10.0], device="cuda")
        rays[:, 3] = 0.0
        rays[:, 4:7] = torch.nn.functional.normalize(torch.randn(n, 3, device="cuda", generator=g), dim=1)
        rays[:, 7] = 1e30
        st.update(rays=rays, hits=torch.zeros(n, 4, dtype=torch.int32, device="cuda"),
                  t=torch.zeros(n, device="cuda"), stream=torch.cuda.Stream())
    elif c["kind"] == "realtime":
        sc = scenes.many_lights(width=c["width"], height=c["height"], emitters=c["emitters"], M_light=c["lights"])
        sc["sampler"]["param"]["seed"] = int(seed) % 65521
        st["scene"] = _scene(sc)
        if c["denoise"]:
            st["scene"].denoiser_enable()
        st.update(path=scenes.camera_spline(64, seed=seed), frame=0)
    elif c["kind"] == "cached":
        st["scene"] = _scene(_move(scenes.box_room(width=c["width"], height=c["height"], dimension=3, sampler="pcg"),
                                   seed, 0.05))
        st["cache"] = _cache(seed)
    elif c["kind"] == "infer":
        st.update(cache=_cache(seed), x=_features(c["n"], seed), y=torch.zeros(c["n"], 4, device="cuda"),
                  stream=torch.cuda.Stream())
    elif c["kind"] == "train":
        st.update(cache=_cache(seed), stream=torch.cuda.Stream(),
                  x=[_features(c["n"], seed + 10 * k) for k in range(c["steps"])],
                  t=[_targets(c["n"], seed + 10 * k) for k in range(c["steps"])])
    else:
        server = vb.Server(context(), paths_per_batch=1 << 22)
        st["server"] = server
        st["ids"] = [server.add_scene(_scene(scenes.box_room(sampler="pcg"))),
                     server.add_scene(_scene(scenes.large_scene(subdivisions=6, grid=400, sky_width=512,
                                                                sky_height=256)))]
        r = np.random.default_rng(seed)
        st["jobs"] = []
        for scene, w, h, spp in _server_jobs(c):
            eye, aim = ((0.0, 0.5, 1.85), (0.0, 0.5, 0.0)) if scene == 0 else ((0.0, 2.2, 5.0), (0.0, 0.9, 0.0))
            eye = np.asarray(eye) + 0.05 * r.uniform(-1.0, 1.0, 3)
            st["jobs"].append((scene, w, h, spp, scenes.camera_c2w(eye, aim)))
    torch.cuda.synchronize()
    return st


def run(state):
    st, c = state, state["case"]
    kind = c["kind"]
    if kind in ("room", "large", "instanced"):
        s, film = st["scene"], c.get("film", "fp32")
        s.render(0, c["spp"], fp64=film == "fp64")
        if film == "fp64":
            return [s.film(), s.film(vb.FILM_SUM64)]
        return s.film(vb.FILM_RGBA8 if film == "rgba8" else vb.FILM_LINEAR)
    if kind == "rays":
        st["scene"].trace_closest_device(st["rays"].data_ptr(), c["n"], st["hits"].data_ptr(), st["t"].data_ptr(),
                                         stream=st["stream"].cuda_stream)
        return [st["hits"], st["t"]]
    if kind == "realtime":
        s, f = st["scene"], st["frame"]
        s.set_camera(st["path"][f % len(st["path"])], 40.0)
        s.restir_frame(f)
        st["frame"] = f + 1
        return s.restir_buffer("denoised") if c["denoise"] else s.film(vb.FILM_RGBA8)
    if kind == "cached":
        s = st["scene"]
        s.render_cached(st["cache"], 0, c["frames"], train_samples=c["train"])
        return [s.film(), st["cache"].weights()]
    if kind == "infer":
        st["cache"].infer(st["x"].data_ptr(), c["n"], st["y"].data_ptr(), stream=st["stream"].cuda_stream)
        return st["y"]
    if kind == "train":
        cache = st["cache"]
        for x, t in zip(st["x"], st["t"]):
            cache.train(x.data_ptr(), t.data_ptr(), c["n"], stream=st["stream"].cuda_stream)
        st["stream"].synchronize()
        return [cache.gradient(), cache.weights()]
    server = st["server"]
    ids = [server.submit(st["ids"][scene], w, h, spp, c2w=c2w, fov_y=40.0) for scene, w, h, spp, c2w in st["jobs"]]
    return [server.result(j) for j in ids]


def _paths_work(paths, pixels, depth, tris, texels, film_bytes=16):
    """A path's few closest-hit and shadow queries (a box and triangle test
    for each level of a binary tree over the triangles) and its shading; the
    scene read once, the film written once."""
    segments = 1.6 * min(depth, 5)
    per = 12.0 * math.log2(max(tris, 2)) + 400.0
    return dict(bytes=64.0 * tris + 24.0 * texels + film_bytes * pixels, flops=paths * segments * per)


def work(case):
    c = case
    kind = c["kind"]
    px = c.get("width", 0) * c.get("height", 0)
    tris = 20 * 4 ** c.get("subdivisions", 0) + 2 * c.get("grid", 0) ** 2
    if kind == "room":
        return _paths_work(px * c["spp"], px, c["depth"], 36, 0, {"rgba8": 4, "fp32": 16, "fp64": 48}[c["film"]])
    if kind == "large":
        return _paths_work(px * c["spp"], px, c["depth"], tris, c["sky"] * c["sky"] // 2)
    if kind == "instanced":
        return _paths_work(px * c["spp"], px, c["depth"], 161920, 2048 * 1024)
    if kind == "rays":
        return dict(bytes=52.0 * c["n"] + 64.0 * tris, flops=c["n"] * 12.0 * math.log2(tris))
    if kind == "realtime":
        # Reservoirs and surfaces of a frame read and written once (64-byte records), the light candidates,
        # two traced paths of a few bounces.
        w = _paths_work(2 * px, px, 8, 36 + c["emitters"], 0, 4)
        return dict(bytes=w["bytes"] + px * (64.0 * 8 + 80.0), flops=w["flops"] + px * c["lights"] * 60.0)
    if kind == "cached":
        n = px * c["frames"]
        w = _paths_work(n, px, 2, 36, 0)
        train = 3.0 * min(c["train"], px) * c["frames"]
        return dict(bytes=w["bytes"] + 144.0 * n, flops=w["flops"] + 2.0 * vb.CACHE_PARAMS * (n + train))
    if kind == "infer":
        return dict(bytes=144.0 * c["n"], flops=2.0 * vb.CACHE_PARAMS * c["n"])
    if kind == "train":
        return dict(bytes=144.0 * c["n"] * c["steps"], flops=6.0 * vb.CACHE_PARAMS * c["n"] * c["steps"])
    parts = [_paths_work(w * h * spp, w * h, 8, 36 if scene == 0 else 401920, 0 if scene == 0 else 512 * 256)
             for scene, w, h, spp in _server_jobs(c)]
    return dict(bytes=sum(p["bytes"] for p in parts), flops=sum(p["flops"] for p in parts))


def _split(w):
    return [w[l * 4096:(l + 1) * 4096].view(64, 64) for l in range(4)] + [w[4 * 4096:].view(64, 3)]


def _forward(w, x):
    acts = [x]
    for l, m in enumerate(_split(w)):
        z = acts[-1] @ m
        acts.append(z if l == 4 else z.clamp_min(0.0))
    return acts


def exact(case, seed):
    c = case
    if c["kind"] == "infer":
        w = torch.from_numpy(_weights(seed)).cuda().double()
        x = _features(c["n"], seed)
        y = torch.zeros(c["n"], 4, dtype=torch.float64, device="cuda")
        for i in range(0, c["n"], 1 << 18):
            y[i:i + (1 << 18), :3] = _forward(w, x[i:i + (1 << 18)].double())[-1]
        return y
    if c["kind"] == "train":
        w = torch.from_numpy(_weights(seed)).cuda().double()
        m, v = torch.zeros_like(w), torch.zeros_like(w)
        for k in range(c["steps"]):
            x, t = _features(c["n"], seed + 10 * k).double(), _targets(c["n"], seed + 10 * k)[:, :3].double()
            acts = _forward(w, x)
            y, scale = acts[-1], 1.0 / (3.0 * c["n"])
            den = y * y + 0.01
            loss = float(((y - t) ** 2 / den).sum() * scale)
            dz, grads = 2.0 * (y - t) / den * scale, []
            for l in range(4, -1, -1):
                grads.append((acts[l].T @ dz).reshape(-1))
                dz = (dz @ _split(w)[l].T) * (acts[l] > 0.0)
            g = torch.cat(grads[::-1])
            m, v = BETA1 * m + (1.0 - BETA1) * g, BETA2 * v + (1.0 - BETA2) * g * g
            w = w - LR * (m / (1.0 - BETA1 ** (k + 1))) / ((v / (1.0 - BETA2 ** (k + 1))).sqrt() + EPS)
        return [(g, loss), w]
    return None
