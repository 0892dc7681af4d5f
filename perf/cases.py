"""Timed cases of the path tracer: what a program that renders with it does,
through the calls such a program makes.

Seven kinds of work, over their real range of sizes:

  preview   a moved camera: reset(), refine(spp) and the image read back;
            from one sample of a small window (latency, launches) to a 1080p
            frame of the million-triangle scene
  render    Renderer::render(): scene preparation, refinement and readback of
            a still in one call
  load      a scene that was edited or just opened: sync() from host memory
            and the first image of it
  frame     many samples of one frame on a resident scene, linear HDR or
            RGBA8 out: offline rendering, and the benchmark's headline frame
  batch     a service's tick: several sessions' samples as one launch
  cache     frames of a trained radiance cache
  train     one training step of the cache's network on host samples

`listed()` names the cases, `draw(rng)` gives another of the same ranges.
Scenes are the package's procedural ones, made from the seed.
"""
import ctypes as C
import math

import numpy as np

import __graft_entry__

# Execution plans as a user's program sets them: the default, the tuner's
# pick for large resident scenes, and what a service's executor runs.
PLANS = {
    "default": {},
    "split": dict(mode=2, graphs=1),
    "large": dict(mode=2, shade_variant=0, trace_variant=4, stack=64, wave_slots=1 << 22, nee_variant=3,
                  shadow_walk=0, graphs=1, refill=16),
    "serve": dict(mode=2, graphs=1, nee_variant=1),
}


def listed():
    return [
        # The smallest interactive call: one sample of a small window after a
        # camera move, the image on the host (launches and latency).
        dict(name="preview 256 cornell", kind="preview", scene="cornell", tris=36, w=256, h=256, spp=1, bounces=8,
             plan="default", out="image"),
        # The same on a full-screen window.
        dict(name="preview 1080p cornell", kind="preview", scene="cornell", tris=36, w=1920, h=1080, spp=1, bounces=8,
             plan="default", out="image"),
        # The million-triangle scene while its camera moves: one sample of
        # every pixel.
        dict(name="preview 1080p 1M", kind="preview", scene="textured", tris=1048820, w=1920, h=1080, spp=1,
             bounces=12, plan="large", out="image"),
        # The reference's own comparison: a Cornell box still, all in one call.
        dict(name="render 256 cornell 16", kind="render", scene="cornell", tris=36, w=256, h=256, spp=16, bounces=8,
             plan="default", out="image"),
        # An asset still: layered materials, transmission, texture and sky, at
        # a size that is no multiple of anything.
        dict(name="frame 641x359 materials", kind="frame", scene="materials", tris=20480, w=641, h=359, spp=32,
             bounces=12, plan="default", out="hdr"),
        # A block model of half a million triangles.
        dict(name="frame 720p boxes", kind="frame", scene="boxes", tris=480000, w=1280, h=720, spp=8, bounces=8,
             plan="split", out="image"),
        # The headline frame: the million-triangle scene at 64 samples.
        dict(name="frame 1080p 1M 64", kind="frame", scene="textured", tris=1048820, w=1920, h=1080, spp=64,
             bounces=12, plan="large", out="image"),
        # Opening the million-triangle scene, to its first image.
        dict(name="load 1M", kind="load", scene="textured", tris=1048820, w=480, h=270, spp=1, bounces=8,
             plan="default", out="image"),
        # An edit of a small scene, to the next image.
        dict(name="load 5k", kind="load", scene="boxes", tris=4800, w=320, h=200, spp=1, bounces=8, plan="default",
             out="image"),
        # A service's tick over mixed sessions (1e3 to 5e5 triangles).
        dict(name="batch 12", kind="batch", scene="mixed", tris=500000, w=768, h=432, spp=4, bounces=8, count=12,
             plan="serve", out="hdr"),
        # Frames of a trained cache, several in one wavefront.
        dict(name="cache 1080p 4", kind="cache", scene="materials", tris=20480, w=1920, h=1080, spp=4, bounces=12,
             plan="split", out="hdr"),
        # One training step of the cache on a frame's samples.
        dict(name="train 65536", kind="train", scene="cornell", tris=36, w=64, h=64, spp=1, bounces=8, n=65536,
             plan="default", out="grad"),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["preview", "preview", "render", "frame", "frame", "load", "batch", "cache", "train"])
    scene = rng.choice(["cornell", "materials", "boxes", "textured"])
    tris = 36 if scene == "cornell" else _log(rng, 1000, 1000000)
    w = _log(rng, 64, 1920)
    h = max(1, min(1080, int(w * rng.choice([0.5625, 0.75, 1.0]))) + rng.choice([0, 0, -1, 1]))
    bounces = rng.choice([4, 8, 8, 12])
    out = rng.choice(["image", "hdr"])
    plan = rng.choice(["default", "default", "split", "large"])
    most = max(1, 30000000 // (w * h))  # a fraction of the largest listed case's paths
    spp = 1
    c = dict(kind=kind, scene=scene, tris=tris, w=w, h=h, bounces=bounces, plan=plan, out=out)
    if kind == "render":
        spp = _log(rng, 1, min(most, 64))
    elif kind == "frame":
        spp = _log(rng, 1, min(most, 256))
    elif kind == "load":
        c["plan"] = "default"
    elif kind == "batch":
        c["scene"], c["plan"], c["out"] = "mixed", "serve", "hdr"
        c["tris"] = _log(rng, 20000, 500000)
        c["count"] = rng.randint(2, 16)
        spp = _log(rng, 1, max(1, min(16, most // (2 * c["count"]))))
    elif kind == "cache":
        c["plan"], c["out"] = "split", "hdr"
        spp = rng.choice([1, 2, 4])
    elif kind == "train":
        c.update(scene="cornell", tris=36, w=64, h=64, plan="default", out="grad", n=_log(rng, 1000, 65536))
    c["spp"] = spp
    return c


def _scene(pkg, what, tris, seed):
    """A seeded scene of about `tris` triangles, and its environment."""
    if what == "cornell":
        return pkg.Scene.cornell(), None
    if what == "boxes":
        return pkg.Scene.box_field(max(1, tris // 12), seed=seed, material_mix=1), pkg.EnvironmentMap.sky(256, 128)
    freq = max(4, int(round(math.sqrt(tris / 20.0))))
    if what == "materials":
        s = pkg.Scene.icosphere(freq=freq, seed=seed, n_materials=16, n_textures=2, tex_size=256, n_punctual=4,
                                n_emissive=16, material_mix=1)
        return s, pkg.EnvironmentMap.sky(256, 128)
    s = pkg.Scene.icosphere(freq=freq, seed=seed, n_materials=64, n_textures=8, tex_size=1024, n_punctual=16,
                            n_emissive=512, material_mix=0)
    return s, pkg.EnvironmentMap.sky(1024, 512, sun_dir=(0.3, 0.8, -0.5), sun_radiance=2000.0)


def _options(pkg, case, seed, w=None, h=None):
    return pkg.RenderOptions(width=w or case["w"], height=h or case["h"], scene_camera=0,
                             path_trace=pkg.PathTraceOptions(samples_per_pixel=case["spp"],
                                                             max_bounces=case["bounces"], rr_start=3, seed=seed))


def _tracer(pkg, case, scene, env, opts, plan):
    t = pkg.GpuPathTracer(0)
    if plan:
        t.set_tuning(**plan)
    if env is not None:
        t.set_environment(env)
    t.sync(scene, opts)
    return t


def _train_inputs(n, seed):
    r = np.random.default_rng(seed)
    x = np.zeros((n, 12), np.float32)
    x[:, :4] = r.random((n, 4))                      # position in the scene box, roughness
    for k in (4, 8):                                 # outgoing direction, normal, mapped to [0, 1]
        d = r.standard_normal((n, 3))
        x[:, k:k + 3] = 0.5 * (d / np.linalg.norm(d, axis=1, keepdims=True) + 1.0)
    t = np.zeros((n, 4), np.float32)
    t[:, :3] = r.gamma(0.7, 0.6, (n, 3))             # radiance: many dim samples, a few bright ones
    return x, t


def _weights(seed):
    """He-initialised FP32 weights, 64x256, three 64x64 and 16x64 (three rows used)."""
    r = np.random.default_rng(seed + 17)
    mats = [r.uniform(-1, 1, s) * math.sqrt(6.0 / s[1]) for s in _SHAPES]
    mats[-1][3:] = 0.0
    return np.concatenate([m.reshape(-1) for m in mats]).astype(np.float32)


_SHAPES = [(64, 256), (64, 64), (64, 64), (64, 64), (16, 64)]


def prepare(case, seed):
    pkg = __graft_entry__.load_package()
    kind, plan = case["kind"], PLANS[case["plan"]]
    if kind == "batch":
        r = np.random.default_rng(seed)
        env = pkg.EnvironmentMap.sky(256, 128)
        tracers = []
        for k in range(case["count"]):
            tris = int(round(math.exp(r.uniform(math.log(1000), math.log(case["tris"])))))
            w, h = (max(16, case[side] * (2 + (k * step) % 5) // 4 - k % 2) for side, step in (("w", 1), ("h", 3)))
            scene, _ = _scene(pkg, "boxes" if k % 2 else "materials", tris, seed + k)
            tracers.append(_tracer(pkg, case, scene, env, _options(pkg, case, seed + k, w, h), {}))
        executor = pkg.GpuPathTracer(0)
        executor.set_tuning(**plan)
        return dict(kind=kind, pkg=pkg, tracers=tracers, executor=executor, spp=case["spp"])
    scene, env = _scene(pkg, case["scene"], case["tris"], seed)
    opts = _options(pkg, case, seed)
    t = _tracer(pkg, case, scene, env, opts, plan)
    state = dict(kind=kind, pkg=pkg, scene=scene, opts=opts, tracer=t, spp=case["spp"], out=case["out"])
    if kind == "train":
        from oxideav_render_vulkan_b200.nrc import RadianceCache
        cache = RadianceCache(t, seed=1)
        cache.set_weights(_weights(seed))
        x, y = _train_inputs(case["n"], seed)
        state.update(cache=cache, x=x, y=y)
    elif kind == "cache":
        from oxideav_render_vulkan_b200.nrc import RadianceCache
        cache = RadianceCache(t, seed=1)
        cache.set_weights(_weights(seed))
        cache.configure(train=0, train_one_in=1 << 16, frames_per_wave=case["spp"])
        state.update(cache=cache)
    return state


def run(state):
    kind = state["kind"]
    if kind == "batch":
        for t in state["tracers"]:
            t.reset()
        state["pkg"].refine_batch(state["tracers"], state["spp"], state["executor"])
        return [t.hdr() for t in state["tracers"]]
    t = state["tracer"]
    if kind == "render":
        f = t.render_hdr if state["out"] == "hdr" else t.render
        return f(state["scene"], state["opts"])
    if kind == "train":
        N = state["pkg"]._native
        loss, grad = C.c_float(), np.empty(N.NRC_PARAMS, np.float32)
        st = N.lib().oxpt_nrc_train(state["cache"]._h, state["x"].ctypes.data, state["y"].ctypes.data,
                                    len(state["x"]), 0, C.byref(loss), grad.ctypes.data)
        if st != N.OK:
            raise RuntimeError(f"training step failed with status {st}")
        return {"loss": loss.value, "grad": grad}
    if kind == "load":
        t.invalidate_scene()
        t.sync(state["scene"], state["opts"])
    else:
        t.reset()
    if kind == "cache":
        state["cache"].refine(state["spp"])
    else:
        t.refine(state["spp"])
    return t.hdr() if state["out"] == "hdr" else t.image()


def work(case):
    if case["kind"] == "train":
        n, macs = case["n"], sum(a * b for a, b in _SHAPES)
        return {"bytes": n * 16 * 4 + 8 * macs, "flops": 6.0 * n * macs}
    count = case.get("count", 1)
    # (a batch's members have half to one and a half of each side, one on average)
    pixels = case["w"] * case["h"] * count
    # Each sample is a few rays: about two path segments in these scenes, and
    # a shadow ray each; a ray takes a box test of two children per level of
    # a balanced tree and a couple of triangles.
    segments = 3.0 if case["scene"] == "cornell" else 2.0
    rays = 2.0 * segments * pixels * case["spp"]
    levels = max(1.0, math.log2(case["tris"]))
    flops = rays * (2.0 * levels * 25.0 + 2.0 * 60.0) + pixels * case["spp"] * segments * 500.0
    out = pixels * (16 if case["out"] == "hdr" else 4)
    scene = 0.0 if count > 1 else case["tris"] * (48 + 64)  # triangles and their nodes
    if case["kind"] in ("load", "render"):
        scene += case["tris"] * 2.0 * 100 + (8 * 1024 * 1024 * 16.0 if case["scene"] == "textured" else 0.0)
    return {"bytes": out + scene, "flops": flops}


def exact(case, seed):
    """The training step's loss and gradient in 64 bits. A traced image has no
    such value: which surface a ray meets and which light it samples are
    decided by comparisons of single-precision numbers."""
    if case["kind"] != "train":
        return None
    n = case["n"]
    x, t = _train_inputs(n, seed)
    w = _weights(seed).astype(np.float64)
    mats, at = [], 0
    for a, b in _SHAPES:
        mats.append(w[at:at + a * b].reshape(a, b))
        at += a * b
    x = x.astype(np.float64)[:, [0, 1, 2, 3, 4, 5, 6, 7, 8, 9]]
    f = np.zeros((n, 256))
    for i in range(10):
        for j in range(12):
            a = np.pi * x[:, i] * 2.0 ** j
            f[:, 24 * i + 2 * j], f[:, 24 * i + 2 * j + 1] = np.sin(a), np.cos(a)
    f[:, 240:250], f[:, 250] = x, 1.0
    ins = [f]
    for m in mats[:-1]:
        ins.append(np.maximum(ins[-1] @ m.T, 0.0))
    y = (ins[-1] @ mats[-1].T)[:, :3]
    t = t.astype(np.float64)[:, :3]
    den = y * y + 0.01
    loss = float(np.sum((y - t) ** 2 / den) / (3 * n))
    g = np.zeros((n, 16))
    g[:, :3] = 2.0 * (y - t) / den / (3 * n)
    grads = []
    for m, a in zip(reversed(mats), reversed(ins)):
        grads.append((g.T @ a).reshape(-1))
        g = (g @ m) * (a > 0)
    return {"loss": loss, "grad": np.concatenate(grads[::-1])}
