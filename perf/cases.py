"""The work a program has this library do, as timed cases.

Eight kinds, each through the package's public entry points:

  draw     Renderer.Draw: one progressive frame of a window, 16 samples per pixel at depth 4 unless
           the program asks for more (the reference's own main loop calls it with 1200 x 800)
  render   Wavefront.render: an offline render into an accumulator and an sRGB image, from a small
           preview to the full 1080p frame; with the default launch shapes or the autotuner's picks
  trace    DeviceScene.trace: closest hits of a caller's own rays (picking, visibility, ambient
           occlusion), coherent and incoherent ones mixed
  rebuild  venu_lbvh_build_noalloc: the LBVH rebuilt into the caller's buffers each frame
  frame    a scene from host spheres to an image in pinned host memory: DeviceScene, render, download
  animate  moving spheres: DeviceScene.update_device (refit), then a few samples per pixel
  batch    Batch.submit_many / run / collect: many renders of uneven scenes in one shared pool
  serve    Server.submit / wait: requests of a few resident scenes, submitted together

Scenes come from the package's seeded generators (the RTIOW final scene, or a ground sphere and
random spheres in a 200 x 20 x 200 box).  Work that scales with the scene is counted from the box and
sphere tests per ray segment that counting renders of those scenes report.
"""
import ctypes as C
import math

import numpy as np
import torch

import venusaur_gb300 as venu
from venusaur_gb300 import _lib

RTIOW_EYE, RANDOM_EYE = (13.0, 2.0, 3.0), (60.0, 15.0, 60.0)
SPHERE_BYTES = 48
# the autotuner's picks on the RTIOW scene at full size, on large random scenes and on small renders
TUNINGS = {
    "default": None,
    "fused256": dict(traverse_variant=2, traverse_block=256),
    "separate256": dict(traverse_variant=3, traverse_block=256),
    "wide128": dict(traverse_variant=4, traverse_block=128, in_place_factor=8),
}


def listed():
    return [
        # the smallest frame a program draws (a thumbnail): launches and host latency
        dict(name="draw_64x36", kind="draw", n=0, W=64, H=36, spp=2, depth=8),
        # the reference's window: 1200 x 800, 16 samples per pixel, depth 4
        dict(name="draw_1200x800", kind="draw", n=0, W=1200, H=800, spp=16, depth=4),
        # the small RTIOW render, with the autotuner's pick for it
        dict(name="render_rtiow_400x225", kind="render", n=0, W=400, H=225, spp=16, depth=50, tuning="wide128"),
        # the full-size RTIOW frame, the headline workload, as a new Wavefront renders it
        dict(name="render_rtiow_1080p", kind="render", n=0, W=1920, H=1080, spp=256, depth=50, tuning="default"),
        # a scene far larger than the caches, ragged image, the autotuner's pick for large scenes
        dict(name="render_1m_1919x1079", kind="render", n=1_000_000, W=1919, H=1079, spp=8, depth=50,
             tuning="separate256"),
        # a handful of queries against a small scene: picking
        dict(name="trace_rtiow_1001", kind="trace", n=0, rays=1001),
        # a million queries against a medium scene: visibility, ambient occlusion
        dict(name="trace_20k_1m", kind="trace", n=20_011, rays=1_000_003),
        # a particle scene rebuilt from scratch each frame
        dict(name="rebuild_40k", kind="rebuild", n=40_009),
        # a new large scene to its first image on the host: upload, build, a low-sample render, download
        dict(name="frame_300k_512x512", kind="frame", n=300_000, W=512, H=512, spp=4, depth=50),
        # one frame of an animation of moving spheres
        dict(name="animate_100k_640x360", kind="animate", n=100_000, W=640, H=360, spp=4, depth=8),
        # many small renders of uneven scenes at once
        dict(name="batch_96", kind="batch", jobs=96, nmax=20_000, spp=4, depth=50),
        # requests of three resident scenes submitted together
        dict(name="serve_16", kind="serve", requests=16, n=5_000, W=256, H=144, spp=8, depth=50),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["draw", "render", "render", "trace", "trace", "rebuild", "frame", "animate", "batch", "serve"])
    if kind == "draw":
        return dict(kind=kind, n=0, W=_log(rng, 33, 1920), H=_log(rng, 33, 1080), spp=rng.choice([1, 2, 4, 16, 16]),
                    depth=rng.choice([4, 4, 8, 50]))
    if kind == "render":
        n = 0 if rng.random() < 0.5 else _log(rng, 100, 1_000_000)
        return dict(kind=kind, n=n, W=_log(rng, 100, 1920), H=_log(rng, 60, 1080),
                    spp=_log(rng, 1, 64) if n == 0 else _log(rng, 1, 8), depth=rng.choice([4, 50, 50]),
                    tuning=rng.choice(sorted(TUNINGS)))
    if kind == "trace":
        return dict(kind=kind, n=0 if rng.random() < 0.3 else _log(rng, 100, 200_000), rays=_log(rng, 100, 2_000_000))
    if kind == "rebuild":
        return dict(kind=kind, n=_log(rng, 100, 65_536))
    if kind == "frame":
        return dict(kind=kind, n=0 if rng.random() < 0.5 else _log(rng, 100, 500_000), W=_log(rng, 64, 1280),
                    H=_log(rng, 64, 720), spp=rng.choice([1, 4, 8]), depth=rng.choice([4, 50]))
    if kind == "animate":
        return dict(kind=kind, n=_log(rng, 100, 500_000), W=_log(rng, 64, 1280), H=_log(rng, 64, 720),
                    spp=rng.choice([1, 2, 4]), depth=rng.choice([4, 8, 50]))
    if kind == "batch":
        return dict(kind=kind, jobs=_log(rng, 4, 128), nmax=_log(rng, 1_000, 100_000), spp=rng.choice([2, 4, 8]),
                    depth=rng.choice([8, 50]))
    return dict(kind=kind, requests=_log(rng, 2, 24), n=_log(rng, 500, 50_000), W=_log(rng, 64, 512),
                H=_log(rng, 64, 512), spp=rng.choice([4, 8, 16]), depth=rng.choice([8, 50]))


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------
def _spheres(n, seed):
    return venu.generate_rtiow(seed) if n == 0 else venu.generate_random(n, seed)


def _camera(n, W, H):
    return venu.Camera.look_at(RTIOW_EYE if n == 0 else RANDOM_EYE, (0.0, 0.0, 0.0), 20.0, W / H, 0.1, 10.0)


def _to_device(spheres):
    return torch.from_numpy(spheres.view(np.uint8).reshape(-1).copy()).cuda()


def _rays(n, m, seed):
    """Half towards the scene from one eye (coherent), half from points in the scene in all directions."""
    g = torch.Generator(device="cuda").manual_seed(seed)
    k = m // 2
    eye = torch.tensor(RTIOW_EYE if n == 0 else RANDOM_EYE, device="cuda")
    size = torch.tensor((22.0, 2.0, 22.0) if n == 0 else (200.0, 20.0, 200.0), device="cuda")
    low = torch.tensor((-11.0, 0.0, -11.0) if n == 0 else (-100.0, 0.0, -100.0), device="cuda")
    at = torch.linspace(0.0, 1.0, max(k, 1), device="cuda")[:k, None]
    target = (torch.rand(k, 3, generator=g, device="cuda") * 0.1 + 0.9 * torch.cat([at, 1 - at, (at * 97) % 1], 1))
    o = torch.cat([eye.expand(k, 3), low + size * torch.rand(m - k, 3, generator=g, device="cuda")])
    d = torch.cat([low + size * target - eye, torch.randn(m - k, 3, generator=g, device="cuda")])
    return torch.cat([o, d], 1).contiguous()


TRACE_TMIN, TRACE_TMAX = 0.001, 1000.0


def _moved(spheres, seed):
    """The next pose: every sphere but the ground shifted a little."""
    rng = np.random.default_rng(seed)
    out = spheres.copy()
    out["center"][1:] += rng.uniform(-0.2, 0.2, (len(out) - 1, 3)).astype(np.float32)
    return out


BATCH_SIZES = ((256, 144), (256, 256), (127, 95), (400, 225))


def _batch_jobs(case, seed):
    """Sizes from the case, scenes from the seed."""
    rng = np.random.default_rng(case["jobs"])
    jobs = []
    for i in range(case["jobs"]):
        n = 0 if rng.random() < 0.5 else int(round(math.exp(rng.uniform(math.log(100), math.log(case["nmax"])))))
        W, H = BATCH_SIZES[int(rng.integers(len(BATCH_SIZES)))]
        jobs.append((n, W, H, seed * 1000 + i))
    return jobs


def prepare(case, seed):
    kind = case["kind"]
    if kind == "draw":
        W, H = case["W"], case["H"]
        r = venu.Renderer(samples_per_pixel=case["spp"], max_depth=case["depth"])
        r.Init(venu.Scene(seed))
        cam = venu.Camera(RTIOW_EYE, 20.0, W / H, 0.1, 10.0)
        cam.SetForward(tuple(-x for x in RTIOW_EYE))
        return dict(kind=kind, renderer=r, camera=cam, out=venu.CUDAOutputBuffer(W, H))
    if kind == "trace":
        return dict(kind=kind, scene=venu.DeviceScene(_spheres(case["n"], seed)), rays=_rays(case["n"], case["rays"], seed))
    if kind == "rebuild":
        n = case["n"]
        f32 = dict(dtype=torch.float32, device="cuda")
        i32 = dict(dtype=torch.int32, device="cuda")
        build = venu.lib().venu_lbvh_build_noalloc
        build.argtypes = [C.c_void_p, C.c_uint32] + [C.c_void_p] * 6
        build.restype = C.c_int
        return dict(kind=kind, n=n, build=build, spheres=_to_device(_spheres(n, seed)),
                    nodes=torch.zeros(max(n - 1, 1) * 8, **f32), sph=torch.zeros(n * 4, **f32),
                    mat=torch.zeros(n * 4, **f32), meta=torch.zeros(n, **i32), morton=torch.zeros(n, **i32))
    if kind == "batch":
        scenes, jobs = {}, _batch_jobs(case, seed)
        pix = sum(W * H for _, W, H, _ in jobs)
        accum = torch.zeros((pix, _lib.ACCUM_FLOATS), dtype=torch.float32, device="cuda")
        image8 = torch.zeros((pix, 4), dtype=torch.uint8, device="cuda")
        args, at = [], 0
        for n, W, H, s in jobs:
            scene = venu.DeviceScene(_spheres(n, s))
            args.append(dict(scene=scene, camera=_camera(n, W, H), width=W, height=H, spp=case["spp"],
                             accum=accum[at:at + W * H], image8=image8[at:at + W * H], subframe=1,
                             max_depth=case["depth"], reset=True))
            at += W * H
        return dict(kind=kind, batch=venu.Batch(pool_paths=16 << 20, max_jobs=128), jobs=args, accum=accum, image8=image8)
    if kind == "serve":
        spheres = [_spheres(case["n"] + k, 10 * seed + k) for k in range(3)]
        cam = _camera(case["n"], case["W"], case["H"])
        asks = [dict(camera=cam, width=case["W"], height=case["H"], spp=case["spp"], spheres=spheres[i % 3],
                     scene_key=1 + i % 3, subframe=1 + i, max_depth=case["depth"]) for i in range(case["requests"])]
        return dict(kind=kind, server=venu.Server(32 << 30, pool_paths=16 << 20, max_jobs=64), asks=asks)
    # render, frame, animate
    n, W, H = case["n"], case["W"], case["H"]
    spheres = _spheres(n, seed)
    wave = venu.Wavefront()
    tuning = TUNINGS[case.get("tuning", "default")]
    if tuning:
        wave.set_tuning(**tuning)
    state = dict(kind=kind, wave=wave, camera=_camera(n, W, H), W=W, H=H, spp=case["spp"], depth=case["depth"],
                 subframe=1 + seed % 1000, accum=venu.new_accum(W, H),
                 image8=torch.zeros((H, W, 4), dtype=torch.uint8, device="cuda"))
    if kind == "frame":
        state["spheres"] = spheres
        state["host8"] = torch.zeros((H, W, 4), dtype=torch.uint8).pin_memory()
    else:
        state["scene"] = venu.DeviceScene(spheres)
    if kind == "animate":
        state["n"] = len(spheres)
        state["pose"] = _to_device(_moved(spheres, seed))
    return state


# ---------------------------------------------------------------------------
# one pass
# ---------------------------------------------------------------------------
def _render(s, scene):
    s["wave"].render(scene, s["camera"], s["W"], s["H"], s["spp"], s["accum"], subframe=s["subframe"],
                     max_depth=s["depth"], reset=True, image8=s["image8"])


def run(state):
    kind = state["kind"]
    if kind == "draw":
        r, out = state["renderer"], state["out"]
        r.Draw(state["camera"], out)
        return {"accum": r.accum, "pixels_f": out.pixels_f, "pixels": out.pixels}
    if kind == "render":
        _render(state, state["scene"])
        return {"accum": state["accum"], "image8": state["image8"]}
    if kind == "trace":
        t, ids, front = state["scene"].trace(state["rays"], TRACE_TMIN, TRACE_TMAX)
        return {"t": t, "id": ids, "front": front}
    if kind == "rebuild":
        s = state
        stream = torch.cuda.current_stream().cuda_stream
        rc = s["build"](s["spheres"].data_ptr(), s["n"], s["nodes"].data_ptr(), s["sph"].data_ptr(), s["mat"].data_ptr(),
                        s["meta"].data_ptr(), s["morton"].data_ptr(), stream)
        if rc:
            raise RuntimeError(venu.lib().venu_last_error())
        # the nodes hold boxes and child words: compared as the 32-bit words they are
        return {"nodes": s["nodes"].view(torch.int32), "sph": s["sph"], "mat": s["mat"], "meta": s["meta"],
                "morton": s["morton"]}
    if kind == "frame":
        scene = venu.DeviceScene(state["spheres"])
        _render(state, scene)
        state["host8"].copy_(state["image8"], non_blocking=True)
        torch.cuda.current_stream().synchronize()
        scene.close()
        return {"accum": state["accum"], "host8": state["host8"]}
    if kind == "animate":
        state["scene"].update_device(state["pose"], state["n"])
        _render(state, state["scene"])
        return {"accum": state["accum"], "image8": state["image8"]}
    if kind == "batch":
        b = state["batch"]
        b.submit_many(state["jobs"])
        b.run()
        b.collect()
        return {"accum": state["accum"], "image8": state["image8"]}
    ids = [state["server"].submit(**ask) for ask in state["asks"]]
    return {"images": np.stack([state["server"].wait(i)["image"] for i in ids])}


# ---------------------------------------------------------------------------
# the work a pass cannot do without
# ---------------------------------------------------------------------------
def _per_segment(n):
    """Flops of one ray segment: 20 a box test, 25 a sphere test, 60 to shade.  Counting renders report
    17.6 box and 3.3 sphere tests on the RTIOW scene, 107 and 8.3 on a million random spheres."""
    x = 0.0 if n == 0 else min(1.0, max(0.0, math.log(n / 485.0) / math.log(1e6 / 485.0)))
    return 20 * (17.6 + x * (107 - 17.6)) + 25 * (3.3 + x * (8.3 - 3.3)) + 60


def _segments(n, depth):
    """Ray segments per path: 2.7 on the RTIOW scene at depth 50, about 14 on a million spheres."""
    x = 0.0 if n == 0 else min(1.0, max(0.0, math.log(n / 485.0) / math.log(1e6 / 485.0)))
    return min(float(depth), 2.7 + x * 11.3)


def _image(n, W, H, spp, depth, out_bytes):
    spheres = 485 if n == 0 else n
    return spheres * SPHERE_BYTES + W * H * out_bytes, W * H * spp * _segments(n, depth) * _per_segment(n)


def work(case):
    kind = case["kind"]
    if kind in ("draw", "render", "frame", "animate"):
        # draw: accumulator read and written, two images; the others: accumulator written, one image
        b, f = _image(case["n"], case["W"], case["H"], case["spp"], case["depth"],
                      32 + 32 + 16 + 4 if kind == "draw" else 32 + 4)
        return {"bytes": b, "flops": f}
    if kind == "trace":
        n, m = case["n"], case["rays"]
        return {"bytes": (485 if n == 0 else n) * SPHERE_BYTES + m * (24 + 12), "flops": m * _per_segment(n)}
    if kind == "rebuild":
        n = case["n"]
        return {"bytes": n * (SPHERE_BYTES + 32 + 16 + 16 + 4 + 4), "flops": n * 100}
    if kind == "batch":
        parts = [_image(n, W, H, case["spp"], case["depth"], 36) for n, W, H, _ in _batch_jobs(case, 0)]
        return {"bytes": sum(p[0] for p in parts), "flops": sum(p[1] for p in parts)}
    b, f = _image(case["n"], case["W"], case["H"], case["spp"], case["depth"], 4)
    return {"bytes": case["requests"] * b, "flops": case["requests"] * f}


# ---------------------------------------------------------------------------
# in 64 bits
# ---------------------------------------------------------------------------
def exact(case, seed):
    """Closest hits by brute force in 64 bits.  A rendered pixel has no such value: each path's random
    decisions follow from its 32-bit hits, so a path traced in 64 bits is soon another path; the LBVH is
    words and copies of its inputs."""
    if case["kind"] != "trace":
        return None
    spheres = _spheres(case["n"], seed)
    if len(spheres) * case["rays"] > 1 << 35:
        return None
    c = torch.from_numpy(spheres["center"].copy()).cuda().double()
    r2 = torch.from_numpy(spheres["radius"].copy()).cuda().double() ** 2
    rays = _rays(case["n"], case["rays"], seed).double()
    best = torch.full((case["rays"],), TRACE_TMAX, dtype=torch.float64, device="cuda")
    step = max(1, (1 << 26) // len(spheres))
    for at in range(0, case["rays"], step):
        o, d = rays[at:at + step, :3], rays[at:at + step, 3:]
        a = (d * d).sum(1)[:, None]
        b = torch.zeros((len(o), len(c)), dtype=torch.float64, device="cuda")  # half of the linear coefficient
        k = -r2.expand(len(o), -1)
        h = [o[:, i:i + 1] - c[None, :, i] for i in range(3)]
        for i in range(3):
            b = b + h[i] * d[:, i:i + 1]
            k = k + h[i] * h[i]
        f = [h[i] - (b / a) * d[:, i:i + 1] for i in range(3)]
        disc = r2[None, :] - (f[0] * f[0] + f[1] * f[1] + f[2] * f[2])
        q = -(b + torch.copysign(torch.sqrt(a * disc.clamp(min=0.0)), b))
        ta, tb = q / a, k / q
        lo, hi = torch.minimum(ta, tb), torch.maximum(ta, tb)
        bad = float("inf")
        t = torch.where(lo >= TRACE_TMIN, lo, hi)
        t = torch.where((disc >= 0.0) & (t >= TRACE_TMIN) & (t <= TRACE_TMAX), t, bad)
        best[at:at + step] = torch.minimum(best[at:at + step], t.min(1).values)
    return {"t": best, "id": None, "front": None}
