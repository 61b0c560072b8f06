"""GPU tests of the paths that sizes choose: ray queries spread over warps or
split into up-front tests and refilled walks, bounces split the same way, the
finishing kernel's shares, the one-block and the tiled sorts of the LBVH build,
and the fast walk against the canonical one on scenes and rays at the edges of
its bounds.  Everything is bit-exact against the oracle (the tolerance of every
closest-hit, render and LBVH test here)."""
import numpy as np
import pytest

from oracle import pyoracle

pytestmark = pytest.mark.gpu


def _query_rays(m, seed, low, high, eye):
    rng = np.random.default_rng(seed)
    o = rng.uniform(low, high, (m, 3))
    d = rng.normal(size=(m, 3))
    k = m // 2
    o[:k] = eye
    d[:k] = rng.uniform(low, high, (k, 3)) - eye
    return np.concatenate([o, d], 1).astype(np.float32)


def _check_trace(venu, oracle, torch, spheres, rays, tmin=0.001, tmax=1e16, oracle_rows=None):
    ds = venu.DeviceScene(spheres)
    t, ids, front = ds.trace(torch.from_numpy(rays).cuda(), tmin, tmax)
    t, ids, front = t.cpu().numpy(), ids.cpu().numpy(), front.cpu().numpy()
    rows = slice(None) if oracle_rows is None else oracle_rows
    wid, wt, wfront, _, _ = oracle.trace_bvh(spheres, rays[rows], tmin, tmax)
    assert np.array_equal(ids[rows], wid)
    assert np.array_equal(t[rows].view(np.uint32), wt.view(np.uint32))
    assert np.array_equal(front[rows].astype(np.uint32), wfront)


# one warp's share of the rays changes at multiples of 152 SMs x 16 warps
@pytest.mark.parametrize("m", [1, 31, 33, 2431, 2432, 2433, 4865, 19457, 77823, 77825])
def test_trace_spread_sizes(venu, oracle, cuda, m):
    sp = oracle.scene_random(3000, 11)
    _check_trace(venu, oracle, cuda, sp, _query_rays(m, m, [-100, 0, -100], [100, 20, 100], (60, 15, 60)))


# the split's first sizes: 65536 spheres, 2^18 rays; and one ray more than warps of 32
@pytest.mark.parametrize("n,m", [(65535, 1 << 18), (65536, (1 << 18) - 1), (65536, 1 << 18), (70001, (1 << 18) + 33)])
def test_trace_split_walk(venu, oracle, cuda, n, m):
    sp = oracle.scene_random(n, 12)
    rays = _query_rays(m, 5, [-100, 0, -100], [100, 20, 100], (60, 15, 60))
    rays[7, 3:] = (0.0, -1.0, 0.0)  # along an axis
    rays[9] = (0.0, 1e5, 0.0, 1e-7, -1.0, 1e-7)  # from far outside: the canonical walk
    rays[11] = (4e4, 3e4, -5e4, -0.8, -0.6, 1.0)
    rows = np.r_[0:2000, m - 2000:m]
    _check_trace(venu, oracle, cuda, sp, rays, oracle_rows=rows)
    # tmin and tmax of the caller, and outputs that are not all asked for
    _check_trace(venu, oracle, cuda, sp, rays, 0.5, 40.0, oracle_rows=rows)
    import ctypes as C
    ds = venu.DeviceScene(sp)
    dev = cuda.from_numpy(rays).cuda()
    full = ds.trace(dev)
    only = cuda.zeros(m, dtype=cuda.float32, device="cuda")
    rc = venu.lib().venu_trace(ds.handle, C.c_void_p(dev.data_ptr()), C.c_uint32(m), C.c_float(0.001), C.c_float(1e16),
                               C.c_void_p(only.data_ptr()), None, None, None)
    assert rc == 0 and cuda.equal(only, full[0])


def _edge_scene(oracle, name):
    sp = oracle.scene_random(400, 21)
    if name == "giants":  # 70 huge spheres: none hoisted, the leaves' extent is theirs
        big = oracle.scene_random(70, 22)
        big["center"] *= 40.0
        big["radius"] = 900.0
        big["center"][:, 1] -= 2000.0
        sp = np.concatenate([sp, big])
    elif name == "four_hoisted":
        sp["center"][:4] = [[0, -1000, 0], [0, 1100, 0], [2500, 0, 0], [0, 0, -2500]]
        sp["radius"][:4] = [1000, 900, 2300, 2300]
    elif name == "two_huge":  # every leaf hoisted: the root's record is empty
        sp = sp[:2].copy()
        sp["center"] = [[0, -1000, 0], [0, 30, 0]]
        sp["radius"] = [1000.0, 400.0]
    elif name == "hollow":  # shells, zero radii, duplicates
        sp["center"][100:200] = sp["center"][0:100]
        sp["radius"][100:200] = -0.9 * sp["radius"][0:100]
        sp["material"][100:200] = 2
        sp["ir"][100:200] = 1.5
        sp["radius"][200:220] = 0.0
        sp["center"][220:240] = sp["center"][240:260]
        sp["radius"][220:240] = sp["radius"][240:260]
    elif name == "far":  # a small scene a long way from the origin
        sp = sp[1:].copy()
        sp["center"] *= 0.05
        sp["center"] += np.float32(1500.0)
    return np.ascontiguousarray(sp)


@pytest.mark.parametrize("name", ["giants", "four_hoisted", "two_huge", "hollow", "far"])
def test_fast_walk_edge_scenes(venu, oracle, cuda, name):
    """The widened boxes of the traversal records never cull a hit: ray queries
    and renders equal the oracle's, whose walk tests every leaf's sphere, on
    scenes whose extent, hoisted leaves or radii are unusual; origins on and
    inside spheres, in the planes of the axes, directions with zero and tiny
    components, grazing rays, negative tmin."""
    torch = cuda
    sp = _edge_scene(oracle, name)
    rng = np.random.default_rng(3)
    c, r = sp["center"], np.abs(sp["radius"])
    k = rng.integers(len(sp), size=6000)
    nrm = rng.normal(size=(6000, 3))
    nrm /= np.linalg.norm(nrm, axis=1)[:, None]
    on = c[k] + r[k, None] * nrm
    d = rng.normal(size=(6000, 3))
    d[:2000] = np.cross(nrm[:2000], d[:2000])       # tangent to the sphere the origin lies on
    d[2000:2500, 0] = 0.0
    d[2500:3000, 1] *= 1e-6
    d[3000:3300, :2] = 0.0
    on[3300:3600, 2] = 0.0
    j = rng.integers(len(sp), size=6000)
    graze = c[j] + r[j, None] * np.cross(nrm, rng.normal(size=(6000, 3)))
    d[4000:] = graze[4000:] - on[4000:]             # towards another sphere's rim
    rays = np.concatenate([on, d], 1).astype(np.float32)
    _check_trace(venu, oracle, cuda, sp, rays)
    _check_trace(venu, oracle, cuda, sp, rays, -5.0, 50.0)
    W, H, spp, depth = 48, 27, 2, 12
    lo, hi = (c - r[:, None]).min(0), (c + r[:, None]).max(0)
    at = c.mean(0) if name != "far" else (lo + hi) / 2
    eye = at + np.array([70, 20, 65]) if name != "far" else at + np.array([12, 4, 11])
    cam = oracle.camera(tuple(eye), tuple(at), 40.0, W / H, 0.1, 10.0)
    want = oracle.render(sp, cam, W, H, spp, subframe=1, max_depth=depth, mode=pyoracle.MODE_GB300)
    ds = venu.DeviceScene(sp)
    for variant in (2, 3, 4, 5):
        wf = venu.Wavefront(0)
        wf.set_tuning(traverse_variant=variant)
        acc = venu.new_accum(W, H)
        wf.render(ds, cam, W, H, spp, acc, subframe=1, max_depth=depth, reset=True)
        torch.cuda.synchronize()
        assert np.array_equal(acc.cpu().numpy().view(np.uint32), want["accum"].view(np.uint32)), variant
        assert wf.stats()["segments"] == want["segments"]


@pytest.mark.parametrize("variant", [0, 3])
def test_split_bounces(venu, oracle, cuda, variant):
    """Bounces of 2^20 rays and more on a scene of 16384 spheres and more: the
    accumulator equals the fused kernel's, whose every path another test pins,
    and the oracle's on sampled rows; one sphere or one sample less does not
    split."""
    torch = cuda
    W, H, depth = 1024, 513, 7
    cam = oracle.camera((60, 15, 60), (0, 0, 0), 20.0, W / H, 0.1, 10.0)
    for n, spp in ((16384, 2), (16383, 2), (16384, 1)):
        sp = oracle.scene_random(n, 31)
        ds = venu.DeviceScene(sp)
        got = {}
        for v in (variant, 2):
            wf = venu.Wavefront(0)
            wf.set_tuning(traverse_variant=v, traverse_block=128)
            acc = venu.new_accum(W, H)
            wf.render(ds, cam, W, H, spp, acc, subframe=3, max_depth=depth, reset=True)
            torch.cuda.synchronize()
            got[v] = (acc.cpu().numpy().view(np.uint32), wf.stats()["segments"])
        assert got[variant][1] == got[2][1]
        assert np.array_equal(got[variant][0], got[2][0])
        want = oracle.render(sp, cam, W, H, spp, subframe=3, max_depth=depth, mode=pyoracle.MODE_GB300, rows=(200, 208))
        rows = slice(200 * W, 208 * W)
        assert np.array_equal(got[2][0][rows], want["accum"].view(np.uint32)[rows])


# one path a warp and less, shares that do not divide, a full grid and one path more
@pytest.mark.parametrize("W,H,spp", [(2, 2, 1), (3, 11, 1), (152, 8, 1), (1217, 2, 1), (608, 256, 1), (311, 501, 1)])
@pytest.mark.parametrize("variant,factor", [(2, 1), (2, 4), (4, 1), (4, 16)])
def test_finishing_shares(venu, oracle, cuda, W, H, spp, variant, factor):
    sp = oracle.scene_rtiow(0)
    cam = oracle.camera((13, 2, 3), (0, 0, 0), 20.0, W / H, 0.1, 10.0)
    ds = venu.DeviceScene(sp)
    want = oracle.render(sp, cam, W, H, spp, subframe=2, max_depth=40, mode=pyoracle.MODE_GB300)
    wf = venu.Wavefront(0)
    wf.set_tuning(traverse_variant=variant, in_place_factor=factor)
    acc = venu.new_accum(W, H)
    acc.fill_(3.0)  # reset has to clear it
    img = cuda.zeros((W * H, 4), dtype=cuda.uint8, device="cuda")
    imf = cuda.zeros((W * H, 4), dtype=cuda.float32, device="cuda")
    wf.render(ds, cam, W, H, spp, acc, subframe=2, max_depth=40, reset=True, image_f=imf, image8=img)
    cuda.cuda.synchronize()
    assert np.array_equal(acc.cpu().numpy().view(np.uint32), want["accum"].view(np.uint32))
    assert np.array_equal(img.cpu().numpy(), want["image8"])
    assert np.array_equal(imf.cpu().numpy().view(np.uint32), want["image_f"].view(np.uint32))
    assert wf.stats()["segments"] == want["segments"]


# scenes of 7168 spheres and more finish over the binary tree with refilled walks
@pytest.mark.parametrize("n", [7167, 7168])
@pytest.mark.parametrize("variant,factor", [(0, 1), (1, 1), (2, 1), (2, 16), (3, 1), (4, 1), (4, 16), (5, 1)])
def test_finishing_walks(venu, oracle, cuda, n, variant, factor):
    W, H, spp, depth = 311, 101, 2, 30
    sp = oracle.scene_random(n, 21, (-40, 0, -40), (40, 12, 40))
    cam = oracle.camera((30, 10, 30), (0, 4, 0), 40.0, W / H, 0.05, 30.0)
    want = oracle.render(sp, cam, W, H, spp, subframe=1, max_depth=depth, mode=pyoracle.MODE_GB300)
    ds = venu.DeviceScene(sp)
    wf = venu.Wavefront(0)
    wf.set_tuning(traverse_variant=variant, in_place_factor=factor)
    acc = venu.new_accum(W, H)
    wf.render(ds, cam, W, H, spp, acc, subframe=1, max_depth=depth, reset=True)
    cuda.cuda.synchronize()
    assert np.array_equal(acc.cpu().numpy().view(np.uint32), want["accum"].view(np.uint32))
    assert wf.stats()["segments"] == want["segments"]


# the block's survivors are placed by a sum over its 2 to 16 warps
@pytest.mark.parametrize("shade_block", [64, 96, 480, 512])
@pytest.mark.parametrize("variant", [0, 3])
def test_separate_shading_blocks(venu, oracle, cuda, variant, shade_block):
    W, H, spp, depth = 641, 487, 2, 6  # twice what one 128-thread block an SM leaves to the finishing kernel
    sp = oracle.scene_random(500, 31, (-10, 0, -10), (10, 3, 10))
    cam = oracle.camera((13, 2, 3), (0, 1, 0), 30.0, W / H, 0.1, 10.0)
    want = oracle.render(sp, cam, W, H, spp, subframe=1, max_depth=depth, mode=pyoracle.MODE_GB300)
    ds = venu.DeviceScene(sp)
    wf = venu.Wavefront(0)
    wf.set_tuning(traverse_variant=variant, traverse_block=128, traverse_blocks_per_sm=1, shade_block=shade_block)
    acc = venu.new_accum(W, H)
    wf.render(ds, cam, W, H, spp, acc, subframe=1, max_depth=depth, reset=True)
    cuda.cuda.synchronize()
    assert np.array_equal(acc.cpu().numpy().view(np.uint32), want["accum"].view(np.uint32))
    assert wf.stats()["segments"] == want["segments"]


def test_waves_accumulate_and_resolve_once(venu, oracle, cuda):
    """Several waves of part of the pixels and of part of the samples: each pixel
    starts from zero (or from what is there) once and is resolved once."""
    sp = oracle.scene_rtiow(0)
    W, H, spp, depth = 64, 36, 5, 6
    cam = oracle.camera((13, 2, 3), (0, 0, 0), 20.0, W / H, 0.1, 10.0)
    ds = venu.DeviceScene(sp)
    first = oracle.render(sp, cam, W, H, spp, subframe=1, max_depth=depth, mode=pyoracle.MODE_GB300)
    both = oracle.render(sp, cam, W, H, spp, subframe=2, max_depth=depth, mode=pyoracle.MODE_GB300,
                         accum=first["accum"].copy())
    first = oracle.render(sp, cam, W, H, spp, subframe=1, max_depth=depth, mode=pyoracle.MODE_GB300)
    for max_paths in (1000, W * H, 2 * W * H, 0):
        wf = venu.Wavefront(max_paths)
        acc = venu.new_accum(W, H)
        acc.fill_(7.0)
        img = cuda.zeros((W * H, 4), dtype=cuda.uint8, device="cuda")
        for sub, want, reset in ((1, first, True), (2, both, False)):
            wf.render(ds, cam, W, H, spp, acc, subframe=sub, max_depth=depth, reset=reset, image8=img)
            cuda.cuda.synchronize()
            assert np.array_equal(acc.cpu().numpy().view(np.uint32), want["accum"].view(np.uint32))
            assert np.array_equal(img.cpu().numpy(), want["image8"])
            assert wf.stats()["segments"] == want["segments"]


# the one-block codes and sort end at 4096; tiles of 128 keys end at 65536, of 256 at 262144
@pytest.mark.parametrize("n", [1, 2, 3, 63, 64, 65, 2047, 4095, 4096, 4097, 65535, 65537, 262144, 262145])
def test_lbvh_sort_paths(venu, oracle, cuda, n):
    sp = oracle.scene_random(n, 41)
    if n > 100:  # runs of equal codes
        sp["center"][n // 2:n // 2 + 50] = sp["center"][n // 2]
    got = venu.DeviceScene(sp).export_bvh()
    want = oracle.lbvh(sp)
    assert np.array_equal(got["keys"], want["keys"]) and np.array_equal(got["ids"], want["ids"])
    assert got["nodes"].tobytes() == want["nodes"].tobytes()


def test_concurrent_traces_of_one_scene(venu, oracle, cuda):
    """Queries of one scene from several threads at once, more of them than the
    scene has error words for."""
    import threading
    sp = oracle.scene_random(2000, 51)
    ds = venu.DeviceScene(sp)
    rays = _query_rays(3000, 6, [-100, 0, -100], [100, 20, 100], (60, 15, 60))
    wid, wt, _, _, _ = oracle.trace_bvh(sp, rays)
    dev = cuda.from_numpy(rays).cuda()
    cuda.cuda.synchronize()
    bad = []

    def work():
        s = cuda.cuda.Stream()
        with cuda.cuda.stream(s):
            for _ in range(5):
                t, ids, _ = ds.trace(dev, stream=s)
                s.synchronize()
                if not (np.array_equal(ids.cpu().numpy(), wid) and np.array_equal(t.cpu().numpy(), wt)):
                    bad.append(1)

    threads = [threading.Thread(target=work) for _ in range(40)]
    for th in threads:
        th.start()
    for th in threads:
        th.join()
    assert not bad
