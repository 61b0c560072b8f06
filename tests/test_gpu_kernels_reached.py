"""GPU tests that put work in front of one kernel each: sizes come from the grids (one
block of 64 or 128 threads an SM), and each test shows from counts of rays that
its kernel has some.  Everything is bit-exact against the oracle."""
import numpy as np
import pytest

from oracle import pyoracle

from test_gpu_parity import DEEP, _nested_scene
from test_gpu_paths import _edge_scene

pytestmark = pytest.mark.gpu


def _same(got, want):
    return np.array_equal(got.cpu().numpy().view(np.uint32), want.view(np.uint32))


def _rays_at(oracle, sp, cam, W, H, spp, sub, bounce):
    """Rays of bounce `bounce` (from 0): segments up to it, less those before it."""
    seg = [oracle.render(sp, cam, W, H, spp, subframe=sub, max_depth=d, mode=pyoracle.MODE_GB300)["segments"] if d else 0
           for d in (bounce, bounce + 1)]
    return seg[1] - seg[0]


def _check_large(venu, oracle, cuda, ds, sp, cam, W, H, spp, sub, depth, tuning, built_from=None, split_from=None):
    """A render too large for the oracle: all of it against the fused kernel's with
    the default tuning, sampled rows against the oracle's.  split_from: the first
    bounce that k_walk takes, which has to have at least 2^20 rays."""
    seg = [0]
    for d in range(1, depth + 1):
        wf = venu.Wavefront(0)
        acc = venu.new_accum(W, H)
        wf.render(ds, cam, W, H, spp, acc, subframe=sub, max_depth=d, reset=True)
        cuda.cuda.synchronize()
        seg.append(wf.stats()["segments"])
    if split_from is not None:
        assert seg[split_from + 1] - seg[split_from] >= 1 << 20
    wf = venu.Wavefront(0)
    wf.set_tuning(**tuning)
    mine = venu.new_accum(W, H)
    wf.render(ds, cam, W, H, spp, mine, subframe=sub, max_depth=depth, reset=True)
    cuda.cuda.synchronize()
    assert wf.stats()["segments"] == seg[depth] and cuda.equal(mine, acc)
    for row in (H // 3, H // 2, H - 9):
        want = oracle.render(sp, cam, W, H, spp, subframe=sub, max_depth=depth, mode=pyoracle.MODE_GB300,
                             rows=(row, row + 8), built_from=built_from)
        rows = slice(row * W, (row + 8) * W)
        assert _same(mine[rows], want["accum"][rows])


# variant 2: whole waves of more than a thread's worth (factor 16), or what the first
# bounce leaves (factor 1); 3, 4 and 5 leave their first bounce's rays to it
@pytest.mark.parametrize("n", [7167, 7168, 20_000])
@pytest.mark.parametrize("variant,factor", [(2, 1), (2, 16), (3, 1), (3, 16), (4, 1), (4, 16), (5, 1), (5, 16)])
def test_refilled_finishing_walks(venu, oracle, cuda, n, variant, factor):
    W, H, spp, sub, depth = 311, 101, 2, 1, 30
    threads = 128 * venu.core.sm_count()
    sp = oracle.scene_random(n, 21, (-40, 0, -40), (40, 12, 40))
    cam = oracle.camera((30, 10, 30), (0, 4, 0), 40.0, W / H, 0.05, 30.0)
    paths = W * H * spp
    assert threads < paths <= 16 * threads  # factor 16: the whole wave, more than a ray a thread
    if factor == 1:  # the first bounce is not the finishing kernel's, and leaves it more than that
        assert threads < _rays_at(oracle, sp, cam, W, H, spp, sub, 1) <= 16 * threads
    want = oracle.render(sp, cam, W, H, spp, subframe=sub, max_depth=depth, mode=pyoracle.MODE_GB300)
    ds = venu.DeviceScene(sp)
    wf = venu.Wavefront(0)
    wf.set_tuning(traverse_variant=variant, in_place_factor=factor, traverse_block=128, traverse_blocks_per_sm=1)
    acc = venu.new_accum(W, H)
    for _ in range(2):  # the second from the kept graph
        acc.fill_(1.0)
        wf.render(ds, cam, W, H, spp, acc, subframe=sub, max_depth=depth, reset=True)
        cuda.cuda.synchronize()
        assert _same(acc, want["accum"]) and wf.stats()["segments"] == want["segments"]


# one path fewer, as many, and one more than the grid has threads, and than it has at
# 16 a thread: the spreading kernel, the refilled walks, and a bounce before them
@pytest.mark.parametrize("per", [1, 16])
@pytest.mark.parametrize("more", [-1, 0, 1])
def test_finishing_walk_edges(venu, oracle, cuda, per, more):
    threads = 64 * venu.core.sm_count()
    paths = per * threads + more
    W = next(w for w in range(2, paths) if paths % w == 0)
    H = paths // W
    sp = oracle.scene_random(7300, 22, (-40, 0, -40), (40, 12, 40))
    cam = oracle.camera((30, 10, 30), (0, 4, 0), 40.0, 1.5, 0.05, 30.0)
    want = oracle.render(sp, cam, W, H, 1, subframe=2, max_depth=20, mode=pyoracle.MODE_GB300)
    ds = venu.DeviceScene(sp)
    wf = venu.Wavefront(0)
    wf.set_tuning(traverse_variant=2, in_place_factor=16, traverse_block=64, traverse_blocks_per_sm=1)
    acc = venu.new_accum(W, H)
    wf.render(ds, cam, W, H, 1, acc, subframe=2, max_depth=20, reset=True)
    cuda.cuda.synchronize()
    assert _same(acc, want["accum"]) and wf.stats()["segments"] == want["segments"]


@pytest.mark.parametrize("variant", [0, 3])
def test_split_bounce_after_the_first(venu, oracle, cuda, variant):
    """Later bounces of 2^20 rays and more, which the finishing kernel does not take,
    through k_traverse's up-front pass and k_walk."""
    W, H, spp, sub, depth = 1024, 1025, 2, 3, 5
    assert 2 * 128 * venu.core.sm_count() < 1 << 20  # what the finishing kernel takes at factor 2
    sp = oracle.scene_random(16384, 31)
    cam = oracle.camera((60, 15, 60), (0, 0, 0), 20.0, W / H, 0.1, 10.0)
    _check_large(venu, oracle, cuda, venu.DeviceScene(sp), sp, cam, W, H, spp, sub, depth,
                 dict(traverse_variant=variant, in_place_factor=2, traverse_block=128, traverse_blocks_per_sm=1),
                 split_from=1)


# The 4-wide tree: at 19456 rays left (2 a thread) the finishing kernel takes over, so
# the first bounces are k_trace_shade_wide's (4) or k_traverse's over that tree (5);
# the counting build of variant 4 stays on it to the end.
WIDE = [(4, False), (4, True), (5, False), (5, True)]


def _wide_render(venu, oracle, cuda, sp, cam, W, H, spp, depth, variant, count, bounces):
    threads = 64 * venu.core.sm_count()
    assert _rays_at(oracle, sp, cam, W, H, spp, 1, bounces - 1) > 2 * threads
    want = oracle.render(sp, cam, W, H, spp, subframe=1, max_depth=depth, mode=pyoracle.MODE_GB300)
    ds = venu.DeviceScene(sp)
    wf = venu.Wavefront(0, count=count)
    wf.set_tuning(traverse_variant=variant, in_place_factor=2, traverse_block=64, traverse_blocks_per_sm=1)
    acc = venu.new_accum(W, H)
    wf.render(ds, cam, W, H, spp, acc, subframe=1, max_depth=depth, reset=True)
    cuda.cuda.synchronize()
    st = wf.stats()  # raises on a stack error
    assert _same(acc, want["accum"]) and st["segments"] == want["segments"]


@pytest.mark.parametrize("variant,count", WIDE)
@pytest.mark.parametrize("name", ["giants", "four_hoisted", "two_huge", "hollow", "far"])
def test_wide_walk_edge_scenes(venu, oracle, cuda, name, variant, count):
    sp = _edge_scene(oracle, name)
    W, H, spp, depth = 192, 108, 12 if name == "far" else 4, 12
    c, r = sp["center"], np.abs(sp["radius"])
    far = name == "far"
    lo, hi = (c - r[:, None]).min(0), (c + r[:, None]).max(0)
    at = (lo + hi) / 2 if far else c.mean(0)
    eye = at + (np.array([12, 4, 11]) if far else np.array([70, 20, 65]))
    cam = oracle.camera(tuple(eye), tuple(at), 40.0, W / H, 0.1, 10.0)
    _wide_render(venu, oracle, cuda, sp, cam, W, H, spp, depth, variant, count, 1 if variant == 4 else 2)


@pytest.mark.parametrize("variant,count", WIDE)
@pytest.mark.parametrize("n,levels,rfrac,ks", DEEP)
def test_wide_walk_deep_stacks(venu, oracle, cuda, n, levels, rfrac, ks, variant, count):
    sp = _nested_scene(oracle, n, levels, rfrac)
    W, H, spp = 192, 108, 4
    cam = oracle.camera((150.0, 30.0, 150.0), (0, 0, 0), 20.0, W / H, 0.1, 10.0)
    _wide_render(venu, oracle, cuda, sp, cam, W, H, spp, 6, variant, count, 1 if variant == 4 else 2)


@pytest.mark.parametrize("variant,factor", [(0, 2), (2, 16), (3, 2), (4, 2)])
def test_refit_with_grown_extent(venu, oracle, cuda, variant, factor):
    """Moved spheres, some of them 1000 times as far as the built scene reaches, then
    renders through the split bounces (0, 3), the refilled finishing walks (2) and
    the 4-wide tree (4): the records follow, there and back."""
    large = variant in (0, 3)
    W, H, spp, sub, depth = (1024, 1025, 2, 1, 4) if large else (311, 101, 2, 1, 20)
    threads = 128 * venu.core.sm_count()
    assert 2 * threads < 1 << 20 and threads < 311 * 101 * 2 <= 16 * threads and 311 * 101 * 2 > 2 * threads
    sp = oracle.scene_random(20_000, 91)
    rng = np.random.default_rng(4)
    to = sp.copy()
    to["center"][1:] += rng.normal(size=(len(to) - 1, 3)).astype(np.float32)
    to["center"][[50, 9000, 19000]] = [[2e5, 0, 0], [0, 1e5, 1e5], [-1e5, 30, 0]]
    cam = oracle.camera((60, 15, 60), (0, 0, 0), 20.0, W / H, 0.1, 10.0)
    tuning = dict(traverse_variant=variant, in_place_factor=factor, traverse_block=128, traverse_blocks_per_sm=1)
    ds = venu.DeviceScene(sp)
    wf = venu.Wavefront(0)
    wf.set_tuning(**tuning)
    acc = venu.new_accum(W, H)
    wf.render(ds, cam, W, H, spp, acc, subframe=sub, max_depth=1, reset=True)  # the 4-wide tree is refit, too
    for pose in (to, sp):
        ds.update(pose)
        if large:
            _check_large(venu, oracle, cuda, ds, pose, cam, W, H, spp, sub, depth, tuning, built_from=sp,
                         split_from=0 if variant == 0 else 1)
            continue
        wf.render(ds, cam, W, H, spp, acc, subframe=sub, max_depth=depth, reset=True)
        cuda.cuda.synchronize()
        want = oracle.render(pose, cam, W, H, spp, subframe=sub, max_depth=depth, mode=pyoracle.MODE_GB300, built_from=sp)
        assert _same(acc, want["accum"]) and wf.stats()["segments"] == want["segments"]
    rays = np.concatenate([rng.uniform([-100, 0, -100], [100, 20, 100], (3000, 3)), rng.normal(size=(3000, 3))], 1)
    rays = rays.astype(np.float32)
    rays[:100, :3] = [150000.0, 5.0, 3.0]  # towards a far sphere
    rays[:100, 3:] = to["center"][50] - rays[:100, :3]
    ds.update(to)
    t, ids, _ = ds.trace(cuda.from_numpy(rays).cuda())
    wid, wt, _, _, _ = oracle.trace_bvh(to, rays)
    assert np.array_equal(ids.cpu().numpy(), wid) and np.array_equal(t.cpu().numpy().view(np.uint32), wt.view(np.uint32))
