"""GPU tests of scenes that are updated while other streams and threads use them."""
import threading

import numpy as np
import pytest

from oracle import pyoracle

pytestmark = pytest.mark.gpu


def _moved(spheres, seed, scale):
    rng = np.random.default_rng(seed)
    out = spheres.copy()
    out["center"][1:] += (rng.normal(size=(len(out) - 1, 3)) * scale).astype(np.float32)
    return out


def test_host_updates_beside_renders(venu, oracle, cuda):
    """Spheres uploaded by venu_scene_update while renders of the scene run on
    another stream: those renders may see old and new spheres mixed but end
    without an error, and once both are through the scene is the last update's."""
    torch = cuda
    n, W, H, spp, depth = 30_000, 320, 180, 4, 8
    sp = oracle.scene_random(n, 72)
    last = _moved(sp, 9, 0.3)
    cam = oracle.camera((60, 15, 60), (0, 0, 0), 20.0, W / H, 0.1, 10.0)
    ds = venu.DeviceScene(sp)
    bytes0 = ds.info()["device_bytes"]
    waves = []
    for variant in (2, 3, 4):
        wf = venu.Wavefront(0)
        wf.set_tuning(traverse_variant=variant, traverse_blocks_per_sm=1)
        waves.append((wf, venu.new_accum(W, H), torch.cuda.Stream()))
        wf.render(ds, cam, W, H, spp, waves[-1][1], subframe=1, max_depth=depth, reset=True)
    torch.cuda.synchronize()
    side = torch.cuda.Stream()
    for k in range(12):
        for wf, acc, st in waves:
            wf.render(ds, cam, W, H, spp, acc, subframe=1, max_depth=depth, reset=True, stream=st)
        ds.update(_moved(sp, k, 0.3), stream=side)
    torch.cuda.synchronize()
    for wf, _, _ in waves:
        wf.stats()  # raises on a traversal error
    ds.update(last)
    assert ds.info()["device_bytes"] >= bytes0 + 48 * n  # the upload's memory is counted
    assert np.array_equal(ds.export_bvh()["nodes"].view(np.uint32), oracle.lbvh_refit(sp, last).view(np.uint32))
    want = oracle.render(last, cam, W, H, spp, subframe=1, max_depth=depth, mode=pyoracle.MODE_GB300)
    for wf, acc, _ in waves:
        wf.render(ds, cam, W, H, spp, acc, subframe=1, max_depth=depth, reset=True)
        torch.cuda.synchronize()
        assert np.array_equal(acc.cpu().numpy().view(np.uint32), want["accum"].view(np.uint32))


def test_host_updates_from_threads(venu, oracle, cuda):
    """Updates to the same pose from several threads and streams: whichever comes
    last, the scene has that pose."""
    n = 20_000
    sp = oracle.scene_random(n, 73)
    to = _moved(sp, 3, 0.5)
    ds = venu.DeviceScene(sp)
    failed = []

    def work():
        s = cuda.cuda.Stream()
        try:
            for _ in range(10):
                ds.update(to, stream=s)
        except venu.VenuError as e:
            failed.append(e)

    threads = [threading.Thread(target=work) for _ in range(4)]
    for th in threads:
        th.start()
    for th in threads:
        th.join()
    assert not failed
    assert np.array_equal(ds.export_bvh()["nodes"].view(np.uint32), oracle.lbvh_refit(sp, to).view(np.uint32))


def test_overlapping_refits_leave_no_trace(venu, oracle, cuda):
    """Refits of one scene from two streams at once, all to the same pose: the scene
    has that pose afterwards, and a later refit is exact."""
    torch = cuda
    n = 60_000
    sp = oracle.scene_random(n, 71)
    a, b = _moved(sp, 1, 0.5), _moved(sp, 2, 0.5)
    want_a, want_b = oracle.lbvh_refit(sp, a), oracle.lbvh_refit(sp, b)
    ds = venu.DeviceScene(sp)
    dev_a = torch.from_numpy(a.view(np.uint8).copy()).cuda()
    dev_b = torch.from_numpy(b.view(np.uint8).copy()).cuda()
    torch.cuda.synchronize()
    streams = [torch.cuda.Stream() for _ in range(2)]
    for _ in range(30):
        for s in streams:
            for _ in range(4):
                ds.update_device(dev_a, n, stream=s)
    torch.cuda.synchronize()
    assert np.array_equal(ds.export_bvh()["nodes"].view(np.uint32), want_a.view(np.uint32))
    ds.update_device(dev_b, n)
    torch.cuda.synchronize()
    assert np.array_equal(ds.export_bvh()["nodes"].view(np.uint32), want_b.view(np.uint32))


def test_captured_refit(venu, oracle, cuda):
    """A refit captured into a graph replays beside refits that are launched, and
    alone."""
    torch = cuda
    n = 60_000
    sp = oracle.scene_random(n, 74)
    a, b = _moved(sp, 1, 0.5), _moved(sp, 2, 0.5)
    want_a, want_b = oracle.lbvh_refit(sp, a), oracle.lbvh_refit(sp, b)
    ds = venu.DeviceScene(sp)
    dev = torch.from_numpy(a.view(np.uint8).copy()).cuda()
    dev_b = torch.from_numpy(b.view(np.uint8).copy()).cuda()
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        ds.update_device(dev, n)
    side = torch.cuda.Stream()
    for _ in range(20):
        graph.replay()
        ds.update_device(dev, n, stream=side)
    torch.cuda.synchronize()
    assert np.array_equal(ds.export_bvh()["nodes"].view(np.uint32), want_a.view(np.uint32))
    ds.update_device(dev_b, n)
    torch.cuda.synchronize()
    assert np.array_equal(ds.export_bvh()["nodes"].view(np.uint32), want_b.view(np.uint32))
    graph.replay()
    torch.cuda.synchronize()
    assert np.array_equal(ds.export_bvh()["nodes"].view(np.uint32), want_a.view(np.uint32))


def test_updates_beside_the_first_wide_render(venu, oracle, cuda):
    """The 4-wide tree, built by the first render that asks for it, while another
    thread moves the spheres: afterwards it is that of the last pose."""
    torch = cuda
    n, W, H, spp, depth = 20_000, 96, 54, 2, 10
    sp = oracle.scene_random(n, 75)
    to = _moved(sp, 5, 0.5)
    cam = oracle.camera((60, 15, 60), (0, 0, 0), 20.0, W / H, 0.1, 10.0)
    want = oracle.render(to, cam, W, H, spp, subframe=1, max_depth=depth, mode=pyoracle.MODE_GB300, built_from=sp)
    dev = torch.from_numpy(to.view(np.uint8).copy()).cuda()
    torch.cuda.synchronize()
    for _ in range(8):
        ds = venu.DeviceScene(sp)
        started = threading.Event()
        failed = []

        def move():
            s = torch.cuda.Stream()
            try:
                for k in range(40):
                    ds.update_device(dev, n, stream=s)
                    started.set()
                s.synchronize()
            except venu.VenuError as e:
                failed.append(e)

        th = threading.Thread(target=move)
        th.start()
        started.wait()
        wf = venu.Wavefront(0, count=True)  # counting renders of variant 4 walk the 4-wide tree to the end
        wf.set_tuning(traverse_variant=4)
        acc = venu.new_accum(W, H)
        side = torch.cuda.Stream()
        wf.render(ds, cam, W, H, spp, acc, subframe=1, max_depth=depth, reset=True, stream=side)
        side.synchronize()
        th.join()
        wf.stats()  # raises on a traversal error
        assert not failed
        wf.render(ds, cam, W, H, spp, acc, subframe=1, max_depth=depth, reset=True)
        torch.cuda.synchronize()
        assert np.array_equal(acc.cpu().numpy().view(np.uint32), want["accum"].view(np.uint32))
        ds.close()
