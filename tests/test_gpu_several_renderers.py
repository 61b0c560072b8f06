"""GPU tests of renderers and batches of different launch shapes that live at the
same time: what one of them sets up must not change what another launches."""
import numpy as np
import pytest

from oracle import pyoracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("variant", [0, 1, 2, 3, 4, 5])
def test_renderers_of_different_blocks(venu, oracle, cuda, variant):
    """A renderer with blocks of 256 threads renders after one with blocks of 64
    has been set up: a scene above 4096 spheres, so its kernels ask for the
    deep stack's 16 KB, four times as much as the other's."""
    sp = oracle.scene_random(5000, 61)
    W, H, spp, depth = 311, 251, 4, 6  # more paths than a grid of one block an SM finishes at once
    cam = oracle.camera((60, 15, 60), (0, 0, 0), 20.0, W / H, 0.1, 10.0)
    want = oracle.render(sp, cam, W, H, spp, subframe=1, max_depth=depth, mode=pyoracle.MODE_GB300)
    ds = venu.DeviceScene(sp)
    big = venu.Wavefront(0)
    big.set_tuning(traverse_variant=variant, traverse_block=256, traverse_blocks_per_sm=1)
    small = venu.Wavefront(0)
    small.set_tuning(traverse_variant=variant, traverse_block=64, traverse_blocks_per_sm=1)
    for wf in (big, small, big):
        acc = venu.new_accum(W, H)
        wf.render(ds, cam, W, H, spp, acc, subframe=1, max_depth=depth, reset=True)
        cuda.cuda.synchronize()
        assert np.array_equal(acc.cpu().numpy().view(np.uint32), want["accum"].view(np.uint32))
        assert wf.stats()["segments"] == want["segments"]


def test_batches_of_different_blocks(venu, oracle, cuda):
    sp = oracle.scene_random(5000, 62)
    W, H, spp, depth = 64, 48, 2, 8
    cam = oracle.camera((60, 15, 60), (0, 0, 0), 20.0, W / H, 0.1, 10.0)
    want = oracle.render(sp, cam, W, H, spp, subframe=1, max_depth=depth, mode=pyoracle.MODE_GB300)
    ds = venu.DeviceScene(sp)
    big, small = venu.Batch(pool_paths=4000, max_jobs=2), venu.Batch(pool_paths=4000, max_jobs=2)
    big.set_tuning(traverse_block=256)
    small.set_tuning(traverse_block=64)
    for b in (big, small, big):
        acc = venu.new_accum(W, H)
        b.submit(ds, cam, W, H, spp, acc, subframe=1, max_depth=depth)
        b.run()
        assert len(b.collect()) == 1
        cuda.cuda.synchronize()
        assert np.array_equal(acc.cpu().numpy().view(np.uint32), want["accum"].view(np.uint32))
