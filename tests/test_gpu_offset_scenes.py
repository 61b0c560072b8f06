"""GPU tests of scenes away from the origin and of scenes with a far sphere: their
boxes must cull as those of the same scene at the origin do."""
import numpy as np
import pytest

from oracle import pyoracle

pytestmark = pytest.mark.gpu

W, H, SPP, DEPTH = 96, 54, 2, 20


def _render(venu, torch, ds, cam, variant, count=False):
    wf = venu.Wavefront(0, count=count)
    wf.set_tuning(traverse_variant=variant)
    acc = venu.new_accum(W, H)
    wf.render(ds, cam, W, H, SPP, acc, subframe=1, max_depth=DEPTH, reset=True)
    torch.cuda.synchronize()
    return acc.cpu().numpy().view(np.uint32), wf.stats()


def _tests_per_segment(venu, torch, ds, cam, want):
    """Box and sphere tests a segment of the 4-wide walk, whose boxes are the
    binary records'; every walk's image is the oracle's."""
    acc, st = _render(venu, torch, ds, cam, 4, count=True)
    assert np.array_equal(acc, want["accum"].view(np.uint32)) and st["segments"] == want["segments"]
    for variant in (2, 3):
        assert np.array_equal(_render(venu, torch, ds, cam, variant)[0], want["accum"].view(np.uint32)), variant
    return st["nodes_visited"] / st["segments"], st["spheres_tested"] / st["segments"]


# A box is widened by a few units in the last place of its own distance from the
# scene's middle and of the scene's radius, neither of which an offset or a few far
# spheres change by more than the rounding of the spheres themselves (0.03 at 1e6,
# against radii of 0.2): half as many tests again is far above that.
@pytest.mark.parametrize("shift", [1e4, 1e5, 1e6])
def test_offset_scene_culls(venu, oracle, cuda, shift):
    tests = []
    for at in (0.0, shift):
        sp = oracle.scene_rtiow(0)
        sp["center"][:, 0] += np.float32(at)
        cam = oracle.camera((13 + at, 2, 3), (at, 0, 0), 20.0, W / H, 0.1, 10.0)
        want = oracle.render(sp, cam, W, H, SPP, subframe=1, max_depth=DEPTH, mode=pyoracle.MODE_GB300)
        tests.append(_tests_per_segment(venu, cuda, venu.DeviceScene(sp), cam, want))
    (nodes0, spheres0), (nodes, spheres) = tests
    assert nodes < 1.5 * nodes0 and spheres < 1.5 * spheres0


def test_far_spheres_keep_the_rest_culling(venu, oracle, cuda):
    """Three spheres moved 1e5 to 3e6 away: the same tree, whose other boxes cull as
    before.  (The boxes above the three are met by most rays, in any walk: the
    4-wide walk's tests are counted against the canonical one's.)"""
    sp = oracle.scene_random(3000, 81, (-40, 0, -40), (40, 12, 40))
    far = sp.copy()
    far["center"][[100, 1500, 2900]] = [[0, 0, 3e6], [-1e5, 0, 0], [0, 2e6, 0]]
    cam = oracle.camera((30, 10, 30), (0, 4, 0), 40.0, W / H, 0.05, 30.0)
    tests = []
    for now in (sp, far):
        ds = venu.DeviceScene(sp)
        ds.update(now)
        want = oracle.render(now, cam, W, H, SPP, subframe=1, max_depth=DEPTH, mode=pyoracle.MODE_GB300, built_from=sp)
        nodes, spheres = _tests_per_segment(venu, cuda, ds, cam, want)
        tests.append((nodes * want["segments"] / want["nodes"], spheres * want["segments"] / want["spheres"]))
    (nodes0, spheres0), (nodes, spheres) = tests
    assert nodes < 1.5 * nodes0 and spheres < 1.5 * spheres0
