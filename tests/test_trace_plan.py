"""The launch shape of ray queries (trace_plan, built for the host): every ray has a
lane, up to the largest count that venu_trace takes."""
import os
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CUDA = os.environ.get("CUDA_HOME", "/usr/local/cuda")
FILL = 152 * 16  # warps that put four on every scheduler's SM


@pytest.fixture(scope="module")
def plan(tmp_path_factory):
    exe = str(tmp_path_factory.mktemp("plan") / "trace_plan")
    cmd = ["g++", "-std=c++17", "-O2", "-I", os.path.join(ROOT, "venusaur_gb300", "csrc"), "-I",
           os.path.join(CUDA, "include"), os.path.join(ROOT, "tests", "cpp", "trace_plan.cpp"), "-o", exe,
           "-L", os.path.join(CUDA, "lib64"), "-lcudart"]
    r = subprocess.run(cmd, capture_output=True, text=True)
    assert r.returncode == 0, r.stderr

    def run(cases):
        args = [str(int(x)) for c in cases for x in c]
        r = subprocess.run([exe] + args, capture_output=True, text=True,
                           env=dict(os.environ, LD_LIBRARY_PATH=os.path.join(CUDA, "lib64")))
        assert r.returncode == 0, (r.returncode, r.stderr)
        return [tuple(int(x) for x in line.split()) for line in r.stdout.splitlines()]

    return run


def test_every_ray_has_a_lane(plan):
    top = 2**32 - 1
    counts = [1, 31, 32, 33, FILL - 1, FILL, FILL + 1, 31 * FILL, 31 * FILL + 1, 32 * FILL, 10**6, 2**31, 2**31 + 1,
              top - 4 * FILL, top - FILL, top - FILL + 2, top - FILL + 3, top - 200, top - 127, top - 1, top]
    cases = [(s, n, b) for n in counts for s in (0, 485, 65535, 65536, 2**28) for b in (0, 1)]
    for (spheres, n, both), (per_warp, grid, walk) in zip(cases, plan(cases)):
        assert 1 <= per_warp <= 32 and grid >= 1
        assert grid * 4 * per_warp >= n > (grid - 1) * 4 * per_warp
        assert grid * 128 <= 2**32  # thread numbers fit 32 bits
        assert walk == (both and spheres >= 65536 and 2**18 <= n <= 2**31)
        if n >= 32 * FILL or walk:
            assert per_warp == 32
