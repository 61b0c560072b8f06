"""The rule by which a ray skips the test of the sphere it leaves (left_behind in
venu_device.cuh), restated in float32 with numpy and held against the oracle's
full test: no ray that the rule passes over may hit."""
import numpy as np
import pytest

F = np.float32


def _left_behind(o, d, c, r, tmin):
    with np.errstate(over="ignore", invalid="ignore", under="ignore"):
        h = o - c
        a = (d * d).sum(1, dtype=F)
        hb = (h * d).sum(1, dtype=F)
        hh = (h * h).sum(1, dtype=F)
        r2 = F(r) * F(r)
        return ((hb > F(1e-15)) & (hb * hb > hh * a * F(2.0**-30))
                & ((hh - r2) - (hh + r2) * F(2.0**-22) > hb * F(tmin) * F(-0.99)))


@pytest.mark.parametrize("r", [1000.0, 1.0, -0.2, 0.2, 1e-3, 1e-7, 1e6, 3e18])
@pytest.mark.parametrize("off", [0.0, 40.0])
def test_left_behind_never_drops_a_hit(oracle, r, off):
    rng = np.random.default_rng(int(abs(np.log2(abs(r))) * 100) + int(off))
    m, R, tmin = 40000, abs(r), 0.001
    c = np.array([off, -R, 0.3 * off], F)
    n = rng.normal(size=(m, 3))
    n /= np.linalg.norm(n, axis=1, keepdims=True)
    if R > 100:  # near one point of a huge sphere, as rays that leave the ground are
        n[: m // 2, 1] += 50.0
        n /= np.linalg.norm(n, axis=1, keepdims=True)
    # origins from on the surface to an r-th off it, on both sides
    depth = rng.choice([0.0, 1e-8, 1e-7, 1e-6, 1e-5, 1e-3, 0.06], m) * rng.choice([-1.0, 1.0], m)
    o = (c.astype(np.float64) + n * R * (1.0 + depth)[:, None]).astype(F)
    u = rng.normal(size=(m, 3))
    u /= np.linalg.norm(u, axis=1, keepdims=True)
    d = n + u * rng.choice([0.1, 1.0, 1.0, 30.0], m)[:, None]
    k = m // 4  # grazing
    t = u[:k] - (u[:k] * n[:k]).sum(1, keepdims=True) * n[:k]
    d[:k] = t + n[:k] * 10.0 ** rng.uniform(-9, -1, (k, 1))
    d = (d * rng.choice([1.0, 1e-6, 1e4], m)[:, None]).astype(F)
    sp = oracle.scene_random(1, 1)
    sp["center"][0] = c
    sp["radius"][0] = r
    ids = oracle.trace_bvh(sp, np.concatenate([o, d], 1), tmin, 1e16)[0]
    skipped = _left_behind(o, d, c, r, tmin)
    assert not (skipped & (ids >= 0)).any()
    if 1e-3 <= R <= 1000:  # and it does pass over most rays that head outwards
        assert skipped.sum() > m // 4
