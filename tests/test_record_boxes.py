"""The boxes of the traversal records and the fast walk's test of them
(frame_box, far_margin and Tracer::interval, meets), restated in float32 with
numpy and held against the oracle's full sphere test: wherever a sphere is hit,
its own box and any box around it must be met up to the hit's distance, for any
frame (G, E), with reciprocals an ulp off, unless the margin sends the ray to the
canonical walk."""
import numpy as np
import pytest

F = np.float32


def _down(x):
    r = x.astype(F)
    return np.where(r.astype(np.float64) > x, np.nextafter(r, F(-np.inf)), r)


def _up(x):
    return -_down(-x)


def _fma(a, b, c):
    return (a.astype(np.float64) * b.astype(np.float64) + c.astype(np.float64)).astype(F)


def _record(lo, hi, G, E):
    """frame_box: lo, hi (n, 3) float32 -> centres and half extents."""
    d = np.float64
    lo, hi = _down(lo.astype(d) - G.astype(d)), _up(hi.astype(d) - G.astype(d))
    far = np.maximum(np.abs(lo), np.abs(hi))
    e = ((far[:, 0] + far[:, 1]) + far[:, 2] + F(E)) * F(1.5 * 2.0**-20)
    c = F(0.5) * lo + F(0.5) * hi
    h = np.maximum(_up(hi.astype(d) - c.astype(d)), _up(c.astype(d) - lo.astype(d)))
    return c, _up(h.astype(d) + e.astype(d)[:, None])


def _interval(o, inv, G, E, c, h):
    p = G - o
    n0 = p * inv
    far = (np.abs(p[:, 0]) + np.abs(p[:, 1])) + np.abs(p[:, 2])
    m = np.maximum(_fma(far, F(2.0**-18), F(-(2.0**-18) * E)), F(0)) * np.abs(inv).max(1)
    tc = _fma(c, inv, n0)
    return _fma(h, -np.abs(inv), tc).max(1), _fma(h, np.abs(inv), tc).min(1), m


@pytest.mark.parametrize("r", [0.2, 1e-3, 30.0])
@pytest.mark.parametrize("at", [(0.0, 0.0, 0.0), (7.0, 0.2, -9.0), (1e4, 2.0, 3.0), (-1e5, 1e5, 40.0), (1e6, 0.0, 0.0)])
def test_hit_spheres_are_met(oracle, r, at):
    rng = np.random.default_rng(int(1000 * r) + int(abs(at[0])))
    m, tmin = 30000, F(0.001)
    C = np.array(at, F)
    sp = oracle.scene_random(1, 1)
    sp["center"][0], sp["radius"][0] = C, r
    # origins from beside the sphere to far away, towards its rim (from inside to
    # just past it), some along axes
    n = rng.normal(size=(m, 3))
    n /= np.linalg.norm(n, axis=1, keepdims=True)
    dist = r * 10.0 ** rng.uniform(0.0, 5.0, m)
    o = (C + n * dist[:, None]).astype(F)
    u = np.cross(n, rng.normal(size=(m, 3)))
    u /= np.linalg.norm(u, axis=1, keepdims=True)
    rim = C.astype(np.float64) + u * (r * (1.0 + rng.choice([-0.5, -1e-3, -1e-6, 0.0, 1e-6, 1e-4], m)))[:, None]
    d = (rim - o) * 10.0 ** rng.uniform(-2, 2, (m, 1))
    k = m // 5
    axis = rng.integers(0, 3, k)
    d[np.arange(k), axis] *= rng.choice([0.0, 1e-7, 1e-4], k)
    d = d.astype(F)
    ids, t = oracle.trace_bvh(sp, np.concatenate([o, d], 1), float(tmin), 1e16)[:2]
    hit = ids == 0
    assert hit.sum() > m // 4
    d0 = np.where(np.abs(d) < F(1e-20), np.copysign(F(1e-20), d), d)
    inv = F(1.0) / d0
    inv = np.choose(rng.integers(0, 3, inv.shape), [inv, np.nextafter(inv, inv * F(2)), np.nextafter(inv, F(0))])
    # its own box; one that another sphere nearby extends; one that a far one does
    R = F(r)
    lo = np.repeat(_down(C.astype(np.float64) - float(R))[None], m, 0)
    hi = np.repeat(_up(C.astype(np.float64) + float(R))[None], m, 0)
    boxes = [(lo, hi)]
    for size in (5.0 * r, 3e3, 3e6):
        other = (C + rng.normal(size=(m, 3)) * size).astype(F)
        boxes.append((np.minimum(lo, other), np.maximum(hi, other)))
    tested = 0
    for G, E in ((C, 0.0), (C, 20 * r), (C + F(3 * r), 1e3 * r), (np.zeros(3, F), float(np.linalg.norm(C)) + r),
                 (np.array([5.0, -30.0, 2.0], F), 10.0)):
        for blo, bhi in boxes:
            c, h = _record(blo, bhi, G.astype(F), E)
            near, far, margin = _interval(o, inv, G.astype(F), E, c, h)
            met = np.maximum(near, tmin) <= np.minimum(far, t) + margin
            walked = margin <= F(1.0)
            assert (met | ~(hit & walked)).all()
            tested += int((hit & walked).sum())
    assert tested > 5 * m // 2
