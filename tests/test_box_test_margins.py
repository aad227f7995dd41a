"""The box tests of the distance kernels (csrc/cmg_sdf.cuh: box_ball, box_disc, cell_disc)
restated in FP32: a triangle that can matter to a cell of a box is never dropped. Cells,
triangles (well shaped, slivers, points, collinear) and surface points are drawn over
scales; the truth is the FP64 point-triangle distance: a triangle matters to cell p when
its distance is at most |p - q| + eps (box tests) or the cell's bound (cell test)."""
import numpy as np
import pytest

F = np.float32
U = F(2.0 ** -24)


def _dist(p, a, b, c):
    """FP64 distance of points p (n, 3) from the triangle (a, b, c)."""
    best = np.full(len(p), np.inf)
    for u, v in ((a, b), (b, c), (c, a)):
        d = v - u
        t = np.clip(((p - u) @ d) / max(d @ d, 1e-300), 0, 1)
        best = np.minimum(best, np.linalg.norm(p - (u + t[:, None] * d), axis=1))
    n = np.cross(b - a, c - a)
    nn = n @ n
    if nn > 0:
        wb = np.cross(p - a, c - a) @ n / nn
        wc = np.cross(b - a, p - a) @ n / nn
        best = np.where((wb >= 0) & (wc >= 0) & (wb + wc <= 1), np.abs((p - a) @ n) / np.sqrt(nn), best)
    return best


def _box(q, h, r, eps, pos):
    q2 = F((q * q).sum(dtype=F))
    qr = F((np.sqrt(q2) + r + eps) * (1 + 8 * U))
    e2 = F(eps * (2 * qr + eps) * (1 + 8 * U))
    add = F(64 * U * (q2 + r * r) + 8 * pos * (qr + pos) + F(1e-36))
    return q, h, q2, F(r * r), qr, e2, add


def _ball(box, c, w, pos):
    q, h, q2, r2, qr, e2, add = box
    c2 = F((c * c).sum(dtype=F))
    lin = F(F(-2) * F((h * np.abs(c - q)).sum(dtype=F)) + (c2 - q2))
    m = F(64 * U * c2 + (8 * pos * w + add))
    return not lin > F(w * (1 + 32 * U) * (2 * qr + w) + e2 + m)


def _disc(box, c, w, n, nerr):
    q, h, q2, r2, qr, e2, add = box
    c2 = F((c * c).sum(dtype=F))
    lin = F(F(-2) * F((h * np.abs(c - q)).sum(dtype=F)) + (c2 - q2))
    m = F((64 * U + 8 * nerr) * (c2 + r2) + (8 * nerr * q2 + add))
    nc = F((n * c).sum(dtype=F))
    gs = F((h * np.abs(nc * n - q)).sum(dtype=F))
    s2 = F(F(2) * gs + (q2 + r2 - nc * nc) + (e2 + m))
    s = F(np.sqrt(max(s2, F(0))))
    return not s2 < 0 and not lin > F(w * (1 + 32 * U) * (2 * s + w) + e2 + m)


def _cell(d2, pn, b, w):
    s = F(np.sqrt(max(F((b - abs(pn)) * (b + abs(pn))), F(0))))
    return abs(pn) <= b and not d2 > F(F(w * (2 * s + w) + b * b) * (1 + 16 * U))


def _triangle(rng, size):
    v = rng.normal(size=(3, 3)) * size
    k = rng.integers(5)
    if k == 1:
        v[2] = v[1] + (v[1] - v[0]) * 1e-4 + rng.normal(size=3) * size * 1e-7   # sliver
    elif k == 2:
        v[2] = 0.5 * (v[0] + v[1])                                              # collinear
    elif k == 3:
        v[1] = v[2] = v[0]                                                      # a point
    elif k == 4:
        v[:, 2] = v[0, 2]                                                       # axis-parallel
    return v - v.mean(0)


@pytest.mark.parametrize("half", [(1.5, 1.5, 1.5), (1.5, 1.5, 0.5), (7.5, 7.5, 7.5), (0.0, 0.0, 0.0)])
def test_no_triangle_that_matters_is_dropped(half):
    rng = np.random.default_rng(11)
    matters = dropped_far = far = 0
    for _ in range(1000):
        h = np.array(half) * 10.0 ** rng.uniform(-3, 1)
        hf = h.astype(F)
        r = F(np.linalg.norm(h) * (1 + 1e-9))
        r = np.nextafter(r, F(np.inf))
        far_off = 10.0 ** rng.uniform(-1, 2) * max(float(r), 1e-3)
        q = (rng.normal(size=3) * far_off).astype(F)
        size = 10.0 ** rng.uniform(-2, 0.5) * max(float(r), 1e-3)
        tri = _triangle(rng, size)
        # centres near the sphere of the surface point's distance: the deciding region
        d = rng.normal(size=3)
        d *= np.linalg.norm(q) * rng.choice([0.9, 1.0, 1.0, 1.02, 1.3]) / np.linalg.norm(d)
        if rng.random() < 0.5:
            d = q + rng.normal(size=3) * size * rng.choice([0.5, 2, 5])
        c = d.astype(F)
        V = tri + c.astype(np.float64)
        w = np.nextafter(F(np.linalg.norm(tri, axis=1).max() * (1 + 1e-12)), F(np.inf))
        n = np.cross(tri[1] - tri[0], tri[2] - tri[0])
        nl = np.linalg.norm(n)
        lu, lv = np.linalg.norm(tri[1] - tri[0]), np.linalg.norm(tri[2] - tri[0])
        nerr = F(50 * 1.1102230246251565e-16 * lu * lv / nl + 1.2e-7) if nl > 0 else F(0)
        n = (n / nl if nl > 0 else n * 0).astype(F)
        eps = F(200 * U * (np.linalg.norm(q) + r + w))
        box = _box(q, hf, r, eps, F(0))
        corners = np.array([[i, j, k] for i in (-1, 1) for j in (-1, 1) for k in (-1, 1)])
        p = np.concatenate([corners * h, rng.uniform(-1, 1, size=(24, 3)) * h])
        dist = _dist(p, *V)
        bound = np.linalg.norm(p - q.astype(np.float64), axis=1) + float(eps)
        keep_ball, keep_disc = _ball(box, c, w, F(0)), _disc(box, c, w, n, nerr)
        if (dist <= bound).any():
            matters += 1
            assert keep_ball and keep_disc
        elif dist.min() > bound.max() + float(w):
            far += 1
            dropped_far += not keep_disc
        # the cell test: the cell's bound at, just above and well above the distance
        unit = n if nl > 0 else np.array([0, 0, 1], F)
        reach = F(w * (1 + 20 * U) + 17 * U * r)
        for i in range(0, len(p), 5):
            pf = p[i].astype(F)
            o = (pf - c).astype(F)
            true = float(_dist(pf[None].astype(np.float64), *V)[0])
            for b in (np.nextafter(F(true), F(np.inf)), F(true * 1.01)):
                pr = F(F(b + 4 * (w + r)) * (F(2.4e-7) + 64 * U) + b)
                pn = F((o * unit).sum(dtype=F))
                if nl > 0 and nerr > 2.4e-7:  # the record's frame normal is rounded only
                    continue
                if nl == 0:
                    # a frame of the kernel's choosing holds the collinear triangle
                    e = tri[np.argmax(np.linalg.norm(tri, axis=1))]
                    a = np.cross(e, [1.0, 0, 0]) if abs(e[0]) <= np.abs(e).max() * 0.9 else np.cross(e, [0, 1.0, 0])
                    a = a / np.linalg.norm(a) if np.linalg.norm(a) > 0 else np.array([0, 0, 1.0])
                    pn = F((o * a.astype(F)).sum(dtype=F))
                assert _cell(F((o * o).sum(dtype=F)), pn, pr, reach)
    assert matters > 100
    assert far == 0 or dropped_far > far // 2  # the tests do drop
