"""The distance kernels' pruning tests, compiled from csrc/cmg_sdf.cuh itself
(tests/cpp/box_tests.cpp), with the normals the records hold: each triangle's own frame as
k_sdf_tri_prep builds it, rounded to FP32, and the one error bound of every record. Slivers
of every aspect, down to triangles that the preparation takes as collinear, are drawn beside
well shaped ones: none that can matter to a cell is dropped. Without the margins some are."""
import ctypes
import os
import subprocess

import numpy as np
import pytest

from conftest import ROOT

F = np.float32
L = np.longdouble
U = F(2.0 ** -24)


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    from cybermeshgenerator_gb300 import build
    so = str(tmp_path_factory.mktemp("box") / "libbox.so")
    cuda = os.path.join(build._cuda_home(build._nvcc()), "include")
    r = subprocess.run(["g++", "-std=c++17", "-O2", "-w", "-ffp-contract=off", "-shared", "-fPIC", "-I", build.CSRC,
                        "-I", cuda, os.path.join(ROOT, "tests", "cpp", "box_tests.cpp"), "-o", so],
                       capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    so = ctypes.CDLL(so)
    fp, f = ctypes.POINTER(ctypes.c_float), ctypes.c_float
    so.normal_error.restype = f
    so.ball.argtypes = [fp, fp, f]
    so.disc.argtypes = [fp, fp, f, fp, f]
    so.cell.argtypes = [f, f, f, f]
    return so


def _p(a):
    return a.ctypes.data_as(ctypes.POINTER(ctypes.c_float))


def _frame_normal(a, b, c):
    """The record's normal: u along b - a (else c - a, else x), v from c - a by two
    Gram-Schmidt passes, any direction across u for a collinear triangle."""
    e, f = b - a, c - a
    le, lf = np.linalg.norm(e), np.linalg.norm(f)
    u = e / le if le > 0 else (f / lf if lf > 0 else np.array([1.0, 0, 0]))
    r = f - (f @ u) * u
    r = r - (r @ u) * u
    h = np.linalg.norm(r)
    if h > 1e-9 * max(le, lf):
        v = r / h
    else:
        axis = np.eye(3)[np.argmin(np.abs(u))]
        v = np.cross(axis, u)
        v /= np.linalg.norm(v)
    return np.cross(u, v).astype(F)


def _dist(p, a, b, c):
    """The distance of points p (n, 3) from the triangle, in extended precision."""
    p, a, b, c = (x.astype(L) for x in (p, a, b, c))
    best = np.full(len(p), np.inf, dtype=L)
    for u, v in ((a, b), (b, c), (c, a)):
        d = v - u
        dd = (d * d).sum()
        t = np.clip(((p - u) * d).sum(1) / dd, 0, 1) if dd > 0 else np.zeros(len(p), L)
        best = np.minimum(best, np.sqrt((((p - (u + t[:, None] * d))) ** 2).sum(1)))
    n = np.cross(b - a, c - a)
    nn = (n * n).sum()
    if nn > 0:
        wb = (np.cross(p - a, c - a) * n).sum(1) / nn
        wc = (np.cross(b - a, p - a) * n).sum(1) / nn
        inside = (wb >= 0) & (wc >= 0) & (wb + wc <= 1)
        best = np.where(inside, np.minimum(best, np.abs(((p - a) * n).sum(1)) / np.sqrt(nn)), best)
    return best


def _triangle(rng, size):
    v = rng.normal(size=(3, 3)) * size
    k = rng.integers(6)
    if k < 3:  # slivers: a corner near the opposite edge, or next to another corner
        width = size * 10.0 ** rng.uniform(-13, -1)
        v[2] = v[0] + (v[1] - v[0]) * rng.choice([0.0, 0.5, 0.9999, 1.0, 1.5]) + rng.normal(size=3) * width
    elif k == 3:
        v[2] = 0.5 * (v[0] + v[1])
    elif k == 4:
        v[:, 2] = v[0, 2]
    v = v - v.mean(0)
    return v[rng.permutation(3)]


def _draw(rng, half):
    """A box, a surface point, a triangle near the sphere where the tests decide."""
    h = np.array(half) * 10.0 ** rng.uniform(-3, 1)
    r = np.nextafter(F(np.linalg.norm(h) * (1 + 1e-9)), F(np.inf))
    unit = max(float(r), 1e-3)
    q = (rng.normal(size=3) * 10.0 ** rng.uniform(-1, 2) * unit).astype(F)
    tri = _triangle(rng, 10.0 ** rng.uniform(-2, 1) * unit)
    d = rng.normal(size=3)
    d *= np.linalg.norm(q) * rng.choice([0.9, 1.0, 1.0, 1.02, 1.3]) / np.linalg.norm(d)
    if rng.random() < 0.5:
        d = q + rng.normal(size=3) * np.linalg.norm(tri, axis=1).max() * rng.choice([0.5, 2, 5])
    c = d.astype(F)
    w = np.nextafter(F(np.linalg.norm(tri, axis=1).max() * (1 + 1e-12)), F(np.inf))
    corners = np.array([[i, j, k] for i in (-1, 1) for j in (-1, 1) for k in (-1, 1)])
    p = np.concatenate([corners * h, rng.uniform(-1, 1, size=(16, 3)) * h])
    return h, r, q, tri, c, w, p


@pytest.mark.parametrize("half", [(1.5, 1.5, 1.5), (1.5, 1.5, 0.5), (7.5, 7.5, 7.5), (0.0, 0.0, 0.0)])
def test_no_triangle_that_matters_is_dropped(lib, half):
    rng = np.random.default_rng(23)
    nerr = F(lib.normal_error())
    matters = thin = 0
    for _ in range(1500):
        h, r, q, tri, c, w, p = _draw(rng, half)
        V = tri + c.astype(np.float64)
        n = _frame_normal(*tri)
        eps = F(200 * U * (np.linalg.norm(q) + r + w))
        box = np.concatenate([q, h.astype(F), [r, eps, F(0)]]).astype(F)
        dist = _dist(p, *V)
        bound = np.linalg.norm((p - q.astype(np.float64)).astype(L), axis=1) + L(eps)
        if (dist <= bound).any():
            matters += 1
            area = np.linalg.norm(np.cross(tri[1] - tri[0], tri[2] - tri[0]))
            thin += area < 1e-4 * float(w) ** 2
            assert lib.ball(_p(box), _p(c), w)
            assert lib.disc(_p(box), _p(c), w, _p(n), nerr)
        # one cell: its bound at, just above and well above the distance, widened as the kernel
        # widens it (plane_reach over bound, triangle and sub-brick radius; reach_term)
        reach = F(w * (1 + 20 * U) + 17 * U * r)
        a = tri[0].astype(F)
        for i in range(0, len(p), 5):
            o = (p[i].astype(F) - c).astype(F)
            pn = F(((o - a) * n).sum(dtype=F))
            true = _dist(p[i].astype(F).astype(np.float64)[None], *V)[0]
            for b in (np.nextafter(F(true), F(np.inf)), F(true * L(1.01))):
                pr = F(F(b + 4 * (w + r)) * (nerr + 64 * U) + b)
                assert lib.cell(F((o * o).sum(dtype=F)), pn, pr, reach)
    assert matters > 150 and thin > 50


def test_the_tests_do_drop(lib):
    """Far triangles are dropped, and with a cell's bound that is not widened so are some that
    matter: what keeps them above is the margin."""
    rng = np.random.default_rng(29)
    far = dropped = lost = 0
    for _ in range(3000):
        h, r, q, tri, c, w, p = _draw(rng, (1.5, 1.5, 1.5))
        n = _frame_normal(*tri)
        V = tri + c.astype(np.float64)
        box = np.concatenate([q, h.astype(F), [r, F(0), F(0)]]).astype(F)
        dist = _dist(p, *V)
        bound = np.linalg.norm(p - q.astype(np.float64), axis=1)
        if float(dist.min()) > bound.max() + float(w):
            far += 1
            dropped += not lib.disc(_p(box), _p(c), w, _p(n), F(lib.normal_error()))
        for i in range(0, len(p), 5):
            o = (p[i].astype(F) - c).astype(F)
            pn = F(((o - tri[0].astype(F)) * n).sum(dtype=F))
            true = _dist(p[i].astype(F).astype(np.float64)[None], *V)[0]
            lost += not lib.cell(F((o * o).sum(dtype=F)), pn, np.nextafter(F(true), F(np.inf)), w)
    assert far == 0 or dropped > far // 2
    assert lost > 5
