"""CPU: the screened map evaluation against the oracle's arithmetic.

The image kernels take a point's box from a cheaper evaluation of the map where a bound on
its distance from the map's own arithmetic proves the same box.  The library's host probe
runs the kernels' operations; here every proven box has to be the oracle's, every image has
to lie within the bound, and the benchmark maps' points have to be proven almost always.
"""
import ctypes as C

import numpy as np
import pytest

from oracle import oracle as O


def probe(spec, depth, codes, offsets, reach, from_centre):
    from b12_b200 import _lib
    L = _lib.lib()
    d, m = _lib.Domain(), _lib.Map()
    dim = spec["dim"]
    d.dim = dim
    for j in range(dim):
        d.center[j], d.radius[j] = spec["center"][j], spec["radius"][j]
    ms = spec["map"]
    m.kind, m.arith, m.steps, m.h = ms["kind"], ms.get("fma", 0), ms.get("steps", 1), ms.get("h", 0.0)
    for i, v in enumerate(ms.get("p", [])):
        m.p[i] = v
    n = len(codes)
    codes = np.ascontiguousarray(codes, dtype=np.uint64)
    offsets = np.ascontiguousarray(offsets, dtype=np.float64)
    applies = C.c_int()
    bound, images = np.zeros(dim), np.zeros((n, dim))
    decided, boxes = np.zeros(n, dtype=np.uint8), np.zeros(n, dtype=np.uint64)
    st = L.b12g_screen_probe(C.byref(d), C.byref(m), depth, reach, codes.ctypes.data, offsets.ctypes.data, n,
                             from_centre, C.byref(applies), bound.ctypes.data, images.ctypes.data,
                             decided.ctypes.data, boxes.ctypes.data)
    assert st == 0, L.b12g_last_error()
    return bool(applies.value), bound, images, decided.astype(bool), boxes


def exact(spec, depth, codes, offsets):
    """(images, depth-d box codes or ~0 outside) by the oracle."""
    o = O.Oracle(spec)
    dim = spec["dim"]
    images, boxes = np.zeros((len(codes), dim)), np.zeros(len(codes), dtype=np.uint64)
    c, r = np.zeros(dim), np.zeros(dim)
    for i, code in enumerate(codes):
        o.L.orc_box_coordinates(C.byref(o.dom), int(code), depth, O._ptr(c, C.c_double), O._ptr(r, C.c_double))
        images[i] = o.map_apply(c + offsets[i] * r)
        p64, inside = o.point_code64(images[i])
        boxes[i] = p64 >> (64 - depth) if inside and depth else (0 if inside else 0xFFFFFFFFFFFFFFFF)
    return images, boxes


def check(spec, depth, codes, offsets, reach=1.0):
    """(the screen applies, the share of the points it decides)"""
    share = 0.0
    want = None
    for from_centre in (0, 1):
        on, bound, images, decided, boxes = probe(spec, depth, codes, offsets, reach, from_centre)
        if not on:
            return False, 0.0
        want = want or exact(spec, depth, codes, offsets)
        assert np.array_equal(boxes[decided], want[1][decided])
        # the images, moved back to the map's coordinates (roundings of the scaling aside)
        far = np.abs(images - want[0])[decided]
        slack = 2.0 ** -48 * (np.abs(want[0][decided]) + np.abs(np.array(spec["center"])) + 64.0)
        assert (far <= bound + slack).all(), (far.max(axis=0), bound)
        share = decided.mean()
    return True, share


def random_boxes(rng, dim, depth, n, on_faces=0.5):
    """Boxes and points in them: grid-like offsets, faces and corners among them."""
    codes = rng.integers(0, 2 ** min(depth, 63), size=n, dtype=np.uint64) if depth else np.zeros(n, np.uint64)
    offsets = rng.uniform(-1.0, 1.0, size=(n, dim))
    grid = rng.choice([-1.0, -0.8, -0.4, 0.0, 0.4, 0.8, 1.0], size=(n, dim))
    return codes, np.where(rng.random((n, 1)) < on_faces, grid, offsets)


def lorenz(rho=28.0, fma=0, h=0.01, steps=20, sigma=10.0, beta=8.0 / 3.0, center=(0.0, 0.0, 27.0),
           radius=(30.0, 30.0, 40.0)):
    return dict(dim=3, center=list(center), radius=list(radius),
                map=dict(kind=O.MAP_LORENZ, steps=steps, h=h, fma=fma, p=[sigma, rho, beta]),
                grid=dict(kind=O.GRID_INNER, n=5))


def box_codes(spec, x, depth):
    """The depth-d boxes holding the points x (all inside the domain)."""
    o = O.Oracle(spec)
    return np.array([o.point_code64(p)[0] >> (64 - depth) if depth else 0 for p in x], dtype=np.uint64)


def trajectory_points(spec, x0, n, burn):
    o = O.Oracle(spec)
    x, out = np.array(x0, dtype=np.float64), []
    for i in range(burn + n):
        x = o.map_apply(x)
        if i >= burn:
            out.append(x)
    return np.array(out)


@pytest.mark.parametrize("fma", [0, 1])
@pytest.mark.parametrize("depth", [0, 1, 2, 7, 18, 22, 27, 30, 33])
def test_lorenz_depths(depth, fma):
    rng = np.random.default_rng([depth, fma])
    spec = lorenz(fma=fma)
    codes, off = random_boxes(rng, 3, depth, 1500)
    on, _ = check(spec, depth, codes, off)
    assert on
    # boxes the attractor passes through: almost every point is decided
    x = trajectory_points(spec, (1.0, 2.0, 20.0), 400, 50)
    codes = np.repeat(box_codes(spec, x, depth), 3)
    _, off = random_boxes(rng, 3, depth, len(codes))
    on, share = check(spec, depth, codes, off)
    # (coarse boxes have grid points on the axis x = y = 0, which is mapped into itself and
    # bounds four boxes: those points are for the map's own arithmetic, and too many to count)
    assert on and (share >= 0.995 or depth < 18)


@pytest.mark.parametrize("case", range(24))
def test_lorenz_parameters(case):
    """Other parameters, domains, steps and backward time; a wide reach of the grid."""
    rng = np.random.default_rng([case, 5])
    spec = lorenz(rho=rng.uniform(0.5, 60.0), fma=case % 2, h=rng.choice([0.001, 0.005, 0.01, -0.004]),
                  steps=int(rng.integers(1, 24)), sigma=rng.uniform(1.0, 16.0), beta=rng.uniform(0.2, 4.0),
                  center=rng.uniform(-20.0, 30.0, size=3), radius=np.exp(rng.uniform(np.log(0.5), np.log(60.0), size=3)))
    depth = int(rng.integers(0, 40))
    codes, off = random_boxes(rng, 3, depth, 800)
    reach = float(rng.choice([1.0, 1.5, 4.0]))
    check(spec, depth, codes, off * reach, reach)


def coupled(h=0.05, steps=10, center=(0.0,) * 4, radius=(2.0,) * 4):
    return dict(dim=4, center=list(center), radius=list(radius),
                map=dict(kind=O.MAP_COUPLED_DUFFING, steps=steps, h=h), grid=dict(kind=O.GRID_PHILOX, points=8))


@pytest.mark.parametrize("depth", [0, 1, 3, 8, 16, 24, 30, 41])
def test_coupled_duffing_depths(depth):
    rng = np.random.default_rng([depth, 2])
    codes, off = random_boxes(rng, 4, depth, 3000, 0.2)
    on, share = check(coupled(), depth, codes, off)
    # (points on the faces of coarse boxes stay on the planes q = 0 or p = 0 or meet them)
    assert on and (share >= 0.99 or depth < 16)


@pytest.mark.parametrize("case", range(16))
def test_coupled_duffing_parameters(case):
    rng = np.random.default_rng([case, 6])
    spec = coupled(h=rng.choice([0.003, 0.05, -0.05, 0.11]), steps=int(rng.integers(1, 16)),
                   center=rng.uniform(-1.0, 1.0, size=4), radius=np.exp(rng.uniform(np.log(0.2), np.log(6.0), size=4)))
    codes, off = random_boxes(rng, 4, depth := int(rng.integers(0, 44)), 800)
    reach = float(rng.choice([1.0, 2.0]))
    check(spec, depth, codes, off * reach, reach)


def forced(steps=200, p=(0.25, -1.0, 1.0, 0.3), center=(0.0, 0.0), radius=(2.0, 2.0)):
    return dict(dim=2, center=list(center), radius=list(radius),
                map=dict(kind=O.MAP_FORCED_DUFFING, steps=steps, h=O.FORCED_PERIOD / steps, p=list(p)),
                grid=dict(kind=O.GRID_INNER, n=4))


@pytest.mark.parametrize("depth", [0, 1, 6, 14, 19, 22, 26, 31])
def test_forced_duffing_depths(depth):
    rng = np.random.default_rng([depth, 4])
    spec = forced()
    codes, off = random_boxes(rng, 2, depth, 2000)
    on, _ = check(spec, depth, codes, off)
    assert on == (depth <= 26)       # 200 steps: the bound passes a sixteenth of the warps' budget at 14 bisections
    if not on:
        return
    x = trajectory_points(spec, (0.5, 0.1), 500, 50)
    codes = box_codes(spec, x, depth)
    _, off = random_boxes(rng, 2, depth, len(codes))
    on, share = check(spec, depth, codes, off)
    assert on and (share >= 0.99 or depth < 14)


@pytest.mark.parametrize("case", range(16))
def test_forced_duffing_parameters(case):
    rng = np.random.default_rng([case, 8])
    p = (rng.uniform(-0.1, 0.6), rng.uniform(-1.5, 1.5), rng.uniform(0.1, 2.0), rng.uniform(-0.6, 0.6))
    spec = forced(steps=int(rng.choice([40, 100, 200, 333])), p=p, center=rng.uniform(-0.5, 0.5, size=2),
                  radius=np.exp(rng.uniform(np.log(0.3), np.log(3.0), size=2)))
    depth = int(rng.integers(0, 34))
    codes, off = random_boxes(rng, 2, depth, 600)
    check(spec, depth, codes, off)


def test_points_beside_box_boundaries():
    """Images a few roundings, and a little more, beside a boundary."""
    spec = lorenz(h=2.0 ** -39, steps=1)     # the image is the point itself but for its last digits
    rng = np.random.default_rng(3)
    depth = 18
    codes = rng.integers(0, 2 ** depth, size=3000, dtype=np.uint64)
    off = np.where(rng.random((3000, 3)) < 0.5, rng.choice([-1.0, 1.0], size=(3000, 3)),
                   rng.uniform(-1, 1, size=(3000, 3)))
    off = off * (1.0 + rng.choice([-1.0, 1.0], size=(3000, 3)) * 10.0 ** rng.uniform(-16, -8, size=(3000, 3)))
    on, _ = check(spec, depth, codes, off, 1.001)
    assert on


def test_screening_is_left_out_where_it_cannot_prove():
    from_zero = [np.zeros(1, np.uint64), np.zeros((1, 3))]
    assert not probe(lorenz(), 57, *from_zero, 1.0, 0)[0]                   # more than 18 bisections of x
    assert not probe(lorenz(steps=400), 27, *from_zero, 1.0, 0)[0]          # the bound grows past the boxes
    assert not probe(lorenz(radius=(4000.0, 4000.0, 4000.0)), 27, *from_zero, 1.0, 0)[0]
    assert not probe(lorenz(h=0.0), 27, *from_zero, 1.0, 0)[0]
    assert not probe(lorenz(sigma=float("nan")), 27, *from_zero, 1.0, 0)[0]
    assert not probe(lorenz(steps=0), 27, *from_zero, 1.0, 0)[0]
    assert not probe(forced(p=(0.25, -1.0, -1.0, 0.3)), 16, np.zeros(1, np.uint64), np.zeros((1, 2)), 1.0, 0)[0]
    assert not probe(forced(p=(0.25, -1.0, 0.0, 0.3)), 16, np.zeros(1, np.uint64), np.zeros((1, 2)), 1.0, 0)[0]
