"""The 8-wide traversal's leaf queue (leaves of a warp's rays tested by all of
its lanes) against the reference-order traversal, which tests each leaf where
it meets it: batch sizes around warps and blocks, leaves of one and of many
primitives, spheres among triangles, intervals of no length, and rays whose
interval ends at a hit."""
import itertools

import numpy as np
import pytest

from bulbit_b200 import abi, lib, scenes

pytestmark = pytest.mark.gpu


def stacked(copies, n=120):
    """n triangles of the soup, each `copies` times: leaves hold several
    primitives, all hit at exactly the same t."""
    s = scenes.triangle_soup(n, seed=8, sigma=0.2)
    s.tri_indices = np.repeat(s.tri_indices, copies, axis=0)
    m = s.tri_indices.shape[0]
    s.prim_kind, s.prim_index = np.zeros(m, np.int32), np.arange(m, dtype=np.int32)
    s.prim_material = np.full(m, -1, np.int32)
    return s


def with_spheres():
    s = scenes.triangle_soup(3000, seed=5, sigma=0.05)
    g = np.random.default_rng(3)
    for k in range(60):
        sph = abi.Sphere()
        sph.p[:] = g.uniform(-1, 1, 3).tolist()
        sph.q[:] = [0.0, 0.0, 0.0, 1.0]
        sph.s[:] = [1.0, 1.0, 1.0]
        sph.radius = float(g.uniform(0.03, 0.15))
        s.spheres.append(sph)
    s.prim_kind = np.concatenate([s.prim_kind, np.full(60, abi.BBG_PRIM_SPHERE, np.int32)])
    s.prim_index = np.concatenate([s.prim_index, np.arange(60, dtype=np.int32)])
    s.prim_material = np.full(3060, -1, np.int32)
    return s


def corner_fans(cubes=60):
    """Per cube, 24 triangles of three of its corners whose box is the whole cube:
    no split separates them, so a leaf holds them all, at different t."""
    g = np.random.default_rng(12)
    corner = np.array([[k & 1, k >> 1 & 1, k >> 2] for k in range(8)], np.float32)
    tri = [c for c in itertools.combinations(range(8), 3) if np.ptp(corner[list(c)], axis=0).min() == 1][:24]
    lo, size = g.uniform(-1, 0.7, (cubes, 1, 3)), g.uniform(0.1, 0.3, (cubes, 1, 3))
    s = scenes.triangle_soup(1, seed=8)
    s.positions = (lo + corner[None] * size).reshape(-1, 3).astype(np.float32)
    s.tri_indices = (8 * np.arange(cubes)[:, None, None] + np.array(tri)[None]).reshape(-1, 3).astype(np.int32)
    s.normals = np.tile(np.float32([0, 1, 0]), (8 * cubes, 1))
    s.tangents = np.tile(np.float32([1, 0, 0]), (8 * cubes, 1))
    s.uvs = np.zeros((8 * cubes, 2), np.float32)
    m = s.tri_indices.shape[0]
    s.prim_kind, s.prim_index = np.zeros(m, np.int32), np.arange(m, dtype=np.int32)
    s.prim_material = np.full(m, -1, np.int32)
    return s


SCENES = {"soup": lambda: scenes.triangle_soup(50_000, seed=7, sigma=0.03), "cornell": lambda: scenes.cornell_icosphere(5),
          "stacked3": lambda: stacked(3), "stacked31": lambda: stacked(31), "spheres": with_spheres,
          "one": lambda: scenes.triangle_soup(1, seed=3, sigma=0.5)}


def check(scene, acc, rays):
    """Same t and occlusion; the primitive kept may be another one only where
    several are hit at exactly the same t."""
    acc.set_traversal(abi.BBG_TRAVERSAL_REFERENCE)
    ref, occ = acc.intersect(rays), acc.intersect_any(rays)
    acc.set_traversal(abi.BBG_TRAVERSAL_WIDE)
    got = acc.intersect(rays)
    assert np.array_equal(acc.intersect_any(rays), occ)
    assert np.array_equal(got[1].view(np.uint32), ref[1].view(np.uint32))
    assert np.array_equal(got[0] < 0, ref[0] < 0)
    # Copies of a triangle differ in their number only; no two spheres are alike.
    other = got[0] != ref[0]
    if scene.spheres:
        assert np.count_nonzero(other) <= 2
    elif other.any():
        corners = scene.positions[scene.tri_indices]
        same = np.all(corners[got[0][other]] == corners[ref[0][other]], axis=(1, 2))
        assert np.count_nonzero(~same) <= 2
    return ref


@pytest.mark.parametrize("name", SCENES)
@pytest.mark.parametrize("n", [1, 31, 33, 129, 5000, 200_001])
def test_wide_matches_reference_order(name, n):
    scene = SCENES[name]()
    acc = lib.GpuAccel(scene)
    assert acc.export_wide8().shape[0] > 0
    closest, short = scenes.soup_rays(n, seed=n)
    check(scene, acc, closest)
    check(scene, acc, short)
    acc.close()


@pytest.mark.parametrize("name", ["soup", "stacked3", "spheres"])
def test_intervals_around_hits(name):
    scene = SCENES[name]()
    acc = lib.GpuAccel(scene)
    closest, _ = scenes.soup_rays(20_011, seed=4)
    ref = check(scene, acc, closest)
    hit = ref[0] >= 0
    assert hit.sum() > 500
    for lo, hi in ((ref[1], np.inf), (1e-4, ref[1]), (ref[1], ref[1]), (2.0, 1.0)):
        rays = closest[hit].copy()
        rays[:, 6] = lo[hit] if isinstance(lo, np.ndarray) else lo
        rays[:, 7] = hi[hit] if isinstance(hi, np.ndarray) else hi
        if isinstance(lo, np.ndarray) and isinstance(hi, np.ndarray):
            # An interval of no length ends at the first primitive tested, which
            # depends on the order: a hit must be the one at that t, and about as
            # many rays have one as in the reference's order (0.977 to 0.998 of
            # them in these scenes).
            acc.set_traversal(abi.BBG_TRAVERSAL_REFERENCE)
            count = np.count_nonzero(acc.intersect(rays)[0] >= 0)
            acc.set_traversal(abi.BBG_TRAVERSAL_WIDE)
            got = acc.intersect(rays)
            assert np.all((got[0] < 0) | (got[1] == rays[:, 6]))
            assert 0.9 * count <= np.count_nonzero(got[0] >= 0) <= 1.1 * count
            assert np.array_equal(acc.intersect_any(rays) != 0, got[0] >= 0)
        else:
            check(scene, acc, rays)
    acc.close()


@pytest.mark.parametrize("make", [SCENES["one"], lambda: corner_fans(1)], ids=["one", "fan"])
def test_no_length_intervals_in_one_leaf(make):
    """In a tree of one leaf the first primitive tested is known, the leaf's
    first: an interval of no length is answered as in the reference's order."""
    acc = lib.GpuAccel(make())
    assert acc.export()[0].shape[0] == 1
    closest, _ = scenes.soup_rays(60_000, seed=4)
    acc.set_traversal(abi.BBG_TRAVERSAL_REFERENCE)
    ref = acc.intersect(closest)
    rays = closest[ref[0] >= 0].copy()
    rays[:, 6] = rays[:, 7] = ref[1][ref[0] >= 0]
    want, occ = acc.intersect(rays), acc.intersect_any(rays)
    assert len(rays) > 200 and occ.any()
    acc.set_traversal(abi.BBG_TRAVERSAL_WIDE)
    got = acc.intersect(rays)
    assert np.array_equal(acc.intersect_any(rays), occ)
    assert all(np.array_equal(got[k].view(np.uint32), want[k].view(np.uint32)) for k in range(4))
    acc.close()


@pytest.mark.parametrize("make", [corner_fans, lambda: stacked(31)], ids=["fans", "stacked31"])
def test_records_of_large_leaves(make):
    """32 waiting leaves of two dozen primitives are tested in many rounds: each
    ray's record (primitive, t, u, v) is one primitive's."""
    acc = lib.GpuAccel(make())
    assert acc.export_wide8().shape[0] > 0
    closest, _ = scenes.soup_rays(100_003, seed=5)
    acc.set_traversal(abi.BBG_TRAVERSAL_REFERENCE)
    ref = acc.intersect(closest)
    acc.set_traversal(abi.BBG_TRAVERSAL_WIDE)
    got = acc.intersect(closest)
    assert (ref[0] >= 0).sum() > 5000
    assert np.array_equal(got[1].view(np.uint32), ref[1].view(np.uint32))
    # Copies share u and v; two triangles of a fan meet at one t only along the
    # line they cross in.
    other = np.any([got[k].view(np.uint32) != ref[k].view(np.uint32) for k in (2, 3)], axis=0)
    assert np.count_nonzero(other) <= 4
    acc.close()
