"""Axis-parallel rays that run exactly in box faces: meshes whose vertices have
whole-number coordinates up to 1,024 (where the boxes' padding of 10 epsilon is
rounded away) and spheres, whose boxes are never padded, with ray origins on
those coordinates, borders and tangents included. The ordered and 8-wide
traversals against the reference-order traversal."""
import numpy as np
import pytest

from bulbit_b200 import abi, lib, scenes

pytestmark = pytest.mark.gpu


def mesh(positions, triangles, name):
    s = scenes.triangle_soup(1, seed=1)
    s.name = name
    s.positions = np.ascontiguousarray(positions, np.float32)
    s.normals = np.tile(np.float32([0, 1, 0]), (len(positions), 1))
    s.tangents = np.tile(np.float32([1, 0, 0]), (len(positions), 1))
    s.uvs = np.zeros((len(positions), 2), np.float32)
    s.tri_indices = np.ascontiguousarray(triangles, np.int32)
    m = len(triangles)
    s.prim_kind, s.prim_index = np.zeros(m, np.int32), np.arange(m, dtype=np.int32)
    s.prim_material = np.full(m, -1, np.int32)
    return s


def height_field(base, n=40):
    """(n + 1)^2 vertices at (base + i, base + 0..6, base + j)."""
    g = np.random.default_rng(base + 1)
    i, j = np.meshgrid(np.arange(n + 1), np.arange(n + 1), indexing="ij")
    p = np.stack([base + i, base + g.integers(0, 7, (n + 1, n + 1)), base + j], 2).reshape(-1, 3)
    a = (i[:-1, :-1] * (n + 1) + j[:-1, :-1]).ravel()
    t = np.concatenate([np.stack([a, a + 1, a + n + 2], 1), np.stack([a, a + n + 2, a + n + 1], 1)])
    return mesh(p, t, "height field")


def boxes(base, count=60, n=40):
    g = np.random.default_rng(base + 2)
    corner = np.array([[k & 1, k >> 1 & 1, k >> 2] for k in range(8)])
    quads = np.array([[0, 2, 6, 4], [1, 3, 7, 5], [0, 1, 5, 4], [2, 3, 7, 6], [0, 1, 3, 2], [4, 5, 7, 6]])
    tri = np.concatenate([quads[:, [0, 1, 2]], quads[:, [0, 2, 3]]])
    lo, size = g.integers(0, n - 6, (count, 1, 3)), g.integers(1, 7, (count, 1, 3))
    p = (base + lo + corner[None] * size).reshape(-1, 3)
    return mesh(p, (8 * np.arange(count)[:, None, None] + tri[None]).reshape(-1, 3), "boxes")


def stacked(base):
    """40 copies of each of a few triangles: no 8-wide layout, so the ordered
    traversal over the binary one is the default."""
    s = height_field(base, 4)
    return mesh(s.positions, np.repeat(s.tri_indices, 40, axis=0), "stacked")


def spheres(base, count=40, n=40):
    g = np.random.default_rng(base + 3)
    s = scenes.triangle_soup(1, seed=1)
    s.spheres = []
    for _ in range(count):
        sph = abi.Sphere()
        sph.p[:] = (base + g.integers(0, n, 3)).astype(float).tolist()
        sph.q[:] = [0.0, 0.0, 0.0, 1.0]
        sph.s[:] = [1.0, 1.0, 1.0]
        sph.radius = float(g.integers(1, 5))
        s.spheres.append(sph)
    s.prim_kind = np.concatenate([s.prim_kind, np.full(count, abi.BBG_PRIM_SPHERE, np.int32)])
    s.prim_index = np.concatenate([s.prim_index, np.arange(count, dtype=np.int32)])
    s.prim_material = np.full(count + 1, -1, np.int32)
    return s


def rays_on_planes(base, rays, seed, n=40):
    """Origins at whole coordinates in [base - 1, base + n + 1], a third of them
    on the border; axis directions (lengths 1 and 3, either zero)."""
    g = np.random.default_rng(seed)
    o = (base + g.integers(-1, n + 2, (rays, 3))).astype(np.float32)
    edge = g.random((rays, 3)) < 0.3
    o[edge] = np.where(g.random(edge.sum()) < 0.5, base, base + n)
    axis = g.integers(0, 3, rays)
    d = np.where(g.random((rays, 3)) < 0.5, np.float32(0.0), np.float32(-0.0)).astype(np.float32)
    d[np.arange(rays), axis] = np.where(g.random(rays) < 0.5, 1.0, -1.0) * np.where(g.random(rays) < 0.2, 3.0, 1.0)
    out = np.zeros((rays, 8), np.float32)
    out[:, 0:3], out[:, 3:6] = o, d
    far = g.random(rays) < 0.7
    out[np.arange(rays), axis] -= np.where(far, 2.0 * n * np.sign(d[np.arange(rays), axis]), 0).astype(np.float32)
    out[:, 6], out[:, 7] = 1e-4, np.where(g.random(rays) < 0.3, 15.0, np.inf)
    return out


@pytest.mark.parametrize("base", [0, 33, 100, 1000])
@pytest.mark.parametrize("make", [height_field, boxes, stacked, spheres])
def test_rays_in_box_faces(make, base):
    acc = lib.GpuAccel(make(base))
    rays = rays_on_planes(base, 60_001, base + 7, 4 if make is stacked else 40)
    assert (acc.export_wide8().shape[0] == 0) == (make is stacked)
    default = acc.intersect(rays), acc.intersect_any(rays)
    acc.set_traversal(abi.BBG_TRAVERSAL_REFERENCE)
    ref, occ = acc.intersect(rays), acc.intersect_any(rays)
    hit = ref[0] >= 0
    assert hit.sum() > 1000 and (~hit).sum() > 1000
    got = [default]
    for mode in (abi.BBG_TRAVERSAL_ORDERED,) + (() if make is stacked else (abi.BBG_TRAVERSAL_WIDE,)):
        acc.set_traversal(mode)
        got.append((acc.intersect(rays), acc.intersect_any(rays)))
    for closest, any_hit in got:
        # Equal to the last bit: whole coordinates make the triangle tests exact,
        # and a box that is opened though the reference does not adds no hit.
        assert np.array_equal(closest[0] >= 0, hit)
        assert np.array_equal(closest[1].view(np.uint32), ref[1].view(np.uint32))
        assert np.array_equal(any_hit, occ)
    acc.close()
