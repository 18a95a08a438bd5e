"""Rays with direction components of zero (either sign) or far below the
others: the ordered and 8-wide traversals, whose box tests use a finite
reciprocal there, against the reference-order traversal, which uses 1/0."""
import numpy as np
import pytest

from bulbit_b200 import abi, lib, scenes

pytestmark = pytest.mark.gpu


def axis_rays(n, seed, tiny):
    """Rays from points in [-1.2, 1.2]^3 with one or two components replaced
    by +-0 or +-tiny; every eighth ray is axis-parallel, every third short, and
    every fifth direction is not of unit length."""
    g = np.random.default_rng(seed)
    r = np.zeros((n, 8), np.float32)
    r[:, 0:3] = g.uniform(-1.2, 1.2, (n, 3))
    d = g.standard_normal((n, 3)).astype(np.float32)
    d /= np.linalg.norm(d, axis=1, keepdims=True)
    small = np.where(g.random((n, 3)) < 0.5, np.float32(tiny), np.float32(-tiny)).astype(np.float32)
    axis = g.integers(0, 3, n)
    d[np.arange(n), axis] = small[np.arange(n), axis]
    d[::8, :][np.arange(len(d[::8])), (axis[::8] + 1) % 3] = small[::8][np.arange(len(d[::8])), (axis[::8] + 1) % 3]
    r[:, 3:6] = d * np.where(np.arange(n) % 5 == 0, 7.0, 1.0)[:, None].astype(np.float32)
    r[:, 6] = 1e-4
    r[:, 7] = np.where(np.arange(n) % 3 == 0, 0.4, np.inf)
    return r


@pytest.mark.parametrize("tiny", [0.0, 1e-41, 1e-30, 1e-12])
@pytest.mark.parametrize("make", [lambda: scenes.triangle_soup(20_000, seed=4, sigma=0.03),
                                  lambda: scenes.cornell_icosphere(levels=4), lambda: scenes.readme_sphere()],
                         ids=["soup20k", "cornell", "sphere"])
def test_parallel_rays_match_reference_order(make, tiny):
    acc = lib.GpuAccel(make())
    rays = axis_rays(40_003, 11, tiny)
    acc.set_traversal(abi.BBG_TRAVERSAL_REFERENCE)
    ref, occ = acc.intersect(rays), acc.intersect_any(rays)
    for mode in (abi.BBG_TRAVERSAL_WIDE, abi.BBG_TRAVERSAL_ORDERED):
        acc.set_traversal(mode)
        got = acc.intersect(rays)
        assert np.array_equal(acc.intersect_any(rays), occ)
        # t to the last bit; the primitive may differ only where two are hit
        # at exactly the same t (shared edges of the box's quads).
        assert np.array_equal(got[1].view(np.uint32), ref[1].view(np.uint32))
        assert np.count_nonzero(got[0] != ref[0]) <= 4
    assert occ.any() and not occ.all()
    acc.close()
