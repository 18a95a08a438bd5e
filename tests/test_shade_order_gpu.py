"""The shading order of scenes whose primitives all have one kind of material,
which the default leaves unsorted where shading them is cheap: the same film
either way, and no slower by default than in queue order where it is not."""
import numpy as np
import pytest

from bulbit_b200 import abi, lib, scenes

pytestmark = pytest.mark.gpu

MATERIALS = {
    "diffuse": scenes.diffuse((0.5, 0.5, 0.5)),
    "mirror": scenes.conductor(scenes.GOLD_ETA, scenes.GOLD_K, 0.0),
    "glass": scenes.dielectric(1.5),
    "rough_glass_compensated": scenes.dielectric(1.5, roughness=0.4, energy_compensation=True),
    "metal": scenes.metallic_roughness((0.8, 0.6, 0.3), 0.7, 0.4),
}


def open_soup(material, width, height):
    """3,000 triangles of one material under a spot and an infinite light: most
    of a level's rays escape."""
    s, r = scenes.triangle_soup(3000, seed=1, sigma=0.05), scenes.readme_sphere(width, height, 16, 8)
    s.materials, s.prim_material = [material], np.zeros(3000, np.int32)
    s.lights, s.camera, s.spp, s.max_bounces = r.lights, r.camera, 16, 8
    return s


@pytest.mark.parametrize("regularize", [0, 1])
@pytest.mark.parametrize("name", MATERIALS)
def test_orders_give_the_same_film(name, regularize):
    s = open_soup(MATERIALS[name], 97, 61)
    acc = lib.GpuAccel(s)
    integ = lib.GpuPathIntegrator(acc, s, regularize=regularize)
    a, b = (integ.render(shade_order=o, path_L=True) for o in (abi.BBG_SHADE_SORTED, abi.BBG_SHADE_QUEUE))
    assert np.array_equal(a.path_L, b.path_L) and np.array_equal(a.rgb_sum, b.rgb_sum)
    assert a.path_L.any()
    integ.close()
    acc.close()


def test_expensive_shading_is_sorted():
    """Rough glass with energy compensation: sorted 7.3 ms, in queue order 10.9
    ms on one B200, so the default has to be at least a tenth faster."""
    s = open_soup(MATERIALS["rough_glass_compensated"], 640, 480)
    acc = lib.GpuAccel(s)
    integ = lib.GpuPathIntegrator(acc, s)
    times = {o: [] for o in (abi.BBG_SHADE_SORTED, abi.BBG_SHADE_QUEUE)}
    for _ in range(8):
        for o, t in times.items():
            t.append(integ.render(shade_order=o).stats.device_ms)
    default, queue = (np.median(t[2:]) for t in times.values())
    assert default < 0.9 * queue, (default, queue)
    integ.close()
    acc.close()
