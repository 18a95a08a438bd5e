"""The queue and work counters of a bounce level, which the passes around their
use clear: the same paths in one wave and in many, captured in a graph or
launched one by one, in a second render, with levels drained after the last
bounce, with and without the shading sort and with a guide, and after a render
that stopped in the middle."""
import numpy as np
import pytest

from bulbit_b200 import abi, lib, scenes

pytestmark = pytest.mark.gpu


def cornell(material=None):
    return scenes.cornell_icosphere(levels=2, width=41, height=37, spp=4, max_bounces=5, sphere_material=material)


def shells():
    """Six material-less spheres around the camera: paths outlive the levels of
    a wave and are drained."""
    s = scenes.cornell_icosphere(levels=1, width=24, height=24, spp=4, max_bounces=1)
    for k in range(6):
        sph = abi.Sphere()
        sph.p[:] = s.camera.position[:]
        sph.q[:], sph.s[:], sph.radius = [0, 0, 0, 1], [1, 1, 1], 0.05 + 0.04 * k
        s.spheres.append(sph)
    s.prim_kind = np.concatenate([s.prim_kind, np.ones(6, np.int32)]).astype(np.int32)
    s.prim_index = np.concatenate([s.prim_index, np.arange(6)]).astype(np.int32)
    s.prim_material = np.concatenate([s.prim_material, -np.ones(6, np.int32)]).astype(np.int32)
    return s


SCENES = {"sorted": cornell, "one_kind": lambda: cornell(scenes.diffuse((0.4, 0.5, 0.6))),
          "sphere": lambda: scenes.readme_sphere(40, 30, 4, 6), "drained": shells}


@pytest.mark.parametrize("guided", [False, True])
@pytest.mark.parametrize("name", SCENES)
def test_waves_and_graphs_agree(name, guided):
    scene = SCENES[name]()
    acc = lib.GpuAccel(scene)
    integ = lib.GpuPathIntegrator(acc, scene)
    guide = lib.GpuGuide(np.array([-1.1, -1.1, -1.1, 1.1, 2.1, 1.1], np.float32), seed=2) if guided else None
    want = integ.render(path_L=True, use_graph=False, guide=guide)
    assert want.path_L.any()
    paths = want.path_L.shape[0]
    for kw in (dict(use_graph=True), dict(use_graph=True), dict(use_graph=True, wave_paths=paths // 3),
               dict(use_graph=False, wave_paths=paths // 5), dict(use_graph=False)):
        got = integ.render(path_L=True, guide=guide, **kw)
        assert np.array_equal(got.path_L, want.path_L), kw
        assert np.array_equal(got.rgb_sum, want.rgb_sum) and np.array_equal(got.count, want.count)
        assert got.stats.closest_rays == want.stats.closest_rays and got.stats.shadow_rays == want.stats.shadow_rays
    integ.close()
    acc.close()


@pytest.mark.parametrize("use_graph", [True, False])
def test_render_after_a_stopped_one(use_graph):
    scene = shells()
    acc = lib.GpuAccel(scene)
    integ = lib.GpuPathIntegrator(acc, scene)
    want = integ.render(path_L=True)
    with pytest.raises(lib.BbgError) as e:
        integ.render(pass_through_levels=2, use_graph=use_graph, wave_paths=500)
    assert e.value.status == abi.BBG_ERR_TIMEOUT
    got = integ.render(path_L=True, use_graph=use_graph)
    assert np.array_equal(got.path_L, want.path_L)
    assert got.stats.closest_rays == want.stats.closest_rays
    integ.close()
    acc.close()
