"""Stored distances so large that a march step's quotient by the units per
world unit leaves FP32: the single-volume pass leaves the brick there, as the
counting pass does, which divides."""
import dataclasses

import numpy as np
import pytest

from denrimrendererkit_gb300 import Camera, DenrimRenderer, RenderOutput, compile_scene, scenes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("scale", [1.0, 2.0, 1.0e4])  # 1, 0.5 and 1e-4 local units per world unit
@pytest.mark.parametrize("far", [1.0e30, 3.0e38, float(np.finfo(np.float32).max)])
def test_far_distances_equal_the_counting_pass(dk_lib, scale, far):
    wl = scenes.sdf_spheres(96, 64, 2, resolution=48, seed=9, narrow_band=0.1, fp16=False)
    build = compile_scene(wl.scene)
    volumes, samples = build.volumes.copy(), build.volume_brick_samples.copy()
    for name in ("world_bounds_min", "world_bounds_max"):
        volumes[name][..., :3] *= scale
    volumes["world_to_local"][..., :3, :3] /= scale
    samples["distance"][samples["distance"] > 0.5 * samples["distance"].max()] = far
    build = dataclasses.replace(build, volumes=volumes, volume_brick_samples=samples)
    camera = Camera((0.0, 0.9 * scale, 3.1 * scale), (0.0, 0.0, 0.0), vertical_field_of_view_degrees=40.0)
    scene = dataclasses.replace(wl.scene, camera=camera)
    counting = dataclasses.replace(wl.settings, collects_traversal_stats=True)
    renderer = DenrimRenderer(0)
    with renderer.make_session(scene, wl.settings, build=build) as a, \
            renderer.make_session(scene, counting, build=build) as b:
        a.render(2)
        b.render(2)
        assert b.sdf_traversal_stats()["sparse_brick_marches"] > 0
        for kind in RenderOutput:
            assert np.array_equal(a.pixels(kind).view(np.uint32), b.pixels(kind).view(np.uint32)), kind
