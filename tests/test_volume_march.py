"""The single-volume pass (k_volume_march) against the counting pass, which
walks the same volume through the reference's nested loops: every plane bit
for bit, over grids, sample formats, cameras inside and along the axes."""
import dataclasses

import numpy as np
import pytest

from denrimrendererkit_gb300 import Camera, DenrimRenderer, RenderOutput, compile_scene, scenes

pytestmark = pytest.mark.gpu

CAMERAS = [Camera((0.0, 0.9, 3.1), (0.0, 0.0, 0.0), vertical_field_of_view_degrees=40.0),
           Camera((0.05, 0.02, 0.4), (0.0, 0.0, -1.0), vertical_field_of_view_degrees=70.0),  # inside the grid
           Camera((0.0, 0.0, 3.0), (0.0, 0.0, 0.0), orthographic_scale=2.0),  # directions with two zero components
           Camera((5.0, 5.0, 5.0), (9.0, 9.0, 9.0), vertical_field_of_view_degrees=30.0)]  # misses the bounds


@pytest.mark.parametrize("resolution,width,height,fp16,band", [(24, 1, 1, False, 0.2), (48, 33, 17, False, 0.1),
                                                               (192, 130, 70, True, 0.02), (256, 96, 64, False, 0.03)])
def test_equals_the_counting_pass(dk_lib, resolution, width, height, fp16, band):
    wl = scenes.sdf_spheres(width, height, 2, resolution=resolution, seed=resolution, narrow_band=band, fp16=fp16)
    build = compile_scene(wl.scene)
    renderer = DenrimRenderer(0)
    for camera in CAMERAS:
        scene = dataclasses.replace(wl.scene, camera=camera)
        counting = dataclasses.replace(wl.settings, collects_traversal_stats=True)
        with renderer.make_session(scene, wl.settings, build=build) as a, \
                renderer.make_session(scene, counting, build=build) as b:
            a.render(2)
            b.render(2)
            for kind in RenderOutput:
                assert np.array_equal(a.pixels(kind).view(np.uint32), b.pixels(kind).view(np.uint32)), (camera, kind)
