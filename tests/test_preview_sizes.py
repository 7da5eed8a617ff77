"""The preview kernels' three block sizes draw the same frame: whole, in tiles
that run in blocks of 128 threads and in tiles that run in blocks of a warp,
bit for bit, on triangles and on a distance volume."""
import dataclasses

import numpy as np
import pytest

from denrimrendererkit_gb300 import DenrimRenderer, RenderOutput, RenderQuality, compile_scene, scenes

pytestmark = pytest.mark.gpu

SCENES = {"materials": lambda w, h: scenes.material_zoo(w, h),
          "spheres": lambda w, h: scenes.spheres_large(w, h, subdivisions=2),
          "volume": lambda w, h: scenes.sdf_spheres(w, h, 1, resolution=96, narrow_band=0.05)}


@pytest.mark.parametrize("quality", [RenderQuality.PREVIEW, RenderQuality.INTERACTIVE])
@pytest.mark.parametrize("scene", SCENES)
def test_block_sizes_agree(quality, scene):
    width, height = 642, 403  # 258,726 pixels; tiles of 321 x 202 and of 107 x 81, some cut
    wl = SCENES[scene](width, height)
    build = compile_scene(wl.scene)
    settings = dataclasses.replace(wl.settings, quality=quality)
    renderer = DenrimRenderer(0)
    planes = []
    for tw, th in ((width, height), (321, 202), (107, 81)):
        with renderer.make_session(wl.scene, settings, build=build) as session:
            for y in range(0, height, th):
                for x in range(0, width, tw):
                    session.render_next_tile(x, y, tw, th, x + tw >= width and y + th >= height)
            planes.append({kind: session.pixels(kind).view(np.uint32) for kind in RenderOutput})
    assert len(np.unique(planes[0][RenderOutput.DEPTH])) > 100
    for other in planes[1:]:
        for kind in RenderOutput:
            assert np.array_equal(planes[0][kind], other[kind]), kind
