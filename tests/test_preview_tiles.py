"""The preview kernels at the edges of their blocks: a frame drawn in ragged
tiles is the frame drawn at once, bit for bit."""
import dataclasses

import numpy as np
import pytest

from denrimrendererkit_gb300 import DenrimRenderer, RenderOutput, RenderQuality, compile_scene, scenes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("quality", [RenderQuality.PREVIEW, RenderQuality.INTERACTIVE])
@pytest.mark.parametrize("width,height,cuts_x,cuts_y", [(1, 1, (), ()), (9, 5, (8,), (4,)), (70, 43, (1, 33), (7, 40)),
                                                        (160, 130, (96, 159), (128,))])
def test_ragged_tiles_equal_the_frame(quality, width, height, cuts_x, cuts_y):
    wl = scenes.material_zoo(width, height)
    build = compile_scene(wl.scene)
    settings = dataclasses.replace(wl.settings, quality=quality)
    renderer = DenrimRenderer(0)
    with renderer.make_session(wl.scene, settings, build=build) as whole, \
            renderer.make_session(wl.scene, settings, build=build) as tiled:
        whole.render(1)
        xs, ys = (0, *cuts_x, width), (0, *cuts_y, height)
        tiles = [(x0, y0, x1 - x0, y1 - y0) for y0, y1 in zip(ys, ys[1:]) for x0, x1 in zip(xs, xs[1:])]
        for k, tile in enumerate(tiles):
            tiled.render_next_tile(*tile, k == len(tiles) - 1)
        for kind in RenderOutput:
            assert np.array_equal(whole.pixels(kind).view(np.uint32), tiled.pixels(kind).view(np.uint32)), kind
