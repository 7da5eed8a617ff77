"""A wave of so many paths that the survivors' block counts are scanned in a
kernel of their own: the image is that of its quarters, bit for bit, and each
bounce has that one launch more."""
import dataclasses

import pytest

torch = pytest.importorskip("torch")

from denrimrendererkit_gb300 import DenrimRenderer, RenderOutput, compile_scene, scenes

pytestmark = pytest.mark.gpu


def test_large_wave_equals_its_quarters(dk_lib):
    size = 5800  # 33.6 M paths, 8,213 blocks
    wl = scenes.cornell_small(size, size, 1)
    settings = dataclasses.replace(wl.settings, max_bounces=4)
    build = compile_scene(wl.scene)
    renderer = DenrimRenderer(0)
    images, launches = [], []
    for rows in (size, size // 4):
        with renderer.make_session(wl.scene, settings, build=build) as session:
            if rows == size:
                session.render(1)
            else:
                for y in range(0, size, rows):
                    session.render_next_tile(0, y, size, rows, y + rows == size)
            launches.append(session.stats().last_launches)
            planes = [RenderOutput.BEAUTY, RenderOutput.ALBEDO]
            images.append([session.copy_output(k, torch.empty(size, size, 4, device="cuda")) for k in planes])
            torch.cuda.synchronize()
    assert all(torch.equal(a, b) for a, b in zip(*images))
    assert launches[0] - launches[1] == settings.max_bounces
