"""Temporal filtering of images far taller than wide: every radius takes what
the filter's other passes take, and rows far from a cut equal those of the
image cut there."""
import pytest

torch = pytest.importorskip("torch")

pytestmark = pytest.mark.gpu

HEIGHT, CUT = 600_000, 4096


def _planes(height):
    g = torch.Generator(device="cuda").manual_seed(3)
    plane = torch.rand(HEIGHT, 2, 4, generator=g, device="cuda")
    beauty = plane[:height] * 2.0
    depth = plane[:height, :, :1].expand(-1, -1, 4) * 0.2 + 2.0
    normal = torch.ones(height, 2, 4, device="cuda")
    normal[..., :2] = 0.5 + 0.1 * plane[:height, :, :2]
    return [p.contiguous() for p in (beauty, depth, normal, torch.zeros(height, 2, 4, device="cuda"))]


@pytest.mark.parametrize("radius", [1, 2, 3, 4])
def test_tall_image(dk_lib, radius):
    from denrimrendererkit_gb300.denoiser import SvgfDenoiser
    images = []
    for height in (HEIGHT, CUT):
        out = torch.full((height, 2, 4), -1.0, device="cuda")
        SvgfDenoiser(2, height).denoise(*_planes(height), out, radius=radius, iterations=2)
        torch.cuda.synchronize()
        images.append(out)
    tall, short = images
    margin = 32  # rows the two passes, the variance estimate and its prefilter reach
    assert torch.equal(tall[:CUT - margin], short[:CUT - margin])
    assert bool((tall >= 0.0).all())  # every row is written
