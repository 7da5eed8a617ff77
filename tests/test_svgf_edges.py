"""The SVGF passes at every radius on images whose edges cut their taps and
row groups, against the numpy restatement."""
import numpy as np
import pytest

from oracle import svgf_oracle as so

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("radius,iterations,width,height", [(1, 1, 1, 1), (1, 5, 40, 37), (2, 5, 33, 3), (2, 4, 131, 70),
                                                            (3, 3, 64, 33), (4, 5, 97, 65), (2, 1, 5, 64)])
def test_every_radius_and_ragged_sizes(dk_lib, radius, iterations, width, height):
    torch = pytest.importorskip("torch")
    from denrimrendererkit_gb300.denoiser import SvgfDenoiser
    rng = np.random.default_rng(radius * 100 + width)
    shape = (height, width, 4)
    beauty = rng.uniform(0.1, 2.0, shape).astype(np.float32)
    depth = np.repeat(rng.uniform(2.0, 2.2, shape[:2] + (1,)), 4, -1).astype(np.float32)
    direction = rng.normal(0.0, 0.1, shape[:2] + (3,)) + (0.0, 0.0, 1.0)
    direction /= np.linalg.norm(direction, axis=-1, keepdims=True)
    normal = np.concatenate([direction * 0.5 + 0.5, np.ones(shape[:2] + (1,))], -1).astype(np.float32)
    normal[rng.uniform(size=shape[:2]) < 0.05] = 0.0  # no surface
    motion = np.zeros(shape, np.float32)
    motion[..., :2] = (0.6, -0.3)
    motion[..., 3] = 1.0
    p = so.params(radius=radius, iterations=iterations)
    gpu, cpu = SvgfDenoiser(width, height), so.Svgf(width, height)
    planes = [torch.from_numpy(a).cuda() for a in (beauty, depth, normal, motion)]
    out = torch.empty(shape, device="cuda")
    for _ in range(2):  # a fresh history, then a reprojected one
        gpu.denoise(*planes, out, radius=radius, iterations=iterations)
        want = cpu.denoise(beauty, depth, normal, motion, p)
        got = out.cpu().numpy()
        assert np.array_equal(got[..., 3], want[..., 3])
        # FP32 sums of at most 81 taps with the two-ulp special functions on both sides, five passes
        assert np.abs(got[..., :3] - want[..., :3]).max() <= 1e-3 * want[..., :3].mean()
