"""The tensor-memory weight gradient where a CTA takes several blocks of input
channels, two sets of accumulators, a ragged last block, or many tiles: against
FP64 sums, to the error of sums no longer than the rule allows."""
import pytest

torch = pytest.importorskip("torch")

from denrimrendererkit_gb300 import DenrimRenderer, library

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def lib(dk_lib):
    DenrimRenderer(0)
    return library.load()


# Two blocks per CTA with an even and an odd number of them, ragged edges, channel slices; two accumulator sets,
# with CTAs of one tile among them; a last block of 16 channels; more than 160 output channels; images 17 pixels
# wide; and enough pixels that the number of sums has to follow them.
@pytest.mark.parametrize("n,h,w,cin,cout,pad", [
    (16, 33, 31, 32, 32, 0), (16, 128, 128, 64, 32, 0), (16, 128, 128, 96, 32, 0), (8, 131, 117, 96, 32, 8),
    (4, 128, 128, 160, 64, 16), (128, 16, 15, 96, 32, 0), (16, 272, 15, 96, 32, 0), (16, 272, 17, 96, 64, 0),
    (16, 64, 64, 112, 176, 0), (40, 17, 130, 288, 160, 24), (16, 256, 256, 192, 192, 0), (4, 256, 256, 512, 512, 0)])
def test_sums_are_short_enough(lib, n, h, w, cin, cout, pad):
    g = torch.Generator(device="cuda").manual_seed(cin + 3 * cout + w)
    x = torch.randn(n, h, w, cin + pad, generator=g, device="cuda").relu().to(torch.bfloat16)
    dy = torch.randn(n, h, w, cout + pad, generator=g, device="cuda").to(torch.bfloat16)
    start = torch.randn(cout, 9, cin, generator=g, device="cuda")
    gw = start.clone()
    library.check(lib.dk_unet_conv3x3_wgrad(x.data_ptr() + 2 * pad, cin + pad, dy.data_ptr() + 2 * pad, cout + pad, n, h,
                                            w, cin, cout, gw.data_ptr(), None))
    # channel corners: the first and the last 48 on both sides
    ci = sorted({*range(min(48, cin)), *range(max(0, cin - 48), cin)})
    co = sorted({*range(min(48, cout)), *range(max(0, cout - 48), cout)})
    p = torch.nn.functional.pad(x[..., pad:][..., ci], (0, 0, 1, 1, 1, 1))
    flat = dy[..., pad:][..., co].double().reshape(-1, len(co))
    want = torch.stack([flat.T @ p[:, a:a + h, b:b + w].double().reshape(-1, len(ci))
                        for a in range(3) for b in range(3)], dim=1)
    got = (gw.double() - start.double())[co][:, :, ci]
    # A sum's K steps of 16 pixels: a part of the pixels for each of the blocks of 64 x 64 channels and one tap that
    # give an SM eight, at least 512 pixels, a third more for ragged tiles, at most 64 tiles of 16 steps.  Each step
    # truncates: half a unit of 2^-23 on average.  Then FP32 additions of the sums onto values of about their size.
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    blocks = 9 * -(-cin // 64) * -(-cout // 64)
    pixels = max(512, n * h * w / -(-8 * sms // blocks))
    steps = min(1.3 * pixels / 16 + 1, 1024)
    scale = float(want.norm() / start[co][:, :, ci].double().norm())  # the start's rounding, relative to the sums
    assert float((got - want).norm() / want.norm()) <= (steps + 8) * 2.0 ** -24 + 2.0 ** -24 * (1.0 + 1.0 / scale)
