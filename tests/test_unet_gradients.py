"""The gradient kernels of the learned denoiser's layers at the edges of their
tiles, against the same sums in FP64."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

from denrimrendererkit_gb300 import library

pytestmark = pytest.mark.gpu


def _ptr(t, offset=0):
    return t.data_ptr() + offset * t.element_size()


def rel_rms(a, b):
    return float((a.double() - b.double()).norm() / b.double().norm().clamp(min=1e-300))


@pytest.fixture(scope="module")
def lib():
    return library.load()


# Tiles of 16 x 16 pixels, blocks of 32 input channels, up to 160 output
# channels per CTA: one pixel, whole tiles, one over, narrow and wide images,
# a last block of 16 channels, two output blocks, strided channel slices.
@pytest.mark.parametrize("n,h,w,cin,cout,pad", [(1, 1, 1, 16, 16, 0), (1, 16, 16, 32, 32, 0), (2, 17, 15, 48, 32, 8),
                                                (3, 5, 70, 288, 160, 0), (2, 33, 31, 32, 176, 16),
                                                (16, 64, 64, 64, 96, 0), (1, 40, 130, 160, 64, 24),
                                                (5, 16, 160, 96, 32, 0), (1, 8, 300, 16, 288, 0)])
def test_weight_gradient_tiles(lib, n, h, w, cin, cout, pad):
    g = torch.Generator().manual_seed(cin + 3 * cout + w)
    x = torch.randn(n, h, w, cin + pad, generator=g).to(torch.bfloat16)
    dy = torch.randn(n, h, w, cout + pad, generator=g).to(torch.bfloat16)
    xd, dyd = x.cuda(), dy.cuda()
    off = pad // 16 * 8  # a slice that starts inside the pixel's channels
    start = torch.randn(cout, 9, cin, generator=g)
    gw = start.cuda()
    library.check(lib.dk_unet_conv3x3_wgrad(_ptr(xd, off), cin + pad, _ptr(dyd, off), cout + pad, n, h, w, cin, cout,
                                            _ptr(gw), None))
    p = torch.nn.functional.pad(x[..., off:off + cin].double(), (0, 0, 1, 1, 1, 1))
    flat = dy[..., off:off + cout].double().reshape(-1, cout)
    want = torch.stack([flat.T @ p[:, dy_:dy_ + h, dx:dx + w].reshape(-1, cin) for dy_ in range(3) for dx in range(3)],
                       dim=1)
    torch.cuda.synchronize()
    # FP32 sums of exact products: at most one rounding of 2^-23 per K step of 16 pixels and per added partial sum
    tol = 4 * (n * h * w / 16 + 160) * 2.0 ** -23
    assert rel_rms(gw.cpu().double() - start.double(), want) <= tol


@pytest.mark.parametrize("c,pad", [(8, 0), (16, 0), (24, 8), (32, 2), (96, 0), (160, 128), (256, 0), (2, 0)])
@pytest.mark.parametrize("pixels", [1, 63, 4099])
def test_relu_and_bias_gradient(lib, c, pad, pixels):
    g = torch.Generator().manual_seed(c + pixels)
    ld = c + pad
    out = torch.randn(pixels, ld, generator=g).relu().to(torch.bfloat16)
    dout = torch.randn(pixels, ld, generator=g).to(torch.bfloat16)
    outd, doutd = out.cuda(), dout.cuda()
    want = torch.where(out[:, :c] > 0, dout[:, :c], torch.zeros_like(dout[:, :c]))
    sums = want.double().sum(0)
    # sums of at most `pixels` FP32 terms in any order
    tol = pixels * 2.0 ** -23 * want.double().abs().sum(0).max().item() + 1e-30

    def fresh():
        return torch.full((pixels, ld), 9.0, dtype=torch.bfloat16, device="cuda"), torch.zeros(c, device="cuda")

    both, db = fresh()
    library.check(lib.dk_unet_relu_bias_backward(_ptr(outd), ld, _ptr(doutd), ld, _ptr(both), ld, c, pixels, _ptr(db),
                                                 None))
    one, db1 = fresh()
    library.check(lib.dk_unet_relu_backward(_ptr(outd), ld, _ptr(doutd), ld, _ptr(one), ld, c, pixels, None))
    library.check(lib.dk_unet_bias_grad(_ptr(one), ld, c, pixels, _ptr(db1), None))
    torch.cuda.synchronize()
    for t, b in ((both, db), (one, db1)):
        assert torch.equal(t[:, :c].cpu(), want) and bool((t[:, c:] == 9.0).all())
        assert float((b.cpu().double() - sums).abs().max()) <= tol
