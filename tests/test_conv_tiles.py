"""The 2-D halo-tile convolution at the edges of its tiles, channel blocks and
weight stages: against FP64 sums, and bit for bit against the per-tap kernel
where both sum in the same order (images narrower than 128 pixels)."""
import ctypes as C

import pytest

torch = pytest.importorskip("torch")

from denrimrendererkit_gb300 import DenrimRenderer, library

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def lib(dk_lib):
    DenrimRenderer(0)
    lib = library.load()
    yield lib
    err = C.c_int(0)
    library.check(lib.dk_unet_error(C.byref(err)))
    library.check(lib.dk_unet_set_conv_path(3))
    assert err.value == 0, "a tensor-core wait timed out"


@pytest.mark.parametrize("n,h,w,cin,cout,pad,accumulate", [
    (1, 1, 1, 16, 16, 0, 0), (1, 16, 8, 64, 96, 0, 0), (2, 17, 9, 96, 96, 8, 0), (1, 15, 7, 48, 80, 0, 1),
    (3, 16, 16, 160, 160, 0, 0), (16, 64, 64, 96, 96, 0, 0), (3, 32, 32, 288, 128, 0, 0), (2, 33, 100, 224, 176, 2, 0),
    (1, 24, 60, 256, 256, 0, 0), (4, 40, 64, 512, 32, 0, 1), (1, 34, 140, 160, 64, 0, 0), (1, 20, 300, 112, 128, 24, 0),
    (16, 64, 64, 96, 224, 0, 0), (16, 64, 64, 96, 224, 0, 1), (8, 63, 61, 64, 192, 8, 0)])
def test_tiles_match(lib, n, h, w, cin, cout, pad, accumulate):
    g = torch.Generator().manual_seed(cin + cout + w)
    x = torch.randn(n, h, w, cin + pad, generator=g).to(torch.bfloat16).cuda()
    weight = (torch.randn(cout, 9, cin, generator=g) / (3 * cin ** 0.5)).to(torch.bfloat16).cuda()
    bias = torch.randn(cout, generator=g).cuda()
    prior = torch.randn(n, h, w, cout + pad, generator=g).to(torch.bfloat16).cuda()
    ldi = (cin + pad) // 8 * 8 if pad % 8 else cin + pad
    if ldi != cin + pad:
        x = x[..., :ldi].contiguous()
    outs = []
    for path in (3, 2):
        library.check(lib.dk_unet_set_conv_path(path))
        out = prior.clone()
        library.check(lib.dk_unet_conv3x3(x.data_ptr(), n, h, w, cin, ldi, weight.data_ptr(), bias.data_ptr(), cout,
                                          out.data_ptr(), cout + pad, pad, 1 - accumulate, accumulate, None))
        torch.cuda.synchronize()
        outs.append(out)
    library.check(lib.dk_unet_set_conv_path(3))
    assert torch.equal(outs[0][..., :pad], prior[..., :pad])
    if w < 128:
        assert torch.equal(outs[0], outs[1])
    p = torch.nn.functional.pad(x[..., :cin].double(), (0, 0, 1, 1, 1, 1))
    want = bias.double() + sum(p[:, dy:dy + h, dx:dx + w] @ weight[:, 3 * dy + dx].double().T
                               for dy in range(3) for dx in range(3))
    want = want + prior[..., pad:].double() if accumulate else want.clamp(min=0.0)
    got = outs[0][..., pad:].double()
    # one bf16 rounding of the result (2^-9) over the FP32 sum
    assert float((got - want).norm() / want.norm().clamp(min=1e-30)) <= 2.0 ** -8


@pytest.mark.parametrize("n,h,w,cin,cout,accumulate", [
    (1, 1, 1, 16, 272, 0), (2, 17, 9, 128, 288, 1), (16, 32, 32, 128, 288, 0), (1, 20, 150, 48, 320, 0),
    (3, 16, 8, 512, 512, 0), (1, 5, 30, 528, 272, 0)])
def test_more_output_channels_than_one_accumulator(lib, n, h, w, cin, cout, accumulate):
    g = torch.Generator().manual_seed(cin + cout + w)
    x = torch.randn(n, h, w, cin, generator=g).to(torch.bfloat16).cuda()
    weight = (torch.randn(cout, 9, cin, generator=g) / (3 * cin ** 0.5)).to(torch.bfloat16).cuda()
    bias = torch.randn(cout, generator=g).cuda()
    prior = torch.randn(n, h, w, cout, generator=g).to(torch.bfloat16).cuda()
    p = torch.nn.functional.pad(x.double(), (0, 0, 1, 1, 1, 1))
    want = bias.double() + sum(p[:, dy:dy + h, dx:dx + w] @ weight[:, 3 * dy + dx].double().T
                               for dy in range(3) for dx in range(3))
    want = want + prior.double() if accumulate else want.clamp(min=0.0)
    for path in (3, 0):
        library.check(lib.dk_unet_set_conv_path(path))
        out = prior.clone()
        library.check(lib.dk_unet_conv3x3(x.data_ptr(), n, h, w, cin, cin, weight.data_ptr(), bias.data_ptr(), cout,
                                          out.data_ptr(), cout, 0, 1 - accumulate, accumulate, None))
        torch.cuda.synchronize()
        # one bf16 rounding of the result (2^-9) over the FP32 sum
        assert float((out.double() - want).norm() / want.norm()) <= 2.0 ** -8
    library.check(lib.dk_unet_set_conv_path(3))
