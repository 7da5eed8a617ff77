"""The ReLU gradient alone: of more channels than one block of threads holds,
of pixel counts around a block's, in place, and its time on a small tensor."""
import pytest

torch = pytest.importorskip("torch")

from denrimrendererkit_gb300 import DenrimRenderer, library

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def lib(dk_lib):
    DenrimRenderer(0)
    return library.load()


@pytest.mark.parametrize("c,pad", [(8, 0), (96, 8), (2040, 8), (2048, 0), (2056, 0), (4104, 24)])
@pytest.mark.parametrize("pixels", [1, 21, 300, 1000])
def test_relu_gradient(lib, c, pad, pixels):
    g = torch.Generator(device="cuda").manual_seed(c + pixels)
    ld = c + pad
    out = torch.randn(pixels, ld, generator=g, device="cuda").relu().to(torch.bfloat16)
    dout = torch.randn(pixels, ld, generator=g, device="cuda").to(torch.bfloat16)
    want = torch.where(out[:, :c] > 0, dout[:, :c], torch.zeros_like(dout[:, :c]))
    dpre = torch.full((pixels, ld), 9.0, dtype=torch.bfloat16, device="cuda")
    library.check(lib.dk_unet_relu_backward(out.data_ptr(), ld, dout.data_ptr(), ld, dpre.data_ptr(), ld, c, pixels,
                                            None))
    assert torch.equal(dpre[:, :c], want) and bool((dpre[:, c:] == 9.0).all())
    library.check(lib.dk_unet_relu_backward(out.data_ptr(), ld, dout.data_ptr(), ld, dout.data_ptr(), ld, c, pixels,
                                            None))
    assert torch.equal(dout[:, :c], want)


def microseconds(call):
    """Of one call among others on the device (median of 15 runs of ten)."""
    begin, end = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    times = []
    for _ in range(15):
        torch.cuda._sleep(400_000)  # the launches queue up behind it
        begin.record()
        for _ in range(10):
            call()
        end.record()
        torch.cuda.synchronize()
        times.append(begin.elapsed_time(end) * 100.0)
    return sorted(times)[7]


def relu_time(lib, c, pixels):
    a, b, d = (torch.randn(pixels, c, device="cuda").to(torch.bfloat16) for _ in range(3))
    return microseconds(lambda: library.check(lib.dk_unet_relu_backward(a.data_ptr(), c, b.data_ptr(), c, d.data_ptr(), c,
                                                                        c, pixels, None)))


def test_a_small_tensor_costs_a_launch(lib):
    # 2.4 MB, 0.35 us of memory time: one wave of blocks, each thread one load deep, like a single pixel; eight
    # pixels a thread in two rounds of loads took twice as long
    assert relu_time(lib, 96, 4096) <= 1.65 * relu_time(lib, 96, 1)


def test_many_channels_go_at_the_rate_of_few(lib):
    # the same 1.6 GB in rows of 4,096 and of 1,024 channels
    assert relu_time(lib, 4096, 65536) <= 1.2 * relu_time(lib, 1024, 4 * 65536)
