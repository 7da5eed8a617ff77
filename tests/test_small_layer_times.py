"""The convolution calls on layers of a few pixels: the kernel that large
layers want has set-up of its own, which a small one must not pay."""
import pytest

torch = pytest.importorskip("torch")

from denrimrendererkit_gb300 import DenrimRenderer, library

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def lib(dk_lib):
    DenrimRenderer(0)
    return library.load()


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


def weight_gradient(lib, n, h, w, cin, cout):
    x = torch.randn(n, h, w, cin, device="cuda").to(torch.bfloat16)
    dy = torch.randn(n, h, w, cout, device="cuda").to(torch.bfloat16)
    gw = torch.zeros(cout, 9, cin, device="cuda")
    return lambda: library.check(lib.dk_unet_conv3x3_wgrad(x.data_ptr(), cin, dy.data_ptr(), cout, n, h, w, cin, cout,
                                                           gw.data_ptr(), None))


@pytest.mark.parametrize("small,large", [((1, 8, 8, 128, 128), (16, 64, 64, 128, 128)),
                                         ((1, 4, 4, 160, 160), (16, 64, 64, 160, 160))])
def test_small_weight_gradient(lib, small, large):
    # a 1,024th and a 4,096th of the work; set-up and read-out alone took 0.7 of the large one's time
    assert microseconds(weight_gradient(lib, *small)) <= 0.4 * microseconds(weight_gradient(lib, *large))


def forward(lib, n, h, w, cin, cout):
    x = torch.randn(n, h, w, cin, device="cuda").to(torch.bfloat16)
    weight = (torch.randn(cout, 9, cin, device="cuda") / (3 * cin ** 0.5)).to(torch.bfloat16)
    bias = torch.randn(cout, device="cuda")
    out = torch.empty(n, h, w, cout, device="cuda", dtype=torch.bfloat16)
    return out, lambda: library.check(lib.dk_unet_conv3x3(x.data_ptr(), n, h, w, cin, cin, weight.data_ptr(),
                                                          bias.data_ptr(), cout, out.data_ptr(), cout, 0, 1, 0, None))


# Many images a pixel or a few wide or high, which fill little of an 8 x 16 tile; and one that fills tiles well.
@pytest.mark.parametrize("n,h,w,cin,cout,other", [(353, 40, 1, 160, 192, 2), (620, 4, 33, 176, 208, 2),
                                                  (1299, 1, 3, 208, 288, 0), (16, 64, 64, 96, 96, 2)])
def test_forward_takes_the_better_kernel(lib, n, h, w, cin, cout, other):
    out, call = forward(lib, n, h, w, cin, cout)
    chosen = microseconds(call)
    image = out.clone()
    library.check(lib.dk_unet_set_conv_path(other))
    try:
        alternative = microseconds(call)
    finally:
        library.check(lib.dk_unet_set_conv_path(3))
    assert torch.equal(image, out)  # the same products in the same order
    assert chosen <= 1.15 * alternative
