"""The optimiser's moments are rounded the same way in both entry points: the
decayed moment, then one fused addition of the new term."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

from denrimrendererkit_gb300 import DenrimRenderer, abi, library

pytestmark = pytest.mark.gpu


def fused(a, b, c):  # the product of two FP32 values is exact in FP64
    return (a.astype(np.float64) * b.astype(np.float64) + c.astype(np.float64)).astype(np.float32)


@pytest.mark.parametrize("grouped", [False, True])
def test_moments(dk_lib, grouped):
    DenrimRenderer(0)
    lib = library.load()
    n, beta1, beta2 = 9 * 32 * 36, np.float32(0.9), np.float32(0.999)
    g = torch.Generator(device="cuda").manual_seed(4)
    w, grad, m = (torch.randn(n, generator=g, device="cuda") * s for s in (0.1, 1e-3, 3e-4))
    v = torch.rand(n, generator=g, device="cuda") * 1e-6
    gh, mh, vh = (t.cpu().numpy() for t in (grad, m, v))
    one = np.float32(1.0)
    want_m = fused(np.full(n, one - beta1), gh, beta1 * mh)
    want_v = fused((one - beta2) * gh, gh, beta2 * vh)
    flip = torch.empty(n, dtype=torch.bfloat16, device="cuda")
    if grouped:
        group = abi.AdamGroup(w.data_ptr(), grad.data_ptr(), m.data_ptr(), v.data_ptr(), None, flip.data_ptr(), n, 32, 36, 0)
        library.check(lib.dk_unet_adam_groups((abi.AdamGroup * 1)(group), 1, 1e-3, 0.9, 0.999, 1e-8, 100, None))
    else:
        library.check(lib.dk_unet_adam(w.data_ptr(), grad.data_ptr(), m.data_ptr(), v.data_ptr(), n, 1e-3, 0.9, 0.999, 1e-8,
                                       100, None, flip.data_ptr(), 32, 36, None))
    torch.cuda.synchronize()
    assert np.array_equal(m.cpu().numpy(), want_m) and np.array_equal(v.cpu().numpy(), want_v)
