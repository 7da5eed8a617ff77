"""The loss and output kernels with tensors that take their wide loads and
stores and with ones that do not: the same values."""
import pytest

torch = pytest.importorskip("torch")

from denrimrendererkit_gb300 import library

pytestmark = pytest.mark.gpu


def _ptr(t, offset=0):
    return t.data_ptr() + offset * t.element_size()


@pytest.mark.parametrize("residual", [False, True])
@pytest.mark.parametrize("pixels", [1, 255, 4097])
def test_layouts_agree(residual, pixels):
    lib = library.load()
    g = torch.Generator().manual_seed(pixels)
    pred, base = (torch.randn(pixels, 3, generator=g).to(torch.bfloat16) for _ in range(2))
    target = torch.rand(pixels, 4, generator=g).cuda()
    grads, losses, images = [], [], []
    for ldp, ldb, ldg, off in ((16, 16, 16, 0), (3, 16, 16, 0), (16, 5, 16, 0), (16, 16, 17, 0), (20, 20, 16, 1)):
        p = torch.zeros(pixels * ldp + 8, dtype=torch.bfloat16, device="cuda")
        b = torch.zeros(pixels * ldb + 8, dtype=torch.bfloat16, device="cuda")
        p[off:off + pixels * ldp].view(pixels, ldp)[:, :3] = pred.cuda()
        b[off:off + pixels * ldb].view(pixels, ldb)[:, :3] = base.cuda()
        grad = torch.full((pixels, ldg), 5.0, dtype=torch.bfloat16, device="cuda")
        loss, out = torch.zeros(1, device="cuda"), torch.empty(pixels, 4, device="cuda")
        if residual:
            library.check(lib.dk_unet_l1_loss_residual(_ptr(p, off), ldp, _ptr(b, off), ldb, _ptr(target), pixels,
                                                       _ptr(grad), ldg, _ptr(loss), None))
            library.check(lib.dk_unet_unpack_output_residual(_ptr(p, off), ldp, _ptr(b, off), ldb, 1, pixels,
                                                             _ptr(target), pixels, 1, 0, 0, _ptr(out), None))
        else:
            library.check(lib.dk_unet_l1_loss(_ptr(p, off), ldp, _ptr(target), pixels, _ptr(grad), ldg, _ptr(loss),
                                              None))
            library.check(lib.dk_unet_unpack_output(_ptr(p, off), ldp, 1, pixels, _ptr(target), pixels, 1, 0, 0,
                                                    _ptr(out), None))
        torch.cuda.synchronize()
        grads.append(grad[:, :16].cpu())
        losses.append(float(loss))
        images.append(out.cpu())
    for other, image, loss in zip(grads[1:], images[1:], losses[1:]):
        assert torch.equal(other, grads[0]) and torch.equal(image, images[0])
        assert abs(loss - losses[0]) <= 1e-5 * losses[0]
    want = pred.float() + (base.float() if residual else 0.0)
    d = (want - torch.log1p(target.cpu()[:, :3])).abs().mean()
    assert abs(losses[0] - float(d)) <= 1e-4 * float(d)
