"""The grouped optimiser step against one call per tensor and against FP64."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

from denrimrendererkit_gb300 import abi, library

pytestmark = pytest.mark.gpu

# (cout, cin): whole 32 x 32 tiles, 16-channel remainders, one below four, more groups than one launch takes
LAYERS = [(32, 32), (16, 48), (160, 288), (96, 16), (6, 5), (1, 1)] + [(16, 16)] * 40


def test_groups_equal_single_calls():
    lib = library.load()
    g = torch.Generator().manual_seed(3)
    sets = [[], []]
    for cout, cin in LAYERS:
        n = cout * 9 * cin
        base = [torch.randn(n, generator=g), torch.randn(n, generator=g) * 1e-3, torch.randn(n, generator=g) * 1e-4,
                torch.rand(n, generator=g) * 1e-6]
        for s in sets:
            s.append([t.clone().cuda() for t in base] + [torch.zeros(n, dtype=torch.bfloat16, device="cuda")
                                                         for _ in range(2)])
    lr, b1, b2, eps, step = 1e-3, 0.9, 0.999, 1e-8, 7
    rows = []
    for k, ((cout, cin), t) in enumerate(zip(LAYERS, sets[0])):
        flip = t[5].data_ptr() if k % 5 != 4 or k < 5 else None  # some without a transposed copy
        rows.append(tuple(x.data_ptr() for x in t[:5]) + (flip, t[0].numel(), cout, cin, 0))
        t1 = sets[1][k]
        library.check(lib.dk_unet_adam(*(x.data_ptr() for x in t1[:4]), t1[0].numel(), lr, b1, b2, eps, step,
                                       t1[4].data_ptr(), t1[5].data_ptr() if flip else None, cout, cin, None))
    library.check(lib.dk_unet_adam_groups((abi.AdamGroup * len(rows))(*rows), len(rows), lr, b1, b2, eps, step, None))
    torch.cuda.synchronize()
    for a, b in zip(*sets):
        for x, y in zip(a, b):
            assert torch.equal(x, y)


def test_group_without_a_tensor_is_refused():
    lib = library.load()
    row = abi.AdamGroup()
    row.count = 4
    with pytest.raises(library.DenrimError):
        library.check(lib.dk_unet_adam_groups(row, 1, 1e-3, 0.9, 0.999, 1e-8, 1, None))
