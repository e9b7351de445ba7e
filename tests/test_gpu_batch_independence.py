"""An image's output and input gradient do not depend on the batch it sits in, bit for bit: kernels and tiles follow the size of
the launch, the order in which an element's terms are added does not.  Both forms of the clamp; windows of the standard and of
other extents; batches that take different tiles."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"

# (ci, co, h, w, k, stride, pad, batches)
CASES = [(128, 128, 14, 14, 3, 1, 1, (1, 8, 16, 64)), (64, 64, 15, 15, 3, 1, 1, (1, 8, 64)), (256, 256, 14, 14, 3, 1, 1, (1, 8, 64)),
         (40, 72, 9, 11, 3, 1, 1, (1, 5, 64)), (96, 64, 16, 16, 3, 2, 1, (1, 8, 100)), (256, 64, 14, 14, 1, 1, 0, (1, 8, 64)),
         (100, 60, 7, 9, 1, 1, 0, (1, 8, 64)), (64, 128, 28, 28, 1, 2, 0, (1, 8, 64)), (16, 16, 32, 32, 3, 1, 1, (1, 8, 64))]
# beyond the standard geometries: blocks of channels below, at and past 16 and 32, even and odd numbers of taps
OTHER = [(48, 40, 20, 20, 5, 1, 2, (1, 6, 64)), (36, 33, 18, 18, 2, 2, 0, (1, 16, 64)), (16, 24, 21, 23, 7, 2, 3, (1, 8, 64)),
         (17, 20, 12, 12, 5, 1, 2, (1, 8, 128)), (64, 64, 14, 14, 4, 1, 1, (1, 8, 64))]


@pytest.mark.parametrize("fast", [False, True], ids=["exact", "saturating"])
@pytest.mark.parametrize("case", CASES + OTHER, ids=lambda c: "c%dto%d_%dx%d_k%ds%dp%d" % c[:7])
def test_an_image_does_not_see_its_batch(case, fast, monkeypatch):
    from addernetcuda_b200 import adder
    ci, co, h, w, k, s, p, batches = case
    monkeypatch.setattr(adder, "FAST_CLAMP", fast)
    gen = torch.Generator(device=DEV).manual_seed(ci + co)
    layer = adder.adder2d(ci, co, k, stride=s, padding=p).to(DEV)
    x = torch.randn(max(batches), ci, h, w, device=DEV, generator=gen)
    g = None
    results = []
    for n in sorted(batches, reverse=True):
        xn = x[:n].clone().requires_grad_()
        out = layer(xn)
        if g is None:
            g = torch.randn(out.shape, device=DEV, generator=gen)
        out.backward(g[:n].contiguous())
        results.append((n, out.detach(), xn.grad))
    for n, out, gx in results[1:]:
        assert torch.equal(out, results[0][1][:n]), f"output of batch {n}"
        assert torch.equal(gx, results[0][2][:n]), f"input gradient of batch {n}"
