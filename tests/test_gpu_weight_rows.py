"""Staging of the weights in 16-byte copies: the input gradient's copy by taps.  It does not change the order of addition, so it is
compared bit for bit with the form without scratch, and with the oracle."""
import pytest
import torch

from oracle import adder_oracle as O

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def _tensors(n, ci, co, h, w, k, s, p):
    gen = torch.Generator(device=DEV).manual_seed(n + ci + co)
    x = torch.randn(n, ci, h, w, device=DEV, generator=gen)
    wt = torch.randn(co, ci, k, k, device=DEV, generator=gen)
    g = torch.randn(n, co, (h + 2 * p - k) // s + 1, (w + 2 * p - k) // s + 1, device=DEV, generator=gen)
    return x, wt, g


@pytest.mark.parametrize("fast", [False, True], ids=["exact", "saturating"])
@pytest.mark.parametrize("shape", [(128, 64, 64, 28, 28, 3, 1, 1), (160, 36, 130, 17, 29, 3, 1, 1), (224, 128, 66, 28, 28, 3, 2, 1),
                                   (24, 20, 33, 90, 90, 5, 1, 2)], ids=lambda s: "n%d_c%dto%d_%dx%d_k%ds%dp%d" % s)
def test_input_gradient_from_a_copy_by_taps(shape, fast):
    from addernetcuda_b200 import _lib
    x, w, g = _tensors(*shape)
    n, ci, co, h, wd, k, s, p = shape
    lib = _lib.load()
    geom = (n, ci, h, wd, co, k, k, s, s, p, p, 1, 1)
    need = lib.adder_b200_conv_backward_input_workspace_bytes(*geom)
    assert need == w.numel() * 4
    stream = torch.cuda.current_stream().cuda_stream

    def run(bytes_given):
        gx = torch.empty_like(x)
        ws = torch.empty(max(bytes_given, 16), dtype=torch.uint8, device=DEV)
        _lib.check(lib.adder_b200_conv_backward_input_with_workspace(g.data_ptr(), x.data_ptr(), w.data_ptr(), gx.data_ptr(), ws.data_ptr(),
                                                                     bytes_given, *geom, int(fast), stream), "backward_input")
        return gx

    gx = run(need)
    assert torch.equal(gx, run(need - 4))          # too small: as without
    if k == 3:
        ok, _, msg = O.compare("grad_x", gx[:1], O.adder2d_backward_direct(g[:1].cpu(), x[:1].cpu(), w.cpu(), s, p)[0])
        assert ok, msg
