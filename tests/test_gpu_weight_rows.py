"""Staging of the weights in 16-byte copies: the forward's rows as they lie, the input gradient's copy by taps.  Neither changes the
order of addition, so both are compared bit for bit with the forms that a misaligned or missing buffer takes, and with the oracle."""
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


def _shifted(t):
    """The same values at an address that is no multiple of 16 bytes."""
    buf = torch.empty(t.numel() + 1, device=t.device)
    buf[1:] = t.flatten()
    return buf[1:].view(t.shape)


# one block of channels and less, ragged outputs and inputs, odd and even numbers of channel pairs, several blocks
@pytest.mark.parametrize("shape", [(64, 64, 64, 14, 14, 3, 1, 1), (40, 36, 100, 17, 9, 3, 1, 1), (64, 128, 128, 28, 28, 3, 1, 1),
                                   (73, 4, 96, 8, 12, 3, 1, 1), (20, 32, 64, 20, 20, 1, 1, 0), (64, 512, 128, 14, 14, 1, 1, 0), (48, 68, 60, 12, 20, 1, 1, 0)],
                         ids=lambda s: "n%d_c%dto%d_%dx%d_k%ds%dp%d" % s)
def test_forward_rows(shape):
    from addernetcuda_b200 import adder_cuda as ac
    x, w, _ = _tensors(*shape)
    s, p = shape[6:]
    out = ac.forward(x, w, s, p)
    assert torch.equal(out, ac.forward(x, _shifted(w), s, p))
    ok, _, msg = O.compare("out", out[:2], O.adder2d_forward_direct(x[:2].cpu(), w.cpu(), s, p))
    assert ok, msg


@pytest.mark.parametrize("fast", [False, True], ids=["exact", "saturating"])
@pytest.mark.parametrize("shape", [(128, 64, 64, 28, 28, 3, 1, 1), (160, 60, 130, 17, 29, 3, 1, 1), (224, 128, 66, 28, 28, 3, 2, 1),
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
