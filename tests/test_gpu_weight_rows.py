"""Staging of the weights in 16-byte copies: the forward's rows as they lie, the input gradient's copy by taps.  Neither changes the
order of addition, so both are compared bit for bit with the forms that a misaligned or missing buffer takes, and with the oracle or
float64.  The plans say that the forms in question are the ones that run."""
import pytest
import torch
import torch.nn.functional as F

from oracle import adder_oracle as O

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
U = 2.0 ** -24


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


# two chunks of two channels (the last 36 floats of w), one block of channels and less, ragged outputs and inputs, several blocks, stride 2;
# the fourth runs the tiled kernel where w is not aligned
@pytest.mark.parametrize("shape", [(64, 64, 64, 14, 14, 3, 1, 1), (40, 36, 100, 17, 9, 3, 1, 1), (64, 128, 128, 28, 28, 3, 1, 1),
                                   (73, 4, 96, 8, 12, 3, 1, 1), (100, 8, 60, 30, 9, 3, 2, 1), (20, 32, 64, 20, 20, 1, 1, 0),
                                   (64, 512, 128, 14, 14, 1, 1, 0), (48, 68, 60, 12, 20, 1, 1, 0)],
                         ids=lambda s: "n%d_c%dto%d_%dx%d_k%ds%dp%d" % s)
def test_forward_rows(shape):
    from addernetcuda_b200 import _lib
    from addernetcuda_b200 import adder_cuda as ac
    n, ci, co, h, wd, k, s, p = shape
    plan = lambda flags: _lib.describe_plan(0, n, ci, h, wd, co, k, s, p, flags).split(";")[0]
    assert "_rows" in plan(0) and "_rows" not in plan(_lib.FLAG_UNALIGNED)
    x, w, _ = _tensors(*shape)
    out = ac.forward(x, w, s, p)
    assert torch.equal(out, ac.forward(x, _shifted(w), s, p))
    assert torch.equal(out, ac.forward(_shifted(x), w, s, p))
    ok, _, msg = O.compare("out", out[:2], O.adder2d_forward_direct(x[:2].cpu(), w.cpu(), s, p))
    assert ok, msg


def _gradient_of_one_image(x, w, g, k, s, p):
    """(input gradient, sum of |g| over its taps) in float64."""
    cols = F.unfold(x.double()[None], k, padding=p, stride=s)[0]
    w64, g64 = w.double().reshape(w.shape[0], -1), g.double().reshape(g.shape[0], -1)
    gcols = torch.zeros_like(cols)
    for c in range(w.shape[0]):
        gcols += (w64[c, :, None] - cols).clamp(-1, 1) * g64[c]
    back = lambda t: F.fold(t[None], x.shape[1:], k, padding=p, stride=s)[0]
    return back(gcols), back(g64.abs().sum(0).expand(cols.shape[0], -1))


# tiles of 64 and 32 input channels, ragged channels and planes, classes of a stride, windows of 25 and 49 taps (5x5: the first for the
# saturating form alone, the last on the tile of 16)
COPIES = [(128, 64, 64, 28, 28, 3, 1, 1), (160, 60, 130, 17, 29, 3, 1, 1), (224, 128, 66, 28, 28, 3, 2, 1), (24, 20, 33, 90, 90, 5, 1, 2),
          (8, 512, 512, 14, 14, 3, 1, 1), (1, 512, 512, 16, 16, 7, 1, 3), (7, 640, 720, 7, 7, 5, 1, 2)]


@pytest.mark.parametrize("fast", [0, 1], ids=["exact", "saturating"])
@pytest.mark.parametrize("shape", COPIES, ids=lambda s: "n%d_c%dto%d_%dx%d_k%ds%dp%d" % s)
def test_input_gradient_from_a_copy_by_taps(shape, fast):
    from addernetcuda_b200 import _lib
    x, w, g = _tensors(*shape)
    n, ci, co, h, wd, k, s, p = shape
    lib = _lib.load()
    geom = (n, ci, h, wd, co, k, k, s, s, p, p, 1, 1)
    need = lib.adder_b200_conv_backward_input_workspace_bytes(*geom)
    assert need == w.numel() * 4
    if k == 3:
        assert "staging=tap_rows" in _lib.describe_plan(1, n, ci, h, wd, co, k, s, p, fast)
    stream = torch.cuda.current_stream().cuda_stream
    ws = torch.empty(w.numel() + 8, device=DEV)
    poison = 1234.5

    def run(pointer, bytes_given, flags=0, gx=None):
        ws.fill_(poison)
        gx = torch.full_like(x, float("nan")) if gx is None else gx
        _lib.check(lib.adder_b200_conv_backward_input_with_workspace(g.data_ptr(), x.data_ptr(), w.data_ptr(), gx.data_ptr(), pointer,
                                                                     bytes_given, *geom, flags | fast, stream), "backward_input")
        return gx

    gx = run(ws.data_ptr(), need)
    # the copy is made, in [tap][output channel][input channel], and nothing lies behind it
    if fast or shape != (24, 20, 33, 90, 90, 5, 1, 2):
        assert torch.equal(ws[:w.numel()], w.permute(2, 3, 0, 1).flatten())
        assert (ws[w.numel():] == poison).all()
    else:
        assert (ws == poison).all()
    start = torch.full_like(x, 0.5)
    assert torch.equal(run(ws.data_ptr(), need, _lib.FLAG_ACCUMULATE, start.clone()), start + gx)
    for pointer, size in ((ws.data_ptr(), need - 4), (ws.data_ptr() + 4, need), (None, need)):      # too small, misaligned, none: as without
        assert torch.equal(gx, run(pointer, size))
        assert (ws == poison).all()
    want, size = _gradient_of_one_image(x[0], w, g[0], k, s, p)
    assert ((gx[0].double() - want).abs() <= 4 * (co * k * k + 4) * U * size).all()


def test_layers_take_the_scratch_from_torch():
    """The module's backward, other windows through the C++ path, with the copy's scratch: the bits of the entry point without."""
    from addernetcuda_b200 import _lib, adder
    shape = (8, 64, 64, 64, 64, 5, 1, 2)
    n, ci, co, h, wd, k, s, p = shape
    x, w, g = _tensors(*shape)
    geom = (n, ci, h, wd, co, k, k, s, s, p, p, 1, 1)
    lib = _lib.load()
    assert lib.adder_b200_conv_backward_input_workspace_bytes(*geom) > 0
    layer = adder.adder2d(ci, co, k, stride=s, padding=p).to(DEV)
    with torch.no_grad():
        layer.adder.copy_(w)
    xg = x.clone().requires_grad_()
    layer(xg).backward(g)
    want = torch.empty_like(x)
    _lib.check(lib.adder_b200_conv_backward_input(g.data_ptr(), x.data_ptr(), w.data_ptr(), want.data_ptr(), *geom, int(adder.FAST_CLAMP),
                                                  torch.cuda.current_stream().cuda_stream), "backward_input")
    assert torch.equal(xg.grad, want)
