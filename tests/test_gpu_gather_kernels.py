"""The gathering kernels (csrc/adder_fwd_gather.cu, csrc/adder_gx_gather.cu) at the edges of their tiles: one output a thread up to
full tiles, ragged channels and pixels, blocks of channels with a remainder, 16-byte and 4-byte staging, the residue classes of a
stride, windows of any extent; the folded batch norm, residual and ReLU of their epilogue, and the statistics made beside them.

Against float64 on the same device, element by element.  u = 2^-24 bounds each rounding, K terms are added in fp32 in some order:
  forward     every term |x - w| has one sign: |error| <= (K + 1) u |out|
  gradient    |error| <= (K + 3) u sum |g| for clamp(w - x) (|clamp| <= 1); the saturating form adds 2 sat((w - x + 1) / 2) g and
              takes sum g off again, so 4 (K + 4) u sum |g| holds for both
  epilogue    a product and two sums more: 3 u (|out scale| + |shift| + |residual|)."""
import pytest
import torch
import torch.nn.functional as F

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
U = 2.0 ** -24

# (n, ci, co, h, w, k, stride, pad)
CASES = [(1, 16, 16, 32, 32, 3, 1, 1), (1, 5, 7, 5, 5, 3, 1, 1), (1, 66, 67, 8, 8, 3, 1, 1), (3, 64, 64, 9, 7, 3, 1, 0),
         (2, 27, 45, 29, 31, 3, 1, 1), (6, 130, 129, 14, 14, 3, 1, 1), (40, 65, 70, 15, 13, 3, 2, 1), (2, 64, 72, 16, 16, 3, 2, 1),
         (1, 33, 36, 4, 4, 1, 1, 0), (3, 70, 130, 12, 12, 1, 1, 0), (20, 100, 260, 11, 11, 1, 1, 0), (2, 64, 96, 28, 28, 1, 2, 0),
         (3, 40, 33, 13, 15, 1, 2, 0), (300, 3, 20, 20, 20, 3, 1, 1), (64, 160, 24, 28, 28, 1, 1, 0), (2, 9, 12, 17, 19, 5, 1, 2),
         (3, 40, 16, 14, 14, 1, 2, 0), (3, 40, 16, 13, 14, 1, 2, 0), (2, 70, 16, 34, 34, 1, 2, 0),
         (1, 6, 33, 23, 30, 3, 4, 1), (2, 20, 18, 12, 16, 2, 2, 0), (1, 3, 40, 33, 33, 7, 2, 3)]


def _columns(t, k, s, p):
    return F.unfold(t.double(), k, padding=p, stride=s)


@pytest.mark.parametrize("case", CASES, ids=lambda c: "n%d_c%dto%d_%dx%d_k%ds%dp%d" % c)
def test_gathering_kernels(case):
    from addernetcuda_b200 import adder_cuda as ac
    from addernetcuda_b200.adder import adder2d
    n, ci, co, h, w, k, s, p = case
    gen = torch.Generator(device=DEV).manual_seed(sum(case))
    rand = lambda *shape: torch.randn(*shape, device=DEV, generator=gen)
    layer = adder2d(ci, co, k, stride=s, padding=p).to(DEV)
    with torch.no_grad():
        layer.adder.copy_(rand(co, ci, k, k))
    wt = layer.adder.detach()
    x, terms = rand(n, ci, h, w), ci * k * k
    xg = x.clone().requires_grad_()
    out = layer(xg)
    g, scale, shift, res = rand(*out.shape), rand(co), rand(co), rand(*out.shape)
    out.backward(g)
    grads = [xg.grad]
    with torch.no_grad():
        fused = layer.forward_affine(x, scale, shift, res, True)
    assert (fused is not None) == (k in (1, 3) and s in (1, 2))
    if fused is not None:
        grads += [ac.backward_input(g, x, wt, s, p, fast_clamp=fast) for fast in (False, True)]
        y, st = ac.forward(x, wt, s, p, stats=True)
        assert torch.equal(y, out)
        if st.shape[1]:
            y64 = y.double()
            torch.testing.assert_close(st[:, :, 0].sum(1), y64.sum((0, 2, 3)), rtol=1e-6, atol=0)
            torch.testing.assert_close(st[:, :, 1].sum(1), (y64 * y64).sum((0, 2, 3)), rtol=1e-6, atol=0)

    w64 = wt.double().reshape(co, terms)
    for i in range(n):
        cols = _columns(x[i:i + 1], k, s, p)[0]                                   # terms x positions
        want = torch.empty(co, cols.shape[1], device=DEV, dtype=torch.float64)
        gcols = torch.zeros_like(cols)
        g64 = g[i].double().reshape(co, -1)
        for c in range(co):
            d = w64[c, :, None] - cols
            want[c] = -d.abs().sum(0)
            gcols += d.clamp(-1, 1) * g64[c]
        want = want.reshape(out[i].shape)
        assert ((out[i].double() - want).abs() <= (terms + 1) * U * want.abs()).all()
        sc, sh, r = scale.double()[:, None, None], shift.double()[:, None, None], res[i].double()
        bound = (terms + 1) * U * (want * sc).abs() + 3 * U * ((want * sc).abs() + sh.abs() + r.abs())
        if fused is not None:
            assert ((fused[i].double() - (want * sc + sh + r).relu()).abs() <= bound).all()

        back = lambda t: F.fold(t[None], (h, w), k, padding=p, stride=s)[0]
        want_gx = back(gcols)
        size = back(g64.abs().sum(0).expand(terms, -1))
        for got in grads:
            assert ((got[i].double() - want_gx).abs() <= 4 * (co * k * k + 4) * U * size).all()


@pytest.mark.parametrize("fast", [0, 1], ids=["exact", "saturating"])
@pytest.mark.parametrize("hw", [(9, 11), (10, 11), (9, 12), (10, 12), (8, 16), (1, 1), (2, 1), (1, 2)], ids=lambda v: "%dx%d" % v)
@pytest.mark.parametrize("strides", [(2, 2), (2, 3), (3, 2), (3, 3), (1, 2), (2, 1), (5, 2)], ids=lambda v: "s%dx%d" % v)
def test_unsampled_pixels_get_zeros(strides, hw, fast):
    """A strided 1x1 layer reads one pixel of each block: the input gradient writes a zero to every other one, whatever lay there, with
    16-byte, 8-byte or single stores."""
    from addernetcuda_b200 import _lib
    (h, w), (sh, sw), n, ci, co = hw, strides, 3, 70, 66
    gen = torch.Generator(device=DEV).manual_seed(h * w + sh)
    x, wt = torch.randn(n, ci, h, w, device=DEV, generator=gen), torch.randn(co, ci, device=DEV, generator=gen)
    g = torch.randn(n, co, -(-h // sh), -(-w // sw), device=DEV, generator=gen)
    gx = torch.full_like(x, float("nan"))
    _lib.check(_lib.load().adder_b200_conv_backward_input(g.data_ptr(), x.data_ptr(), wt.data_ptr(), gx.data_ptr(), n, ci, h, w, co, 1, 1,
                                                          sh, sw, 0, 0, 1, 1, fast, torch.cuda.current_stream().cuda_stream), "backward_input")
    want = torch.zeros(n, ci, h, w, device=DEV, dtype=torch.float64)
    d = (wt.double()[None, :, :, None, None] - x.double()[:, None, :, ::sh, ::sw]).clamp(-1, 1)
    want[:, :, ::sh, ::sw] = (d * g.double()[:, :, None]).sum(1)
    size = torch.zeros_like(want)
    size[:, :, ::sh, ::sw] = g.double().abs().sum(1, keepdim=True)
    assert ((gx.double() - want).abs() <= 4 * (co + 4) * U * size).all()
