"""Weight gradient on the tensor cores (csrc/adder_gw_mma.cu): exact three-way bf16 splits with fp32 accumulation.

Compared with a float64 evaluation on the same device, at the edges of its tiles: channels below, at and past a tile, both ways
of issuing (stacked, split), strides, halos, planes narrower than a step, slices with one chunk, and sums long enough to be
drained many times.  Bound: a slice's sum loses at most 16 truncations of 2^-23 of the running sum before it is moved (2e-6, reached
only if all values have one sign; random signs stay near 1e-7), and everything after that is rounded to nearest."""
import pytest
import torch
import torch.nn.functional as F

pytestmark = pytest.mark.gpu
DEV = "cuda:0"

# (n, ci, co, h, w, k, stride, pad)
CASES = [(64, 32, 32, 18, 18, 3, 1, 1), (70, 16, 48, 20, 20, 3, 1, 1), (50, 27, 45, 29, 31, 3, 1, 1), (60, 40, 41, 13, 17, 3, 2, 1),
         (9, 130, 70, 15, 13, 3, 1, 1), (40, 128, 129, 9, 7, 3, 2, 1), (16, 256, 256, 14, 14, 3, 1, 0), (9, 200, 264, 11, 11, 1, 1, 0),
         (9, 96, 520, 28, 26, 1, 2, 0), (2, 64, 64, 112, 112, 3, 1, 1), (1, 64, 72, 7, 200, 3, 1, 1)]


@pytest.mark.parametrize("one_sign", [False, True])
@pytest.mark.parametrize("case", CASES, ids=lambda c: "n%d_c%dto%d_%dx%d_k%ds%dp%d" % c)
def test_tensor_core_weight_gradient(case, one_sign):
    from addernetcuda_b200 import _lib, adder_cuda as ac
    n, ci, co, h, w, k, s, p = case
    assert _lib.describe_plan(2, n, ci, h, w, co, k, s, p).startswith("gw mma")
    gen = torch.Generator(device=DEV).manual_seed(n + ci + co)
    x = torch.randn(n, ci, h, w, device=DEV, generator=gen)
    wt = torch.randn(co, ci, k, k, device=DEV, generator=gen)
    ho, wo = (h + 2 * p - k) // s + 1, (w + 2 * p - k) // s + 1
    g = torch.randn(n, co, ho, wo, device=DEV, generator=gen)
    if one_sign:
        x, g = x.abs() + 1, g.abs() + 1
    got = ac.backward_weight(g, x, wt, s, p, eta=0.0)
    want = torch.zeros(co, ci * k * k, device=DEV, dtype=torch.float64)
    for i in range(n):
        cols = F.unfold(x[i:i + 1].double(), k, padding=p, stride=s)[0]
        gi = g[i].double().reshape(co, -1)
        want += gi @ cols.T - wt.double().reshape(co, -1) * gi.sum(1, keepdim=True)
    want = want.reshape(wt.shape)
    rel = float((got.double() - want).norm() / want.norm())
    print("    rel", rel)
    assert rel <= (2e-6 if one_sign else 5e-7), rel
    assert torch.equal(ac.backward_weight(g, x, wt, s, p, eta=0.0), got)     # same bits twice


# gradients of 9 to 65,790 elements: both block widths of the one-launch finish, its largest size and the first beyond it, with remainders
@pytest.mark.parametrize("ci,co", [(1, 1), (16, 29), (17, 31), (85, 85), (85, 86)])
def test_finish_of_the_weight_gradient(ci, co):
    """Norm and rescale.  The slices are added in double, so what the sums of 192 products lose before that (192 u of their
    size, u = 2^-24) and the roundings of scale and product bound the norm of the error."""
    from addernetcuda_b200 import adder_cuda as ac
    gen = torch.Generator(device=DEV).manual_seed(ci + co)
    x = torch.randn(3, ci, 8, 8, device=DEV, generator=gen)
    w = torch.randn(co, ci, 3, 3, device=DEV, generator=gen)
    g = torch.randn(3, co, 8, 8, device=DEV, generator=gen)
    got, norm = ac.backward_weight(g, x, w, 1, 1, eta=0.2, return_norm=True)
    cols = F.unfold(x.double(), 3, padding=1)
    g64 = g.double().reshape(3, co, -1)
    want = torch.einsum("ncp,nkp->ck", g64, cols) - w.double().reshape(co, -1) * g64.sum((0, 2))[:, None]
    size = torch.einsum("ncp,nkp->ck", g64.abs(), cols.abs()) + w.double().reshape(co, -1).abs() * g64.abs().sum((0, 2))[:, None]
    bound = float((192 + 8) * 2.0 ** -24 * size.norm() / want.norm())
    assert abs(float(norm) - float(want.norm())) <= bound * float(want.norm())
    want *= 0.2 * want.numel() ** 0.5 / want.norm()
    assert float((got.double().reshape(co, -1) - want).norm()) <= 2 * bound * float(want.norm())


@pytest.mark.parametrize("case", [(8, 128, 128, 28, 28, 3, 1, 1), (8, 256, 256, 14, 14, 3, 1, 1), (1, 128, 128, 32, 32, 3, 1, 1)],
                         ids=lambda c: "n%d_c%dto%d_%dx%d_k%ds%dp%d" % c)
def test_fixed_scratch_takes_layers_whose_tensor_core_slices_do_not_fit(case):
    """The entry point with 8 MiB of its own falls back to the fp32 kernels, which need less.  K = n ho wo products added in fp32, in
    slices that are added in double: (K + 8) u of their size (u = 2^-24) bounds the error, as below for the finish."""
    from addernetcuda_b200 import _lib
    n, ci, co, h, w, k, s, p = case
    lib = _lib.load()
    assert lib.adder_b200_backward_weight_workspace_bytes(n, ci, h, w, co, k, s, p) > lib.adder_b200_static_scratch_bytes()
    gen = torch.Generator(device=DEV).manual_seed(n + ci)
    x = torch.randn(n, ci, h, w, device=DEV, generator=gen)
    wt = torch.randn(co, ci, k, k, device=DEV, generator=gen)
    g = torch.randn(n, co, h, w, device=DEV, generator=gen)
    got, want, size = torch.full_like(wt, 7.0), 0.0, 0.0
    stream = torch.cuda.current_stream().cuda_stream
    status = lib.adder_b200_backward_weight_static(g.data_ptr(), x.data_ptr(), wt.data_ptr(), got.data_ptr(), 0.0, None, n, ci, h, w, co,
                                                   k, s, p, stream)
    assert status == 0, status
    for i in range(n):
        cols, gi, w64 = F.unfold(x[i:i + 1].double(), k, padding=p)[0], g[i].double().reshape(co, -1), wt.double().reshape(co, -1)
        want += gi @ cols.T - w64 * gi.sum(1, keepdim=True)
        size += gi.abs() @ cols.abs().T + w64.abs() * gi.abs().sum(1, keepdim=True)
    assert ((got.double().reshape(co, -1) - want).abs() <= (n * h * w + 8) * 2.0 ** -24 * size).all()


@pytest.mark.parametrize("value", [float("inf"), float("nan")])
@pytest.mark.parametrize("case", [(9, 130, 70, 15, 13, 3, 1, 1), (40, 128, 129, 9, 7, 3, 2, 1), (3, 16, 16, 8, 8, 3, 1, 1), (3, 85, 86, 8, 8, 3, 1, 1)],
                         ids=lambda c: "n%d_c%dto%d_%dx%d_k%ds%dp%d" % c)
def test_a_value_that_is_not_finite_does_not_blow_up_the_gradient(case, value):
    """adder.py:78 of the reference divides by norm(p=2).clamp(min=1e-12): a norm of NaN gives NaN everywhere, one of infinity zero for
    what is finite.  Tensor-core and fp32 kernels, finish in one launch and in three."""
    from addernetcuda_b200 import adder_cuda as ac
    n, ci, co, h, w, k, s, p = case
    gen = torch.Generator(device=DEV).manual_seed(ci)
    x = torch.randn(n, ci, h, w, device=DEV, generator=gen)
    g = torch.randn(n, co, (h + 2 * p - k) // s + 1, (w + 2 * p - k) // s + 1, device=DEV, generator=gen)
    x[0, 0, h // 2, w // 2] = value
    got = ac.backward_weight(g, x, torch.randn(co, ci, k, k, device=DEV, generator=gen), s, p)
    assert got.isnan().any() and (got[~got.isnan()] == 0).all()
