"""The C++ host path of the eager layer calls (csrc/host.cpp) beside what torch and the caller may do around a layer."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def _rand(*shape, seed=0):
    return torch.randn(*shape, device=DEV, generator=torch.Generator(device=DEV).manual_seed(seed + sum(shape)))


def _calls():
    """(name, function of an input that requires grad, shape of the input) of every autograd node the path makes."""
    from addernetcuda_b200 import adder
    l3, l5 = (adder.adder2d(6, 8, k, padding=k // 2).to(DEV) for k in (3, 5))
    w = torch.nn.Parameter(_rand(8, 24))
    return [("3x3", l3, l3.adder, (2, 6, 9, 10)), ("5x5", l5, l5.adder, (2, 6, 9, 10)),
            ("columns", lambda x: adder.adder.apply(w, x), w, (24, 70))]


def _grads(x, w):
    r = x.grad.clone(), w.grad.clone()
    x.grad = w.grad = None
    return r


def test_a_refused_call_raises():
    """A status other than 0 is a ValueError with the library's words, in forward and in backward: more channels than a launch has rows
    of blocks."""
    from addernetcuda_b200 import adder
    n = 4_500_000
    one = torch.ones(1, 1, device=DEV)
    with pytest.raises(ValueError, match="adder_b200_forward: .*status 3"):
        adder.adder.apply(torch.ones(n, 1, device=DEV), one)
    x = torch.ones(n, 1, device=DEV, requires_grad=True)
    out = adder.adder.apply(torch.zeros(1, n, device=DEV), x)
    with pytest.raises(ValueError, match="adder_b200_backward_input: .*status 3"):
        out.backward(one)


@pytest.mark.parametrize("i", range(3), ids=["3x3", "5x5", "columns"])
def test_a_forward_before_a_tuning_block_may_run_its_backward_inside(i):
    """The nodes keep the product library's entry points while another library is active."""
    from addernetcuda_b200 import _lib
    _, call, w, shape = _calls()[i]
    x = _rand(*shape).requires_grad_()
    out = call(x)
    g = _rand(*out.shape, seed=1)
    out.backward(g)
    want = _grads(x, w)
    out = call(x)
    with _lib.tuning():
        out.backward(g)
    got = _grads(x, w)
    call(x).backward(g)                                  # and the path is on again behind it
    again = _grads(x, w)
    for a, b, c in zip(want, got, again):
        assert torch.equal(a, b) and torch.equal(a, c)


@pytest.mark.parametrize("grad", [False, True], ids=["no_grad", "grad"])
@pytest.mark.parametrize("i", range(3), ids=["3x3", "5x5", "columns"])
def test_a_trace_records_the_operation(i, grad):
    """torch.jit.trace: the traced module follows a new input instead of returning the output of the traced one."""
    _, call, w, shape = _calls()[i]

    class Net(torch.nn.Module):
        def __init__(self):
            super().__init__()
            self.w = w

        def forward(self, x):
            return call(x)

    net, a, b = Net(), _rand(*shape), _rand(*shape, seed=1)
    with torch.set_grad_enabled(grad):
        traced = torch.jit.trace(net, a, check_trace=False)
        # (a traced 5x5 layer runs as columns, which adds in another order)
        torch.testing.assert_close(traced(b), net(b), rtol=1e-5, atol=1e-4)
        assert float((traced(b) - traced(a)).abs().max()) > 1.0


@pytest.mark.parametrize("i", range(3), ids=["3x3", "5x5", "columns"])
def test_forward_mode_is_refused(i):
    """No derivative is defined for it, so a dual input is an error, whether or not a gradient is wanted as well."""
    import torch.autograd.forward_ad as fw
    _, call, w, shape = _calls()[i]
    for grad, frozen in ((True, False), (True, True), (False, False)):
        w.requires_grad_(not frozen)
        with torch.set_grad_enabled(grad), fw.dual_level():
            x = fw.make_dual(_rand(*shape), torch.ones(shape, device=DEV))
            with pytest.raises(NotImplementedError, match="jvp"):
                call(x)


@pytest.mark.parametrize("change", [lambda t: t.cpu(), lambda t: t.double(), lambda t: t.mT.contiguous().mT, lambda t: t[:-1].contiguous()],
                         ids=["cpu", "double", "strided", "shorter"])
@pytest.mark.parametrize("i", range(3), ids=["3x3", "5x5", "columns"])
def test_backward_looks_at_what_saved_tensor_hooks_return(i, change):
    """Tensors in another form than the kernels take are an error, not an address."""
    _, call, w, shape = _calls()[i]
    x = _rand(*shape).requires_grad_()
    with torch.autograd.graph.saved_tensors_hooks(lambda t: t, change):
        out = call(x)
    with pytest.raises((RuntimeError, TypeError, ValueError)):
        out.backward(_rand(*out.shape))
    with torch.autograd.graph.saved_tensors_hooks(lambda t: t.cpu(), lambda t: t.to(DEV)):
        out = call(x)
    g = _rand(*out.shape)
    out.backward(g)
    got = _grads(x, w)
    call(x).backward(g)
    for a, b in zip(got, _grads(x, w)):
        assert torch.equal(a, b)


@pytest.mark.parametrize("i,names", [(0, ("forward", "backward")), (1, ("ADDER_CONV", "ADDER_BACKWARD")), (2, ("ADDER_CONV", "ADDER_BACKWARD"))],
                         ids=["3x3", "5x5", "columns"])
def test_replaced_operations_are_called(i, names, monkeypatch):
    """Code that wraps the operations of `adder_cuda` sees the calls of layers and of the column op."""
    from addernetcuda_b200 import adder_cuda
    _, call, w, shape = _calls()[i]
    x = _rand(*shape).requires_grad_()
    out = call(x)
    out.backward(_rand(*out.shape, seed=1))
    want, seen = _grads(x, w), []

    def wrapped(name, fn):
        return lambda *a, **kw: (seen.append(name), fn(*a, **kw))[1]
    for name in names:
        monkeypatch.setattr(adder_cuda, name, wrapped(name, getattr(adder_cuda, name)))
    again = call(x)
    again.backward(_rand(*out.shape, seed=1))
    assert seen == list(names)
    torch.testing.assert_close(again, out, rtol=1e-5, atol=1e-4)
    for a, b in zip(_grads(x, w), want):
        torch.testing.assert_close(a, b, rtol=1e-5, atol=1e-4)


def test_a_folded_network_runs_the_modules_that_someone_looks_at():
    """A layer and the folded batch norm behind it are one call only while nothing hangs on the call of either: global hooks, hooks
    on a module, a forward of a subclass or of an instance are seen as without that."""
    from addernetcuda_b200 import adder, inference, resnet
    torch.manual_seed(0)
    net, images = resnet.resnet20().to(DEV), _rand(8, 3, 32, 32)
    for m in net.modules():                              # statistics of these images: outputs on both sides of the ReLU
        if isinstance(m, torch.nn.BatchNorm2d):
            m.momentum = 1.0
    with torch.no_grad():
        net.train()(images)
    inference.fold_batchnorm(net)
    block = net.layer1[0]

    class Doubled(adder.adder2d):
        def forward(self, x):
            return 2.0 * super().forward(x)

    with torch.no_grad():
        want = net(images)
        assert not torch.equal(want, net(_rand(8, 3, 32, 32, seed=1)))
        seen = []
        hook = torch.nn.modules.module.register_module_forward_hook(lambda m, i, o: seen.append(m))
        assert torch.equal(net(images), want)
        hook.remove()
        assert {m for m in net.modules() if isinstance(m, (adder.adder2d, inference.FoldedBatchNorm2d))} <= set(seen)
        for m in (block.conv1, block.bn1):
            hook = m.register_forward_hook(lambda m, i, o: 2.0 * o)
            doubled = net(images)
            assert not torch.equal(doubled, want)
            hook.remove()
            own = m.forward
            m.forward = lambda *a, **kw: 2.0 * own(*a, **kw)
            assert torch.equal(net(images), doubled)
            del m.forward
        block.conv1.__class__ = Doubled
        assert not torch.equal(net(images), want)
        block.conv1.__class__ = adder.adder2d
        assert torch.equal(net(images), want)


def test_wide_strides_go_through_columns():
    """Strides whose input gradient is nearly all zeros: same results, from the path that is faster on them."""
    from addernetcuda_b200 import _native, adder
    for stride, native in ((16, True), (25, False), ((1, 601), False)):
        layer = adder.adder2d(3, 4, 2, stride=stride).to(DEV)
        sh, sw = (stride, stride) if isinstance(stride, int) else stride
        x = _rand(2, 3, 40, 320 if sw < 320 else 620).requires_grad_()
        assert (_native.conv(x, layer.adder, sh, sw, 0, 0, 1, 1) is not None) == native
        out = layer(x)
        g = _rand(*out.shape, seed=1)
        out.backward(g)
        cols = torch.nn.functional.unfold(x.detach().double(), 2, stride=stride).requires_grad_()
        d = layer.adder.detach().double().reshape(4, 12, 1) - cols[:, None]
        torch.testing.assert_close(out.double().reshape(2, 4, -1), -d.abs().sum(2), rtol=1e-5, atol=1e-5)
        gc = (d.clamp(-1, 1) * g.double().reshape(2, 4, 1, -1)).sum(1)
        want = torch.nn.functional.fold(gc.detach(), x.shape[2:], 2, stride=stride)
        torch.testing.assert_close(x.grad.double(), want, rtol=1e-5, atol=1e-5)
