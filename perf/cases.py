"""The work that users of this framework have it do, as cases that can be timed and compared.

Four kinds, each through the public entry points:

  layer   one `adder2d` module, forward and backward through autograd (the unit every network is built of);
  column  the column-matrix op `adder.apply(W_col, X_col)`, forward and backward (code written against the
          reference's own extension);
  infer   a ResNet-20 / ResNet-50 with folded batch norm, evaluation mode, no gradients (`inference.py`);
  train   one SGD training step of ResNet-20 (`train.TrainStep`, CUDA graph).

Inputs follow the benchmark definitions of the repository: x ~ N(0,1), Kaiming-normal weights,
grad_out ~ N(0,1), synthetic images ~ N(0,1) with uniform random labels; all tensors fp32.
"""
import math

import torch

from addernetcuda_b200 import adder, inference, resnet, strict_fp32, train

DEV = "cuda:0"
_CAP_OPS = 2.7e11        # drawn layers: operations of forward + backward, about the largest listed layer
_CAP_ELEMENTS = 1 << 28  # drawn layers: values of any one tensor (the im2col matrix included)


def listed():
    def layer(name, n, ci, co, h, w, k, stride, pad, fast):
        return dict(name=name, kind="layer", n=n, ci=ci, co=co, h=h, w=w, k=k, stride=stride, pad=pad, fast=fast)

    return [
        # the shape of the reference's extension test: small column matrices, where launches and host time count
        dict(name="column_k288_p1024", kind="column", K=288, P=1024, Co=32),
        # one image at a time through a trained CIFAR network: the smallest end of evaluation
        dict(name="infer_resnet20_n1", kind="infer", depth=20, n=1),
        # a single CIFAR layer at a small batch, the first benchmark configuration
        layer("layer_n32_c16_32x32", 32, 16, 16, 32, 32, 3, 1, 1, False),
        # stage transition of the CIFAR network at the training batch, saturating clamp as bench.py trains
        layer("layer_n256_c16to32_32x32_s2", 256, 16, 32, 32, 32, 3, 2, 1, True),
        # last stage of the CIFAR network: many channels on small planes, the module's default clamp
        layer("layer_n256_c64_8x8", 256, 64, 64, 8, 8, 3, 1, 1, False),
        # a user's own network: no size is a multiple of a tile
        layer("layer_n50_c27to45_29x31", 50, 27, 45, 29, 31, 3, 1, 1, False),
        # a geometry beyond 1x1 and 3x3 kernels
        layer("layer_n32_c16to32_32x32_k5", 32, 16, 32, 32, 32, 5, 1, 2, False),
        # ImageNet bottleneck layers: the strided shortcut, the channel reduction and the 3x3 in the middle
        layer("layer_n64_c256to512_56x56_k1s2", 64, 256, 512, 56, 56, 1, 2, 0, True),
        layer("layer_n256_c1024to256_14x14_k1", 256, 1024, 256, 14, 14, 1, 1, 0, False),
        layer("layer_n256_c256_14x14", 256, 256, 256, 14, 14, 3, 1, 1, True),
        # the headline: a training step of the CIFAR network at batch 256
        dict(name="train_resnet20_n256", kind="train", n=256, fast=True),
        # evaluation of the ImageNet network, the largest work listed
        dict(name="infer_resnet50_n64", kind="infer", depth=50, n=64),
    ]


# ------------------------------------------------------------------------------------------ drawn cases

def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _channels(rng, lo, hi):
    """Mostly multiples of 8 or 16 as in published networks, one in four as it falls."""
    c = _log_int(rng, lo, hi)
    m = rng.choice((1, 8, 16, 16))
    return max(lo, (c + m - 1) // m * m)


def _draw_layer(rng):
    while True:
        k = rng.choice((3, 3, 3, 3, 3, 3, 1, 1, 1, rng.choice((2, 5, 7))))
        stride = rng.choice((1, 1, 1, 2)) if k in (1, 3) else rng.choice((1, 2, 3))
        top = 1024 if k == 1 else 512 if k == 3 else 64
        ci, co = _channels(rng, 3, top), _channels(rng, 4, top)
        h = _log_int(rng, 6, 64)
        w = h if rng.random() < 0.7 else _log_int(rng, 6, 64)
        n = _log_int(rng, 1, 256)
        case = dict(kind="layer", n=n, ci=ci, co=co, h=h, w=w, k=k, stride=stride, pad=k // 2, fast=rng.random() < 0.5)
        ho, wo = _out_hw(case)
        unfolded = ci * k * k if k not in (1, 3) else 0
        if 9 * _layer_triples(case) <= _CAP_OPS and n * max(ci * h * w, co * ho * wo, unfolded * ho * wo) <= _CAP_ELEMENTS:
            return case


def _draw_column(rng):
    while True:
        K, P, Co = _log_int(rng, 9, 4608), _log_int(rng, 64, 1 << 18), _log_int(rng, 4, 512)
        if 9 * K * P * Co <= _CAP_OPS and K * P <= _CAP_ELEMENTS:
            return dict(kind="column", K=K, P=P, Co=Co)


def draw(rng):
    """One more case of the listed kinds: layers most often, over the sizes of small and large networks."""
    r = rng.random()
    if r < 0.6:
        return _draw_layer(rng)
    if r < 0.7:
        return _draw_column(rng)
    if r < 0.8:
        return dict(kind="infer", depth=20, n=_log_int(rng, 1, 1024))
    if r < 0.88:
        return dict(kind="infer", depth=50, n=_log_int(rng, 1, 60))
    return dict(kind="train", n=_log_int(rng, 16, 400), fast=rng.random() < 0.7)


# ------------------------------------------------------------------------------------------ inputs

def _generator(seed):
    return torch.Generator(device=DEV).manual_seed(int(seed))


def _out_hw(case):
    return tuple((case[d] + 2 * case["pad"] - case["k"]) // case["stride"] + 1 for d in ("h", "w"))


def _network(depth, gen):
    strict_fp32()      # stem and classifier in fp32 too, as the benchmark definitions have it
    with torch.device(DEV):
        net = resnet.resnet20() if depth == 20 else resnet.resnet50()
    with torch.no_grad():
        for name, p in net.named_parameters():
            if p.dim() == 4:      # convolution and adder weights: Kaiming-normal; batch norm keeps weight 1, bias 0
                p.normal_(0.0, math.sqrt(2.0 / (p.shape[1] * p.shape[2] * p.shape[3])), generator=gen)
            elif name == "fc.bias":
                p.zero_()
    return net


def _images(depth, n, gen):
    side = 32 if depth == 20 else 224
    return torch.randn((n, 3, side, side), device=DEV, generator=gen)


def _prepare_layer(case, gen):
    n, ci, co, k = case["n"], case["ci"], case["co"], case["k"]
    layer = adder.adder2d(ci, co, k, stride=case["stride"], padding=case["pad"]).to(DEV)
    with torch.no_grad():
        layer.adder.normal_(0.0, math.sqrt(2.0 / (ci * k * k)), generator=gen)
    x = torch.randn((n, ci, case["h"], case["w"]), device=DEV, generator=gen).requires_grad_()
    g = torch.randn((n, co, *_out_hw(case)), device=DEV, generator=gen)
    return dict(kind="layer", layer=layer, x=x, g=g, fast=case["fast"])


def _prepare_column(case, gen):
    K, P, Co = case["K"], case["P"], case["Co"]
    w = (torch.randn((Co, K), device=DEV, generator=gen) * math.sqrt(2.0 / K)).requires_grad_()
    x = torch.randn((K, P), device=DEV, generator=gen).requires_grad_()
    return dict(kind="column", w=w, x=x, g=torch.randn((Co, P), device=DEV, generator=gen))


def _prepare_infer(case, gen):
    # Running statistics as training leaves them: each batch norm takes those of one batch that it normalises.
    net = _network(case["depth"], gen).train()
    norms = [m for m in net.modules() if isinstance(m, torch.nn.BatchNorm2d)]
    for m in norms:
        m.momentum = 1.0
    with torch.no_grad():
        net(_images(case["depth"], 16, gen))
    for m in norms:
        m.momentum = 0.1
    return dict(kind="infer", net=inference.fold_batchnorm(net), images=_images(case["depth"], case["n"], gen))


def _prepare_train(case, gen):
    adder.FAST_CLAMP = case["fast"]
    net = _network(20, gen).train()
    first = {k: v.clone() for k, v in net.state_dict().items()}
    images = _images(20, case["n"], gen)
    labels = torch.randint(0, 10, (case["n"],), device=DEV, generator=gen)
    step = train.TrainStep(net, images.shape, 10, lr=0.1, momentum=0.9, device=DEV)
    step.load_batch(images, labels)
    step.warmup()
    step.capture()
    # warm-up made real steps: training starts from the first weights, with no momentum
    net.load_state_dict(first)
    for s in step.opt.state.values():
        s["momentum_buffer"].zero_()
    weights = [p for p in net.parameters() if p.dim() == 4]
    vectors = [p for p in net.parameters() if p.dim() == 1]
    return dict(kind="train", step=step, images=images, labels=labels, weights=weights, vectors=vectors)


_PREPARE = {"layer": _prepare_layer, "column": _prepare_column, "infer": _prepare_infer, "train": _prepare_train}


def prepare(case, seed):
    return _PREPARE[case["kind"]](case, _generator(seed))


# ------------------------------------------------------------------------------------------ one pass

def run(state):
    kind = state["kind"]
    if kind == "layer":
        layer, x = state["layer"], state["x"]
        adder.FAST_CLAMP = state["fast"]
        x.grad = layer.adder.grad = None
        out = layer(x)
        out.backward(state["g"])
        return {"out": out, "grad_x": x.grad, "grad_w": layer.adder.grad}
    if kind == "column":
        w, x = state["w"], state["x"]
        w.grad = x.grad = None
        out = adder.adder.apply(w, x)
        out.backward(state["g"])
        return {"out": out, "grad_x": x.grad, "grad_w": w.grad}
    if kind == "infer":
        with torch.no_grad():
            return state["net"](state["images"])
    step = state["step"]
    loss = step.step(state["images"], state["labels"])
    return {"loss": loss, "logits": step.logits, "weights": state["weights"],
            "batch_norm": torch.cat([p.detach() for p in state["vectors"]])}


# ------------------------------------------------------------------------------------------ work and tolerance

def _layer_triples(case):
    ho, wo = _out_hw(case)
    return case["n"] * ho * wo * case["co"] * case["ci"] * case["k"] ** 2


def _network_work(depth, n):
    """(|x-w| terms of the adder layers, multiply-adds of stem and classifier, parameters) of one forward."""
    triples = params = 0

    def conv(ci, co, k, side):
        nonlocal triples, params
        triples += n * side * side * ci * co * k * k
        params += ci * co * k * k

    if depth == 20:
        cin, side = 16, 32
        for width, stride in ((16, 1), (32, 2), (64, 2)):
            for block in range(3):
                s = stride if block == 0 else 1
                side //= s
                if s != 1:
                    conv(cin, width, 1, side)
                conv(cin, width, 3, side)
                conv(width, width, 3, side)
                cin = width
        return triples, n * (32 * 32 * 3 * 16 * 9 + 640), params + 3 * 16 * 9 + 640
    cin, side = 64, 56
    for width, blocks, stride in ((64, 3, 1), (128, 4, 2), (256, 6, 2), (512, 3, 2)):
        for block in range(blocks):
            s = stride if block == 0 else 1
            conv(cin, width, 1, side)
            side //= s
            if block == 0:
                conv(cin, width * 4, 1, side)
            conv(width, width, 3, side)
            conv(width, width * 4, 1, side)
            cin = width * 4
    return triples, n * (112 * 112 * 3 * 64 * 49 + 2048000), params + 3 * 64 * 49 + 2048000


def work(case):
    """Operations by the benchmark's rule: 3 per |x - w| term forward, 6 backward; 2 per multiply-add."""
    kind = case["kind"]
    if kind == "layer":
        ho, wo = _out_hw(case)
        x = case["n"] * case["ci"] * case["h"] * case["w"]
        out = case["n"] * case["co"] * ho * wo
        w = case["co"] * case["ci"] * case["k"] ** 2
        return {"bytes": 4 * 2 * (x + out + w), "flops": 9 * _layer_triples(case)}
    if kind == "column":
        K, P, Co = case["K"], case["P"], case["Co"]
        return {"bytes": 4 * 2 * (K * P + Co * P + Co * K), "flops": 9 * K * P * Co}
    n = case["n"]
    depth = case["depth"] if kind == "infer" else 20
    triples, macs, params = _network_work(depth, n)
    pixels = n * 3 * (32 * 32 if depth == 20 else 224 * 224)
    if kind == "infer":
        return {"bytes": 4 * (pixels + params + n * (10 if depth == 20 else 1000)), "flops": 3 * triples + 2 * macs}
    # weights and momentum read and written
    return {"bytes": 4 * (pixels + 4 * params + n * 10) + 8 * n, "flops": 9 * triples + 6 * macs}


def tolerance(case):
    if case["kind"] in ("layer", "column"):
        return {"rel": 1e-5}       # 32-bit sums in any order
    if case["kind"] == "infer":
        return {"rel": 1e-4}       # the same through 20 or 52 layers, each followed by a normalisation
    return {"rel": 1e-3}           # a ReLU gate near zero that opens or closes moves whole terms of a gradient
