"""Tile planners of the three kernel families, exercised without a GPU.

`adder_b200_describe_plan` runs the same host code that precedes a launch and returns the plan as text: first the
kernel that is launched, then, behind a ";", the form that the layer would take without it ("tiled form", "fp32
form").  For a seeded sample of layer geometries (the benchmark shapes plus random ones) every plan must be
launchable: status 0, at most 256 threads (384 on the tensor cores) in whole warps, shared memory within the 227 KB
a CTA can have, a non-empty grid, and the special-case kernels chosen exactly where they apply.
"""
import random
import re

import pytest

from addernetcuda_b200 import _lib

SMEM_LIMIT = 227 * 1024

BENCH_SHAPES = [  # (n, ci, h, w, co, k, stride, pad)
    (256, 16, 32, 32, 16, 3, 1, 1), (256, 16, 32, 32, 32, 3, 2, 1), (256, 32, 16, 16, 32, 3, 1, 1),
    (256, 64, 8, 8, 64, 3, 1, 1), (256, 256, 14, 14, 256, 3, 1, 1), (256, 512, 7, 7, 512, 3, 1, 1),
    (256, 1024, 14, 14, 256, 1, 1, 0), (256, 16, 32, 32, 32, 1, 2, 0), (256, 32, 16, 16, 64, 1, 2, 0),
    (64, 64, 56, 56, 64, 3, 1, 1), (64, 128, 56, 56, 128, 3, 2, 1), (64, 256, 56, 56, 512, 1, 2, 0),
    (64, 2048, 7, 7, 512, 1, 1, 0), (32, 16, 32, 32, 16, 3, 1, 1), (1, 3, 224, 224, 64, 3, 1, 1),
]


def _random_shapes(count, seed):
    rng = random.Random(seed)
    out = []
    while len(out) < count:
        k = rng.choice((1, 3))
        s = rng.choice((1, 2))
        p = rng.randrange(0, k)
        h, w = rng.randrange(1, 70), rng.randrange(1, 70)
        if h + 2 * p < k or w + 2 * p < k:
            continue
        out.append((rng.randrange(1, 40), rng.randrange(1, 200), h, w, rng.randrange(1, 200), k, s, p))
    return out


def _field(plan, name):
    m = re.search(r"(?<![\w/])%s=(\d+)" % re.escape(name), plan)
    return int(m.group(1)) if m else None


def _launched(op, *shape):
    """The part of the text that describes the launched kernel."""
    return _lib.describe_plan(op, *shape).split(";")[0]


def _fp32_form(*shape):
    """The weight gradient's fp32 kernel, whether or not the tensor cores take the layer."""
    return _lib.describe_plan(2, *shape).split("; fp32 form: ")[-1]


@pytest.mark.parametrize("op", [0, 1, 2], ids=["forward", "grad_x", "grad_w"])
def test_plans_are_launchable(op):
    for shape in BENCH_SHAPES + _random_shapes(150, 20 + op):
        for flags in ((0, 1) if op == 1 else (0,)):
            for plan in _lib.describe_plan(op, *shape, flags).split(";"):
                assert _field(plan, "status") == 0, (shape, plan)
                threads = _field(plan, "threads")
                assert threads is not None and 32 <= threads <= (384 if "mma" in plan else 256) and threads % 32 == 0, (shape, plan)
                smem = _field(plan, "smem")
                if smem is not None:          # the one-thread-per-position kernels use static shared memory
                    assert smem <= SMEM_LIMIT, (shape, plan)
                grid = re.search(r"grid=\((\d+),(\d+)\)", plan)
                if grid:
                    assert int(grid.group(1)) >= 1 and 1 <= int(grid.group(2)) <= 65535, (shape, plan)
                splits = _field(plan, "splits")
                if splits is not None:
                    assert splits >= 1, (shape, plan)


def test_a_plan_that_cannot_be_launched_says_so():
    """More blocks of channels than a grid has rows, on the gathering kernels of 1x1 layers."""
    for op, shape in ((0, (1, 1, 1, 1, 4_500_000, 1, 1, 0)), (1, (1, 4_500_000, 1, 1, 1, 1, 1, 0))):
        plan = _launched(op, *shape)
        assert "gather" in plan and _field(plan, "status") == 3, plan
    assert ";" not in _lib.describe_plan(0, 64, 256, 56, 56, 512, 1, 2, 0)      # the tiled forward has no 1x1 form


def test_special_case_kernels_are_chosen_where_they_apply():
    # 1x1 stride-2, few channels: one thread per output position, all three passes
    for op in (0, 1):
        assert "pointwise" in _launched(op, 256, 16, 32, 32, 32, 1, 2, 0, 1)
        assert "gather k=1x1" in _launched(op, 64, 256, 56, 56, 512, 1, 2, 0, 1)     # too many channels
        assert "gather k=1x1" in _launched(op, 256, 16, 32, 32, 32, 1, 1, 0, 1)      # stride 1
    assert _field(_launched(2, 256, 16, 32, 32, 32, 1, 2, 0), "pointwise") == 1
    # 1x1 with many channels: the tensor cores; below the pixels that pay for them the GEMM-style fp32 kernel
    for shape in ((256, 1024, 14, 14, 256, 1, 1, 0), (64, 256, 56, 56, 512, 1, 2, 0)):
        assert _launched(2, *shape).startswith("gw mma"), _launched(2, *shape)
        assert _field(_fp32_form(*shape), "gemm1x1") == 1 and _field(_fp32_form(*shape), "pointwise") == 0
    assert _field(_launched(2, 1, 1024, 14, 14, 256, 1, 1, 0), "gemm1x1") == 1
    assert _field(_launched(2, 256, 16, 32, 32, 16, 3, 1, 1), "gemm1x1") == 0
    # 3x3 stride-2 input gradient: two segments per thread with 4-pixel segments and whole row pairs (also a ragged last one);
    # the gathering kernel from 64 channels on
    assert _field(_launched(1, 256, 16, 32, 32, 32, 3, 2, 1, 1), "segs/thread") == 2
    assert _field(_launched(1, 256, 16, 32, 32, 16, 3, 1, 1, 1), "segs/thread") == 1
    assert _field(_launched(1, 64, 60, 28, 28, 60, 3, 2, 1, 1), "segs/thread") == 2
    assert "gather k=3x3" in _launched(1, 64, 256, 28, 28, 256, 3, 2, 1, 1)


def test_chunking_does_not_depend_on_the_batch():
    """Sub-batches must be computed by the same kernel, and in the tiled input gradient, whose two-level summation folds one
    partial sum per chunk, with the same chunk boundaries (bitwise-equal results per image).  The gathering kernels fold after a
    fixed number of terms, and the forward keeps one running sum per output over all input channels, so their bits do not
    depend on the tile, which follows the size of the launch."""
    for ci, h, w, co, k, s in ((64, 8, 8, 64, 3, 1), (32, 16, 16, 32, 3, 1), (32, 16, 16, 60, 3, 2), (256, 14, 14, 256, 3, 1),
                               (64, 15, 15, 64, 3, 1), (128, 28, 28, 128, 3, 2), (256, 14, 14, 64, 1, 1), (64, 28, 28, 128, 1, 2)):
        for flags in (0, 1):
            plans = [_launched(1, n, ci, h, w, co, k, s, k // 2, flags) for n in (1, 2, 3, 8, 64, 256)]
            gathers = {"gather" in p for p in plans}
            assert len(gathers) == 1, plans
            if not gathers.pop():
                chunks = {_field(p, "CKO") for p in plans}
                assert len(chunks) == 1 and None not in chunks, plans


def test_unsupported_geometry_is_reported_not_planned():
    lib = _lib.load()
    import ctypes
    buf = ctypes.create_string_buffer(256)
    assert lib.adder_b200_describe_plan(0, 4, 8, 16, 16, 8, 5, 1, 2, 0, buf, 256) != 0       # 5x5 kernel
    assert lib.adder_b200_describe_plan(0, 4, 8, 16, 16, 8, 3, 3, 1, 0, buf, 256) != 0       # stride 3
    assert lib.adder_b200_describe_plan(0, 4, 0, 16, 16, 8, 3, 1, 1, 0, buf, 256) != 0       # no channels


def test_empty_batch_plans_have_at_least_one_split():
    """An empty batch still defines the weight gradient (all zeros): the plan must keep one CTA per output
    tile to write the zero slices, also on the geometry that otherwise takes the pointwise kernels."""
    for shape in ((0, 16, 32, 32, 32, 1, 2, 0), (0, 16, 32, 32, 16, 3, 1, 1), (0, 1024, 14, 14, 256, 1, 1, 0)):
        plan = _launched(2, *shape)
        assert _field(plan, "status") == 0 and _field(plan, "pointwise") == 0, plan
        assert _field(plan, "splits") >= 1, plan


def test_imagenet_plane_rules():
    """Planner rules for the ResNet-50 shapes (resnet50.py:84-90 and the 7/14/28-wide stages): which kernel
    family and which segment width a geometry gets.  Host-side only: the plans are computed without a GPU."""
    # wide 3x3 weight gradients run on the tensor cores; their fp32 form on 28-, 14- and 7-wide planes is the warp-tile kernel
    # with 4- or 7-pixel segments, on 56-wide planes its bulk-copy form
    for hw, rw in ((28, 4), (14, 7), (7, 7)):
        shape = (64, 128, hw, hw, 128, 3, 1, 1)
        assert _launched(2, *shape).startswith("gw mma"), _launched(2, *shape)
        fp32 = _fp32_form(*shape)
        assert "warp-tile" in fp32 and "tma" not in fp32 and _field(fp32, "RW") == rw, fp32
    assert "warp-tile tma" in _fp32_form(64, 64, 56, 56, 64, 3, 1, 1)
    # ... which small planes with few channels launch
    assert _launched(2, 256, 64, 8, 8, 64, 3, 1, 1).startswith("gw warp-tile tma")
    # 1x1 layers: the gathering kernels, at stride 2 on the class of sampled pixels alone
    for op in (0, 1):
        for shape in ((64, 256, 56, 56, 512, 1, 2, 0), (64, 256, 56, 56, 64, 1, 1, 0), (64, 1024, 14, 14, 256, 1, 1, 0)):
            assert "gather k=1x1" in _launched(op, *shape, 1)
    assert _field(_launched(1, 64, 256, 56, 56, 512, 1, 2, 0, 1), "classes") == 1
    # 3x3 stride-2 input gradients: four classes of pixels in the gathering kernel, two complementary segments per thread
    # in the tiled one
    for hw in (32, 56, 28, 14):
        assert _field(_launched(1, 64, 128, hw, hw, 128, 3, 2, 1, 1), "classes") == 4
        assert _field(_launched(1, 64, 32, hw, hw, 32, 3, 2, 1, 1), "segs/thread") == 2


def test_waits_for_the_copy_engine_outlast_a_time_slice():
    """A kernel whose wait runs out leaves its result unwritten and a flag on the device, which a caller need not read: the bound
    is for a copy that never lands, not for a GPU that another process has for a second (2^18 polls)."""
    from addernetcuda_b200 import build
    text = (build.CSRC / "tma.cuh").read_text()
    assert int(re.search(r"MBAR_WAIT_LIMIT = 1 << (\d+);", text).group(1)) >= 22


def test_forward_kernel_by_predicted_time():
    """Stride-1 3x3 forwards: the tiled kernel where it is the faster one - few input channels, or output channels that fill a
    fraction of the gathering kernel's tiles - and the gathering kernel for wide layers, ragged planes and small launches."""
    for shape in ((147, 16, 60, 60, 40), (241, 416, 10, 24, 33), (231, 112, 15, 57, 19), (31, 425, 62, 62, 5), (256, 16, 32, 32, 16),
                  (256, 64, 8, 8, 64)):
        assert "gather" not in _launched(0, *shape, 3, 1, 1), shape
    for shape in ((64, 64, 56, 56, 64), (256, 256, 14, 14, 256), (50, 27, 29, 31, 45), (1, 16, 32, 32, 16), (1, 512, 7, 7, 512)):
        assert "gather" in _launched(0, *shape, 3, 1, 1), shape
    # the 2x8 tile of 8 channels only where nothing better fits (it cost half of what it takes)
    for shape in ((256, 32, 16, 16, 21), (80, 64, 30, 30, 24), (72, 24, 38, 38, 24)):
        plan = _launched(0, *shape, 3, 1, 1)
        assert not (_field(plan, "RM") == 2 and _field(plan, "RP") == 8), plan


def test_weight_gradient_kernel_by_size():
    """Tensor cores: more than 8 output channels, and on small planes with few channels more work than elsewhere."""
    for shape in ((40, 304, 32, 32, 7), (244, 112, 29, 29, 6), (64, 64, 16, 16, 64), (256, 64, 8, 8, 64)):
        assert not _launched(2, *shape, 3, 1, 1).startswith("gw mma"), shape
    for shape in ((40, 304, 32, 32, 9), (115, 8, 32, 32, 282), (128, 64, 16, 16, 64), (400, 64, 8, 8, 64), (64, 64, 36, 36, 64)):
        assert _launched(2, *shape, 3, 1, 1).startswith("gw mma"), shape


def test_statistics_pass_has_a_row_of_blocks_per_channel():
    """Beyond the rows of a grid there are no fused statistics (the batch norm reads the output itself), not a launch that fails."""
    lib = _lib.load()
    for co, some in ((65535, True), (65536, False)):
        assert (lib.adder_b200_forward_stat_slices(8, 4, 3, 3, co, 1, 1, 0) > 0) == some
        assert (lib.adder_b200_forward_stat_slices(8, 128, 3, 3, co, 3, 1, 1) > 0) == some


def test_copy_by_taps_where_it_pays():
    """The input gradient's copy of w by taps costs by the weight and saves by the term: scratch is asked for where outputs enough share
    a weight, and where a tile that gains by it is launched (of at least 32 input channels, mostly)."""
    lib = _lib.load()

    def scratch(n, ci, h, w, co, k, s):
        return lib.adder_b200_conv_backward_input_workspace_bytes(n, ci, h, w, co, k, k, s, s, k // 2, k // 2, 1, 1)

    # few outputs a weight (the copy took 5 to 30 % more than it saved), tiles of 8 and 16 channels (7 % slower with it), small layers
    for shape in ((2, 2048, 7, 7, 2048, 3, 1), (1, 4096, 5, 5, 4096, 3, 1), (7, 1024, 7, 7, 1024, 3, 1), (9, 72, 56, 56, 176, 3, 1),
                  (152, 48, 59, 11, 80, 3, 1), (47, 176, 8, 8, 176, 3, 1), (256, 1024, 14, 14, 256, 1, 1)):
        assert scratch(*shape) == 0, shape
    for shape in ((256, 256, 14, 14, 256, 3, 1), (64, 128, 56, 56, 128, 3, 2), (64, 512, 14, 14, 512, 3, 2), (4, 1024, 14, 14, 1024, 3, 1),
                  (16, 256, 14, 14, 256, 5, 1), (1, 512, 16, 16, 512, 7, 1)):
        assert scratch(*shape) == 4 * shape[1] * shape[4] * shape[5] ** 2, shape


def test_register_budget_of_the_exact_input_gradient():
    """Tiled 3x3 stride-1 layers: the budget of three CTAs an SM where more than 8 warps share one (with that of two, two CTAs of 5 warps
    were 11 % slower than before the packed loop), that of two below; the saturating form by what fits."""
    for shape, exact, fast in (((355, 144, 6, 12, 48), 3, 2), ((173, 144, 12, 24, 48), 3, 2), ((256, 64, 8, 8, 64), 3, 2),
                               ((128, 64, 8, 8, 64), 2, 2), ((3, 3, 4, 4, 208), 2, 2), ((256, 16, 32, 32, 16), 3, 3), ((1, 16, 32, 32, 16), 2, 3),
                               ((256, 32, 14, 14, 32), 2, 2)):
        assert _field(_launched(1, *shape, 3, 1, 1, 0), "MB") == exact, shape
        assert _field(_launched(1, *shape, 3, 1, 1, 1), "MB") == fast, shape


def test_forward_plan_by_alignment():
    """Tiles that profit from weights in 16-byte copies are planned as cheaper only where the operands allow those: without
    alignment the layers below ran 5 to 8 % slower on them than on the tile (the last one: kernel) that is planned otherwise."""
    def tile(*shape):
        plan = _launched(0, *shape)
        return "gather" in plan and tuple(_field(plan, k) for k in ("RM", "RP", "TC", "TP"))

    unaligned = _lib.FLAG_UNALIGNED
    for shape in ((19, 944, 22, 22, 144, 1, 1, 0), (100, 64, 30, 30, 64, 3, 1, 1), (106, 16, 9, 9, 129, 3, 1, 1)):
        assert "_rows" in _launched(0, *shape) and "_rows" not in _launched(0, *shape, unaligned)
        assert tile(*shape) == (4, 8, 64, 64), shape
        assert tile(*shape, unaligned) not in (False, (4, 8, 64, 64)), shape
    assert tile(73, 4, 8, 12, 96, 3, 1, 1) and not tile(73, 4, 8, 12, 96, 3, 1, 1, unaligned)
    # no rows of whole quads: the plan is the same
    for shape in ((50, 27, 29, 31, 45, 3, 1, 1), (64, 250, 14, 14, 64, 1, 1, 0), (256, 16, 32, 32, 16, 3, 1, 1)):
        assert tile(*shape) == tile(*shape, unaligned), shape
        assert "_rows" not in _launched(0, *shape) + _launched(0, *shape, unaligned)
