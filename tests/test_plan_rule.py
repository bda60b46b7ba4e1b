"""The segment length and the recommendation that a plan gets when the caller names none, at the lines of the rule, and
the product through such a plan against float64."""
import ctypes

import pytest
import torch

import macko_spmv_b200 as macko_spmv
from macko_spmv_b200 import cabi

DEV = "cuda:0"
GROUPS = 148 * 32 * 4


# 57408 columns are the most that two CTAs of an SM can hold; with one the groups are half as many
@pytest.mark.parametrize("cols,groups", [(8192, GROUPS), (57408, GROUPS), (57409, GROUPS // 2), (100000, GROUPS // 2)])
def test_plan_bytes_follow_the_default_segment(cols, groups):
    lib = cabi.load()
    for share, seg in ((0, 512), (496, 512), (497, 768), (752, 768), (1008, 1024), (1009, 1280), (1088, 1280), (1089, 1536), (9000, 1536)):
        padded = share * groups
        assert lib.macko_spmv_plan_bytes(5000, cols, padded, 0) == lib.macko_spmv_plan_bytes(5000, cols, padded, seg), share


@pytest.mark.gpu
@pytest.mark.parametrize("rows,dense_rows,cols,planned,seg", [
    (3000, 300, 10232, False, 512),    # 162 elements per group, 39.97 sub-steps of a warp over the longest row: no plan
    (3000, 300, 10240, True, 512),     # 40 sub-steps
    (512, 20, 65536, True, 512),       # 138 elements per group (of one CTA per SM), 256 sub-steps
    (900, 200, 30000, True, 512),      # 317, 117 sub-steps
    (900, 240, 30000, True, 512),      # 380
    (8192, 1700, 4000, False, 512),    # 358 elements per group, 31 sub-steps of 16 lanes
    (8192, 1740, 4000, True, 512),     # 367
    (2000, 400, 30000, True, 768),     # 634
    (900, 800, 30000, False, 1536),    # 1267, but no row is far longer than the mean
    (4000, 640, 30000, True, 1280),    # 1014
])
def test_default_plans(rows, dense_rows, cols, planned, seg):
    M = torch.zeros(rows, cols, dtype=torch.float16, device=DEV)
    M[:dense_rows] = torch.randn(dense_rows, cols, device=DEV).half()
    M = M[torch.randperm(rows, device=DEV)].contiguous()
    lib = cabi.load()
    comp = macko_spmv.compress(M)
    frozen = macko_spmv.freeze(comp)
    assert (frozen.plan is not None) == planned and frozen.plan_meta[1] == seg
    x = torch.randn(cols, device=DEV).half()
    ref, l1 = M.double() @ x.double(), M.double().abs() @ x.double().abs()
    lanes, steps = ctypes.c_int(), ctypes.c_int()
    cabi.check(lib, lib.macko_spmv_shape(rows, cols, comp[0].numel(), torch.cuda.get_device_properties(0).multi_processor_count,
                                         ctypes.byref(lanes), ctypes.byref(steps)))
    for fz in (frozen, macko_spmv.freeze(comp, plan=True)):
        # Additions that a product goes through in a row: in one of the four sums of a lane (8 lanes walk a segment), over the
        # sums and the lanes, over the segments. A lost segment of n elements shifts a row by about sqrt(n), at least 40 times this.
        chain = fz.plan_meta[1] // 32 + 5 + -(-cols // fz.plan_meta[1]) + 1 if fz.plan is not None else cols // (4 * lanes.value) + 8
        y = macko_spmv.multiply(fz, x).double()
        # half a unit in the last place of y, and 2^-24 of the absolute sum per fp32 addition
        assert bool(((y - ref).abs() <= 2.0 ** -11 * ref.abs() + chain * 2.0 ** -24 * l1 + 2.0 ** -24).all())


@pytest.mark.gpu
def test_chain_is_that_of_the_launch_that_would_run():
    """Where one CTA per SM holds x the default launch has 1024 threads and a warp per row up to 5209 rows, `macko_spmv_shape` (two
    CTAs of 512 threads) 16 lanes: 8000 elements are 31 sub-steps of a warp, too few for a plan, and would be 62 of 16 lanes."""
    rows, cols = 3000, 60000
    M = torch.zeros(rows, cols, dtype=torch.float16, device=DEV)
    M[:, :800] = torch.randn(rows, 800, device=DEV).half()
    M[70, :8000] = 0.5
    frozen = macko_spmv.freeze(macko_spmv.compress(M))
    assert frozen.plan_meta[2] == 8000 and frozen.plan is None


@pytest.mark.gpu
def test_no_plan_where_x_does_not_fit():
    """120 000 columns: the planned launch would refuse the matrix that `freeze` made."""
    rows, cols = 300, 120_000
    M = torch.zeros(rows, cols, dtype=torch.float16, device=DEV)
    M[::4, ::7] = 0.01
    M[:70] = torch.randn(70, cols, device=DEV).half()
    comp = macko_spmv.compress(M)
    frozen = macko_spmv.freeze(comp)
    assert frozen.plan is None
    x = torch.randn(cols, device=DEV).half()
    assert torch.equal(macko_spmv.multiply(frozen, x), macko_spmv.multiply(comp, x))
