"""Which kernel a tcgen05 product takes, by its sizes, and what the library says that it needs (nothing is run)."""
import pytest

from llm_b200 import ops
from llm_b200.ops import tactics


@pytest.mark.parametrize("m,n,k", [(350, 4096, 4096), (1300, 4096, 4096), (160, 4096, 14336), (400, 4096, 14336), (300, 6144, 4096)])
def test_a_product_on_the_row_side_asks_for_nothing(m, n, k):
    """Its pairs meet in shared memory: one kernel, no partial sums, no counters, and neither sums for the next norm nor a rotation
    inside. With the pairs of SMs switched off another kernel runs, and the answers are that kernel's."""
    for target in ops.TARGETS:
        plan = ops.product_plan(m, n, k, target)
        if plan.kernel == "row_side":
            assert (plan.scratch_floats, plan.counters, plan.kernels, plan.emit_parts, plan.tail) == (0, 0, 1, 0, 0)
            assert 64 <= plan.width <= 256 and plan.width % 32 == 0 and 1 <= plan.splits <= 3
    assert ops.product_plan(m, n, k).kernel == "row_side"
    tactics.disable("gemm_tc_pair")
    try:
        assert ops.product_plan(m, n, k).kernel == "blocks"
    finally:
        tactics.enable("gemm_tc_pair")


@pytest.mark.parametrize("m,n,k,target,kernel,tail", [
    (2048, 28672, 4096, "gated", "pairs", True), (3001, 28672, 4096, "gated", "pairs", True), (2500, 4096, 14336, "residual", "pairs", True),
    (2048, 4096, 4096, "residual", "pairs", False), (64, 4096, 4096, "bfloat16", "blocks", False), (8, 28672, 4096, "gated", "blocks", False)])
def test_what_the_other_kernels_need(m, n, k, target, kernel, tail):
    """Tiles cut along K leave two pieces of a tile for every pair and a second kernel adds them; split products leave a tile for
    every split, and what is left for the next norm is a sum for every block of columns."""
    plan = ops.product_plan(m, n, k, target)
    assert plan.kernel == kernel and (plan.tail > 0) == tail
    if kernel == "pairs":
        assert (plan.scratch_floats > 0, plan.kernels) == (tail, 2 if tail else 1) and plan.emit_parts == 0
    elif plan.splits > 1:
        tiles = -(-n // 128) * -(-m // plan.width)
        assert plan.counters == tiles and plan.scratch_floats == tiles * plan.splits * plan.width * 128
        assert plan.emit_parts == (-(-n // 256) if m > 16 else -(-n // 128) if n <= 8192 else 0)


@pytest.mark.parametrize("m,n,k,target,others,row_side", [
    # (microseconds of both ways on a B200, more than a twentieth apart)
    (598, 113152, 128, "bfloat16", 107.1, 149.6), (331, 51760, 272, "bfloat16", 44.5, 54.7), (1365, 16000, 512, "bfloat16", 41.4, 51.1),
    (684, 12568, 792, "bfloat16", 30.2, 36.5), (1341, 99120, 224, "bfloat16", 175.3, 259.3), (399, 5760, 256, "bfloat16", 8.5, 9.3),
    (611, 28544, 256, "residual", 25.2, 31.9), (609, 16384, 320, "residual", 32.3, 37.4), (417, 20736, 496, "residual", 22.9, 26.1),
    (798, 16384, 13992, "residual", 486.3, 520.9), (1054, 12848, 16104, "residual", 537.4, 581.8),
    (1941, 640, 5440, "gated", 33.0, 35.0), (350, 6144, 4096, "bfloat16", 27.0, 19.3), (149, 3328, 256, "bfloat16", 8.1, 5.4),
    (299, 1024, 128, "residual", 10.0, 5.8), (600, 4096, 14336, "residual", 85.9, 64.1), (350, 28672, 4096, "gated", 100.7, 85.8),
    (1150, 4096, 4096, "residual", 45.6, 34.3), (777, 6144, 4096, "bfloat16", 46.1, 33.8)])
def test_the_faster_kernel_is_chosen(m, n, k, target, others, row_side):
    """Products that were timed both ways go to the faster one: with a short K what leaves a tile sets the pace, and the row side's
    tiles leave more slowly."""
    assert (ops.product_plan(m, n, k, target).kernel == "row_side") == (row_side < others)
