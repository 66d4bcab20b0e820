"""Which kernel a tcgen05 product takes, by its sizes, and what the library says that it needs (nothing is run)."""
import pytest

from llm_b200 import ops
from llm_b200.ops import tactics


@pytest.mark.parametrize("m,n,k", [(350, 4096, 4096), (1300, 4096, 4096), (160, 4096, 14336), (400, 4096, 14336), (300, 6144, 4096)])
def test_a_product_on_the_row_side_asks_for_nothing(m, n, k):
    """Its pairs meet in shared memory: one kernel, no partial sums, no counters, and neither sums for the next norm nor a rotation
    inside. With the pairs of SMs switched off another kernel runs, and the answers are that kernel's."""
    for glu in (False, True):
        plan = ops.product_plan(m, n, k, glu)
        if plan.kernel == "row_side":
            assert (plan.scratch_floats, plan.counters, plan.kernels, plan.emit_parts, plan.tail) == (0, 0, 1, 0, 0)
            assert 64 <= plan.width <= 256 and plan.width % 32 == 0 and 1 <= plan.splits <= 3
    assert ops.product_plan(m, n, k).kernel == "row_side"
    tactics.disable("gemm_tc_pair")
    try:
        assert ops.product_plan(m, n, k).kernel == "blocks"
    finally:
        tactics.enable("gemm_tc_pair")


@pytest.mark.parametrize("m,n,k,glu,kernel,tail", [(2048, 28672, 4096, True, "pairs", True), (3001, 28672, 4096, True, "pairs", True),
                                                   (2500, 4096, 14336, False, "pairs", True), (2048, 4096, 4096, False, "pairs", False),
                                                   (64, 4096, 4096, False, "blocks", False), (8, 28672, 4096, True, "blocks", False)])
def test_what_the_other_kernels_need(m, n, k, glu, kernel, tail):
    """Tiles cut along K leave two pieces of a tile for every pair and a second kernel adds them; split products leave a tile for
    every split, and what is left for the next norm is a sum for every block of columns."""
    plan = ops.product_plan(m, n, k, glu)
    assert plan.kernel == kernel and (plan.tail > 0) == tail
    if kernel == "pairs":
        assert (plan.scratch_floats > 0, plan.kernels) == (tail, 2 if tail else 1) and plan.emit_parts == 0
    elif plan.splits > 1:
        tiles = -(-n // 128) * -(-m // plan.width)
        assert plan.counters == tiles and plan.scratch_floats == tiles * plan.splits * plan.width * 128
        assert plan.emit_parts == (-(-n // 256) if m > 16 else -(-n // 128) if n <= 8192 else 0)
