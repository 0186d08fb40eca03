"""Grouped expert products where a group's row count decides the kernel and the operand
layout: up to 16 rows packed (8 and 9 rows: the accumulator halves), up to 32 and 64 rows
stacked two-term tiles, more unstacked; groups of all kinds in one call.  Same bars as
tests/test_gpu_tc.py."""
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():
    pytest.skip("no CUDA device", allow_module_level=True)

from tests import test_gpu_tc as tc            # noqa: E402


@pytest.mark.parametrize("gathered", [False, True])
@pytest.mark.parametrize("counts", [
    [1, 2, 7, 8, 9, 15, 16, 17],
    [31, 32, 33, 47, 48, 63, 64, 65],
    [3, 0, 96, 127, 20, 128, 129, 40],
    [5, 5, 5, 5, 5, 5, 5, 5],
])
def test_row_counts_at_the_dispatch_edges(oracle, counts, gathered):
    tc.test_grouped_expert_products_block_scaled(oracle, counts, gathered)
