"""GPU: rows of more than 8,192 samples in builds of up to 65,536, which one launch finishes: three CTAs per such row, one value lane
each (k_rows_small), against the oracle; and what they cost beside the same row in a larger build."""
import pytest

from kernel_scheduling_b200.pair_table import PairTableBuilder
from oracle import pair_table_oracle as O
from tests.helpers import assert_tables_match
from tests.test_gpu_row_sizes import trace_with_rows

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("sizes", [[8193], [8193] * 7, [12_000, 9001, 1, 600], [16_384, 16_385, 16_383], [20_000, 513, 8192, 8191, 5], [48_200, 3], [65_000], [50_000, 14_000, 700]])
@pytest.mark.parametrize("kind", ["spread", "steps", "equal", "clusters"])
def test_long_rows_against_the_oracle(sizes, kind):
    rec = trace_with_rows(sizes, kind, len(sizes))
    want = O.build_pair_table(rec)
    with PairTableBuilder(device=0) as b:
        for ordered in (True, False, True):  # counts read back, then the same for an order that is not vouched for, then guessed sizes
            assert_tables_match(*b.build(rec, time_ordered=ordered), *want)


@pytest.mark.parametrize("kind", ["spread", "steps", "clusters"])
def test_long_rows_cost_no_more_than_in_a_larger_build(kind):
    """The same work and a few per cent more in kernels that spread a row over the chip; one CTA that searched an unstaged row
    took 5 to 13 times as long."""
    def reduce_ms(n):
        rec = trace_with_rows([n], kind, 1)
        with PairTableBuilder(device=0) as b:
            times = []
            for _ in range(8):
                b.build_device(rec)  # sizes read back: the samples are n and three solo launches
                times.append(b.info["ms_reduce"])
        return min(times)

    assert reduce_ms(62_000) < 2.5 * reduce_ms(66_000)
