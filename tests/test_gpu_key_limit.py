"""GPU: traces at and beyond the 65,535 distinct kernel keys a table can hold, behind successful builds.  The stages of such a call
are queued before the host has seen the key count: the status must come back and the handle must stay usable."""
import pytest

from kernel_scheduling_b200 import _lib
from kernel_scheduling_b200.pair_table import PairTableBuilder
from oracle import pair_table_oracle as O
from tests.helpers import assert_tables_match
from tests.test_gpu_row_sizes import trace_with_rows

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("pairs", [32_768, 35_000, 60_000])
@pytest.mark.parametrize("before", [300, 32_767])
def test_too_many_keys_behind_a_smaller_build(before, pairs):
    """Every pair has two keys of its own.  With 600 keys before, the guessed sizes do not hold; with 65,534 they do."""
    good, bad = trace_with_rows([1] * before, "spread", before), trace_with_rows([1] * pairs, "spread", pairs)
    want = O.build_pair_table(good)
    with PairTableBuilder(device=0) as b:
        for _ in range(2):
            assert_tables_match(*b.build(good, time_ordered=True), *want)
            with pytest.raises(_lib.KsError) as e:
                b.build(bad, time_ordered=True)
            assert e.value.status == _lib.ERR_TOO_MANY_KEYS
        for _ in range(2):
            assert_tables_match(*b.build(good, time_ordered=True), *want)
