"""GPU: the resident table when rows cross the borders of its merge kernels: 32 and 64 new samples per window (register merge,
warp, CTA), 64 and 1,024 kept values, ties and equal values.  After every window against the oracle over all launches so far."""
import numpy as np
import pytest

from kernel_scheduling_b200.pair_table import PairTableBuilder
from oracle import pair_table_oracle as O
from tests.helpers import assert_tables_match
from tests.test_gpu_row_sizes import trace_with_rows

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind", ["spread", "steps", "equal"])
@pytest.mark.parametrize("per_window", [[1, 2, 31, 32, 33], [63, 64, 65, 1, 30], [500, 524, 1, 32, 3], [1024, 1025, 40, 1100, 64], [0, 9000, 9000, 1, 33]])
def test_rows_across_the_borders(kind, per_window):
    parts, shift = [], 0
    for w, m in enumerate(per_window):
        rec = trace_with_rows([max(m, 1), 1, max(m // 2, 1), 7], kind, 10 * w + 1)  # the same four pairs in every window
        rec["start_ns"] += np.uint64(shift)
        rec["end_ns"] += np.uint64(shift)
        shift = int(rec["end_ns"].max()) + 5
        parts.append(rec)
    with PairTableBuilder(device=0) as b:
        b.update_begin()
        for w in range(len(parts)):
            b.update(parts[w])
            assert_tables_match(*b.update_table(), *O.build_pair_table(np.concatenate(parts[: w + 1])))
        b.update_end()
