"""GPU: dense key ids are ranks of the keys, at the counts where the ranking kernel takes two and four keys per lane (two CTAs of 32
lanes' keys per SM: 9,472 and 18,944 on 148 SMs) and at the largest count."""
import numpy as np
import pytest

from kernel_scheduling_b200.records import pack_records
from oracle import pair_table_oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n_keys", [1, 2, 31, 32, 33, 63, 64, 65, 1023, 9471, 9472, 9473, 9537, 18_943, 18_944, 18_945, 19_071, 37_889, 65_535])
def test_keys_come_out_ranked(builder, n_keys):
    name = np.repeat(np.arange(n_keys), 1 + np.arange(n_keys) % 3)
    np.random.default_rng(n_keys).shuffle(name)
    n = len(name)
    start = 1000 + 10 * np.arange(n)
    rec = pack_records(name, np.full((n, 3), [7, 2, 1]), np.full((n, 3), [128, 1, 1]), np.zeros(n, int), np.zeros(n, int), np.zeros(n, bool), start, start + 5)
    keys, pairs = builder.build(rec, time_ordered=True)
    ukeys, counts = np.unique(O.kernel_keys(rec), return_counts=True)
    assert len(pairs) == 0 and np.array_equal(keys["key"], ukeys) and np.array_equal(keys["launches"], counts)
    first = dict(zip(O.kernel_keys(rec).tolist(), name.tolist()))
    assert all(first[int(k)] == int(i) for k, i in zip(keys["key"], keys["name_id"]))  # the launch fields of its own slot
