"""GPU: launch counts per key and the solo stream of the decode kernel at the borders of its tiles (384 records), of its count
cache (4,096 entries, emptied when the key mix changes) and of its solo queue, against numpy."""
import numpy as np
import pytest

from kernel_scheduling_b200.records import pack_records
from oracle import pair_table_oracle as O

pytestmark = pytest.mark.gpu


def one_tenant_trace(n, n_keys, order, solo, seed):
    """n launches of n_keys kernels, Zipf-distributed, one at a time (no overlaps)."""
    rng = np.random.default_rng(seed)
    p = 1.0 / np.arange(1, n_keys + 1)
    name = rng.choice(n_keys, n, p=p / p.sum())
    if order == "stretches":  # four models one after the other, each with keys of its own
        name = name + n_keys * (4 * np.arange(n) // n)
    dur = rng.integers(1, 5000, n)
    start = 1000 + np.cumsum(dur + 5) - dur
    is_solo = {"none": np.zeros(n, bool), "all": np.ones(n, bool), "some": rng.random(n) < 0.3, "front": np.arange(n) < n // 3}[solo]
    return pack_records(name, np.full((n, 3), [7, 2, 1]), np.full((n, 3), [128, 1, 1]), np.zeros(n, int), np.full(n, 3), is_solo, start, start + dur)


@pytest.mark.parametrize("n", [1, 383, 384, 385, 769, 444 * 384 + 1, 1_300_001])
@pytest.mark.parametrize("n_keys, order, solo", [(1, "mixed", "all"), (300, "mixed", "some"), (3000, "stretches", "front"), (15_000, "stretches", "some"), (9000, "mixed", "none")])
def test_counts_and_solo_times(builder, n, n_keys, order, solo):
    rec = one_tenant_trace(n, n_keys, order, solo, n + n_keys)
    keys, pairs = builder.build(rec, time_ordered=True)
    ukeys, kid, counts = np.unique(O.kernel_keys(rec), return_inverse=True, return_counts=True)
    is_solo = (rec["smem_word"] & (1 << 23)) != 0
    assert len(pairs) == 0 and np.array_equal(keys["key"], ukeys) and np.array_equal(keys["launches"], counts)
    assert np.array_equal(keys["solo_launches"], np.bincount(kid[is_solo], minlength=len(ukeys)))
    assert builder.info["n_solo"] == is_solo.sum()
    dur = (rec["end_ns"] - rec["start_ns"]).astype(np.int64)
    for k in range(0, len(ukeys), max(1, len(ukeys) // 50)):
        mine = dur[(kid == k) & is_solo]
        assert (np.isnan(keys["solo_ns"][k]) and len(mine) == 0) or keys["solo_ns"][k] == np.median(mine), k
