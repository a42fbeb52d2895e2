"""GPU: a time-ordered build behind one with so few keys that the sort covers too few bits of its sort keys: rows of a hot pair lie
interleaved with those of another one, run out of their tiles and are taken for one that goes on behind them, more chunks than the
lists hold.  The host throws that table away and builds again; nothing may be touched out of range on the way."""
import numpy as np
import pytest

from kernel_scheduling_b200.pair_table import PairTableBuilder
from kernel_scheduling_b200.records import pack_records
from oracle import c_oracle as CO
from oracle import pair_table_oracle as O
from tests.helpers import assert_tables_match
from tests.test_gpu_row_sizes import trace_with_rows

pytestmark = pytest.mark.gpu
NAMES = 30  # kernels per tenant: 60 keys, sort keys of 12 bits; two keys before: one pass of 9 bits


def launches(name_a, name_b, seed):
    """Launch i of tenant 0 (name_a[i]) overlaps launch i of tenant 1 (name_b[i]); then every kernel once by itself."""
    rng = np.random.default_rng(seed)
    n = len(name_a)
    da, db = rng.integers(1, 900, n), rng.integers(1, 900, n)
    t = 10_000 + 2000 * np.arange(n)
    every = np.tile(np.arange(NAMES), 2)
    te = t[-1] + 5000 + 2000 * np.arange(2 * NAMES)
    name = np.concatenate([name_a, name_b, every])
    start = np.concatenate([t, t, te])
    tenant = np.concatenate([np.zeros(n, int), np.ones(n, int), np.repeat([0, 1], NAMES)])
    dur = np.concatenate([da, db, np.full(2 * NAMES, 10)])
    order, m = np.argsort(start, kind="stable"), len(name)
    return pack_records(name[order], np.ones((m, 3)), np.ones((m, 3)), np.zeros(m, int), tenant[order], np.zeros(m, bool), start[order], (start + dur)[order])


def colliding_pairs():
    """Two pairs of kernels whose sort keys agree in the low nine bits."""
    rec = launches(np.array([0]), np.array([0]), 0)
    keys = O.kernel_keys(rec)
    ukeys = np.unique(keys)
    rank = {(int(r["smem_word"]) >> 24, int(r["name_id"])): int(np.searchsorted(ukeys, k)) for r, k in zip(rec, keys)}
    assert len(ukeys) == 2 * NAMES
    seen = {}
    for i in range(NAMES):
        for j in range(NAMES):
            low = (2 * NAMES + rank[0, i] * 2 * NAMES + rank[1, j]) & 511
            if low in seen and seen[low][0] != i and seen[low][1] != j:
                return seen[low], (i, j)
            seen.setdefault(low, (i, j))


@pytest.mark.parametrize("n, every", [(400_000, 1500), (40_000, 1500), (700_000, 40_000)])
def test_rows_of_an_unsorted_table_stay_in_range(n, every):
    (a0, b0), (a1, b1) = colliding_pairs()
    rng = np.random.default_rng(n)
    rare = rng.random(n) < 1.0 / every
    rec = launches(np.where(rare, a1, a0), np.where(rare, b1, b0), n)
    small = trace_with_rows([n], "spread", 5)
    want = CO.build_pair_table(rec)
    with PairTableBuilder(device=0) as b:
        for _ in range(2):
            b.build(small, time_ordered=True)
            assert_tables_match(*b.build(rec, time_ordered=True), *want)
