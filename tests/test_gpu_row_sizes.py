"""GPU: the statistics of table rows and segments at the borders of their size classes (the kernels of ks_tilestats.cuh and
ks_segstats.cuh), against the oracle and numpy's partition.  Everything is an integer or one IEEE division of one: bit for bit,
sums and means within the table contract of 1e-6 (tests/helpers.py)."""
import numpy as np
import pytest

from kernel_scheduling_b200.records import pack_records
from oracle import pair_table_oracle as O
from tests.helpers import assert_tables_match, sample_places

pytestmark = pytest.mark.gpu

BORDERS = [1, 2, 3, 4, 5, 8, 9, 16, 17, 31, 32, 33, 64, 65, 128, 129, 256, 257, 511, 512, 513, 514, 2047, 2048, 2049, 2560, 8191, 8192, 8193, 50_001]


def durations(kind, n, rng):
    if kind == "spread":
        return rng.integers(1, 60_000, n)
    if kind == "steps":  # a coarse clock: few distinct values
        return 500 * rng.integers(1, 12, n)
    if kind == "equal":
        return np.full(n, 777)
    return np.where(rng.random(n) < 0.5, 1000 + rng.integers(0, 50, n), 900_000 + rng.integers(0, 50, n))  # two far-off clusters


def trace_with_rows(counts, kind, seed):
    """Pair p of keys (0, p) and (1, p) meets counts[p] times; every third key of tenant 0 has solo launches."""
    rng = np.random.default_rng(seed)
    pair = np.repeat(np.arange(len(counts)), counts)
    rng.shuffle(pair)
    n = len(pair)
    da, db = durations(kind, n, rng), durations(kind, n, rng)
    t = 10_000 + np.cumsum(da + db + 10) - (da + db + 10)
    solo = np.repeat(np.arange(0, len(counts), 3), 3)
    ts = t[-1] + 2_000_000 + 70_000 * np.arange(len(solo))
    name = np.concatenate([pair, pair, solo])
    start = np.concatenate([t, t + np.minimum(da - 1, 1), ts])
    tenant = np.concatenate([np.zeros(n, int), np.ones(n, int), np.zeros(len(solo), int)])
    dur = np.concatenate([da, db, rng.integers(1, 60_000, len(solo))])
    is_solo = np.arange(len(name)) >= 2 * n
    order = np.argsort(start, kind="stable")
    m = len(name)
    return pack_records(name[order], np.ones((m, 3)), np.ones((m, 3)), np.zeros(m, int), tenant[order], is_solo[order], start[order], (start + dur)[order])


@pytest.mark.parametrize("kind", ["spread", "steps", "equal", "clusters"])
def test_rows_at_the_borders_of_the_size_classes(builder, kind):
    rec = trace_with_rows(BORDERS, kind, 7)
    want = O.build_pair_table(rec)
    assert sorted(want[1]["count"].tolist()) == BORDERS
    for _ in range(2):  # counts read back, then queued with the counts of the call before
        assert_tables_match(*builder.build(rec, time_ordered=True), *want)


def test_rows_that_end_with_a_tile(builder):
    """Rows of one tile of samples (2,048), the window behind it (512) and one more or less, many times over."""
    for sizes in ([2048] * 5, [2560] * 3 + [1], [512] * 9, [511, 1] * 6, [2047, 1, 2049, 3, 513] * 2, [1] * 5000):
        rec = trace_with_rows(sizes, "spread", len(sizes))
        assert_tables_match(*builder.build(rec, time_ordered=True), *O.build_pair_table(rec))


@pytest.mark.parametrize("sizes", [[8191, 8192, 8193, 20_001, 2, 513], [60_000], [30_000, 30_001], [64_000, 1500], [65_530], [600] * 105])
def test_long_rows_of_small_builds(builder, sizes):
    """Up to 65,536 samples one launch finishes the rows of every length; the last cases lie on both sides of that."""
    rec = trace_with_rows(sizes, "spread", sum(sizes))
    want = O.build_pair_table(rec)
    for _ in range(2):
        assert_tables_match(*builder.build(rec, time_ordered=True), *want)


def middle(v):
    lo, hi = (len(v) - 1) // 2, len(v) // 2
    p = np.partition(v, [lo, hi])
    return [len(v), int(v.astype(np.uint64).sum()), int(v.min()), int(v.max()), int(p[lo]), int(p[hi])]


@pytest.mark.parametrize("n", [8193, 20_000, 60_001, 400_002])
@pytest.mark.parametrize("kind", ["random", "misled_low", "misled_high", "misled_wide", "two_values", "top"])
def test_long_segments_whose_sample_misleads(builder, n, kind):
    """The pivots of a long segment come from 1,024 (8,192) of its values; here those values, and as many evenly spaced ones, say
    little about the others: the middle lies below or above the pivots, or everything lies between them."""
    rng = np.random.default_rng(n)
    v = rng.integers(1000, 2**32 - 1000, n, dtype=np.uint64).astype(np.uint32)
    seen = np.concatenate([(np.arange(1024, dtype=np.int64) * n) // 1024, sample_places(n, 8192 if n >= 1 << 17 else 1024).astype(np.int64)])
    if kind == "misled_low":
        v[seen] = 0xFFFFFFFF
    elif kind == "misled_high":
        v[seen] = np.arange(len(seen)) % 1000
    elif kind == "misled_wide":
        v[:] = 0x80000000 + rng.integers(0, 1000, n)
        v[seen] = np.where(np.arange(len(seen)) % 2, 5, 0xFFFFFFF0)
    elif kind == "two_values":
        v = np.where(rng.random(n) < 0.5, 3, 0xFFFFFFFF).astype(np.uint32)
    elif kind == "top":
        v[:] = 0xFFFFFFFF
    off = np.array([0, n], dtype=np.uint64)
    assert builder.segment_stats(v, off).tolist() == [middle(v)]


@pytest.mark.parametrize("samples", [1, 511, 512, 513, 4095, 4096, 4097, 8193])
def test_sample_counts_at_the_borders_of_the_sort_tiles(builder, samples):
    """Tiles of the first sort pass and of the partition by key range: 512 threads, 4,096 samples."""
    rec = trace_with_rows([1] * (samples // 3) + [2] * (samples - samples // 3), "spread", samples)
    rec = rec[(rec["smem_word"] & (1 << 23)) == 0]  # no solo launches: the pairs are all the samples
    want = O.build_pair_table(rec)
    for _ in range(2):
        assert_tables_match(*builder.build(rec, time_ordered=True), *want)
    builder.build_streamed_device(rec, window_records=max(1, len(rec) // 2), n_parts=5)
    assert_tables_match(*builder.fetch(), *want)


def test_quotients_are_ieee_divisions(builder):
    """Sums, means, minima and maxima of every row: the integers of the row divided by the solo time, to the last bit (the
    kernel multiplies by a reciprocal and corrects)."""
    rng = np.random.default_rng(11)
    rec = trace_with_rows(rng.integers(1, 40, 3000).tolist(), "spread", 12)
    keys, pairs = builder.build(rec, time_ordered=True)
    dur = (rec["end_ns"] - rec["start_ns"]).astype(np.int64)
    tenant, solo = rec["smem_word"] >> 24, (rec["smem_word"] & (1 << 23)) != 0
    name_of = {int(k): int(n) for k, n in zip(keys["key"], keys["name_id"])}
    solo_of = {int(k): float(s) for k, s in zip(keys["key"], keys["solo_ns"])}
    mine = (tenant == 0) & ~solo
    name, d = rec["name_id"][mine].astype(int), dur[mine]
    total, count = np.bincount(name, d).astype(np.int64), np.bincount(name)
    low, high = np.full(len(total), 2**40), np.zeros(len(total), np.int64)
    np.minimum.at(low, name, d)
    np.maximum.at(high, name, d)
    seen = 0
    for row in pairs:
        p, s = name_of[int(row["key_a"])], solo_of[int(row["key_a"])]
        if np.isnan(s):
            continue
        seen += 1
        total_q = np.float64(total[p]) / s
        assert (row["sum_a"], row["mean_a"], row["min_a"], row["max_a"]) == (total_q, total_q / np.float64(count[p]), np.float64(low[p]) / s, np.float64(high[p]) / s)
    assert seen == 1000
