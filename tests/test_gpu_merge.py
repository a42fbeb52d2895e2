"""GPU: traces that consist of a few ordered runs are merged, not sorted (ks_merge.cuh).  Against the same launches in start
order and against numpy's stable sort, at the borders of the merge tiles (2,048 launches) and of the number of runs (32)."""
import numpy as np
import pytest

from kernel_scheduling_b200 import trace

pytestmark = pytest.mark.gpu


def in_runs(rec, runs, seed):
    """The trace cut into `runs` pieces that come in reverse order."""
    cuts = np.sort(np.random.default_rng(seed).choice(np.arange(1, len(rec)), runs - 1, replace=False))
    return np.concatenate(np.split(rec, cuts)[::-1])


def pairs_of(idx):
    return sorted(zip(idx[0].tolist(), idx[1].tolist()))


@pytest.mark.parametrize("n", [40, 2047, 2048, 2049, 6145, 60_000])
@pytest.mark.parametrize("runs", [2, 3, 5, 31, 32, 33, 40])
def test_runs_give_the_table_of_the_ordered_trace(builder, n, runs):
    rec = trace.generate(trace.config("c3", n), interleave_solo=True)
    rec["start_ns"] -= rec["start_ns"] % np.uint64(5000)  # many equal starts
    rec = rec[np.argsort(rec["start_ns"], kind="stable")]
    keys, pairs = builder.build(rec, time_ordered=True)
    mixed = in_runs(rec, runs, n)
    mkeys, mpairs = builder.build(mixed)
    assert keys.tobytes() == mkeys.tobytes() and pairs.tobytes() == mpairs.tobytes()
    assert builder.info["was_time_ordered"] == 0
    assert builder.info["min_start_ns"] == rec["start_ns"][0] and builder.info["max_start_ns"] == rec["start_ns"][-1]
    # equal starts keep the order of the input: the join's positions are those in numpy's stable order
    stable = mixed[np.argsort(mixed["start_ns"], kind="stable")]
    assert pairs_of(builder.join_overlaps(mixed)) == pairs_of(builder.join_overlaps(stable))


def test_one_log_per_tenant(builder):
    rec = trace.generate(trace.config("c3", 50_000))
    logs = rec[np.argsort(rec["smem_word"] >> 24, kind="stable")]
    want, got = builder.build(rec, time_ordered=True), builder.build(logs)
    assert all(w.tobytes() == g.tobytes() for w, g in zip(want, got))


@pytest.mark.parametrize("ordered", [(True, True), (True, False), (False, True), (False, False)])
def test_batches_of_ordered_and_unordered_logs(builder, ordered):
    rng = np.random.default_rng(5)
    pool = rng.permutation(300_000).astype(np.uint64) + np.uint64(10**12)
    s1, s2 = pool[:70_001], rng.permutation(pool[50_000:170_000])
    both = 20_001
    s1, s2 = (np.sort(s) if o else s for s, o in zip((s1, s2), ordered))
    assert builder.count_batches(s1, s2) == [len(s1) + len(s2) - 2 * both, both]
