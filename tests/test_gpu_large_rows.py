"""GPU: rows of more than 8,192 samples at the sizes where their way changes -- a warp's or a CTA's sample for the pivots (2^17), a
second narrowing over many CTAs (2^19, if more than 2^15 values were collected: a sixteenth) -- against numpy's partition, bit
for bit; and what they cost."""
import ctypes
import time

import numpy as np
import pytest
import torch

from kernel_scheduling_b200 import _lib
from oracle import pair_table_oracle as O
from tests.helpers import assert_tables_match, sample_places
from tests.test_gpu_row_sizes import middle, trace_with_rows

pytestmark = pytest.mark.gpu


def values(kind, n, rng):
    if kind == "wide":
        return rng.integers(0, 2**32, n, dtype=np.uint64).astype(np.uint32)
    if kind == "ties":  # every value many times, the pivots among them
        return rng.integers(0, 90, n).astype(np.uint32)
    if kind == "ascending":
        return (np.arange(n) // 3).astype(np.uint32)
    if kind == "periodic":
        return rng.permutation(4096).astype(np.uint32)[np.arange(n) % 4096]
    if kind == "clusters":
        return np.where(rng.random(n) < 0.5, rng.integers(0, 1000, n), 0xFFFFFFFF - rng.integers(0, 1000, n)).astype(np.uint32)
    v = rng.integers(1000, 2**32 - 1000, n, dtype=np.uint64).astype(np.uint32)
    seen = sample_places(n, 8192 if n >= 1 << 17 else 1024)
    if kind == "misled_low":  # the sample says that the middle lies at the top
        v[seen] = 0xFFFFFFFF
    elif kind == "misled_high":
        v[seen] = np.arange(len(seen))
    elif kind == "misled_wide":  # everything lies between the pivots
        v[:] = 0x80000000 + rng.integers(0, 1000, n)
        v[seen] = np.where(np.arange(len(seen)) % 2, 5, 0xFFFFFFF0)
    return v


@pytest.mark.parametrize("n", [8193, (1 << 17) - 1, 1 << 17, (1 << 17) + 1, (1 << 19) - 1, 1 << 19, 620_001, 1_500_002])
@pytest.mark.parametrize("kind", ["wide", "ties", "ascending", "periodic", "clusters", "misled_low", "misled_high", "misled_wide"])
def test_large_segments(builder, n, kind):
    rng = np.random.default_rng(n)
    v = values(kind, n, rng)
    other = values("wide", 20_000, rng)
    off = np.cumsum([0, 5, n, 7, 9000, 20_000 - 5 - 7 - 9000]).astype(np.uint64)
    v = np.concatenate([other[:5], v, other[5:]])
    want = [middle(v[int(a):int(b)]) for a, b in zip(off[:-1], off[1:])]
    assert builder.segment_stats(v, off).tolist() == want


@pytest.mark.parametrize("sizes", [[130_000, 132_000, 3], [700_001, 20_000, 8193], [1_200_000]])
@pytest.mark.parametrize("kind", ["spread", "steps", "clusters"])
def test_large_table_rows(builder, sizes, kind):
    rec = trace_with_rows(sizes, kind, len(sizes))
    want = O.build_pair_table(rec)
    for _ in range(2):
        assert_tables_match(*builder.build(rec, time_ordered=True), *want)


def best_ms(builder, values, offsets):
    """Wall time of the stage call on device arrays, best of several."""
    v, off = torch.from_numpy(values.view(np.int32)).cuda(), torch.from_numpy(offsets.view(np.int64)).cuda()
    out = torch.zeros((len(offsets) - 1, 6), dtype=torch.int64, device="cuda")
    torch.cuda.synchronize()
    best = 1e9
    for _ in range(8):
        t0 = time.perf_counter()
        builder._check(builder._lib.ks_segment_stats(builder._h, ctypes.c_void_p(v.data_ptr()), ctypes.c_void_p(off.data_ptr()), len(offsets) - 1, _lib.ON_DEVICE,
                                                     ctypes.c_void_p(out.data_ptr())), "ks_segment_stats")
        best = min(best, 1e3 * (time.perf_counter() - t0))
    return best


def test_a_large_segment_costs_about_what_its_values_cost(builder):
    """One segment of 16 M values against the same values in 2,048 segments, and whatever order its values come in."""
    n = 1 << 24
    rng = np.random.default_rng(1)
    v = rng.integers(1, 60_000, n).astype(np.uint32)
    one = np.array([0, n], dtype=np.uint64)
    many = best_ms(builder, v, np.arange(0, n + 1, 8192, dtype=np.uint64))
    assert best_ms(builder, v, one) < 4 * many
    for period in (2, 64, 4096, 1 << 16):
        assert best_ms(builder, rng.integers(1, 60_000, period).astype(np.uint32)[np.arange(n) % period], one) < 4 * many, period
