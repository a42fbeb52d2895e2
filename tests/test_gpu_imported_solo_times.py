"""GPU: the quotients of a table over solo times that a caller imports (ks_mg_solo), which may be any positive numbers: IEEE
divisions to the last bit, also where a reciprocal, a quotient or a remainder is no normal number."""
import numpy as np
import pytest
import torch

from kernel_scheduling_b200 import parallel
from kernel_scheduling_b200.pair_table import PairTableBuilder
from kernel_scheduling_b200.records import KEY_ROW_DTYPE, PAIR_ROW_DTYPE
from tests.test_gpu_row_sizes import trace_with_rows

pytestmark = pytest.mark.gpu

EXTREMES = [5e-324, 3e-310, 2.3e-308, 1e-290, 2.0**-901, 2.0**-900, 2.0**-899, 1e-100, 0.3, 1.0, 3.0, 1e17, 1e200, 2.0**900, 2.0**901, 1e300, 8e307, 1.7976931348623157e308, np.inf, np.nan, 0.0]


def test_quotients_over_imported_solo_times():
    rec = trace_with_rows(np.random.default_rng(3).integers(1, 700, 200).tolist(), "spread", 4)
    stream = torch.cuda.Stream()
    with torch.cuda.stream(stream), PairTableBuilder(device=0, stream=stream.cuda_stream) as b:
        s = parallel.GpuStages(b, torch.from_numpy(rec.view(np.uint8).copy()).cuda())
        s.begin(False)
        s.global_keys(*s.local_keys())
        s.samples()
        s.reduce(s.partition([], 0, 1))

        def pairs_over(solo):
            s.solo_import(torch.from_numpy(solo).cuda())
            s.finalize()
            keys, pairs = s.tables()
            torch.cuda.synchronize()
            return keys.cpu().numpy().view(KEY_ROW_DTYPE), pairs.cpu().numpy().view(PAIR_ROW_DTYPE)

        keys, whole = pairs_over(np.ones(s.n_keys))  # over 1.0: the integers themselves (a median: half of the sum of two)
        solo = np.array([EXTREMES[i % len(EXTREMES)] for i in range(s.n_keys)])
        with np.errstate(all="ignore"):
            solo[:: 5] *= 1.0 + 1e-3 * np.arange(len(solo[:: 5])) / len(solo)
        keys, pairs = pairs_over(solo)
    at = {int(k): i for i, k in enumerate(keys["key"])}
    seen = set()
    with np.errstate(all="ignore"):
        for row, ints in zip(pairs, whole):
            for side in ("a", "b"):
                d = solo[at[int(row["key_" + side])]]
                got = [row[c + side] for c in ("sum_", "mean_", "min_", "max_")]
                if not d > 0:
                    assert np.isnan(got).all()
                    continue
                total = np.float64(ints["sum_" + side]) / d
                want = [total, total / np.float64(row["count"]), np.float64(ints["min_" + side]) / d, np.float64(ints["max_" + side]) / d]
                assert np.array_equal(got, want, equal_nan=True), (d, got, want)
                if row["count"] % 2:  # one middle value
                    mid = np.float64(ints["median_" + side]) / d
                    assert np.array_equal([row["median_" + side]], [(mid + mid) * 0.5], equal_nan=True), d
                seen.add(float(d))
    assert {5e-324, 1e300, np.inf} <= seen
