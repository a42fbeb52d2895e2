"""The calls that programs make of this library, as timed cases: what an offline rebuild of the interference table, an
online scheduler that keeps the table resident, and the stage calls behind the drop-in scripts do.

The traces are the benchmark configurations of ``kernel_scheduling_b200.trace`` (c1 .. c5) at their own sizes and at
sizes around them.  Records that are already on the GPU (an agent that stages its launches there, or the ingest of this
library) stay there and so do the tables; where a caller holds host data the whole call with its copies counts.
"""
import ctypes
import math

import numpy as np
import torch

from kernel_scheduling_b200 import _lib, trace
from kernel_scheduling_b200.make_pair_eff import TraceIngest, records_from_log
from kernel_scheduling_b200.pair_table import PairTableBuilder

# overlapping launch pairs per record of each workload (a property of its tenants' utilisations)
PAIRS_PER_RECORD = {"c1": 0.42, "c2": 0.438, "c3": 2.014, "c4": 3.32, "c5": 0.44}


def listed():
    return [
        # a short profiling run (some seconds of two small models): launches and host waits are what it costs
        {"name": "build_c1_20k", "kind": "build", "workload": "c1", "n": 20_000, "order": "start", "key_type": False},
        # the offline program on its 200,000 launches, host arrays in log order, SHAPE and TYPE tables (make_pair_eff)
        {"name": "make_tables_c1_200k", "kind": "make_tables", "workload": "c1", "n": 200_000},
        # a medium trace, TYPE keys (the fallback rows of the daemon), a size that is no multiple of anything
        {"name": "build_c2_type_2345677", "kind": "build", "workload": "c2", "n": 2_345_677, "order": "start", "key_type": True},
        # the two-tenant LLM + speech configuration at its full size
        {"name": "build_c2_10M", "kind": "build", "workload": "c2", "n": 10_000_000, "order": "start", "key_type": False},
        # the agents' logs one behind the other (every log ordered, their concatenation not): ordered on the GPU first
        {"name": "build_c3_20M_logs", "kind": "build", "workload": "c3", "n": 20_000_000, "order": "logs", "key_type": False},
        # the four-tenant configuration at its full size, the largest that goes through one call
        {"name": "build_c3_100M", "kind": "build", "workload": "c3", "n": 100_000_000, "order": "start", "key_type": False},
        # host records in (page-locked), host tables out (new arrays)
        {"name": "build_c2_3M_host", "kind": "build_host", "workload": "c2", "n": 3_000_000},
        # the eight-tenant configuration in windows and key ranges (a trace beyond one call, at a 32nd of its size)
        {"name": "streamed_c4_32M", "kind": "streamed", "workload": "c4", "n": 32_000_000, "window": 1 << 23, "parts": 8},
        # an online session: windows of 65,536 launches merged into the resident table, then the table read out
        {"name": "online_c5_24x64k", "kind": "online", "workload": "c5", "n": 65_536, "windows": 24},
        # the grouping primitive by itself (joins of decision logs, group-bys): 64-bit keys with payload
        {"name": "sort_pairs_u64_12M", "kind": "sort", "n": 12_000_003, "bits": 64},
        # the batch counter of postprocess.py on two logs of its 200,000 rows
        {"name": "count_batches_200k", "kind": "batches", "n": 200_000},
        # an agent's timing log (text, host memory) into launch records
        {"name": "ingest_log_100k", "kind": "ingest", "n": 100_000},
    ]


def _log_uniform(rng, lo, hi):
    return int(math.exp(rng.uniform(math.log(lo), math.log(hi))))


def draw(rng):
    kind = rng.choice(["build", "build", "build", "build", "make_tables", "build_host", "streamed", "online", "sort", "batches", "ingest"])
    if kind == "build":
        workload = rng.choice(["c1", "c2", "c2", "c3", "c3", "c4"])
        most = {"c1": 2_000_000, "c2": 20_000_000, "c3": 40_000_000, "c4": 20_000_000}[workload]
        return {"kind": kind, "workload": workload, "n": _log_uniform(rng, 5_000, most) | 1, "order": rng.choice(["start", "start", "logs", "shuffled"]),
                "key_type": rng.random() < 0.25, "mix": rng.randrange(1000)}
    if kind == "make_tables":
        return {"kind": kind, "workload": "c1", "n": _log_uniform(rng, 20_000, 1_000_000), "mix": rng.randrange(1000)}
    if kind == "build_host":
        return {"kind": kind, "workload": rng.choice(["c2", "c3"]), "n": _log_uniform(rng, 100_000, 6_000_000), "mix": rng.randrange(1000)}
    if kind == "streamed":
        return {"kind": kind, "workload": rng.choice(["c3", "c4"]), "n": _log_uniform(rng, 2_000_000, 30_000_000), "window": 1 << rng.randrange(20, 24),
                "parts": rng.randrange(2, 17), "mix": rng.randrange(1000)}
    if kind == "online":
        return {"kind": kind, "workload": "c5", "n": _log_uniform(rng, 8_192, 131_072), "windows": rng.randrange(4, 33), "mix": rng.randrange(1000)}
    if kind == "sort":
        return {"kind": kind, "n": _log_uniform(rng, 10_000, 20_000_000), "bits": rng.choice([32, 64])}
    if kind == "batches":
        return {"kind": kind, "n": _log_uniform(rng, 5_000, 1_000_000)}
    return {"kind": kind, "n": _log_uniform(rng, 5_000, 200_000)}


# ---- inputs ---------------------------------------------------------------------------------------------------------
_staging = {}


def _host_trace(case, seed):
    """The launches of the case in start order, in a page-locked array that the next call overwrites."""
    n = case["n"] * case.get("windows", 1)
    if _staging.get("n", 0) < n:
        _staging.clear()
        _staging["n"], _staging["buffer"] = n, torch.empty(n * 48, dtype=torch.uint8, pin_memory=True)
    out = trace.to_dtype(_staging["buffer"].numpy()[: n * 48])
    spec = trace.config(case["workload"], n, seed=case.get("mix"))
    return trace.generate_fast(spec, window=seed, out=out, interleave_solo=case["kind"] == "online")


def _device_trace(case, seed):
    rec = torch.from_numpy(_host_trace(case, seed).view(np.uint8)).cuda()
    if case.get("order") in ("logs", "shuffled"):
        words = rec.view(torch.int32).view(-1, 12)
        if case["order"] == "logs":  # one ordered run per tenant
            at = torch.sort((words[:, 7] >> 24) & 255, stable=True).indices
        else:
            at = torch.randperm(len(words), device="cuda", generator=torch.Generator("cuda").manual_seed(seed))
        rec = words[at].contiguous().view(torch.uint8).view(-1)
    return rec


def _log_text(case, seed):
    """One process's timing log with the 17 columns the agent writes."""
    rec = _host_trace({"kind": "ingest", "workload": "c1", "n": case["n"]}, seed)
    cols = "kernel_id kernel_us prefetch_us prefetch_to_kernel_gap_us hook_tag prefetch_bytes prefetched_tensors args_check kernel_name start_ns end_ns batch_id batch_size batch_pos block model grid"
    lines = ["\t".join(cols.split())]
    rows = zip(rec["name_id"].tolist(), rec["start_ns"].tolist(), rec["end_ns"].tolist(), rec["block"].tolist(), rec["grid"].tolist())
    for i, (name, start, end, b, g) in enumerate(rows):
        lines.append(f"{i}\t{(end - start) / 1000:.3f}\t\t\tunknown\t0\t\t-\tvoid ns::kernel_{name}<float>(float*)\t{start}\t{end}\t{i + 1}\t1\t0\t"
                     f"({b[0]}, {b[1]}, {b[2]})\tqwen\t({g[0]}, {g[1]}, {g[2]})")
    return ("\n".join(lines) + "\n").encode()


def _batch_starts(case, seed):
    """start_ns of two logs without repeats inside a log; a tenth to a third of them agree."""
    rng = np.random.default_rng([seed, 11])
    pool = 1_000_000_000_000 + np.cumsum(rng.integers(1, 20_000, 2 * case["n"], dtype=np.int64))
    rng.shuffle(pool)
    n, both = case["n"], int(rng.integers(case["n"] // 10, case["n"] // 3))
    return np.sort(pool[:n]).astype(np.uint64), np.sort(pool[n - both: 2 * n - both]).astype(np.uint64)


def prepare(case, seed):
    kind = case["kind"]
    state = {"case": case}
    if kind in ("build", "streamed", "online", "sort"):
        # launched on a stream of the program's own, so that its tensors and the library's work are ordered
        state["stream"] = torch.cuda.Stream()
        state["builder"] = PairTableBuilder(stream=state["stream"].cuda_stream)
    else:
        state["builder"] = PairTableBuilder()
    if kind in ("build", "streamed", "online"):
        state["records"] = _device_trace(case, seed)
    elif kind == "make_tables":
        state["records"] = trace.to_dtype(_device_trace(dict(case, order="logs"), seed).cpu().numpy())
    elif kind == "build_host":
        state["records"] = state["builder"].pinned_records(case["n"])
        state["records"][:] = _host_trace(case, seed)
    elif kind == "sort":
        gen = torch.Generator("cuda").manual_seed(seed)
        dtype = torch.int64 if case["bits"] == 64 else torch.int32
        bound = torch.iinfo(dtype)
        state["keys"] = torch.randint(bound.min, bound.max, (case["n"],), dtype=dtype, device="cuda", generator=gen)
        state["vals"] = torch.arange(case["n"], dtype=dtype, device="cuda")
    elif kind == "batches":
        state["starts"] = _batch_starts(case, seed)
    else:
        state["text"] = _log_text(case, seed)
    if kind in ("build", "streamed"):
        state["tables"] = [_table_buffers(case, device="cuda")]
    elif kind in ("build_host", "online", "make_tables"):
        state["tables"] = [_table_buffers(case, pin_memory=True) for _ in range(2 if kind == "make_tables" else 1)]
    torch.cuda.synchronize()
    return state


# ---- one pass -------------------------------------------------------------------------------------------------------
def _capacity(case):
    """Rows of the caller's pair table: every pair of keys of different tenants, or twice the expected rows where that is far less."""
    sizes = [t.n_keys for t in trace.config(case["workload"]).tenants]
    return min((sum(sizes) ** 2 - sum(k * k for k in sizes)) // 2, max(10_000_000, 10_000 + 2 * int(_expected_rows(case))))


def _table_buffers(case, **where):
    """The caller's buffers of a table: key rows as 18 and pair rows as 16 words (rows behind the table stay zero)."""
    n_keys = sum(t.n_keys for t in trace.config(case["workload"]).tenants)
    return torch.zeros((n_keys, 18), dtype=torch.int32, **where), torch.zeros((_capacity(case), 16), dtype=torch.int64, **where)


def _copy_table(b, tables):
    """The tables of the last build into the caller's buffers."""
    lib, flags = _lib.load(), _lib.ON_DEVICE if tables[0].is_cuda else 0
    rows = []
    for copy, t in ((lib.ks_copy_key_rows, tables[0]), (lib.ks_copy_pair_rows, tables[1])):
        rows.append(copy(b._h, ctypes.c_void_p(t.data_ptr()), len(t), flags))
        if rows[-1] < 0:
            raise RuntimeError(lib.ks_last_error(b._h).decode())
    return _columns(*tables, rows)


def _columns(keys, pairs, rows):
    """Whole and floating columns of a table."""
    return {"rows": np.array(rows), "keys": keys[:, :16], "solo_ns": keys.view(torch.float64)[:, 8], "pairs": pairs[:, :4], "span": pairs[:, 15],
            "stats": pairs.view(torch.float64)[:, 4:15]}


def run(state):
    case, b = state["case"], state["builder"]
    kind = case["kind"]
    if kind == "build":
        b.build_device(state["records"].data_ptr(), case["n"], time_ordered=case["order"] == "start", key_type=case["key_type"])
        return _copy_table(b, state["tables"][0])
    if kind == "streamed":
        b.build_streamed_device(state["records"].data_ptr(), case["n"], window_records=case["window"], n_parts=case["parts"])
        return _copy_table(b, state["tables"][0])
    if kind == "online":
        b.update_begin()
        samples = [b.update(state["records"].data_ptr() + w * case["n"] * 48, case["n"]) for w in range(case["windows"])]
        if _lib.load().ks_update_table(b._h) < 0:
            raise RuntimeError(_lib.load().ks_last_error(b._h).decode())
        return {"samples": np.array(samples), **_copy_table(b, state["tables"][0])}
    if kind == "make_tables":
        out = []
        for key_type, tables in zip((False, True), state["tables"]):
            b.build_device(state["records"], key_type=key_type)
            out.append(_copy_table(b, tables))
        return out
    if kind == "build_host":
        b.build_device(state["records"], time_ordered=True)
        return _copy_table(b, state["tables"][0])
    if kind == "sort":  # in place, so on a copy
        lib = _lib.load()
        with torch.cuda.stream(state["stream"]):
            keys, vals = state["keys"].clone(), state["vals"].clone()
            fn = lib.ks_sort_pairs_u64 if case["bits"] == 64 else lib.ks_sort_pairs_u32
            if fn(b._h, ctypes.c_void_p(keys.data_ptr()), ctypes.c_void_p(vals.data_ptr()), case["n"], 0, case["bits"], _lib.ON_DEVICE) < 0:
                raise RuntimeError(lib.ks_last_error(b._h).decode())
            return keys, vals
    if kind == "batches":
        return b.count_batches(*state["starts"])
    return records_from_log(TraceIngest(), b, state["text"], solo=False).view(np.int32).reshape(-1, 12)


# ---- what a pass cannot do without ----------------------------------------------------------------------------------
def _expected_rows(case):
    """Expected distinct key pairs among the overlapping launches."""
    n = case["n"] * case.get("windows", 1)
    spec = trace.config(case["workload"], n)
    probs = [1.0 / np.arange(1, t.n_keys + 1) ** t.zipf_s for t in spec.tenants]
    probs = [p / p.sum() for p in probs]
    mean = np.array([t.dur_median_ns * np.exp(0.5 * t.dur_sigma**2) for t in spec.tenants])
    rate = np.array([t.utilisation for t in spec.tenants]) / mean
    busy = np.array([t.utilisation for t in spec.tenants])
    share = {(a, c): rate[a] * busy[c] + rate[c] * busy[a] for a in range(len(probs)) for c in range(a)}
    pairs = PAIRS_PER_RECORD[case["workload"]] * n
    return sum((1.0 - np.exp(-pairs * s / sum(share.values()) * np.outer(probs[a], probs[c]))).sum() for (a, c), s in share.items())


def work(case):
    kind, n = case["kind"], case["n"]
    if kind in ("build", "build_host", "streamed", "online", "make_tables"):
        keys = sum(t.n_keys for t in trace.config(case["workload"]).tenants)
        once = 48.0 * n * case.get("windows", 1) + 128.0 * _expected_rows(case) + 72.0 * keys
        return {"bytes": once * (2 if kind == "make_tables" else 1), "flops": 0}
    if kind == "sort":
        return {"bytes": 2.0 * 2 * n * case["bits"] / 8, "flops": 0}
    if kind == "batches":
        return {"bytes": 2.0 * 8 * n, "flops": 0}
    return {"bytes": (132.0 + 48.0) * n, "flops": 0}


def tolerance(case):
    # whole numbers and their IEEE quotients: every value of the tables is defined bit for bit
    return "exact"


# ---- the same tables from plain torch in 64 bits --------------------------------------------------------------------
_SIGN = -(1 << 63)


def _signed(v):
    return v - (1 << 64) if v >= 1 << 63 else v


def _mix64(x):
    for shift, factor in ((30, 0xBF58476D1CE4E5B9), (27, 0x94D049BB133111EB), (31, 1)):
        x = (x ^ ((x >> shift) & ((1 << (64 - shift)) - 1))) * _signed(factor)
    return x


def _kernel_keys(w, key_type):
    """Keys of the records (12 words each as int64), as signed numbers that sort like the unsigned keys."""
    name, gx, gy, gz, bx, by, bz, word = (w[:, i] & 0xFFFFFFFF for i in range(8))
    word = word & ~(1 << 23)
    if key_type:
        gx, gy, gz, word = gx * 0, gy * 0, gz * 0, word & 0xFF000000
    h = torch.zeros_like(name)
    for lo, hi in ((name, gx), (gy, gz), (bx, by), (bz, word)):
        h = _mix64((h ^ (lo | (hi << 32))) + _signed(0x9E3779B97F4A7C15))
    return torch.where(h == 0, torch.ones_like(h), h) ^ _SIGN


def _middle(sorted_vals, first, count):
    return sorted_vals[first + (count - 1) // 2].double(), sorted_vals[first + count // 2].double()


def _exact_table(case, rec, key_type=False):
    words = rec.view(torch.int32).view(-1, 12)
    start, end = (rec.view(torch.int64).view(-1, 6)[:, i] for i in (4, 5))
    _, kid = torch.unique(_kernel_keys(words.long(), key_type), return_inverse=True)
    nk = int(kid.max()) + 1
    solo = (words[:, 7] >> 23 & 1).bool()
    # solo times
    sk, sd = kid[solo], (end - start)[solo]
    sorted_solo = torch.sort(sk << 32 | sd).values
    count = torch.bincount(sk, minlength=nk)
    first = torch.cumsum(count, 0) - count
    has = count > 0
    solo_ns = torch.full((nk,), math.nan, dtype=torch.float64, device=rec.device)
    lo, hi = _middle(sorted_solo & 0xFFFFFFFF, first[has], count[has])
    solo_ns[has] = (lo + hi) * 0.5
    # overlapping launches of different tenants, each pair once from its earlier launch
    s, at = torch.sort(start[~solo], stable=True)
    e, k, t = end[~solo][at], kid[~solo][at], (words[:, 7] >> 24 & 255)[~solo][at]
    here = torch.arange(len(s), device=rec.device)
    run_len = (torch.searchsorted(s, e) - here - 1).clamp_(min=0)
    i = torch.repeat_interleave(here, run_len)
    j = i + 1 + torch.arange(len(i), device=rec.device) - (torch.cumsum(run_len, 0) - run_len)[i]
    ok = (t[i] != t[j]) & (s[i] < e[j])
    i, j = i[ok], j[ok]
    swap = t[i] > t[j]
    a, c = torch.where(swap, j, i), torch.where(swap, i, j)
    row, count = torch.unique(k[a] * nk + k[c], return_inverse=True, return_counts=True)[1:]
    ids = torch.empty(len(count), dtype=torch.int64, device=rec.device).scatter_(0, row, k[a] * nk + k[c])
    solo_a, solo_c = solo_ns[ids // nk], solo_ns[ids % nk]
    first = torch.cumsum(count, 0) - count
    out = []
    for value, base in (((e - s)[a], solo_a), ((e - s)[c], solo_c)):
        v = torch.sort(row << 32 | value).values & 0xFFFFFFFF
        upto = torch.cumsum(v, 0)
        total = upto[first + count - 1] - upto[first] + v[first]
        lo, hi = _middle(v, first, count)
        base = torch.where(base > 0, base, math.nan)
        out += [total / base, total / base / count, v[first] / base, v[first + count - 1] / base, (lo / base + hi / base) * 0.5]
    span = torch.maximum(e[i], e[j]) - s[i]
    lo, hi = _middle(torch.sort(row << 32 | span).values & 0xFFFFFFFF, first, count)
    both = torch.where((solo_a > 0) & (solo_c > 0), solo_a + solo_c, math.nan)
    out.append((both / lo + both / hi) * 0.5)
    keys, pairs = _table_buffers(case, device=rec.device)
    keys.view(torch.float64)[:nk, 8] = solo_ns
    pairs.view(torch.float64)[: len(ids), 4:15] = torch.stack(out, 1)
    return dict(_columns(keys, pairs, [nk, len(ids)]), keys=None, pairs=None, span=None)


def exact(case, seed):
    kind = case["kind"]
    if kind in ("build", "streamed", "build_host"):
        return _exact_table(case, _device_trace(case, seed), case.get("key_type", False))
    if kind == "online":
        return {"samples": None, **_exact_table(case, _device_trace(case, seed))}
    if kind == "make_tables":
        rec = _device_trace(dict(case, order="logs"), seed)
        return [_exact_table(case, rec, key_type) for key_type in (False, True)]
    return None  # whole numbers throughout
