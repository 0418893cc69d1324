"""Autotuner for the transform launch schedule (vfhe_cuda_ntt_set_schedule).

For a (log2 P, rows-per-launch) class the tuner times every candidate schedule of the
FP64 transform -- tile bits (one pass, or a radix-2^(logP - tile_bits) column pass
followed by tiles), tiles per CTA, and one-CTA-per-tile-group vs a persistent grid of
k CTAs per SM -- on forward + inverse transforms of several row counts of the class (odd
and even, from its start to its end), and keeps the one whose times, relative to the built-in
schedule's, have the least mean.  Schedules never change results (the transform is exact),
so a tuned table can be applied at any time.  The table is a JSON file keyed "logP/rows_log2";
``apply`` loads it into the engine and missing classes use the nearest tuned bucket
of the same logP.

A transform's schedule also sets what a key switch's fused column pass and division finds to
do behind it (2^tile_bits columns a polynomial), which is not timed here: few rows of 2^13
points and more want larger tiles than the transform alone does (one multiply at N = 2^15,
9 limbs: 88 us on 2^11 and 2^12 tiles, 106 on the tiles this tuner prefers).

    python -m vfhe_b200.autotune --out vfhe_b200/tuned/ntt_schedule_b200.json
"""

from __future__ import annotations

import argparse
import json
from pathlib import Path

import numpy as np

from .native import Engine, cuda_engine

DEFAULT_TABLE = Path(__file__).resolve().parent / "tuned" / "ntt_schedule_b200.json"
MAX_ELEMS = 1 << 28  # at most 2 GiB of rows per timed buffer
BUCKETS = tuple(range(4, 16))
KEEP_DEFAULT_MARGIN = 0.01  # a tuned schedule must beat the built-in one by 1%


def candidates(logP: int) -> list[tuple[int, int, int]]:
    """(tile_bits, tiles_per_cta, ctas_per_sm) triples worth timing for one logP."""
    if logP <= 13:  # one pass, or a short column pass in front of smaller tiles
        tiles = {k for k in (logP, logP - 1, logP - 2, logP - 3) if k >= 8}
    else:  # a column pass of radix 2^(logP - k) is required
        tiles = set(range(max(8, logP - 5), 14))
    out = []
    for k in sorted(tiles):
        tpt = 1 << (k - 4)
        tpcs = [0] + [t for t in (1, 2, 4, 8) if tpt * t <= max(256, tpt) and tpt * t >= 64]
        for tpc in sorted(set(tpcs)):
            for cps in (0, 2, 4):
                out.append((k, tpc, cps))
    # fused split transforms on a thread-block cluster of 2^(logP - k) CTAs (ctas_per_sm = -1)
    for k in (11, 12, 13):
        if 1 <= logP - k <= 3:
            out.append((k, 0, -1))
    # column pass and tile pass as one dataflow launch (ctas_per_sm = -2; tiles_per_cta =
    # work items per ticket)
    for k in (10, 11, 12, 13):
        if flow_supported(k, logP - k):
            out.extend((k, per, -2) for per in (1, 2))
    return out


def flow_supported(k: int, k1: int) -> bool:
    """Shapes of the dataflow launch (ntt_flow.cu): 2^k-point tiles, a radix-2^k1 column
    pass, and the tiles of one 256-thread item in one row."""
    if not (10 <= k <= 13 and 2 <= k1 <= 4):
        return False
    per_item = 1 if k >= 12 else (2 if k == 11 else 4)
    return per_item <= (1 << k1)


def row_counts(bucket: int) -> list[int]:
    """Row counts a class is timed at, multiples of the three limbs of a timed polynomial: odd
    ones near its start and past its middle (tiles that do not fill CTAs evenly), three times a
    power of two (tiles that do), and one near its end."""
    n = 1 << bucket
    polys = ((n + n // 8) // 3 | 1, n // 2, n // 2 + 1 | 1, (2 * n - n // 8) // 3)
    return sorted({3 * b for b in polys if n <= 3 * b < 2 * n})


def _device_ms(call, captured: bool, reps: int) -> float:
    """Device time of call(stream) the two ways a program launches, averaged: queued on a stream
    (behind a wait of the device: one by one, the host's launch rate would hide what a schedule
    does below some 10 us) and, where it can be, captured in a CUDA graph (queued launches start
    on a grid of about 2 us, which hides smaller differences)."""
    import torch

    stream = torch.cuda.Stream()
    ev0, ev1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)

    def best_of(enqueue, count: int) -> float:
        best = float("inf")
        for _ in range(reps):
            torch.cuda._sleep(50_000 * (count + 1))
            ev0.record(stream)
            enqueue()
            ev1.record(stream)
            stream.synchronize()
            best = min(best, ev0.elapsed_time(ev1) / count)
        return best

    with torch.cuda.stream(stream):
        call(stream)
        ev0.record(stream)
        call(stream)
        ev1.record(stream)
        stream.synchronize()
        count = max(1, min(20, int(0.5 / max(ev0.elapsed_time(ev1), 1e-3))))

        def several() -> None:
            for _ in range(count):
                call(stream)

        queued = best_of(several, count)
        if not captured:
            return queued
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=stream):
            several()
        return (queued + best_of(graph.replay, count)) / 2


def _time_shape(engine: Engine, logP: int, rows: int, cands, reps: int = 5) -> dict[tuple, float]:
    """Device ms of one forward and one inverse transform of `rows` rows by candidate."""
    import torch

    from .arith import Ring

    ffi, lib = engine.ffi, engine.lib
    N = 1 << logP
    L = 3
    R = Ring(N, prime_size=[50] * L, split_degree=1, engine=engine)
    batch = rows // L
    buf = torch.empty((batch, L, N), dtype=torch.int64, device="cuda")
    for k, q in enumerate(R.primes):
        buf[:, k].random_(0, q)
    limbs = ffi.new("uint32_t[]", R.prime_indices)
    p = ffi.cast("uint64_t*", buf.data_ptr())

    def both(stream) -> None:
        for inverse in (0, 1):
            lib.vfhe_cuda_ntt_batch(R.NTT, inverse, p, p, batch, limbs, L, ffi.cast("void*", stream.cuda_stream))

    bucket = (batch * L).bit_length() - 1
    res = {}
    for c in cands:
        if lib.vfhe_cuda_ntt_set_schedule(logP, bucket, *c) != 0:
            lib.vfhe_cuda_clear_error()
            continue
        res[c] = _device_ms(both, c[2] != -2, reps)  # (the dataflow launch does not run under capture)
    lib.vfhe_cuda_ntt_set_schedule(logP, bucket, 0, 0, 0)
    engine.check("autotune")
    return res


def choose(timed: list[dict[tuple, float]], default: tuple) -> tuple[tuple, float, float | None]:
    """The schedule of one class from the times at its row counts: (schedule, its mean ms, the
    built-in one's), the built-in one unless another's mean relative time is 1% less."""
    cands = set.intersection(*(set(t) for t in timed))
    mean = lambda c: sum(t[c] for t in timed) / len(timed)  # noqa: E731
    base = [t.get(default) or min(t.values()) for t in timed]
    ratio = {c: sum(t[c] / b for t, b in zip(timed, base)) / len(timed) for c in cands}
    best = min(sorted(cands), key=ratio.__getitem__)
    if default in cands and ratio[best] > 1.0 - KEEP_DEFAULT_MARGIN:
        best = default
    return best, mean(best), mean(default) if default in cands else None


def tune(engine: Engine | None = None, logps=range(8, 18), buckets=BUCKETS, reps: int = 5,
         verbose: bool = False) -> dict:
    """Time every candidate for each (logP, bucket) that fits MAX_ELEMS; returns the table."""
    engine = engine or cuda_engine()
    table = {}
    for logP in logps:
        cands = candidates(logP)
        default = (logP if logP <= 13 else 12, 0, 0)
        for b in buckets:
            timed = [_time_shape(engine, logP, rows, cands, reps) for rows in row_counts(b) if rows << logP <= MAX_ELEMS]
            if not timed or not all(timed):
                continue
            best, best_ms, default_ms = choose(timed, default)
            table[f"{logP}/{b}"] = {"schedule": list(best), "ms": best_ms, "default_ms": default_ms}
            if verbose:
                print(f"logP={logP} rows=2^{b}: best {best} {best_ms:.4f} ms (default {default_ms})", flush=True)
    return table


def apply(engine: Engine, table: dict) -> int:
    """Load a tuned table into the engine; every bucket of a tuned logP gets the nearest
    tuned entry.  Returns the number of (logP, bucket) classes set."""
    by_logp: dict[int, dict[int, list[int]]] = {}
    for key, val in table.items():
        lp, b = (int(x) for x in key.split("/"))
        by_logp.setdefault(lp, {})[b] = val["schedule"]
    n = 0
    for lp, entries in by_logp.items():
        tuned = sorted(entries)
        for b in range(32):
            near = min(tuned, key=lambda t: (abs(t - b), t))
            if engine.lib.vfhe_cuda_ntt_set_schedule(lp, b, *entries[near]) != 0:
                engine.lib.vfhe_cuda_clear_error()
                continue
            n += 1
    return n


def load(path: Path = DEFAULT_TABLE) -> dict | None:
    try:
        return json.loads(Path(path).read_text())["table"]
    except (OSError, ValueError, KeyError):
        return None


def main() -> None:
    ap = argparse.ArgumentParser()
    ap.add_argument("--out", default=str(DEFAULT_TABLE))
    ap.add_argument("--reps", type=int, default=5)
    ap.add_argument("--logp", type=int, nargs="*", default=None, help="tune only these log2 P (default 8..17)")
    ap.add_argument("--merge", action="store_true", help="keep the --out table's entries for other log2 P")
    args = ap.parse_args()
    import torch

    eng = cuda_engine(apply_tuned=False)
    table = tune(eng, logps=args.logp or range(8, 18), reps=args.reps, verbose=True)
    if args.merge:
        old = load(Path(args.out)) or {}
        old.update(table)
        table = old
    out = {"device": torch.cuda.get_device_name(0), "table": table,
           "note": "ms = forward + inverse transform of rows of 2^logP, mean over row counts from 2^bucket on, "
                   "device time"}
    Path(args.out).parent.mkdir(parents=True, exist_ok=True)
    Path(args.out).write_text(json.dumps(out, indent=1, sort_keys=True))
    gains = [v["default_ms"] / v["ms"] for v in table.values() if v.get("default_ms")]
    print(f"tuned {len(table)} classes; median gain over default {np.median(gains):.3f}x, max {max(gains):.3f}x")


if __name__ == "__main__":
    main()
