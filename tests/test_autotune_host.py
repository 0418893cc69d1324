"""Autotuner host logic: candidate schedules are valid, tables apply to every bucket."""

from __future__ import annotations

import json


def test_candidates_respect_kernel_limits():
    from vfhe_b200.autotune import candidates

    for logP in range(8, 18):
        cands = candidates(logP)
        assert cands, logP
        assert (logP if logP <= 13 else 12, 0, 0) in cands  # the built-in schedule is always timed
        for k, tpc, cps in cands:
            assert 8 <= k <= 13 and k <= logP and logP - k <= 5
            assert tpc in (0, 1, 2, 4, 8) and cps in (0, 2, 4, -1, -2)
            if cps == -1:
                assert 11 <= k <= 13 and 1 <= logP - k <= 3
            if cps == -2:  # dataflow launch: 10..13 tile bits, radix 4..16 columns, one row per item
                assert 10 <= k <= 13 and 2 <= logP - k <= 4 and tpc in (1, 2)
                assert (max(256, 1 << (k - 4)) >> (k - 4)) <= (1 << (logP - k))
            if tpc and cps != -2:  # tiles one CTA holds (for -2: work items per ticket)
                assert (1 << (k - 4)) * tpc <= max(256, 1 << (k - 4))


class _FakeLib:
    def __init__(self):
        self.calls = []

    def vfhe_cuda_ntt_set_schedule(self, lp, b, tb, tpc, cps):
        self.calls.append((lp, b, tb, tpc, cps))
        return 0

    def vfhe_cuda_clear_error(self):
        pass


class _FakeEngine:
    def __init__(self):
        self.lib = _FakeLib()


def test_apply_fills_every_bucket_with_the_nearest_entry(tmp_path):
    from vfhe_b200 import autotune

    table = {"14/7": {"schedule": [13, 0, 0]}, "14/13": {"schedule": [12, 1, 2]}, "10/9": {"schedule": [10, 2, 0]}}
    eng = _FakeEngine()
    assert autotune.apply(eng, table) == 64
    got = {(lp, b): (tb, tpc, cps) for lp, b, tb, tpc, cps in eng.lib.calls}
    assert got[(14, 0)] == (13, 0, 0) and got[(14, 10)] == (13, 0, 0)  # ties go to the smaller bucket
    assert got[(14, 11)] == (12, 1, 2) and got[(14, 31)] == (12, 1, 2)
    assert all(got[(10, b)] == (10, 2, 0) for b in range(32))

    p = tmp_path / "t.json"
    p.write_text(json.dumps({"table": table}))
    assert autotune.load(p) == table
    assert autotune.load(tmp_path / "missing.json") is None


def test_dataflow_candidates_cover_the_two_pass_sizes():
    from vfhe_b200.autotune import candidates

    flows = {logP: sorted({k for k, _, cps in candidates(logP) if cps == -2}) for logP in range(8, 18)}
    assert flows[12] == [10] and flows[13] == [10, 11] and flows[14] == [10, 11, 12]
    assert flows[16] == [12, 13] and flows[17] == [13]
    assert all(not flows[lp] for lp in range(8, 12))


def test_a_class_is_timed_over_its_range():
    from vfhe_b200.autotune import BUCKETS, row_counts

    for b in BUCKETS:
        counts = row_counts(b)
        assert len(counts) in (3, 4) and all(c >> b == 1 and c % 3 == 0 for c in counts)
        assert any(c % 2 for c in counts) and any(c % (1 << (b - 1)) == 0 for c in counts)
        assert counts[-1] > 1.7 * (1 << b)


def test_choice_holds_over_every_row_count():
    """A schedule that is fast at the class's power of two and twice as slow at an odd count
    loses to one that is a little faster everywhere; less than 1% keeps the built-in one."""
    from vfhe_b200.autotune import choose

    default, peaky, steady = (9, 0, 0), (9, 4, 2), (9, 2, 0)
    timed = [{default: 1.0, peaky: 0.8, steady: 0.95}, {default: 1.3, peaky: 2.6, steady: 1.2},
             {default: 1.9, peaky: 1.7, steady: 1.8}]
    assert choose(timed, default)[0] == steady
    assert choose([{default: 1.0, steady: 0.995}], default) == (default, 1.0, 1.0)
    assert choose([{peaky: 2.0, steady: 1.0}], default) == (steady, 1.0, None)
