"""FP64 transforms at the edges of their tile and column kernels' rules: rows on 16 but not 32
bytes (the narrow form of the edge pass's accesses), and row counts on both sides of a rule,
against the CPU oracle."""

from __future__ import annotations

import numpy as np
import pytest

from .helpers import twin_rings

pytestmark = pytest.mark.gpu


def _check(cuda, oracle_engine, log_p: int, rows: int, schedule, offset: int, in_place: bool) -> None:
    import torch

    from vfhe_b200.arith import Polynomial, repr as domain

    N = 1 << log_p
    ring, ref = twin_rings([cuda, oracle_engine], N, [50], 1)
    lib, ffi = cuda.lib, cuda.ffi
    rng = np.random.default_rng(log_p * 1000 + rows)
    q = ring.primes[0]
    x = rng.integers(0, q, (rows, N), dtype=np.uint64)
    x[0, :], x[-1, ::2] = q - 1, 0
    limbs = ffi.new("uint32_t[]", ring.prime_indices)
    st = ffi.cast("void*", torch.cuda.current_stream().cuda_stream)
    bucket, old = min(15, rows.bit_length() - 1), ffi.new("int32_t[3]")
    lib.vfhe_cuda_ntt_get_schedule(log_p, rows, old)
    assert lib.vfhe_cuda_ntt_set_schedule(log_p, bucket, *schedule) == 0
    sample = sorted({0, rows // 2, rows - 1})
    try:
        for inverse in (0, 1):
            buf = torch.empty(rows * N + offset, dtype=torch.int64, device="cuda")[offset:]
            out = buf if in_place else torch.empty(rows * N + offset, dtype=torch.int64, device="cuda")[offset:]
            assert buf.data_ptr() % 32 == (16 if offset else 0)
            buf.copy_(torch.from_numpy(x.view(np.int64).reshape(-1)))
            assert lib.vfhe_cuda_ntt_batch(ring.NTT, inverse, ffi.cast("uint64_t*", out.data_ptr()),
                                           ffi.cast("uint64_t*", buf.data_ptr()), rows, limbs, 1, st) == 0
            got = out.cpu().numpy().view(np.uint64).reshape(rows, N)
            for r in sample:
                p = Polynomial(ref)
                p.set_rows(x[r:r + 1])
                p.repr = domain.ntt if inverse else domain.coeff
                p.to_coeff() if inverse else p.to_NTT()
                assert np.array_equal(got[r], p.rows()[0]), (inverse, r)
    finally:
        lib.vfhe_cuda_ntt_set_schedule(log_p, bucket, *list(old))


@pytest.mark.parametrize("log_p,schedule", [(8, (8, 0, 0)), (9, (9, 2, 0)), (10, (10, 1, 0)), (11, (11, 1, 0)),
                                            (12, (12, 1, 0)), (13, (13, 1, 0)), (14, (10, 1, 0)), (14, (11, 0, -1)),
                                            (15, (12, 0, -1)), (15, (13, 0, -1)), (12, (12, 1, 1)), (13, (12, 1, 0))])
@pytest.mark.parametrize("in_place", [True, False])
def test_rows_on_16_bytes(cuda, oracle_engine, log_p, schedule, in_place):
    _check(cuda, oracle_engine, log_p, 37, schedule, 2, in_place)


@pytest.mark.parametrize("log_p,tile,rows", [(9, 8, 5), (11, 10, 3), (13, 12, 1), (13, 11, 3), (14, 13, 3)])
def test_short_column_passes(cuda, oracle_engine, log_p, tile, rows):
    """Column passes of two and four points, in CTAs of 128 and 64 threads."""
    _check(cuda, oracle_engine, log_p, rows, (tile, 0, 0), 0, True)


@pytest.mark.parametrize("log_p,tile", [(9, 9), (10, 10), (11, 11), (12, 12), (13, 11), (14, 13)])
@pytest.mark.parametrize("side", [0, 1])
def test_inverse_forms(cuda, oracle_engine, log_p, tile, side):
    """Tile counts on both sides of the inverse kernels' rule: one CTA's threads an SM at 2^10
    and 2^11, four tiles an SM at 2^12."""
    import torch

    sms = torch.cuda.get_device_properties(0).multi_processor_count
    tiles = {9: 8 * sms, 10: 4 * sms, 11: 2 * sms, 12: 4 * sms, 13: sms}[tile]
    _check(cuda, oracle_engine, log_p, (tiles >> (log_p - tile)) + side, (tile, 1, 0), 0, False)
