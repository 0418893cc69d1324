"""Reading a polynomial's rows: into an array the caller gives, on both engines, and through
vfhe_cuda_poly_read_rows."""

from __future__ import annotations

import numpy as np
import pytest

N, SIZES = 64, [50, 40, 45]


def _poly(engine):
    from vfhe_b200.arith import Polynomial, Ring

    ring = Ring(N, prime_size=SIZES, split_degree=1, engine=engine)
    p = Polynomial(ring)
    rng = np.random.default_rng(3)
    rows = np.stack([rng.integers(0, q, N, dtype=np.uint64) for q in ring.primes])
    p.set_rows(rows)
    return p, rows


def _given_arrays(engine):
    p, rows = _poly(engine)
    out = np.zeros((len(SIZES) + 1, N), dtype=np.uint64)
    assert p.rows(out) is out
    assert np.array_equal(out[:-1], rows) and not out[-1].any()
    signed = np.zeros((len(SIZES), N), dtype=np.int64)
    assert np.array_equal(p.rows(signed).view(np.uint64), rows)
    locked = np.zeros((len(SIZES), N), dtype=np.uint64)
    locked.flags.writeable = False
    for bad in (np.zeros((len(SIZES) - 1, N), dtype=np.uint64), np.zeros(len(SIZES) * N - 1, dtype=np.uint64),
                np.zeros((len(SIZES), 2 * N), dtype=np.uint64)[:, ::2], np.zeros((len(SIZES), N), dtype=np.uint32),
                locked):
        with pytest.raises(ValueError):
            p.rows(bad)
        assert not bad.any()


def test_rows_into_a_given_array(oracle_engine):
    _given_arrays(oracle_engine)


@pytest.mark.gpu
def test_rows_into_a_given_array_cuda(cuda):
    _given_arrays(cuda)


@pytest.mark.gpu
@pytest.mark.parametrize("rows", [[0, 1, 2], [0, 2], [2, 1, 0], [1, 2], [0, 1, 1, 2], [2], []])
def test_read_rows_over_gaps_and_runs(cuda, rows):
    """Runs of neighbouring rows go in one copy; any order, gaps and repeats give the same rows."""
    p, want = _poly(cuda)
    idx = [p.ring.prime_indices[k] for k in rows]
    out = np.zeros((len(rows) + 1, N), dtype=np.uint64)
    assert cuda.lib.vfhe_cuda_poly_read_rows(p.obj, cuda.ffi.from_buffer("uint64_t[]", out),
                                             cuda.ffi.new("uint32_t[]", idx), len(idx)) == 0
    assert np.array_equal(out[:-1], want[rows]) and not out[-1].any()


@pytest.mark.gpu
def test_read_rows_refusals(cuda):
    p, _ = _poly(cuda)
    lib, ffi = cuda.lib, cuda.ffi
    out = np.zeros((2, N), dtype=np.uint64)
    buf, one = ffi.from_buffer("uint64_t[]", out), ffi.new("uint32_t[]", [p.ring.prime_indices[0]])
    outside = ffi.new("uint32_t[]", [p.ring.prime_indices[0], 63])
    for args, what in (((p.obj, buf, outside, 2), "row outside"), ((p.obj, ffi.NULL, one, 1), "null"),
                       ((p.obj, buf, ffi.NULL, 1), "null"), ((ffi.NULL, buf, one, 1), "")):
        assert lib.vfhe_cuda_poly_read_rows(*args) != 0
        assert what in ffi.string(lib.vfhe_cuda_last_error()).decode()
        lib.vfhe_cuda_clear_error()
    assert not out.any()
    assert lib.vfhe_cuda_poly_read_rows(p.obj, ffi.NULL, ffi.NULL, 0) == 0  # nothing asked for


@pytest.mark.gpu
def test_read_rows_follow_the_row_pointers(cuda):
    """Rows whose pointers the caller has exchanged are read where the pointers say."""
    p, want = _poly(cuda)
    c = cuda.ffi.cast("RNS_Polynomial", p.obj).coeffs
    i, j = p.ring.prime_indices[0], p.ring.prime_indices[2]
    c[i], c[j] = c[j], c[i]
    got, seen = p.rows(), np.stack([p.row(k).copy() for k in p.ring.prime_indices])
    c[i], c[j] = c[j], c[i]
    assert np.array_equal(got, seen) and np.array_equal(got, want[[2, 1, 0]])
