"""Batched CGGI16 bootstrap (vfhe_cuda_cggi_bootstrap_batch) against the reference API
path (CGGI16.functional_bootstrap over mgsw_CMUX), bit for bit, and LUT correctness."""

from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _setup(cuda, N, n_lwe, count, seed, msg_prec=5):
    from vfhe_b200.arith import Ring
    from vfhe_b200.fhe import CGGI16
    from vfhe_b200.mlwe import LWE_Key, MLWE_Scheme, encrypt_lwe
    from vfhe_b200.native import use_engine

    with use_engine(cuda):
        rng = np.random.default_rng(seed)
        Rq = Ring(N, prime_size=[50, 50, 50], split_degree=1)
        in_ring = Rq.quotient_ring(ell=2)
        s = MLWE_Scheme(Rq, special_primes=1, module_rank=1, max_lvl=1)
        in_key_s = [int(v) for v in rng.integers(0, 2, n_lwe)]
        in_key = LWE_Key(ring=in_ring, key=in_key_s, n=n_lwe)
        out_key = s.key_gen_sparse(64, 3.2, ternary=False, rng=rng)
        cg = CGGI16(s)
        bk = cg.generate_bootstrap_key(in_key, out_key, rng=rng)
        t = 1 << (msg_prec - 1)
        lut = [int(v) for v in rng.integers(0, t, t)]
        tv = cg.LUT_packing(lut, t, msg_prec)
        msgs = [int(v) for v in rng.integers(0, t, count)]
        lwes = []
        for m in msgs:
            scaled = round(m * in_ring.q_l / (1 << msg_prec)) % in_ring.q_l
            lwes.append(encrypt_lwe(in_ring, in_key_s, [scaled % q for q in in_ring.primes], 3.2, rng))
        ok = out_key.extract_lwe_key()
        key2 = LWE_Key(ring=in_ring, key=ok.get_s(), n=ok.n)
        return s, cg, bk, tv, lwes, msgs, lut, t, in_ring, key2


@pytest.mark.parametrize("N,n_lwe,count", [(256, 16, 4), (1024, 64, 8)])
def test_batched_bootstrap_matches_reference_path(cuda, N, n_lwe, count):
    import torch

    from vfhe_b200.batch import CggiBatch, bootstrap_key_tensor, to_device, to_host
    from vfhe_b200.mlwe import LWE

    s, cg, bk, tv, lwes, msgs, lut, t, in_ring, key2 = _setup(cuda, N, n_lwe, count, seed=N + n_lwe)
    ref_a, ref_b = [], []
    for lwe in lwes:
        out = LWE(ring=in_ring)
        cg.functional_bootstrap(out, tv, lwe, bk, torus_base=t)
        ref_a.append(np.array(out.get_a(), dtype=np.uint64))
        ref_b.append(np.array(out.get_b(), dtype=np.uint64))

    a = to_device(np.stack([np.array(l.get_a(), dtype=np.uint64) for l in lwes]))
    b = to_device(np.stack([np.array(l.get_b(), dtype=np.uint64) for l in lwes]))
    tv.to_coeff()
    tvt = to_device(np.stack([tv.component_rows(0), tv.component_rows(1)]))
    oa, ob = CggiBatch(s).bootstrap(a, b, bootstrap_key_tensor(bk), tvt, t)
    torch.cuda.synchronize()
    assert np.array_equal(to_host(oa), np.stack(ref_a))
    assert np.array_equal(to_host(ob), np.stack(ref_b))

    # decryption of the batched outputs
    for i, m in enumerate(msgs):
        o = LWE(ring=in_ring, n=N)
        o.set_rows(to_host(oa)[i], to_host(ob)[i])
        ph = o.phase(key2, recompose=True)
        assert round(ph * (2 * t) / in_ring.q_l) % (2 * t) == lut[m]


@pytest.mark.parametrize("N,L0", [(256, 1), (256, 2), (512, 1), (512, 2), (1024, 1), (1024, 2), (2048, 2), (4096, 1)])
def test_fused_forms_match_one_launch_per_stage(cuda, N, L0):
    """A key off the 16-byte boundary takes one launch per stage.  The same key on it takes
    whole rotations on clusters for a few LWEs (N <= 2048) and one launch per step for many
    (512 <= N): the same residues from uniform keys, ciphertexts and test vectors."""
    import torch

    from vfhe_b200.arith import Ring

    n, few, many, t = 9, 3, 150, 16
    R = Ring(N, prime_size=[50] * (L0 + 1), split_degree=1, engine=cuda)
    q, limbs = R.primes, cuda.ffi.new("uint32_t[]", R.prime_indices[:L0])
    gen = torch.Generator(device="cuda")
    gen.manual_seed(N + L0)

    def uniform(shape, axis, primes):
        x = torch.empty(shape, dtype=torch.int64, device="cuda")
        for k, p in enumerate(primes):
            x.select(axis, k).random_(0, p, generator=gen)
        return x

    a, b = uniform((many, L0, n), 1, q[:L0]), uniform((many, L0), 1, q[:L0])
    a[1] = 0  # rotations by zero
    bk, tv = uniform((n, 2 * L0, 2, L0 + 1, N), 3, q), uniform((2, L0, N), 1, q[:L0])
    off = torch.empty(bk.numel() + 1, dtype=torch.int64, device="cuda")
    off[1:] = bk.flatten()

    def run(count, key_ptr):
        oa = torch.empty((count, L0, N), dtype=torch.int64, device="cuda")
        ob = torch.empty((count, L0), dtype=torch.int64, device="cuda")
        ws = torch.empty(cuda.lib.vfhe_cuda_cggi_workspace_bytes(R.NTT, count, n, L0) // 8 + 1, dtype=torch.int64,
                         device="cuda")
        p = lambda x: cuda.ffi.cast("uint64_t*", x.data_ptr())  # noqa: E731
        rc = cuda.lib.vfhe_cuda_cggi_bootstrap_batch(
            R.NTT, p(oa), p(ob), p(a), p(b), count, n, limbs, L0, R.prime_indices[L0],
            cuda.ffi.cast("uint64_t*", key_ptr), p(tv), t, cuda.ffi.cast("void*", ws.data_ptr()),
            cuda.ffi.cast("void*", torch.cuda.current_stream().cuda_stream))
        cuda.check("bootstrap")
        assert rc == 0
        torch.cuda.synchronize()
        return oa, ob

    assert bk.data_ptr() % 16 == 0 and off.data_ptr() % 16 == 0
    want_a, want_b = run(many, off.data_ptr() + 8)
    for count in (few, many):
        oa, ob = run(count, bk.data_ptr())
        assert torch.equal(oa, want_a[:count]) and torch.equal(ob, want_b[:count])
