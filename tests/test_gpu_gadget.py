"""The one-call key switch and multiply with every digit at once (abi_mlwe.cu): against the
batched key switch where the digits' scratch takes several rounds, and against the oracle
on pools whose active limbs are not neighbours and at every split's product form."""

from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("logn,L", [(8, 1), (12, 2), (13, 5), (15, 20)])
def test_one_call_key_switch_matches_batched(cuda, logn, L):
    """N = 2^15 with 20 limbs has 110 MB of digit spectra: two rounds of the 64 MB scratch."""
    import torch

    from vfhe_b200.worklist import per_call_workspace, run_job_on_engine, run_per_call, uneven_jobs

    seed = next(s for s in range(100) if uneven_jobs_kind(s) == "keyswitch")
    jobs = [j for j in uneven_jobs(cuda, 1, seed=seed, logn=(logn, logn), limbs=(L, L))]
    assert jobs[0].kind == "keyswitch"
    out = torch.empty_like(jobs[0].out)
    run_per_call(cuda, jobs, [out], per_call_workspace(cuda, jobs))
    torch.cuda.synchronize()
    got = run_job_on_engine(cuda, jobs[0])
    assert np.array_equal(got, out.cpu().numpy().view(np.uint64))


def uneven_jobs_kind(seed: int) -> str:
    rng = np.random.default_rng(seed)
    rng.integers(0, 1), rng.integers(0, 1)
    return "chain" if rng.random() < 0.5 else "keyswitch"


@pytest.mark.parametrize("N,split,rank", [(2**9, 1, 1), (2**10, 2, 1), (2**11, 4, 2), (2**10, 1, 3)])
def test_limbs_with_gaps_match_the_oracle(cuda, oracle_engine, N, split, rank):
    """Ciphertext limbs at pool rows 0, 2, 3 and 5 and the special prime at 1: the digits are
    not evenly spaced and the rows between are inactive."""
    from vfhe_b200.arith import Ring, repr as domain
    from vfhe_b200.mlwe import MLWE, MLWE_Scheme, MLWE_Set
    from vfhe_b200.native import use_engine

    outs = []
    for eng in (cuda, oracle_engine):
        with use_engine(eng):
            rng = np.random.default_rng(N + rank)
            q = Ring(N, prime_size=[50, 45, 40, 42, 44, 41], split_degree=split).primes
            lims, special = [q[0], q[2], q[3], q[5]], q[1]

            def ring(primes):
                return Ring(N, prime_size=[int(p).bit_length() for p in primes], primes=primes, split_degree=split)

            s = MLWE_Scheme([ring(lims)], special_rings=[ring(lims + [special])], module_rank=rank)

            def sample(r):
                m = MLWE(s, ring=r)
                for c in range(rank + 1):
                    m.set_component_rows(c, np.stack([rng.integers(0, p, N, dtype=np.uint64) for p in r.primes]))
                m.repr = domain.ntt
                return m

            key = MLWE_Set([[sample(s.special_rings[0]) for _ in lims] for _ in range(rank)])
            ct = sample(s.rings[0])
            sw = s.keyswitch(ct, key)
            rlk = MLWE_Set([[sample(s.special_rings[0]) for _ in lims] for _ in range(rank * (rank + 1) // 2)]
                           + [None] * rank)
            prod = s.multiply(sample(s.rings[0]), sample(s.rings[0]), rlk)
            outs.append([np.stack([m.component_rows(c) for c in range(rank + 1)]) for m in (sw, prod)])
    for got, want in zip(*outs):
        assert np.array_equal(got, want)


@pytest.mark.parametrize("split", [1, 2])
def test_digit_of_a_large_prime_outside_the_key(cuda, oracle_engine, split):
    """A ciphertext limb of a 58-bit prime, whose digit is no double, under a key without that
    limb: the external product still equals the oracle's."""
    from vfhe_b200.arith import Ring, repr as domain
    from vfhe_b200.mlwe import MLWE, MLWE_Scheme
    from vfhe_b200.native import use_engine

    N, outs = 2**9, []
    for eng in (cuda, oracle_engine):
        with use_engine(eng):
            rng = np.random.default_rng(split)
            q = Ring(N, prime_size=[50, 45, 58, 40], split_degree=split).primes
            lims, key_lims = [q[0], q[2], q[3]], [q[0], q[1], q[3]]

            def ring(primes):
                return Ring(N, prime_size=[int(p).bit_length() for p in primes], primes=primes, split_degree=split)

            s = MLWE_Scheme([ring(lims)], special_rings=[ring(key_lims)], module_rank=1)

            def sample(r):
                m = MLWE(s, ring=r)
                for c in range(2):
                    m.set_component_rows(c, np.stack([rng.integers(0, p, N, dtype=np.uint64) for p in r.primes]))
                return m

            rows = [sample(s.special_rings[0]) for _ in range(6)]
            ct, out = sample(s.rings[0]), MLWE(s, ring=s.special_rings[0])
            ct.repr = domain.coeff
            eng.lib.mgsw_external_product(out.obj, eng.ffi.new("void*[]", [r.obj for r in rows]), ct.obj, 3, 0)
            eng.check("mgsw_external_product")
            outs.append(np.stack([out.component_rows(c) for c in range(2)]))
    assert np.array_equal(*outs)
