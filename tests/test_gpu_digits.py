"""All key-switch digits in one transform launch (digit mode of a row set, ckks.cu): the
batched multiply (which leaves out the digits' own primes), rotation and key switch equal
the one-op-per-call path at the smallest and largest limb counts and ring sizes of each
transform schedule, odd batches and split degrees."""

from __future__ import annotations

import numpy as np
import pytest

from tests.test_gpu_batch import _setup

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("N,n_mid,split,pairs", [(2**9, 1, 1, 1), (2**11, 1, 2, 3), (2**13, 1, 1, 1), (2**13, 4, 4, 5),
                                                 (2**15, 2, 1, 3), (2**16, 1, 1, 2)])
def test_digits_in_one_launch_match_single_calls(cuda, N, n_mid, split, pairs):
    import torch

    from vfhe_b200.batch import CkksBatch, ciphertext_rows, key_tensor, to_device, to_host

    s, key, rlk, gks, cts = _setup(cuda, N, n_mid, 2 * pairs, [2], seed=N + pairs, split=split)
    c1, c2 = cts[0::2], cts[1::2]
    ref_prod, ref_rot = [], []
    for a, b in zip(c1, c2):
        p = s.multiply(a, b, rlk)
        p.round_division(lvl=1)
        ref_prod.append(ciphertext_rows(p))
        ref_rot.append(ciphertext_rows(s.automorphism(p, s.galois_gen(2), gks[2])))
    for c in cts:
        c.to_NTT()
    t1 = to_device(np.stack([ciphertext_rows(c) for c in c1]))
    t2 = to_device(np.stack([ciphertext_rows(c) for c in c2]))
    special = s.special_rings[0].prime_indices[-1]
    out = CkksBatch(s.rings[0], special).mul_relin_rescale(t1, t2, key_tensor(rlk))
    gk = key_tensor(gks[2])
    rot = CkksBatch(s.rings[1], special).rotate(out, [s.galois_gen(2)] * pairs, [gk] * pairs)
    torch.cuda.synchronize()
    assert np.array_equal(to_host(out), np.stack(ref_prod))
    assert np.array_equal(to_host(rot), np.stack(ref_rot))
