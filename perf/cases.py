"""Timed workloads of the cuda engine, each through the entry point a program calls.

The listed cases cover the engine's use: batched CKKS evaluation from one small
ciphertext to the largest parameters, the RNS transforms in both directions, the fused
ring product, both CGGI16 bootstraps at a few and at thousands of ciphertexts, the uneven
work list, and the one-operation-per-call surface.  ``draw`` gives more cases of the same
ranges.

Residues are uniform in [0, q): what ciphertexts, transformed polynomials and evaluation
keys of these schemes look like.  Torus keys and ciphertexts are real ones.
"""

from __future__ import annotations

import math

import numpy as np
import torch

from vfhe_b200.arith import Ring, repr as domain
from vfhe_b200.batch import CggiBatch, CkksBatch, ciphertext_rows
from vfhe_b200.cggi_fft import CggiFft, TorusParams, generate_device_keys
from vfhe_b200.cggi_fft import test_vector as lookup_vector
from vfhe_b200.cggi_fft import to_device as torus_to_device
from vfhe_b200.fhe import CKKS_Scheme
from vfhe_b200.mlwe import MLWE, MLWE_Scheme, MLWE_Set
from vfhe_b200.native import cuda_engine
from vfhe_b200.worklist import Job, WorkList

# Rotations are drawn from the steps 1, 2, 4, ..., 2^12 (a program keeps one Galois key
# for each), so a batch reads at most this many keys.
ROTATION_STEPS = 13


def listed() -> list[dict]:
    return [
        # An interactive request: one ciphertext pair at the smallest served parameters.
        # Launches and latency count, not bandwidth.
        {"name": "ckks_mul_single", "kind": "ckks_mul", "log_n": 13, "limbs": 4, "batch": 1},
        # The CKKS arithmetic benchmark: 256 pairs at N = 2^14, one 50-bit and eight 40-bit
        # primes.
        {"name": "ckks_mul_256", "kind": "ckks_mul", "log_n": 14, "limbs": 9, "batch": 256},
        # Rotations at the largest served parameters, an odd batch over several Galois keys.
        {"name": "ckks_rotate_deep", "kind": "ckks_rotate", "log_n": 16, "limbs": 24, "batch": 3},
        # The transform throughput benchmark: 64 polynomials of 24 limbs, N = 2^16, at the
        # default split degree of 50-bit primes.
        {"name": "ntt_forward_deep", "kind": "ntt", "log_n": 16, "limbs": 24, "batch": 64, "split": 4,
         "inverse": False},
        # Results leaving the transform domain: an odd number of polynomials and limbs.
        {"name": "ntt_inverse_odd", "kind": "ntt", "log_n": 14, "limbs": 11, "batch": 29, "split": 1,
         "inverse": True},
        # The plain RNS round trip: 64 pairs, N = 4096, L = 3, transform, product, inverse.
        {"name": "ring_product_64", "kind": "ring_product", "log_n": 12, "limbs": 3, "batch": 64, "split": 4},
        # RNS-gadget CGGI16 bootstraps: a request with a few ciphertexts, and the largest
        # request the serving loop admits.
        {"name": "rns_bootstrap_few", "kind": "rns_bootstrap", "lwe_dim": 630, "batch": 3},
        {"name": "rns_bootstrap_1024", "kind": "rns_bootstrap", "lwe_dim": 630, "batch": 1024},
        # Torus CGGI16 bootstraps (blind rotation and key switch): a few ciphertexts, and the
        # 4096 of the bootstrap benchmark.
        {"name": "torus_bootstrap_few", "kind": "torus_bootstrap", "log_n": 10, "lwe_dim": 630, "batch": 7},
        {"name": "torus_bootstrap_4096", "kind": "torus_bootstrap", "log_n": 10, "lwe_dim": 630, "batch": 4096},
        # The uneven workload: ring products and key switches, N from 2^12 to 2^16 and L from
        # 2 to 24, run together.
        {"name": "uneven_64", "kind": "worklist", "jobs": 64, "shapes": 3},
        # One ciphertext product and rotation through the one-operation-per-call surface, as
        # the library's unchanged callers run it, and the result read on the host.
        {"name": "one_call_per_op", "kind": "one_call", "log_n": 14, "limbs": 9},
    ]


def draw(rng) -> dict:
    kind = rng.choice(["ckks_mul", "ckks_rotate", "ntt", "ring_product", "rns_bootstrap", "torus_bootstrap",
                       "worklist", "one_call"])

    def spread(low: int, high: int) -> int:
        return max(low, min(high, int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))))

    if kind in ("ckks_mul", "ckks_rotate"):
        log_n, limbs = rng.randint(13, 16), rng.randint(4, 24)
        most = (256 * 9 * 10 << 14) // (limbs * (limbs + 1) << log_n)
        return {"kind": kind, "log_n": log_n, "limbs": limbs, "batch": spread(1, max(1, min(256, most)))}
    if kind == "ntt":
        log_n, limbs = rng.randint(12, 16), rng.randint(1, 24)
        most = (64 * 24 << 16) // (limbs << log_n)
        return {"kind": kind, "log_n": log_n, "limbs": limbs, "batch": spread(1, max(1, min(512, most))),
                "split": rng.choice([1, 4]), "inverse": rng.random() < 0.5}
    if kind == "ring_product":
        return {"kind": kind, "log_n": rng.randint(11, 14), "limbs": rng.randint(1, 6), "batch": spread(1, 256),
                "split": rng.choice([1, 2, 4])}
    if kind == "rns_bootstrap":
        return {"kind": kind, "lwe_dim": rng.randint(64, 630), "batch": spread(1, 1024)}
    if kind == "torus_bootstrap":
        log_n = rng.choice([9, 10, 10, 11])
        return {"kind": kind, "log_n": log_n, "lwe_dim": rng.randint(64, 630),
                "batch": spread(1, 4096 >> max(0, log_n - 10))}
    if kind == "worklist":
        return {"kind": kind, "jobs": spread(8, 64), "shapes": rng.randint(10, 10**6)}
    return {"kind": kind, "log_n": rng.randint(12, 15), "limbs": rng.randint(3, 12)}


# ---- inputs


def _generator(seed: int) -> torch.Generator:
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    return g


def _uniform(gen: torch.Generator, shape: tuple, axis: int, primes: list[int]) -> torch.Tensor:
    """Residues uniform in [0, q), q the prime at the index along `axis`."""
    t = torch.empty(shape, dtype=torch.int64, device="cuda")
    for k, q in enumerate(primes):
        t.select(axis, k).random_(0, int(q), generator=gen)
    return t


def _host_uniform(gen: torch.Generator, primes: list[int], n: int) -> np.ndarray:
    return _uniform(gen, (len(primes), n), 0, primes).cpu().numpy().view(np.uint64)


def _pointer(eng, t: torch.Tensor):
    return eng.ffi.cast("uint64_t*", t.data_ptr())


def _stream(eng):
    return eng.ffi.cast("void*", torch.cuda.current_stream().cuda_stream)


def _ckks_ring(log_n: int, limbs: int) -> Ring:
    """`limbs` ciphertext primes (one of 50 bits, the others of 40) and one special prime."""
    return Ring(1 << log_n, prime_size=[50] + [40] * (limbs - 1) + [50], split_degree=1)


def _prepare_ckks(case: dict, seed: int) -> dict:
    n, L, B = 1 << case["log_n"], case["limbs"], case["batch"]
    ring = _ckks_ring(case["log_n"], L)
    level = ring.quotient_ring(ell=L)
    gen = _generator(seed)
    q = list(ring.primes)
    st = {"batch": CkksBatch(level, ring.prime_indices[-1]), "kind": case["kind"]}
    if case["kind"] == "ckks_mul":
        st["ct1"] = _uniform(gen, (B, 2, L, n), 2, q[:L])
        st["ct2"] = _uniform(gen, (B, 2, L, n), 2, q[:L])
        st["rlk"] = _uniform(gen, (L, 2, L + 1, n), 2, q)
        return st
    st["ct"] = _uniform(gen, (B, 2, L, n), 2, q[:L])
    steps = np.random.default_rng(seed).integers(0, ROTATION_STEPS, B)
    keys = {int(s): _uniform(gen, (L, 2, L + 1, n), 2, q) for s in np.unique(steps)}
    st["gens"] = [pow(5, 1 << int(s), 2 * n) for s in steps]
    st["keys"] = [keys[int(s)] for s in steps]
    return st


def _prepare_ntt(case: dict, seed: int) -> dict:
    n, L, B = 1 << case["log_n"], case["limbs"], case["batch"]
    eng = cuda_engine()
    ring = Ring(n, prime_size=[50] * L, split_degree=case["split"])
    return {"kind": case["kind"], "eng": eng, "ring": ring, "limbs": eng.ffi.new("uint32_t[]", ring.prime_indices),
            "L": L, "B": B, "inverse": int(case["inverse"]),
            "x": _uniform(_generator(seed), (B, L, n), 1, ring.primes)}


def _prepare_ring_product(case: dict, seed: int) -> dict:
    n, L, B = 1 << case["log_n"], case["limbs"], case["batch"]
    eng = cuda_engine()
    ring = Ring(n, prime_size=[50] * L, split_degree=case["split"])
    gen = _generator(seed)
    return {"kind": case["kind"], "eng": eng, "ring": ring, "limbs": eng.ffi.new("uint32_t[]", ring.prime_indices),
            "L": L, "B": B, "a": _uniform(gen, (B, L, n), 1, ring.primes),
            "b": _uniform(gen, (B, L, n), 1, ring.primes)}


RNS_N, RNS_L, RNS_TABLE = 1024, 2, 16


def _prepare_rns_bootstrap(case: dict, seed: int) -> dict:
    n, B = case["lwe_dim"], case["batch"]
    ring = Ring(RNS_N, prime_size=[50] * (RNS_L + 1), split_degree=1)
    scheme = MLWE_Scheme(ring, special_primes=1, module_rank=1, max_lvl=1)
    gen = _generator(seed)
    q = list(ring.primes)
    tv = torch.zeros((2, RNS_L, RNS_N), dtype=torch.int64, device="cuda")
    lut = np.random.default_rng(seed).integers(0, RNS_TABLE, RNS_TABLE)
    Q = math.prod(int(p) for p in q[:RNS_L])
    for k in range(RNS_L):
        row = [(int(lut[j * RNS_TABLE // RNS_N]) * Q // (2 * RNS_TABLE)) % int(q[k]) for j in range(RNS_N)]
        tv[1, k] = torch.tensor(row, dtype=torch.int64)
    return {"kind": case["kind"], "cggi": CggiBatch(scheme),
            "a": _uniform(gen, (B, RNS_L, n), 1, q[:RNS_L]), "b": _uniform(gen, (B, RNS_L), 1, q[:RNS_L]),
            "bk": _uniform(gen, (n, 2 * RNS_L, 2, RNS_L + 1, RNS_N), 3, q), "tv": tv}


def _prepare_torus_bootstrap(case: dict, seed: int) -> dict:
    params = TorusParams(n=case["lwe_dim"], N=1 << case["log_n"])
    eng = cuda_engine()
    rng = np.random.default_rng(seed)
    eng.lib.vfhe_prng_set_deterministic_seed(seed)
    keys = generate_device_keys(params, rng)
    dev = CggiFft(keys)
    eng.lib.vfhe_prng_clear_deterministic_seed()
    lut = rng.integers(0, params.t, params.t)
    lwe = keys.encrypt(rng.integers(0, params.t, case["batch"]), rng)
    return {"kind": case["kind"], "cggi": dev, "lwe": torus_to_device(lwe),
            "tv": torus_to_device(lookup_vector(lut, params))}


def _job_shapes(case: dict) -> list[tuple[str, int, int]]:
    """(kind, N, L) of every job: N uniform over 2^12..2^16, L over 2..24, half of each kind."""
    rng = np.random.default_rng(case["shapes"])
    return [("chain" if rng.random() < 0.5 else "keyswitch", 1 << int(rng.integers(12, 17)), int(rng.integers(2, 25)))
            for _ in range(case["jobs"])]


def _prepare_worklist(case: dict, seed: int) -> dict:
    shapes = _job_shapes(case)
    gen = _generator(seed)
    rings = {n: Ring(n, prime_size=[50] * 25) for n in sorted({n for _, n, _ in shapes})}
    sizes = [(1 if kind == "chain" else 2) * L * n for kind, n, L in shapes]
    out = torch.empty(sum(sizes), dtype=torch.int64, device="cuda")
    wl, at = WorkList(), 0
    for (kind, n, L), size in zip(shapes, sizes):
        ring, q = rings[n], rings[n].primes
        limbs = list(ring.prime_indices[:L])
        o = out[at:at + size]
        at += size
        if kind == "chain":
            wl.add(Job("chain", ring, L, limbs, None, o.view(L, n), _uniform(gen, (L, n), 0, q[:L]),
                       b=_uniform(gen, (L, n), 0, q[:L])))
        else:
            wl.add(Job("keyswitch", ring, L, limbs, ring.prime_indices[L], o.view(2, L, n),
                       _uniform(gen, (2, L, n), 1, q[:L]), ksk=_uniform(gen, (L, 2, L + 1, n), 2, q[:L + 1])))
    wl.compile()
    return {"kind": case["kind"], "wl": wl, "out": out}


def _prepare_one_call(case: dict, seed: int) -> dict:
    n, L = 1 << case["log_n"], case["limbs"]
    q = list(_ckks_ring(case["log_n"], L).primes)

    def level(primes: list[int]) -> Ring:
        return Ring(n, prime_size=[int(p).bit_length() for p in primes], primes=primes, split_degree=1)

    # the two levels the product and the rotation use, and each with the special prime
    scheme = CKKS_Scheme([level(q[:L]), level(q[:L - 1])], scaling_factor=2**40,
                         special_rings=[level(q), level(q[:L - 1] + q[L:])])
    gen = _generator(seed)

    def sample(level_ring: Ring, ciphertext: bool = False) -> MLWE:
        c = scheme.ciphertext_type(scheme) if ciphertext else MLWE(scheme, ring=level_ring)
        for i in range(2):
            c.set_component_rows(i, _host_uniform(gen, level_ring.primes, n))
        c.repr = domain.ntt
        return c

    def key(lvl: int) -> list[MLWE]:
        special = scheme.special_rings[lvl]
        return [sample(special) for _ in range(special.ell - 1)]

    return {"kind": case["kind"], "scheme": scheme, "ct1": sample(scheme.rings[0], True),
            "ct2": sample(scheme.rings[0], True), "rlk": MLWE_Set([key(0), None]), "gk": MLWE_Set([key(1)]),
            "gen": scheme.galois_gen(1)}


_PREPARE = {"ckks_mul": _prepare_ckks, "ckks_rotate": _prepare_ckks, "ntt": _prepare_ntt,
            "ring_product": _prepare_ring_product, "rns_bootstrap": _prepare_rns_bootstrap,
            "torus_bootstrap": _prepare_torus_bootstrap, "worklist": _prepare_worklist,
            "one_call": _prepare_one_call}


def prepare(case: dict, seed: int) -> dict:
    return _PREPARE[case["kind"]](case, seed)


# ---- one pass


def run(st: dict):
    kind = st["kind"]
    if kind == "ckks_mul":
        return st["batch"].mul_relin_rescale(st["ct1"], st["ct2"], st["rlk"])
    if kind == "ckks_rotate":
        return st["batch"].rotate(st["ct"], st["gens"], st["keys"])
    if kind == "ntt":
        eng, x = st["eng"], st["x"]
        out = torch.empty_like(x)
        if eng.lib.vfhe_cuda_ntt_batch(st["ring"].NTT, st["inverse"], _pointer(eng, out), _pointer(eng, x), st["B"],
                                       st["limbs"], st["L"], _stream(eng)) != 0:
            eng.check("ntt_batch")
        return out
    if kind == "ring_product":
        eng, a = st["eng"], st["a"]
        out = torch.empty_like(a)
        if eng.lib.vfhe_cuda_ntt_mul_intt_batch(st["ring"].NTT, _pointer(eng, out), _pointer(eng, a),
                                                _pointer(eng, st["b"]), st["B"], st["limbs"], st["L"],
                                                _stream(eng)) != 0:
            eng.check("ntt_mul_intt_batch")
        return out
    if kind == "rns_bootstrap":
        return st["cggi"].bootstrap(st["a"], st["b"], st["bk"], st["tv"], RNS_TABLE)
    if kind == "torus_bootstrap":
        return st["cggi"].bootstrap(st["lwe"], st["tv"])
    if kind == "worklist":
        st["wl"].run()
        return st["out"]
    s = st["scheme"]
    product = s.multiply(st["ct1"], st["ct2"], st["rlk"])
    product.round_division(lvl=1)
    return ciphertext_rows(s.automorphism(product, st["gen"], st["gk"]))


# ---- what a pass cannot do without


def _transforms(rows: int, n: int, split: int = 1) -> float:
    """Operations of `rows` transforms: log2(n / split) stages of n / 2 butterflies, each a
    modular product, a sum and a difference."""
    return 3.0 * rows * (n / 2) * math.log2(n / split)


def _switch_flops(L: int, n: int, split: int = 1) -> float:
    """A key switch of one L-limb polynomial: L (L + 1) digit transforms, the products with
    both key components, and 2 (L + 1) inverse transforms."""
    return _transforms(L * (L + 1) + 2 * (L + 1), n, split) + 2 * 2.0 * L * (L + 1) * n * split


def work(case: dict) -> dict:
    kind = case["kind"]
    if kind in ("ckks_mul", "ckks_rotate"):
        n, L, B = 1 << case["log_n"], case["limbs"], case["batch"]
        key = 8.0 * L * 2 * (L + 1) * n
        if kind == "ckks_mul":
            return {"bytes": 8.0 * B * n * (4 * L + 2 * (L - 1)) + key,
                    "flops": B * (_switch_flops(L, n) + _transforms(L, n) + 5.0 * L * n)}
        return {"bytes": 8.0 * B * n * 4 * L + key * min(B, ROTATION_STEPS), "flops": B * _switch_flops(L, n)}
    if kind == "ntt":
        n, rows = 1 << case["log_n"], case["limbs"] * case["batch"]
        return {"bytes": 16.0 * rows * n, "flops": _transforms(rows, n, case["split"])}
    if kind == "ring_product":
        n, rows = 1 << case["log_n"], case["limbs"] * case["batch"]
        return {"bytes": 24.0 * rows * n,
                "flops": 3 * _transforms(rows, n, case["split"]) + 2.0 * rows * n * case["split"]}
    if kind == "rns_bootstrap":
        n, B, L, N = case["lwe_dim"], case["batch"], RNS_L, RNS_N
        digits, limbs = 2 * L, L + 1
        step = _transforms(digits * limbs + 2 * limbs, N) + 4.0 * digits * limbs * N
        return {"bytes": 8.0 * (n * digits * 2 * limbs * N + B * (n + 1) * L + 2 * L * N + B * L * (N + 1)),
                "flops": n * B * step}
    if kind == "torus_bootstrap":
        p = TorusParams(n=case["lwe_dim"], N=1 << case["log_n"])
        B, M, rows = case["batch"], p.N // 2, 2 * p.bs_levels
        step = (rows + 2) * 5.0 * M * math.log2(M) + rows * 2 * 8.0 * M
        return {"bytes": 16.0 * p.n * rows * 2 * M + 4.0 * (p.N * p.ks_levels * (p.n + 1) + 2 * B * (p.n + 1)),
                "flops": p.n * B * step + 2.0 * B * p.N * p.ks_levels * (p.n + 1)}
    if kind == "worklist":
        total, flops = 0.0, 0.0
        for job, n, L in _job_shapes(case):
            if job == "chain":
                total += 24.0 * L * n
                flops += 3 * _transforms(L, n, 4) + 8.0 * L * n
            else:
                total += 8.0 * n * (4 * L + L * 2 * (L + 1))
                flops += _switch_flops(L, n, 4)
        return {"bytes": total, "flops": flops}
    n, L = 1 << case["log_n"], case["limbs"]
    keys = 8.0 * n * (L * 2 * (L + 1) + (L - 1) * 2 * L)
    return {"bytes": 8.0 * n * (4 * L + 2 * (L - 1)) + keys,
            "flops": _switch_flops(L, n) + _switch_flops(L - 1, n) + _transforms(L, n)}


def exact(case: dict, seed: int):
    """Every output is a residue or a torus word, a whole number that has to be equal."""
    return None
