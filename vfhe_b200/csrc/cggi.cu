// Batched CGGI16 functional bootstrap with the RNS gadget (the reference's CGGI16:
// modules/fhe/python/src/vfhe/fhe/cggi16.py:46-128 over mgsw_CMUX / mgsw_external_product,
// modules/mlwe/c/src/mgsw.c:6-72).
//
// For every LWE of the batch (all sharing one bootstrapping key):
//   rotations  rot_b = round((b + floor(Q / 4t)) 2N / Q) mod 2N,  a_i' = round(a_i 2N / Q) mod 2N
//              (cggi16.py:56-79; Q = product of the LWE's primes, values by exact CRT)
//   acc        = tv * X^(2N - rot_b)
//   step i     acc = CMUX(acc, acc X^(a_i'), bk_i) = acc + ExtProd(bk_i, acc X^(a_i') - acc)
//   output     sample extraction at coefficient 0 (mlwe.c:40-68)
// ExtProd: digit d = limb l of component c of the difference, lifted to the key's
// extended limbs and transformed; accumulated against bk_i[d]; inverse transform;
// rounded division by the special prime.
// Three forms with the same residues: whole rotations on clusters (small batches), one
// launch per step for the external product and one for the division (k_cggi_step), and one
// launch per stage (rings or keys the fused kernels do not take).
//
// The accumulator stays in the coefficient domain: the reference transforms the CMUX
// output forward (mgsw.c:48,67) and the next step back (cggi16.py:84); both maps are
// exact inverses on canonical residues, so skipping them leaves every bit unchanged.
// A step with a_i' = 0 (skipped by the reference) adds ExtProd(bk_i, 0) = 0 here.
#include <cooperative_groups.h>
#include <cuda_runtime.h>
#include <string.h>

#include <vector>

#include "abi_common.cuh"
#include "fp64mod.cuh"
#include "ntt_f64_r8.cuh"

namespace vc {

namespace {

struct CggiShape {
    uint32_t lwe_prime[4];   // pool indices of the LWE / accumulator limbs (L0 of them)
    uint32_t ext_prime[5];   // extended limbs: lwe_prime then the special prime
    int L0;                  // accumulator limbs
    int n;                   // LWE dimension
    long long N;
};

__device__ __forceinline__ unsigned __int128 crt2(uint64_t r0, uint64_t r1, uint64_t q0, uint64_t q1,
                                                   uint64_t q0inv_mod_q1, const PrimeInfo& p1) {
    // v = r0 + q0 * ((r1 - r0) * q0^-1 mod q1)
    const uint64_t d = sub_mod(r1, r0 % q1, q1);
    const uint64_t k = mul_mod(d, q0inv_mod_q1, p1);
    return (unsigned __int128)r0 + (unsigned __int128)q0 * k;
}

// round(v * 2N / Q) mod 2N for 0 <= v < 2Q; v 2N has no exact half-integer quotient
// because Q is odd, so round-half-up equals the reference's rounding.
__device__ __forceinline__ uint32_t rotation(unsigned __int128 v, unsigned __int128 Q, long long N) {
    const unsigned __int128 num = v * (unsigned __int128)(2 * N);
    const unsigned __int128 k = (2 * num + Q) / (2 * Q);
    return (uint32_t)(k % (unsigned __int128)(2 * N));
}

// rots[i][b] = a_i' and rot0[b] = 2N - rot_b, for L0 = 1 or 2 LWE limbs.
// a: [B][L0][n], bb: [B][L0].
__global__ void k_rotations(uint32_t* __restrict__ rots, uint32_t* __restrict__ rot0, const uint64_t* __restrict__ a,
                            const uint64_t* __restrict__ bb, const __grid_constant__ CggiShape sh,
                            const PrimeInfo* __restrict__ primes, long long B, uint64_t q0inv, uint64_t offset_lo,
                            uint64_t offset_hi) {
    const PrimeInfo p0 = primes[sh.lwe_prime[0]];
    const PrimeInfo p1 = primes[sh.lwe_prime[sh.L0 > 1 ? 1 : 0]];
    const unsigned __int128 Q = sh.L0 > 1 ? (unsigned __int128)p0.q * p1.q : (unsigned __int128)p0.q;
    const long long total = B * (sh.n + 1);
    for (long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x; e < total;
         e += (long long)gridDim.x * blockDim.x) {
        const long long b = e / (sh.n + 1);
        const int i = (int)(e - b * (sh.n + 1));
        unsigned __int128 v;
        if (i < sh.n) {
            const uint64_t* ab = a + (b * sh.L0) * sh.n;
            v = sh.L0 > 1 ? crt2(ab[i], ab[sh.n + i], p0.q, p1.q, q0inv, p1) : (unsigned __int128)ab[i];
            rots[(long long)i * B + b] = rotation(v, Q, sh.N);
        } else {
            const uint64_t* bv = bb + b * sh.L0;
            v = sh.L0 > 1 ? crt2(bv[0], bv[1], p0.q, p1.q, q0inv, p1) : (unsigned __int128)bv[0];
            v += ((unsigned __int128)offset_hi << 64) | offset_lo;
            const uint32_t r = rotation(v, Q, sh.N);
            rot0[b] = (uint32_t)((2 * sh.N - r) % (2 * sh.N));
        }
    }
}

// acc[b][c][l] = tv[c][l] * X^rot0[b]   (mlwe_RNSc_mul_by_xai, rns_polynomial.c:1048-1106)
__global__ void k_init_acc(uint64_t* __restrict__ acc, const uint64_t* __restrict__ tv, const uint32_t* __restrict__ rot0,
                           const __grid_constant__ CggiShape sh, const PrimeInfo* __restrict__ primes) {
    const long long N = sh.N;
    const int rows = 2 * sh.L0;
    const long long b = blockIdx.y / rows;
    const int cl = blockIdx.y - (int)(b * rows);
    const uint64_t q = primes[sh.lwe_prime[cl % sh.L0]].q;
    const uint64_t a = rot0[b];
    const uint64_t* src = tv + (long long)cl * N;
    uint64_t* dst = acc + (b * rows + cl) * N;
    for (long long x = blockIdx.x * (long long)blockDim.x + threadIdx.x; x < N; x += (long long)gridDim.x * blockDim.x) {
        const uint64_t s = ((uint64_t)x + 2 * N - a) & (2 * N - 1);
        dst[x] = s < (uint64_t)N ? src[s] : neg_mod(src[s - N], q);
    }
}

// diff[b][c][l] = acc X^r - acc, r = rots[step][b]  (mgsw_CMUX's in2 - in1, mgsw.c:60-61)
__global__ void k_rot_diff(uint64_t* __restrict__ diff, const uint64_t* __restrict__ acc,
                           const uint32_t* __restrict__ rots_step, const __grid_constant__ CggiShape sh,
                           const PrimeInfo* __restrict__ primes) {
    const long long N = sh.N;
    const int rows = 2 * sh.L0;
    const long long b = blockIdx.y / rows;
    const int cl = blockIdx.y - (int)(b * rows);
    const uint64_t q = primes[sh.lwe_prime[cl % sh.L0]].q;
    const uint64_t a = rots_step[b];
    const uint64_t* src = acc + (b * rows + cl) * N;
    uint64_t* dst = diff + (b * rows + cl) * N;
    for (long long x = blockIdx.x * (long long)blockDim.x + threadIdx.x; x < N; x += (long long)gridDim.x * blockDim.x) {
        const uint64_t s = ((uint64_t)x + 2 * N - a) & (2 * N - 1);
        const uint64_t v = s < (uint64_t)N ? src[s] : neg_mod(src[s - N], q);
        dst[x] = sub_mod(v, src[x], q);
    }
}

// ext[b][c'][e] = sum_d D[b][d][e] * G[d][c'][e]   (gadget_mul_addto_polynomial, gadget.c:5-20)
// D: [B][nd][ne][N]; G: [nd][2][ne][N] (one MGSW of the key); ext: [B][2][ne][N].
__global__ void k_mac_shared(uint64_t* __restrict__ ext, const uint64_t* __restrict__ D, const uint64_t* __restrict__ G,
                             const __grid_constant__ CggiShape sh, const PrimeInfo* __restrict__ primes, int nd) {
    const long long N = sh.N;
    const int ne = sh.L0 + 1;
    const long long b = blockIdx.y / ne;
    const int e = blockIdx.y - (int)(b * ne);
    const PrimeInfo pi = primes[sh.ext_prime[e]];
    const double q = pi.qd, qinv = pi.qinv;
    const long long dstr = (long long)ne * N, gstr = 2LL * ne * N;
    const uint64_t* d = D + b * nd * dstr + (long long)e * N;
    const uint64_t* ga = G + (long long)e * N;
    const uint64_t* gb = ga + dstr;
    uint64_t* oa = ext + b * 2 * dstr + (long long)e * N;
    uint64_t* ob = oa + dstr;
    if ((N & 1) == 0 &&
        ((reinterpret_cast<uintptr_t>(d) | reinterpret_cast<uintptr_t>(ga) | reinterpret_cast<uintptr_t>(oa)) & 15) ==
            0) {
        // two residues per thread with 16-byte accesses; the digit is the multiplier of
        // both key products (one quotient; uncentred operands below 2^50, |t| <= 3q/4)
        for (long long x = 2 * (blockIdx.x * (long long)blockDim.x + threadIdx.x); x < N;
             x += 2 * (long long)gridDim.x * blockDim.x) {
            double sa0 = 0.0, sb0 = 0.0, sa1 = 0.0, sb1 = 0.0;
            for (int j = 0; j < nd; ++j) {
                const ulonglong2 dv = __ldcs(reinterpret_cast<const ulonglong2*>(d + j * dstr + x));
                const ulonglong2 av = *reinterpret_cast<const ulonglong2*>(ga + j * gstr + x);
                const ulonglong2 bv = *reinterpret_cast<const ulonglong2*>(gb + j * gstr + x);
                const double v0 = f_from_u64(dv.x), v1 = f_from_u64(dv.y);
                const double vq0 = __dmul_rn(v0, qinv), vq1 = __dmul_rn(v1, qinv);
                sa0 = __dadd_rn(sa0, f_mulmod(f_from_u64(av.x), v0, vq0, q));
                sa1 = __dadd_rn(sa1, f_mulmod(f_from_u64(av.y), v1, vq1, q));
                sb0 = __dadd_rn(sb0, f_mulmod(f_from_u64(bv.x), v0, vq0, q));
                sb1 = __dadd_rn(sb1, f_mulmod(f_from_u64(bv.y), v1, vq1, q));
                if ((j & 3) == 3) {
                    sa0 = f_reduce(sa0, q, qinv);
                    sa1 = f_reduce(sa1, q, qinv);
                    sb0 = f_reduce(sb0, q, qinv);
                    sb1 = f_reduce(sb1, q, qinv);
                }
            }
            ulonglong2 ra, rb;
            ra.x = f_to_canonical(sa0, q, qinv, pi.q);
            ra.y = f_to_canonical(sa1, q, qinv, pi.q);
            rb.x = f_to_canonical(sb0, q, qinv, pi.q);
            rb.y = f_to_canonical(sb1, q, qinv, pi.q);
            *reinterpret_cast<ulonglong2*>(oa + x) = ra;
            *reinterpret_cast<ulonglong2*>(ob + x) = rb;
        }
        return;
    }
    for (long long x = blockIdx.x * (long long)blockDim.x + threadIdx.x; x < N; x += (long long)gridDim.x * blockDim.x) {
        double sa = 0.0, sb = 0.0;
        for (int j = 0; j < nd; ++j) {
            const double v = f_from_u64(d[j * dstr + x]);
            const double wa = f_from_u64(ga[j * gstr + x]);
            const double wb = f_from_u64(gb[j * gstr + x]);
            sa = __dadd_rn(sa, f_mulmod(v, wa, __dmul_rn(wa, qinv), q));
            sb = __dadd_rn(sb, f_mulmod(v, wb, __dmul_rn(wb, qinv), q));
            if ((j & 3) == 3) {
                sa = f_reduce(sa, q, qinv);
                sb = f_reduce(sb, q, qinv);
            }
        }
        oa[x] = f_to_canonical(sa, q, qinv, pi.q);
        ob[x] = f_to_canonical(sb, q, qinv, pi.q);
    }
}

struct DivConsts {
    uint64_t half_sp[4], inv_sp[4], inv_sp_sh[4];
    uint64_t p, half_p;
    // FP64 form (every prime below 2^50): p^-1 centred with its quotient fl(w/q)
    int fp64;
    double half_sp_d[4], inv_sp_d[4], inv_sp_dq[4];
};

// acc[b][c][l] += round(ext[b][c] / p) limb l   (round division by the special prime,
// rns_polynomial.c:939-976, then the CMUX's + in1, mgsw.c:65-68)
__global__ void k_moddown_acc(uint64_t* __restrict__ acc, const uint64_t* __restrict__ ext,
                              const __grid_constant__ CggiShape sh, const __grid_constant__ DivConsts dc,
                              const PrimeInfo* __restrict__ primes) {
    const long long N = sh.N;
    const int L0 = sh.L0, ne = L0 + 1;
    const long long b = blockIdx.y >> 1;
    const int c = blockIdx.y & 1;
    const uint64_t* ex = ext + (b * 2 + c) * ne * N;
    uint64_t* ac = acc + (b * 2 + c) * L0 * N;
    if (dc.fp64 && (N & 1) == 0 && ((reinterpret_cast<uintptr_t>(ex) | reinterpret_cast<uintptr_t>(ac)) & 15) == 0) {
        // exact FP64 form of the loop below (every intermediate an integer below 2^52),
        // two coefficients per thread
        for (long long x = 2 * (blockIdx.x * (long long)blockDim.x + threadIdx.x); x < N;
             x += 2 * (long long)gridDim.x * blockDim.x) {
            const ulonglong2 sp = __ldcs(reinterpret_cast<const ulonglong2*>(ex + (long long)L0 * N + x));
            uint64_t t0 = sp.x + dc.half_p, t1 = sp.y + dc.half_p;
            t0 -= t0 >= dc.p ? dc.p : 0;
            t1 -= t1 >= dc.p ? dc.p : 0;
            const double td0 = f_from_u64(t0), td1 = f_from_u64(t1);
            for (int l = 0; l < L0; ++l) {
                const PrimeInfo& pi = primes[sh.lwe_prime[l]];
                const ulonglong2 ev = __ldcs(reinterpret_cast<const ulonglong2*>(ex + (long long)l * N + x));
                ulonglong2* ap = reinterpret_cast<ulonglong2*>(ac + (long long)l * N + x);
                const ulonglong2 av = *ap;
                const double y0 = __dadd_rn(__dadd_rn(f_from_u64(ev.x), dc.half_sp_d[l]), -td0);
                const double y1 = __dadd_rn(__dadd_rn(f_from_u64(ev.y), dc.half_sp_d[l]), -td1);
                const double v0 = __dadd_rn(f_mulmod(y0, dc.inv_sp_d[l], dc.inv_sp_dq[l], pi.qd), f_from_u64(av.x));
                const double v1 = __dadd_rn(f_mulmod(y1, dc.inv_sp_d[l], dc.inv_sp_dq[l], pi.qd), f_from_u64(av.y));
                ulonglong2 r;
                r.x = f_to_canonical(v0, pi.qd, pi.qinv, pi.q);
                r.y = f_to_canonical(v1, pi.qd, pi.qinv, pi.q);
                *ap = r;
            }
        }
        return;
    }
    for (long long x = blockIdx.x * (long long)blockDim.x + threadIdx.x; x < N; x += (long long)gridDim.x * blockDim.x) {
        const uint64_t t = add_mod(ex[(long long)L0 * N + x], dc.half_p, dc.p);
        for (int l = 0; l < L0; ++l) {
            const PrimeInfo& pi = primes[sh.lwe_prime[l]];
            uint64_t v = add_mod(ex[(long long)l * N + x], dc.half_sp[l], pi.q);
            v = sub_mod(v, reduce64(t, pi), pi.q);
            v = shoup(v, dc.inv_sp[l], dc.inv_sp_sh[l], pi.q);
            ac[(long long)l * N + x] = add_mod(ac[(long long)l * N + x], v, pi.q);
        }
    }
}

// ---- whole blind rotations on a cluster
//
// One cluster of L0 + 1 blocks runs one LWE's n CMUX steps, block e for extended prime e.
// Group d of N / 8 threads keeps limb d % L0 of component d / L0 of the accumulator in
// registers (every block a copy), forms digit d of acc X^r - acc, transforms it modulo the
// block's prime; the block multiplies the digits with its limb of the key and transforms the
// two outputs back.  The outputs go through L2 to the other blocks, which divide by the
// special prime and add: one cluster barrier a step.
//
// For batches of up to one block per SM, where a step's latency counts.  The transforms hold
// 8 residues a thread (three stages a pass) instead of the 16 of the tile kernels, so that a
// block has twice the warps.
//
// N = 1024, L0 = 2, n = 630: 18 us a step with five launches, 8.5 us here (about 4000 cycles
// forward, 1300 products, 4000 inverse, the rest barriers and the exchange through L2).

// A key pair loaded where the call stands (not moved to its use).
__device__ __forceinline__ ulonglong2 load_key(const uint64_t* p) {
    ulonglong2 v;
    asm volatile("ld.global.nc.v2.u64 {%0, %1}, [%2];" : "=l"(v.x), "=l"(v.y) : "l"(p));
    return v;
}

template <int K, int L0>
struct ClusterShape {
    static constexpr int N = 1 << K, NE = L0 + 1, ND = 2 * L0, TPT = 1 << (K - 3), THREADS = ND * TPT;
    static constexpr int PADDED = N + (N >> 3);
    static constexpr size_t smem = 8 * (size_t)(ND * PADDED);  // exchange buffers
};

template <int K, int L0>
__global__ void __launch_bounds__(ClusterShape<K, L0>::THREADS)
    k_cggi_cluster(uint64_t* __restrict__ out_a, uint64_t* __restrict__ out_b, double* ext0, double* ext1,
                   const uint64_t* __restrict__ tv, const uint64_t* __restrict__ bk, const uint32_t* __restrict__ rots,
                   const uint32_t* __restrict__ rot0, const __grid_constant__ CggiShape sh,
                   const __grid_constant__ DivConsts dc, const PrimeInfo* __restrict__ primes, long long B) {
    using C = ClusterShape<K, L0>;
    constexpr int N = C::N, NE = C::NE, ND = C::ND, TPT = C::TPT, T = C::THREADS, PADDED = C::PADDED;
    constexpr int NP = Passes8<K>::count;
    extern __shared__ __align__(128) double ex[];
    namespace cgx = cooperative_groups;
    cgx::cluster_group cluster = cgx::this_cluster();
    const int e = (int)cluster.block_rank();
    const long long b = blockIdx.x / NE;
    const int tid = threadIdx.x, g = tid / TPT, t = tid - g * TPT;
    const PrimeInfo& pi = primes[sh.ext_prime[e]];
    const double q = pi.qd, qinv = pi.qinv;
    const double2* fwd = reinterpret_cast<const double2*>(pi.fwd_d);
    double* exg = ex + g * PADDED;
    // this LWE's outputs [2][NE][N] as doubles, in the buffer of the step's parity
    ext0 += b * 2 * NE * N;
    ext1 += b * 2 * NE * N;
    // group g keeps limb dl of component dcomp of the accumulator, 8 residues a thread
    const int dl = g % L0, dcomp = g / L0;
    const PrimeInfo& pl = primes[sh.lwe_prime[dl]];
    const uint64_t ql = pl.q;
    uint64_t u[8];
    {  // acc = tv X^rot0 (mlwe_RNSc_mul_by_xai, rns_polynomial.c:1048-1106)
        const uint32_t a = rot0[b];
#pragma unroll
        for (int m = 0; m < 8; ++m) {
            const uint32_t s = ((uint32_t)Pass8<K, 0>::index(t, m) + 2 * N - a) & (2 * N - 1);
            const uint64_t v = tv[(long long)g * N + (s & (N - 1))];
            u[m] = s < (uint32_t)N ? v : neg_mod(v, ql);
        }
    }
    uint32_t r = rots[b];
    for (int i = 0; i < sh.n; ++i) {
        const uint32_t r_next = i + 1 < sh.n ? __ldg(rots + (long long)(i + 1) * B + b) : 0;
        const uint64_t* key = bk + (long long)i * (ND * 2 * NE) * N + (long long)e * N;
        if (i + 1 < sh.n && tid < ND * 2)  // the next step's limb rows on their way to L2
            asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(key + (long long)(ND * 2 + tid) * NE * N),
                         "n"(N * 8)
                         : "memory");
        // this step's key at the thread's multiply positions, on its way during the transforms
        constexpr int TURNS = N / (2 * T);
        ulonglong2 kv[TURNS][ND][2];
#pragma unroll
        for (int k = 0; k < TURNS; ++k)
#pragma unroll
            for (int d = 0; d < ND; ++d)
#pragma unroll
                for (int c = 0; c < 2; ++c)
                    kv[k][d][c] = load_key(key + (long long)(2 * d + c) * NE * N + 2 * (tid + k * T));
        // digit g of acc X^r - acc (mgsw_CMUX's in2 - in1, mgsw.c:60-61), modulo this prime;
        // the rotated limb through the group's buffer
        double x[8];
        Twiddles8 tw0;
        load_twiddles<K, 0>(tw0, fwd, t);
        {
            uint64_t* rowbuf = reinterpret_cast<uint64_t*>(exg);
#pragma unroll
            for (int m = 0; m < 8; ++m) rowbuf[Pass8<K, 0>::index(t, m)] = u[m];
            group_sync(g, TPT);
#pragma unroll
            for (int m = 0; m < 8; ++m) {
                const uint32_t s = ((uint32_t)Pass8<K, 0>::index(t, m) + 2 * N - r) & (2 * N - 1);
                const uint64_t v = rowbuf[s & (N - 1)];
                uint64_t d = s < (uint32_t)N ? v - u[m] : 0 - v - u[m];
                // d is in (-2q, q) modulo 2^64
                if ((long long)d < 0) d += ql;
                if ((long long)d < 0) d += ql;
                x[m] = f_from_u64(d);
                if (dl != e) x[m] = f_reduce(x[m], q, qinv);
            }
        }
        fwd8<K, 0>(x, tw0, exg, t, g, fwd, q, qinv);
#pragma unroll
        for (int m = 0; m < 8; ++m) x[m] = f_reduce(x[m], q, qinv);
        group_sync(g, TPT);  // the last exchange is read
        put_regs<K, NP - 1>(exg, x, t);
        __syncthreads();
        // both outputs at two positions a turn: sums of ND products, |sum| <= 3q
        double s[TURNS][2][2];
#pragma unroll
        for (int k = 0; k < TURNS; ++k) {
            const int xx = 2 * (tid + k * T);
            s[k][0][0] = s[k][0][1] = s[k][1][0] = s[k][1][1] = 0.0;
#pragma unroll
            for (int d = 0; d < ND; ++d) {
                const ulonglong2 ka = kv[k][d][0], kb = kv[k][d][1];
                const double2 v = *reinterpret_cast<const double2*>(ex + d * PADDED + pad8(xx));
                const double w0 = __dmul_rn(v.x, qinv), w1 = __dmul_rn(v.y, qinv);
                s[k][0][0] = __dadd_rn(s[k][0][0], f_mulmod(f_from_u64(ka.x), v.x, w0, q));
                s[k][0][1] = __dadd_rn(s[k][0][1], f_mulmod(f_from_u64(ka.y), v.y, w1, q));
                s[k][1][0] = __dadd_rn(s[k][1][0], f_mulmod(f_from_u64(kb.x), v.x, w0, q));
                s[k][1][1] = __dadd_rn(s[k][1][1], f_mulmod(f_from_u64(kb.y), v.y, w1, q));
            }
        }
        __syncthreads();  // every spectrum is read
#pragma unroll
        for (int k = 0; k < TURNS; ++k) {
            const int xx = 2 * (tid + k * T);
#pragma unroll
            for (int c = 0; c < 2; ++c)
                *reinterpret_cast<double2*>(ex + c * PADDED + pad8(xx)) =
                    make_double2(f_reduce(s[k][c][0], q, qinv), f_reduce(s[k][c][1], q, qinv));
        }
        __syncthreads();
        double* ext = (i & 1) ? ext1 : ext0;
        if (g < 2) {  // output g back to coefficients, for every block of the cluster
            Twiddles8 twi;
            load_twiddles<K, NP - 1>(twi, reinterpret_cast<const double2*>(pi.inv_d), t);
            get_regs<K, NP - 1>(x, exg, t);
            inv8<K, NP - 1>(x, twi, exg, t, g, pi);
            double* o = ext + (g * NE + e) * N;
#pragma unroll
            for (int m = 0; m < 8; ++m) {
                if (e == L0) {  // the special prime's: (x + p/2) mod p
                    uint64_t v = f_to_canonical(x[m], q, qinv, pi.q) + dc.half_p;
                    v -= v >= dc.p ? dc.p : 0;
                    x[m] = f_from_u64(v);
                }
                o[Pass8<K, 0>::index(t, m)] = x[m];
            }
        }
        cluster.sync();
        // round division by the special prime (rns_polynomial.c:939-976) + in1 (mgsw.c:65-68).
        // The other parity's buffer is written meanwhile; this one again only after the next
        // barrier, which every block reaches past these reads.
        {
            const double* ev = ext + (dcomp * NE + dl) * N;
            const double* tp = ext + (dcomp * NE + L0) * N;
            double y[8], td[8];
#pragma unroll
            for (int m = 0; m < 8; ++m) {
                y[m] = __ldcg(ev + Pass8<K, 0>::index(t, m));
                td[m] = __ldcg(tp + Pass8<K, 0>::index(t, m));
            }
#pragma unroll
            for (int m = 0; m < 8; ++m) {
                const double z = __dadd_rn(__dadd_rn(y[m], dc.half_sp_d[dl]), -td[m]);
                const double v = __dadd_rn(f_mulmod(z, dc.inv_sp_d[dl], dc.inv_sp_dq[dl], pl.qd), f_from_u64(u[m]));
                u[m] = f_to_canonical(v, pl.qd, pl.qinv, ql);
            }
        }
        r = r_next;
    }
    // sample extraction at coefficient 0 (mlwe.c:40-68)
    if (e == 0) {
#pragma unroll
        for (int m = 0; m < 8; ++m) {
            const int j = Pass8<K, 0>::index(t, m);
            if (dcomp == 0) out_a[(b * L0 + dl) * N + ((N - j) & (N - 1))] = j == 0 ? u[m] : neg_mod(u[m], ql);
            else if (j == 0) out_b[b * L0 + dl] = u[m];
        }
    }
}

template <int K, int L0>
int launch_cluster_t(uint64_t* out_a, uint64_t* out_b, double* ext0, double* ext1, const uint64_t* tv, const uint64_t* bk, const uint32_t* rots,
                     const uint32_t* rot0, const CggiShape& sh, const DivConsts& dc, const PrimeInfo* dp, uint64_t B,
                     cudaStream_t st) {
    using C = ClusterShape<K, L0>;
    int e = (int)cudaFuncSetAttribute(k_cggi_cluster<K, L0>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)C::smem);
    if (e) return e;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)(B * C::NE), 1, 1);
    cfg.blockDim = dim3(C::THREADS, 1, 1);
    cfg.dynamicSmemBytes = C::smem;
    cfg.stream = st;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = C::NE;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    e = (int)cudaLaunchKernelEx(&cfg, k_cggi_cluster<K, L0>, out_a, out_b, ext0, ext1, tv, bk, rots, rot0, sh, dc, dp, (long long)B);
    if (e) return e;
    note_launch();
    return (int)cudaGetLastError();
}

// -1 for shapes without a cluster kernel.
int launch_cluster(int K, uint64_t* out_a, uint64_t* out_b, double* ext0, double* ext1, const uint64_t* tv, const uint64_t* bk, const uint32_t* rots,
                   const uint32_t* rot0, const CggiShape& sh, const DivConsts& dc, const PrimeInfo* dp, uint64_t B,
                   cudaStream_t st) {
    switch (K * 4 + sh.L0) {
        case 8 * 4 + 1: return launch_cluster_t<8, 1>(out_a, out_b, ext0, ext1, tv, bk, rots, rot0, sh, dc, dp, B, st);
        case 8 * 4 + 2: return launch_cluster_t<8, 2>(out_a, out_b, ext0, ext1, tv, bk, rots, rot0, sh, dc, dp, B, st);
        case 9 * 4 + 1: return launch_cluster_t<9, 1>(out_a, out_b, ext0, ext1, tv, bk, rots, rot0, sh, dc, dp, B, st);
        case 9 * 4 + 2: return launch_cluster_t<9, 2>(out_a, out_b, ext0, ext1, tv, bk, rots, rot0, sh, dc, dp, B, st);
        case 10 * 4 + 1: return launch_cluster_t<10, 1>(out_a, out_b, ext0, ext1, tv, bk, rots, rot0, sh, dc, dp, B, st);
        case 10 * 4 + 2: return launch_cluster_t<10, 2>(out_a, out_b, ext0, ext1, tv, bk, rots, rot0, sh, dc, dp, B, st);
        case 11 * 4 + 1: return launch_cluster_t<11, 1>(out_a, out_b, ext0, ext1, tv, bk, rots, rot0, sh, dc, dp, B, st);
        case 11 * 4 + 2: return launch_cluster_t<11, 2>(out_a, out_b, ext0, ext1, tv, bk, rots, rot0, sh, dc, dp, B, st);
        default: return -1;
    }
}

// ---- one CMUX step's external product in one launch
//
// Block (extended prime e, LWE b): the 2 L0 digits of acc X^r - acc modulo prime e (group d
// of 2^(K-4) threads reads digit d's limb of the accumulator through L2), their transforms,
// the products with limb e of the key, and both outputs' inverse transforms into
// ext [B][2][L0 + 1][N].  Only the accumulator, the key and ext pass through L2; as four
// launches (rotation difference, transforms, products, inverse) the digits and their spectra
// did too.  Bound by the FP64 pipe's latency and rate: 1.1 M operations per LWE and step at
// N = 1024, L0 = 2, 9 us of one SM.  1024 bootstraps at n = 630: 99 ms before, 67.3 ms.
template <int K, int L0>
struct StepShape {
    static constexpr int N = 1 << K, NE = L0 + 1, ND = 2 * L0, TPT = 1 << (K - 4), THREADS = ND * TPT;
    static constexpr int PADDED = N + (N >> 4);
    static constexpr size_t smem = 8 * (size_t)(ND * PADDED);
    static constexpr int min_ctas = THREADS <= 256 ? 768 / THREADS < 6 ? 768 / THREADS : 6 : 1;  // 85 registers
};

template <int K, int L0>
__global__ void __launch_bounds__(StepShape<K, L0>::THREADS, StepShape<K, L0>::min_ctas)
    k_cggi_step(uint64_t* __restrict__ ext, const uint64_t* __restrict__ acc, const uint64_t* __restrict__ key0,
                const uint32_t* __restrict__ rots_step, const __grid_constant__ CggiShape sh,
                const PrimeInfo* __restrict__ primes, int B) {
    using C = StepShape<K, L0>;
    constexpr int N = C::N, NE = C::NE, ND = C::ND, TPT = C::TPT, T = C::THREADS, PADDED = C::PADDED;
    extern __shared__ __align__(128) double sm[];
    // the blocks of one prime are neighbours: an SM's blocks then share its limb of the key in L1
    const int e = blockIdx.x / B, b = blockIdx.x - e * B;
    const int tid = threadIdx.x, g = tid / TPT, t = tid - g * TPT;
    const PrimeInfo& pi = primes[sh.ext_prime[e]];
    const double q = pi.qd, qinv = pi.qinv;
    const FCtx fc = fwd_ctx(pi);
    double* smg = sm + g * PADDED;
    const uint64_t* key = key0 + (long long)e * N;
    double x[16];
    {
        PassTw<K - 4, K - 1, K - 4> tw1;
        f_fwd_tw<K, K - 4, K - 1, K - 4>(tw1, t, 0, K, fc);
        // digit g: limb g % L0 of component g / L0 of acc X^r - acc (mgsw_CMUX's in2 - in1, mgsw.c:60-61)
        const int dl = g % L0;
        const uint64_t ql = primes[sh.lwe_prime[dl]].q;
        const uint64_t* a = acc + ((long long)b * ND + g) * N;
        const uint32_t r = rots_step[b];
#pragma unroll
        for (int m = 0; m < 16; ++m) {
            const int j = own<K - 4>(t, m);
            const uint32_t s = ((uint32_t)j + 2 * N - r) & (2 * N - 1);
            const uint64_t v = __ldg(a + (s & (N - 1))), u = __ldg(a + j);
            uint64_t d = s < (uint32_t)N ? v - u : 0 - v - u;
            // d is in (-2q, q) modulo 2^64
            if ((long long)d < 0) d += ql;
            if ((long long)d < 0) d += ql;
            x[m] = f_from_u64(d);
            if (dl != e) x[m] = f_reduce(x[m], q, qinv);
        }
        tile_fwd_passes<K, true>(fc, K, 0, smg, t, x, tw1, g);
    }
    tile_sync<K, true>(g);  // the last exchange is read
#pragma unroll
    for (int m = 0; m < 16; ++m) smg[pad(edge<K>(t, m))] = f_reduce(x[m], q, qinv);
    __syncthreads();
    // both outputs at two positions a turn: sums of ND products, |sum| <= 3q
    constexpr int TURNS = N / (2 * T);
    double s[TURNS][2][2];
#pragma unroll
    for (int k = 0; k < TURNS; ++k) {
        const int xx = 2 * (tid + k * T);
        s[k][0][0] = s[k][0][1] = s[k][1][0] = s[k][1][1] = 0.0;
#pragma unroll
        for (int d = 0; d < ND; ++d) {
            const ulonglong2 ka = __ldg(reinterpret_cast<const ulonglong2*>(key + (long long)(2 * d) * NE * N + xx));
            const ulonglong2 kb = __ldg(reinterpret_cast<const ulonglong2*>(key + (long long)(2 * d + 1) * NE * N + xx));
            const double v0 = sm[d * PADDED + pad(xx)], v1 = sm[d * PADDED + pad(xx + 1)];
            const double w0 = __dmul_rn(v0, qinv), w1 = __dmul_rn(v1, qinv);
            s[k][0][0] = __dadd_rn(s[k][0][0], f_mulmod(f_from_u64(ka.x), v0, w0, q));
            s[k][0][1] = __dadd_rn(s[k][0][1], f_mulmod(f_from_u64(ka.y), v1, w1, q));
            s[k][1][0] = __dadd_rn(s[k][1][0], f_mulmod(f_from_u64(kb.x), v0, w0, q));
            s[k][1][1] = __dadd_rn(s[k][1][1], f_mulmod(f_from_u64(kb.y), v1, w1, q));
        }
    }
    __syncthreads();  // every spectrum is read
#pragma unroll
    for (int k = 0; k < TURNS; ++k) {
        const int xx = 2 * (tid + k * T);
#pragma unroll
        for (int c = 0; c < 2; ++c) {
            sm[c * PADDED + pad(xx)] = f_reduce(s[k][c][0], q, qinv);
            sm[c * PADDED + pad(xx + 1)] = f_reduce(s[k][c][1], q, qinv);
        }
    }
    __syncthreads();
    if (g >= 2) return;
#pragma unroll
    for (int m = 0; m < 16; ++m) x[m] = smg[pad(edge<K>(t, m))];
    tile_inv_regs<K, true, true>(pi, K, 0, smg, t, x, g);
    uint64_t* o = ext + (((long long)b * 2 + g) * NE + e) * N;
#pragma unroll
    for (int m = 0; m < 16; ++m) o[own<K - 4>(t, m)] = f_to_canonical(x[m], q, qinv, pi.q);
}

template <int K, int L0>
int launch_step_t(uint64_t* ext, const uint64_t* acc, const uint64_t* key, const uint32_t* rots_step, const CggiShape& sh,
                  const PrimeInfo* dp, uint64_t B, cudaStream_t st) {
    using C = StepShape<K, L0>;
    if (C::smem > 48 * 1024) {
        const int e = (int)cudaFuncSetAttribute(k_cggi_step<K, L0>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)C::smem);
        if (e) return e;
    }
    k_cggi_step<K, L0><<<(unsigned)(B * C::NE), C::THREADS, C::smem, st>>>(ext, acc, key, rots_step, sh, dp, (int)B);
    note_launch();
    return (int)cudaGetLastError();
}

// -1 for shapes without a step kernel.
int launch_step(int K, uint64_t* ext, const uint64_t* acc, const uint64_t* key, const uint32_t* rots_step,
                const CggiShape& sh, const PrimeInfo* dp, uint64_t B, cudaStream_t st) {
    switch (K * 4 + sh.L0) {
        case 9 * 4 + 1: return launch_step_t<9, 1>(ext, acc, key, rots_step, sh, dp, B, st);
        case 9 * 4 + 2: return launch_step_t<9, 2>(ext, acc, key, rots_step, sh, dp, B, st);
        case 10 * 4 + 1: return launch_step_t<10, 1>(ext, acc, key, rots_step, sh, dp, B, st);
        case 10 * 4 + 2: return launch_step_t<10, 2>(ext, acc, key, rots_step, sh, dp, B, st);
        case 11 * 4 + 1: return launch_step_t<11, 1>(ext, acc, key, rots_step, sh, dp, B, st);
        case 11 * 4 + 2: return launch_step_t<11, 2>(ext, acc, key, rots_step, sh, dp, B, st);
        default: return -1;
    }
}

// Sample extraction at coefficient 0 (mlwe.c:40-68): out_a[b][l][i] = a[0] for i = 0,
// -a[N - i] otherwise; out_b[b][l] = b[0].
__global__ void k_extract0(uint64_t* __restrict__ out_a, uint64_t* __restrict__ out_b, const uint64_t* __restrict__ acc,
                           const __grid_constant__ CggiShape sh, const PrimeInfo* __restrict__ primes) {
    const long long N = sh.N;
    const int L0 = sh.L0;
    const long long b = blockIdx.y / L0;
    const int l = blockIdx.y - (int)(b * L0);
    const uint64_t q = primes[sh.lwe_prime[l]].q;
    const uint64_t* a = acc + (b * 2 * L0 + l) * N;
    const uint64_t* bv = acc + (b * 2 * L0 + L0 + l) * N;
    uint64_t* o = out_a + (b * L0 + l) * N;
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < N; i += (long long)gridDim.x * blockDim.x)
        o[i] = i == 0 ? a[0] : neg_mod(a[N - i], q);
    if (blockIdx.x == 0 && threadIdx.x == 0) out_b[b * L0 + l] = bv[0];
}

dim3 cg_grid(long long n, long long y) {
    note_launch();
    long long blocks = (n + 255) / 256;
    if (blocks > 64) blocks = 64;
    if (blocks < 1) blocks = 1;
    return dim3((unsigned)blocks, (unsigned)y, 1);
}

struct GraphKey {
    const void* ptrs[8];
    uint64_t batch;
    uint32_t n;
    uint32_t primes[5];  // LWE limbs then the special prime (kernel arguments baked into the graph)
    bool operator==(const GraphKey& o) const {
        return batch == o.batch && n == o.n && memcmp(ptrs, o.ptrs, sizeof ptrs) == 0 &&
               memcmp(primes, o.primes, sizeof primes) == 0;
    }
};

}  // namespace

uint64_t cggi_ws_elems(uint64_t N, uint64_t B, uint64_t n, uint32_t L0) {
    const uint64_t ne = L0 + 1, nd = 2 * (uint64_t)L0;
    // acc + diff + digits + ext, plus rotation tables (uint32, rounded up to words)
    return B * N * (2 * L0 + 2 * L0 + nd * ne + 2 * ne) + (B * (n + 1) + 1) / 2 + 64;
}

int cggi_bootstrap(IncNtt* t, uint64_t* out_a, uint64_t* out_b, const uint64_t* in_a, const uint64_t* in_b,
                   uint64_t B, uint32_t n, const uint32_t* limbs, uint32_t L0, uint32_t special, const uint64_t* bk,
                   const uint64_t* tv, uint64_t torus_base, uint64_t* ws, cudaStream_t st) {
    const char* where = "vfhe_cuda_cggi_bootstrap_batch";
    if (!t || L0 < 1 || L0 > 2 || !limbs || special >= t->pub.l || t->pub.split_degree != 1 || n == 0 ||
        torus_base == 0) {
        set_error(where, "needs split_degree 1, one or two LWE limbs, a special prime and n > 0");
        return 1;
    }
    if (B == 0 || B > 16383) {  // grid.y carries batch x 4 rows
        set_error(where, "batch must be in [1, 16383]");
        return 1;
    }
    for (uint32_t k = 0; k < L0; ++k)
        if (limbs[k] >= t->pub.l || !t->info[limbs[k]].fp64) {
            set_error(where, "limb outside the pool or prime above 2^50");
            return 1;
        }
    if (!t->info[special].fp64) {
        set_error(where, "special prime above 2^50");
        return 1;
    }
    const long long N = (long long)t->pub.N;
    CggiShape sh;
    memset(&sh, 0, sizeof sh);
    for (uint32_t k = 0; k < L0; ++k) sh.lwe_prime[k] = sh.ext_prime[k] = limbs[k];
    sh.ext_prime[L0] = special;
    sh.L0 = (int)L0;
    sh.n = (int)n;
    sh.N = N;
    const int ne = (int)L0 + 1, nd = 2 * (int)L0;

    uint64_t* acc = ws;                                  // [B][2][L0][N]  coefficient domain
    uint64_t* diff = acc + B * 2 * L0 * N;               // [B][2][L0][N]
    uint64_t* D = diff + B * 2 * L0 * N;                 // [B][nd][ne][N] NTT domain
    uint64_t* ext = D + B * (uint64_t)nd * ne * N;       // [B][2][ne][N]
    uint32_t* rot0 = (uint32_t*)(ext + B * 2 * ne * N);  // [B]
    uint32_t* rots = rot0 + B;                           // [n][B]

    // constants
    const uint64_t q0 = t->info[limbs[0]].q, q1 = L0 > 1 ? t->info[limbs[1]].q : 1;
    const uint64_t q0inv = L0 > 1 ? host_inv_mod(q0 % q1, q1) : 0;
    const unsigned __int128 Q = (unsigned __int128)q0 * q1;
    const unsigned __int128 off = Q / (4 * (unsigned __int128)torus_base);
    DivConsts dc;
    memset(&dc, 0, sizeof dc);
    const uint64_t p = t->info[special].q;
    dc.p = p;
    dc.half_p = p / 2;
    for (uint32_t l = 0; l < L0; ++l) {
        const uint64_t q = t->info[limbs[l]].q;
        dc.half_sp[l] = (p / 2) % q;
        dc.inv_sp[l] = host_inv_mod(p % q, q);
        dc.inv_sp_sh[l] = host_shoup(dc.inv_sp[l], q);
    }
    dc.fp64 = p < (1ULL << 50);
    for (uint32_t l = 0; l < L0; ++l) {
        const uint64_t q = t->info[limbs[l]].q;
        dc.fp64 = dc.fp64 && q < (1ULL << 50);
        const uint64_t w = dc.inv_sp[l];
        dc.half_sp_d[l] = (double)dc.half_sp[l];
        dc.inv_sp_d[l] = w > q / 2 ? (double)w - (double)q : (double)w;
        dc.inv_sp_dq[l] = dc.inv_sp_d[l] / (double)q;
    }
    const PrimeInfo* dp = t->d_info;

    // digit transforms: slot k = d * ne + e, d = c * L0 + l: diff row (b, c, l) lifted to ext limb e
    RowSet dig;
    memset(&dig, 0, sizeof dig);
    for (int d = 0; d < nd; ++d)
        for (int e = 0; e < ne; ++e) {
            const int k = d * ne + e;
            dig.in[k] = diff + (long long)d * N;
            dig.out[k] = D + (long long)k * N;
            dig.prime[k] = sh.ext_prime[e];
        }
    dig.nlimbs = nd * ne;
    dig.split = 1;
    dig.logP = t->logP;
    dig.batch = (int)B;
    dig.batch_stride = (long long)nd * ne * N;
    dig.in_batch_stride = 2LL * L0 * N;
    dig.reduce_input = 1;
    mark_fp64(dig, t);
    RowSet inv;
    memset(&inv, 0, sizeof inv);
    for (int e = 0; e < ne; ++e) {
        inv.in[e] = ext + (long long)e * N;
        inv.out[e] = ext + (long long)e * N;
        inv.prime[e] = sh.ext_prime[e];
    }
    inv.nlimbs = ne;
    inv.split = 1;
    inv.logP = t->logP;
    inv.batch = (int)(2 * B);
    inv.batch_stride = (long long)ne * N;
    inv.in_batch_stride = inv.batch_stride;
    mark_fp64(inv, t);

    k_rotations<<<cg_grid(B * (n + 1), 1), 256, 0, st>>>(rots, rot0, in_a, in_b, sh, dp, (long long)B, q0inv,
                                                         (uint64_t)off, (uint64_t)(off >> 64));
    // The fused kernels take 16-byte key pairs and N = 256 (clusters only) to 2048; one launch
    // per stage otherwise.  Clusters of one block per SM do best while all of the batch's fit
    // (44 clusters of 3 do on 148 SMs, 47 do not: 973 and 1519 us at n = 100, where a launch
    // per step takes 1335); past that the launches, whose blocks never wait for one another.
    const bool fused = dc.fp64 && t->info[special].fp64 && (reinterpret_cast<uintptr_t>(bk) & 15) == 0;
    if (fused && B * ne * 9 <= (uint64_t)sm_count() * 8) {
        const int ec = launch_cluster(t->logP, out_a, out_b, (double*)ext, (double*)D, tv, bk, rots, rot0, sh, dc, dp, B, st);
        if (ec != -1) return check_cuda(ec, where) ? 0 : 1;
    }
    k_init_acc<<<cg_grid(N, B * 2 * L0), 256, 0, st>>>(acc, tv, rot0, sh, dp);
    if (!check_cuda(cudaGetLastError(), where)) return 1;

    // the n blind-rotation steps: one CUDA graph per (shape, buffers), replayed
    struct Cached {
        GraphKey key;
        cudaGraphExec_t exec;
        uint64_t launches;  // kernels per replay
    };
    static std::vector<Cached> graphs;
    GraphKey key;
    memset(&key, 0, sizeof key);
    const void* ptrs[8] = {t, acc, diff, D, ext, rots, bk, dp};
    memcpy(key.ptrs, ptrs, sizeof ptrs);
    key.batch = B;
    key.n = n;
    memcpy(key.primes, sh.ext_prime, sizeof key.primes);
    cudaGraphExec_t exec = nullptr;
    uint64_t per_replay = 0;
    for (auto& g : graphs)
        if (g.key == key) {
            exec = g.exec;
            per_replay = g.launches;
        }
    if (!exec) {
        if (!check_cuda(prepare_ntt_kernels(), where)) return 1;
        const uint64_t counted0 = launch_counter();
        cudaStream_t cs = nullptr;
        if (!check_cuda(cudaStreamCreateWithFlags(&cs, cudaStreamNonBlocking), where)) return 1;
        if (!check_cuda(cudaStreamBeginCapture(cs, cudaStreamCaptureModeThreadLocal), where)) return 1;
        const uint64_t bk_stride = (uint64_t)nd * 2 * ne * N;
        int err = 0;
        for (uint32_t i = 0; i < n && !err; ++i) {
            err = fused ? launch_step(t->logP, ext, acc, bk + i * bk_stride, rots + (uint64_t)i * B, sh, dp, B, cs) : -1;
            if (err == 0) {
                k_moddown_acc<<<cg_grid((N + 1) / 2, B * 2), 256, 0, cs>>>(acc, ext, sh, dc, dp);
                continue;
            }
            if (err != -1) break;
            // four coefficients per thread: at N = 1024 one block per row, so the launch is
            // not bound by the block rate
            k_rot_diff<<<cg_grid((N + 3) / 4, B * 2 * L0), 256, 0, cs>>>(diff, acc, rots + (uint64_t)i * B, sh, dp);
            err = launch_ntt(dig, dp, false, cs);
            if (err) break;
            k_mac_shared<<<cg_grid((N + 1) / 2, B * ne), 256, 0, cs>>>(ext, D, bk + i * bk_stride, sh, dp, nd);
            err = launch_ntt(inv, dp, true, cs);
            if (err) break;
            k_moddown_acc<<<cg_grid((N + 1) / 2, B * 2), 256, 0, cs>>>(acc, ext, sh, dc, dp);
        }
        cudaGraph_t graph = nullptr;
        const cudaError_t e1 = cudaStreamEndCapture(cs, &graph);
        cudaStreamDestroy(cs);
        per_replay = launch_counter() - counted0;  // counted at capture: taken back, noted per replay
        forget_launches(per_replay);
        if (err || !check_cuda(e1, where)) {
            if (graph) cudaGraphDestroy(graph);
            if (err) check_cuda(err, where);
            return 1;
        }
        const cudaError_t e2 = cudaGraphInstantiate(&exec, graph, 0);
        cudaGraphDestroy(graph);
        if (!check_cuda(e2, where)) return 1;
        graphs.push_back(Cached{key, exec, per_replay});
    }
    if (!check_cuda(cudaGraphLaunch(exec, st), where)) return 1;
    note_launch((int)per_replay);
    k_extract0<<<cg_grid(N, B * L0), 256, 0, st>>>(out_a, out_b, acc, sh, dp);
    return check_cuda(cudaGetLastError(), where) ? 0 : 1;
}

}  // namespace vc
