// FP64 transforms with 8 residues a thread (three stages a pass) of one row held by a group
// of 2^(K-3) threads, for kernels whose few blocks leave SMs short of warps: twice the warps
// of the 16-residue tiles (ntt_f64_dev.cuh) at half the registers, for one more exchange.
// Used by the CGGI cluster kernel and the small-batch ring product.
#pragma once
#include "ntt_f64_dev.cuh"

namespace vc {

namespace {

__device__ __forceinline__ void group_sync(int grp, int threads) {
    asm volatile("bar.sync %0, %1;" ::"r"(1 + grp), "r"(threads) : "memory");
}

__device__ __forceinline__ int pad8(int i) { return i + ((i >> 4) << 1); }

// Pass P of a 2^K-point transform in 8-residue passes: three index bits from the top, the
// last pass the K mod 3 bits left (none: K / 3 passes).  index() is residue k's place for
// thread t; a partial pass takes its low bits and the index's top bits, so that the lanes
// of a warp own consecutive groups.
template <int K, int P>
struct Pass8 {
    static constexpr int FULL = K / 3;
    static constexpr bool PARTIAL = P >= FULL;
    static constexpr int LO = PARTIAL ? 0 : K - 3 * (P + 1);
    static constexpr int NST = PARTIAL ? K % 3 : 3;
    __device__ __forceinline__ static int index(int t, int k) {
        if constexpr (PARTIAL) {
            return ((k >> NST) << (K - 3 + NST)) | (t << NST) | (k & ((1 << NST) - 1));
        } else {
            return ((t >> LO) << (LO + 3)) | (k << LO) | (t & ((1 << LO) - 1));
        }
    }
    // The butterflies at field bit bb have 2^(2-bb) twiddles (partial pass: 8 / 2^(bb+1)), by
    // k >> (bb + 1); stage bb's start at offset(bb).
    static constexpr int offset(int bb) { return bb == 0 ? 0 : bb == 1 ? 4 : 6; }
};

// The pass's twiddles, requested before the exchange that precedes it so that their latency
// overlaps the barrier (tables by 2^(K-1-b) + (i >> (b + 1)) for index bit b).
struct Twiddles8 {
    double2 w[7];
};

template <int K, int P>
__device__ __forceinline__ void load_twiddles(Twiddles8& T, const double2* tw, int t) {
    using Q = Pass8<K, P>;
#pragma unroll
    for (int bb = 0; bb < Q::NST; ++bb) {
        const int b = Q::LO + bb;
#pragma unroll
        for (int h = 0; h < (4 >> bb); ++h)
            T.w[Q::offset(bb) + h] = __ldg(&tw[(1 << (K - 1 - b)) + (Q::index(t, h << (bb + 1)) >> (b + 1))]);
    }
}

template <int K>
struct Passes8 {
    static constexpr int count = (K + 2) / 3;
};

template <int K, int P>
__device__ __forceinline__ void put_regs(double* sm, const double (&x)[8], int t) {
#pragma unroll
    for (int k = 0; k < 8; ++k) sm[pad8(Pass8<K, P>::index(t, k))] = x[k];
}

template <int K, int P>
__device__ __forceinline__ void get_regs(double (&x)[8], const double* sm, int t) {
#pragma unroll
    for (int k = 0; k < 8; ++k) x[k] = sm[pad8(Pass8<K, P>::index(t, k))];
}

// Forward (Cooley-Tukey) passes P.. of 8 residues a thread in pass P's layout; every fourth
// stage of the transform ends with a reduction (|x| <= q in, each stage adds at most 3q/4,
// so every product's operand stays below 4q < 2^52).  Out: the last pass's layout, |x| < 4q.
template <int K, int P>
__device__ __forceinline__ void fwd8(double (&x)[8], const Twiddles8& T, double* sm, int t, int grp, const double2* tw,
                                     double q, double qinv) {
    using Q = Pass8<K, P>;
#pragma unroll
    for (int bb = Q::NST - 1; bb >= 0; --bb) {
#pragma unroll
        for (int k = 0; k < 8; ++k) {
            if (k & (1 << bb)) continue;
            const double2 w = T.w[Q::offset(bb) + (k >> (bb + 1))];
            const double v = f_mulmod(x[k | (1 << bb)], w.x, w.y, q);
            const double u = x[k];
            x[k] = __dadd_rn(u, v);
            x[k | (1 << bb)] = __dsub_rn(u, v);
        }
        const int stage = K - (Q::LO + bb);  // stages done so far
        if ((stage & 3) == 0 && stage != K) {
#pragma unroll
            for (int k = 0; k < 8; ++k) x[k] = f_reduce(x[k], q, qinv);
        }
    }
    if constexpr (P + 1 < Passes8<K>::count) {
        Twiddles8 next;
        load_twiddles<K, P + 1>(next, tw, t);
        group_sync(grp, 1 << (K - 3));  // the buffer's last contents are read
        put_regs<K, P>(sm, x, t);
        group_sync(grp, 1 << (K - 3));
        get_regs<K, P + 1>(x, sm, t);
        fwd8<K, P + 1>(x, next, sm, t, grp, tw, q, qinv);
    }
}

// Inverse (Gentleman-Sande) passes P down to 0, residues in pass P's layout, |x| <= q / 2 + 1
// in.  Sums double with every stage: three stages reach 4q < 2^52, so the sums are reduced at
// the end of each pass.  P^-1 is folded into the last stage; |x| <= 3q/4 out, pass 0's layout.
template <int K, int P>
__device__ __forceinline__ void inv8(double (&x)[8], const Twiddles8& T, double* sm, int t, int grp, const PrimeInfo& pi) {
    using Q = Pass8<K, P>;
    const double q = pi.qd, qinv = pi.qinv;
#pragma unroll
    for (int bb = 0; bb < Q::NST; ++bb) {
        const bool last = P == 0 && bb == Q::NST - 1;
#pragma unroll
        for (int k = 0; k < 8; ++k) {
            if (k & (1 << bb)) continue;
            const double u = x[k], v = x[k | (1 << bb)];
            if (last) {
                x[k] = f_mulmod(__dadd_rn(u, v), pi.pinv_d, pi.pinv_q, q);
                x[k | (1 << bb)] = f_mulmod(__dsub_rn(u, v), pi.ilast_d, pi.ilast_q, q);
            } else {
                const double2 w = T.w[Q::offset(bb) + (k >> (bb + 1))];
                x[k] = __dadd_rn(u, v);
                x[k | (1 << bb)] = f_mulmod(__dsub_rn(u, v), w.x, w.y, q);
            }
        }
    }
    if constexpr (P > 0) {
        Twiddles8 next;
        load_twiddles<K, P - 1>(next, reinterpret_cast<const double2*>(pi.inv_d), t);
#pragma unroll
        for (int k = 0; k < 8; ++k) x[k] = f_reduce(x[k], q, qinv);
        group_sync(grp, 1 << (K - 3));
        put_regs<K, P>(sm, x, t);
        group_sync(grp, 1 << (K - 3));
        get_regs<K, P - 1>(x, sm, t);
        inv8<K, P - 1>(x, next, sm, t, grp, pi);
    }
}

}  // namespace

}  // namespace vc
