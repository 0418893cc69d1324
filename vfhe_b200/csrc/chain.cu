// NTT -> product -> INTT chains in one kernel (vfhe_cuda_ntt_mul_intt_batch).
//
// The chain polynomial_RNSc_to_RNS(a), polynomial_RNSc_to_RNS(b),
// polynomial_mul_RNS_polynomial, polynomial_RNS_to_RNSc (rns_polynomial.c:311-356,
// 582-614) run as four launches moves every residue through HBM five times.  Here one
// CTA takes one (polynomial, limb) row of N = S P residues, S the ring's split degree
// and P = 2^K the per-block transform size: group g of its threads (2^(K-4) of them,
// 16 residues each) transforms block g of a, parks the spectrum in shared memory,
// transforms block g of b, and then every thread forms its output block's 16 slots of
// the incomplete product
//   out_o[x] = sum_{i <= o} a_i[x] b_{o-i}[x] + w[x] sum_{i > o} a_i[x] b_{o-i+S}[x]
// (w the pool's twist table) and runs the inverse transform of block o from registers.
// The row is read once per operand and written once.  Arithmetic is the exact FP64 form
// of fp64mod.cuh throughout: every product of two reduced operands (|.| <= q/2 + 1) is
// exact modulo q, so the canonical output equals the four-launch chain's bit for bit.
//
// Shapes: FP64 primes, N <= 2^13 (so S P <= 8192 residues of both operands fit in
// shared memory: 17 N bytes), P from 2^9 to 2^13 (a block's threads are whole warps,
// so each group meets at its own named barrier).
#include <cuda_runtime.h>

#include <mutex>

#include "engine.cuh"
#include "ntt_f64_r8.cuh"

namespace vc {

namespace {

struct ChainLimbs {
    uint32_t p[kMaxLimbs];  // pool index of each limb slot's prime
};

// Ring products take their tile addresses split at every size (2^12, 1200 rows: 82.0 us, 84.0
// whole).  Blocks of 2^11 points in a split ring keep 16 consecutive residues a thread between
// the transforms: the spectra stay in shared memory, so the coalesced edge pass saves no global
// access, and its wide twiddle loads cost more there than its fewer bank conflicts give (us,
// edge and linear: (11, 2) 192 rows 26.4 and 24.6, 1200 rows 102.4 and 98.4; (11, 4) 1200 rows
// 221.4 and 216.9; but (10, 4) 95.8 and 101.5, (9, 2) 26.7 and 28.7, (11, 1) 40.9 and 43.0).
template <int K, int S>
constexpr TileForm chain_form() {
    return K == 11 && S > 1 ? kLinear : kSplit;
}

// Up to 128 registers for 256-thread CTAs (two per SM, 70 KB of shared memory each at
// N = 4096; a three-per-SM cap of 85 registers spilled 100-190 bytes per thread) and
// 512-thread CTAs (N = 8192, 139 KB, one per SM); smaller CTAs are left to the compiler.
template <int K, int S>
__global__ void __launch_bounds__(S << (K - 4), (S << (K - 4)) <= 256 ? 2 : 1) k_chain_f(uint64_t* __restrict__ out, const uint64_t* __restrict__ a,
                                                          const uint64_t* __restrict__ b,
                                                          const __grid_constant__ ChainLimbs cl,
                                                          const PrimeInfo* __restrict__ primes, int nl) {
    constexpr int TPT = 1 << (K - 4), P = 1 << K, PADDED = P + (P >> 4);
    constexpr bool GROUP = S > 1;
    constexpr TileForm F = chain_form<K, S>();
    extern __shared__ __align__(128) double csm[];
    double* spec = csm;            // [S][PADDED]: a's spectra, reduced, at pad(edge_base) + pad(edge_step)
    double* ex = csm + S * PADDED;  // [S][PADDED]: each block's exchanges, then b's spectra
    const int g = threadIdx.x / TPT;
    const int t = threadIdx.x - g * TPT;
    const long long row = blockIdx.x;  // polynomial * nl + limb slot
    const int slot = (int)(row % nl);
    const PrimeInfo& pi = primes[cl.p[slot]];
    const double q = pi.qd, qinv = pi.qinv;
    const long long off = row * (long long)(S * P) + (long long)g * P;
    double* exg = ex + g * PADDED;
    const int eb = edge_base<K, F>(t), pe = pad(eb);  // steps have bits that bases lack: pad adds up

    Tile tile;
    tile.hi = 0;
    tile.pi = &pi;
    tile.dst = nullptr;
    double x[16];
    // a's block g
    tile.src = a + off;
    tile_fwd_regs<K, false, false, GROUP, F>(tile, K, false, exg, t, x, g);
#pragma unroll
    for (int m = 0; m < 16; ++m) spec[g * PADDED + pe + pad(edge_step<K, F>(m))] = f_reduce(x[m], q, qinv);
    tile_sync<K, GROUP>(g);  // the block's last exchange reads are over before b's first write
    // b's block g.  Its twiddles are a's again; the prime's address goes through an
    // opaque move so that the compiler reloads them instead of keeping a's ~90 registers
    // of twiddles alive across both transforms.
    tile.src = b + off;
    const PrimeInfo* pib;
    asm volatile("mov.b64 %0, %1;" : "=l"(pib) : "l"(&pi));
    tile.pi = pib;
    tile_fwd_regs<K, false, false, GROUP, F>(tile, K, false, exg, t, x, g);
    if constexpr (S == 1) {
        // pointwise: this thread's own slots of a's spectrum (written by this thread)
#pragma unroll
        for (int m = 0; m < 16; ++m) {
            const double w = f_reduce(x[m], q, qinv);
            x[m] = f_mulmod(spec[pe + pad(edge_step<K, F>(m))], w, __dmul_rn(w, qinv), q);  // |x| <= 3q/4
        }
    } else {
        tile_sync<K, GROUP>(g);  // the block's exchanges are over: its buffer takes b's spectrum
#pragma unroll
        for (int m = 0; m < 16; ++m) exg[pe + pad(edge_step<K, F>(m))] = f_reduce(x[m], q, qinv);
        __syncthreads();  // every block's spectra of a and b are in shared memory
        const ulonglong2* tw = reinterpret_cast<const ulonglong2*>(pi.twist) + eb;
#pragma unroll
        for (int m = 0; m < 16; ++m) {
            const int px = pe + pad(edge_step<K, F>(m));
            double acc = 0.0, wrap = 0.0;
#pragma unroll
            for (int i = 0; i < S; ++i) {
                const double u = spec[i * PADDED + px];
                if (i <= g) {
                    const double v = ex[(g - i) * PADDED + px];
                    acc = __dadd_rn(acc, f_mulmod(u, v, __dmul_rn(v, qinv), q));
                } else {
                    const double v = ex[(g - i + S) * PADDED + px];
                    wrap = __dadd_rn(wrap, f_mulmod(u, v, __dmul_rn(v, qinv), q));
                }
            }
            // at most 8 terms of at most 3q/4 each: below 6q < 2^53
            acc = f_reduce(acc, q, qinv);
            wrap = f_reduce(wrap, q, qinv);
            const uint64_t wi = tw[edge_step<K, F>(m)].x;
            const double wd = wi > pi.q / 2 ? (double)wi - q : (double)wi;
            x[m] = f_reduce(__dadd_rn(acc, f_mulmod(wrap, wd, __dmul_rn(wd, qinv), q)), q, qinv);
        }
        __syncthreads();  // every block's b spectrum is read before the exchanges reuse it
    }
    tile_inv_regs<K, true, GROUP, F>(pi, K, 0, exg, t, x, g);
    uint64_t* o = out + off;
#pragma unroll
    for (int m = 0; m < 16; ++m) o[own<K - 4>(t, m)] = f_to_canonical(x[m], q, qinv, pi.q);
}

// The same chain with 8 residues a thread (ntt_f64_r8.cuh): twice the warps a row, for the
// shapes whose rows leave an SM too few of them (16 residues: 4 warps a row at (K, S) = (9, 4),
// 8 at (10, 4)).  The kernel is bound by one block's chain of exchanges and barriers there,
// not by FP64 issue.  Three limbs, 16 -> 8 residues a thread, us per call with its launch:
//   (9, 4)   48 rows 13.4 -> 10.5, 192 rows 16.5 -> 14.4, 1200 rows 61.7 -> 50.5
//   (10, 4)  48 rows 16.5 -> 14.4, 144 rows 16.6 -> 14.4, 192 rows 24.7 -> 24.7, 1200 rows 96 -> 104
//   (11, 2)  48 rows 16.5 -> 14.5, 144 rows 16.5 -> 15.5, 1200 rows 104 -> 116
//   (12, 1)  48 rows 12.4 -> 14.4; (11, 1) and (10, 2) equal; 1024 threads spill (1.5x slower)
// Hence chain8_rows.
template <int K, int S>
__global__ void __launch_bounds__(S << (K - 3), S << (K - 3) <= 256 ? 2 : 1)
    k_chain8_f(uint64_t* __restrict__ out, const uint64_t* __restrict__ a, const uint64_t* __restrict__ b,
               const __grid_constant__ ChainLimbs cl, const PrimeInfo* __restrict__ primes, int nl) {
    constexpr int TPT = 1 << (K - 3), P = 1 << K, PADDED = P + (P >> 3), NP = Passes8<K>::count;
    extern __shared__ __align__(128) double csm[];
    double* spec = csm;             // [S][PADDED]: a's spectra, reduced
    double* ex = csm + S * PADDED;  // [S][PADDED]: each block's exchanges, then b's spectra
    const int g = threadIdx.x / TPT, t = threadIdx.x - g * TPT;
    const long long row = blockIdx.x;  // polynomial * nl + limb slot
    const PrimeInfo& pi = primes[cl.p[(int)(row % nl)]];
    const double q = pi.qd, qinv = pi.qinv;
    const double2* fwd = reinterpret_cast<const double2*>(pi.fwd_d);
    const long long off = row * (long long)(S * P) + (long long)g * P;
    double* exg = ex + g * PADDED;
    double* specg = spec + g * PADDED;
    double x[8];
    Twiddles8 tw;
    load_twiddles<K, 0>(tw, fwd, t);
#pragma unroll
    for (int m = 0; m < 8; ++m) x[m] = f_from_u64(a[off + Pass8<K, 0>::index(t, m)]);
    fwd8<K, 0>(x, tw, exg, t, g, fwd, q, qinv);
#pragma unroll
    for (int m = 0; m < 8; ++m) specg[pad8(Pass8<K, NP - 1>::index(t, m))] = f_reduce(x[m], q, qinv);
#pragma unroll
    for (int m = 0; m < 8; ++m) x[m] = f_from_u64(b[off + Pass8<K, 0>::index(t, m)]);
    load_twiddles<K, 0>(tw, fwd, t);
    fwd8<K, 0>(x, tw, exg, t, g, fwd, q, qinv);
    group_sync(g, TPT);  // the block's exchanges are over: its buffer takes b's spectrum
#pragma unroll
    for (int m = 0; m < 8; ++m) exg[pad8(Pass8<K, NP - 1>::index(t, m))] = f_reduce(x[m], q, qinv);
    __syncthreads();  // every block's spectra of a and b are in shared memory
    const ulonglong2* twist = reinterpret_cast<const ulonglong2*>(pi.twist);
#pragma unroll
    for (int m = 0; m < 8; ++m) {
        const int xs = Pass8<K, NP - 1>::index(t, m), px = pad8(xs);
        double acc = 0.0, wrap = 0.0;
#pragma unroll
        for (int i = 0; i < S; ++i) {
            const double u = spec[i * PADDED + px];
            const int k = i <= g ? g - i : g - i + S;
            const double v = ex[k * PADDED + px];
            const double p = f_mulmod(u, v, __dmul_rn(v, qinv), q);
            if (i <= g) acc = __dadd_rn(acc, p);
            else wrap = __dadd_rn(wrap, p);
        }
        // at most 8 terms of at most 3q/4 each: below 6q < 2^53
        acc = f_reduce(acc, q, qinv);
        wrap = f_reduce(wrap, q, qinv);
        const uint64_t wi = twist[xs].x;
        const double wd = wi > pi.q / 2 ? (double)wi - q : (double)wi;
        x[m] = f_reduce(__dadd_rn(acc, f_mulmod(wrap, wd, __dmul_rn(wd, qinv), q)), q, qinv);
    }
    __syncthreads();  // every block's b spectrum is read before the exchanges reuse it
    Twiddles8 twi;
    load_twiddles<K, NP - 1>(twi, reinterpret_cast<const double2*>(pi.inv_d), t);
    inv8<K, NP - 1>(x, twi, exg, t, g, pi);
#pragma unroll
    for (int m = 0; m < 8; ++m) out[off + Pass8<K, 0>::index(t, m)] = f_to_canonical(x[m], q, qinv, pi.q);
}

template <int K, int S>
constexpr size_t chain8_smem() {
    return sizeof(double) * 2 * (size_t)S * ((1 << K) + (1 << (K - 3)));
}

template <int K, int S>
constexpr size_t chain_smem() {
    return sizeof(double) * 2 * (size_t)S * ((1 << K) + (1 << (K - 4)));
}

// Most rows the 8-residue kernel takes: any number at (9, 4), one row an SM where a row is
// 512 threads in split blocks (two of the 16-residue kernel's CTAs share an SM beyond that).
// Other shapes have no such kernel.
template <int K, int S>
constexpr bool chain8_built() {
    return S > 1 && ((K == 9 && S == 4) || S << (K - 3) == 512);
}
template <int K, int S>
long long chain8_rows() {
    return K == 9 && S == 4 ? 0x7fffffffLL : sm_count();
}

template <int K, int S>
int chain_attr() {
    int e = 0;
    if (chain_smem<K, S>() > 48 * 1024)
        e = (int)cudaFuncSetAttribute(k_chain_f<K, S>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                      (int)chain_smem<K, S>());
    if constexpr (chain8_built<K, S>()) {
        if (!e && chain8_smem<K, S>() > 48 * 1024)
            e = (int)cudaFuncSetAttribute(k_chain8_f<K, S>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                          (int)chain8_smem<K, S>());
    }
    return e;
}

template <int K, int S>
int chain_launch(uint64_t* out, const uint64_t* a, const uint64_t* b, long long rows, const ChainLimbs& cl,
                 const PrimeInfo* d, int nl, cudaStream_t st) {
    // the shared-memory limit is raised at the first launch (and by prepare_chain_kernels
    // before any stream capture)
    static std::once_flag once;
    static int attr_err = 0;
    std::call_once(once, [] { attr_err = chain_attr<K, S>(); });
    if (attr_err) return attr_err;
    bool eight = false;
    if constexpr (chain8_built<K, S>()) {
        eight = rows <= chain8_rows<K, S>();
        if (eight) k_chain8_f<K, S><<<(unsigned)rows, S << (K - 3), chain8_smem<K, S>(), st>>>(out, a, b, cl, d, nl);
    }
    if (!eight) k_chain_f<K, S><<<(unsigned)rows, S << (K - 4), chain_smem<K, S>(), st>>>(out, a, b, cl, d, nl);
    note_launch();
    return (int)cudaGetLastError();
}

}  // namespace

int prepare_chain_kernels() {
    int e = chain_attr<9, 1>();
    if (!e) e = chain_attr<9, 2>();
    if (!e) e = chain_attr<9, 4>();
    if (!e) e = chain_attr<9, 8>();
    if (!e) e = chain_attr<10, 1>();
    if (!e) e = chain_attr<10, 2>();
    if (!e) e = chain_attr<10, 4>();
    if (!e) e = chain_attr<10, 8>();
    if (!e) e = chain_attr<11, 1>();
    if (!e) e = chain_attr<11, 2>();
    if (!e) e = chain_attr<11, 4>();
    if (!e) e = chain_attr<12, 1>();
    if (!e) e = chain_attr<12, 2>();
    if (!e) e = chain_attr<13, 1>();
    return e;
}

int launch_chain(IncNtt* t, uint64_t* out, const uint64_t* a, const uint64_t* b, uint64_t batch,
                 const uint32_t* limbs, uint32_t nlimbs, cudaStream_t st) {
    const uint64_t N = t->pub.N, S = t->pub.split_degree;
    const int K = t->logP;
    if (N > 8192 || K < 9 || K > 13 || nlimbs == 0 || nlimbs > (uint32_t)kMaxLimbs || batch == 0 ||
        batch * nlimbs > 0x7fffffffULL)
        return kChainUnavailable;
    if (((reinterpret_cast<uintptr_t>(out) | reinterpret_cast<uintptr_t>(a) | reinterpret_cast<uintptr_t>(b)) & 15) != 0)
        return kChainUnavailable;
    ChainLimbs cl;
    for (uint32_t k = 0; k < nlimbs; ++k) {
        if (limbs[k] >= t->pub.l || !t->info[limbs[k]].fp64) return kChainUnavailable;
        cl.p[k] = limbs[k];
    }
    const long long rows = (long long)(batch * nlimbs);
    switch (K * 16 + (int)S) {
        case 9 * 16 + 1: return chain_launch<9, 1>(out, a, b, rows, cl, t->d_info, (int)nlimbs, st);
        case 9 * 16 + 2: return chain_launch<9, 2>(out, a, b, rows, cl, t->d_info, (int)nlimbs, st);
        case 9 * 16 + 4: return chain_launch<9, 4>(out, a, b, rows, cl, t->d_info, (int)nlimbs, st);
        case 9 * 16 + 8: return chain_launch<9, 8>(out, a, b, rows, cl, t->d_info, (int)nlimbs, st);
        case 10 * 16 + 1: return chain_launch<10, 1>(out, a, b, rows, cl, t->d_info, (int)nlimbs, st);
        case 10 * 16 + 2: return chain_launch<10, 2>(out, a, b, rows, cl, t->d_info, (int)nlimbs, st);
        case 10 * 16 + 4: return chain_launch<10, 4>(out, a, b, rows, cl, t->d_info, (int)nlimbs, st);
        case 10 * 16 + 8: return chain_launch<10, 8>(out, a, b, rows, cl, t->d_info, (int)nlimbs, st);
        case 11 * 16 + 1: return chain_launch<11, 1>(out, a, b, rows, cl, t->d_info, (int)nlimbs, st);
        case 11 * 16 + 2: return chain_launch<11, 2>(out, a, b, rows, cl, t->d_info, (int)nlimbs, st);
        case 11 * 16 + 4: return chain_launch<11, 4>(out, a, b, rows, cl, t->d_info, (int)nlimbs, st);
        case 12 * 16 + 1: return chain_launch<12, 1>(out, a, b, rows, cl, t->d_info, (int)nlimbs, st);
        case 12 * 16 + 2: return chain_launch<12, 2>(out, a, b, rows, cl, t->d_info, (int)nlimbs, st);
        case 13 * 16 + 1: return chain_launch<13, 1>(out, a, b, rows, cl, t->d_info, (int)nlimbs, st);
        default: return kChainUnavailable;
    }
}

}  // namespace vc
