// CGGI bootstrap over the 32-bit torus with FP64 complex-FFT external products.
//
// The algorithm is the published TFHE bootstrap (Chillotti, Gama, Georgieva,
// Izabachene, J. Cryptology 33, 2020) with the reference's CGGI16 orchestration
// (modules/fhe/python/src/vfhe/fhe/cggi16.py:46-128: rotation with a half-box
// offset, CMUX(acc, acc X^a_i) per LWE coefficient, extraction at coefficient 0),
// then a base-2^kb LWE key switch back to the input key.  Conventions are those of
// oracle/cggi_torus_oracle.c (the exact-integer checker): uint32 torus, GLWE phase
// b - a S, signed gadget digits, GGSW row (component c, level l) at c * levels + l.
//
// Negacyclic products through a half-size complex FFT: a real polynomial p of N
// coefficients folds to z_j = p_j + i p_{j+M}, M = N/2, its residue modulo X^M - i (the
// other factor X^M + i of X^N + 1 carries the conjugate).  The forward transform splits
// X^m - e^{i f} = (X^{m/2} - w)(X^{m/2} + w), w = e^{i f/2}, down to degree one: element i
// of the result is p at the root zeta^{4k+1}, zeta = e^{i pi/N}, k = i with its bits
// reversed, so pointwise products of spectra are spectra of negacyclic products.  The
// inverse undoes the same splits (bit-reversed in, natural out) and scales by 1/M.  No
// permutation pass and no separate twist.  Key spectra come from the same forward code,
// so both operands are in the same order.
//
// Precision: digits |d| <= 2^(g-1) (64 at base 2^7), key values as signed 32-bit,
// 2 levels-by-components rows x N terms: sums below 2^50; FP64 (53-bit) FFTs then
// round each coefficient to the nearest integer, usually exact; the tests measure
// the maximum deviation from the exact integer product.
//
// One persistent launch runs whole blind rotations: each CTA owns one LWE at a time,
// keeps the accumulator and the spectra in shared memory for all n CMUX steps, and
// reads step i's key spectra (same for every CTA, so they stay in L2) directly.
#include <cuda_runtime.h>
#include <math.h>
#include <string.h>

#include <mutex>
#include <vector>

#include "engine.cuh"

namespace vc {

namespace {

constexpr int kMaxLevels = 4;

// Twiddles of the register-blocked passes (ct_pass below), per N.  The block b of a pass
// over index bits LO..LO+2 starts at split level s = log2 M - 3 - LO; it needs
// w1 = w(s, b), w2 = w(s + 1, 2b), w3 = w(s + 2, 4b) and w3p = w(s + 2, 4b + 2), where
// w(s, b) = e^{i f(s, b)/2}, f(0, 0) = pi/2, f(s + 1, 2b) = f(s, b)/2 and f(s + 1, 2b + 1)
// = f(s, b)/2 + pi: the split of an odd block uses i times its even sibling's w.  Each
// pass stores its w1, w2, w3, w3p as four arrays over the blocks, so that a warp's
// lookups are consecutive or broadcast.
struct FourierTables {
    int N = 0;
    double2* d_tw = nullptr;
};

// split level s, block b -> the angle of w(s, b)
long double split_angle(int s, int b) {
    long double f = 1.570796326794896619231321691639751442L;  // pi/2
    for (int k = s - 1; k >= 0; --k) f = f / 2 + (((b >> k) & 1) ? 3.141592653589793238462643383279502884L : 0.0L);
    return f / 2;
}

// low index bit of pass p of a 2^logm-point transform (three bits a pass from the top, the
// last pass at bit 0) and the number of passes
int pass_lo(int logm, int p) { return p < logm / 3 ? logm - 3 * (p + 1) : 0; }
int pass_count(int logm) { return (logm + 2) / 3; }

std::mutex g_ft_mu;
std::vector<FourierTables*> g_ft;

const FourierTables* fourier_tables(int N) {
    std::lock_guard<std::mutex> lk(g_ft_mu);
    for (const FourierTables* t : g_ft)
        if (t->N == N) return t;
    int logm = 0;
    while ((2 << logm) < N) ++logm;
    std::vector<double2> tw;
    for (int p = 0; p < pass_count(logm); ++p) {
        const int lo = pass_lo(logm, p), s = logm - 3 - lo, nb = 1 << s;
        for (int q = 0; q < 4; ++q)
            for (int b = 0; b < nb; ++b) {
                const long double a = q == 0   ? split_angle(s, b)
                                      : q == 1 ? split_angle(s + 1, 2 * b)
                                               : split_angle(s + 2, 4 * b + (q == 3 ? 2 : 0));
                tw.push_back(make_double2((double)cosl(a), (double)sinl(a)));
            }
    }
    FourierTables t;
    t.N = N;
    if (cudaMalloc(&t.d_tw, sizeof(double2) * tw.size()) != cudaSuccess ||
        cudaMemcpy(t.d_tw, tw.data(), sizeof(double2) * tw.size(), cudaMemcpyHostToDevice) != cudaSuccess ||
        cudaStreamSynchronize(0) != cudaSuccess)  // the upload has landed before other streams read it
        return nullptr;
    g_ft.push_back(new FourierTables(t));
    return g_ft.back();
}

// Table loads issued where they stand: ordinary (coherent) loads that neither the
// compiler nor the assembler moves across the exchange barriers.  Through the read-only
// path they count as invariant, and every level's key and twiddle loads of a step would
// be hoisted to its top, keeping well over a hundred values live in registers.
__device__ __forceinline__ double2 ld_table(const double2* p) {
    double2 v;
    asm volatile("ld.global.v2.f64 {%0, %1}, [%2];" : "=d"(v.x), "=d"(v.y) : "l"(p));
    return v;
}

__device__ __forceinline__ int modswitch(uint32_t v, int logN2) {
    return (int)((((uint64_t)v + (1ULL << (31 - logN2))) >> (32 - logN2)) & ((1ULL << logN2) - 1));
}

// acc X^e at coefficient k (negacyclic, 0 <= e < 2N)
template <int N>
__device__ __forceinline__ uint32_t rot_at(const uint32_t* p, int k, int e) {
    int s = k - e;
    s = s < 0 ? s + 2 * N : s;
    return s < N ? p[s] : (uint32_t)(0u - p[s - N]);
}

// ---- register-blocked radix-8 FFT passes
//
// An M-point transform (M = 2^LOGM) of one array is done by M/8 threads holding 8
// values each.  Pass p covers index bits [LO, LO + NST): thread t holds the elements
// pidx<LO>(t, k), k < 8 (k supplies bits LO..LO+2), so all butterflies of the pass are
// in registers; passes exchange through shared memory with an XOR swizzle that keeps
// every pass's accesses free of bank conflicts.  Forward: LOGM/3 full passes from the
// top bits, then one partial pass (LOGM mod 3 stages) at bit 0; the inverse runs the
// same passes in reverse.  The final forward pass leaves element f = 8t + k in thread
// t, which is also the order of the key spectra in memory (position k * M/8 + t), so
// the multiply-accumulate reads both coalesced.

template <int LO>
__device__ __forceinline__ int pidx(int t, int k) {
    return ((t >> LO) << (LO + 3)) | (k << LO) | (t & ((1 << LO) - 1));
}

__device__ __forceinline__ int swz(int i) { return i ^ ((i >> 3) & 7); }

template <int LOGM, int P>
struct PassOf {
    static constexpr int FULL = LOGM / 3;
    static constexpr int LO = P < FULL ? LOGM - 3 * (P + 1) : 0;
    static constexpr int NST = P < FULL ? 3 : LOGM % 3;
    static constexpr int BLOCKS = 1 << (LOGM - 3 - LO);
    // entries of the twiddle table before this pass's
    static constexpr int tw_offset() {
        int n = 0;
        for (int p = 0; p < P; ++p) n += 4 << (LOGM - 3 - (p < FULL ? LOGM - 3 * (p + 1) : 0));
        return n;
    }
};

template <int LOGM>
struct Passes {
    static constexpr int count = (LOGM + 2) / 3;
    static constexpr int tw_entries = PassOf<LOGM, count - 1>::tw_offset() + 4 * PassOf<LOGM, count - 1>::BLOCKS;
};

// Split of one block pair: (u, v) -> (u + w v, u - w v), both sides by FMAs: fewer
// roundings than a product, a sum and a difference in as many operations.
__device__ __forceinline__ void split(double2& u, double2& v, double2 w) {
    const double2 a = u, b = v;
    u.x = __fma_rn(w.x, b.x, __fma_rn(-w.y, b.y, a.x));
    u.y = __fma_rn(w.x, b.y, __fma_rn(w.y, b.x, a.y));
    v.x = __fma_rn(-w.x, b.x, __fma_rn(w.y, b.y, a.x));
    v.y = __fma_rn(-w.x, b.y, __fma_rn(-w.y, b.x, a.y));
}
__device__ __forceinline__ void split_i(double2& u, double2& v, double2 w) {  // by i w
    split(u, v, make_double2(-w.y, w.x));
}
// The inverse up to the factor 2: (u, v) -> (u + v, (u - v) conj(w)).
__device__ __forceinline__ void join(double2& u, double2& v, double2 w) {
    const double dx = u.x - v.x, dy = u.y - v.y;
    u = make_double2(u.x + v.x, u.y + v.y);
    v = make_double2(__fma_rn(dx, w.x, dy * w.y), __fma_rn(dy, w.x, -dx * w.y));
}
__device__ __forceinline__ void join_i(double2& u, double2& v, double2 w) {  // by i w
    join(u, v, make_double2(-w.y, w.x));
}

struct PassTwiddles {
    double2 w1, w2, w3, w3p;
};

template <int LOGM, int P>
__device__ __forceinline__ PassTwiddles pass_twiddles(const double2* tw, int t) {
    using Q = PassOf<LOGM, P>;
    PassTwiddles r;
    if constexpr (P == 0) {  // one block: constants e^{i pi/4}, e^{i pi/8}, e^{i pi/16}, e^{i 5 pi/16}
        r.w1 = make_double2(0.70710678118654752440, 0.70710678118654752440);
        r.w2 = make_double2(0.92387953251128675613, 0.38268343236508977173);
        r.w3 = make_double2(0.98078528040323044913, 0.19509032201612826785);
        r.w3p = make_double2(0.55557023301960222474, 0.83146961230254523708);
    } else {
        const double2* T = tw + Q::tw_offset() + (t >> Q::LO);
        r.w1 = T[0];
        r.w2 = T[Q::BLOCKS];
        r.w3 = T[2 * Q::BLOCKS];
        r.w3p = T[3 * Q::BLOCKS];
    }
    return r;
}

// The last NST of the three split levels of a pass (NST < 3: the partial pass at bit 0).
template <int LOGM, int P>
__device__ __forceinline__ void split_pass(double2 (&v)[8], int t, const double2* tw) {
    constexpr int NST = PassOf<LOGM, P>::NST;
    const PassTwiddles T = pass_twiddles<LOGM, P>(tw, t);
    if constexpr (NST >= 3) {
#pragma unroll
        for (int k = 0; k < 4; ++k) split(v[k], v[k + 4], T.w1);
    }
    if constexpr (NST >= 2) {
        split(v[0], v[2], T.w2);
        split(v[1], v[3], T.w2);
        split_i(v[4], v[6], T.w2);
        split_i(v[5], v[7], T.w2);
    }
    split(v[0], v[1], T.w3);
    split_i(v[2], v[3], T.w3);
    split(v[4], v[5], T.w3p);
    split_i(v[6], v[7], T.w3p);
}

template <int LOGM, int P>
__device__ __forceinline__ void join_pass(double2 (&v)[8], int t, const double2* tw) {
    constexpr int NST = PassOf<LOGM, P>::NST;
    const PassTwiddles T = pass_twiddles<LOGM, P>(tw, t);
    join(v[0], v[1], T.w3);
    join_i(v[2], v[3], T.w3);
    join(v[4], v[5], T.w3p);
    join_i(v[6], v[7], T.w3p);
    if constexpr (NST >= 2) {
        join(v[0], v[2], T.w2);
        join(v[1], v[3], T.w2);
        join_i(v[4], v[6], T.w2);
        join_i(v[5], v[7], T.w2);
    }
    if constexpr (NST >= 3) {
#pragma unroll
        for (int k = 0; k < 4; ++k) join(v[k], v[k + 4], T.w1);
    }
}

template <int LO>
__device__ __forceinline__ void put8(double2* a, const double2 (&v)[8], int t) {
#pragma unroll
    for (int k = 0; k < 8; ++k) a[swz(pidx<LO>(t, k))] = v[k];
}

template <int LO>
__device__ __forceinline__ void get8(double2 (&v)[8], const double2* a, int t) {
#pragma unroll
    for (int k = 0; k < 8; ++k) v[k] = a[swz(pidx<LO>(t, k))];
}

// ---- group-split external product
//
// The GLWE of one LWE is handled by two groups of TPA = M/8 threads, group c owning
// component c: it forms the LEVELS digit polynomials of component c (one after another,
// each transformed in registers with exchanges through the group's own two shared
// buffers under a named barrier of TPA threads), and multiplies each spectrum with the
// GGSW rows (c, level) of both outputs, keeping the two partial sums in registers.  The
// groups then swap the partial sums of each other's output through shared memory (the
// only point where they meet) and each runs the inverse transform of output c, adding
// the rounded result into its own accumulator component.  Every thread works in every
// phase, and a group never waits for the other group except at the swap.

__device__ __forceinline__ void group_bar(int id, int threads) {
    asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(threads) : "memory");
}

// Signed gadget digits without a per-digit carry loop: adding B/2 to every base-B
// digit of the rounded value r (mod B^levels) makes digit l of the sum, minus B/2, the
// balanced digit in [-B/2, B/2) (the representation is unique, so it equals the
// carry-propagating decomposition).  Digit 0 is the most significant.
struct Gadget {
    int total;       // base_log * levels
    int base_log;
    uint32_t mask;   // 2^total - 1
    uint32_t half;   // sum over digits of B/2 at each digit position
    double bias;     // -(2^52 + B/2): takes 2^52 + a digit field to the balanced digit
    int small_sums;  // every coefficient of an external product stays below 2^51
};

inline Gadget make_gadget(int N, int base_log, int levels) {
    Gadget g;
    g.total = base_log * levels;
    g.base_log = base_log;
    g.mask = g.total >= 32 ? 0xFFFFFFFFu : ((1u << g.total) - 1u);
    g.half = 0;
    for (int l = 0; l < levels; ++l) g.half += 1u << (base_log * l + base_log - 1);
    g.bias = -(4503599627370496.0 + (double)(1u << (base_log - 1)));
    // 2 levels rows of N products of a digit (at most B/2) and a signed 32-bit word
    g.small_sums = 2.0 * levels * N * (double)(1u << (base_log - 1)) * 2147483648.0 < 2251799813685248.0;
    return g;
}

__device__ __forceinline__ uint32_t gadget_prepare(uint32_t v, const Gadget& g) {
    const uint32_t r = g.total >= 32 ? v : (uint32_t)(((uint64_t)v + (1ULL << (31 - g.total))) >> (32 - g.total));
    return (r + g.half) & g.mask;
}

template <int LEVELS>
__device__ __forceinline__ double gadget_digit(uint32_t prepared, const Gadget& g, int l) {
    const int sh = g.base_log * (LEVELS - 1 - l);
    const uint32_t field = (prepared >> sh) & ((1u << g.base_log) - 1u);
    // 2^52 + field, less 2^52 + B/2: exact, and off the slow integer-to-double conversions
    return __dadd_rn(__hiloint2double(0x43300000, (int)field), g.bias);
}

// Nearest integer of z 2^-LOGM modulo 2^32; `rounded` receives the integer itself.  Below
// 2^51 (Gadget::small_sums) it is the low word of the sum with 1.5 2^52.
template <int LOGM>
__device__ __forceinline__ uint32_t round_scaled(double z, const Gadget& g, double& rounded) {
    constexpr double magic = 6755399441055744.0, scale = 1.0 / (double)(1 << LOGM);
    if (g.small_sums) {
        const double r = __fma_rn(z, scale, magic);
        rounded = r - magic;
        return (uint32_t)__double2loint(r);
    }
    const long long r = __double2ll_rn(z * scale);
    rounded = (double)r;
    return (uint32_t)r;
}

// Exchange through buffer `b`: registers in the layout of pass PFROM, out in pass PTO's.
template <int LOGM, int PFROM, int PTO>
__device__ __forceinline__ void exchange(double2 (&v)[8], double2* b, int t, int bar) {
    put8<PassOf<LOGM, PFROM>::LO>(b, v, t);
    group_bar(bar, (1 << LOGM) / 8);
    get8<PassOf<LOGM, PTO>::LO>(v, b, t);
}

// forward passes P .. count-1, registers holding pass P-1's output; exchange e uses buffer e & 1
template <int LOGM, int P, int E>
__device__ __forceinline__ void group_fwd(double2 (&v)[8], double2* bufs, int t, int bar, const double2* tw) {
    if constexpr (P < Passes<LOGM>::count) {
        exchange<LOGM, P - 1, P>(v, bufs + (E & 1) * (1 << LOGM), t, bar);
        split_pass<LOGM, P>(v, t, tw);
        group_fwd<LOGM, P + 1, E + 1>(v, bufs, t, bar, tw);
    }
}

// inverse passes P down to 0, registers holding pass P+1's output
template <int LOGM, int P, int E>
__device__ __forceinline__ void group_inv(double2 (&v)[8], double2* bufs, int t, int bar, const double2* tw) {
    if constexpr (P >= 0) {
        exchange<LOGM, P + 1, P>(v, bufs + (E & 1) * (1 << LOGM), t, bar);
        join_pass<LOGM, P>(v, t, tw);
        group_inv<LOGM, P - 1, E + 1>(v, bufs, t, bar, tw);
    }
}

// v += x k
__device__ __forceinline__ void cmac(double2& v, double2 x, double2 k) {
    v.x = __fma_rn(x.x, k.x, __fma_rn(-x.y, k.y, v.x));
    v.y = __fma_rn(x.x, k.y, __fma_rn(x.y, k.x, v.y));
}

template <int LOGM, int LEVELS>
struct GroupSplit {
    static constexpr int M = 1 << LOGM, N = 2 * M, TPA = M / 8, THREADS = 2 * TPA;
    static constexpr int NP = Passes<LOGM>::count;
    static constexpr int FWD_EX = LEVELS * (NP - 1);  // exchanges of the forward transforms
    // acc[2][N] uint32 | bufs[2 groups][2][M] double2 | xbufs[2][M] double2 | twiddles
    static constexpr size_t smem = sizeof(uint32_t) * 2 * N + sizeof(double2) * (6 * M + Passes<LOGM>::tw_entries);
    // resident blocks the register budget is sized for: about 168 registers a thread
    static constexpr int min_ctas = 65536 / (THREADS * 168) > 0 ? 65536 / (THREADS * 168) : 1;
};

// Rounded, digit-prepared coefficients j and j + M, j = k TPA + t (pass 0's layout), of
// component c of the block's acc X^ai - acc.
template <int LOGM>
__device__ __forceinline__ void rotated_difference(uint32_t (&plo)[8], uint32_t (&phi)[8], const uint32_t* pc, int ai,
                                                   int t, const Gadget& gd) {
    constexpr int M = 1 << LOGM, N = 2 * M, TPA = M / 8;
#pragma unroll
    for (int k = 0; k < 8; ++k) {
        const int j = k * TPA + t;
        plo[k] = gadget_prepare(rot_at<N>(pc, j, ai) - pc[j], gd);
        phi[k] = gadget_prepare(rot_at<N>(pc, j + M, ai) - pc[j + M], gd);
    }
}

// One external product on the block's GLWE, by group c (thread t of TPA).  Source
// (MODE 0): acc X^ai - acc from the block's accumulator; (MODE 1) the GLWE `src`.
// Result: MODE 0 adds the rounded output c into acc component c; MODE 1 writes it to
// dst and returns the largest distance of an unrounded coefficient to its integer.
// bufs: this group's two exchange buffers; xbufs: the two groups' receive buffers
// (xbufs + c M collects output c's share from the other group).  The caller has made
// the accumulator's last writes visible and the receive buffers free (__syncthreads).
template <int LOGM, int LEVELS, int MODE>
__device__ __forceinline__ double group_ext_product(uint32_t* acc, double2* bufs, double2* xbufs, int c, int t,
                                                    const double2* __restrict__ key, int ai, const Gadget& gd,
                                                    const uint32_t* __restrict__ src, uint32_t* __restrict__ dst,
                                                    const double2* tw) {
    using G = GroupSplit<LOGM, LEVELS>;
    constexpr int M = G::M, N = G::N, TPA = G::TPA, NP = G::NP;
    // Fresh copies of the thread coordinates: every shared-memory and table address of
    // the step derives from them, and without this the compiler hoists all of those
    // addresses out of the caller's step loop and keeps them live in registers.
    asm volatile("mov.b32 %0, %0;" : "+r"(t));
    asm volatile("mov.b32 %0, %0;" : "+r"(c));
    const int bar = 1 + c;
    uint32_t plo[8], phi[8];
    if (MODE == 0) {
        rotated_difference<LOGM>(plo, phi, acc + c * N, ai, t, gd);
    } else {
#pragma unroll
        for (int k = 0; k < 8; ++k) {
            plo[k] = gadget_prepare(src[c * N + k * TPA + t], gd);
            phi[k] = gadget_prepare(src[c * N + k * TPA + t + M], gd);
        }
    }
    // both outputs' partial sums stay in registers over the levels; output 1 - c's goes to
    // the other group once, at the end
    double2 pm[8], po[8];
#pragma unroll
    for (int k = 0; k < 8; ++k) pm[k] = po[k] = make_double2(0.0, 0.0);
#pragma unroll
    for (int l = 0; l < LEVELS; ++l) {
        double2 v[8];
#pragma unroll
        for (int k = 0; k < 8; ++k)
            v[k] = make_double2(gadget_digit<LEVELS>(plo[k], gd, l), gadget_digit<LEVELS>(phi[k], gd, l));
        split_pass<LOGM, 0>(v, t, tw);
        if (l == 0) group_fwd<LOGM, 1, 0>(v, bufs, t, bar, tw);
        else if (l == 1) group_fwd<LOGM, 1, (NP - 1)>(v, bufs, t, bar, tw);
        else if (l == 2) group_fwd<LOGM, 1, 2 * (NP - 1)>(v, bufs, t, bar, tw);
        else group_fwd<LOGM, 1, 3 * (NP - 1)>(v, bufs, t, bar, tw);
        // spectrum element 8 t + k meets key position k TPA + t (key order)
        const double2* km = key + (long long)((c * LEVELS + l) * 2 + c) * M;
        const double2* ko = key + (long long)((c * LEVELS + l) * 2 + (1 - c)) * M;
#pragma unroll
        for (int k = 0; k < 8; ++k) cmac(pm[k], v[k], ld_table(&km[k * TPA + t]));
#pragma unroll
        for (int k = 0; k < 8; ++k) cmac(po[k], v[k], ld_table(&ko[k * TPA + t]));
    }
    put8<0>(xbufs + (1 - c) * M, po, t);
    __syncthreads();  // both groups' contributions to each other's output are in place
    {
        double2 other[8];
        get8<0>(other, xbufs + c * M, t);
#pragma unroll
        for (int k = 0; k < 8; ++k) pm[k] = make_double2(pm[k].x + other[k].x, pm[k].y + other[k].y);
    }
    join_pass<LOGM, NP - 1>(pm, t, tw);
    group_inv<LOGM, NP - 2, G::FWD_EX>(pm, bufs, t, bar, tw);
    // unfold, round (element j = k TPA + t)
    double worst = 0.0;
#pragma unroll
    for (int k = 0; k < 8; ++k) {
        const int j = k * TPA + t;
        double rx, ry;
        const uint32_t lo = round_scaled<LOGM>(pm[k].x, gd, rx), hi = round_scaled<LOGM>(pm[k].y, gd, ry);
        if (MODE == 0) {
            acc[c * N + j] += lo;
            acc[c * N + j + M] += hi;
        } else {
            constexpr double inv_m = 1.0 / (double)M;
            dst[c * N + j] = lo;
            dst[c * N + j + M] = hi;
            worst = fmax(worst, fmax(fabs(pm[k].x * inv_m - rx), fabs(pm[k].y * inv_m - ry)));
        }
    }
    return worst;
}

// Extracted LWE of the accumulator at coefficient 0 (threads t of T): mask, then body.
template <int N>
__device__ __forceinline__ void extract_lwe(uint32_t* o, const uint32_t* acc, int t, int T) {
    for (int k = t; k < N; k += T) o[k] = k == 0 ? acc[0] : (uint32_t)(0u - acc[N - k]);
    if (t == 0) o[N] = acc[N];
}

// Blind rotation + sample extraction of B LWEs (in: [B][n+1], mask then body) into
// out [B][N+1] (extracted mask, body).  bsk_f: [n][2 levels][2][M] spectra in key order.
// Block: two groups of M/8 threads (one per GLWE component); persistent over the LWEs.
//
// Bound by shared-memory and L1 traffic (exchanges, key spectra): about 500 KB per LWE and
// step at N = 1024, 3 levels, 4000 cycles at 128 bytes a clock, beside 2900 cycles of the
// FP64 pipe.  Keeping both outputs' sums in registers takes 130 KB a step off that, and
// splits without a twist 100 KB.  4096 rotations at n = 630: 61 ms before, 51 ms with both.
// (Differences as 2u - (u + w v), six operations a split instead of eight, ran in 48 ms but
// left coefficients 4 to 8% further from their integers.)
template <int LOGM, int LEVELS>
__global__ void __launch_bounds__(GroupSplit<LOGM, LEVELS>::THREADS, GroupSplit<LOGM, LEVELS>::min_ctas)
    k_cggi_fft_bootstrap(uint32_t* __restrict__ out, const uint32_t* __restrict__ in, long long B,
                         const double2* __restrict__ bsk_f, const uint32_t* __restrict__ tv, int n, Gadget gd,
                         uint32_t offset, const double2* __restrict__ g_tw) {
    using G = GroupSplit<LOGM, LEVELS>;
    constexpr int M = G::M, N = G::N, TPA = G::TPA, R = 2 * LEVELS;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    uint32_t* acc = reinterpret_cast<uint32_t*>(smem_raw);
    double2* bufs_all = reinterpret_cast<double2*>(acc + 2 * N);
    const int c = threadIdx.x / TPA, t = threadIdx.x - c * TPA;
    double2* bufs = bufs_all + c * 2 * M;
    double2* xbufs = bufs_all + 4 * M;
    // the transforms' twiddles, read from shared memory
    double2* stw = bufs_all + 6 * M;
    for (int k = threadIdx.x; k < Passes<LOGM>::tw_entries; k += blockDim.x) stw[k] = g_tw[k];
    __syncthreads();
    constexpr int logN2 = LOGM + 2;
    for (long long lwe = blockIdx.x; lwe < B; lwe += gridDim.x) {
        const uint32_t* a = in + lwe * (long long)(n + 1);
        const int rb = modswitch(a[n] + offset, logN2);
        const int e0 = (2 * N - rb) & (2 * N - 1);
        for (int k = t; k < N; k += TPA) acc[c * N + k] = c == 0 ? 0u : rot_at<N>(tv, k, e0);
        for (int i = 0; i < n; ++i) {
            // accumulator writes visible; last step's receive-buffer reads done
            __syncthreads();
            const int ai = modswitch(__ldg(a + i), logN2);
            group_ext_product<LOGM, LEVELS, 0>(acc, bufs, xbufs, c, t, bsk_f + (long long)i * R * 2 * M, ai, gd,
                                               nullptr, nullptr, stw);
        }
        __syncthreads();
        extract_lwe<N>(out + lwe * (long long)(N + 1), acc, threadIdx.x, G::THREADS);
        __syncthreads();  // extraction reads done before the next LWE rewrites acc
    }
}

// ---- one rotation on a wide block
//
// The same blind rotation with 2 LEVELS groups of M/8 threads, one per gadget digit
// polynomial, so that a step's forward transforms run side by side instead of one after
// another: for batches that leave SMs without a second block, where the latency of a step
// counts.  The groups leave their spectra in their exchange buffers, every thread of the
// block multiplies: position p of both outputs (key order) sums the spectra with the key
// rows, read into registers one step ahead where the register budget allows; groups 0 and 1
// run the two inverse transforms.  A step moves about 590 KB through shared memory and L1
// (4700 cycles, 65% of the 3.8 us a step takes at N = 1024, 3 levels) and has four block
// barriers.  7 LWEs at n = 630: 7.6 ms of blind rotation before (one block of 128 threads
// each), 2.4 ms on wide blocks.
template <int LOGM, int LEVELS>
struct WideSplit {
    static constexpr int M = 1 << LOGM, N = 2 * M, TPA = M / 8, GROUPS = 2 * LEVELS;
    static constexpr int THREADS = M;  // one multiply position a thread (N <= 1024, so 2 LEVELS <= 8 groups fit)
    // a thread's 4 LEVELS key values are loaded a step ahead where they fit 128 registers
    static constexpr bool AHEAD = LEVELS <= 3;
    // acc[2][N] uint32 | bufs[GROUPS][M] | out[2][M] double2 | twiddles
    static constexpr size_t smem =
        sizeof(uint32_t) * 2 * N + sizeof(double2) * ((GROUPS + 2) * M + Passes<LOGM>::tw_entries);
};

// forward passes P .. count-1 through one buffer (a barrier before and after each write)
template <int LOGM, int P>
__device__ __forceinline__ void wide_fwd(double2 (&v)[8], double2* buf, int t, int bar, const double2* tw) {
    if constexpr (P < Passes<LOGM>::count) {
        if (P > 1) group_bar(bar, (1 << LOGM) / 8);
        exchange<LOGM, P - 1, P>(v, buf, t, bar);
        split_pass<LOGM, P>(v, t, tw);
        wide_fwd<LOGM, P + 1>(v, buf, t, bar, tw);
    }
}

// inverse passes P down to 0 through one buffer
template <int LOGM, int P>
__device__ __forceinline__ void wide_inv(double2 (&v)[8], double2* buf, int t, int bar, const double2* tw) {
    if constexpr (P >= 0) {
        if (P < Passes<LOGM>::count - 2) group_bar(bar, (1 << LOGM) / 8);
        exchange<LOGM, P + 1, P>(v, buf, t, bar);
        join_pass<LOGM, P>(v, t, tw);
        wide_inv<LOGM, P - 1>(v, buf, t, bar, tw);
    }
}

template <int LOGM, int LEVELS>
__global__ void __launch_bounds__(WideSplit<LOGM, LEVELS>::THREADS)
    k_cggi_fft_bootstrap_wide(uint32_t* __restrict__ out, const uint32_t* __restrict__ in,
                              const double2* __restrict__ bsk_f, const uint32_t* __restrict__ tv, int n, Gadget gd,
                              uint32_t offset, const double2* __restrict__ g_tw) {
    using W = WideSplit<LOGM, LEVELS>;
    constexpr int M = W::M, N = W::N, TPA = W::TPA, GROUPS = W::GROUPS, T = W::THREADS, R = 2 * LEVELS;
    constexpr int NP = Passes<LOGM>::count;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    uint32_t* acc = reinterpret_cast<uint32_t*>(smem_raw);
    double2* bufs = reinterpret_cast<double2*>(acc + 2 * N);
    double2* outs = bufs + GROUPS * M;
    double2* stw = outs + 2 * M;
    const int tid = threadIdx.x, g = tid / TPA, t = tid - g * TPA;
    for (int k = tid; k < Passes<LOGM>::tw_entries; k += T) stw[k] = g_tw[k];
    constexpr int logN2 = LOGM + 2;
    {
        const long long lwe = blockIdx.x;
        const uint32_t* a = in + lwe * (long long)(n + 1);
        const int rb = modswitch(a[n] + offset, logN2);
        const int e0 = (2 * N - rb) & (2 * N - 1);
        for (int k = tid; k < 2 * N; k += T) acc[k] = k < N ? 0u : rot_at<N>(tv, k - N, e0);
        double2 kv[W::AHEAD ? 2 * R : 1];
        if (W::AHEAD) {
#pragma unroll
            for (int r = 0; r < 2 * R; ++r) kv[r] = ld_table(bsk_f + (long long)r * M + tid);
        }
        for (int i = 0; i < n; ++i) {
            const double2* key = bsk_f + (long long)i * R * 2 * M;
            const int ai = modswitch(__ldg(a + i), logN2);
            __syncthreads();  // accumulator writes visible; the last step's outputs read
            if (g < GROUPS) {
                const int c = g / LEVELS, l = g - c * LEVELS;
                uint32_t plo[8], phi[8];
                rotated_difference<LOGM>(plo, phi, acc + c * N, ai, t, gd);
                const int sh = gd.base_log * (LEVELS - 1 - l);
                double2 v[8];
#pragma unroll
                for (int k = 0; k < 8; ++k)
                    v[k] = make_double2(gadget_digit<1>(plo[k] >> sh, gd, 0), gadget_digit<1>(phi[k] >> sh, gd, 0));
                split_pass<LOGM, 0>(v, t, stw);
                wide_fwd<LOGM, 1>(v, bufs + g * M, t, 1 + g, stw);
                group_bar(1 + g, TPA);  // the last exchange is read
                put8<0>(bufs + g * M, v, t);
            }
            __syncthreads();
            {
                const int p = tid, f = swz(8 * (p & (TPA - 1)) + p / TPA);  // element 8 t + k of key position k TPA + t
                double2 s0 = make_double2(0.0, 0.0), s1 = s0;
#pragma unroll
                for (int r = 0; r < R; ++r) {
                    const double2 x = bufs[r * M + f];
                    cmac(s0, x, W::AHEAD ? kv[W::AHEAD ? 2 * r : 0] : ld_table(key + (long long)(2 * r) * M + p));
                    cmac(s1, x, W::AHEAD ? kv[W::AHEAD ? 2 * r + 1 : 0] : ld_table(key + (long long)(2 * r + 1) * M + p));
                }
                outs[f] = s0;
                outs[M + f] = s1;
            }
            if (W::AHEAD && i + 1 < n) {
#pragma unroll
                for (int r = 0; r < 2 * R; ++r) kv[r] = ld_table(key + (long long)(2 * R + r) * M + tid);
            }
            __syncthreads();
            if (g < 2) {
                double2 v[8];
                get8<0>(v, outs + g * M, t);
                join_pass<LOGM, NP - 1>(v, t, stw);
                wide_inv<LOGM, NP - 2>(v, bufs + g * M, t, 1 + g, stw);
#pragma unroll
                for (int k = 0; k < 8; ++k) {
                    const int j = g * N + k * TPA + t;
                    double rx, ry;
                    acc[j] += round_scaled<LOGM>(v[k].x, gd, rx);
                    acc[j + M] += round_scaled<LOGM>(v[k].y, gd, ry);
                }
            }
        }
        __syncthreads();
        extract_lwe<N>(out + lwe * (long long)(N + 1), acc, tid, T);
    }
}

// out[B][2N] = ExtProd(ggsw_f, c[B][2N]) rounded; frac[b] = largest distance of an
// unrounded coefficient to its integer.  Same code path as a blind-rotation step.
template <int LOGM, int LEVELS>
__global__ void __launch_bounds__(GroupSplit<LOGM, LEVELS>::THREADS) k_cggi_fft_extprod(
    uint32_t* __restrict__ out, const uint32_t* __restrict__ c_in, const double2* __restrict__ ggsw_f, Gadget gd,
    const double2* __restrict__ g_tw, double* __restrict__ frac) {
    using G = GroupSplit<LOGM, LEVELS>;
    constexpr int M = G::M, N = G::N, TPA = G::TPA;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    uint32_t* acc = reinterpret_cast<uint32_t*>(smem_raw);
    double2* bufs_all = reinterpret_cast<double2*>(acc + 2 * N);
    const int c = threadIdx.x / TPA, t = threadIdx.x - c * TPA;
    double2* stw = bufs_all + 6 * M;
    for (int k = threadIdx.x; k < Passes<LOGM>::tw_entries; k += blockDim.x) stw[k] = g_tw[k];
    __syncthreads();
    const double worst = group_ext_product<LOGM, LEVELS, 1>(
        acc, bufs_all + c * 2 * M, bufs_all + 4 * M, c, t, ggsw_f, 0, gd,
        c_in + (long long)blockIdx.x * 2 * N, out + (long long)blockIdx.x * 2 * N, stw);
    // block maximum through the exchange buffers (no longer needed)
    double* red = reinterpret_cast<double*>(bufs_all);
    __syncthreads();
    red[threadIdx.x] = worst;
    __syncthreads();
    if (threadIdx.x == 0 && frac) {
        double m = 0.0;
        for (int i = 0; i < (int)blockDim.x; ++i) m = fmax(m, red[i]);
        frac[blockIdx.x] = m;
    }
}

// Spectra of rows of N signed 32-bit coefficients (torus values read as int32), in key
// order: out[r][k * M/8 + t] = spectrum element 8 t + k.  One block of M/8 threads per row.
template <int LOGM>
__global__ void __launch_bounds__((1 << LOGM) / 8) k_rows_to_fourier(double2* __restrict__ outp,
                                                                   const uint32_t* __restrict__ rows,
                                                                   const double2* __restrict__ g_tw) {
    constexpr int M = 1 << LOGM, TPA = M / 8;
    __shared__ double2 x[2 * M];
    const int t = threadIdx.x;
    const uint32_t* p = rows + (long long)blockIdx.x * 2 * M;
    double2 v[8];
#pragma unroll
    for (int k = 0; k < 8; ++k)
        v[k] = make_double2((double)(int32_t)p[k * TPA + t], (double)(int32_t)p[k * TPA + t + M]);
    split_pass<LOGM, 0>(v, t, g_tw);
    group_fwd<LOGM, 1, 0>(v, x, t, 1, g_tw);
    double2* o = outp + (long long)blockIdx.x * M;
#pragma unroll
    for (int k = 0; k < 8; ++k) o[k * TPA + t] = v[k];
}

// ---- LWE key switch: out[b] = (0, in[b].body) - sum_{j,l} d_{b,j,l} KSK[j][l], digits of
// in[b].mask[j] (base 2^kb, kt levels), modulo 2^32.
//
// A matrix product of signed digits (8 bits) with key words on the integer tensor path:
// the key words are taken apart into their four bytes, each byte plane is one product
// with 32-bit sums (exact modulo 2^32), and the planes are added at their shifts.  One
// block takes KS_M ciphertexts x KS_N columns x a share of the mask coefficients; warp w
// takes 16 MT ciphertexts (w / 4) and 8 columns (w % 4).  Shares past the first add into
// out with atomics (integers, so the order does not matter), after k_ks_body wrote the
// bodies; the launcher splits the mask where ciphertexts x columns leave SMs idle.
// Measured at n = 630, N = 1024, 8 levels, against 32-bit multiply-adds on 32 ciphertexts
// x 128 columns a block over the whole mask: 7 ciphertexts 3100 -> 26 us, 4096 3400 -> 984.
// Digits of more than 8 bits (PARTS > 1) are taken apart into balanced bytes, byte i meeting
// the key word 2^(8 i): d + sum 128 2^(8 i) has the bytes plus 128, which PARTS bytes hold for
// d in [-2^(b-1), 2^(b-1)) when b <= 8 PARTS - 1; with four bytes it holds modulo 2^32 for any b.
constexpr int KS_J = 32;       // mask coefficients decomposed per round
constexpr int KS_COLS = 32;    // columns per block

__global__ void k_ks_body(uint32_t* __restrict__ out, const uint32_t* __restrict__ in, long long B, int Nin, int n) {
    const long long total = B * (n + 1);
    for (long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x; e < total;
         e += (long long)gridDim.x * blockDim.x) {
        const long long b = e / (n + 1);
        out[e] = e - b * (n + 1) == n ? in[b * (Nin + 1) + Nin] : 0u;
    }
}

__device__ __forceinline__ void mma_s8u8(int (&c)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
    asm volatile(
        "mma.sync.aligned.m16n8k32.row.col.s32.s8.u8.s32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, "
        "%3};"
        : "+r"(c[0]), "+r"(c[1]), "+r"(c[2]), "+r"(c[3])
        : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}

// byte i of words w0..w3 -> b[i] (a 4 x 4 byte transpose)
__device__ __forceinline__ void byte_planes(uint32_t (&b)[4], uint32_t w0, uint32_t w1, uint32_t w2, uint32_t w3) {
    const uint32_t lo01 = __byte_perm(w0, w1, 0x5140), hi01 = __byte_perm(w0, w1, 0x7362);
    const uint32_t lo23 = __byte_perm(w2, w3, 0x5140), hi23 = __byte_perm(w2, w3, 0x7362);
    b[0] = __byte_perm(lo01, lo23, 0x5410);
    b[1] = __byte_perm(lo01, lo23, 0x7632);
    b[2] = __byte_perm(hi01, hi23, 0x5410);
    b[3] = __byte_perm(hi01, hi23, 0x7632);
}

// MT: 16-row tiles of ciphertexts a warp takes; the block takes MROWS = 16 MT x 2.
template <int MT, int PARTS>
__global__ void __launch_bounds__(256) k_cggi_keyswitch(uint32_t* __restrict__ out, const uint32_t* __restrict__ in,
                                                        long long B, const uint32_t* __restrict__ ksk, int Nin, int n,
                                                        int base_log, int levels, int j_share) {
    constexpr int MROWS = 32 * MT;
    extern __shared__ __align__(16) unsigned char ksm[];
    const int dj = levels * PARTS;  // digit bytes of one mask coefficient
    const int kc = KS_J * dj;       // of one round, a multiple of 32
    const int pitch = kc + 16;     // bytes; the 16 keep a fragment's 8 rows on different banks
    int8_t* dig = reinterpret_cast<int8_t*>(ksm);  // [MROWS][pitch]
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int wm = warp >> 2, wn = warp & 3;
    const long long b0 = (long long)blockIdx.y * MROWS;
    const int col = blockIdx.x * KS_COLS + wn * 8 + (lane >> 2);
    const bool col_ok = col <= n;
    const int j_begin = blockIdx.z * j_share;
    const int j_end = j_begin + j_share < Nin ? j_begin + j_share : Nin;
    const int total = base_log * levels;
    const uint32_t keep = total >= 32 ? 0xFFFFFFFFu : (1u << total) - 1u;
    const uint32_t field = base_log >= 32 ? 0xFFFFFFFFu : (1u << base_log) - 1u;
    uint32_t half_sum = 0;
    for (int l = 0; l < levels; ++l) half_sum += 1u << (base_log * l + base_log - 1);
    int acc[MT][4][4];
#pragma unroll
    for (int m = 0; m < MT; ++m)
#pragma unroll
        for (int p = 0; p < 4; ++p)
#pragma unroll
            for (int k = 0; k < 4; ++k) acc[m][p][k] = 0;
    for (int j0 = j_begin; j0 < j_end; j0 += KS_J) {
        __syncthreads();  // the previous round's digits are read
        // balanced digits without a carry loop (see Gadget); coefficients past the end: zeros
        for (int e = threadIdx.x; e < MROWS * KS_J; e += 256) {
            const int row = e / KS_J, jj = e - row * KS_J;
            const long long b = b0 + row;
            const bool ok = b < B && j0 + jj < j_end;
            uint32_t v = ok ? in[b * (Nin + 1) + j0 + jj] : 0u;
            v = total >= 32 ? v : (uint32_t)(((uint64_t)v + (1ULL << (31 - total))) >> (32 - total));
            v = (v + half_sum) & keep;
            int8_t* d = dig + row * pitch + jj * dj;
            for (int l = 0; l < levels; ++l) {
                const uint32_t x = ((v >> (base_log * (levels - 1 - l))) & field) - (1u << (base_log - 1));
                if constexpr (PARTS == 1) {
                    d[l] = ok ? (int8_t)(int)x : 0;
                } else {
                    const uint32_t y = x + (0x80808080u >> (8 * (4 - PARTS)));
#pragma unroll
                    for (int i = 0; i < PARTS; ++i)
                        d[l * PARTS + i] = ok ? (int8_t)((int)((y >> (8 * i)) & 255u) - 128) : 0;
                }
            }
        }
        __syncthreads();
        const long long k_rows = (long long)Nin * dj, k0 = (long long)j0 * dj;
        for (int kk = 0; kk < kc; kk += 32) {
            uint32_t w[8];
#pragma unroll
            for (int r = 0; r < 8; ++r) {
                const long long kr = k0 + kk + (lane & 3) * 4 + (r & 3) + (r >> 2) * 16;
                w[r] = col_ok && kr < k_rows ? __ldg(ksk + kr / PARTS * (n + 1) + col) << (8 * (int)(kr % PARTS)) : 0u;
            }
            uint32_t p0[4], p1[4];
            byte_planes(p0, w[0], w[1], w[2], w[3]);
            byte_planes(p1, w[4], w[5], w[6], w[7]);
#pragma unroll
            for (int m = 0; m < MT; ++m) {
                const int8_t* base = dig + ((wm * MT + m) * 16 + (lane >> 2)) * pitch + kk + (lane & 3) * 4;
                uint32_t a[4];
                a[0] = *reinterpret_cast<const uint32_t*>(base);
                a[1] = *reinterpret_cast<const uint32_t*>(base + 8 * pitch);
                a[2] = *reinterpret_cast<const uint32_t*>(base + 16);
                a[3] = *reinterpret_cast<const uint32_t*>(base + 8 * pitch + 16);
#pragma unroll
                for (int p = 0; p < 4; ++p) mma_s8u8(acc[m][p], a, p0[p], p1[p]);
            }
        }
    }
    // accumulator (row lane / 4 (+ 8), columns 2 (lane % 4) + {0, 1})
    const bool shared_out = gridDim.z > 1;
#pragma unroll
    for (int m = 0; m < MT; ++m)
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            const long long b = b0 + (wm * MT + m) * 16 + (lane >> 2) + (k >> 1) * 8;
            const int c = blockIdx.x * KS_COLS + wn * 8 + (lane & 3) * 2 + (k & 1);
            if (b >= B || c > n) continue;
            uint32_t v = 0u;
#pragma unroll
            for (int p = 0; p < 4; ++p) v -= (uint32_t)acc[m][p][k] << (8 * p);
            uint32_t* o = out + b * (n + 1) + c;
            if (shared_out) atomicAdd(o, v);
            else *o = c == n ? v + in[b * (Nin + 1) + Nin] : v;
        }
}

bool check_shape(int N, int levels, int base_log, const char* where) {
    if (N != 512 && N != 1024 && N != 2048) {
        set_error(where, "N must be 512, 1024 or 2048");
        return false;
    }
    if (levels < 1 || levels > kMaxLevels || base_log < 1 || base_log * levels > 32) {
        set_error(where, "gadget needs 1..4 levels and base_log * levels <= 32");
        return false;
    }
    return true;
}

template <int LOGM, int LEVELS>
int launch_bootstrap_t(uint32_t* out, const uint32_t* in, long long B, const double2* bsk_f, const uint32_t* tv,
                       int n, int base_log, uint32_t offset, const FourierTables* ft, cudaStream_t st) {
    using G = GroupSplit<LOGM, LEVELS>;
    using W = WideSplit<LOGM, LEVELS>;
    // Wide blocks where every LWE has an SM to itself: 2.4 against 4.1-4.6 ms at N = 1024,
    // n = 630, 3 levels for 1 to 148 LWEs, 244 against 381 us at N = 512, n = 100.  Past
    // that a second block per SM does more (296 LWEs: 4.65 ms against 4.79 in two rounds),
    // and at N = 2048 two groups already fill an SM's issue slots (709 against 833 us, n = 100).
    if constexpr (LOGM <= 9) {
        if (B <= sm_count()) {
            const int e = (int)cudaFuncSetAttribute(k_cggi_fft_bootstrap_wide<LOGM, LEVELS>,
                                                    cudaFuncAttributeMaxDynamicSharedMemorySize, (int)W::smem);
            if (e) return e;
            k_cggi_fft_bootstrap_wide<LOGM, LEVELS><<<(unsigned)B, W::THREADS, W::smem, st>>>(
                out, in, bsk_f, tv, n, make_gadget(2 << LOGM, base_log, LEVELS), offset, ft->d_tw);
            note_launch();
            return (int)cudaGetLastError();
        }
    }
    int e = (int)cudaFuncSetAttribute(k_cggi_fft_bootstrap<LOGM, LEVELS>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                      (int)G::smem);
    if (e) return e;
    int per_sm = 0;
    e = (int)cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_cggi_fft_bootstrap<LOGM, LEVELS>, G::THREADS,
                                                           G::smem);
    if (e) return e;
    long long grid = (long long)(per_sm > 0 ? per_sm : 1) * sm_count();
    if (grid > B) grid = B;
    k_cggi_fft_bootstrap<LOGM, LEVELS><<<(unsigned)grid, G::THREADS, G::smem, st>>>(
        out, in, B, bsk_f, tv, n, make_gadget(2 << LOGM, base_log, LEVELS), offset, ft->d_tw);
    note_launch();
    return (int)cudaGetLastError();
}

template <int LOGM, int LEVELS>
int launch_extprod_t(uint32_t* out, const uint32_t* c, long long B, const double2* ggsw_f, int base_log,
                     const FourierTables* ft, double* frac, cudaStream_t st) {
    using G = GroupSplit<LOGM, LEVELS>;
    int e = (int)cudaFuncSetAttribute(k_cggi_fft_extprod<LOGM, LEVELS>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                      (int)G::smem);
    if (e) return e;
    k_cggi_fft_extprod<LOGM, LEVELS><<<(unsigned)B, G::THREADS, G::smem, st>>>(
        out, c, ggsw_f, make_gadget(2 << LOGM, base_log, LEVELS), ft->d_tw, frac);
    note_launch();
    return (int)cudaGetLastError();
}

// (N, levels) -> template instance
template <template <int, int> class F, typename... A>
int dispatch_nl(int N, int levels, A... args) {
    const int logm = N == 512 ? 8 : N == 1024 ? 9 : 10;
    switch (logm * 8 + levels) {
        case 8 * 8 + 1: return F<8, 1>::run(args...);
        case 8 * 8 + 2: return F<8, 2>::run(args...);
        case 8 * 8 + 3: return F<8, 3>::run(args...);
        case 8 * 8 + 4: return F<8, 4>::run(args...);
        case 9 * 8 + 1: return F<9, 1>::run(args...);
        case 9 * 8 + 2: return F<9, 2>::run(args...);
        case 9 * 8 + 3: return F<9, 3>::run(args...);
        case 9 * 8 + 4: return F<9, 4>::run(args...);
        case 10 * 8 + 1: return F<10, 1>::run(args...);
        case 10 * 8 + 2: return F<10, 2>::run(args...);
        case 10 * 8 + 3: return F<10, 3>::run(args...);
        default: return F<10, 4>::run(args...);
    }
}

template <int LOGM, int LEVELS>
struct BootstrapF {
    template <typename... A>
    static int run(A... a) { return launch_bootstrap_t<LOGM, LEVELS>(a...); }
};
template <int LOGM, int LEVELS>
struct ExtprodF {
    template <typename... A>
    static int run(A... a) { return launch_extprod_t<LOGM, LEVELS>(a...); }
};

template <int MT, int PARTS>
int launch_keyswitch_t(uint32_t* out, const uint32_t* in, long long B, const uint32_t* ksk, int N, int n, int base_log,
                       int levels, cudaStream_t st) {
    const size_t smem = (size_t)32 * MT * (KS_J * levels * PARTS + 16);
    if (smem > 48 * 1024) {
        const int e = (int)cudaFuncSetAttribute(k_cggi_keyswitch<MT, PARTS>,
                                                cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        if (e) return e;
    }
    const long long cols = (n + 1 + KS_COLS - 1) / KS_COLS, rows = (B + 32 * MT - 1) / (32 * MT);
    // shares of the mask coefficients: enough blocks for two per SM, no share below one round
    long long shares = (2LL * sm_count() + cols * rows - 1) / (cols * rows);
    const long long rounds = (N + KS_J - 1) / KS_J;
    if (shares > rounds) shares = rounds;
    const int j_share = (int)((rounds + shares - 1) / shares) * KS_J;
    shares = (N + j_share - 1) / j_share;
    if (shares > 1) {
        long long blocks = (B * (n + 1) + 255) / 256;
        if (blocks > 4LL * sm_count()) blocks = 4LL * sm_count();
        k_ks_body<<<(unsigned)blocks, 256, 0, st>>>(out, in, B, N, n);
        note_launch();
    }
    k_cggi_keyswitch<MT, PARTS><<<dim3((unsigned)cols, (unsigned)rows, (unsigned)shares), 256, smem, st>>>(
        out, in, B, ksk, N, n, base_log, levels, j_share);
    note_launch();
    return (int)cudaGetLastError();
}

// Warps take four 16-row tiles of ciphertexts where the batch fills them, one otherwise.
template <int PARTS>
int launch_keyswitch_p(uint32_t* out, const uint32_t* in, long long B, const uint32_t* ksk, int N, int n, int base_log,
                       int levels, cudaStream_t st) {
    return B > 32 ? launch_keyswitch_t<4, PARTS>(out, in, B, ksk, N, n, base_log, levels, st)
                  : launch_keyswitch_t<1, PARTS>(out, in, B, ksk, N, n, base_log, levels, st);
}

// Bytes a digit takes: one up to 8 bits ([-128, 128) as it stands), else those that hold it
// balanced, at most the word's four.
int launch_keyswitch(uint32_t* out, const uint32_t* in, long long B, const uint32_t* ksk, int N, int n, int base_log,
                     int levels, cudaStream_t st) {
    if (base_log <= 8) return launch_keyswitch_p<1>(out, in, B, ksk, N, n, base_log, levels, st);
    if (base_log <= 15) return launch_keyswitch_p<2>(out, in, B, ksk, N, n, base_log, levels, st);
    if (base_log <= 23) return launch_keyswitch_p<3>(out, in, B, ksk, N, n, base_log, levels, st);
    return launch_keyswitch_p<4>(out, in, B, ksk, N, n, base_log, levels, st);
}

int launch_to_fourier(int N, double2* outp, const uint32_t* rows, long long count, const FourierTables* ft,
                      cudaStream_t st) {
    for (long long off = 0; off < count; off += 65535LL * 16) {
        const long long m = count - off < 65535LL * 16 ? count - off : 65535LL * 16;
        switch (N) {
            case 512: k_rows_to_fourier<8><<<(unsigned)m, 32, 0, st>>>(outp + off * 256, rows + off * 512, ft->d_tw); break;
            case 1024: k_rows_to_fourier<9><<<(unsigned)m, 64, 0, st>>>(outp + off * 512, rows + off * 1024, ft->d_tw); break;
            default: k_rows_to_fourier<10><<<(unsigned)m, 128, 0, st>>>(outp + off * 1024, rows + off * 2048, ft->d_tw); break;
        }
        note_launch();
        const int e = (int)cudaGetLastError();
        if (e) return e;
    }
    return 0;
}

}  // namespace

}  // namespace vc

using namespace vc;

namespace vc {
namespace {

// ---- torus key generation on the device (the big random material of the keys; the
// secret keys s and S are the caller's)
//
// Bootstrapping key: row (i, r), r = c levels + l, is a GLWE encryption of zero under
// S, (a, a S + e), with s_i 2^(32 - base_log (l + 1)) added to coefficient 0 of
// component c -- GGSW(s_i) in the layout vfhe_cuda_cggi_fft_bootstrap_batch reads.
// Key-switching key: row (j, l) is an LWE encryption under s of S_j 2^(32 - ks_base_log
// (l + 1)).  a is uniform over the torus, e a rounded Gaussian of width sigma 2^32.
// Randomness: the engine's ChaCha20 stream, uniform and Gaussian nonces, blocks counted
// from u0 / g0 per row.

__device__ __forceinline__ int32_t torus_gauss(const PrngKey& key, uint64_t counter, int k, double sigma32) {
    uint32_t blk[16];
    chacha20_block(key, counter, kStreamGaussian, blk);
    const double u1 = unit_open_low(block_u64(blk, 2 * (k & 3))), u2 = unit_closed_low(block_u64(blk, 2 * (k & 3) + 1));
    return (int32_t)(int64_t)llrint(sigma32 * sqrt(-2.0 * log(u1)) * cospi(2.0 * u2));
}

// One CTA per bootstrapping-key row, its threads over the coefficients k (N = 2048 has more of
// them than a CTA has threads).
constexpr int kBskThreads = 1024;

__global__ void __launch_bounds__(kBskThreads) k_torus_bsk_rows(uint32_t* __restrict__ rows, const int32_t* __restrict__ s,
                                                                const int32_t* __restrict__ S, int N, int levels,
                                                                int base_log, double sigma32,
                                                                const __grid_constant__ PrngKey key, uint64_t u0,
                                                                uint64_t g0) {
    extern __shared__ uint32_t tsm[];  // a [N], S [N]
    uint32_t* a = tsm;
    uint32_t* Ssh = tsm + N;
    const long long row = blockIdx.x;  // i * 2 levels + r
    const int i = (int)(row / (2 * levels)), r = (int)(row - (long long)i * 2 * levels);
    const uint64_t per_row = (uint64_t)(N / 16);
    for (int k = threadIdx.x; k < N; k += blockDim.x) {
        if ((k & 15) == 0) {
            uint32_t blk[16];
            chacha20_block(key, u0 + (uint64_t)row * per_row + (uint64_t)(k >> 4), kStreamUniform, blk);
#pragma unroll
            for (int w = 0; w < 16; ++w) a[k + w] = blk[w];
        }
        Ssh[k] = (uint32_t)S[k];
    }
    __syncthreads();
    const int c = r / levels, l = r - c * levels;
    uint32_t* out = rows + (size_t)row * 2 * N;
    for (int k = threadIdx.x; k < N; k += blockDim.x) {
        // (a S)_k = sum_j a_j S_(k-j) with the sign of the wrap (X^N = -1)
        uint32_t acc = 0;  // products mod 2^32: a small signed key entry multiplies as its residue
        for (int j = 0; j <= k; ++j) acc += a[j] * Ssh[k - j];
        for (int j = k + 1; j < N; ++j) acc -= a[j] * Ssh[k - j + N];
        const int32_t e = torus_gauss(key, g0 + (uint64_t)row * (uint64_t)(N / 4) + (uint64_t)(k >> 2), k, sigma32);
        uint32_t b = acc + (uint32_t)e;
        uint32_t av = a[k];
        if (k == 0) {
            const uint32_t m = (uint32_t)s[i] << (32 - base_log * (l + 1));
            if (c == 0) av += m;
            else b += m;
        }
        out[k] = av;
        out[N + k] = b;
    }
}

// one thread per key-switching-key row (j, l): mask, then body
__global__ void k_torus_ksk_rows(uint32_t* __restrict__ ksk, const int32_t* __restrict__ s,
                                 const int32_t* __restrict__ S, int n, int N, int levels, int base_log, double sigma32,
                                 const __grid_constant__ PrngKey key, uint64_t u0, uint64_t g0) {
    const long long rows = (long long)N * levels;
    for (long long row = blockIdx.x * (long long)blockDim.x + threadIdx.x; row < rows;
         row += (long long)gridDim.x * blockDim.x) {
        const int j = (int)(row / levels), l = (int)(row - (long long)j * levels);
        uint32_t* out = ksk + (size_t)row * (n + 1);
        const uint64_t per_row = (uint64_t)((n + 15) / 16);
        uint32_t dot = 0;
        for (int c = 0; c < n; c += 16) {
            uint32_t blk[16];
            chacha20_block(key, u0 + (uint64_t)row * per_row + (uint64_t)(c >> 4), kStreamUniform, blk);
            for (int w = 0; w < 16 && c + w < n; ++w) {
                out[c + w] = blk[w];
                dot += blk[w] * (uint32_t)s[c + w];
            }
        }
        const int32_t e = torus_gauss(key, g0 + (uint64_t)row, 0, sigma32);
        out[n] = dot + (uint32_t)e + ((uint32_t)S[j] << (32 - base_log * (l + 1)));
    }
}

}  // namespace
}  // namespace vc

extern "C" {

int vfhe_cuda_cggi_fft_to_fourier(double* d_out, const uint32_t* d_rows, uint64_t count, uint32_t N, void* stream) {
    if (!ensure_ready()) return 1;
    const char* where = "vfhe_cuda_cggi_fft_to_fourier";
    if (!check_shape((int)N, 1, 1, where)) return 1;
    const FourierTables* ft = fourier_tables((int)N);
    if (!ft) return check_cuda(cudaErrorMemoryAllocation, where) ? 0 : 1;
    const int e = launch_to_fourier((int)N, (double2*)d_out, d_rows, (long long)count, ft, (cudaStream_t)stream);
    return check_cuda(e, where) ? 0 : 1;
}

int vfhe_cuda_cggi_fft_bootstrap_batch(uint32_t* d_out, const uint32_t* d_in, uint64_t batch, const double* d_bsk_f,
                                       const uint32_t* d_tv, uint32_t n, uint32_t N, uint32_t base_log, uint32_t levels,
                                       uint32_t torus_base, void* stream) {
    if (!ensure_ready()) return 1;
    const char* where = "vfhe_cuda_cggi_fft_bootstrap_batch";
    if (!check_shape((int)N, (int)levels, (int)base_log, where)) return 1;
    if (n == 0 || torus_base == 0 || batch == 0) {
        set_error(where, "need n > 0, torus_base > 0 and a nonempty batch");
        return 1;
    }
    const FourierTables* ft = fourier_tables((int)N);
    if (!ft) return check_cuda(cudaErrorMemoryAllocation, where) ? 0 : 1;
    const uint32_t offset = (uint32_t)((1ULL << 32) / (4ULL * torus_base));
    const int e = dispatch_nl<BootstrapF>((int)N, (int)levels, d_out, d_in, (long long)batch, (const double2*)d_bsk_f,
                                          d_tv, (int)n, (int)base_log, offset, ft, (cudaStream_t)stream);
    return check_cuda(e, where) ? 0 : 1;
}

int vfhe_cuda_cggi_fft_keyswitch_batch(uint32_t* d_out, const uint32_t* d_in, uint64_t batch, const uint32_t* d_ksk,
                                       uint32_t N, uint32_t n, uint32_t base_log, uint32_t levels, void* stream) {
    if (!ensure_ready()) return 1;
    const char* where = "vfhe_cuda_cggi_fft_keyswitch_batch";
    if (base_log < 1 || levels < 1 || levels > 16 || base_log * levels > 32 || n == 0 || N == 0 || batch == 0) {
        set_error(where, "need 1..16 levels, base_log * levels <= 32, n, N > 0");
        return 1;
    }
    if (batch > 65535ULL * 32) {
        set_error(where, "batch too large (at most 65535 x 32)");
        return 1;
    }
    const int e = launch_keyswitch(d_out, d_in, (long long)batch, d_ksk, (int)N, (int)n, (int)base_log, (int)levels,
                                   (cudaStream_t)stream);
    return check_cuda(e, where) ? 0 : 1;
}

int vfhe_cuda_cggi_fft_external_product(uint32_t* d_out, const uint32_t* d_c, uint64_t batch, const double* d_ggsw_f,
                                        uint32_t N, uint32_t base_log, uint32_t levels, double* d_frac,
                                        void* stream) {
    if (!ensure_ready()) return 1;
    const char* where = "vfhe_cuda_cggi_fft_external_product";
    if (!check_shape((int)N, (int)levels, (int)base_log, where)) return 1;
    if (batch == 0 || batch > 65535) {
        set_error(where, "batch must be in [1, 65535]");
        return 1;
    }
    const FourierTables* ft = fourier_tables((int)N);
    if (!ft) return check_cuda(cudaErrorMemoryAllocation, where) ? 0 : 1;
    const int e = dispatch_nl<ExtprodF>((int)N, (int)levels, d_out, d_c, (long long)batch, (const double2*)d_ggsw_f,
                                        (int)base_log, ft, d_frac, (cudaStream_t)stream);
    return check_cuda(e, where) ? 0 : 1;
}

// Torus CGGI keys generated on the device from the caller's secret keys (binary or
// small signed int32): d_bsk_rows [n][2 bs_levels][2][N] uint32 (then to_fourier for the
// spectra the bootstrap reads) and d_ksk [N][ks_levels][n+1] uint32.
int vfhe_cuda_cggi_fft_gen_keys(uint32_t* d_bsk_rows, uint32_t* d_ksk, const int32_t* d_s, const int32_t* d_S,
                                uint32_t n, uint32_t N, uint32_t bs_base_log, uint32_t bs_levels, uint32_t ks_base_log,
                                uint32_t ks_levels, double lwe_sigma, double glwe_sigma, void* stream) {
    if (!ensure_ready()) return 1;
    const char* where = "vfhe_cuda_cggi_fft_gen_keys";
    if (!d_bsk_rows || !d_ksk || !d_s || !d_S || n == 0 || n > (1u << 16) || (N != 512 && N != 1024 && N != 2048) ||
        bs_levels == 0 || bs_levels * bs_base_log > 32 || ks_levels == 0 || ks_levels * ks_base_log > 32 ||
        !(lwe_sigma >= 0.0) || !(glwe_sigma >= 0.0)) {
        set_error(where, "bad buffers, n, N (512/1024/2048), gadget shapes or noise widths");
        return 1;
    }
    cudaStream_t st = (cudaStream_t)stream;
    const uint64_t bsk_rows = (uint64_t)n * 2 * bs_levels;
    const uint64_t ksk_rows = (uint64_t)N * ks_levels;
    const uint64_t u0 = prng_advance(bsk_rows * (N / 16) + ksk_rows * ((n + 15) / 16));
    const uint64_t g0 = prng_advance(bsk_rows * (N / 4) + ksk_rows);
    const PrngKey key = prng_key();
    k_torus_bsk_rows<<<(unsigned)bsk_rows, N < kBskThreads ? N : kBskThreads, 2 * N * sizeof(uint32_t), st>>>(
        d_bsk_rows, d_s, d_S, (int)N, (int)bs_levels, (int)bs_base_log, glwe_sigma * 4294967296.0, key, u0, g0);
    note_launch();
    if (!check_cuda(cudaGetLastError(), where)) return 1;
    k_torus_ksk_rows<<<(unsigned)((ksk_rows + 255) / 256), 256, 0, st>>>(
        d_ksk, d_s, d_S, (int)n, (int)N, (int)ks_levels, (int)ks_base_log, lwe_sigma * 4294967296.0, key,
        u0 + bsk_rows * (N / 16), g0 + bsk_rows * (N / 4));
    note_launch();
    return check_cuda(cudaGetLastError(), where) ? 0 : 1;
}

}  // extern "C"
