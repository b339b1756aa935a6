// ntt_kernels.cuh - two-pass negacyclic NTT / INTT over RNS limbs for sm_100a.
//
// Decomposition. N = N1 * N2 (N1 = 2^LOG_A rows, N2 = 2^LOG_B columns of the row-major limb).
//   forward:  pass A = first LOG_A Cooley-Tukey stages = N2 independent N1-point transforms down
//             the columns; pass B = last LOG_B stages = N1 independent N2-point transforms on the
//             contiguous rows. Natural order in, bit-reversed order out, twiddle index m + k
//             (the reference's convention: src/ntt/ntt_1d.cu:41-60, src/host/ntt.cu:22-33).
//   inverse:  the mirror image with Gentleman-Sande butterflies, rows first.
// One kernel template serves both passes: a CTA owns C sub-transforms of T points, every thread
// keeps EPT = 16 (or 8) residues in registers and runs R1 stages, exchanges once through padded
// shared memory, runs the remaining R2 stages and stores. A limb therefore crosses global memory
// twice per transform (the intermediate of the two passes stays in the 126 MB L2).
//
// Twiddle index algebra (P = 1 for the column pass, P = N1 + row for the row pass):
//   forward, local stage s (0-based inside the T-point sub-transform), pair group k':
//       index = (P << s) + k'
//   inverse, local stage with gap 2^u, pair group k':
//       index = ((T >> (u + 1)) * P) + k'
// Lazy ranges are those of the prime's arithmetic policy (below); the last pass stores canonical values.
#pragma once
#include <cstddef>
#include <type_traits>
#include "modarith.cuh"

namespace b2 {

struct Mod {
    uint64_t q, r0, r1;  // r = floor(2^128 / q)
    uint64_t mu;         // floor(2^(62 + n) / q), n = bit length of q
    double qinv;         // 1 / q
};

// One job = one limb transform: where the limb lives and which prime's tables it uses.
// x = slot in the transform's own buffer, y = prime index, z/w = extra slots for epilogues.
// Inverse transforms read limb x of src and write limb w of dst (z selects the final scaling).
using Job = uint4;

// resident threads per SM the pass kernels are compiled for (register cap = 65536 / this)
#ifndef B2_NTT_RESIDENT_THREADS
#define B2_NTT_RESIDENT_THREADS 768
#endif
// (a pass whose threads hold 32 residues each - the 512-point pass of N = 2^17 - gets twice the registers: half the threads)
constexpr int ntt_min_blocks(int threads, int residues_per_thread = 16) {
    return (B2_NTT_RESIDENT_THREADS / (residues_per_thread > 16 ? 2 : 1)) / threads > 0 ? (B2_NTT_RESIDENT_THREADS / (residues_per_thread > 16 ? 2 : 1)) / threads : 1;
}

// One output limb of a base conversion: sum_i y_i[n] M_i mod p over `ni` input limbs from slot in_slot0 on; M_i at mat_off + i
// as {M, floor(M 2^64 / p)}; bit i of `wide`: input limb i holds residues of a prime of 2^50 or more
struct BcJob {
    uint32_t in_slot0, ni, mat_off, wide;
};
struct NttArgs {
    const uint64_t *src;  // limb `slot` at src + slot * N
    uint64_t *dst;
    const Job *jobs;       // nullptr: slot = job, prime = first_prime + job
    uint32_t first_prime;
    uint32_t logN;
    const W2 *tw;          // [size_QP][N] {w, shoup(w)}
    const Mod *mod;        // [size_QP]
    const W2 *fin;         // inverse only: [idx][2] = {scale of the x outputs, last-stage twiddle}
    // A batch of polynomial sets in one launch (the two-pass kernels only): blockIdx.y = set b, and limb slot s of set b
    // lives at slot s * (lm1 + 1) + b * bs of the buffer. Zero-initialised fields mean one set, slots as they are.
    // Batch-major buffers [b][slots] use lm1 = 0, bs = slots per set; limb-major ones [slot][b] use lm1 = batch - 1, bs = 1.
    // (At an 8-byte boundary, so that a pair of them can be read as one: with the word below before them, and no pair aligned, every
    // transform in one launch took 0.02 to 0.05 us longer, those in two up to 0.1; B200, 8 limbs, 2^12 to 2^16.)
    uint32_t src_lm1, src_bs, dst_lm1, dst_bs;
    uint32_t period;       // without a job list: limb j uses prime first_prime + j % period (0: + j), a batch of polynomials
    const uint32_t *perm;  // inverse row pass: the input is read through a Galois element's permutation (a rotation's c1)
    const BcJob *bc;       // SRC_CONV: one per job, the conversion that makes its limb, and the matrix entries
    const W2 *mat;
    // SRC_REM: the dropped limbs of a rescale, residues mod rem_q in coefficient form; limb job.x takes slot job.x / rem_div, set b's
    // start b * rem_bs limbs further; words above rem_half stand for word - rem_q (rounding to nearest; all ones: floor)
    const uint64_t *rem;
    uint32_t rem_div, rem_bs;
    uint64_t rem_q, rem_half;
};
static_assert(offsetof(NttArgs, src_lm1) % 8 == 0 && offsetof(NttArgs, dst_lm1) % 8 == 0, "pairs of strides are read as one word");
// What a forward transform reads: canonical words (0), words below 2 q as the base conversion leaves them (SRC_WORDS), the base
// conversion of other limbs (SRC_CONV), the remainder that a rescale subtracts (SRC_REM: floor, SRC_REM | SRC_NEAR: nearest), or the
// sum of a remainder (either) and one of the last two before it
enum { SRC_REM = 1, SRC_CONV = 2, SRC_WORDS = 4, SRC_NEAR = 8 };

// The sets of a batched launch are the slow grid dimension. With the sets fastest (the CTAs of all sets on one tile next to
// one another, sharing its twiddles in L2) the row passes ran as fast and the column passes 8 % slower on B200.
__device__ __forceinline__ uint32_t set_idx(const NttArgs &) { return blockIdx.y; }
__device__ __forceinline__ uint32_t work_idx(const NttArgs &) { return blockIdx.x; }
__device__ __forceinline__ size_t src_slot(const NttArgs &a, uint32_t slot) { return (size_t)slot * (a.src_lm1 + 1) + (size_t)set_idx(a) * a.src_bs; }
__device__ __forceinline__ size_t dst_slot(const NttArgs &a, uint32_t slot) { return (size_t)slot * (a.dst_lm1 + 1) + (size_t)set_idx(a) * a.dst_bs; }

template <int SRC>
__device__ __forceinline__ const uint64_t *src_rem(const NttArgs &a, const Job &job, size_t N) {
    return SRC & SRC_REM ? a.rem + ((size_t)(job.x / a.rem_div) + (size_t)set_idx(a) * a.rem_bs) * N : nullptr;
}

__device__ __forceinline__ Job get_job(const NttArgs &a, uint32_t j) {
    if (a.jobs) return a.jobs[j];
    const uint32_t p = a.first_prime + (a.period ? j % a.period : j);
    return make_uint4(j, p, p, j);
}

// 256-bit global accesses (sm_100): one lane moves a whole 32-byte sector, so a thread that owns a run of
// consecutive residues touches every sector once instead of twice with 16-byte accesses. p: 32-byte aligned.
struct u64x4 {
    uint64_t a, b, c, d;
};
// Volatile: a statement that is a function of its address to the compiler may be moved out of a loop and executed where the
// condition around it does not hold (the fused row pass read past the end of its input for the P limbs so), or ahead of the
// wait for the previous kernel. Tables of the context have neither problem: any index of theirs is there to be read.
__device__ __forceinline__ u64x4 ld256(const uint64_t *p) {
    u64x4 v;
    asm volatile("ld.global.v4.u64 {%0, %1, %2, %3}, [%4];" : "=l"(v.a), "=l"(v.b), "=l"(v.c), "=l"(v.d) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ u64x4 ld256_table(const uint64_t *p) {
    u64x4 v;
    asm("ld.global.v4.u64 {%0, %1, %2, %3}, [%4];" : "=l"(v.a), "=l"(v.b), "=l"(v.c), "=l"(v.d) : "l"(p));
    return v;
}
__device__ __forceinline__ void st256(uint64_t *p, uint64_t a, uint64_t b, uint64_t c, uint64_t d) {
    asm volatile("st.global.v4.u64 [%0], {%1, %2, %3, %4};" ::"l"(p), "l"(a), "l"(b), "l"(c), "l"(d) : "memory");
}

// one table entry, or two at a 32-byte boundary
template <int CNT>
__device__ __forceinline__ void ld_pairs(W2 (&w)[CNT], const W2 *p) {
    if constexpr (CNT == 1) {
        w[0] = ldg_w2(p);
    } else {
        const u64x4 v = ld256_table(reinterpret_cast<const uint64_t *>(p));
        w[0] = W2{v.a, v.b}, w[1] = W2{v.c, v.d};
    }
}

// ---- epilogues of the last forward (row) pass ---------------------------------------------------
// The row pass leaves every thread with E canonical residues in runs of four, `step` apart, the first at limb offset o.
// An epilogue first preloads whatever else it needs for those positions (before the butterflies, so
// the loads are in flight while the ALUs work) and then finishes and stores them.
__host__ __device__ inline bool aligned32(const void *p) { return ((uintptr_t)p & 31) == 0; }

struct EpiStore {
    uint64_t *dst;
    bool aligned() const { return true; }  // dst is the transform's own output, checked by the launcher
    template <int E> struct Regs {};
    __device__ __forceinline__ void init(const NttArgs &a, const Job &job, size_t N) { dst = a.dst + dst_slot(a, job.x) * N; }
    template <int E> __device__ __forceinline__ void preload(Regs<E> &, size_t, int) const {}
    template <int E> __device__ __forceinline__ void finish(const Regs<E> &, size_t o, int step, uint64_t (&x)[E], uint64_t) const {
#pragma unroll
        for (int i = 0; i < E / 4; i++) st256(dst + o + i * step, x[4 * i], x[4 * i + 1], x[4 * i + 2], x[4 * i + 3]);
    }
};

// out[job.w] = (ACCUM ? out[job.w] : 0) + (minuend[job.z] - v) * k[prime]
// ModDown (src/rns_bconv.cu:820-821 with include/ntt_radix8_tmpl.cuh:203-233) followed by the
// add-to-ciphertext (:763-769) when ACCUM; rescale (src/rns.cu:1146-1158) without.
template <bool ACCUM>
struct EpiSubMul {
    const uint64_t *minuend;  // [slots][N]
    uint64_t *out;            // [slots][N]
    const W2 *k;              // per prime
    uint32_t m_bs = 0, o_bs = 0;  // batch strides in limbs (set b of a batched launch: see NttArgs)
    const uint64_t *m_ = nullptr;
    uint64_t *o_ = nullptr;
    W2 kk = W2{0, 0};
    bool aligned() const { return aligned32(minuend) && aligned32(out); }
    template <int E> struct Regs {
        u64x4 m[E / 4];
        u64x4 acc[ACCUM ? E / 4 : 1];
    };
    __device__ __forceinline__ void init(const NttArgs &a, const Job &job, size_t N) {
        m_ = minuend + ((size_t)job.z + (size_t)set_idx(a) * m_bs) * N;
        o_ = out + ((size_t)job.w + (size_t)set_idx(a) * o_bs) * N;
        kk = k[job.y];
    }
    template <int E> __device__ __forceinline__ void preload(Regs<E> &r, size_t o, int step) const {
#pragma unroll
        for (int i = 0; i < E / 4; i++) {
            r.m[i] = ld256(m_ + o + i * step);
            if (ACCUM) r.acc[i] = ld256(o_ + o + i * step);
        }
    }
    template <int E> __device__ __forceinline__ void finish(const Regs<E> &r, size_t o, int step, uint64_t (&x)[E], uint64_t q) const {
#pragma unroll
        for (int i = 0; i < E / 4; i++) {
            uint64_t r0 = mul_shoup(sub_mod(r.m[i].a, x[4 * i], q), kk, q);
            uint64_t r1 = mul_shoup(sub_mod(r.m[i].b, x[4 * i + 1], q), kk, q);
            uint64_t r2 = mul_shoup(sub_mod(r.m[i].c, x[4 * i + 2], q), kk, q);
            uint64_t r3 = mul_shoup(sub_mod(r.m[i].d, x[4 * i + 3], q), kk, q);
            if (ACCUM) {
                r0 = add_mod(r.acc[i].a, r0, q);
                r1 = add_mod(r.acc[i].b, r1, q);
                r2 = add_mod(r.acc[i].c, r2, q);
                r3 = add_mod(r.acc[i].d, r3, q);
            }
            st256(o_ + o + i * step, r0, r1, r2, r3);
        }
    }
};

// out[job.w] -= v  (the fused key switch: the inner-product kernel has already left
// ct + cx * P^-1 in `out`, and the ModDown matrix carries P^-1, so only the subtraction remains)
struct EpiSubFrom {
    uint64_t *out;
    uint32_t bs = 0;  // batch stride of `out` in limbs (set b of a batched launch: see NttArgs)
    uint64_t *o_ = nullptr;
    bool aligned() const { return aligned32(out); }
    template <int E> struct Regs {
        u64x4 u[E / 4];
    };
    __device__ __forceinline__ void init(const NttArgs &a, const Job &job, size_t N) { o_ = out + ((size_t)job.w + (size_t)set_idx(a) * bs) * N; }
    template <int E> __device__ __forceinline__ void preload(Regs<E> &r, size_t o, int step) const {
#pragma unroll
        for (int i = 0; i < E / 4; i++) r.u[i] = ld256(o_ + o + i * step);
    }
    template <int E> __device__ __forceinline__ void finish(const Regs<E> &r, size_t o, int step, uint64_t (&x)[E], uint64_t q) const {
#pragma unroll
        for (int i = 0; i < E / 4; i++)
            st256(o_ + o + i * step, sub_mod(r.u[i].a, x[4 * i], q), sub_mod(r.u[i].b, x[4 * i + 1], q), sub_mod(r.u[i].c, x[4 * i + 2], q),
                  sub_mod(r.u[i].d, x[4 * i + 3], q));
    }
};

// the same with a buffer per set of the batch (hoisted rotations: every result is a ciphertext of its own)
constexpr int EPI_TAB_MAX = 16;
struct EpiSubFromTab : EpiSubFrom {
    uint64_t *tab[EPI_TAB_MAX];
    bool aligned() const {
        for (auto p : tab)
            if (!aligned32(p)) return false;
        return true;
    }
};

// the epilogue of the job at hand; one with a table becomes the one without (the table stays in the kernel's parameters: indexed in a
// copy, every thread wrote it to local memory)
template <class Epi>
__device__ __forceinline__ Epi live_epi(const Epi &epi, const NttArgs &a, const Job &job, size_t N) {
    Epi e = epi;
    e.init(a, job, N);
    return e;
}
__device__ __forceinline__ EpiSubFrom live_epi(const EpiSubFromTab &epi, const NttArgs &a, const Job &job, size_t N) {
    EpiSubFrom e{};
    e.o_ = epi.tab[set_idx(a)] + (size_t)job.w * N;
    return e;
}

template <int LOG_T, int RC>
__device__ __forceinline__ int pad_idx(int e) { return e + (e >> RC); }

// ================================================================================================
// arithmetic policies
// ================================================================================================
// On B200 a 32x32->64-bit integer multiply issues at less than half the rate of a double-precision
// FMA (measured: ~26 against ~62 lanes per clock per SM), and a 64-bit Shoup product needs six of
// them. Primes below 2^50 therefore run their butterflies in FP64: residues are held as doubles with
// exact integer values, a modular product is
//     h = y*w,  l = fma(y,w,-h)            (h + l = y*w exactly)
//     c = rint(y * (w/q))                  (quotient estimate)
//     r = fma(-c, q, h) + l                (exact: |h - c q| < 2^53), r = y*w (mod q)
// and a butterfly costs 8 FP64 instructions and no integer multiply. Results are converted back to
// canonical uint64 at the end, so outputs are bit-identical to the integer path.
//
// Every policy says how large a residue may be where, in units of its own, and the stage runners below
// evaluate those rules at compile time: a correction is emitted only where a bound would be passed.
//   ct_out(B)          bound after a forward stage whose inputs are bounded by B; ct<B> is that butterfly
//   gs_sum / gs_prod   bounds of the two outputs of an inverse butterfly; gs(.., ba, bb) is that butterfly
//   group_end          what is done to a residue that changes thread between two stage groups of a pass
//   pass_end           what is done to a residue that is stored between the passes of an inverse transform
//   B_CANON / B_WORDS / B_PASS / GS_PASS   bounds of canonical input, of words below 2 q as the tensor-core conversion leaves them,
//                       of what a forward / an inverse pass stores
constexpr uint64_t FP_SMALL_LIMIT = 1ull << 41;
constexpr uint64_t FP_LIMIT = 1ull << 50;
constexpr uint64_t INT_LAZY_LIMIT = 1ull << 60;
constexpr double FP_MAGIC = 6755399441055744.0;  // 1.5 * 2^52: (v + M) - M = rint(v) for |v| < 2^51
constexpr double FP_2_52 = 4503599627370496.0;

// Primes of [2^50, 2^60): residues run up to 16 q in a 64-bit word, bounds in units of q. The quotient of the Shoup product
// leaves out the lowest of its four partial products (one low at most, so the product is below 3 q), and instead of a
// conditional subtraction per butterfly (six ALU instructions on 64-bit words) a residue is brought below 2 q by a 32-bit
// quotient estimate (four instructions) every fourth stage or so.
struct ArithIntLazy {
    using T = uint64_t;
    using Tw = W2;
    struct K {
        uint64_t q, nq;   // nq = -q mod 2^64
        uint32_t m, s;    // floor(2^(64 + s) / q), normalised to 32 bits
    };
    static constexpr int LIM = 16, RED = 2, PROD = 3, B_CANON = 1, B_WORDS = 2, B_PASS = 16, GS_PASS = 6, B_BCONV = RED;
    __device__ __forceinline__ static K make(const Mod &md, int) {
        const uint32_t s = __clz((uint32_t)md.r1);  // r1 = floor(2^64 / q), in [2^4, 2^14]
        return K{md.q, 0 - md.q, (uint32_t)((md.r1 << s) | (md.r0 >> (64 - s))), s};
    }
    using TwRaw = W2;
    static constexpr int TW_RUN = 2;  // twiddles in 32 bytes
    template <int CNT> __device__ __forceinline__ static void ldtws(TwRaw (&w)[CNT], const W2 *tw, size_t idx) { ld_pairs(w, tw + idx); }
    __device__ __forceinline__ static Tw twiddle(TwRaw w, const K &) { return w; }
    __device__ __forceinline__ static Tw ldfin(const W2 *p, const K &) { return ldg_w2(p); }
    __device__ __forceinline__ static T from_u64(uint64_t v, const K &) { return v; }
    __device__ __forceinline__ static T from_raw(uint64_t v) { return v; }
    __device__ __forceinline__ static uint64_t to_raw(T v) { return v; }
    // x - k q with k = floor(x / q) or one less: below 2 q for any x
    __device__ __forceinline__ static T reduce(T x, const K &k) {
        const uint32_t c = __umulhi((uint32_t)(x >> 32), k.m) >> k.s;
        return x + (uint64_t)c * k.nq;
    }
    __device__ __forceinline__ static T mul(T x, W2 w, const K &k) {  // below 3 q for any x
        const uint32_t xl = (uint32_t)x, xh = (uint32_t)(x >> 32), sl = (uint32_t)w.ws, sh = (uint32_t)(w.ws >> 32);
        const uint64_t t = (uint64_t)xh * sl, u = (uint64_t)xl * sh + (uint32_t)t;
        const uint64_t h = (uint64_t)xh * sh + (t >> 32) + (u >> 32);
        return x * w.w + h * k.nq;
    }
    __host__ __device__ static constexpr int ct_out(int B) { return (B + PROD > LIM ? RED : B) + PROD; }
    template <int B>
    __device__ __forceinline__ static void ct(T &a, T &b, W2 w, const K &k) {
        const uint64_t t = mul(b, w, k);
        if (B + PROD > LIM) a = reduce(a, k);
        b = a + (uint64_t)PROD * k.q - t;
        a = a + t;
    }
    // a sum over the limit is avoided by reducing the larger operand, then the other one if that is not enough
    __host__ __device__ static constexpr int red_a(int ba, int bb) { return ba + bb > LIM && (ba >= bb || bb + RED > LIM) ? RED : ba; }
    __host__ __device__ static constexpr int red_b(int ba, int bb) { return red_a(ba, bb) + bb > LIM ? RED : bb; }
    __host__ __device__ static constexpr int gs_sum(int ba, int bb) { return red_a(ba, bb) + red_b(ba, bb); }
    __host__ __device__ static constexpr int gs_prod(int, int) { return PROD; }
    __device__ __forceinline__ static void gs_in(T &a, T &b, const K &k, int ba, int bb) {
        if (red_a(ba, bb) != ba) a = reduce(a, k);
        if (red_b(ba, bb) != bb) b = reduce(b, k);
    }
    __device__ __forceinline__ static void gs(T &a, T &b, W2 w, const K &k, int ba, int bb) {
        gs_in(a, b, k, ba, bb);
        const uint64_t d = a + (uint64_t)red_b(ba, bb) * k.q - b;
        a = a + b;
        b = mul(d, w, k);
    }
    __device__ __forceinline__ static void gs_last(T &a, T &b, W2 sx, W2 sy, const K &k, int ba, int bb) {
        gs_in(a, b, k, ba, bb);
        const uint64_t d = a + (uint64_t)red_b(ba, bb) * k.q - b, s = a + b;
        a = mul_shoup(s, sx, k.q);
        b = mul_shoup(d, sy, k.q);
    }
    __host__ __device__ static constexpr int group_end_out(int B) { return B > GS_PASS ? RED : B; }
    __device__ __forceinline__ static T group_end(T v, const K &k, int B) { return B > GS_PASS ? reduce(v, k) : v; }
    __device__ __forceinline__ static T pass_end(T v, const K &k, int B) { return group_end(v, k, B); }
    __device__ __forceinline__ static uint64_t canon_fwd(T v, const K &k) { return csub(reduce(v, k), k.q); }
    // a base conversion of up to eight terms, each below 2 q (B_BCONV bounds the result of bc_end)
    __device__ __forceinline__ static T bc_add(T x, uint64_t t, const K &) { return x + t; }
    __device__ __forceinline__ static T bc_end(T x, const K &k) { return reduce(x, k); }
    __device__ __forceinline__ static uint64_t canon_inv(T v, const K &) { return v; }  // gs_last is canonical
};

// Primes of 61 bits (and whatever else does not fit above): Harvey butterflies, one conditional subtraction each; forward
// residues stay below 4 q, inverse ones below 2 q, and no bound needs tracking
struct ArithInt {
    using T = uint64_t;
    using Tw = W2;
    struct K {
        uint64_t q, q2;
    };
    static constexpr int B_CANON = 0, B_WORDS = 0, B_PASS = 0, GS_PASS = 0, B_BCONV = 0;
    __device__ __forceinline__ static K make(const Mod &md, int) { return K{md.q, 2 * md.q}; }
    using TwRaw = W2;
    static constexpr int TW_RUN = 2;  // twiddles in 32 bytes
    template <int CNT> __device__ __forceinline__ static void ldtws(TwRaw (&w)[CNT], const W2 *tw, size_t idx) { ld_pairs(w, tw + idx); }
    __device__ __forceinline__ static Tw twiddle(TwRaw w, const K &) { return w; }
    __device__ __forceinline__ static Tw ldfin(const W2 *p, const K &) { return ldg_w2(p); }
    __device__ __forceinline__ static T from_u64(uint64_t v, const K &) { return v; }
    __device__ __forceinline__ static T from_raw(uint64_t v) { return v; }
    __device__ __forceinline__ static uint64_t to_raw(T v) { return v; }
    __host__ __device__ static constexpr int ct_out(int) { return 0; }
    template <int B>
    __device__ __forceinline__ static void ct(T &a, T &b, W2 w, const K &k) { ct_bfly(a, b, w, k.q, k.q2); }
    __host__ __device__ static constexpr int gs_sum(int, int) { return 0; }
    __host__ __device__ static constexpr int gs_prod(int, int) { return 0; }
    __device__ __forceinline__ static void gs(T &a, T &b, W2 w, const K &k, int, int) { gs_bfly(a, b, w, k.q, k.q2); }
    __device__ __forceinline__ static void gs_last(T &a, T &b, W2 sx, W2 sy, const K &k, int, int) {
        const uint64_t s = a + b, d = a - b + k.q2;
        a = mul_shoup(s, sx, k.q);
        b = mul_shoup(d, sy, k.q);
    }
    __host__ __device__ static constexpr int group_end_out(int) { return 0; }
    __device__ __forceinline__ static T group_end(T v, const K &, int) { return v; }
    __device__ __forceinline__ static T pass_end(T v, const K &, int) { return v; }
    __device__ __forceinline__ static uint64_t canon_fwd(T v, const K &k) { return csub(csub(v, k.q2), k.q); }
    __device__ __forceinline__ static T bc_add(T x, uint64_t t, const K &k) { return csub(x + t, k.q2); }
    __device__ __forceinline__ static T bc_end(T x, const K &) { return x; }
    __device__ __forceinline__ static uint64_t canon_inv(T v, const K &) { return v; }
};

// FP64 residues. BIG = false: primes below 2^41, where no residue needs a correction inside a pass (a forward stage grows a
// residue by less than q, 18 q after 17 stages; an inverse pass doubles its bound 9 times at most and is renormalised at its
// end, so products never see |y| >= 2^51).
// BIG = true: primes below 2^50, bounds in sixteenths of q. A factor may be 2 q at most (|y| < 2^51, so that the quotient is
// rounded right), a sum 8 q (2^53, exact); a product of |y| <= B is below (1/2 + B/4) q.
template <bool BIG>
struct ArithFp {
    using T = double;
    struct Tw {
        double w, wq;  // w and w / q
    };
    struct K {
        double q, qinv;
    };
    static constexpr int FACTOR = 32, LIM = 128, RED = 9;
    static constexpr int B_CANON = BIG ? 16 : 0, B_WORDS = 2 * B_CANON, B_PASS = BIG ? LIM : 0, GS_PASS = BIG ? RED : 0, B_BCONV = BIG ? RED : 0;
    static constexpr bool IS_BIG = BIG;
    __host__ __device__ static constexpr int prod(int B) { return 9 + (B + 3) / 4; }
    // table entry i of an FP64 prime is one double (8 bytes); w / q is rebuilt as w * (1/q), whose
    // relative error of 2^-52 is inside the slack of the quotient estimate
    using TwRaw = double;
    static constexpr int TW_RUN = 4;  // twiddles in 32 bytes
    template <int CNT> __device__ __forceinline__ static void ldtws(TwRaw (&w)[CNT], const W2 *tw, size_t idx) {
        const double *p = reinterpret_cast<const double *>(tw) + idx;
        if constexpr (CNT == 1) {
            w[0] = __ldg(p);
        } else if constexpr (CNT == 2) {
            const double2 v = __ldg(reinterpret_cast<const double2 *>(p));
            w[0] = v.x, w[1] = v.y;
        } else {
            const u64x4 v = ld256_table(reinterpret_cast<const uint64_t *>(p));
            w[0] = from_raw(v.a), w[1] = from_raw(v.b), w[2] = from_raw(v.c), w[3] = from_raw(v.d);
        }
    }
    __device__ __forceinline__ static Tw twiddle(TwRaw w, const K &k) { return Tw{w, __dmul_rn(w, k.qinv)}; }
    __device__ __forceinline__ static Tw ldfin(const W2 *p, const K &) {
        const W2 v = ldg_w2(p);
        return Tw{__longlong_as_double((long long)v.w), __longlong_as_double((long long)v.ws)};
    }
    __device__ __forceinline__ static K make(const Mod &md, int) {
        const double q = (double)md.q;
        return K{q, md.qinv};
    }
    __device__ __forceinline__ static T from_u64(uint64_t v, const K &) {
        return __dsub_rn(__longlong_as_double((long long)(v | 0x4330000000000000ull)), FP_2_52);
    }
    __device__ __forceinline__ static T from_raw(uint64_t v) { return __longlong_as_double((long long)v); }
    __device__ __forceinline__ static uint64_t to_raw(T v) { return (uint64_t)__double_as_longlong(v); }
    __device__ __forceinline__ static T mulmod(T y, Tw w, const K &k) {
        const double wd = w.w, wq = w.wq;
        const double h = __dmul_rn(y, wd);
        const double l = __fma_rn(y, wd, -h);
        const double c = __dsub_rn(__fma_rn(y, wq, FP_MAGIC), FP_MAGIC);
        return __dadd_rn(__fma_rn(-c, k.q, h), l);
    }
    // the representative of least magnitude (|v| <= 2^53)
    __device__ __forceinline__ static T reduce(T v, const K &k) {
        const double c = __dsub_rn(__fma_rn(v, k.qinv, FP_MAGIC), FP_MAGIC);
        return __fma_rn(-c, k.q, v);
    }
    __host__ __device__ static constexpr int factor(int B) { return B > FACTOR ? RED : B; }
    __host__ __device__ static constexpr int ct_out(int B) {
        if (!BIG) return 0;
        return (B + prod(factor(B)) > LIM ? RED : B) + prod(factor(B));
    }
    template <int B>
    __device__ __forceinline__ static void ct(T &a, T &b, Tw w, const K &k) {
        if (BIG && B > FACTOR) b = reduce(b, k);
        if (BIG && B + prod(factor(B)) > LIM) a = reduce(a, k);
        const double t = mulmod(b, w, k);
        b = __dsub_rn(a, t);
        a = __dadd_rn(a, t);
    }
    __host__ __device__ static constexpr int gs_in_bound(int ba, int bb) { return ba + bb > LIM ? 2 * RED : ba + bb; }
    __host__ __device__ static constexpr int gs_sum(int ba, int bb) { return BIG ? gs_in_bound(ba, bb) : 0; }
    __host__ __device__ static constexpr int gs_prod(int ba, int bb) { return BIG ? prod(factor(gs_in_bound(ba, bb))) : 0; }
    __device__ __forceinline__ static void gs_in(T &a, T &b, const K &k, int ba, int bb) {
        if (BIG && ba + bb > LIM) a = reduce(a, k), b = reduce(b, k);
    }
    __device__ __forceinline__ static void gs(T &a, T &b, Tw w, const K &k, int ba, int bb) {
        gs_in(a, b, k, ba, bb);
        double d = __dsub_rn(a, b);
        a = __dadd_rn(a, b);
        if (BIG && gs_in_bound(ba, bb) > FACTOR) d = reduce(d, k);
        b = mulmod(d, w, k);
    }
    __device__ __forceinline__ static void gs_last(T &a, T &b, Tw sx, Tw sy, const K &k, int ba, int bb) {
        gs_in(a, b, k, ba, bb);
        double s = __dadd_rn(a, b), d = __dsub_rn(a, b);
        if (BIG && gs_in_bound(ba, bb) > FACTOR) s = reduce(s, k), d = reduce(d, k);
        a = mulmod(s, sx, k);
        b = mulmod(d, sy, k);
    }
    __host__ __device__ static constexpr int group_end_out(int B) { return B; }
    __device__ __forceinline__ static T group_end(T v, const K &, int) { return v; }
    __device__ __forceinline__ static T pass_end(T v, const K &k, int) { return reduce(v, k); }
    __device__ __forceinline__ static uint64_t to_canon(T v, const K &k) {  // |v| < q
        if (v < 0.0) v = __dadd_rn(v, k.q);
        return (uint64_t)__double_as_longlong(__dadd_rn(v, FP_2_52)) & 0x000FFFFFFFFFFFFFull;
    }
    __device__ __forceinline__ static uint64_t canon_fwd(T v, const K &k) { return to_canon(reduce(v, k), k); }
    __device__ __forceinline__ static T bc_end(T x, const K &k) { return reduce(x, k); }
    __device__ __forceinline__ static uint64_t canon_inv(T v, const K &k) { return to_canon(v, k); }
};

// calls f with the policy of the prime (uniform over a CTA)
template <class F>
__device__ __forceinline__ void with_arith(uint64_t q, F &&f) {
    if (q < FP_SMALL_LIMIT) f(ArithFp<false>{});
    else if (q < FP_LIMIT) f(ArithFp<true>{});
    else if (q < INT_LAZY_LIMIT) f(ArithIntLazy{});
    else f(ArithInt{});
}

// ---- stage runners: compile-time recursion keeps every register index a constant --------------
// forward: E residues x[] bounded by B, local stages S..R-1 of this stage group; twiddle index
// (P << (shift + S)) + (k0 << S) + g. The 2^S twiddles of a stage are one aligned run, read 32 bytes at a time: in the row passes,
// which read one per residue, the loads of single entries were a third of the LSU's work (with 1 / q from the table of primes
// instead of a division in every thread: 32 products at 2^14 710 -> 691 us, eight hoisted rotations at 2^15 255 -> 248 us).
// (MAX_RUN 1: one by one, for kernels without the registers for more)
template <class A, int S, int R, int E, int B, int MAX_RUN = A::TW_RUN>
__device__ __forceinline__ void ct_stages(typename A::T (&x)[E], const W2 *tw, size_t P, int shift, size_t k0, const typename A::K &k) {
    if constexpr (S < R) {
        constexpr int half = E >> (S + 1);
        constexpr int RUN = (1 << S) < MAX_RUN ? (1 << S) : MAX_RUN;
        typename A::TwRaw ws[RUN];
#pragma unroll
        for (int g = 0; g < (1 << S); g++) {
            if (g % RUN == 0) A::ldtws(ws, tw, (P << (shift + S)) + (k0 << S) + g);
            const typename A::Tw w = A::twiddle(ws[g % RUN], k);
#pragma unroll
            for (int j = 0; j < half; j++) A::template ct<B>(x[g * 2 * half + j], x[g * 2 * half + j + half], w, k);
        }
        ct_stages<A, S + 1, R, E, A::ct_out(B), MAX_RUN>(x, tw, P, shift, k0, k);
    }
}
// bound after R forward stages
template <class A>
__host__ __device__ constexpr int ct_bound(int B, int R) {
    for (int i = 0; i < R; i++) B = A::ct_out(B);
    return B;
}

// bounds of the E residues of a thread before local stage U of an inverse stage group that starts at bound B everywhere
template <int E>
struct GsBounds {
    int v[E];
};
template <class A, int E>
__host__ __device__ constexpr GsBounds<E> gs_bounds(int B, int U) {
    GsBounds<E> r{};
    for (int i = 0; i < E; i++) r.v[i] = B;
    for (int u = 0; u < U; u++)
        for (int i = 0; i < E; i++)
            if (!(i & (1 << u))) {
                const int j = i | (1 << u), s = A::gs_sum(r.v[i], r.v[j]), p = A::gs_prod(r.v[i], r.v[j]);
                r.v[i] = s, r.v[j] = p;
            }
    return r;
}
// bound of what a stage group of R stages hands to the next one
template <class A, int E>
__host__ __device__ constexpr int gs_group_bound(int B, int R) {
    const GsBounds<E> b = gs_bounds<A, E>(B, R);
    int m = 0;
    for (int i = 0; i < E; i++) m = m > A::group_end_out(b.v[i]) ? m : A::group_end_out(b.v[i]);
    return m;
}

// inverse: local stages U..R-1 (gap 2^U) of a group that starts at bound B; twiddle index (m0 >> U) * P + (k0 >> U) + g
// with m0 = sub-transform size >> (1 + stages already done), k0 = first pair group of this thread at U = 0.
template <class A, int U, int R, int E, int B>
__device__ __forceinline__ void gs_stages(typename A::T (&x)[E], const W2 *tw, size_t P, int m0, size_t k0, const typename A::K &k) {
    if constexpr (U < R) {
        constexpr int gap = 1 << U;
        constexpr GsBounds<E> bd = gs_bounds<A, E>(B, U);
        constexpr int RUN = (E >> (U + 1)) < A::TW_RUN ? (E >> (U + 1)) : A::TW_RUN;
        typename A::TwRaw ws[RUN];
#pragma unroll
        for (int g = 0; g < (E >> (U + 1)); g++) {
            if (g % RUN == 0) A::ldtws(ws, tw, (size_t)(m0 >> U) * P + (k0 >> U) + g);
            const typename A::Tw w = A::twiddle(ws[g % RUN], k);
#pragma unroll
            for (int j = 0; j < gap; j++) {
                const int i = g * 2 * gap + j;
                A::gs(x[i], x[i + gap], w, k, bd.v[i], bd.v[i + gap]);
            }
        }
        gs_stages<A, U + 1, R, E, B>(x, tw, P, m0, k0, k);
    }
}

// term y M of a base conversion added to the running sums (B_BCONV bounds the result of load_src)
template <bool BIG, int E>
__device__ __forceinline__ void bc_term(double (&x)[E], const uint64_t (&y)[E], W2 m, bool wide, const typename ArithFp<BIG>::K &k) {
    using F = ArithFp<BIG>;
    const double w = (double)m.w;
    const typename F::Tw t{w, __dmul_rn(w, k.qinv)};
    if (!wide) {
#pragma unroll
        for (int i = 0; i < E; i++) x[i] = __dadd_rn(x[i], F::mulmod(F::from_u64(y[i], k), t, k));
        return;
    }
    // a residue of up to 61 bits in two parts: y = yl + 2^30 yh
    const double w30 = F::mulmod(1073741824.0, t, k);
    const typename F::Tw u{w30, __dmul_rn(w30, k.qinv)};
#pragma unroll
    for (int i = 0; i < E; i++) {
        const double l = F::from_u64(y[i] & 0x3FFFFFFFu, k), h = F::from_u64(y[i] >> 30, k);
        x[i] = __dadd_rn(x[i], __dadd_rn(F::mulmod(l, t, k), F::mulmod(h, u, k)));
    }
}

// E residues of a limb at positions n0, n0 + step, .. of the transform's source
template <class A, int SRC, int E>
__device__ __forceinline__ void load_src(typename A::T (&x)[E], const NttArgs &a, const BcJob &bc, const uint64_t *src, const uint64_t *rem, size_t N, size_t n0,
                                         size_t step, const Mod &md, const typename A::K &k) {
    if constexpr (SRC & SRC_REM) {
        if constexpr (SRC & SRC_CONV) load_src<A, SRC_CONV>(x, a, bc, src, nullptr, N, n0, step, md, k);
        else if constexpr (SRC & SRC_WORDS) load_src<A, SRC_WORDS>(x, a, bc, src, nullptr, N, n0, step, md, k);
        const uint64_t q_red = SRC == SRC_REM ? 0 : barrett64(a.rem_q, md.q, md.r1);
        uint64_t v[E];
#pragma unroll
        for (int i = 0; i < E; i++) v[i] = rem[n0 + i * step];
#pragma unroll
        for (int i = 0; i < E; i++) {
            uint64_t r = barrett64(v[i], md.q, md.r1);
            if (SRC != SRC_REM && v[i] > a.rem_half) r = sub_mod(r, q_red, md.q);
            x[i] = SRC & (SRC_CONV | SRC_WORDS) ? x[i] + A::from_u64(r, k) : A::from_u64(r, k);
        }
    } else if constexpr (!(SRC & SRC_CONV)) {
#pragma unroll
        for (int i = 0; i < E; i++) x[i] = A::from_u64(src[n0 + i * step], k);
    } else {
        constexpr bool FP = std::is_same<typename A::T, double>::value;
#pragma unroll
        for (int i = 0; i < E; i++) x[i] = 0;
        const W2 *m = a.mat + bc.mat_off;
        for (uint32_t j = 0; j < bc.ni; j++) {
            uint64_t y[E];
            const uint64_t *s = src + (size_t)j * (a.src_lm1 + 1) * N + n0;
#pragma unroll
            for (int i = 0; i < E; i++) y[i] = s[i * step];
            const W2 c = ldg_w2(m + j);
            if constexpr (FP) {
                bc_term<A::IS_BIG, E>(x, y, c, (bc.wide >> j) & 1, k);
                if (A::IS_BIG && j == 3) {
#pragma unroll
                    for (int i = 0; i < E; i++) x[i] = A::reduce(x[i], k);  // eight products at most between two reductions
                }
            } else {
#pragma unroll
                for (int i = 0; i < E; i++) x[i] = A::bc_add(x[i], mul_shoup_lazy(y[i], c, md.q), k);
            }
        }
#pragma unroll
        for (int i = 0; i < E; i++) x[i] = A::bc_end(x[i], k);
    }
}

// bound of what load_src gives. Canonical words have their own: a 50-bit prime with twice the bound asks for a reduction of the factor
// from the second stage on instead of the third (B200, eight limbs forward in one launch, us on the device: 2^14 5.98 instead of 5.96,
// 2^13 6.06 instead of 6.04)
template <class A, int SRC>
__host__ __device__ constexpr int src_bound() {
    if (SRC == 0) return A::B_CANON;
    return (SRC & SRC_REM ? A::B_CANON : 0) + (SRC & SRC_CONV ? A::B_BCONV : SRC & SRC_WORDS ? A::B_WORDS : 0);
}

// ================================================================================================
// forward pass: R1 strided stages, exchange, R2 contiguous stages
// FIRST: the input holds residues as words, SRC says which (else the raw lazy values of the previous pass)
// ================================================================================================
// SRC (column pass only): where the input comes from. LOG_REST: log2(N) - LOG_T where it is known; the column passes are compiled for
// every ring, so that the rows of a column are immediate offsets of one address (sixteen key switches of 24 limbs at 2^16, forward
// columns 28.4 -> 27.1 us a key switch, inverse 13.3 -> 12.6); the row passes have unit strides and gain nothing.
template <class A, int LOG_T, int R1, int R2, int LOG_C, bool COLS, bool LAST, class Epi, int SRC, int LOG_REST>
__device__ __forceinline__ void fwd_body(const NttArgs &a, const Epi &epi, uint64_t *sm, const Job &job, uint32_t jobi, const Mod &md, uint32_t tile) {
    using T = typename A::T;
    static_assert(SRC == 0 || COLS, "the on-the-fly source belongs to the column pass");
    constexpr int B0 = COLS ? src_bound<A, SRC>() : A::B_PASS, B1 = ct_bound<A>(B0, R1);
    static_assert(ct_bound<A>(B1, R2) <= A::B_PASS, "a forward pass stores residues within B_PASS");
    constexpr bool FIRST = COLS;
    constexpr int TT = 1 << LOG_T, E1 = 1 << R1, E2 = 1 << R2, C = 1 << LOG_C;
    constexpr int EPT = E1 > E2 ? E1 : E2;
    constexpr int THREADS = C * TT / EPT;
    constexpr int TPAD = TT + (TT >> R2);
    const size_t N = (size_t)1 << (LOG_REST < 0 ? (int)a.logN : LOG_T + LOG_REST);
    const typename A::K k = A::make(md, (int)a.logN);
    const W2 *tw = a.tw + (size_t)job.y * N;
    BcJob bc{};
    if (SRC & SRC_CONV) bc = a.bc[jobi];
    const uint64_t *src = a.src + src_slot(a, SRC & SRC_CONV ? bc.in_slot0 : job.x) * N, *rem = src_rem<SRC>(a, job, N);
    const size_t estride = COLS ? (N >> LOG_T) : 1;
    const size_t cstride = COLS ? 1 : TT;
    const size_t base = COLS ? (size_t)tile * C : (size_t)tile * C * TT;
    const uint32_t n1 = (uint32_t)(N >> LOG_T);  // number of sub-transforms per limb
    const int tid = threadIdx.x;

    // ---- stage group 1 ---------------------------------------------------------------------------
#pragma unroll
    for (int gi = 0; gi < EPT / E1; gi++) {
        const int gid = tid + gi * THREADS;
        const int c = COLS ? (gid % C) : (gid / E2);
        const int elo = COLS ? (gid / C) : (gid % E2);
        const uint32_t P = COLS ? 1u : (n1 + tile * C + c);
        T x[E1];
        const size_t n0 = base + (size_t)c * cstride + (size_t)elo * estride;
        if (FIRST) {
            load_src<A, SRC>(x, a, bc, src, rem, N, n0, E2 * estride, md, k);
        } else {
#pragma unroll
            for (int i = 0; i < E1; i++) x[i] = A::from_raw(src[n0 + (size_t)i * E2 * estride]);
        }
        ct_stages<A, 0, R1, E1, B0>(x, tw, P, 0, 0, k);
#pragma unroll
        for (int i = 0; i < E1; i++) {
            const int pe = pad_idx<LOG_T, R2>(elo + i * E2);
            sm[COLS ? (pe * C + c) : (c * TPAD + pe)] = A::to_raw(x[i]);
        }
    }
    __syncthreads();
    // ---- stage group 2 ---------------------------------------------------------------------------
    const auto e = [&] {
        if constexpr (LAST) return live_epi(epi, a, job, N);
        else return epi;
    }();
    uint64_t *dst = a.dst + dst_slot(a, job.x) * N;
#pragma unroll
    for (int gi = 0; gi < EPT / E2; gi++) {
        const int gid = tid + gi * THREADS;
        const int c = COLS ? (gid % C) : (gid / E1);
        const int ehi = COLS ? (gid / C) : (gid % E1);
        const uint32_t P = COLS ? 1u : (n1 + tile * C + c);
        const size_t o = base + (size_t)c * cstride + (size_t)ehi * E2 * estride;
        // What the last pass stores goes through the exchange buffer once more: a thread holds a run of E2 residues, but its accesses
        // are to every E1-th run of four, so that those of a warp cover whole lines one after another. With the runs accessed as
        // they are every lane of a 256-bit access falls into a line of its own, and the row pass that subtracts from the ciphertext
        // stood at 84 % of the L1 (sixteen key switches of 24 limbs at 2^16: 15.1 -> 12.6 us a key switch; eight hoisted rotations at
        // 2^15 219.7 -> 212.6 us in all).
        const size_t o4 = base + (size_t)c * cstride + (size_t)ehi * 4;
        typename std::remove_const_t<decltype(e)>::template Regs<E2> regs;
        if (LAST) e.template preload<E2>(regs, o4, 4 * E1);
        T x[E2];
#pragma unroll
        for (int i = 0; i < E2; i++) {
            const int pe = pad_idx<LOG_T, R2>(ehi * E2 + i);
            x[i] = A::from_raw(sm[COLS ? (pe * C + c) : (c * TPAD + pe)]);
        }
        ct_stages<A, 0, R2, E2, B1>(x, tw, P, R1, ehi, k);
        if (LAST) {
            static_assert(!LAST || !COLS, "the last forward pass is the row pass");
            static_assert(!LAST || (32 % E1 == 0 && EPT == E2), "the threads of a sub-transform are lanes of one warp");
            uint64_t y[E2];
#pragma unroll
            for (int i = 0; i < E2; i++) sm[c * TPAD + pad_idx<LOG_T, R2>(ehi * E2 + i)] = A::canon_fwd(x[i], k);  // where this thread alone read
            __syncwarp();
#pragma unroll
            for (int i = 0; i < E2; i++) y[i] = sm[c * TPAD + pad_idx<LOG_T, R2>((i / 4 * E1 + ehi) * 4 + i % 4)];
            e.template finish<E2>(regs, o4, 4 * E1, y, md.q);
        } else {
#pragma unroll
            for (int i = 0; i < E2; i++) dst[o + (size_t)i * estride] = A::to_raw(x[i]);
        }
    }
}

template <int LOG_T, int R1, int R2, int LOG_C, bool COLS, bool LAST, class Epi, int SRC = 0, int LOG_REST = -1>
__global__ void __launch_bounds__((1 << (LOG_C + LOG_T)) / (1 << (R1 > R2 ? R1 : R2)), ntt_min_blocks((1 << (LOG_C + LOG_T)) / (1 << (R1 > R2 ? R1 : R2)), 1 << (R1 > R2 ? R1 : R2)))
ntt_fwd_pass(NttArgs a, const __grid_constant__ Epi epi) {
    pdl_enter();
    static_assert(R1 + R2 == LOG_T, "stage split");
    constexpr int TT = 1 << LOG_T, C = 1 << LOG_C;
    __shared__ uint64_t sm[C * (TT + (TT >> R2))];
    const uint32_t tiles = (uint32_t)(((size_t)1 << a.logN) >> (LOG_T + LOG_C));
    const uint32_t jobi = work_idx(a) / tiles, tile = work_idx(a) % tiles;
    const Job job = get_job(a, jobi);
    const Mod md = a.mod[job.y];
    with_arith(md.q, [&](auto A) { fwd_body<decltype(A), LOG_T, R1, R2, LOG_C, COLS, LAST, Epi, SRC, LOG_REST>(a, epi, sm, job, jobi, md, tile); });
}

// ================================================================================================
// Last forward (row) pass of ModUp fused with the key-switch inner product, for the limbs on FP64 primes (single calls) or
// for all of them (batched calls).
// A CTA owns one tile of one output limb t and walks the digits: the digit that holds limb t itself contributes the
// NTT-form input as it is, every other digit's limb t is finished here (row pass of its column-pass output) and never
// stored. Both polynomials of the key are multiplied in and summed - on FP64 primes in FP64 (|sum| < beta q), on the others
// as Montgomery products in one word (MacAcc) -, reduced once, and ct[k][t] += sum_k * P^-1, or the P limb stored, as the
// stand-alone inner-product kernel does. Same residues as that kernel.
// ================================================================================================
#define B2_MAC_MAX_BETA 8
struct MacArgs {
    const uint64_t *own;                   // NTT-form input of ModUp, [l][N]
    const uint64_t *evk[B2_MAC_MAX_BETA];  // digit d: [2][size_QP][N]
    uint64_t *ct;                          // [2][l][N]
    uint64_t *cxp;                         // [2][alpha][N]: the P limbs of the inner product
    const W2 *pinv;                        // per prime: P^-1 {w, shoup}
    const W2 *fin;                         // per prime, for the integer path: P^-1 * 2^64 mod q (Q), 2^64 mod p (P)
    uint32_t l, lP, alpha, beta, size_Q, size_QP, acc_p;
    uint32_t interleave;                   // consecutive CTAs walk the limbs of one tile (else the tiles of one limb)
    // a batched launch (one key for every set): set b = blockIdx.x, so that the CTAs which read the same key tile run next
    // to one another and all but the first find it in L2; its digits, NTT-form input, ciphertext and P limbs start
    // b * dig_bs / own_bs / ct_bs / cxp_bs limbs further
    uint32_t dig_bs, own_bs, ct_bs, cxp_bs;  // (with the sets as the slow dimension instead the pass took 30.7 instead of 27.8 us per key switch)
    uint32_t p_first, first_limb;          // the grid covers p_first P limbs, then the Q limbs from first_limb on
    uint32_t p_off;                        // index of the first of those P limbs (a rank's slice under limb sharding; else 0)
    // P limb i of polynomial k of set b lands at limb slot i * cxp_i + k * cxp_k + b * cxp_bs of cxp: [set][2][alpha] is
    // (1, alpha, 2 alpha), the limb-major exchange buffer [alpha][2][sets] is (2 sets, sets, 1)
    uint32_t cxp_i, cxp_k;
    // a rotation: `own` and, added to polynomial 0, c0 [l][N] are read through perm; ct_set: ct is overwritten, not added to
    const uint32_t *perm;
    const uint64_t *c0;
    uint32_t ct_set, c0_bs;  // c0 of set b of a batch starts b * c0_bs limbs further
};

__device__ __forceinline__ void cp_async16(void *smem_dst, const void *gsrc) {
    const uint32_t d = (uint32_t)__cvta_generic_to_shared(smem_dst);
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(d), "l"(gsrc) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int KEEP>
__device__ __forceinline__ void cp_async_wait() {
    asm volatile("cp.async.wait_group %0;" ::"n"(KEEP) : "memory");
}

// bytes of dynamic shared memory the kernel wants: the exchange buffer and one digit's two key polynomials for the tile
template <int LOG_T, int R, int LOG_C>
constexpr size_t mac_smem_bytes() {
    return (size_t)((1 << LOG_C) * ((1 << LOG_T) + ((1 << LOG_T) >> R)) + 2 * (1 << (LOG_C + LOG_T))) * 8;
}

// How the fused pass multiplies a finished digit residue into a key word and sums over the digits, per arithmetic.
// FP64 primes: the signed products (below q in magnitude) are summed as doubles and reduced once.
// Integer primes: a Montgomery product y * key * 2^-64 (four 64-bit multiplies, no correction step: the key word is
// below q, so any 64-bit y gives a value below 2q) summed in one 64-bit word - 128-bit accumulators for sixteen residues
// times two polynomials would not fit the register file, and a Barrett reduction per product costs twice the multiplies.
// The factor 2^-64 is undone by the constant of the final multiplication (MacArgs::fin).
template <class A> struct MacAcc {
    using T = uint64_t;
    using K = typename A::K;
    struct C {
        uint64_t q, q2, ninv;  // ninv = -q^-1 mod 2^64
        bool tight;            // 2 * beta * q could pass 2^64: keep the sum below 2q after every term
    };
    __device__ __forceinline__ static C make(const Mod &md) {
        uint64_t x = md.q;  // q * q = 1 mod 8; every Newton step doubles the valid bits
#pragma unroll
        for (int i = 0; i < 5; i++) x *= 2 - md.q * x;
        return C{md.q, 2 * md.q, 0 - x, (md.q >> 59) != 0};
    }
    __device__ __forceinline__ static T zero() { return 0; }
    __device__ __forceinline__ static uint64_t operand(uint64_t y, const K &) { return y; }  // any lazy value does
    __device__ __forceinline__ static void mac(T &acc, uint64_t y, uint64_t key, const K &, const C &c) {
        const uint64_t lo = y * key, hi = __umul64hi(y, key);
        const uint64_t m = lo * c.ninv;
        // (y key + m q) / 2^64: the low words cancel, carrying one unless lo is zero
        acc += hi + __umul64hi(m, c.q) + (lo != 0);
        if (c.tight) acc = csub(acc, c.q2);
    }
    // sum * 2^-64 times the limb's closing constant, canonical
    __device__ __forceinline__ static uint64_t finish(T acc, W2 fin, const K &, const C &c) { return mul_shoup(acc, fin, c.q); }
};
template <bool BIG> struct MacAcc<ArithFp<BIG>> {
    using Fp = ArithFp<BIG>;
    using T = double;
    using K = typename Fp::K;
    struct C {};
    __device__ __forceinline__ static C make(const Mod &) { return C{}; }
    __device__ __forceinline__ static T zero() { return 0.0; }
    __device__ __forceinline__ static double operand(double y, const K &k) { return Fp::reduce(y, k); }
    __device__ __forceinline__ static void mac(T &acc, double y, uint64_t key, const K &k, const C &) {
        const double w = Fp::from_u64(key, k);
        acc = __dadd_rn(acc, Fp::mulmod(y, typename Fp::Tw{w, __dmul_rn(w, k.qinv)}, k));
    }
    // canonical residue of the sum
    __device__ __forceinline__ static uint64_t finish(T acc, W2, const K &k, const C &) { return Fp::canon_fwd(acc, k); }
};

// One tile of one output limb t (logical index: Q limbs 0 .. l-1, then the P limbs) through all digits.
template <class A, int LOG_T, int R, int LOG_C>
__device__ __forceinline__ void mac_body(const NttArgs &a, const MacArgs &m, uint64_t *sm, uint64_t *kb, uint32_t t, uint32_t pp, uint32_t tile,
                                         uint32_t bset, const Mod &md) {
    using T = typename A::T;
    using Acc = MacAcc<A>;
    constexpr int TT = 1 << LOG_T, E = 1 << R, C = 1 << LOG_C;
    constexpr int TPAD = TT + (TT >> R), THREADS = (C * TT) >> R;
    static_assert(E == 16, "the key staging below gives every thread eight 16-byte chunks per polynomial");
    const size_t N = (size_t)1 << a.logN;
    const typename A::K k = A::make(md, (int)a.logN);
    const W2 *tw = a.tw + (size_t)pp * N;
    const uint32_t n1 = (uint32_t)(N >> LOG_T);
    const int tid = threadIdx.x;
    const int c = tid / E, e = tid % E;  // sub-transform of the tile, register group within it (both stage groups)
    const uint32_t P = n1 + tile * C + c;
    const size_t base = (size_t)tile * C * TT;
    const size_t o = base + (size_t)c * TT + (size_t)e * E;  // this thread's E consecutive outputs: tid * 16 into the tile
    const uint32_t own_d = t < m.l ? t / m.alpha : 0xFFFFFFFFu;  // a P limb belongs to no digit
    const typename Acc::C mc = Acc::make(md);
    typename Acc::T acc0[E], acc1[E];
#pragma unroll
    for (int i = 0; i < E; i++) acc0[i] = acc1[i] = Acc::zero();
    for (uint32_t d = 0; d < m.beta; d++) {
        // The digit's key tile starts its way from HBM now (cp.async, L1 bypassed: the key is read once) and is waited for
        // only after this digit's butterflies: a thread's eight 16-byte chunks of a polynomial are XOR-swizzled inside its
        // 128-byte row so that the 128-bit reads below are free of bank conflicts.
        {
            const uint64_t *g0 = m.evk[d] + (size_t)pp * N + base, *g1 = g0 + (size_t)m.size_QP * N;
#pragma unroll
            for (int g = tid; g < C * TT / 2; g += THREADS) {
                const int owner = g >> 3, chunk = g & 7, off = owner * 16 + ((chunk ^ (owner & 7)) << 1);
                cp_async16(kb + off, g0 + 2 * g);
                cp_async16(kb + C * TT + off, g1 + 2 * g);
            }
            cp_async_commit();
        }
        T y[E];
        if (d == own_d && m.perm) {
            const uint64_t *src = m.own + ((size_t)bset * m.own_bs + t) * N;
#pragma unroll
            for (int i = 0; i < E; i += 4) {
                const uint4 v = *reinterpret_cast<const uint4 *>(m.perm + o + i);
                y[i] = A::from_u64(src[v.x], k), y[i + 1] = A::from_u64(src[v.y], k), y[i + 2] = A::from_u64(src[v.z], k), y[i + 3] = A::from_u64(src[v.w], k);
            }
        } else if (d == own_d) {
#pragma unroll
            for (int i = 0; i < E; i += 4) {
                const u64x4 v = ld256(m.own + ((size_t)bset * m.own_bs + t) * N + o + i);
                y[i] = A::from_u64(v.a, k), y[i + 1] = A::from_u64(v.b, k), y[i + 2] = A::from_u64(v.c, k), y[i + 3] = A::from_u64(v.d, k);
            }
        } else {
            const uint64_t *src = a.src + ((size_t)bset * m.dig_bs + (size_t)d * m.lP + t) * N + base + (size_t)c * TT + e;
#pragma unroll
            for (int i = 0; i < E; i++) y[i] = A::from_raw(src[i * E]);
            ct_stages<A, 0, R, E, A::B_PASS, 1>(y, tw, P, 0, 0, k);
#pragma unroll
            for (int i = 0; i < E; i++) sm[c * TPAD + pad_idx<LOG_T, R>(e + i * E)] = A::to_raw(y[i]);
            __syncthreads();
#pragma unroll
            for (int i = 0; i < E; i++) y[i] = A::from_raw(sm[c * TPAD + pad_idx<LOG_T, R>(e * E + i)]);
            ct_stages<A, 0, R, E, ct_bound<A>(A::B_PASS, R), 1>(y, tw, P, R, e, k);
#pragma unroll
            for (int i = 0; i < E; i++) y[i] = Acc::operand(y[i], k);
        }
        cp_async_wait<0>();
        __syncthreads();  // every thread's share of the key tile has landed
#pragma unroll
        for (int i = 0; i < E; i += 2) {
            const int off = tid * 16 + (((i >> 1) ^ (tid & 7)) << 1);
            const ulonglong2 u = *reinterpret_cast<const ulonglong2 *>(kb + off), v = *reinterpret_cast<const ulonglong2 *>(kb + C * TT + off);
            Acc::mac(acc0[i], y[i], u.x, k, mc);
            Acc::mac(acc0[i + 1], y[i + 1], u.y, k, mc);
            Acc::mac(acc1[i], y[i], v.x, k, mc);
            Acc::mac(acc1[i + 1], y[i + 1], v.y, k, mc);
        }
        __syncthreads();  // the key tile and the exchange buffer are free for the next digit
    }
    const uint64_t q = md.q;
    if (t < m.l) {
        // a Q limb: ct[k][t] += sum * P^-1. FP64 sums are canonical first and take P^-1; integer sums carry 2^-64 and
        // take P^-1 * 2^64 in the same single multiplication.
        constexpr bool FP = std::is_same<typename A::T, double>::value;
        const W2 pi = FP ? m.pinv[pp] : m.fin[pp];
        uint64_t *c0 = m.ct + ((size_t)bset * m.ct_bs + t) * N + o, *c1 = c0 + (size_t)m.l * N;
#pragma unroll
        for (int i = 0; i < E; i += 4) {
            uint64_t r[4], s[4];
#pragma unroll
            for (int j = 0; j < 4; j++) {
                r[j] = Acc::finish(acc0[i + j], pi, k, mc);
                s[j] = Acc::finish(acc1[i + j], pi, k, mc);
                if (FP) r[j] = mul_shoup(r[j], pi, q), s[j] = mul_shoup(s[j], pi, q);
            }
            if (m.c0) {
                const uint64_t *src = m.c0 + ((size_t)bset * m.c0_bs + t) * N;
                const uint4 v = *reinterpret_cast<const uint4 *>(m.perm + o + i);
                r[0] = add_mod(r[0], src[v.x], q), r[1] = add_mod(r[1], src[v.y], q), r[2] = add_mod(r[2], src[v.z], q), r[3] = add_mod(r[3], src[v.w], q);
            }
            if (!m.ct_set) {
                const u64x4 u = ld256(c0 + i), v = ld256(c1 + i);
                r[0] = add_mod(u.a, r[0], q), r[1] = add_mod(u.b, r[1], q), r[2] = add_mod(u.c, r[2], q), r[3] = add_mod(u.d, r[3], q);
                s[0] = add_mod(v.a, s[0], q), s[1] = add_mod(v.b, s[1], q), s[2] = add_mod(v.c, s[2], q), s[3] = add_mod(v.d, s[3], q);
            }
            st256(c0 + i, r[0], r[1], r[2], r[3]);
            st256(c1 + i, s[0], s[1], s[2], s[3]);
        }
    } else {
        // a P limb: kept (or, acc_p, added to what is there) in the compact buffer [2][alpha][N] for the ModDown that
        // follows; the closing constant of an integer prime is 2^64 mod p
        const W2 fin = m.fin[pp];
        uint64_t *p0 = m.cxp + ((size_t)bset * m.cxp_bs + (size_t)(t - m.l) * m.cxp_i) * N + o, *p1 = p0 + (size_t)m.cxp_k * N;
#pragma unroll
        for (int i = 0; i < E; i += 4) {
            uint64_t r[4], s[4];
#pragma unroll
            for (int j = 0; j < 4; j++) {
                r[j] = Acc::finish(acc0[i + j], fin, k, mc);
                s[j] = Acc::finish(acc1[i + j], fin, k, mc);
            }
            if (m.acc_p) {
                const u64x4 u = ld256(p0 + i), v = ld256(p1 + i);
                r[0] = add_mod(r[0], u.a, q), r[1] = add_mod(r[1], u.b, q), r[2] = add_mod(r[2], u.c, q), r[3] = add_mod(r[3], u.d, q);
                s[0] = add_mod(s[0], v.a, q), s[1] = add_mod(s[1], v.b, q), s[2] = add_mod(s[2], v.c, q), s[3] = add_mod(s[3], v.d, q);
            }
            st256(p0 + i, r[0], r[1], r[2], r[3]);
            st256(p1 + i, s[0], s[1], s[2], s[3]);
        }
    }
}

template <int LOG_T, int R, int LOG_C>
__global__ void __launch_bounds__((1 << (LOG_C + LOG_T)) >> R, 3) ntt_fwd_rows_mac(NttArgs a, const __grid_constant__ MacArgs m) {
    pdl_enter();
    static_assert(2 * R == LOG_T, "equal stage groups: one register group per thread in both");
    constexpr int TT = 1 << LOG_T, C = 1 << LOG_C;
    constexpr int TPAD = TT + (TT >> R);
    extern __shared__ __align__(16) uint64_t mac_smem[];
    uint64_t *sm = mac_smem;             // [C][TPAD] exchange buffer of the row pass
    uint64_t *kb = mac_smem + C * TPAD;  // [2][C * TT] the tile of both key polynomials of the digit in hand
    const uint32_t tiles = (uint32_t)(((size_t)1 << a.logN) >> (LOG_T + LOG_C));
    // the P limbs (60-bit primes: the long CTAs) go first so that they do not form the tail of the grid
    const uint32_t n_limbs = gridDim.y / tiles, bset = blockIdx.x;
    const uint32_t i = m.interleave ? blockIdx.y % n_limbs : blockIdx.y / tiles, tile = m.interleave ? blockIdx.y / n_limbs : blockIdx.y % tiles;
    const uint32_t t = i < m.p_first ? m.l + m.p_off + i : m.first_limb + (i - m.p_first);
    const uint32_t pp = t < m.l ? t : m.size_Q + (t - m.l);  // the limb's prime
    const Mod md = a.mod[pp];
    with_arith(md.q, [&](auto A) { mac_body<decltype(A), LOG_T, R, LOG_C>(a, m, sm, kb, t, pp, tile, bset, md); });
}

// ================================================================================================
// inverse pass: RA contiguous stages, exchange, RB strided stages
// ================================================================================================
template <class A, int LOG_T, int RA, int RB, int LOG_C, bool COLS, bool LAST, int LOG_REST>
__device__ __forceinline__ void inv_body(const NttArgs &a, uint64_t *sm, const Job &job, const Mod &md, uint32_t tile) {
    using T = typename A::T;
    constexpr bool FIRST = !COLS;
    constexpr int TT = 1 << LOG_T, EA = 1 << RA, EB = 1 << RB, C = 1 << LOG_C;
    constexpr int EPT = EA > EB ? EA : EB;
    constexpr int THREADS = C * TT / EPT;
    constexpr int TPAD = TT + (TT >> RA);
    const size_t N = (size_t)1 << (LOG_REST < 0 ? (int)a.logN : LOG_T + LOG_REST);
    const typename A::K k = A::make(md, (int)a.logN);
    const W2 *tw = a.tw + (size_t)job.y * N;
    const uint64_t *src = a.src + src_slot(a, FIRST ? job.x : job.w) * N;  // the second pass works in place on dst
    uint64_t *dst = a.dst + dst_slot(a, job.w) * N;
    const size_t estride = COLS ? (N >> LOG_T) : 1;
    const size_t cstride = COLS ? 1 : TT;
    const size_t base = COLS ? (size_t)tile * C : (size_t)tile * C * TT;
    const uint32_t n1 = (uint32_t)(N >> LOG_T);
    const int tid = threadIdx.x;
    constexpr int B0 = FIRST ? A::B_CANON : A::GS_PASS, B1 = gs_group_bound<A, EA>(B0, RA);
    constexpr GsBounds<EA> end_a = gs_bounds<A, EA>(B0, RA);

    // ---- stage group 1: contiguous runs of EA residues ----------------------------------------------
#pragma unroll
    for (int gi = 0; gi < EPT / EA; gi++) {
        const int gid = tid + gi * THREADS;
        const int c = COLS ? (gid % C) : (gid / EB);
        const int ehi = COLS ? (gid / C) : (gid % EB);
        const uint32_t P = COLS ? 1u : (n1 + tile * C + c);
        T x[EA];
        const uint64_t *p = src + base + (size_t)c * cstride + (size_t)ehi * EA * estride;
        if (COLS) {
#pragma unroll
            for (int i = 0; i < EA; i++) {
                const uint64_t v = p[(size_t)i * estride];
                x[i] = FIRST ? A::from_u64(v, k) : A::from_raw(v);
            }
        } else if (FIRST && a.perm) {
            // an aligned run of EA values comes from an aligned run of EA values: whole sectors are used
            const uint32_t *pm = a.perm + base + (size_t)c * cstride + (size_t)ehi * EA;
#pragma unroll
            for (int i = 0; i < EA; i += 4) {
                const uint4 v = *reinterpret_cast<const uint4 *>(pm + i);
                x[i] = A::from_u64(src[v.x], k), x[i + 1] = A::from_u64(src[v.y], k);
                x[i + 2] = A::from_u64(src[v.z], k), x[i + 3] = A::from_u64(src[v.w], k);
            }
        } else {
#pragma unroll
            for (int i = 0; i < EA; i += 4) {
                const u64x4 v = ld256(p + i);
                x[i] = FIRST ? A::from_u64(v.a, k) : A::from_raw(v.a);
                x[i + 1] = FIRST ? A::from_u64(v.b, k) : A::from_raw(v.b);
                x[i + 2] = FIRST ? A::from_u64(v.c, k) : A::from_raw(v.c);
                x[i + 3] = FIRST ? A::from_u64(v.d, k) : A::from_raw(v.d);
            }
        }
        gs_stages<A, 0, RA, EA, B0>(x, tw, P, TT >> 1, (size_t)ehi * (EA >> 1), k);
#pragma unroll
        for (int i = 0; i < EA; i++) {
            const int pe = pad_idx<LOG_T, RA>(ehi * EA + i);
            sm[COLS ? (pe * C + c) : (c * TPAD + pe)] = A::to_raw(A::group_end(x[i], k, end_a.v[i]));
        }
    }
    __syncthreads();
    // ---- stage group 2: stride EA ---------------------------------------------------------------------
#pragma unroll
    for (int gi = 0; gi < EPT / EB; gi++) {
        const int gid = tid + gi * THREADS;
        const int c = COLS ? (gid % C) : (gid / EA);
        const int elo = COLS ? (gid / C) : (gid % EA);
        const uint32_t P = COLS ? 1u : (n1 + tile * C + c);
        T x[EB];
#pragma unroll
        for (int i = 0; i < EB; i++) {
            const int pe = pad_idx<LOG_T, RA>(elo + i * EA);
            x[i] = A::from_raw(sm[COLS ? (pe * C + c) : (c * TPAD + pe)]);
        }
        gs_stages<A, 0, (LAST ? RB - 1 : RB), EB, B1>(x, tw, P, TT >> (RA + 1), 0, k);
        constexpr GsBounds<EB> end_b = gs_bounds<A, EB>(B1, LAST ? RB - 1 : RB);
        uint64_t *o = dst + base + (size_t)c * cstride + (size_t)elo * estride;
        if (LAST) {
            // last stage of the whole transform (twiddle index 1): the x outputs take the scale,
            // the y outputs a twiddle that already carries it (src/host/ntt.cu:53-55,
            // include/ntt_radix8_tmpl.cuh:566-568); callers fold further per-limb factors in.
            constexpr int gap = EB / 2;
            const typename A::Tw sx = A::ldfin(a.fin + 2 * (size_t)job.z, k);
            const typename A::Tw sy = A::ldfin(a.fin + 2 * (size_t)job.z + 1, k);
#pragma unroll
            for (int j = 0; j < gap; j++) A::gs_last(x[j], x[j + gap], sx, sy, k, end_b.v[j], end_b.v[j + gap]);
#pragma unroll
            for (int i = 0; i < EB; i++) o[(size_t)i * EA * estride] = A::canon_inv(x[i], k);
        } else {
#pragma unroll
            for (int i = 0; i < EB; i++) o[(size_t)i * EA * estride] = A::to_raw(A::pass_end(x[i], k, end_b.v[i]));
        }
    }
}

template <int LOG_T, int RA, int RB, int LOG_C, bool COLS, bool LAST, int LOG_REST = -1>
__global__ void __launch_bounds__((1 << (LOG_C + LOG_T)) / (1 << (RA > RB ? RA : RB)), ntt_min_blocks((1 << (LOG_C + LOG_T)) / (1 << (RA > RB ? RA : RB)), 1 << (RA > RB ? RA : RB)))
ntt_inv_pass(NttArgs a) {
    pdl_enter();
    static_assert(RA + RB == LOG_T, "stage split");
    constexpr int TT = 1 << LOG_T, C = 1 << LOG_C;
    __shared__ uint64_t sm[C * (TT + (TT >> RA))];
    const uint32_t tiles = (uint32_t)(((size_t)1 << a.logN) >> (LOG_T + LOG_C));
    const uint32_t jobi = work_idx(a) / tiles, tile = work_idx(a) % tiles;
    const Job job = get_job(a, jobi);
    const Mod md = a.mod[job.y];
    with_arith(md.q, [&](auto A) { inv_body<decltype(A), LOG_T, RA, RB, LOG_C, COLS, LAST, LOG_REST>(a, sm, job, md, tile); });
}

}  // namespace b2
