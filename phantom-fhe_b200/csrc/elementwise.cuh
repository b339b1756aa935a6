// elementwise.cuh - everything that works on residues position by position: sums of products (BSGS giants, weighted sums,
// the key-switch inner product), tensor product, limb arithmetic, automorphisms, expansion of signed coefficients.
//
// Layout of every kernel here: blockIdx.y = limb, blockIdx.x = a run of coefficients of that limb, so that the prime and its
// constants are uniform over a CTA and no thread divides by N.
#pragma once
#include "modarith.cuh"
#include "ntt_kernels.cuh"

namespace b2 {

// ---- products of canonical residues ------------------------------------------------------------------------------------
// x y mod q by Barrett with one 64-bit quotient estimate: n = bit length of q, t = floor(x y / 2^(n-2)) < 2^(n+2),
// mu = floor(2^(62+n) / q) < 2^63; the estimate is short by one at most. Eight partial products instead of the sixteen of a
// 128-bit ratio.
__device__ __forceinline__ uint64_t mul_mod(uint64_t x, uint64_t y, const Mod &m) {
    const int n = 64 - __clzll((long long)m.q);
    const uint64_t lo = x * y, hi = __umul64hi(x, y);
    const uint64_t t = (hi << (66 - n)) | (lo >> (n - 2));
    return csub(lo - __umul64hi(t, m.mu) * m.q, m.q);
}

// the same for a sum of up to four products, q below 2^60: t < 2^64, the estimate is short by two at most
__device__ __forceinline__ uint64_t reduce_sum4(u128 x, const Mod &m) {
    const int n = 64 - __clzll((long long)m.q);
    const uint64_t t = (x.hi << (66 - n)) | (x.lo >> (n - 2));
    const uint64_t r = x.lo - __umul64hi(t, m.mu) * m.q;
    return csub(csub(r, 2 * m.q), m.q);
}

// ---- sums of products: how operands are held and summed, per prime class -------------------------------------------------
//   A, B     an operand as the sum wants it (split, or with its quotient); Acc the running sum; FLUSH how many terms it takes
//   flush    brings a full sum back to where it takes FLUSH terms again
//   finish   the canonical residue;  finish_mul the canonical residue times w
// Primes below 2^41: 21-bit pieces, four exact FP64 FMAs per term, no reduction until the end (a term adds less than 2^43).
struct SumFp21 {
    using F = ArithFp<false>;
    struct A {
        double l, h;
    };
    using B = A;
    struct K {
        F::K k;
        double w21, w42;  // 2^21, 2^42 mod q, least magnitude
    };
    struct Acc {
        double a0, a1, a2;
    };
    static constexpr int FLUSH = 120;
    __device__ __forceinline__ static K make(const Mod &m) {
        K r;
        r.k = F::make(m, 0);
        r.w21 = F::reduce(2097152.0, r.k), r.w42 = F::reduce(4398046511104.0, r.k);
        return r;
    }
    __device__ __forceinline__ static void zero(Acc &a) { a.a0 = a.a1 = a.a2 = 0.0; }
    __device__ __forceinline__ static A ld_a(uint64_t v, const K &) {
        return A{__dsub_rn(__longlong_as_double((long long)((v & 0x1FFFFF) | 0x4330000000000000ull)), FP_2_52),
                 __dsub_rn(__longlong_as_double((long long)((v >> 21) | 0x4330000000000000ull)), FP_2_52)};
    }
    __device__ __forceinline__ static B ld_b(uint64_t v, const K &k) { return ld_a(v, k); }
    __device__ __forceinline__ static void mac(Acc &s, const A &x, const B &y, const K &) {
        s.a0 = __fma_rn(x.l, y.l, s.a0);
        s.a1 = __fma_rn(x.l, y.h, __fma_rn(x.h, y.l, s.a1));
        s.a2 = __fma_rn(x.h, y.h, s.a2);
    }
    // a0 + a1 2^21 + a2 2^42, within 2 q + |a0|; |a1|, |a2| < 2^50
    __device__ __forceinline__ static double value(const Acc &s, const K &k) {
        const double u = F::mulmod(s.a1, F::Tw{k.w21, __dmul_rn(k.w21, k.k.qinv)}, k.k), v = F::mulmod(s.a2, F::Tw{k.w42, __dmul_rn(k.w42, k.k.qinv)}, k.k);
        return __dadd_rn(s.a0, __dadd_rn(u, v));
    }
    __device__ __forceinline__ static void flush(Acc &s, const K &k) { s = Acc{F::reduce(value(s, k), k.k), 0.0, 0.0}; }
    __device__ __forceinline__ static uint64_t finish(const Acc &s, const K &k) { return F::canon_fwd(value(s, k), k.k); }
    __device__ __forceinline__ static uint64_t finish_mul(const Acc &s, W2 w, const K &k) {
        const double wd = (double)w.w;
        return F::to_canon(F::mulmod(F::reduce(value(s, k), k.k), F::Tw{wd, __dmul_rn(wd, k.k.qinv)}, k.k), k.k);
    }
};
// Primes below 2^50: FP64 modular products (below 3/4 q in magnitude), summed up to 8 q = 2^53.
struct SumFp {
    using F = ArithFp<true>;
    using A = F::Tw;
    using B = double;
    using K = F::K;
    using Acc = double;
    static constexpr int FLUSH = 8;
    __device__ __forceinline__ static K make(const Mod &m) { return F::make(m, 0); }
    __device__ __forceinline__ static void zero(Acc &a) { a = 0.0; }
    __device__ __forceinline__ static A ld_a(uint64_t v, const K &k) {
        const double w = F::from_u64(v, k);
        return A{w, __dmul_rn(w, k.qinv)};
    }
    __device__ __forceinline__ static B ld_b(uint64_t v, const K &k) { return F::from_u64(v, k); }
    __device__ __forceinline__ static void mac(Acc &s, const A &x, B y, const K &k) { s = __dadd_rn(s, F::mulmod(y, x, k)); }
    __device__ __forceinline__ static void flush(Acc &s, const K &k) { s = F::reduce(s, k); }
    __device__ __forceinline__ static uint64_t finish(const Acc &s, const K &k) { return F::canon_fwd(s, k); }
    __device__ __forceinline__ static uint64_t finish_mul(const Acc &s, W2 w, const K &k) {
        return F::to_canon(F::mulmod(F::reduce(s, k), ld_a(w.w, k), k), k);
    }
};
// Primes below 2^60: 30-bit halves, four wide multiply-adds per term straight into 64-bit sums (two terms a sum of the
// middle weight, each below 2^60: sixteen fit), against four wide multiplies and eight carry instructions of a 128-bit sum.
struct SumInt30 {
    struct A {
        uint32_t l, h;
    };
    using B = A;
    using K = Mod;
    struct Acc {
        uint64_t s0, s1, s2;
        uint32_t s3;  // weights 2^0, 2^30, 2^60, 2^120
    };
    static constexpr int FLUSH = 8;
    __device__ __forceinline__ static K make(const Mod &m) { return m; }
    __device__ __forceinline__ static void zero(Acc &a) { a.s0 = a.s1 = a.s2 = 0, a.s3 = 0; }
    __device__ __forceinline__ static A ld_a(uint64_t v, const K &) { return A{(uint32_t)v & 0x3FFFFFFFu, (uint32_t)(v >> 30)}; }
    __device__ __forceinline__ static B ld_b(uint64_t v, const K &k) { return ld_a(v, k); }
    __device__ __forceinline__ static void mac(Acc &s, const A &x, const B &y, const K &) {
        s.s0 += (uint64_t)x.l * y.l;
        s.s1 += (uint64_t)x.l * y.h;
        s.s1 += (uint64_t)x.h * y.l;
        s.s2 += (uint64_t)x.h * y.h;
    }
    __device__ __forceinline__ static void carry(Acc &s) {
        s.s1 += s.s0 >> 30, s.s0 &= 0x3FFFFFFFu;
        s.s2 += s.s1 >> 30, s.s1 &= 0x3FFFFFFFu;
        s.s3 += (uint32_t)(s.s2 >> 60), s.s2 &= 0x0FFFFFFFFFFFFFFFull;
    }
    __device__ __forceinline__ static u128 total(Acc s) {
        carry(s);
        const uint64_t low = s.s0 | (s.s1 << 30);  // 60 bits
        return u128{low | (s.s2 << 60), (s.s2 >> 4) | ((uint64_t)s.s3 << 56)};
    }
    __device__ __forceinline__ static void flush(Acc &s, const K &k) {
        carry(s);
        if (s.s3 >= 128) {  // the sum nears 2^128
            const uint64_t r = barrett128(total(s), k.q, k.r0, k.r1);
            s = Acc{r & 0x3FFFFFFFu, r >> 30, 0, 0};
        }
    }
    __device__ __forceinline__ static uint64_t finish(const Acc &s, const K &k) { return barrett128(total(s), k.q, k.r0, k.r1); }
    __device__ __forceinline__ static uint64_t finish_mul(const Acc &s, W2 w, const K &k) { return mul_shoup(finish(s, k), w, k.q); }
};
// at most four terms: half the multiplications at the end
struct SumInt30Short : SumInt30 {
    __device__ __forceinline__ static uint64_t finish(const Acc &s, const K &k) { return reduce_sum4(total(s), k); }
    __device__ __forceinline__ static uint64_t finish_mul(const Acc &s, W2 w, const K &k) { return mul_shoup(finish(s, k), w, k.q); }
};
// Any prime up to 61 bits: 128-bit sums
struct SumInt {
    using A = uint64_t;
    using B = uint64_t;
    using K = Mod;
    using Acc = u128;
    static constexpr int FLUSH = 31;
    __device__ __forceinline__ static K make(const Mod &m) { return m; }
    __device__ __forceinline__ static void zero(Acc &a) { a = u128{0, 0}; }
    __device__ __forceinline__ static A ld_a(uint64_t v, const K &) { return v; }
    __device__ __forceinline__ static B ld_b(uint64_t v, const K &) { return v; }
    __device__ __forceinline__ static void mac(Acc &s, A x, B y, const K &) { mac128(s, x, y); }
    __device__ __forceinline__ static void flush(Acc &s, const K &k) { s = u128{barrett128(s, k.q, k.r0, k.r1), 0}; }
    __device__ __forceinline__ static uint64_t finish(const Acc &s, const K &k) { return barrett128(s, k.q, k.r0, k.r1); }
    __device__ __forceinline__ static uint64_t finish_mul(const Acc &s, W2 w, const K &k) { return mul_shoup(finish(s, k), w, k.q); }
};
template <class F>
__device__ __forceinline__ void with_sum(uint64_t q, F &&f) {
    if (q < FP_SMALL_LIMIT) f(SumFp21{});
    else if (q < FP_LIMIT) f(SumFp{});
    else if (q < INT_LAZY_LIMIT) f(SumInt30{});
    else f(SumInt{});
}

// ---- BSGS giant step (src/bsgs.cu:51-96): out_g[k] = sum_b pt[g][b] (.) baby_b[k], up to G giants per launch --------------
// Every baby value is loaded once and multiplied into each giant's own plaintext, so the babies (two thirds of the bytes of a
// single giant) cross HBM once per launch. pts[g * M + b] may be null: that giant has no diagonal for baby b.
// The table of pointers is read through shared memory, MAC_CHUNK babies at a time, and MAC_U babies' loads are issued before
// the first multiply. With 128-bit integer sums and the pointers read in the loop (b then p then data) the launch of four
// giants x 32 babies at N = 2^16, 16 limbs took 747 us for 1.6 GB.
constexpr int MAC_CHUNK = 64, MAC_U = 4;

template <class S, int G>
__device__ __forceinline__ void bsgs_mac_body(const uint64_t *const *pts, const uint64_t *const *babies, uint64_t *const *outs, uint64_t *out,
                                              const uint64_t **sp, const Mod &md, size_t S_words, size_t idx, uint32_t M, uint32_t n_g) {
    const typename S::K k = S::make(md);
    typename S::Acc acc[G][2];
#pragma unroll
    for (int g = 0; g < G; g++) S::zero(acc[g][0]), S::zero(acc[g][1]);
    int pending = 0;
    for (uint32_t c0 = 0; c0 < M; c0 += MAC_CHUNK) {
        const uint32_t n = min(M - c0, (uint32_t)MAC_CHUNK), n4 = (n + MAC_U - 1) / MAC_U * MAC_U;
        __syncthreads();
        for (uint32_t i = threadIdx.x; i < n4 * (G + 1); i += blockDim.x) {
            const uint32_t b = i / (G + 1), w = i % (G + 1);
            const uint64_t *p = nullptr;
            if (b < n) p = w == 0 ? babies[c0 + b] : (w - 1 < n_g ? pts[(size_t)(w - 1) * M + c0 + b] : nullptr);
            sp[i] = p;
        }
        __syncthreads();
        for (uint32_t b = 0; b < n4; b += MAC_U) {
            uint64_t y0[MAC_U], y1[MAC_U], p[MAC_U][G];
#pragma unroll
            for (int u = 0; u < MAC_U; u++) {
                const uint64_t *bb = sp[(b + u) * (G + 1)];
                y0[u] = bb ? bb[idx] : 0;
                y1[u] = bb ? bb[S_words + idx] : 0;
#pragma unroll
                for (int g = 0; g < G; g++) {
                    const uint64_t *pp = sp[(b + u) * (G + 1) + 1 + g];
                    p[u][g] = pp ? __ldcs(pp + idx) : 0;  // a diagonal is read once
                }
            }
            if (pending + MAC_U > S::FLUSH) {
#pragma unroll
                for (int g = 0; g < G; g++) S::flush(acc[g][0], k), S::flush(acc[g][1], k);
                pending = 0;
            }
            pending += MAC_U;
#pragma unroll
            for (int u = 0; u < MAC_U; u++) {
                const typename S::B v0 = S::ld_b(y0[u], k), v1 = S::ld_b(y1[u], k);
#pragma unroll
                for (int g = 0; g < G; g++) {
                    const typename S::A a = S::ld_a(p[u][g], k);
                    S::mac(acc[g][0], a, v0, k);
                    S::mac(acc[g][1], a, v1, k);
                }
            }
        }
    }
#pragma unroll
    for (int g = 0; g < G; g++) {
        if (g < (int)n_g) {
            uint64_t *o = outs ? outs[g] : out;
            o[idx] = S::finish(acc[g][0], k);
            o[S_words + idx] = S::finish(acc[g][1], k);
        }
    }
}

template <int G>
__global__ void __launch_bounds__(256, 2) bsgs_mac_kernel(const uint64_t *const *pts, const uint64_t *const *babies, uint64_t *const *outs, uint64_t *out,
                                                          const Mod *mod, uint32_t N, uint32_t l, uint32_t M, uint32_t n_g) {
    pdl_enter();
    __shared__ const uint64_t *sp[MAC_CHUNK * (G + 1)];
    const Mod md = mod[blockIdx.y];
    const size_t idx = (size_t)blockIdx.y * N + blockIdx.x * 256 + threadIdx.x;
    with_sum(md.q, [&](auto s) { bsgs_mac_body<decltype(s), G>(pts, babies, outs, out, sp, md, (size_t)l * N, idx, M, n_g); });
}

// ---- weighted sum: out = sum_t x_t * s_t (+ c on polynomial 0 of every ciphertext of `per` polynomials) with per-limb integer weights,
// one reduction per value. The terms may sit at higher levels than the output (more limbs per polynomial): lt[t] is term t's limb count.
#define B2_LINCOMB_MAX_TERMS 8
#define B2_LINCOMB_MAX_LIMBS 32
struct LincombArgs {
    const uint64_t *x[B2_LINCOMB_MAX_TERMS];
    uint32_t lt[B2_LINCOMB_MAX_TERMS];
    uint64_t s[B2_LINCOMB_MAX_TERMS][B2_LINCOMB_MAX_LIMBS];
    uint64_t c[B2_LINCOMB_MAX_LIMBS];
};
template <class S>
__device__ __forceinline__ void lincomb_body(const LincombArgs &a, uint64_t *out, const Mod &md, uint32_t N, uint32_t l, uint32_t n_terms, uint32_t per) {
    const typename S::K k = S::make(md);
    const uint32_t limb = blockIdx.y % l, p = blockIdx.y / l, i = blockIdx.x * 256 + threadIdx.x;
    typename S::Acc acc;
    S::zero(acc);
    uint64_t v[B2_LINCOMB_MAX_TERMS];
#pragma unroll
    for (int t = 0; t < B2_LINCOMB_MAX_TERMS; t++) v[t] = t < (int)n_terms ? a.x[t][((size_t)p * a.lt[t] + limb) * N + i] : 0;
#pragma unroll
    for (int t = 0; t < B2_LINCOMB_MAX_TERMS; t++) {
        if (t == S::FLUSH) S::flush(acc, k);
        if (t < (int)n_terms) S::mac(acc, S::ld_a(a.s[t][limb], k), S::ld_b(v[t], k), k);
    }
    const uint64_t r = S::finish(acc, k);
    out[(size_t)blockIdx.y * N + i] = p % per == 0 ? add_mod(r, a.c[limb], md.q) : r;
}
__global__ void __launch_bounds__(256) lincomb_kernel(const __grid_constant__ LincombArgs a, uint64_t *out, const Mod *mod, uint32_t N, uint32_t l,
                                                     uint32_t n_terms, uint32_t per) {
    pdl_enter();
    const Mod md = mod[blockIdx.y % l];
    with_sum(md.q, [&](auto s) { lincomb_body<decltype(s)>(a, out, md, N, l, n_terms, per); });
}

// ---- vector access: V = 4 words with 256-bit loads where every buffer is 32-byte aligned, else one word -------------------
template <int V>
__device__ __forceinline__ void ldv(uint64_t (&x)[V], const uint64_t *p) {
    if constexpr (V == 4) {
        const u64x4 v = ld256(p);
        x[0] = v.a, x[1] = v.b, x[2] = v.c, x[3] = v.d;
    } else {
        x[0] = *p;
    }
}
template <int V>
__device__ __forceinline__ void stv(uint64_t *p, const uint64_t (&x)[V]) {
    if constexpr (V == 4) st256(p, x[0], x[1], x[2], x[3]);
    else *p = x[0];
}

// (a0, a1) x (b0, b1): a0 <- a0 b0, b0 <- a0 b1 + a1 b0, a1 <- a1 b1
template <int V>
__device__ __forceinline__ void tensor_values(uint64_t (&a0)[V], uint64_t (&a1)[V], uint64_t (&b0)[V], const uint64_t (&b1)[V], const Mod &md) {
    const uint64_t q = md.q;
    if (q < FP_LIMIT) {
        using F = ArithFp<true>;
        const F::K k = F::make(md, 0);
#pragma unroll
        for (int i = 0; i < V; i++) {
            const double x0 = F::from_u64(a0[i], k), x1 = F::from_u64(a1[i], k), y0 = F::from_u64(b0[i], k), y1 = F::from_u64(b1[i], k);
            const F::Tw w0{y0, __dmul_rn(y0, k.qinv)}, w1{y1, __dmul_rn(y1, k.qinv)};
            a0[i] = F::to_canon(F::mulmod(x0, w0, k), k);
            b0[i] = F::canon_fwd(__dadd_rn(F::mulmod(x0, w1, k), F::mulmod(x1, w0, k)), k);
            a1[i] = F::to_canon(F::mulmod(x1, w1, k), k);
        }
    } else {
#pragma unroll
        for (int i = 0; i < V; i++) {
            const uint64_t d0 = mul_mod(a0[i], b0[i], md), d2 = mul_mod(a1[i], b1[i], md);
            const uint64_t m = mul_mod(add_mod(a0[i], a1[i], q), add_mod(b0[i], b1[i], q), md);
            a0[i] = d0, b0[i] = sub_mod(sub_mod(m, d0, q), d2, q), a1[i] = d2;
        }
    }
}

// HMult tensor product (src/polymath.cu:463-498): d0 = a0 b0, d1 = a0 b1 + a1 b0, d2 = a1 b1. d0, d1 go to out[0..2S), d2 to
// out2[0..S): the relinearising caller keeps d2 in scratch and the rest in its result. blockIdx.z = pair of a batch, whose
// operands, result and d2 start z * bs.x / .y / .z / .w limbs further. Streams seven limbs; FP64 products below 2^50
// (24 limbs at N = 2^16: 27.1 us with 128-bit integer products on one word per thread).
template <int V>
__global__ void __launch_bounds__(256) tensor_mul_kernel(const uint64_t *a, const uint64_t *b, uint64_t *out, uint64_t *out2, const Mod *mod, uint32_t N,
                                                        uint32_t l, uint4 bs) {
    pdl_enter();
    const size_t o = (size_t)blockIdx.y * N + (blockIdx.x * 256 + threadIdx.x) * V, S = (size_t)l * N;
    a += (size_t)blockIdx.z * bs.x * N + o, b += (size_t)blockIdx.z * bs.y * N + o, out += (size_t)blockIdx.z * bs.z * N + o,
        out2 += (size_t)blockIdx.z * bs.w * N + o;
    const Mod md = mod[blockIdx.y];
    uint64_t a0[V], a1[V], b0[V], b1[V];
    ldv<V>(a0, a), ldv<V>(a1, a + S), ldv<V>(b0, b), ldv<V>(b1, b + S);
    tensor_values<V>(a0, a1, b0, b1, md);
    stv<V>(out, a0), stv<V>(out + S, b0), stv<V>(out2, a1);
}

// The same for products whose operands lie apart and may sit at higher levels (more limbs per polynomial): blockIdx.z =
// product p * sets + set, operand p at a[p] + set * 2 la[p] limbs. dbl: the doubled product.
constexpr int TENSOR_MANY_MAX = 16;
struct TensorMany {
    const uint64_t *a[TENSOR_MANY_MAX], *b[TENSOR_MANY_MAX];
    uint32_t la[TENSOR_MANY_MAX], lb[TENSOR_MANY_MAX];
    uint32_t sets, dbl;
    uint32_t out_bs, d2;  // a product's results lie out_bs limbs apart, its third polynomial d2 limbs behind the first
};
__global__ void __launch_bounds__(256) tensor_many_kernel(const __grid_constant__ TensorMany t, uint64_t *out, const Mod *mod, uint32_t N, uint32_t l) {
    pdl_enter();
    constexpr int V = 4;
    const uint32_t p = blockIdx.z / t.sets, set = blockIdx.z % t.sets;
    const size_t o = (size_t)blockIdx.y * N + (blockIdx.x * 256 + threadIdx.x) * V, S = (size_t)l * N;
    const uint64_t *a = t.a[p] + (size_t)set * 2 * t.la[p] * N + o, *b = t.b[p] + (size_t)set * 2 * t.lb[p] * N + o;
    const Mod md = mod[blockIdx.y];
    uint64_t d0[V], d1[V], d2[V], b1[V];
    ldv<V>(d0, a), ldv<V>(d2, a + (size_t)t.la[p] * N), ldv<V>(d1, b), ldv<V>(b1, b + (size_t)t.lb[p] * N);
    tensor_values<V>(d0, d2, d1, b1, md);
    if (t.dbl) {
#pragma unroll
        for (int i = 0; i < V; i++) d0[i] = add_mod(d0[i], d0[i], md.q), d1[i] = add_mod(d1[i], d1[i], md.q), d2[i] = add_mod(d2[i], d2[i], md.q);
    }
    out += (size_t)blockIdx.z * t.out_bs * N + o;
    stv<V>(out, d0), stv<V>(out + S, d1), stv<V>(out + (size_t)t.d2 * N, d2);
}

// The dropped limb of a rescale after ModDown, in coefficient form: r -= sum_i P_i M_i mod q over the alpha P limbs (M: the last
// prime's row of the ModDown matrix). blockIdx.y = polynomial, blockIdx.z = set, bs limbs apart.
__global__ void __launch_bounds__(256) rescale_remainder_kernel(const uint64_t *P, uint64_t *r, const W2 *m, const Mod *mod, uint32_t N, uint32_t alpha, uint32_t bs) {
    pdl_enter();
    constexpr int V = 4;
    const Mod md = *mod;
    const bool tight = md.q >= INT_LAZY_LIMIT;  // eight terms below 2 q could pass 2^64
    const size_t o = (size_t)blockIdx.z * bs * N + (blockIdx.x * 256 + threadIdx.x) * V;
    P += o + (size_t)blockIdx.y * alpha * N, r += o + (size_t)blockIdx.y * N;
    uint64_t x[V], s[V] = {0, 0, 0, 0};
    ldv<V>(x, r);
    for (uint32_t i = 0; i < alpha; i++) {
        const W2 w = ldg_w2(m + i);
        uint64_t y[V];
        ldv<V>(y, P + (size_t)i * N);
#pragma unroll
        for (int j = 0; j < V; j++) {
            s[j] += mul_shoup_lazy(y[j], w, md.q);
            if (tight) s[j] = csub(s[j], 2 * md.q);
        }
    }
#pragma unroll
    for (int j = 0; j < V; j++) x[j] = sub_mod(x[j], barrett64(s[j], md.q, md.r1), md.q);
    stv<V>(r, x);
}

// x y mod q for V pairs, FP64 below 2^50
template <int V>
__device__ __forceinline__ void mul_limb(uint64_t (&x)[V], const uint64_t (&y)[V], const Mod &md) {
    if (md.q < FP_LIMIT) {
        using F = ArithFp<true>;
        const F::K k = F::make(md, 0);
#pragma unroll
        for (int i = 0; i < V; i++) {
            const double w = F::from_u64(y[i], k);
            x[i] = F::to_canon(F::mulmod(F::from_u64(x[i], k), F::Tw{w, __dmul_rn(w, k.qinv)}, k), k);
        }
    } else {
#pragma unroll
        for (int i = 0; i < V; i++) x[i] = mul_mod(x[i], y[i], md);
    }
}

// src/polymath.cu:17-180. `period` limbs per polynomial: limb t of the buffer uses prime t % period, so one launch covers a
// whole ciphertext. b_wrap: the second operand is one polynomial shared by all (a plaintext).
template <int V>
__global__ void __launch_bounds__(256) poly_op_kernel(int op, const uint64_t *a, const uint64_t *b, uint64_t *out, const Mod *mod, uint32_t N, uint32_t period,
                                                     int b_wrap) {
    pdl_enter();
    const uint32_t limb = blockIdx.y % period, i = (blockIdx.x * 256 + threadIdx.x) * V;
    const size_t o = (size_t)blockIdx.y * N + i;
    const Mod md = mod[limb];
    uint64_t x[V], y[V];
    ldv<V>(x, a + o);
    if (op != 3) ldv<V>(y, b + (b_wrap ? (size_t)limb * N + i : o));
    if (op == 2) {
        mul_limb<V>(x, y, md);
    } else {
#pragma unroll
        for (int j = 0; j < V; j++) x[j] = op == 0 ? add_mod(x[j], y[j], md.q) : op == 1 ? sub_mod(x[j], y[j], md.q) : (x[j] ? md.q - x[j] : 0);
    }
    stv<V>(out + o, x);
}

// Per-limb integer constants (src/bootstrap.cu:1535-1565, multiply_scalar_per_tower_kernel; adding a constant polynomial c to
// NTT-form data adds c to every value of the limb).
struct ScalarTab {
    uint64_t v[64];
};
template <int V>
__global__ void __launch_bounds__(256) poly_scalar_kernel(int op, const uint64_t *a, const __grid_constant__ ScalarTab tab, uint64_t *out, const Mod *mod,
                                                         uint32_t N, uint32_t period) {
    pdl_enter();
    const uint32_t limb = blockIdx.y % period;
    const size_t o = (size_t)blockIdx.y * N + (blockIdx.x * 256 + threadIdx.x) * V;
    const Mod md = mod[limb];
    uint64_t x[V], y[V];
    ldv<V>(x, a + o);
#pragma unroll
    for (int j = 0; j < V; j++) y[j] = tab.v[limb];
    if (op == 0) {
#pragma unroll
        for (int j = 0; j < V; j++) x[j] = add_mod(x[j], y[j], md.q);
    } else {
        mul_limb<V>(x, y, md);
    }
    stv<V>(out + o, x);
}

// symmetric encryption (src/secretkey.cu:236-299): out0 holds the error e, out1 the mask a; out0 <- m - (a s + e)
// (m null: an encryption of zero). encrypt = 0, decryption (src/secretkey.cu:883-919): out0 <- m + a s
template <int V>
__global__ void __launch_bounds__(256) mask_kernel(const uint64_t *m, const uint64_t *a, const uint64_t *s, uint64_t *out0, const Mod *mod, uint32_t N, int encrypt) {
    pdl_enter();
    const size_t o = (size_t)blockIdx.y * N + (blockIdx.x * 256 + threadIdx.x) * V;
    const Mod md = mod[blockIdx.y];
    uint64_t x[V], y[V], z[V];
    ldv<V>(x, a + o), ldv<V>(y, s + o);
    if (encrypt) {
        ldv<V>(z, out0 + o);
    }
    mul_limb<V>(x, y, md);
    if (m) ldv<V>(y, m + o);
#pragma unroll
    for (int j = 0; j < V; j++) {
        if (encrypt) {
            x[j] = add_mod(x[j], z[j], md.q);
            x[j] = m ? sub_mod(y[j], x[j], md.q) : (x[j] ? md.q - x[j] : 0);
        } else {
            x[j] = add_mod(x[j], y[j], md.q);
        }
    }
    stv<V>(out0 + o, x);
}

// NTT-domain automorphism (src/galois.cu:11-18): dst[l][i] = src[l][perm[i]]. An aligned run of 2^k values comes from an
// aligned run of 2^k values (the low bits of a bit-reversed index are the high bits of the exponent), so the four reads of a
// thread fall into one sector.
template <int V>
__global__ void __launch_bounds__(256) galois_gather_kernel(const uint64_t *__restrict__ src, uint64_t *__restrict__ dst, const uint32_t *__restrict__ perm,
                                                           uint32_t N) {
    pdl_enter();
    const uint32_t i = (blockIdx.x * 256 + threadIdx.x) * V;
    const uint64_t *s = src + (size_t)blockIdx.y * N;
    uint64_t x[V];
    if constexpr (V == 4) {
        const uint4 p = *reinterpret_cast<const uint4 *>(perm + i);
        x[0] = s[p.x], x[1] = s[p.y], x[2] = s[p.z], x[3] = s[p.w];
    } else {
        x[0] = s[perm[i]];
    }
    stv<V>(dst + (size_t)blockIdx.y * N + i, x);
}

// the same for several polynomials, each through a permutation of its own: blockIdx.z = polynomial, src_bs limbs apart
constexpr int GATHER_TAB_MAX = 16;
struct GatherTab {
    const uint32_t *perm[GATHER_TAB_MAX];
};
__global__ void __launch_bounds__(256) galois_gather_tab_kernel(const uint64_t *__restrict__ src, uint64_t *__restrict__ dst, const __grid_constant__ GatherTab tab,
                                                               uint32_t N, uint32_t src_bs) {
    pdl_enter();
    const uint32_t i = (blockIdx.x * 256 + threadIdx.x) * 4;
    const uint64_t *s = src + ((size_t)blockIdx.z * src_bs + blockIdx.y) * N;
    const uint4 p = *reinterpret_cast<const uint4 *>(tab.perm[blockIdx.z] + i);
    st256(dst + ((size_t)blockIdx.z * gridDim.y + blockIdx.y) * N + i, s[p.x], s[p.y], s[p.z], s[p.w]);
}

// Signed coefficient vectors -> their residues in each of l primes from first_prime on (src/bootstrap.cu:660-686,
// light_pt_expand_per_tower_kernel): src [M][N] -> dst [M][l][N], blockIdx.z = vector
template <int V>
__global__ void __launch_bounds__(256) expand_signed_kernel(const int64_t *__restrict__ src, uint64_t *__restrict__ dst, const Mod *mod, uint32_t N, uint32_t l,
                                                           uint32_t first_prime) {
    pdl_enter();
    const uint32_t i = (blockIdx.x * 256 + threadIdx.x) * V;
    const Mod md = mod[first_prime + blockIdx.y];
    uint64_t x[V];
    ldv<V>(x, reinterpret_cast<const uint64_t *>(src) + (size_t)blockIdx.z * N + i);
#pragma unroll
    for (int j = 0; j < V; j++) {
        const int64_t c = (int64_t)x[j];
        const uint64_t r = barrett64(c >= 0 ? (uint64_t)c : (uint64_t)0 - (uint64_t)c, md.q, md.r1);
        x[j] = (c >= 0 || r == 0) ? r : md.q - r;
    }
    stv<V>(dst + ((size_t)blockIdx.z * l + blockIdx.y) * N + i, x);
}

// M separate vectors that the device can read where they are (pinned host memory) -> one array. One CTA with as many loads in
// flight as the link needs, 112 KB: reads over the link beyond that only queue, and everything else that the GPU loads queues
// behind them. 8 MB take 167 us (50 GB/s) with 96 KB to 400 KB in flight on 2 to 96 CTAs, but a transform of 384 limbs of 2^14
// beside them 35 + 42 us with 96 KB, 60 + 65 with 400 KB, 120 + 125 with 800 KB; alone 26 + 32. (256 copies of 128 KB took 6.4
// us each, a quarter of the link's rate, plus a host call each.)
constexpr int GATHER_MAX = 128, GATHER_U = 7, GATHER_CTAS = 1, GATHER_THREADS = 1024;
struct GatherPtrs {
    const ulonglong2 *p[GATHER_MAX];
};
__global__ void __launch_bounds__(GATHER_THREADS) gather_vectors_kernel(const __grid_constant__ GatherPtrs src, ulonglong2 *__restrict__ dst, uint32_t logN,
                                                                       uint32_t M) {
    pdl_enter();
    const uint32_t log_per = logN - 1, total = M << log_per, mask = (1u << log_per) - 1;  // pairs; at least 2048 in a vector
    for (uint32_t i = blockIdx.x * (GATHER_THREADS * GATHER_U) + threadIdx.x; i < total; i += gridDim.x * (GATHER_THREADS * GATHER_U)) {
        ulonglong2 x[GATHER_U];
#pragma unroll
        for (int u = 0; u < GATHER_U; u++) {
            const uint32_t k = i + u * GATHER_THREADS;
            if (k < total) x[u] = __ldcs(src.p[k >> log_per] + (k & mask));
        }
#pragma unroll
        for (int u = 0; u < GATHER_U; u++) {
            const uint32_t k = i + u * GATHER_THREADS;
            if (k < total) dst[k] = x[u];
        }
    }
}

// ---- key-switch inner product (src/eval_key_switch.cu:175-230) ---------------------------------------------------------------
// For logical limb t (physical prime pp):  acc[k][t][n] = sum_d digits[d][t][n] * evk[d][k][pp][n],  k = 0, 1.
// Pure streaming: two coefficients per thread, 16-byte loads, two digits at a time so that 32 warps fit an SM (three digits and
// 24: eight hoisted rotations at N = 2^15 the same, 32 products at 2^14 724 against 707 us), the loads of the key before
// those that wait for a permutation. CTAs of 128 threads: with 256 the warps of an SM load and multiply more
// in step (247.7 -> 245.3 us, 689 -> 684.6 us, a bootstrap 25.48 -> 25.37 ms).
constexpr int IP_MAX_STEPS = 16, IP_MAX_EVK = 256;
struct IpArgs {
    const uint64_t *digits;
    // `own` (optional): the NTT-form input of ModUp; limb t of digit t / alpha is that input itself (src/rns_bconv.cu:522-528),
    // so the digit buffer need not hold a copy of it
    const uint64_t *own;
    uint64_t *out;  // fused: the P limbs, else [2][l + alpha][N]
    uint64_t *ct;   // fused: acc * P^-1 goes straight into the Q limbs of the ciphertext [2][l][N]
    const uint64_t *c0;  // fused, optional: the first polynomial of a ciphertext being rotated, read through perm and added
    const W2 *pinv;
    const Mod *mod;
    uint32_t logN, l, lP, size_Q, size_QP, beta;
    uint32_t q0, nq, p0, np;  // the Q limbs and P limbs this launch covers (a rank's slice under limb sharding)
    uint32_t fused, ct_acc, acc_p;  // ct_acc / acc_p: add to what ct / the P limbs hold (else overwrite)
    // blockIdx.z = set of a batch with one key: its digits, own, ct start z * dig_bs / own_bs / ct_bs limbs further, and P limb
    // i of polynomial k lands at slot (i * p_mul_i + k * p_mul_k) * (p_lm1 + 1) + z * p_bs of the P-limb buffer
    uint32_t dig_bs, own_bs, ct_bs, p_mul_i, p_mul_k, p_lm1, p_bs;
    uint32_t c0_bs;  // a batch of rotations: c0 of set z starts z * c0_bs limbs further
    // hoisted rotations: steps > 0. Step s reads digits and own through perm[s] and has the key evk[s * beta ..]. each = 1: one
    // set per step, written to ct_tab[z] (P limbs as above); each = 0: the steps are summed.
    // A rotation whose c1 was permuted before ModUp: steps = 0 and perm[0] set; own and c0 are read through it, digits are not.
    uint32_t steps, each;
    // steps that are summed and have ciphertexts of their own, c1 permuted before ModUp: step s reads digits and own s * dig_ss /
    // own_ss limbs further, as they are, and c0 s * c0_ss limbs further through perm[s]
    uint32_t apart, dig_ss, own_ss, c0_ss;
    const uint32_t *perm[IP_MAX_STEPS];
    uint64_t *ct_tab[IP_MAX_STEPS];
    const uint64_t *evk[IP_MAX_EVK];
};

// the pair of values at positions n, n + 1 (n even) behind the permutation: an aligned pair, in either order
__device__ __forceinline__ ulonglong2 ld_pair(const uint64_t *p, uint32_t n, uint32_t pn, bool permuted) {
    const ulonglong2 v = *reinterpret_cast<const ulonglong2 *>(p + (permuted ? (pn & ~1u) : n));
    return permuted && (pn & 1u) ? make_ulonglong2(v.y, v.x) : v;
}

// FEW: four terms at most in a sum, one step
template <class S, bool FEW>
__device__ __forceinline__ void ip_body(const IpArgs &a, uint32_t t, uint32_t n, uint32_t pp, const Mod &md) {
    constexpr int U = 2;
    const size_t N = (size_t)1 << a.logN;
    const uint32_t z = blockIdx.z, lim = a.size_QP;
    const typename S::K k = S::make(md);
    typename S::Acc acc[2][2];
#pragma unroll
    for (int i = 0; i < 2; i++) S::zero(acc[i][0]), S::zero(acc[i][1]);
    const uint64_t *digits = a.digits + ((size_t)z * a.dig_bs + t) * N, *own = a.own ? a.own + ((size_t)z * a.own_bs + t) * N : nullptr;
    const uint32_t own_d = (own && t < a.l) ? t / (a.lP - a.l) : 0xFFFFFFFFu;
    const uint32_t s0 = a.each ? z : 0, n_s = !FEW && a.steps && !a.each ? a.steps : 1;
    const bool hoist = a.steps != 0 && !a.apart;
    uint64_t g0 = 0, g1 = 0;  // permuted c0
    int pending = 0;
    for (uint32_t s = s0; s < s0 + n_s; s++, digits += (size_t)a.dig_ss * N, own += (size_t)a.own_ss * N) {
        const bool pm = a.perm[s] != nullptr;
        const uint32_t pn = pm ? a.perm[s][n] : 0;
        for (uint32_t d0 = 0; d0 < a.beta; d0 += U) {
            // the key's loads go first: they do not wait for the permutation
            ulonglong2 x[U], e0[U], e1[U];
#pragma unroll
            for (int i = 0; i < U; i++) {
                e0[i] = e1[i] = make_ulonglong2(0, 0);
                if (d0 + i < a.beta) {
                    const uint64_t *e = a.evk[s * a.beta + d0 + i] + (size_t)pp * N + n;
                    e0[i] = __ldcs(reinterpret_cast<const ulonglong2 *>(e));
                    e1[i] = __ldcs(reinterpret_cast<const ulonglong2 *>(e + (size_t)lim * N));
                }
            }
#pragma unroll
            for (int i = 0; i < U; i++) {
                x[i] = make_ulonglong2(0, 0);
                if (d0 + i < a.beta)
                    x[i] = d0 + i == own_d ? ld_pair(own, n, pn, pm && !a.apart) : ld_pair(digits + (size_t)(d0 + i) * a.lP * N, n, pn, hoist);
            }
            if (d0 == 0 && a.c0 && t < a.l) {
                const ulonglong2 c = ld_pair(a.c0 + ((size_t)z * a.c0_bs + (size_t)s * a.c0_ss + t) * N, n, pn, pm);
                g0 = add_mod(g0, c.x, md.q), g1 = add_mod(g1, c.y, md.q);
            }
            if (!FEW && pending + U > S::FLUSH) {
#pragma unroll
                for (int i = 0; i < 2; i++) S::flush(acc[i][0], k), S::flush(acc[i][1], k);
                pending = 0;
            }
            pending += U;
#pragma unroll
            for (int i = 0; i < U; i++) {
                if (d0 + i < a.beta) {
                    const typename S::A x0 = S::ld_a(x[i].x, k), x1 = S::ld_a(x[i].y, k);
                    S::mac(acc[0][0], x0, S::ld_b(e0[i].x, k), k);
                    S::mac(acc[0][1], x1, S::ld_b(e0[i].y, k), k);
                    S::mac(acc[1][0], x0, S::ld_b(e1[i].x, k), k);
                    S::mac(acc[1][1], x1, S::ld_b(e1[i].y, k), k);
                }
            }
        }
    }
    uint64_t r[4];
    uint64_t *o0, *o1;
    bool add;
    if (a.fused && t < a.l) {
        // together with a ModDown matrix that carries P^-1, ct + acc * P^-1 - delta equals ct + (acc - delta') * P^-1
        const W2 pi = a.pinv[pp];
#pragma unroll
        for (int i = 0; i < 4; i++) r[i] = S::finish_mul(acc[i >> 1][i & 1], pi, k);
        if (a.c0) r[0] = add_mod(r[0], g0, md.q), r[1] = add_mod(r[1], g1, md.q);
        o0 = (a.each ? a.ct_tab[z] : a.ct + (size_t)z * a.ct_bs * N) + (size_t)t * N + n;
        o1 = o0 + (size_t)a.l * N;
        add = a.ct_acc;
    } else {
#pragma unroll
        for (int i = 0; i < 4; i++) r[i] = S::finish(acc[i >> 1][i & 1], k);
        if (a.fused) {
            o0 = a.out + ((size_t)(t - a.l) * a.p_mul_i * (a.p_lm1 + 1) + (size_t)z * a.p_bs) * N + n;
            o1 = o0 + (size_t)a.p_mul_k * (a.p_lm1 + 1) * N;
            add = a.acc_p;
        } else {
            o0 = a.out + (size_t)t * N + n, o1 = o0 + (size_t)a.lP * N;
            add = false;
        }
    }
    if (add) {
        const ulonglong2 u0 = *reinterpret_cast<const ulonglong2 *>(o0), u1 = *reinterpret_cast<const ulonglong2 *>(o1);
        r[0] = add_mod(r[0], u0.x, md.q), r[1] = add_mod(r[1], u0.y, md.q), r[2] = add_mod(r[2], u1.x, md.q), r[3] = add_mod(r[3], u1.y, md.q);
    }
    *reinterpret_cast<ulonglong2 *>(o0) = make_ulonglong2(r[0], r[1]);
    *reinterpret_cast<ulonglong2 *>(o1) = make_ulonglong2(r[2], r[3]);
}

// FEW (a digit per term, at most four, single rotations): FP64 products and one reduction cost less than pieces and their
// recombination - 78 FP64 instructions a coefficient against 102 and 85 of the integer pipe at three digits. Kernels of their own:
// in one, 132 bytes of spills at the 64 registers of eight CTAs an SM; apart 8 (few) and 92 (eight hoisted rotations at 2^15 209.0 ->
// 204.0 us, a bootstrap at 2^16 22.81 -> 22.57 ms).
template <bool FEW>
__global__ void __launch_bounds__(128, 8) ks_inner_prod_kernel(const __grid_constant__ IpArgs a) {
    pdl_enter();
    // the limbs of the special primes (the longer arithmetic) first
    const uint32_t y = blockIdx.y, t = y < a.np ? a.l + a.p0 + y : a.q0 + (y - a.np);
    const uint32_t pp = t < a.l ? t : a.size_Q + (t - a.l);
    const uint32_t n = 2 * (blockIdx.x * 128 + threadIdx.x);
    const Mod md = a.mod[pp];
    if constexpr (FEW) {
        if (md.q < FP_LIMIT) ip_body<SumFp, true>(a, t, n, pp, md);
        else if (md.q < INT_LAZY_LIMIT) ip_body<SumInt30Short, true>(a, t, n, pp, md);
        else ip_body<SumInt, true>(a, t, n, pp, md);
    } else {
        with_sum(md.q, [&](auto s) { ip_body<decltype(s), false>(a, t, n, pp, md); });
    }
}

}  // namespace b2
