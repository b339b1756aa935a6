// ntt_whole.cuh - whole transforms of one limb in one launch for the rings 2^12 .. 2^14, at 2^12 with the base conversion of a
// key switch (or the reduction of a rescale) made while loading.
//
// A limb belongs to a thread-block cluster of four CTAs (eight at N = 2^14), 1024 or 2048 residues each. Forward: every CTA
// runs the column pass on its N2 / CL columns, leaves the result in its shared memory, the cluster meets at the hardware
// barrier, and every CTA gathers its N1 / CL rows from the slabs of the cluster (distributed shared memory) for the row pass;
// inverse: the mirror image. What this removes is one launch, one trip through global memory and - with the conversion
// fused - a second launch and trip: a key switch at 2^12 is five launches instead of eleven.
//
// When it pays (B200, us on the device, the launches queued behind a busy stream so that the host does not count; two passes ->
// whole):
//   2^12, plain transforms and rescales, up to 192 limbs a launch: a 60-bit prime among eight, 8 limbs 5.1 -> 5.0, 96 6.7 -> 6.4,
//     192 8.4 -> 8.1, 256 10.8 -> 11.3, 1024 28.8 -> 30.9; FP64 primes 192 7.9 -> 7.6, 256 9.2 -> 9.9, 1024 25.1 -> 28.0; 60-bit
//     primes 192 12.3 -> 11.9, 256 15.2 -> 15.1, 512 24.9 -> 25.2. Above, every SM has CTAs enough for either form, and the whole
//     one's rendezvous and its reads of the neighbours' slabs show.
//   2^12, conversions: every output limb reads its alpha inputs again and multiplies in FP64 or 64-bit integers, where the tensor
//     cores convert all outputs from one read: the larger alpha, the earlier that weighs more than the saved launch and
//     trip. Whole relinearisations: alpha 1, 25 limbs 35.5 -> 28.4, 3200 411 -> 316; alpha 2, 32 35.0 -> 28.6, 4096 507 -> 466;
//     alpha 3, 3456 502 -> 493; alpha 4, 512 79.0 -> 77.0, 1024 134.6 -> 135.9; alpha 5, 360 73.3 -> 72.0, 540 93.1 -> 95.5;
//     alpha 6, 96 38.5 -> 35.3, 192 43.8 -> 44.5; alpha 7, 84 42.1 -> 40.3, 112 45.0 -> 46.9; alpha 8, 72 37.1 -> 35.6, 144
//     42.4 -> 44.8, 576 91.5 -> 111.3.
//   2^13 and 2^14, plain transforms on FP64 primes, up to 32 limbs. What they save is the host's second launch, which a program
//     that issues transforms one by one waits for (forward, 8 limbs: 2^13 9.9 -> 7.6, 2^14 9.8 -> 7.4, whatever the limbs).
//     On the device alone: 2^14, 8 limbs 6.4 -> 5.9, 16 5.9 -> 6.7, 32 7.7 -> 7.3, 60 11.4 -> 10.9; 2^13, 8 limbs 5.3 -> 5.8, 32
//     5.7 -> 6.1, 60 7.2 -> 7.3 (a thread's stages run alone on its scheduler, and two launches spread them over twice the SMs).
//     With a 60-bit prime among the limbs 2^13 takes 7.1 -> 8.1 on the device, 9.8 -> 8.1 with the host; 2^14 9.2 -> 8.2 and
//     9.9 -> 8.3: there the line could go. Key switches (job lists) lose at 2^13 (a rotation 44 -> 48 us).
// At 2^15 a limb would want sixteen CTAs; with eight everything loses. The loops over a thread's register groups are not
// unrolled: the code a lone CTA streams through is fetched once per launch (unrolled, the rotation took 57 us).
//
// No flag and no spin: cluster.sync() is the only rendezvous, and every thread of every CTA reaches it.
#pragma once
#include <cooperative_groups.h>

#include "ntt_kernels.cuh"

namespace b2 {
namespace cg = cooperative_groups;

template <int LOGN> struct WholeCfg;
//                                          column pass            row pass              log2 of CTAs per limb, threads
template <> struct WholeCfg<12> { static constexpr int LOG_A = 6, RA1 = 3, RA2 = 3, LOG_B = 6, RB1 = 3, RB2 = 3, LOG_CL = 2, THREADS = 128; };
template <> struct WholeCfg<13> { static constexpr int LOG_A = 6, RA1 = 3, RA2 = 3, LOG_B = 7, RB1 = 3, RB2 = 4, LOG_CL = 2, THREADS = 128; };
template <> struct WholeCfg<14> { static constexpr int LOG_A = 7, RA1 = 3, RA2 = 4, LOG_B = 7, RB1 = 3, RB2 = 4, LOG_CL = 3, THREADS = 128; };
template <int LOGN>
__host__ __device__ constexpr int whole_slab() { return 1 << (LOGN - WholeCfg<LOGN>::LOG_CL); }  // residues per CTA
// the slab, and an exchange buffer of as many residues padded by one word per 2^R
template <int LOGN>
constexpr size_t whole_smem() {
    using C = WholeCfg<LOGN>;
    constexpr int ra = C::RA1 < C::RA2 ? C::RA1 : C::RA2, rb = C::RB1 < C::RB2 ? C::RB1 : C::RB2;
    return 8 * (size_t)(2 * whole_slab<LOGN>() + (whole_slab<LOGN>() >> (ra < rb ? ra : rb)));
}

// R1 strided stages, exchange, R2 contiguous stages on 2^LOG_C sub-transforms of 2^LOG_T points (see fwd_body). ld(c, e) gives
// element e of sub-transform c, st(c, e0, x) takes the E2 elements from e0 on; P0: twiddle row of sub-transform 0 (rows), 1 (columns).
template <class A, int LOG_T, int R1, int R2, int LOG_C, bool COLS, int THREADS, int B0, class Ld, class St>
__device__ __forceinline__ void whole_fwd_tile(uint64_t *sm, const W2 *tw, uint32_t P0, const typename A::K &k, Ld &&ld, St &&st) {
    using T = typename A::T;
    constexpr int TT = 1 << LOG_T, E1 = 1 << R1, E2 = 1 << R2, C = 1 << LOG_C, EPT = C * TT / THREADS, TPAD = TT + (TT >> R2);
    constexpr int B1 = ct_bound<A>(B0, R1);
    static_assert(EPT >= E1 && EPT >= E2, "a thread holds a whole stage group");
    static_assert(ct_bound<A>(B1, R2) <= A::B_PASS, "residues stay within the policy's bounds");
#pragma unroll 1
    for (int gi = 0; gi < EPT / E1; gi++) {
        const int gid = threadIdx.x + gi * THREADS;
        const int c = COLS ? gid % C : gid / E2, elo = COLS ? gid / C : gid % E2;
        T x[E1];
        ld(c, elo, E2, x);
        ct_stages<A, 0, R1, E1, B0>(x, tw, COLS ? 1u : P0 + c, 0, 0, k);
#pragma unroll
        for (int i = 0; i < E1; i++) {
            const int pe = pad_idx<LOG_T, R2>(elo + i * E2);
            sm[COLS ? pe * C + c : c * TPAD + pe] = A::to_raw(x[i]);
        }
    }
    __syncthreads();
#pragma unroll 1
    for (int gi = 0; gi < EPT / E2; gi++) {
        const int gid = threadIdx.x + gi * THREADS;
        const int c = COLS ? gid % C : gid / E1, ehi = COLS ? gid / C : gid % E1;
        T x[E2];
#pragma unroll
        for (int i = 0; i < E2; i++) {
            const int pe = pad_idx<LOG_T, R2>(ehi * E2 + i);
            x[i] = A::from_raw(sm[COLS ? pe * C + c : c * TPAD + pe]);
        }
        ct_stages<A, 0, R2, E2, B1>(x, tw, COLS ? 1u : P0 + c, R1, ehi, k);
        st(c, ehi * E2, x);
    }
}

template <class A, int LOGN, class Epi, int SRC>
__device__ __forceinline__ void whole_fwd_body(const NttArgs &a, const Epi &epi, uint64_t *smem, const Job &job, uint32_t jobi, const Mod &md) {
    using Cfg = WholeCfg<LOGN>;
    constexpr int LOG_CC = Cfg::LOG_B - Cfg::LOG_CL, LOG_CR = Cfg::LOG_A - Cfg::LOG_CL;
    constexpr int N2 = 1 << Cfg::LOG_B, CC = 1 << LOG_CC;
    constexpr int B0 = src_bound<A, SRC>();
    constexpr size_t N = (size_t)1 << LOGN;
    uint64_t *slab = smem, *ex = smem + whole_slab<LOGN>();
    const typename A::K k = A::make(md, LOGN);
    const W2 *tw = a.tw + (size_t)job.y * N;
    const uint32_t rank = cg::this_cluster().block_rank();
    BcJob bc{};
    if (SRC & SRC_CONV) bc = a.bc[jobi];
    const uint64_t *src = a.src + src_slot(a, SRC & SRC_CONV ? bc.in_slot0 : job.x) * N, *rem = src_rem<SRC>(a, job, N);
    whole_fwd_tile<A, Cfg::LOG_A, Cfg::RA1, Cfg::RA2, LOG_CC, true, Cfg::THREADS, B0>(
        ex, tw, 1u, k,
        [&](int c, int e, int step, auto &x) {
            load_src<A, SRC>(x, a, bc, src, rem, N, (size_t)e * N2 + rank * CC + c, (size_t)step * N2, md, k);
        },
        [&](int c, int e0, auto &x) {
#pragma unroll
            for (int i = 0; i < (int)(sizeof(x) / 8); i++) slab[(e0 + i) * CC + c] = A::to_raw(x[i]);
        });
    cg::this_cluster().sync();
    const auto e = live_epi(epi, a, job, N);
    const uint32_t row0 = rank << LOG_CR;
    whole_fwd_tile<A, Cfg::LOG_B, Cfg::RB1, Cfg::RB2, LOG_CR, false, Cfg::THREADS, A::B_PASS>(
        ex, tw, (uint32_t)(N >> Cfg::LOG_B) + row0, k,
        [&](int c, int el, int step, auto &x) {
#pragma unroll
            for (int i = 0; i < (int)(sizeof(x) / 8); i++) {
                const int col = el + i * step;
                const uint64_t *peer = cg::this_cluster().map_shared_rank(slab, col >> LOG_CC);
                x[i] = A::from_raw(peer[(row0 + c) * CC + (col & (CC - 1))]);
            }
        },
        [&](int c, int e0, auto &x) {
            constexpr int E = (int)(sizeof(x) / 8);
            const size_t o = (size_t)(row0 + c) * N2 + e0;
            typename std::remove_const_t<decltype(e)>::template Regs<E> regs;
            e.template preload<E>(regs, o, 4);
            uint64_t y[E];
#pragma unroll
            for (int i = 0; i < E; i++) y[i] = A::canon_fwd(x[i], k);
            e.template finish<E>(regs, o, 4, y, md.q);
        });
    cg::this_cluster().sync();  // nobody leaves while a peer may still read its slab
}

template <int LOGN, class Epi, int SRC>
__global__ void __launch_bounds__(WholeCfg<LOGN>::THREADS, 512 / WholeCfg<LOGN>::THREADS) ntt_fwd_whole(NttArgs a, const __grid_constant__ Epi epi) {
    pdl_enter();
    extern __shared__ __align__(16) uint64_t whole_sm[];
    const uint32_t jobi = blockIdx.x >> WholeCfg<LOGN>::LOG_CL;
    const Job job = get_job(a, jobi);
    const Mod md = a.mod[job.y];
    with_arith(md.q, [&](auto A) { whole_fwd_body<decltype(A), LOGN, Epi, SRC>(a, epi, whole_sm, job, jobi, md); });
}

// inverse tile: RA contiguous stages, exchange, RB strided stages; LAST: the transform's final stage with the scaling constants
template <class A, int LOG_T, int RA, int RB, int LOG_C, bool COLS, bool LAST, int THREADS, int B0, class Ld, class St>
__device__ __forceinline__ void whole_inv_tile(uint64_t *sm, const W2 *tw, uint32_t P0, const W2 *fin, const typename A::K &k, Ld &&ld, St &&st) {
    using T = typename A::T;
    constexpr int TT = 1 << LOG_T, EA = 1 << RA, EB = 1 << RB, C = 1 << LOG_C, EPT = C * TT / THREADS, TPAD = TT + (TT >> RA);
    constexpr int B1 = gs_group_bound<A, EA>(B0, RA);
    constexpr GsBounds<EA> end_a = gs_bounds<A, EA>(B0, RA);
    constexpr GsBounds<EB> end_b = gs_bounds<A, EB>(B1, LAST ? RB - 1 : RB);
    static_assert(EPT >= EA && EPT >= EB, "a thread holds a whole stage group");
#pragma unroll 1
    for (int gi = 0; gi < EPT / EA; gi++) {
        const int gid = threadIdx.x + gi * THREADS;
        const int c = COLS ? gid % C : gid / EB, ehi = COLS ? gid / C : gid % EB;
        T x[EA];
        ld(c, ehi * EA, x);
        gs_stages<A, 0, RA, EA, B0>(x, tw, COLS ? 1u : P0 + c, TT >> 1, (size_t)ehi * (EA >> 1), k);
#pragma unroll
        for (int i = 0; i < EA; i++) {
            const int pe = pad_idx<LOG_T, RA>(ehi * EA + i);
            sm[COLS ? pe * C + c : c * TPAD + pe] = A::to_raw(A::group_end(x[i], k, end_a.v[i]));
        }
    }
    __syncthreads();
#pragma unroll 1
    for (int gi = 0; gi < EPT / EB; gi++) {
        const int gid = threadIdx.x + gi * THREADS;
        const int c = COLS ? gid % C : gid / EA, elo = COLS ? gid / C : gid % EA;
        T x[EB];
#pragma unroll
        for (int i = 0; i < EB; i++) {
            const int pe = pad_idx<LOG_T, RA>(elo + i * EA);
            x[i] = A::from_raw(sm[COLS ? pe * C + c : c * TPAD + pe]);
        }
        gs_stages<A, 0, (LAST ? RB - 1 : RB), EB, B1>(x, tw, COLS ? 1u : P0 + c, TT >> (RA + 1), 0, k);
        if (LAST) {
            constexpr int gap = EB / 2;
            const typename A::Tw sx = A::ldfin(fin, k), sy = A::ldfin(fin + 1, k);
#pragma unroll
            for (int j = 0; j < gap; j++) A::gs_last(x[j], x[j + gap], sx, sy, k, end_b.v[j], end_b.v[j + gap]);
        } else {
#pragma unroll
            for (int i = 0; i < EB; i++) x[i] = A::pass_end(x[i], k, end_b.v[i]);
        }
        st(c, elo, EA, x);
    }
}

template <class A, int LOGN>
__device__ __forceinline__ void whole_inv_body(const NttArgs &a, uint64_t *smem, const Job &job, const Mod &md) {
    using Cfg = WholeCfg<LOGN>;
    constexpr int LOG_CC = Cfg::LOG_B - Cfg::LOG_CL, LOG_CR = Cfg::LOG_A - Cfg::LOG_CL;
    constexpr int N2 = 1 << Cfg::LOG_B, CC = 1 << LOG_CC, CR = 1 << LOG_CR;
    constexpr size_t N = (size_t)1 << LOGN;
    uint64_t *slab = smem, *ex = smem + whole_slab<LOGN>();
    const typename A::K k = A::make(md, LOGN);
    const W2 *tw = a.tw + (size_t)job.y * N;
    const uint32_t rank = cg::this_cluster().block_rank(), row0 = rank << LOG_CR;
    const uint64_t *src = a.src + src_slot(a, job.x) * N;
    uint64_t *dst = a.dst + dst_slot(a, job.w) * N;
    whole_inv_tile<A, Cfg::LOG_B, Cfg::RB2, Cfg::RB1, LOG_CR, false, false, Cfg::THREADS, A::B_CANON>(
        ex, tw, (uint32_t)(N >> Cfg::LOG_B) + row0, nullptr, k,
        [&](int c, int e0, auto &x) {
            constexpr int E = (int)(sizeof(x) / 8);
            const size_t o = (size_t)(row0 + c) * N2 + e0;
            if (a.perm) {
#pragma unroll
                for (int i = 0; i < E; i += 4) {
                    const uint4 v = *reinterpret_cast<const uint4 *>(a.perm + o + i);
                    x[i] = A::from_u64(src[v.x], k), x[i + 1] = A::from_u64(src[v.y], k), x[i + 2] = A::from_u64(src[v.z], k), x[i + 3] = A::from_u64(src[v.w], k);
                }
            } else {
#pragma unroll
                for (int i = 0; i < E; i += 4) {
                    const u64x4 v = ld256(src + o + i);
                    x[i] = A::from_u64(v.a, k), x[i + 1] = A::from_u64(v.b, k), x[i + 2] = A::from_u64(v.c, k), x[i + 3] = A::from_u64(v.d, k);
                }
            }
        },
        [&](int c, int e, int step, auto &x) {
#pragma unroll
            for (int i = 0; i < (int)(sizeof(x) / 8); i++) slab[c * N2 + e + i * step] = A::to_raw(x[i]);
        });
    cg::this_cluster().sync();
    whole_inv_tile<A, Cfg::LOG_A, Cfg::RA2, Cfg::RA1, LOG_CC, true, true, Cfg::THREADS, A::GS_PASS>(
        ex, tw, 1u, a.fin + 2 * (size_t)job.z, k,
        [&](int c, int e0, auto &x) {
#pragma unroll
            for (int i = 0; i < (int)(sizeof(x) / 8); i++) {
                const int row = e0 + i;
                const uint64_t *peer = cg::this_cluster().map_shared_rank(slab, row >> LOG_CR);
                x[i] = A::from_raw(peer[(row & (CR - 1)) * N2 + rank * CC + c]);
            }
        },
        [&](int c, int e, int step, auto &x) {
#pragma unroll
            for (int i = 0; i < (int)(sizeof(x) / 8); i++) dst[(size_t)(e + i * step) * N2 + rank * CC + c] = A::canon_inv(x[i], k);
        });
    cg::this_cluster().sync();
}

template <int LOGN>
__global__ void __launch_bounds__(WholeCfg<LOGN>::THREADS, 512 / WholeCfg<LOGN>::THREADS) ntt_inv_whole(NttArgs a) {
    pdl_enter();
    extern __shared__ __align__(16) uint64_t whole_sm[];
    const Job job = get_job(a, blockIdx.x >> WholeCfg<LOGN>::LOG_CL);
    const Mod md = a.mod[job.y];
    with_arith(md.q, [&](auto A) { whole_inv_body<decltype(A), LOGN>(a, whole_sm, job, md); });
}

static_assert(whole_smem<14>() <= 48 * 1024, "no opt-in to a larger shared memory is asked for");

// ---- launchers (ntt_whole.cu); they set no error state of their own: the caller reads cudaGetLastError -----------------------
void launch_inv_whole(const NttArgs &a, uint32_t njobs, uint32_t batch, cudaStream_t s);
template <class Epi, int SRC>
void launch_fwd_whole(const NttArgs &a, const Epi &epi, uint32_t njobs, uint32_t batch, cudaStream_t s);

}  // namespace b2
