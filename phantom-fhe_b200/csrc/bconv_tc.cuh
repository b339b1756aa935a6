// bconv_tc.cuh - fast base conversion on the sm_100a tensor cores (tcgen05.mma kind::i8, accumulators in TMEM).
// The formulation, the data structures, the reduction and the host-side planning are in bconv_tc_plan.h.
//
// A tile is 256 coefficients of one job: 128 rows of two coefficients, so that an input limb's share of the tile is 2 KB of
// consecutive memory AND, as it lies there, one 16-byte K slice of all rows of A. One cp.async.bulk per limb brings it in, no
// thread touches it, and a thread of the epilogue (TMEM lane = row) holds both coefficients of an output: one record, one
// address and one 16-byte store for the two. The price is a B whose blocks for the other coefficient of a row are zero, twice
// the multiplications, on a unit that has them to spare.
//
// Fourteen warps a CTA, two CTAs an SM, each walking a run of consecutive items (job part, set, tile): warp 13 loads (a ring of
// A tiles, the part's B image when the part changes), warp 12 issues the MMAs of three column groups at a time into one of two
// 96-column accumulators, warps 0 to 11 (TMEM lanes 32 (w % 4) .. +31, a group each) reduce and store the other. Groups a
// buffer, ModUp and ModDown of sixteen key switches of 24 limbs and 8 special primes at 2^16, us a key switch: two 18.6, three
// 17.1, four 17.8 (spills). Six warps of the epilogue on an SM sub-partition hide a warp's chain of TMEM load, reduction and store:
// with four, of two groups each in turn, and the records read from global memory, 21.8.
// Two A tiles in flight: three or four are no faster, and their shared memory keeps the CTAs of other streams' kernels off the
// SM, and this kernel's CTAs off an SM that those have not left (four streams of key switches 7420 a second with two, 6700
// with four).
// The form before (a coefficient a row, rows filled by cp.async of eight bytes, a barrier pair per tile of 128 coefficients)
// took 73 warp instructions an output and 25.0 us; the bytes alone take 12.9 at the copy rate. A launch that gives a CTA one
// tile takes 0.5 us longer than it did then: a bulk copy arrives a microsecond after its issue. The first tile filled by all
// threads was slower still (rotations at 2^14, 16 limbs, alpha 8 60.8 -> 64.2 us): the instructions of a kernel that runs for
// three microseconds are fetched as they are executed.
// No multicast, no cluster; every wait is bounded and reports through a status word instead of spinning forever; copies and
// MMAs in flight are waited for, with a limit of their own when another wait has run out, and TMEM is released on every path.
#pragma once
#include <cstdint>
#include <cuda_runtime.h>

#include "bconv_tc_plan.h"
#include "modarith.cuh"

namespace b2 {

constexpr uint32_t TC_TILE = 256;                   // coefficients of a tile
constexpr uint32_t TC_SLICE = TC_TILE * 8;          // bytes of one input limb's share of it: one K slice of A
constexpr uint32_t TC_STAGES = 2;                   // A tiles in flight
constexpr uint32_t TC_CHUNK = 3;                    // column groups of one accumulator buffer: one per warp of a TMEM quadrant
constexpr uint32_t TC_ACC_COLS = 32 * TC_CHUNK, TC_TMEM_COLS = 256, TC_BUFS = TC_TMEM_COLS / TC_ACC_COLS;
constexpr uint32_t TC_EPI_WARPS = 4 * TC_CHUNK, TC_THREADS = 32 * (TC_EPI_WARPS + 2);
constexpr uint32_t TC_CTRL_BYTES = 256;             // barriers and the like
constexpr uint32_t TC_SM_SMEM = 233472;             // shared memory of one SM (228 KB)
constexpr uint32_t TC_SMEM_MAX_REQUEST = TC_SM_SMEM / 2 - 1024;  // two CTAs an SM, a kilobyte each for the system

__device__ __forceinline__ uint32_t tc_smem_u32(const void *p) { return (uint32_t)__cvta_generic_to_shared(p); }

// shared-memory matrix descriptor: K-major, no swizzle; lbo = bytes between K-adjacent core matrices, 128 bytes between groups
// of eight rows; descriptor version 1 (sm_100)
__device__ __forceinline__ uint64_t tc_desc(uint32_t smem_addr, uint32_t lbo) {
    return (uint64_t)((smem_addr & 0x3FFFFu) >> 4) | ((uint64_t)(lbo >> 4) << 16) | ((uint64_t)(128u >> 4) << 32) | ((uint64_t)1 << 46);
}

__device__ __forceinline__ void tc_mma_i8(uint32_t d_tmem, uint64_t adesc, uint64_t bdesc, uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n\t"
        ".reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::i8 [%0], %1, %2, %3, p;\n\t"
        "}\n" ::"r"(d_tmem),
        "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate)
        : "memory");
}
__device__ __forceinline__ void tc_commit(uint32_t bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ void tc_bar_init(uint32_t bar, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count) : "memory");
}
__device__ __forceinline__ void tc_expect(uint32_t bar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}
__device__ __forceinline__ void tc_arrive(uint32_t bar) { asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory"); }
// bytes and both addresses multiples of 16
__device__ __forceinline__ void tc_bulk(uint32_t smem_dst, const void *gsrc, uint32_t bytes, uint32_t bar) {
    asm volatile("cp.async.bulk.shared::cta.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(smem_dst), "l"(gsrc), "r"(bytes), "r"(bar)
                 : "memory");
}
// waits for the phase of the given parity to end (tc_poll has the limits)
template <bool DRAIN = false>
__device__ __forceinline__ bool tc_wait(uint32_t bar, uint32_t parity, volatile uint32_t *gave_up) {
    return tc_poll(
        [&] {
            uint32_t done;
            asm volatile(
                "{\n\t"
                ".reg .pred P1;\n\t"
                "mbarrier.try_wait.parity.shared::cta.b64 P1, [%1], %2;\n\t"
                "selp.b32 %0, 1, 0, P1;\n\t"
                "}\n"
                : "=r"(done)
                : "r"(bar), "r"(parity)
                : "memory");
            return done != 0;
        },
        gave_up, DRAIN);
}

// 32 consecutive accumulator columns of this thread's TMEM lane, and the wait as a statement that owns the registers: a
// group's planes can be on their way while the previous group is reduced
__device__ __forceinline__ void tc_ld32(uint32_t taddr, uint32_t (&c)[32]) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
        "%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];\n"
        : "=r"(c[0]), "=r"(c[1]), "=r"(c[2]), "=r"(c[3]), "=r"(c[4]), "=r"(c[5]), "=r"(c[6]), "=r"(c[7]), "=r"(c[8]), "=r"(c[9]), "=r"(c[10]),
          "=r"(c[11]), "=r"(c[12]), "=r"(c[13]), "=r"(c[14]), "=r"(c[15]), "=r"(c[16]), "=r"(c[17]), "=r"(c[18]), "=r"(c[19]), "=r"(c[20]),
          "=r"(c[21]), "=r"(c[22]), "=r"(c[23]), "=r"(c[24]), "=r"(c[25]), "=r"(c[26]), "=r"(c[27]), "=r"(c[28]), "=r"(c[29]), "=r"(c[30]), "=r"(c[31])
        : "r"(taddr)
        : "memory");
}
__device__ __forceinline__ void tc_wait_ld(uint32_t (&c)[32]) {
    asm volatile("tcgen05.wait::ld.sync.aligned;\n"
                 : "+r"(c[0]), "+r"(c[1]), "+r"(c[2]), "+r"(c[3]), "+r"(c[4]), "+r"(c[5]), "+r"(c[6]), "+r"(c[7]), "+r"(c[8]), "+r"(c[9]), "+r"(c[10]),
                   "+r"(c[11]), "+r"(c[12]), "+r"(c[13]), "+r"(c[14]), "+r"(c[15]), "+r"(c[16]), "+r"(c[17]), "+r"(c[18]), "+r"(c[19]), "+r"(c[20]),
                   "+r"(c[21]), "+r"(c[22]), "+r"(c[23]), "+r"(c[24]), "+r"(c[25]), "+r"(c[26]), "+r"(c[27]), "+r"(c[28]), "+r"(c[29]), "+r"(c[30]), "+r"(c[31])
                 :
                 : "memory");
}

// the NV outputs of a group, two coefficients each
template <int NB, int NV>
__device__ __forceinline__ void tc_group(const uint32_t (&c)[32], const TcGroup *g, uint32_t slot_words, uint64_t *__restrict__ out_n) {
#pragma unroll
    for (int o = 0; o < NV; o++) {
        const uint4 r = *reinterpret_cast<const uint4 *>(&g->o[o]);
        // r: {2^64 - p as two words, mu, slot}
        const TcWord e = tc_residue<NB>(c + 2 * NB * o, r.x, r.y, r.z), f = tc_residue<NB>(c + 2 * NB * o + NB, r.x, r.y, r.z);
        asm volatile("st.global.v4.u32 [%0], {%1, %2, %3, %4};" ::"l"(out_n + r.w * slot_words), "r"(e.lo), "r"(e.hi), "r"(f.lo), "r"(f.hi) : "memory");
    }
}
__device__ __forceinline__ void tc_group_any(const uint32_t (&c)[32], uint2 hdr, const TcGroup *g, uint32_t slot_words, uint64_t *__restrict__ out_n) {
    switch (hdr.x * 8 + hdr.y) {  // (bytes per output, outputs in the group): no slot is processed in vain
        case 4 * 8 + 1: tc_group<4, 1>(c, g, slot_words, out_n); break;
        case 4 * 8 + 2: tc_group<4, 2>(c, g, slot_words, out_n); break;
        case 4 * 8 + 3: tc_group<4, 3>(c, g, slot_words, out_n); break;
        case 4 * 8 + 4: tc_group<4, 4>(c, g, slot_words, out_n); break;
        case 5 * 8 + 1: tc_group<5, 1>(c, g, slot_words, out_n); break;
        case 5 * 8 + 2: tc_group<5, 2>(c, g, slot_words, out_n); break;
        case 5 * 8 + 3: tc_group<5, 3>(c, g, slot_words, out_n); break;
        case 6 * 8 + 1: tc_group<6, 1>(c, g, slot_words, out_n); break;
        case 6 * 8 + 2: tc_group<6, 2>(c, g, slot_words, out_n); break;
        case 7 * 8 + 1: tc_group<7, 1>(c, g, slot_words, out_n); break;
        case 7 * 8 + 2: tc_group<7, 2>(c, g, slot_words, out_n); break;
        case 8 * 8 + 1: tc_group<8, 1>(c, g, slot_words, out_n); break;
        case 8 * 8 + 2: tc_group<8, 2>(c, g, slot_words, out_n); break;
        default: break;  // an empty group: the planner makes none
    }
}

constexpr uint32_t TC_JOBS_INLINE = 8;
struct TcArgs {
    const uint64_t *in;
    uint64_t *out;
    const uint64_t *copy_src;  // optional (one set): the digit's own limbs go from here to the jobs' copy slots
    const TcJob *jobs;         // the first TC_JOBS_INLINE of them in job[] as well: a load from memory less before the first copy
    const TcGroup *groups;     // device form: o[].p holds 2^64 - p
    const uint8_t *images;
    uint32_t *err;
    uint32_t N;
    uint32_t items, more;      // a CTA works on `items` (job part, set, tile)s, the first `more` CTAs on one more
    uint32_t parts;            // a job's groups are dealt over this many parts, items of their own
    uint32_t stage_bytes, b_bytes;
    uint32_t part_recs;        // most groups of a part: the output records of a CTA's parts lie that far apart
    // A batch of conversions in one launch: set b reads input limb slot s at s * (in_lm1 + 1) + b * in_bs and writes output
    // limb slot s at s * (out_lm1 + 1) + b * out_bs (batch-major and limb-major buffers as for the transforms, ntt_kernels.cuh)
    uint32_t batch, in_lm1, in_bs, out_lm1, out_bs;
    TcJob job[TC_JOBS_INLINE];
};
__device__ __forceinline__ TcJob tc_job(const TcArgs &a, uint32_t j) { return j < TC_JOBS_INLINE ? a.job[j] : a.jobs[j]; }

// part `part` of a job: groups [g0, g1)
__device__ __forceinline__ void tc_part(const TcJob &job, uint32_t part, uint32_t parts, uint32_t &g0, uint32_t &g1) {
    g0 = job.n_groups * part / parts, g1 = job.n_groups * (part + 1) / parts;
}

__global__ void __launch_bounds__(TC_THREADS, 2) bconv_tc_pairs(const __grid_constant__ TcArgs a) {
    pdl_enter();
    extern __shared__ __align__(1024) uint8_t tc_smem[];
    const uint32_t sA = tc_smem_u32(tc_smem), sB = sA + TC_STAGES * a.stage_bytes;
    uint8_t *ctrl = tc_smem + TC_STAGES * a.stage_bytes + a.b_bytes;
    const uint32_t bar = tc_smem_u32(ctrl);
    const uint32_t full_a = bar, empty_a = bar + 32, full_t = bar + 64, empty_t = bar + 96, full_b = bar + 128, drained = bar + 136;
    uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(ctrl + 144);
    volatile uint32_t *gave_up = reinterpret_cast<volatile uint32_t *>(ctrl + 148);
    static_assert(TC_STAGES <= 4 && TC_BUFS <= 4, "four barriers of a kind");
    const uint32_t tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const uint32_t log_tiles = 31 - __clz(a.N / TC_TILE), per_part = a.batch << log_tiles, tile_mask = (1u << log_tiles) - 1;
    // consecutive items: a CTA changes its part as seldom as can be
    const uint32_t v0 = blockIdx.x * a.items + min(blockIdx.x, a.more), v1 = v0 + a.items + (blockIdx.x < a.more);

    TcGroup *recs = reinterpret_cast<TcGroup *>(ctrl + TC_CTRL_BYTES);
    const uint32_t first_part = v0 / per_part;

    // ---- loads: one warp, a lane a copy. The first item's are under way before the CTA meets for the first time ---------------
    uint32_t cur = 0xFFFFFFFFu, n_b = 0;
    TcJob job{};
    auto load_item = [&](uint32_t v, uint32_t k) {
        const uint32_t pi = v / per_part, st = k % TC_STAGES;
        if (pi != cur) {
            // the part's columns of the job's B image; the MMAs that read the old one are done when the last item's are
            if (k && !__all_sync(0xFFFFFFFFu, tc_wait(empty_a + 8 * ((k - 1) % TC_STAGES), ((k - 1) / TC_STAGES) & 1, gave_up))) return false;
            job = tc_job(a, pi / a.parts);
            uint32_t g0, g1;
            tc_part(job, pi % a.parts, a.parts, g0, g1);
            const uint32_t slices = tc_slices(job.ni), row = job.n_groups * 512, part_row = (g1 - g0) * 512;
            if (lane == 0) tc_expect(full_b, slices * part_row);
            __syncwarp();
            if (lane < slices) tc_bulk(sB + lane * part_row, a.images + job.img_off + g0 * 512 + lane * row, part_row, full_b);
            cur = pi, n_b++;
        }
        if (k >= TC_STAGES && !__all_sync(0xFFFFFFFFu, tc_wait(empty_a + 8 * st, (k / TC_STAGES - 1) & 1, gave_up))) return false;
        const uint32_t tile = v & tile_mask, set = (v - pi * per_part) >> log_tiles;
        if (lane == 0) tc_expect(full_a + 8 * st, job.ni * TC_SLICE);
        __syncwarp();
        if (lane < job.ni) {
            const size_t slot = (size_t)(job.in_slot0 + lane * (job.in_stride1 + 1)) * (a.in_lm1 + 1) + (size_t)set * a.in_bs;
            tc_bulk(sA + st * a.stage_bytes + lane * TC_SLICE, a.in + slot * a.N + (size_t)tile * TC_TILE, TC_SLICE, full_a + 8 * st);
        }
        return true;
    };
    if (warp == TC_EPI_WARPS + 1) {
        // barriers 0 .. 17 as laid out above; those of empty_t take an arrival from every warp of the epilogue
        if (lane < 18) tc_bar_init(bar + 8 * lane, lane >= 12 && lane < 16 ? TC_EPI_WARPS : 1);
        if (lane == 0) *gave_up = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        __syncwarp();
        load_item(v0, 0);
    } else if (warp == TC_EPI_WARPS) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(tc_smem_u32(tmem_slot)), "r"(TC_TMEM_COLS) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    } else {
        // the output records of every part the CTA will work on
        for (uint32_t pi = first_part + warp; pi <= (v1 - 1) / per_part; pi += TC_EPI_WARPS) {
            const TcJob j = tc_job(a, pi / a.parts);
            uint32_t g0, g1;
            tc_part(j, pi % a.parts, a.parts, g0, g1);
            const uint4 *src = reinterpret_cast<const uint4 *>(a.groups + j.grp_off + g0);
            uint4 *dst = reinterpret_cast<uint4 *>(recs + (pi - first_part) * a.part_recs);
            for (uint32_t i = lane; i < (g1 - g0) * (sizeof(TcGroup) / 16); i += 32) dst[i] = __ldg(src + i);
        }
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem = *tmem_slot;

    if (warp == TC_EPI_WARPS + 1) {
        uint32_t k = 1;
        for (uint32_t v = v0 + 1; v < v1; v++, k++)
            if (!load_item(v, k)) break;
        // nothing may be in flight when the CTA ends
        for (uint32_t i = k > TC_STAGES ? k - TC_STAGES : 0; i < k; i++) tc_wait<true>(full_a + 8 * (i % TC_STAGES), (i / TC_STAGES) & 1, gave_up);
        tc_wait<true>(full_b, (n_b - 1) & 1, gave_up);
    } else if (warp == TC_EPI_WARPS) {
        // ---- MMAs -------------------------------------------------------------------------------------------------
        if (lane == 0) {
            uint32_t n_t = 0, k = 0, cols = 0, steps = 0;
            bool ok = true;
            for (uint32_t v = v0; v < v1 && ok; v++, k++) {
                const uint32_t pi = v / per_part, st = k % TC_STAGES;
                if (pi != cur) {
                    job = tc_job(a, pi / a.parts);
                    uint32_t g0, g1;
                    tc_part(job, pi % a.parts, a.parts, g0, g1);
                    cols = (g1 - g0) * 32, steps = (job.ni + 1) / 2;
                    if (!(ok = tc_wait(full_b, n_b & 1, gave_up))) break;
                    cur = pi, n_b++;
                }
                if (!(ok = tc_wait(full_a + 8 * st, (k / TC_STAGES) & 1, gave_up))) break;
                const uint64_t adesc = tc_desc(sA + st * a.stage_bytes, TC_SLICE);
                for (uint32_t c0 = 0; c0 < cols; c0 += TC_ACC_COLS, n_t++) {
                    const uint32_t buf = n_t % TC_BUFS, n = min(cols - c0, TC_ACC_COLS);
                    if (n_t >= TC_BUFS && !(ok = tc_wait(empty_t + 8 * buf, (n_t / TC_BUFS - 1) & 1, gave_up))) break;
                    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                    const uint64_t bdesc = tc_desc(sB + c0 * 16, cols * 16);
                    // D s32, A and B u8, both K-major, M = 128, N = the columns of up to TC_CHUNK groups
                    const uint32_t idesc = (2u << 4) | ((n >> 3) << 17) | ((128u >> 4) << 24);
                    for (uint32_t s = 0; s < steps; s++)  // 32 bytes of K: two input limbs
                        tc_mma_i8(tmem + buf * TC_ACC_COLS, adesc + s * (2 * TC_SLICE >> 4), bdesc + s * (2 * cols * 16 >> 4), idesc, s != 0);
                    tc_commit(full_t + 8 * buf);
                }
                tc_commit(empty_a + 8 * st);
            }
            tc_commit(drained);
            tc_wait<true>(drained, 0, gave_up);
        }
    } else {
        // ---- reduction and stores -----------------------------------------------------------------------------------
        const uint32_t lane_base = tmem + ((warp & 3) << 21), mine = warp >> 2, n_row = 2 * ((warp & 3) * 32 + lane);
        const uint32_t slot_words = (a.out_lm1 + 1) * a.N;
        uint32_t n_t = 0, k = 0, g0 = 0, g1 = 0;
        bool ok = true;
        for (uint32_t v = v0; v < v1 && ok; v++, k++) {
            const uint32_t pi = v / per_part, tile = v & tile_mask, set = (v - pi * per_part) >> log_tiles;
            if (pi != cur) {
                job = tc_job(a, pi / a.parts);
                tc_part(job, pi % a.parts, a.parts, g0, g1);
                cur = pi;
            }
            if (a.copy_src != nullptr && g0 == 0 && job.copy_dst_slot0 != 0xFFFFFFFFu && tid < TC_TILE)
                for (uint32_t i = 0; i < job.ni; i++)
                    a.out[(size_t)(job.copy_dst_slot0 + i) * a.N + (size_t)tile * TC_TILE + tid] =
                        a.copy_src[(size_t)(job.in_slot0 + i) * a.N + (size_t)tile * TC_TILE + tid];
            uint64_t *out_n = a.out + (size_t)set * a.out_bs * a.N + (tile * TC_TILE + n_row);
            // a last chunk that is not full is shared out evenly over the items
            const uint32_t own = (mine + k) % TC_CHUNK;
            for (uint32_t c0 = 0; c0 < g1 - g0; c0 += TC_CHUNK, n_t++) {
                const uint32_t buf = n_t % TC_BUFS, g = c0 + own;
                const bool work = g < g1 - g0;
                const TcGroup *G = recs + (pi - first_part) * a.part_recs + (work ? g : 0);
                const uint2 hdr = *reinterpret_cast<const uint2 *>(G);
                ok = __all_sync(0xFFFFFFFFu, tc_wait(full_t + 8 * buf, (n_t / TC_BUFS) & 1, gave_up));
                if (!ok) break;
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                uint32_t c[32];
                if (work) {
                    tc_ld32(lane_base + buf * TC_ACC_COLS + own * 32, c);
                    tc_wait_ld(c);
                }
                asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
                __syncwarp();
                if (lane == 0) tc_arrive(empty_t + 8 * buf);  // the planes are in registers
                if (work) tc_group_any(c, hdr, G, slot_words, out_n);
            }
        }
    }
    __syncwarp();
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (tid == 0 && *gave_up) atomicExch(a.err, 1u);  // a barrier never completed: outputs from there on are not written
    if (warp == TC_EPI_WARPS) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(TC_TMEM_COLS) : "memory");
}

}  // namespace b2
