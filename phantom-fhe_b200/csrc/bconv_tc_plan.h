// bconv_tc_plan.h - data structures, reduction and host-side planning of the tensor-core base conversion (kernel: bconv_tc.cuh).
// Plain C++: also compiled by the CPU test-suite, which emulates the matrix product on the byte images built here.
//
// The conversion (src/rns_bconv.cu:143-168, 455-485; include/rns_bconv.cuh:112-125)
//     out_j[n] = (sum_i y_i[n] * M_ji) mod p_j,      i < ni <= 8 inputs, j over the group's outputs
// is a small u8 x u8 -> s32 matrix product per tile of coefficients:
//   * a residue is its own little-endian bytes, y_i = sum_a 2^(8a) y_{i,a}, so the eight uint64 input
//     limbs of a coefficient ARE the K = 64 bytes of its part of A (k = 8 i + a);
//   * the weight of the input byte is folded into the matrix modulo the output prime:
//         sum_i y_i M_ji  =  sum_{i,a} y_{i,a} * (2^(8a) M_ji mod p_j)      (mod p_j),
//     and that constant, below p_j, is split into its nb_j bytes: column (j, b) of B holds byte b;
//   * D[n][(j,b)] = sum_k A[n][k] B[k][(j,b)] < 64 * 255^2 < 2^22 is exact in int32, and
//         V_j = sum_b D[n][(j,b)] 2^(8b)  =  out_j[n]  (mod p_j),   V_j < 2^(8 nb_j + 14.01).
// The epilogue shift-adds nb_j (4 to 8) int32 words into one 64- or 96-bit integer and reduces it once:
// quotient estimate from the top 32 bits times a 32-bit reciprocal (never above the true quotient, at most
// one below), so the result is below 2 p_j; the transform that follows takes it so (SRC_WORDS). The canonical residue is
// unique: behind the transform the limbs equal those of the integer and FP64 kernels bit for bit.
//
// A row of A holds TWO coefficients: K slice i (16 bytes) is input limb i of both, as it lies in memory. Outputs are packed into
// groups of floor(16 / nb) outputs of equal byte count nb, 32 accumulator columns a group: output o in columns 2 nb o .. (the first
// coefficient's nb bytes, then the second's), zero in the half of every slice that belongs to the other coefficient. A job (a digit
// of ModUp, a polynomial of ModDown) has at most TC_MAX_GROUPS groups. Its image of B is an even number of slices (an MMA takes
// two) one after another, in each the columns' 16 bytes: the canonical K-major no-swizzle form of the sm_100 shared-memory matrix
// descriptor (core matrices of 8 rows x 16 bytes), K neighbours one slice apart.
#pragma once
#include <algorithm>
#include <cstdint>
#include <utility>
#include <vector>

#if defined(__CUDACC__)
#define B2_HD __host__ __device__ __forceinline__
#else
#define B2_HD inline
#endif

namespace b2 {

struct TcOut {
    uint64_t p;     // output prime
    uint32_t mu;    // floor(2^(8 nb + 15) / p)
    uint32_t slot;  // output limb (absolute slot in the output buffer)
};
struct TcGroup {
    uint32_t nb;       // bytes per output of this group (4..8)
    uint32_t n_valid;  // outputs present (1 .. 16 / nb)
    uint32_t pad0, pad1;
    TcOut o[4];
};
struct TcJob {
    uint32_t in_slot0, ni;     // first input limb, number of input limbs (<= 8)
    uint32_t copy_dst_slot0;   // ModUp: where the digit's own limbs are copied to (0xFFFFFFFF: no copy)
    uint32_t n_groups;         // column groups (<= TC_MAX_GROUPS)
    uint32_t img_off;          // byte offset of the B image (512 bytes a group and slice)
    uint32_t grp_off;          // first TcGroup of the job
    uint32_t pad;
    uint32_t in_stride1;       // input limb i sits at slot in_slot0 + i * (in_stride1 + 1)
};
static_assert(sizeof(TcOut) == 16 && sizeof(TcGroup) == 80 && sizeof(TcJob) == 32, "device layouts");

// slices of 16 bytes of K: one per input limb, an even number
B2_HD uint32_t tc_slices(uint32_t ni) { return (ni + 1) & ~1u; }

// sum_b c[b] 2^(8b) mod p, below 2 p, for NB words below 2^22 each: paired with shift-adds, joined by one (7 and 8 planes: two)
// wide multiply-adds, the quotient estimate one high multiply, v + qhat (2^64 - p) one wide multiply-add and one narrow one.
// The true value is below 2 p < 2^62: the wrap-around is harmless. np: 2^64 - p as two words; mu = floor(2^(8 NB + 15) / p)
struct TcWord {
    uint32_t lo, hi;
};
// (hi:lo >> s) mod 2^32 for s < 32, and the high word of a product (as plain expressions on the device too, eight hoisted rotations at
// 2^15 took 204.9 instead of 203.3 us)
B2_HD uint32_t tc_funnel(uint32_t lo, uint32_t hi, int s) {
#if defined(__CUDA_ARCH__)
    return __funnelshift_r(lo, hi, s);
#else
    return (uint32_t)((((uint64_t)hi << 32) | lo) >> s);
#endif
}
B2_HD uint32_t tc_mulhi(uint32_t a, uint32_t b) {
#if defined(__CUDA_ARCH__)
    return __umulhi(a, b);
#else
    return (uint32_t)(((uint64_t)a * b) >> 32);
#endif
}
template <int NB>
B2_HD TcWord tc_residue(const uint32_t *c, uint32_t np_lo, uint32_t np_hi, uint32_t mu) {
    static_assert(NB >= 4 && NB <= 8, "4 to 8 bytes per output prime");
    constexpr int SH = 8 * NB - 17;  // V >> SH fits 32 bits
    const uint32_t x0 = c[0] + (c[1] << 8), x1 = c[2] + (c[3] << 8);
    uint32_t vl, vh, vq;  // V mod 2^64 as two words; V >> SH
    if constexpr (NB <= 6) {
        const uint32_t x2 = NB == 4 ? 0u : (NB == 5 ? c[4] : c[4] + (c[5] << 8));
        const uint64_t v = (uint64_t)x1 * 65536u + (((uint64_t)x2 << 32) | x0);
        vl = (uint32_t)v, vh = (uint32_t)(v >> 32);
        vq = tc_funnel(vl, vh, SH);
    } else {
        const uint32_t x2 = c[4] + (c[5] << 8), x3 = NB == 7 ? c[6] : c[6] + (c[7] << 8);
        const uint64_t a = (uint64_t)x1 * 65536u + x0, b = (uint64_t)x3 * 65536u + x2;
        const uint64_t mid = (a >> 32) + b;  // V >> 32, below 2^47
        vl = (uint32_t)a, vh = (uint32_t)mid;
        vq = tc_funnel((uint32_t)mid, (uint32_t)(mid >> 32), SH - 32);
    }
    const uint32_t qhat = tc_mulhi(vq, mu);
    const uint64_t t = (uint64_t)qhat * np_lo + (((uint64_t)vh << 32) | vl);
    return TcWord{(uint32_t)t, (uint32_t)(t >> 32) + qhat * np_hi};
}

// How long a warp polls a barrier: until its phase has ended, TC_WAIT_LIMIT polls at most, and ONE poll once another wait of the
// CTA has run out, so that the CTA ends soon. `drain`: the waits before the CTA ends for what it has in flight itself. Whether
// another wait gave up says nothing about them, and the hardware still writes to shared and tensor memory until they are over:
// they take their own limit.
constexpr uint32_t TC_WAIT_LIMIT = 1u << 22;
template <class Poll>
B2_HD bool tc_poll(Poll &&poll, volatile uint32_t *gave_up, bool drain) {
    for (uint32_t it = 0; it < TC_WAIT_LIMIT; it++) {
        if (poll()) return true;
        if (!drain && *gave_up) return false;
    }
    *gave_up = 1u;
    return false;
}

struct TcSpecOut {
    uint32_t slot;        // absolute output limb
    uint64_t p;           // its prime
    const uint64_t *row;  // M[j][0..ni)
};

static inline uint32_t tc_nbytes(uint64_t p) { return std::max(4u, (uint32_t)((64 - __builtin_clzll(p) + 7) / 8)); }

constexpr uint32_t TC_MAX_GROUPS = 16;  // column groups of a job

struct TcBuild {
    std::vector<TcJob> jobs;
    std::vector<TcGroup> groups;
    std::vector<uint8_t> images;
    bool ok = true;
    // One conversion (a digit, a polynomial): outputs are packed, in order, into groups of equal byte count; more than
    // TC_MAX_GROUPS groups are dealt evenly over further jobs on the same inputs. Returns the number of jobs added.
    uint32_t add(uint32_t in_slot0, uint32_t ni, uint32_t copy_dst, const std::vector<TcSpecOut> &outs, uint32_t in_stride = 1) {
        if (ni < 1 || ni > 8 || outs.empty()) {
            ok = false;
            return 0;
        }
        uint32_t added = 0;
        size_t i = 0;
        // groups the outputs need in all -> jobs of equal size
        uint32_t total_groups = 0;
        for (size_t k = 0; k < outs.size();) {
            const uint32_t nb = tc_nbytes(outs[k].p), opg = 16 / nb;
            uint32_t cnt = 0;
            while (k < outs.size() && cnt < opg && tc_nbytes(outs[k].p) == nb) cnt++, k++;
            total_groups++;
        }
        const uint32_t n_split = (total_groups + TC_MAX_GROUPS - 1) / TC_MAX_GROUPS, per_job = (total_groups + n_split - 1) / n_split;
        while (i < outs.size()) {
            TcJob job{in_slot0, ni, added == 0 ? copy_dst : 0xFFFFFFFFu, 0, (uint32_t)images.size(), (uint32_t)groups.size(), 0, in_stride - 1};
            std::vector<std::pair<size_t, uint32_t>> placed;  // (output index, first column) of this job
            while (i < outs.size() && job.n_groups < per_job) {
                const uint32_t nb = tc_nbytes(outs[i].p), opg = 16 / nb;
                TcGroup g{};
                g.nb = nb;
                while (i < outs.size() && g.n_valid < opg && tc_nbytes(outs[i].p) == nb) {
                    const uint64_t p = outs[i].p;
                    const unsigned __int128 mu = ((unsigned __int128)1 << (8 * nb + 15)) / p;
                    if (p <= (1ull << 16) || (mu >> 32)) ok = false;
                    g.o[g.n_valid] = TcOut{p, (uint32_t)mu, outs[i].slot};
                    placed.push_back({i, 32 * job.n_groups + g.n_valid * 2 * nb});
                    g.n_valid++;
                    i++;
                }
                groups.push_back(g);
                job.n_groups++;
            }
            const size_t img0 = images.size(), cols = 32 * job.n_groups;
            images.resize(img0 + tc_slices(ni) * cols * 16, 0);
            for (auto &pl : placed) {
                const TcSpecOut &o = outs[pl.first];
                const uint32_t nb = tc_nbytes(o.p);
                for (uint32_t ii = 0; ii < ni; ii++)
                    for (uint32_t a = 0; a < 8; a++) {
                        const uint64_t e = (uint64_t)((((unsigned __int128)(o.row[ii] % o.p)) << (8 * a)) % o.p);
                        for (uint32_t b = 0; b < nb; b++)
                            for (uint32_t c = 0; c < 2; c++)  // the row's coefficients
                                images[img0 + (ii * cols + pl.second + c * nb + b) * 16 + 8 * c + a] = (uint8_t)(e >> (8 * b));
                    }
            }
            jobs.push_back(job);
            added++;
        }
        return added;
    }
};

}  // namespace b2
