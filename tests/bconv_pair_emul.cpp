// CPU emulation of the tensor-core base conversion as the kernel lays it out (bconv_tc.cuh): the planner's groups and images
// (bconv_tc_plan.h), rows of A of two coefficients, K slices copied as they lie in memory, the image of B cut into parts by column
// groups, accumulator columns addressed as the matrix descriptors and tcgen05.ld address them, and the kernel's own reduction.
// Every output is compared with (sum_i y_i M_ji) mod p_j in 128-bit integers. Usage: bconv_pair_emul <seed>; prints "ok <cases>" or the first mismatch.
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <vector>

#include "bconv_tc_plan.h"

typedef unsigned __int128 u128;
static uint64_t rng_state;
static uint64_t rnd() {
    uint64_t z = (rng_state += 0x9E3779B97F4A7C15ull);
    z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
    z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
    return z ^ (z >> 31);
}
static uint64_t odd_bits(int bits) { return (rnd() >> (64 - bits)) | (1ull << (bits - 1)) | 1ull; }

static const uint32_t SLICE = 2048;

static uint64_t residue(uint32_t nb, const uint32_t *c, const b2::TcOut &m) {
    const uint64_t np = 0 - m.p;
    const uint32_t lo = (uint32_t)np, hi = (uint32_t)(np >> 32);
    b2::TcWord w;
    switch (nb) {
        case 4: w = b2::tc_residue<4>(c, lo, hi, m.mu); break;
        case 5: w = b2::tc_residue<5>(c, lo, hi, m.mu); break;
        case 6: w = b2::tc_residue<6>(c, lo, hi, m.mu); break;
        case 7: w = b2::tc_residue<7>(c, lo, hi, m.mu); break;
        default: w = b2::tc_residue<8>(c, lo, hi, m.mu); break;
    }
    return ((uint64_t)w.hi << 32) | w.lo;
}

static int run_case(int ni, const std::vector<int> &in_bits, const std::vector<int> &out_bits, uint32_t parts, bool extremes) {
    std::vector<uint64_t> q(ni), p(out_bits.size()), mat(out_bits.size() * ni);
    std::vector<b2::TcSpecOut> outs;
    for (int i = 0; i < ni; i++) q[i] = odd_bits(in_bits[i]);
    for (size_t j = 0; j < out_bits.size(); j++) {
        p[j] = odd_bits(out_bits[j]);
        for (int i = 0; i < ni; i++) mat[j * ni + i] = extremes ? p[j] - 1 : rnd() % p[j];
        outs.push_back(b2::TcSpecOut{(uint32_t)(100 + j), p[j], &mat[j * ni]});
    }
    b2::TcBuild tb;
    const uint32_t n_jobs = tb.add(3, (uint32_t)ni, 0xFFFFFFFFu, outs);
    if (!tb.ok || n_jobs == 0) return printf("planner refused a valid case\n"), 1;
    std::vector<uint64_t> y((size_t)ni * 256);
    for (int i = 0; i < ni; i++)
        for (int n = 0; n < 256; n++) y[(size_t)i * 256 + n] = (extremes || n == 5) ? q[i] - 1 : (n == 8 ? 0 : rnd() % q[i]);
    const uint32_t slices = b2::tc_slices((uint32_t)ni);
    std::vector<uint8_t> A((size_t)slices * SLICE, 0xA5);  // a slice without a limb holds whatever was there
    for (int i = 0; i < ni; i++) memcpy(&A[(size_t)i * SLICE], &y[(size_t)i * 256], SLICE);
    std::vector<char> seen(out_bits.size(), 0);
    for (uint32_t jb = 0; jb < n_jobs; jb++) {
        const b2::TcJob &job = tb.jobs[jb];
        if (job.n_groups < 1 || job.n_groups > b2::TC_MAX_GROUPS || job.in_slot0 != 3 || job.ni != (uint32_t)ni || (job.img_off & 15) ||
            job.img_off + (size_t)slices * job.n_groups * 512 != (jb + 1 < n_jobs ? tb.jobs[jb + 1].img_off : tb.images.size()))
            return printf("bad job header\n"), 1;
        const uint8_t *img = tb.images.data() + job.img_off;
        const uint32_t np = parts < job.n_groups ? parts : job.n_groups;
        for (uint32_t part = 0; part < np; part++) {
            const uint32_t g0 = job.n_groups * part / np, g1 = job.n_groups * (part + 1) / np, cols = (g1 - g0) * 32;
            if (g0 == g1) return printf("an empty part\n"), 1;
            std::vector<uint8_t> B((size_t)slices * cols * 16);
            for (uint32_t i = 0; i < slices; i++) memcpy(&B[(size_t)i * cols * 16], &img[(size_t)i * job.n_groups * 512 + g0 * 512], cols * 16);
            for (uint32_t g = g0; g < g1; g++) {
                const b2::TcGroup &G = tb.groups[job.grp_off + g];
                if (G.nb < 4 || G.nb > 8 || G.n_valid < 1 || G.n_valid > 16 / G.nb) return printf("bad group header\n"), 1;
                for (uint32_t row = 0; row < 128; row++) {
                    uint32_t c[32];
                    for (uint32_t col = 0; col < 32; col++) {
                        const uint32_t bc = (g - g0) * 32 + col;
                        uint32_t acc = 0;
                        for (uint32_t k = 0; k < slices * 16; k++)  // core matrices of 8 rows x 16 bytes, K neighbours one slice apart
                            acc += (uint32_t)A[(k / 16) * SLICE + (row / 8) * 128 + (row % 8) * 16 + k % 16] *
                                   B[(k / 16) * cols * 16 + (bc / 8) * 128 + (bc % 8) * 16 + k % 16];
                        c[col] = acc;
                    }
                    for (uint32_t o = 0; o < G.n_valid; o++)
                        for (uint32_t h = 0; h < 2; h++) {
                            const b2::TcOut &m = G.o[o];
                            const uint32_t *d = c + 2 * G.nb * o + h * G.nb;
                            for (uint32_t b = 0; b < G.nb; b++)
                                if (d[b] >= (1u << 22)) return printf("accumulator out of range\n"), 1;
                            const uint64_t got = residue(G.nb, d, m);
                            const size_t j = m.slot - 100;
                            if (j >= out_bits.size() || m.p != p[j]) return printf("bad output record\n"), 1;
                            seen[j] = 1;
                            u128 want = 0;
                            for (int i = 0; i < ni; i++) want += (u128)y[(size_t)i * 256 + 2 * row + h] * mat[j * ni + i];
                            if (got >= 2 * p[j] || got % p[j] != (uint64_t)(want % p[j]))
                                return printf("mismatch: ni=%d nb=%u row=%u half=%u out=%zu\n", ni, G.nb, row, h, j), 1;
                        }
                }
            }
        }
    }
    for (char s : seen)
        if (!s) return printf("an output was never produced\n"), 1;
    return 0;
}

int main(int argc, char **argv) {
    rng_state = argc > 1 ? strtoull(argv[1], nullptr, 10) : 1;
    int cases = 0;
    // 24 limbs, one of 60 bits and 23 of 40, and eight special primes of 60: ModDown, the first digit of ModUp and a later one
    std::vector<int> dn(1, 60), up0(16, 40), up1(1, 60), d0(8, 40), many;
    for (int i = 0; i < 23; i++) dn.push_back(40);
    for (int i = 0; i < 15; i++) up1.push_back(40);
    for (int i = 0; i < 8; i++) up0.push_back(60), up1.push_back(60);
    d0[0] = 60;
    for (int i = 0; i < 70; i++) many.push_back(i % 2 ? 60 : 36);  // more outputs than one job holds
    for (uint32_t parts : {1u, 2u, 5u, 16u})
        for (int ex = 0; ex < 2; ex++) {
            if (run_case(8, std::vector<int>(8, 60), dn, parts, ex) || run_case(8, d0, up0, parts, ex) || run_case(8, std::vector<int>(8, 40), up1, parts, ex) ||
                run_case(3, std::vector<int>(3, 50), many, parts, ex) || run_case(8, std::vector<int>(8, 60), many, parts, ex))
                return 1;
            cases += 5;
        }
    // every byte count, ragged inputs
    for (int bits = 17; bits <= 61; bits++)
        for (int ni = 1; ni <= 8; ni += bits & 1 ? 1 : 1 + bits % 3) {
            std::vector<int> in(ni, 17 + (bits * 11 + ni * 5) % 45);
            if (bits & 2) in[0] = 61;
            if (run_case(ni, in, {bits, bits, 61, bits, bits, bits, 17 + (bits * 7) % 45}, 1 + ni % 3, bits & 4)) return 1;
            cases++;
        }
    printf("ok %d\n", cases);
    return 0;
}
