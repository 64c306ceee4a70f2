// The exact fixed-point key of one combination of order K (3 or 4), by one warp,
// from the data set itself, for a kernel that meets few combinations above its bound and
// would pay more for keeping the tables' derivation beside the bound's.
//
// Bound by the latency of its loads: lanes are (genotype x of the first SNP,
// word mod 8), so a step brings seven or ten words a lane, all independent, from
// rows read 64 bytes at a time, and the next step's are on their way while the 9
// or 27 cells of x are counted.  With a lane per cell instead (three of the 81 in turn, four
// loads in flight) a key of 18 800 samples of order 4 took 70 us.
//
// A launch whose candidate buffer has overflowed is made again in smaller pieces, so at order 4 no more keys
// are made for it (the least one is returned): 100 SNPs x 8 000 samples, all combinations tied, 644 -> 233 ms.
// At order 3 the check cost the searches without ties 0.6 % and gained the others 25 %: left out.
#pragma once

#include "internal.h"

namespace fiu {

template <int K>
__device__ __noinline__ long long warp_exact_key(const DevData* dp, long long base_key, int c0, int c1, int c2,
                                                  int c3, const unsigned* overflow) {
    // (one decision for the warp)
    if (K == 4 && __any_sync(0xffffffffu, *(volatile const unsigned*)overflow != 0))
        return (long long)0x8000000000000000ull;
    const DevData& d = *dp;
    const int lane = threadIdx.x & 31, x = lane >> 3, wl = lane & 7;  // x == 3: idle
    const size_t per_snp = 3 * (size_t)(d.cw + d.tw);
    constexpr int kRows = 1 + 3 * (K - 1), kCells = K == 4 ? 27 : 9;
    uint32_t cnt[kCells];  // cells (y, z[, g]): cases | controls << 16, each at most 65535
#pragma unroll
    for (int c = 0; c < kCells; ++c) cnt[c] = 0;
#pragma unroll 1
    for (int cls = 0; cls < 2; ++cls) {
        const int W = x < 3 ? (cls ? d.tw : d.cw) : 0;
        const size_t at = (cls ? 3 * (size_t)d.cw : 0) + wl;
        const uint64_t* r0 = d.ref + (size_t)c0 * per_snp + at + (size_t)x * W;
        const uint64_t* r1 = d.ref + (size_t)c1 * per_snp + at;
        const uint64_t* r2 = d.ref + (size_t)c2 * per_snp + at;
        const uint64_t* r3 = d.ref + (size_t)c3 * per_snp + at;
        const uint32_t one = cls ? 1u << 16 : 1u;
        uint64_t v[kRows];
        auto load = [&](int w) {
            v[0] = __ldg(r0 + w);
#pragma unroll
            for (int g = 0; g < 3; ++g) {
                v[1 + g] = __ldg(r1 + g * W + w);
                v[4 + g] = __ldg(r2 + g * W + w);
                if (K == 4) v[kRows - 3 + g] = __ldg(r3 + g * W + w);
            }
        };
        if (wl < W) load(0);
#pragma unroll 1
        for (int w = 0; w + wl < W; w += 8) {
            uint64_t u[kRows];
#pragma unroll
            for (int e = 0; e < kRows; ++e) u[e] = v[e];
            if (w + 8 + wl < W) load(w + 8);
#pragma unroll
            for (int y = 0; y < 3; ++y) {
                const uint64_t a = u[0] & u[1 + y];
#pragma unroll
                for (int z = 0; z < 3; ++z) {
                    const uint64_t b = a & u[4 + z];
                    if constexpr (K == 4) {
#pragma unroll
                        for (int g = 0; g < 3; ++g)
                            cnt[9 * y + 3 * z + g] += (uint32_t)__popcll(b & u[7 + g]) * one;
                    } else {
                        cnt[3 * y + z] += (uint32_t)__popcll(b) * one;
                    }
                }
            }
        }
    }
    __syncwarp();
    long long key = 0;
#pragma unroll
    for (int c = 0; c < kCells; ++c) {  // over the eight lanes of an x; each then takes the cells wl, wl + 8, ..
#pragma unroll
        for (int o = 4; o > 0; o >>= 1) cnt[c] += __shfl_xor_sync(0xffffffffu, cnt[c], o);
    }
#pragma unroll
    for (int s = 0; s < (kCells + 7) / 8; ++s) {
        uint32_t v = 0;
#pragma unroll
        for (int c = 0; c < 8; ++c)
            if (8 * s + c < kCells && wl == c) v = cnt[8 * s + c < kCells ? 8 * s + c : 0];
        const uint32_t a = v & 0xffffu, b = v >> 16;
        key += __ldg(d.ftab + a) + __ldg(d.ftab + b) - __ldg(d.ftab + a + b);  // 0 of an empty cell
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) key += __shfl_xor_sync(0xffffffffu, key, o);
    return key + base_key;
}

}  // namespace fiu
