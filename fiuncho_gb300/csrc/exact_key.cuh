// The exact fixed-point key of one combination, by one warp, from the data set
// itself: lane c counts the cells c, c + 32, .. of the 3^K table (an AND and a
// popcount a word).  For kernels that meet so few combinations above their bound
// that keeping the tables' derivation beside the bound's would cost more.
#pragma once

#include "internal.h"

namespace fiu {

template <int K>
__device__ __noinline__ long long warp_exact_key(const DevData* dp, long long base_key, int c0, int c1, int c2,
                                                 int c3) {
    const DevData& d = *dp;
    const int lane = threadIdx.x & 31;
    constexpr int kCells = K == 4 ? 81 : 27;
    const size_t per_snp = 3 * (size_t)(d.cw + d.tw);
    const int cmb[4] = {c0, c1, c2, c3};
    long long key = 0;
    for (int cell = lane; cell < kCells; cell += 32) {
        const uint64_t* row[K];
        uint32_t cnt[2];
#pragma unroll
        for (int cls = 0; cls < 2; ++cls) {
            const int W = cls ? d.tw : d.cw;
            int r = cell;
#pragma unroll
            for (int t = K - 1; t >= 0; --t) {  // first SNP most significant
                row[t] = d.ref + (size_t)cmb[t] * per_snp + (cls ? 3 * (size_t)d.cw : 0) + (size_t)(r % 3) * W;
                r /= 3;
            }
            uint32_t n = 0;
#pragma unroll 4
            for (int w = 0; w < W; ++w) {
                uint64_t v = __ldg(row[0] + w);
#pragma unroll
                for (int t = 1; t < K; ++t) v &= __ldg(row[t] + w);
                n += (uint32_t)__popcll(v);
            }
            cnt[cls] = n;
        }
        key += __ldg(d.ftab + cnt[0]) + __ldg(d.ftab + cnt[1]) - __ldg(d.ftab + cnt[0] + cnt[1]);
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) key += __shfl_xor_sync(0xffffffffu, key, o);
    return key + base_key;
}

}  // namespace fiu
