// Host side of the order-3 kernel for data with missing calls (tensor3m.cu).
#pragma once

#include <vector>

#include "tensor3x.h"

namespace fiu {

constexpr int kPmJ = 64;  // j per pair item (32 per CTA)
constexpr int kPmG = 5;   // most groups of 16 l per item

// The l-tiles of the row of items whose first j is jf, as t3x_tiles with groups of 16 SNPs.
__host__ __device__ __forceinline__ int t3m_groups(int n, int jf) { return (n - ((jf + 1) & ~7) + 15) >> 4; }
__host__ __device__ __forceinline__ int t3m_tiles(int n, int jf) { return (t3m_groups(n, jf) + kPmG - 1) / kPmG; }
// First item of each i (host), [n + 1].
std::vector<long long> t3m_items(int n);
// Maps over the three-genotype layout (f4_prepare).
cudaError_t f4_missing_maps(F4Plan& f, int snps);
cudaError_t launch_tensor3m(const ScanWork& w, const F4Plan& f, const long long* item_begin, long long g0, long long g1,
                            const CandSink& sink, double est_margin, int* status, cudaStream_t s, int sms);

}  // namespace fiu
