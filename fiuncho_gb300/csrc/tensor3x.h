// Host side of the 4-bit operand layout and of the order-3 pair kernel (tensor3x.cu).
#pragma once

#include <vector>

#include "internal.h"

namespace fiu {

constexpr int kPxJ = 64;   // j per pair item (32 per CTA)
constexpr int kPxG = 15;   // most groups of 8 l per item

// The l-tiles of the row of items whose first j is jf: groups of 8 SNPs from
// the one holding jf + 1, split evenly into tiles of at most kPxG groups.
__host__ __device__ __forceinline__ int t3x_groups(int n, int jf) { return (n - ((jf + 1) & ~7) + 7) >> 3; }
__host__ __device__ __forceinline__ int t3x_tiles(int n, int jf) { return (t3x_groups(n, jf) + kPxG - 1) / kPxG; }

// Sizes of the 4-bit layout (host).
void f4_sizes(const DevData& d, F4Plan& f);
// Operand planes and bit rows of a data set (built once, on stream s), of 2 genotypes a SNP or of 3 (data
// with missing calls).
cudaError_t f4_prepare(const DevData& d, F4Plan& f, int genotypes, cudaStream_t s);
void f4_release(F4Plan& f);
cudaError_t f4_bit_map(CUtensorMap* m, const F4Plan& f, const uint32_t* bits, int rows, int box_rows);
// log2 of the control weight W when cases + W controls fit one FP32
// accumulator exactly (n_cases < W, n_cases + W n_ctrls < 2^24), else 0.
int f4_pack(int n_cases, int n_ctrls);
// First item of each i (host), [n + 1].
std::vector<long long> t3x_items(int n);

struct T3xRange {                        // where the items of a request are listed
    const long long* item_begin;         // first item of each i, [n + 1]
    const CUtensorMap* map_j;            // bit rows of the j operand
    const long long* jl_begin = nullptr; // a Distribution layer: first listed j of each i, [n + 1]
    const int* jlist = nullptr;          // ... and the listed j
};
cudaError_t launch_tensor3x(const ScanWork& w, const F4Plan& f, const T3xRange& r, long long g0, long long g1,
                            const CandSink& sink, uint32_t* dump, const uint32_t* single, const uint4* pairs,
                            double est_margin, int* status, cudaStream_t s, int sms, bool cores = false);
// The packed cores of all pairs and triples (F4Plan::tri, pairf), by the pair kernel over the order-3 items;
// waits for them.
cudaError_t f4_triples(const DevData& d, F4Plan& f, const long long* item_begin, long long items, const uint4* pairs,
                       cudaStream_t s, int sms);

// Order-4 pair kernel (tensor4x.cu): items (i, j, 32 k, up to 112 l).
constexpr int kP4K = 32;   // k per pair item (16 per CTA)
constexpr int kP4G = 7;    // most groups of 16 l per item
__host__ __device__ __forceinline__ int t4x_groups(int n, int kf) { return (n - ((kf + 1) & ~7) + 15) >> 4; }
__host__ __device__ __forceinline__ int t4x_tiles(int n, int kf) { return (t4x_groups(n, kf) + kP4G - 1) / kP4G; }
cudaError_t f4_order4_maps(F4Plan& f, int snps);
struct T4xRange {                   // where the items of a request are listed
    const long long* begin;         // first item of the pairs with second SNP j, [n + 1] (a layer: of each listed pair)
    const long long* per;           // items of a pair with second SNP j
    const CUtensorMap* map_k;       // bit rows of the k operand
    const int4* pinfo = nullptr;    // a Distribution layer: (i, j, first owned k) of each listed pair
    int n_pairs = 0;
};
cudaError_t launch_tensor4x(const ScanWork& w, const F4Plan& f, const T4xRange& r, long long g0, long long g1,
                            const CandSink& sink, uint32_t* dump, const uint32_t* single, const uint4* pairs,
                            int* status, cudaStream_t s, int sms);

}  // namespace fiu
