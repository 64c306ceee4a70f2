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

// Operand planes and bit rows of a data set (built once, on stream s).
cudaError_t f4_prepare(const DevData& d, F4Plan& f, cudaStream_t s);
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
                            float thr_f, float thr_q, int* status, cudaStream_t s, int sms);

}  // namespace fiu
