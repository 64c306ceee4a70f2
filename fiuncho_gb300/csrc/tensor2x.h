// Host side of the order-2 pair kernel (tensor2x.cu).
#pragma once

#include <vector>

#include "internal.h"

namespace fiu {

constexpr int kP2I = 128;   // i per pair item (64 per CTA)
constexpr int kP2J = 120;   // j per item
constexpr int kP2Band = 4;  // i-tiles per band (512 i)

// Items of `count` owned i = first + step m (the whole scan: 0, 1, n - 1 of them): tiles of 128
// consecutive owned i in bands of 4, a band listed j-tile by j-tile from the one that holds its
// first i + 1.  Returns the first item of each band, [bands + 1]; tiles = i-tiles.
std::vector<long long> t2x_items(int n, long long count, long long first, long long step, int& tiles);
// e2m1 planes of `count` SNPs first + step m (1.0 where the genotype is g) in rows f4_row(m, g), `wpr`
// 16-byte chunks each; allocates, launches on s.
cudaError_t f4_ones_planes(const DevData& d, const F4Plan& f, int count, int first, int step, uint8_t*& planes,
                           cudaStream_t s);
// Maps over such planes: boxes of 128 B x 128 rows (the i operand) and x 120 rows (the j operand).
cudaError_t f4_map_a2(CUtensorMap* m, const F4Plan& f, const uint8_t* planes, int count);
cudaError_t f4_map_b2(CUtensorMap* m, const F4Plan& f, const uint8_t* planes, int count);

struct T2xRange {
    const long long* item_begin;  // first item of each band
    int tiles;
    const CUtensorMap *map_a, *map_b;
    int first, step;              // owned i = first + step m (layer_step's)
};
cudaError_t launch_tensor2x(const ScanWork& w, const F4Plan& f, const T2xRange& r, long long g0, long long g1,
                            const CandSink& sink, uint32_t* dump, const uint32_t* single, int* status, cudaStream_t s,
                            int sms);

}  // namespace fiu
