// Device pieces of the top-N reduction shared by topn.cu and batch.cu:
// the total order of candidates, a one-CTA bitonic sort, and the FP64
// re-scoring of a combination from its recomputed full table.
#pragma once

#include "internal.h"

namespace fiu {

constexpr unsigned kSortCap = 8192;  // largest set sorted inside one CTA
constexpr int kSortThreads = 1024;

struct CandBetter {
    __device__ bool operator()(const Cand& a, const Cand& b) const {
        return a.key > b.key || (a.key == b.key && a.code < b.code);
    }
};

struct Scored {
    double v;
    unsigned long long code;
    long long key;
};

struct ScoredBetter {
    __device__ bool operator()(const Scored& a, const Scored& b) const {
        return a.v > b.v || (a.v == b.v && a.code < b.code);
    }
};

// Best-first bitonic sort of s[0..p) (p a power of two) by the whole block.
template <typename T, typename Better>
__device__ __forceinline__ void block_bitonic(T* s, unsigned p) {
    Better better;
    for (unsigned k = 2; k <= p; k <<= 1) {
        for (unsigned j = k >> 1; j > 0; j >>= 1) {
            for (unsigned i = threadIdx.x; i < p; i += blockDim.x) {
                const unsigned ixj = i ^ j;
                if (ixj > i) {
                    const T a = s[i], b = s[ixj];
                    const bool first_half = (i & k) == 0;
                    if (first_half ? better(b, a) : better(a, b)) {
                        s[i] = b;
                        s[ixj] = a;
                    }
                }
            }
            __syncthreads();
        }
    }
}

// Sorts n <= kSortCap elements best-first in one CTA (bitonic network in
// shared memory, padded to a power of two with `worst`).
template <typename T, typename Better>
__global__ void __launch_bounds__(kSortThreads) sort_block(T* data, unsigned n, T worst) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    T* s = reinterpret_cast<T*>(smem_raw);
    unsigned p = 1;
    while (p < n) p <<= 1;
    for (unsigned i = threadIdx.x; i < p; i += blockDim.x) s[i] = i < n ? data[i] : worst;
    __syncthreads();
    block_bitonic<T, Better>(s, p);
    for (unsigned i = threadIdx.x; i < n; i += blockDim.x) data[i] = s[i];
}

// ---- tables of given combinations and FP64 MI --------------------------------
// One warp per combination: for every cell (x_0..x_{K-1}) the lanes stride the
// words of the AND of the K rows, then reduce.  FP64 MI follows the definition
// H(X) + H(Y) - H(X,Y) with p = count / N, cells in index order.
__device__ inline void combo_tables(const DevData& d, int K, const int* c, int lane, uint32_t* cases_out,
                             uint32_t* ctrls_out, double* mi) {
    const size_t per_snp = 3 * (size_t)(d.cw + d.tw);
    int cells = 1;
    for (int t = 0; t < K; ++t) cells *= 3;
    const double N = (double)d.n_cases + (double)d.n_ctrls;
    double h_y = 0.0, h_x = 0.0, h_xy = 0.0;
    if (d.n_cases) h_y -= (d.n_cases / N) * log(d.n_cases / N);
    if (d.n_ctrls) h_y -= (d.n_ctrls / N) * log(d.n_ctrls / N);
    for (int cell = 0; cell < cells; ++cell) {
        uint32_t cnt[2];
        for (int cls = 0; cls < 2; ++cls) {
            const int W = cls ? d.tw : d.cw;
            const size_t roff = cls ? 3 * (size_t)d.cw : 0;
            uint32_t acc = 0;
            for (int w = lane; w < W; w += 32) {
                uint64_t v = ~0ull;
                int rem = cell;
                for (int t = K - 1; t >= 0; --t) {
                    const int x = rem % 3;
                    rem /= 3;
                    v &= __ldg(d.ref + (size_t)c[t] * per_snp + roff + (size_t)x * W + w);
                }
                acc += __popcll(v);
            }
            for (int o = 16; o; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
            cnt[cls] = acc;
        }
        if (cases_out && lane == 0) {
            cases_out[cell] = cnt[0];
            ctrls_out[cell] = cnt[1];
        }
        const double pc = cnt[0] / N, pt = cnt[1] / N, pa = pc + pt;
        if (cnt[0]) h_xy -= pc * log(pc);
        if (cnt[1]) h_xy -= pt * log(pt);
        if (cnt[0] + cnt[1]) h_x -= pa * log(pa);
    }
    if (mi) *mi = h_x + h_y - h_xy;
}

// ---- FP64 re-scoring of one combination by one CTA -----------------------------
// The value is combo_tables' to the last bit: the same terms, added in cell order.
// Bound by latency: a warp counts a cell at a time (one warp for all of them took
// the loads of 3^K cells one after the other), the logarithms go one to a thread
// (FP64 has two lanes a cycle and SM quarter; a warp that evaluates all of them
// pays 32 lanes for each), and what is left in sequence is one FP64 multiply-add a
// term.  Eighty combinations: order 3, 8 000 samples
// 19 us, order 4, 18 800 samples 35 us (before, with the sort and the copies: 0.25 to
// 0.74 ms of a search).
constexpr int kScoreThreads = 256, kScoreCells = 243;  // cells of a pass
struct ScoreShared {
    uint32_t cnt[2][kScoreCells];
    double p[3][kScoreCells], lg[3][kScoreCells];  // case, control and joint frequencies and their logarithms
};

// Samples of class cls in a cell (lanes over words), on every lane.
template <int K>
__device__ __forceinline__ uint32_t cell_count(const DevData& d, const int* c, int cell, int cls, int lane) {
    const int W = cls ? d.tw : d.cw;
    const size_t per_snp = 3 * (size_t)(d.cw + d.tw), off = cls ? 3 * (size_t)d.cw : 0;
    const uint64_t* row[K];
#pragma unroll
    for (int t = K - 1; t >= 0; --t) {
        row[t] = d.ref + (size_t)c[t] * per_snp + off + (size_t)(cell % 3) * W;
        cell /= 3;
    }
    uint32_t acc = 0;
#pragma unroll 4
    for (int w = lane; w < W; w += 32) {
        uint64_t v = __ldg(row[0] + w);
#pragma unroll
        for (int t = 1; t < K; ++t) v &= __ldg(row[t] + w);
        acc += __popcll(v);
    }
    return __reduce_add_sync(0xffffffffu, acc);
}

// The MI of combination c (K SNPs) on thread 0; every thread of the CTA (kScoreThreads) calls it.
__device__ inline double block_mi(const DevData& d, int K, const int* c, ScoreShared& sh) {
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    int cells = 1;
    for (int t = 0; t < K; ++t) cells *= 3;
    const double N = (double)d.n_cases + (double)d.n_ctrls;
    double h_y = 0.0, h_x = 0.0, h_xy = 0.0;
    if (tid == 0) {
        if (d.n_cases) h_y -= (d.n_cases / N) * log(d.n_cases / N);
        if (d.n_ctrls) h_y -= (d.n_ctrls / N) * log(d.n_ctrls / N);
    }
    for (int base = 0; base < cells; base += kScoreCells) {
        const int m = min(kScoreCells, cells - base);
        for (int q = warp; q < m; q += kScoreThreads / 32) {
            uint32_t n[2];
#pragma unroll
            for (int cls = 0; cls < 2; ++cls) {
                switch (K) {
                    case 1: n[cls] = cell_count<1>(d, c, base + q, cls, lane); break;
                    case 2: n[cls] = cell_count<2>(d, c, base + q, cls, lane); break;
                    case 3: n[cls] = cell_count<3>(d, c, base + q, cls, lane); break;
                    case 4: n[cls] = cell_count<4>(d, c, base + q, cls, lane); break;
                    case 5: n[cls] = cell_count<5>(d, c, base + q, cls, lane); break;
                    case 6: n[cls] = cell_count<6>(d, c, base + q, cls, lane); break;
                    case 7: n[cls] = cell_count<7>(d, c, base + q, cls, lane); break;
                    default: n[cls] = cell_count<8>(d, c, base + q, cls, lane); break;
                }
            }
            if (lane == 0) {
                sh.cnt[0][q] = n[0];
                sh.cnt[1][q] = n[1];
            }
        }
        __syncthreads();
        for (int e = tid; e < 3 * m; e += kScoreThreads) {
            const int k = e / m, q = e - k * m;
            const double pc = sh.cnt[0][q] / N, pt = sh.cnt[1][q] / N;
            const double p = k == 0 ? pc : k == 1 ? pt : pc + pt;
            sh.p[k][q] = p;
            sh.lg[k][q] = p > 0 ? log(p) : 0.0;
        }
        __syncthreads();
        if (tid == 0) {
            for (int q = 0; q < m; ++q) {
                if (sh.cnt[0][q]) h_xy -= sh.p[0][q] * sh.lg[0][q];
                if (sh.cnt[1][q]) h_xy -= sh.p[1][q] * sh.lg[1][q];
                if (sh.cnt[0][q] + sh.cnt[1][q]) h_x -= sh.p[2][q] * sh.lg[2][q];
            }
        }
        __syncthreads();
    }
    return h_x + h_y - h_xy;
}

}  // namespace fiu
