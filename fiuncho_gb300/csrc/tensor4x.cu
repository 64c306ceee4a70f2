// Order-4 contingency tables on CTA pairs with 4-bit operands.
//
// A cluster of two CTAs runs one GEMM per work item (i, j, 32 k, up to 112 l):
//     D[(k,x,y,z), (l,w)] = sum_s A[(k,x,y,z), s] B[(l,w), s]    (M 256, N <= 224)
// as the order-3 pair kernel does (tensor3x.cu: operand formats, roles,
// handover, scales).  CTA r builds the A rows of its 16 k -- the AND of the i, j
// and k bit rows, spread to nibbles -- and stages half r of the l rows.
//
// Accumulator rows are ordered (k / 4, x, y, z, k % 4).  A 16x256b load of a
// 16-row block gives a thread the rows (x, y = 0, 1) of one z and one k; it loads
// two column groups (16 l) and exchanges halves with the lane of the other z (16
// shuffles): each lane then holds all 16 cores of the combinations (k, l) and
// (k, l + 1) of one group.  The lane of z = 1 keeps its rows first, so its z
// runs 1, 0, 2: it reads the tables that depend on k's genotype in that order.
//
// Epilogue.  The 81 cells of both combinations follow slice by slice (genotype of
// l) from the packed cores and marginals in two-wide single precision: per l the
// tables of (i,j,l), (i,l), (j,l), l and per k those of (i,j,k), (i,k), (j,k), k
// are staged in shared memory one item ahead by two warps of their own; the
// triples (i,k,l), (j,k,l) and the pair (k,l) come as packed floats of (l, l + 1)
// side by side (F4Plan::tri, pairf; the triples are made by the order-3 pair
// kernel, whose accumulators they are).  The quartic bound (F4Bound4) rejects
// nearly all combinations of classes that are near in size (300 SNPs x 558/1 012:
// 5 500 of 3.3e8 pass it) and fewer the more one outweighs the other (0.2 % pass at
// 1 000/4 000, 9 % at 800/8 000, 73 % at 1 000/20 000); a group that has some left
// takes their logarithm estimate, whose error bound is proven (t4x_estimate), and what
// passes that gets the exact fixed-point key, so the kept set is the one of the
// exact key.  150 SNPs, exact keys right after the bound -> with the estimate
// between: 1 000/4 000 6.0 -> 4.8 ms, 800/8 000 53 -> 7.2, 1 000/20 000 643 -> 16
// (e4m3 kernel with the estimate for all: 7.3, 10.5 and 22).
//
// Measured (whole searches): 300 SNPs x 4 000/4 000 81.9 -> 33.6 ms, 300 x
// 558/1 012 60.0 -> 28.5 ms, against e4m3 operands, one CTA a tile, 243
// logarithms a combination (1 944 cycles a warp and SM quarter) and triples
// counted by POPC.  Without the evaluation the two take 22 and 13 ms; the
// evaluation of 64 combinations by a warp is 2 240 cycles of bound (81 x 2
// reciprocals 800, splitting the classes 650) and about 700 of derivation and takes
// 5 400 beside the builders, with two warps a quarter to hide latencies.  Tried:
// three warps a quarter on one combination at a time (104 registers) 40 ms; the
// slices in a loop (a third of the code) 32.8; three cells at a time through the
// bound 29.5.  Classes that do not share an accumulator (SPLIT): 100 SNPs x
// 9 000/9 800 6.7 -> 2.9 ms.
//
// Reference semantics: GenotypeTable::combine_and_popcnt for order 4
// (src/base/gt_popcnt.cpp:4-35) and MutualInformation::compute
// (src/base/mi_compute.cpp:16-41) over the combinations ThreadedSearch
// visits (include/fiuncho/ThreadedSearch.h:157-180) with one worker.
#include <algorithm>
#include <cmath>
#include <type_traits>

#include "elided4_prefix.cuh"
#include "exact_key.cuh"
#include "live.cuh"
#include "tensor3x.h"
#include "tensor_fp4.cuh"

namespace fiu {

constexpr int kYK = kP4K / 2;                       // k per CTA
constexpr int kYL = 16 * kP4G;                      // 112 l per item at most
constexpr int kYN = 2 * kYL;                        // columns of an accumulator region
constexpr int kYRow = kF4K / 2;                     // 128 bytes per operand row and stage
constexpr int kYBitRow = kF4K / 8;                  // 32 bytes per bit row and stage
constexpr int kYHalfG = 4;                          // items of at most 4 groups bring 64 l rows a CTA, others 112
template <bool SPLIT>
constexpr int kYStages = SPLIT ? 4 : 8;             // rings of the copies and of A, as in the order-3 kernel
template <bool SPLIT>
constexpr int kYAStages = SPLIT ? 3 : 4;
constexpr int kYSA = 8 * kYK * kYRow;               // 16 KB
constexpr int kYSB = kYN / 2 * kYRow;               // 14 KB: this CTA's half of the l rows
constexpr int kYSK = 2 * kYK * kYBitRow;            //  1 KB
constexpr int kYSI = 2 * kYBitRow;                  // 64 bytes of i, 64 of j (on 128-byte boundaries)
constexpr int kYBits = kYSK + 256;                  // the bit rows of a stage, behind all stages' B tiles
constexpr int kYColOne = 2 * kYN, kYColW = kYColOne + 16;
// 640 threads: copies, MMAs and two staging warps; two groups of four builders
// that take alternate stages; eight epilogue warps.  Registers a thread: 96 at
// launch, then 56 / 56 / 152 (3 x 56 + 2 x 152 <= 5 x 96).
constexpr int kYBuildWarps = 4, kYEpiWarps = 8;
constexpr int kYThreads = 32 * (4 + 2 * kYBuildWarps + kYEpiWarps);
constexpr int kYMeta = 16;                          // items in flight between the copies and the MMAs
// staged tables of an item: per l (ijl (x,y,w), il (x,w), jl (y,w), l (w); w = 0, 1, any), per k of
// this CTA (ijk, ik, jk, k cores, each twice: both halves of a pair; SPLIT: cases and controls
// beside each other, in both) and the item's threshold (key, estimate, bound)
template <bool SPLIT>
constexpr int kYTabL = 27 * kYL * (SPLIT ? 8 : 4);
constexpr int kYTabK = 18 * kYK * 8;
template <bool SPLIT>
constexpr int kYTab = kYTabL<SPLIT> + kYTabK + 16;
constexpr int kYStash = kYEpiWarps * ((kP4G + 1) / 2) * 4 * 32 * 16;  // 64 KB: (warp, its group, x, z, lane), 8 counts
template <bool SPLIT>
constexpr size_t kYSmem = 1024 + (size_t)kYStages<SPLIT> * (kYSB + kYBits) + (size_t)kYAStages<SPLIT> * kYSA +
                          2 * kYTab<SPLIT> + (SPLIT ? kYStash : 0);
static_assert(kYSmem<false> <= 227 * 1024 - 512 && kYSmem<true> <= 227 * 1024 - 512, "order-4 pair kernel shared memory");
static_assert(kYSA % 1024 == 0 && kYSB % 1024 == 0, "operand tiles on swizzle atoms");
static_assert(kYColW + 16 <= 512, "tensor memory columns");
static_assert(kYStages<false> < kYMeta, "an item has a stage at least");

// One item: (i, j, k0 ..), l-tile of ng groups of 16 from l0.
struct T4xItem {
    int i, j, k0, l0, ng;
};

// Item g; at is the walker's position (the items of one walker ascend): the
// second SNP j, or in a layer the listed pair.
template <bool LAYER>
__device__ __forceinline__ T4xItem t4x_item(const long long* __restrict__ begin, const long long* __restrict__ per,
                                            const int4* __restrict__ pinfo, int n_pairs, int n, int step,
                                            long long g, int& at) {
    if (at < 0) {
        int lo = 0, hi = (LAYER ? n_pairs : n) - 1;
        while (lo < hi) {
            const int mid = (lo + hi + 1) >> 1;
            if (__ldg(begin + mid) <= g) lo = mid;
            else hi = mid - 1;
        }
        at = lo;
    } else {
        while (__ldg(begin + at + 1) <= g) ++at;
    }
    T4xItem it;
    const unsigned rel = (unsigned)(g - __ldg(begin + at));
    unsigned q = rel;
    int k;
    if (LAYER) {
        const int4 f = __ldg(pinfo + at);
        it.i = f.x;
        it.j = f.y;
        k = f.z;
    } else {
        const unsigned pj = (unsigned)__ldg(per + at);
        it.j = at;
        it.i = (int)(rel / pj);
        q = rel - it.i * pj;
        k = at + 1;
    }
    for (;; k += kP4K * (LAYER ? step : 1)) {
        const unsigned nl = t4x_tiles(n, k);
        if (q < nl) {
            const int G = t4x_groups(n, k), a = G * (int)q / (int)nl, b = G * ((int)q + 1) / (int)nl;
            it.k0 = k;
            it.l0 = ((k + 1) & ~7) + 16 * a;
            it.ng = b - a;
            return it;
        }
        q -= nl;
    }
}

// Every other item of a walker is turned over: CTA r has the k of half 1 - r, in
// blocks of 4 from the last to the first (position kk holds k kk ^ 12), since in a
// tile on the diagonal the first k have the most l above them and an SM quarter
// keeps its block: with all items one way up the fullest quarter had 1.14 (300
// SNPs) to 1.43 (100) times the mean.
__device__ __forceinline__ int t4x_flip(unsigned item) { return item & 1 ? 12 : 0; }

// Columns the MMA of an item of ng groups multiplies (at least 64).
__device__ __forceinline__ int t4x_n(int ng) { return 32 * max(ng, 2); }

// Counts of both classes: packed (float), or beside each other (f2).
template <class T>
__device__ __forceinline__ T t4x_pk(uint32_t c, uint32_t t, float W) {
    if constexpr (sizeof(T) == 8) return f2_pack(u2f(c), u2f(t));
    else return fmaf(W, u2f(t), u2f(c));
}
template <class T>
__device__ __forceinline__ T t4x_pair(const uint4& v, int x, int y, float W) {
    const uint32_t c = x ? v.y : v.x, t = x ? v.w : v.z;
    return t4x_pk<T>(y ? c >> 16 : c & 0xffffu, y ? t >> 16 : t & 0xffffu, W);
}
// Core e of the triple whose pair-of-l entry is at row (F4Plan::tri).
template <class T>
__device__ __forceinline__ T t4x_tri(const float* row, int l, int e) {
    if constexpr (sizeof(T) == 8) return f4_ab(__ldg(reinterpret_cast<const uint32_t*>(row) + 8 * (l & 1) + e));
    else return __ldg(row + 2 * e + (l & 1));
}

// One 27-cell slice (one genotype of l) from its 8 cores c (x, y, z) and packed
// marginals: mij (x, y), mik (x, z), mil (x), mjk (y, z), mjl (y), mkl (z = 0, 1,
// any).  T is one value or two side by side; use(q, cell) gets cell (x, y, z) at
// q = (x*3+y)*3+z.
__device__ __forceinline__ f2 t4x_less(f2 a, f2 b, f2 c) { return f2_sub(f2_sub(a, b), c); }
__device__ __forceinline__ float t4x_less(float a, float b, float c) { return a - b - c; }
template <class T, class Use>
__device__ __forceinline__ void t4x_slice(const T (&c)[2][2][2], const T (&mij)[2][2], const T (&mik)[2][2],
                                          const T (&mil)[2], const T (&mjk)[2][2], const T (&mjl)[2],
                                          const T (&mkl)[3], Use&& use) {
    T a[2][3][3];  // cells of x = 0, 1
#pragma unroll
    for (int x = 0; x < 2; ++x) {
#pragma unroll
        for (int y = 0; y < 2; ++y) {
            a[x][y][0] = c[x][y][0];
            a[x][y][1] = c[x][y][1];
            a[x][y][2] = t4x_less(mij[x][y], c[x][y][0], c[x][y][1]);
        }
        const T k2 = t4x_less(mil[x], mik[x][0], mik[x][1]);
#pragma unroll
        for (int z = 0; z < 3; ++z) a[x][2][z] = t4x_less(z < 2 ? mik[x][z] : k2, a[x][0][z], a[x][1][z]);
#pragma unroll
        for (int y = 0; y < 3; ++y)
#pragma unroll
            for (int z = 0; z < 3; ++z) use((x * 3 + y) * 3 + z, a[x][y][z]);
    }
    const T j0 = t4x_less(mjl[0], mjk[0][0], mjk[0][1]), j1 = t4x_less(mjl[1], mjk[1][0], mjk[1][1]);
#pragma unroll
    for (int z = 0; z < 3; ++z) {
        const T m0 = z < 2 ? mjk[0][z] : j0, m1 = z < 2 ? mjk[1][z] : j1;
        use(18 + z, t4x_less(m0, a[0][0][z], a[1][0][z]));
        use(21 + z, t4x_less(m1, a[0][1][z], a[1][1][z]));
        use(24 + z, t4x_less(t4x_less(mkl[z], m0, m1), a[0][2][z], a[1][2][z]));
    }
}

// What a lane holds for its combinations: cores (x, y, z, w), the triples (i,k,l) (x, z, w) and
// (j,k,l) (y, z, w), the pair (k,l) (z, w); z in the lane's order.
template <class T>
struct T4xCores {
    T c[2][2][2][2], ik[2][2][2], jk[2][2][2], kl[2][2];
};

// The three slices of the combinations in v.  tabl(e) and tabk(e) return the
// staged entries (kYTabL and kYTabK order, z in the lane's order).
template <class T, class TL, class TK, class Use>
__device__ __forceinline__ void t4x_slices(const T4xCores<T>& v, TL&& tabl, TK&& tabk, Use&& use) {
#pragma unroll
    for (int w = 0; w < 3; ++w) {
        T c[2][2][2], mij[2][2], mik[2][2], mil[2], mjk[2][2], mjl[2], mkl[3];
#pragma unroll
        for (int x = 0; x < 2; ++x)
#pragma unroll
            for (int y = 0; y < 2; ++y) {
                mij[x][y] = tabl((x * 2 + y) * 3 + w);
#pragma unroll
                for (int z = 0; z < 2; ++z)
                    c[x][y][z] = w < 2 ? v.c[x][y][z][w & 1]
                                       : t4x_less(tabk((x * 2 + y) * 2 + z), v.c[x][y][z][0], v.c[x][y][z][1]);
            }
#pragma unroll
        for (int x = 0; x < 2; ++x) {
            mil[x] = tabl(12 + x * 3 + w);
            mjl[x] = tabl(18 + x * 3 + w);
#pragma unroll
            for (int z = 0; z < 2; ++z) {
                mik[x][z] = w < 2 ? v.ik[x][z][w & 1] : t4x_less(tabk(8 + x * 2 + z), v.ik[x][z][0], v.ik[x][z][1]);
                mjk[x][z] = w < 2 ? v.jk[x][z][w & 1] : t4x_less(tabk(12 + x * 2 + z), v.jk[x][z][0], v.jk[x][z][1]);
            }
        }
#pragma unroll
        for (int z = 0; z < 2; ++z) mkl[z] = w < 2 ? v.kl[z][w & 1] : t4x_less(tabk(16 + z), v.kl[z][0], v.kl[z][1]);
        mkl[2] = t4x_less(tabl(24 + w), mkl[0], mkl[1]);
        t4x_slice<T>(c, mij, mik, mil, mjk, mjl, mkl, [&](int q, T cell) { use(w, q, cell); });
    }
}

// The key estimate, in bits, of the combinations in v: of the two side by side, or (SPLIT) of one, in both
// halves.  It is within t4x_margin of the exact key: a cell's three terms a lg a + b lg b - s lg s are added up
// first (at most s in magnitude), so that the running sum stays below the samples.  For the groups in which a
// combination passes the quartic bound; out of line, with the cores through local memory, since its
// registers beside the bound's would slow every group down.  Bound by its 486 logarithms (3 888 cycles a warp and
// SM quarter), against 10 to 70 us for each exact key that it saves.
template <bool SPLIT>
__device__ __noinline__ f2 t4x_estimate(const T4xCores<f2>* v, const std::conditional_t<SPLIT, f2, float>* tl,
                                        const f2* tabk0, int zb, int pack) {
    const f2 tiny = f2_dup(9.5367431640625e-07f);  // 2^-20: x lg2(x + tiny) = 0 at x = 0
    const f2 inv_w = f2_dup(__uint_as_float((uint32_t)(127 - pack) << 23)), neg_w = f2_dup(-(float)(1 << pack));
    const f2 m23 = f2_dup(8388608.0f), neg_m23 = f2_dup(-8388608.0f);
    f2 kf = 0;
    t4x_slices<f2>(
        *v,
        [&](int e) {
            if constexpr (SPLIT) return tl[e * kYL];
            else return *reinterpret_cast<const f2*>(tl + e * kYL);
        },
        [&](int e) { return tabk0[(e ^ zb) * kYK]; },
        [&](int, int, f2 cell) {
            if constexpr (SPLIT) {
                float a, b, k, unused;
                f2_unpack(cell, a, b);
                f2_unpack(kf, k, unused);
                const float t2 = 9.5367431640625e-07f, s = a + b;
                k += fmaf(-s, t3_lg2(s + t2), fmaf(b, t3_lg2(b + t2), a * t3_lg2(a + t2)));
                kf = f2_dup(k);
            } else {
                auto lg = [](f2 x) {
                    float lo, hi;
                    f2_unpack(x, lo, hi);
                    return f2_pack(t3_lg2(lo), t3_lg2(hi));
                };
                const f2 b = f2_add(f2_fma_rz(cell, inv_w, m23), neg_m23), a = f2_fma(neg_w, b, cell), s = f2_add(a, b);
                const f2 ab = f2_fma(b, lg(f2_add(b, tiny)), f2_mul(a, lg(f2_add(a, tiny))));
                kf = f2_add(kf, f2_sub(ab, f2_mul(s, lg(f2_add(s, tiny)))));
            }
        });
    return kf;
}

// SPLIT: the exact key (without the base) of the combination in v, a lane each, from its cells, for groups with
// several left (no threshold yet, or many that tie with it): one a warp from the data set (warp_exact_key) takes
// 10 to 70 us at these classes' samples.  Bound by its gathers from the c ln c table.  100 copies of one SNP x
// 18 000 samples, all combinations tied: 1 920 -> 72 ms (e4m3 kernel 724); a layer of 100 SNPs, step 7, 7 000
// outputs 12.5 -> 8.7.  Classes that share an accumulator stay with warp_exact_key, which is short there: with this
// beside it their kernel's code came out 6 % slower (300 SNPs x 558/1 012 28.5 -> 30.4 ms).
__device__ __noinline__ long long t4x_key(const T4xCores<f2>* v, const f2* tl, const f2* tabk0, int zb,
                                          const DevData* d) {
    const uint32_t nc = (uint32_t)d->n_cases, nt = (uint32_t)d->n_ctrls;
    const long long* ftab = d->ftab;
    long long key = 0;
    t4x_slices<f2>(
        *v, [&](int e) { return tl[e * kYL]; }, [&](int e) { return tabk0[(e ^ zb) * kYK]; },
        [&](int, int, f2 cell) {
            float x, y;
            f2_unpack(cell, x, y);
            // (a lane without a combination holds anything: clamped)
            const uint32_t a = min(__float2uint_rn(x), nc), b = min(__float2uint_rn(y), nt);
            key += __ldg(ftab + a) + __ldg(ftab + b) - __ldg(ftab + a + b);
        });
    return key;
}
constexpr int kYGroupKeys = 4;  // combinations left of a group from which t4x_key makes all their keys

// ALL: every combination takes the exact path (a search's first units, before a threshold; dumps and
// digests).  Otherwise the bound comes first, a group with combinations above it gets their estimates
// (t4x_estimate), and the few that pass those are evaluated from the data set (warp_exact_key): the exact
// path's registers beside the bound's cost 20 % of the whole.
// SPLIT: classes that do not share an accumulator, as in the order-3 kernel: cases accumulate in one region
// and go to shared memory as 16-bit counts, controls in the other; one combination at a time is evaluated
// from both beside each other.
template <bool LAYER, bool ALL, bool SPLIT>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(kYThreads, 1)
    tensor4x_kernel(const __grid_constant__ CUtensorMap map_b, const __grid_constant__ CUtensorMap map_bh,
                    const __grid_constant__ CUtensorMap map_k,
                    const __grid_constant__ CUtensorMap map_i, const __grid_constant__ ScanWork w,
                    const __grid_constant__ CandSink sink, const long long* __restrict__ begin,
                    const long long* __restrict__ per, const int4* __restrict__ pinfo, int n_pairs, long long g0,
                    long long g1, int nw_c, int nw_t, int pack, const __grid_constant__ LiveMap map,
                    const __grid_constant__ F4Quartic quart,
                    uint32_t* dump, const uint32_t* __restrict__ single, const uint4* __restrict__ pairs,
                    const float* __restrict__ tri, const float* __restrict__ pairf, const int* __restrict__ row_p,
                    const int* __restrict__ row_q, int* status) {
    constexpr int kStages = kYStages<SPLIT>, kAStages = kYAStages<SPLIT>, kTab = kYTab<SPLIT>, kTabL = kYTabL<SPLIT>;
    using Tab = std::conditional_t<SPLIT, f2, float>;
    extern __shared__ uint8_t smraw[];
    __shared__ __align__(8) uint64_t full_t[kStages], empty[kStages], full_a[kAStages];
    __shared__ __align__(8) uint64_t acc_full[2], acc_empty[2], tab_full[2], tab_empty[2], done;
    __shared__ uint32_t tmem_base;
    __shared__ int item_ng[kYMeta];  // groups of the items in flight, for the MMA issuer
    __shared__ int abort_flag;
    uint8_t* sm = (uint8_t*)(((uintptr_t)smraw + 1023) & ~(uintptr_t)1023);  // stages: B half; the A tiles; k | i | j
    uint8_t* sma = sm + kStages * kYSB;
    uint8_t* smk = sma + kAStages * kYSA;
    uint8_t* tabs = smk + kStages * kYBits;
    uint4* stash = reinterpret_cast<uint4*>(tabs + 2 * kTab);
    volatile int* abort = &abort_flag;
    const int n = w.d.snps, kstep = LAYER ? layer_step(w.dist_step, w.d.snps) : 1;
    const int tid = threadIdx.x, lane = tid & 31;
    const int warp = __shfl_sync(0xffffffffu, tid >> 5, 0);  // warp-uniform for the compiler too
    const int ksteps = ((nw_c + 3) >> 2) + ((nw_t + 3) >> 2);  // stages of 256 samples
    const uint32_t rank = cluster_rank();  // 0 issues the MMAs
    const long long cid = cluster_id(), ncl = cluster_count();

    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_base)),
                     "r"(512));
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;");
    }
    if (tid == 0) {
        auto init = [](uint64_t* b, int count) {
            asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(b)), "r"(count));
        };
        for (int s = 0; s < kStages; ++s) {
            init(&full_t[s], 1);
            init(&empty[s], 1);
        }
        for (int s = 0; s < kAStages; ++s) init(&full_a[s], 2 * kYBuildWarps);
        for (int b = 0; b < 2; ++b) {
            init(&acc_full[b], 1);
            init(&acc_empty[b], 2 * kYEpiWarps);
            init(&tab_full[b], 2);
            init(&tab_empty[b], kYEpiWarps);
        }
        init(&done, 1);
        asm volatile("fence.mbarrier_init.release.cluster;");
        abort_flag = 0;
    }
    asm volatile("tcgen05.fence::before_thread_sync;");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;");
    const uint32_t tmem = tmem_base;
    if (warp >= 4 && warp < 8) f4_fill_scales<16>(tmem, warp & 3, kYColOne, kYColW, pack);
    asm volatile("tcgen05.fence::before_thread_sync;");
    __syncthreads();
    cluster_sync_all();  // both CTAs' barriers and scales exist before either signals the other
    asm volatile("tcgen05.fence::after_thread_sync;");
    bool ok = true;

    if (warp < 4) {
        asm volatile("setmaxnreg.dec.sync.aligned.u32 56;");
        if (warp == 0) {
            // ---------------------------------------------------------------- TMA producer (both CTAs)
            if (g0 + cid < g1 && elect_one()) {
                unsigned s = 0, par = 1;  // stage and the parity its last release has (first round: free)
                unsigned step = 0, item = 0;
                int at = -1;
                T4xItem it = t4x_item<LAYER>(begin, per, pinfo, n_pairs, n, kstep, g0 + cid, at);
                for (long long g = g0 + cid; g < g1 && ok; g += ncl) {
                    // this CTA's first k row (in a layer the owned k are consecutive residue-ordered rows;
                    // rows past the last owned one are loaded too and ignored by the epilogue)
                    const int krow =
                        2 * ((LAYER ? residue_row(it.k0, kstep, n) : it.k0) + kYK * ((int)rank ^ (int)(item & 1)));
                    const int brow = 2 * it.l0 + t4x_n(it.ng) / 2 * (int)rank, irow = 2 * it.i, jrow = 2 * it.j;
                    const bool half = it.ng <= kYHalfG;
                    item_ng[item++ % kYMeta] = it.ng;
                    T4xItem nx = it;
                    for (int ks = 0; ks < ksteps; ++ks) {
                        if (!t3_wait_cl(smem_u32(&empty[s]), par, abort)) {
                            ok = false;
                            break;
                        }
                        const uint32_t st = smem_u32(sm + s * kYSB), bar = smem_u32(&full_t[s]);
                        const uint32_t sk = smem_u32(smk + s * kYBits);
                        asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar),
                                     "r"((uint32_t)((half ? 16 * kYHalfG * kYRow : kYSB) + kYSK + 2 * kYSI))
                                     : "memory");
                        t3_tma(sk, &map_k, kYBitRow * ks, krow, bar);
                        t3_tma(sk + kYSK, &map_i, kYBitRow * ks, irow, bar);
                        t3_tma(sk + kYSK + 128, &map_i, kYBitRow * ks, jrow, bar);
                        t3_tma(st, half ? &map_bh : &map_b, kYRow * ks, brow, bar);
                        if (step < kStages) ++step;
                        if (++s == kStages) {
                            s = 0;
                            par ^= 1;
                        }
                        // the next item's place is looked up while this item's copies are in flight
                        if (ks == 0 && g + ncl < g1)
                            nx = t4x_item<LAYER>(begin, per, pinfo, n_pairs, n, kstep, g + ncl, at);
                    }
                    it = nx;
                }
                // no copy may be in flight when the CTA exits: the last use of every stage used
                for (unsigned q = 0; q < step; ++q) {
                    // stage q was last filled in the round before `par` names, or in this one when q < s
                    if (!t3_drain(smem_u32(&full_t[q]), q < s ? par ^ 1 : par)) ok = false;
                }
            }
            __syncwarp();
        } else if (warp == 1) {
            // ---------------------------------------------------------------- MMA issuer (CTA 0)
            if (rank == 0 && elect_one()) {
                ok = f4_pair_issue<SPLIT, kAStages, kYSA, kStages, kYSB, kYN, kYColOne, kYColW>(
                    (g1 - g0 - cid + ncl - 1) / ncl, smem_u32(sma), smem_u32(sm), smem_u32(&full_a[0]),
                    smem_u32(&empty[0]), smem_u32(&acc_full[0]), smem_u32(&acc_empty[0]), tmem, nw_c, nw_t, abort,
                    [&](unsigned item) { return t4x_n(item_ng[item % kYMeta]); });
                commit_pair(smem_u32(&done));
                // neither CTA releases shared or tensor memory before the pair's MMAs are
                // done (CTA 1 waits once its own work is over, below)
                if (!t3_drain_cl(smem_u32(&done), 0)) ok = false;
            }
            __syncwarp();
        } else {
            // ---------------------------------------------------------------- table staging (both CTAs)
            const int t = tid - 64;  // 0 .. 63
            const float W = (float)(1u << pack);
            const Tab ntot = t4x_pk<Tab>(w.d.n_cases, w.d.n_ctrls, W);
            const uint4* single4 = reinterpret_cast<const uint4*>(single);
            unsigned item = 0;
            int at = -1;
            for (long long g = g0 + cid; g < g1 && ok; g += ncl, ++item) {
                const T4xItem it = t4x_item<LAYER>(begin, per, pinfo, n_pairs, n, kstep, g, at);
                const unsigned buf = item & 1;
                if (item >= 2 && !t3_wait(smem_u32(&tab_empty[buf]), ((item >> 1) - 1) & 1, abort)) {
                    ok = false;
                    break;
                }
                // the threshold of this item (the pairs take turns at raising the live one)
                if (sink.hist && rank == 0 && warp == 2 && item > 0 && (item < 3 || ((item + cid) & 7) == 0))
                    live_update(sink, lane);
                if (t == 0) {
                    const long long thr = sink.hist ? *(volatile long long*)sink.live : sink.thr;
                    float est, bound;
                    live_tests(map, thr, est, bound);
                    uint8_t* o = tabs + buf * kTab + kTabL + kYTabK;
                    *reinterpret_cast<long long*>(o) = thr;
                    *reinterpret_cast<float2*>(o + 8) = make_float2(bound, est);
                }
                Tab* tl = reinterpret_cast<Tab*>(tabs + buf * kTab);
                f2* tk = reinterpret_cast<f2*>(tabs + buf * kTab + kTabL);
                const int i = it.i, j = it.j;
                const uint4 pij4 = __ldg(pairs + pair_index(i, j, n));
                const uint4 si = __ldg(single4 + i), sj = __ldg(single4 + j);
                const float* tij = tri + 16ll * (__ldg(row_q + i) + __ldg(row_p + j));
                for (int ll = t; ll < 16 * it.ng; ll += 64) {
                    const int l = it.l0 + ll;
                    Tab* o = tl + ll;
                    if (l < n && l > j) {
                        const float* e3 = tij + 16ll * (l >> 1);
                        const uint4 pi = __ldg(pairs + pair_index(i, l, n)), pj = __ldg(pairs + pair_index(j, l, n));
                        const uint4 sl = __ldg(single4 + l);
                        // w = 0, 1 and what is left of the marginal ("any" entries hold what is left after
                        // genotypes 0 and 1, so the slice of genotype 2 reads its marginals as the others do)
                        auto put = [&](int e, Tab a, Tab b, Tab all) {
                            o[e * kYL] = a;
                            o[(e + 1) * kYL] = b;
                            o[(e + 2) * kYL] = t4x_less(all, a, b);
                        };
#pragma unroll
                        for (int xy = 0; xy < 4; ++xy)
                            put(3 * xy, t4x_tri<Tab>(e3, l, 2 * xy), t4x_tri<Tab>(e3, l, 2 * xy + 1),
                                t4x_pair<Tab>(pij4, xy >> 1, xy & 1, W));
#pragma unroll
                        for (int x = 0; x < 2; ++x) {
                            put(12 + 3 * x, t4x_pair<Tab>(pi, x, 0, W), t4x_pair<Tab>(pi, x, 1, W),
                                t4x_pk<Tab>(x ? si.y : si.x, x ? si.w : si.z, W));
                            put(18 + 3 * x, t4x_pair<Tab>(pj, x, 0, W), t4x_pair<Tab>(pj, x, 1, W),
                                t4x_pk<Tab>(x ? sj.y : sj.x, x ? sj.w : sj.z, W));
                        }
                        put(24, t4x_pk<Tab>(sl.x, sl.z, W), t4x_pk<Tab>(sl.y, sl.w, W), ntot);
                    } else {
#pragma unroll
                        for (int e = 0; e < 27; ++e) o[e * kYL] = 0;
                    }
                }
                if (t < kYK) {
                    const int k = layer_snp(it.k0, kstep, kYK * ((int)rank ^ (int)(item & 1)) + t);
                    auto put = [&](int e, Tab v) {
                        if constexpr (SPLIT) tk[e * kYK + t] = v;
                        else tk[e * kYK + t] = f2_dup(v);
                    };
                    if (k < n) {
                        const float* e3 = tij + 16ll * (k >> 1);
                        const uint4 pi = __ldg(pairs + pair_index(i, k, n)), pj = __ldg(pairs + pair_index(j, k, n));
                        const uint4 sk = __ldg(single4 + k);
#pragma unroll
                        for (int e = 0; e < 8; ++e) put(e, t4x_tri<Tab>(e3, k, e));
#pragma unroll
                        for (int e = 0; e < 4; ++e) {
                            put(8 + e, t4x_pair<Tab>(pi, e >> 1, e & 1, W));
                            put(12 + e, t4x_pair<Tab>(pj, e >> 1, e & 1, W));
                        }
                        put(16, t4x_pk<Tab>(sk.x, sk.z, W));
                        put(17, t4x_pk<Tab>(sk.y, sk.w, W));
                    } else {
#pragma unroll
                        for (int e = 0; e < 18; ++e) put(e, 0);
                    }
                }
                __syncwarp();
                if (lane == 0)
                    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(&tab_full[buf])) : "memory");
            }
        }
    } else if (warp < 12) {
        asm volatile("setmaxnreg.dec.sync.aligned.u32 56;");
        // ---------------------------------------------------------------- A builders (both CTAs)
        // thread: 16-byte chunk c (32 samples) of the k rows rg and rg + 16 of every second stage
        const int t = (tid - 128) & (32 * kYBuildWarps - 1), c = t & 7, rg = t >> 3;
        const uint32_t full0 = cluster_addr(smem_u32(&full_a[0]), 0);
        // A row (kk / 4, x, y, z, kk % 4) of staged row (kk, z) = rg + 16 u: u + 1 is 64 rows on (back when turned over)
        const int kk = rg >> 1, z = rg & 1, m0 = 32 * (kk >> 2) + 4 * z + (kk & 3);
        const int dst0 = m0 * kYRow + ((c ^ (m0 & 7)) << 4);
        unsigned s = 0, par = 0, sa = 0;                  // copy stage, A stage
        unsigned se = kStages - kAStages, pe = 1;       // the stage whose MMAs free this A stage
        bool mine = warp < 8;
        int turn = 0;  // an item turned over: block b is block 3 - b
        for (long long g = g0 + cid; g < g1 && ok; g += ncl, turn ^= 96 * kYRow) {
            for (int ks = 0; ks < ksteps; ++ks, mine = !mine) {
                if (mine) {
                    if (!t3_wait(smem_u32(&full_t[s]), par, abort)) {
                        ok = false;
                        break;
                    }
                    const uint32_t* sK = reinterpret_cast<const uint32_t*>(smk + s * kYBits);
                    const uint32_t* sI = sK + kYSK / 4 + c;
                    const uint32_t k0 = sK[rg * 8 + c], k1 = sK[(rg + 16) * 8 + c];
                    const uint32_t i0 = sI[0], i1 = sI[8], j0 = sI[32], j1 = sI[40];
                    if (!t3_wait_cl(smem_u32(&empty[se]), pe, abort)) {
                        ok = false;
                        break;
                    }
                    uint8_t *dst = sma + sa * kYSA + (dst0 ^ turn), *dst2 = sma + sa * kYSA + (dst0 ^ turn ^ 64 * kYRow);
#pragma unroll
                    for (int xy = 0; xy < 4; ++xy) {
                        const uint32_t ij = (xy & 2 ? i1 : i0) & (xy & 1 ? j1 : j0);
                        *reinterpret_cast<uint4*>(dst + 8 * xy * kYRow) = f4_expand_a(ij, k0);
                        *reinterpret_cast<uint4*>(dst2 + 8 * xy * kYRow) = f4_expand_a(ij, k1);
                    }
                    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
                    __syncwarp();
                    if (lane == 0) arrive_cl(full0 + 8 * sa);
                }
                if (++s == kStages) {
                    s = 0;
                    par ^= 1;
                }
                if (++se == kStages) {
                    se = 0;
                    pe ^= 1;
                }
                if (++sa == kAStages) sa = 0;
            }
        }
    } else {
        asm volatile("setmaxnreg.inc.sync.aligned.u32 152;");
        // ---------------------------------------------------------------- epilogue (both CTAs)
        const int q = warp & 3, hh = (warp - 12) >> 2;  // lane quarter (4 k); its two warps take alternate groups
        const int zb = lane >> 4, kk0 = 4 * q + ((lane >> 2) & 3), lc = 2 * (lane & 3);
        const uint32_t wmask = (1u << pack) - 1u;
        uint4* mine = stash + (warp - 12) * ((kP4G + 1) / 2) * 128 + lane;  // written and read by this warp only
        unsigned item = 0;
        int at = -1;
        for (long long g = g0 + cid; g < g1 && ok; g += ncl, ++item) {
            const T4xItem it = t4x_item<LAYER>(begin, per, pinfo, n_pairs, n, kstep, g, at);
            const unsigned buf = item & 1, ph = (item >> 1) & 1;
            const int gi0 = (hh + item) & 1;  // the odd group of an item goes to either warp in turn
            const int kk = kk0 ^ t4x_flip(item), k = layer_snp(it.k0, kstep, kYK * ((int)rank ^ (int)(item & 1)) + kk);
            const bool k_ok = k < n;
            // entries of the rows (i, k), (j, k) and k, in units of 16 bytes
            const int rp = k_ok ? __ldg(row_p + k) : 0;
            const uint4* tik = reinterpret_cast<const uint4*>(tri) + 4 * ((long long)__ldg(row_q + it.i) + rp);
            const uint4* tjk = reinterpret_cast<const uint4*>(tri) + 4 * ((long long)__ldg(row_q + it.j) + rp);
            const uint4* tkl = reinterpret_cast<const uint4*>(pairf) + 2 * (long long)rp;
            // accumulators of one x in group gi: 8 group + 4 w + 2 y (l) and + 1 (l + 1)
            auto acc_ld = [&](int region, int x, int gi, uint32_t (&r)[16]) {
                asm volatile(
                    "tcgen05.ld.sync.aligned.16x256b.x4.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, "
                    "[%16];"
                    : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
                      "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]),
                      "=r"(r[15])
                    : "r"(tmem + ((uint32_t)(32 * q + 16 * x) << 16) + (uint32_t)(kYN * region + 32 * gi)));
                asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
            };
            // SPLIT: the same as 16-bit counts (l | l + 1 << 16), this lane's z first and then the other z,
            // components 2 w + y
            auto acc_counts = [&](int region, int x, int gi, uint4& own, uint4& other) {
                uint32_t r[16], o[8];
                acc_ld(region, x, gi, r);
#pragma unroll
                for (int e = 0; e < 8; ++e)
                    o[e] = __byte_perm(__float_as_uint(__uint_as_float(r[2 * e]) + 8388608.0f),
                                       __float_as_uint(__uint_as_float(r[2 * e + 1]) + 8388608.0f), 0x5410);
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                    (&own.x)[e] = zb ? o[4 + e] : o[e];
                    (&other.x)[e] = __shfl_xor_sync(0xffffffffu, zb ? o[e] : o[4 + e], 16);
                }
            };
            if (SPLIT) {
                // case counts to shared memory; their region is then free
                if (!t3_wait_cl(smem_u32(&acc_full[0]), item & 1, abort)) {
                    ok = false;
                    break;
                }
                asm volatile("tcgen05.fence::after_thread_sync;");
#pragma unroll 1
                for (int gi = gi0; gi < it.ng; gi += 2)
#pragma unroll
                    for (int x = 0; x < 2; ++x) {
                        uint4 o[2];
                        acc_counts(0, x, gi, o[0], o[1]);
                        mine[(2 * (gi & ~1) + 2 * x) * 32] = o[0];
                        mine[(2 * (gi & ~1) + 2 * x + 1) * 32] = o[1];
                    }
                asm volatile("tcgen05.fence::before_thread_sync;");
                __syncwarp();
                if (lane == 0) arrive_cl(cluster_addr(smem_u32(&acc_empty[0]), 0));
            }
            if (!t3_wait(smem_u32(&tab_full[buf]), ph, abort) ||
                !t3_wait_cl(smem_u32(&acc_full[SPLIT ? 1 : buf]), SPLIT ? item & 1 : ph, abort)) {
                ok = false;
                break;
            }
            asm volatile("tcgen05.fence::after_thread_sync;");
            const Tab* tabl0 = reinterpret_cast<const Tab*>(tabs + buf * kTab);
            const f2* tabk0 = reinterpret_cast<const f2*>(tabs + buf * kTab + kTabL) + kk;
            const long long thr = *reinterpret_cast<const long long*>(tabs + buf * kTab + kTabL + kYTabK);
            const float thr_q = *reinterpret_cast<const float*>(tabs + buf * kTab + kTabL + kYTabK + 8);
            auto thr_f = [&] { return reinterpret_cast<const float*>(tabs + buf * kTab + kTabL + kYTabK)[3]; };
            // per-k entries: the index's last bit is z
            auto tabk = [&](int e) { return tabk0[(e ^ zb) * kYK]; };
            auto exact_append = [&](int src, int u, int lu) {  // a survivor of lane src
                const int cmb[4] = {it.i, it.j, __shfl_sync(0xffffffffu, k, src), __shfl_sync(0xffffffffu, lu, src) + u};
                const long long key = warp_exact_key<4>(&w.d, w.base_key, cmb[0], cmb[1], cmb[2], cmb[3], sink.overflow);
                if (lane == 0 && key >= thr) live_append(sink, key, pack_code(cmb, 4, w.bits));
            };
            // the exact path of combination (i, j, k, lu), whose slices walk(use) makes: use(w, cell index,
            // cases, controls)
            auto every = [&](int lu, bool want, auto&& walk) {
                const int cmb[4] = {it.i, it.j, k, lu};
                long long key = w.base_key;
                uint32_t* o = nullptr;
                if (want) {
                    // owned prefix ordinal of (i, j, k): rank offset + m * step
                    if (dump)
                        o = dump + ((size_t)((triple_index(it.i, it.j, k, n) - w.dist_offset) / w.dist_step) * n +
                                    cmb[3]) * 162;
                    const unsigned gt = blockIdx.x * blockDim.x + threadIdx.x;
                    if (sink.digest && gt < sink.dscratch_threads) o = sink.dscratch + (size_t)gt * 162;
                    const uint32_t nc = (uint32_t)w.d.n_cases, nt = (uint32_t)w.d.n_ctrls;
                    walk([&](int sw, int c, uint32_t ua, uint32_t ub) {
                        const uint32_t a = min(ua, nc), b = min(ub, nt);
                        key += __ldg(w.d.ftab + a) + __ldg(w.d.ftab + b) - __ldg(w.d.ftab + a + b);
                        if (o) {
                            const int z = c % 3, zt = z < 2 ? z ^ zb : 2;
                            o[(c - z + zt) * 3 + sw] = a;
                            o[81 + (c - z + zt) * 3 + sw] = b;
                        }
                    });
                }
                if (sink.digest) dg_warp_add(sink.digest, want && o ? dg_table(cmb, 4, n, o, 81) : 0ull);
                if (want && key >= thr) live_append(sink, key, pack_code(cmb, 4, w.bits));
            };
            if constexpr (SPLIT) {
                // (i,k,l), (j,k,l) and (k,l) of combination u of group gi: words of w = 0, 1
                uint2 ik[2][2], jk[2][2], kl[2];
                auto load = [&](int gi, int u) {
                    const int l = it.l0 + 16 * gi + 8 * zb + lc + u;
                    const bool any = gi < it.ng && k_ok && l < n && l > k;
                    auto ld = [&](const uint4* p, int e, uint2& o) {
                        o = make_uint2(0, 0);
                        if (any) o = __ldg(reinterpret_cast<const uint2*>(p) + e);
                    };
#pragma unroll
                    for (int z = 0; z < 2; ++z) {
#pragma unroll
                        for (int x = 0; x < 2; ++x) {
                            ld(tik, 4 * l + 2 * x + (z ^ zb), ik[x][z]);
                            ld(tjk, 4 * l + 2 * x + (z ^ zb), jk[x][z]);
                        }
                        ld(tkl, 2 * l + (z ^ zb), kl[z]);
                    }
                };
                load(gi0, 0);
#pragma unroll 1
                for (int gi = gi0; gi < it.ng; gi += 2) {
                    const int ll = 16 * gi + 8 * zb + lc, l = it.l0 + ll;
                    const bool v0 = k_ok && l < n && l > k, v1 = k_ok && l + 1 < n && l + 1 > k;
                    const unsigned m0 = __ballot_sync(0xffffffffu, v0), m1 = __ballot_sync(0xffffffffu, v1);
                    if (!(m0 | m1)) {
                        load(gi + 2, 0);
                        continue;
                    }
                    if (sink.evaluated && lane == 0)
                        atomicAdd(sink.evaluated, (unsigned long long)(__popc(m0) + __popc(m1)));
                    uint4 t[2][2];  // control counts (x, z)
#pragma unroll
                    for (int x = 0; x < 2; ++x) acc_counts(1, x, gi, t[x][0], t[x][1]);
#pragma unroll 1
                    for (int u = 0; u < 2; ++u) {
                        auto cores = [&](T4xCores<f2>& v) {  // of combination u, whose triples and pair are in ik, jk, kl
#pragma unroll
                            for (int x = 0; x < 2; ++x)
#pragma unroll
                                for (int z = 0; z < 2; ++z) {
                                    const uint4 c = mine[(2 * (gi & ~1) + 2 * x + z) * 32];
#pragma unroll
                                    for (int e = 0; e < 4; ++e)
                                        v.c[x][e & 1][z][e >> 1] = f4_ab((&c.x)[e], (&t[x][z].x)[e], u);
                                    v.ik[x][z][0] = f4_ab(ik[x][z].x);
                                    v.ik[x][z][1] = f4_ab(ik[x][z].y);
                                    v.jk[x][z][0] = f4_ab(jk[x][z].x);
                                    v.jk[x][z][1] = f4_ab(jk[x][z].y);
                                }
#pragma unroll
                            for (int z = 0; z < 2; ++z) {
                                v.kl[z][0] = f4_ab(kl[z].x);
                                v.kl[z][1] = f4_ab(kl[z].y);
                            }
                        };
                        T4xCores<f2> v;
                        cores(v);
                        load(u ? gi + 2 : gi, u ^ 1);  // the next one's, on their way while this one is evaluated
                        const Tab* tl = tabl0 + ll + u;
                        auto tabl = [&](int e) { return tl[e * kYL]; };
                        const bool want = u ? v1 : v0;
                        if constexpr (!ALL) {
                            F4Bound4AB bd(quart);
                            t4x_slices<f2>(v, tabl, tabk, [&](int, int, f2 cell) { bd.one(cell); });
                            unsigned sv = __ballot_sync(0xffffffffu, want && bd.acc >= thr_q);
                            if (sv) {
                                load(gi, u);  // (the next one's triples have taken the place of this one's)
                                T4xCores<f2> again;
                                cores(again);
                                float est, unused;
                                f2_unpack(t4x_estimate<true>(&again, tl, tabk0, zb, pack), est, unused);
                                sv &= __ballot_sync(0xffffffffu, est >= thr_f());
                                if (__popc(sv) >= kYGroupKeys) {
                                    const int cmb[4] = {it.i, it.j, k, l + u};
                                    const long long key = t4x_key(&again, tl, tabk0, zb, &w.d) + w.base_key;
                                    if ((sv >> lane & 1) && key >= thr) live_append(sink, key, pack_code(cmb, 4, w.bits));
                                    sv = 0;
                                }
                                for (; sv; sv &= sv - 1) exact_append(__ffs(sv) - 1, u, l);
                                load(u ? gi + 2 : gi, u ^ 1);
                            }
                        } else {
                            every(l + u, want, [&](auto&& use) {
                                t4x_slices<f2>(v, tabl, tabk, [&](int sw, int c, f2 cell) {
                                    float a, b;
                                    f2_unpack(cell, a, b);
                                    use(sw, c, __float2uint_rn(a), __float2uint_rn(b));
                                });
                            });
                        }
                    }
                }
            } else {
                // (i,k,l), (j,k,l) and (k,l) of group gi: 16 bytes hold one (x, z) and both w
                T4xCores<f2> v;
                auto load = [&](int gi) {
                    const int l = it.l0 + 16 * gi + 8 * zb + lc, m = l >> 1;
                    const bool any = gi < it.ng && k_ok && l < n && l + 1 > k;
                    auto ld = [&](const uint4* p, f2 (&o)[2]) {
                        uint4 x = make_uint4(0, 0, 0, 0);
                        if (any) x = __ldg(p);
                        o[0] = f2_pack(__uint_as_float(x.x), __uint_as_float(x.y));
                        o[1] = f2_pack(__uint_as_float(x.z), __uint_as_float(x.w));
                    };
#pragma unroll
                    for (int x = 0; x < 2; ++x)
#pragma unroll
                        for (int z = 0; z < 2; ++z) {
                            ld(tik + 4 * m + 2 * x + (z ^ zb), v.ik[x][z]);
                            ld(tjk + 4 * m + 2 * x + (z ^ zb), v.jk[x][z]);
                        }
#pragma unroll
                    for (int z = 0; z < 2; ++z) ld(tkl + 2 * m + (z ^ zb), v.kl[z]);
                };
                load(gi0);
#pragma unroll 1
                for (int gi = gi0; gi < it.ng; gi += 2) {
                    const int ll = 16 * gi + 8 * zb + lc, l = it.l0 + ll;
                    const bool v0 = k_ok && l < n && l > k, v1 = k_ok && l + 1 < n && l + 1 > k;
                    const unsigned m0 = __ballot_sync(0xffffffffu, v0), m1 = __ballot_sync(0xffffffffu, v1);
                    if (!(m0 | m1)) {
                        load(gi + 2);
                        continue;
                    }
                    if (sink.evaluated && lane == 0)
                        atomicAdd(sink.evaluated, (unsigned long long)(__popc(m0) + __popc(m1)));
#pragma unroll
                    for (int x = 0; x < 2; ++x) {
                        uint32_t r[16];
                        acc_ld(buf, x, gi, r);
#pragma unroll
                        for (int y = 0; y < 2; ++y)
#pragma unroll
                            for (int w2 = 0; w2 < 2; ++w2) {
                                const int e = 4 * w2 + 2 * y;
                                const uint32_t o0 = zb ? r[8 + e] : r[e], o1 = zb ? r[9 + e] : r[1 + e];
                                const uint32_t s0 = zb ? r[e] : r[8 + e], s1 = zb ? r[1 + e] : r[9 + e];
                                const uint32_t p0 = __shfl_xor_sync(0xffffffffu, s0, 16);
                                const uint32_t p1 = __shfl_xor_sync(0xffffffffu, s1, 16);
                                v.c[x][y][0][w2] = f2_pack(__uint_as_float(o0), __uint_as_float(o1));
                                v.c[x][y][1][w2] = f2_pack(__uint_as_float(p0), __uint_as_float(p1));
                            }
                    }
                    const float* tl = tabl0 + ll;
                    if constexpr (!ALL) {
                        F4Bound4 bd(pack, quart);
                        t4x_slices<f2>(
                            v, [&](int e) { return *reinterpret_cast<const f2*>(tl + e * kYL); }, tabk,
                            [&](int sw, int c, f2 cell) {
                                // the last slice has read the triples: the next group's are on their way
                                // while its cells are summed
                                if (sw == 2 && c == 0) load(gi + 2);
                                bd.one(cell);
                            });
                        float b0, b1;
                        f2_unpack(bd.acc, b0, b1);
                        unsigned s0 = __ballot_sync(0xffffffffu, v0 && b0 >= thr_q);
                        unsigned s1 = __ballot_sync(0xffffffffu, v1 && b1 >= thr_q);
                        if (s0 | s1) {
                            load(gi);  // (the next group's triples have taken the place of this one's)
                            const T4xCores<f2> again = v;
                            f2_unpack(t4x_estimate<false>(&again, tl, tabk0, zb, pack), b0, b1);
                            s0 &= __ballot_sync(0xffffffffu, b0 >= thr_f());
                            s1 &= __ballot_sync(0xffffffffu, b1 >= thr_f());
                            while (s0 | s1) {
                                const int u = s0 ? 0 : 1, src = __ffs(u ? s1 : s0) - 1;
                                if (u) s1 &= s1 - 1;
                                else s0 &= s0 - 1;
                                exact_append(src, u, l);
                            }
                            load(gi + 2);
                        }
                    } else {
#pragma unroll 1
                        for (int u = 0; u < 2; ++u) {
                            const bool want = u ? v1 : v0;
                            auto at1 = [&](f2 a) {
                                float lo, hi;
                                f2_unpack(a, lo, hi);
                                return u ? hi : lo;
                            };
                            T4xCores<float> s;
#pragma unroll
                            for (int e = 0; e < 16; ++e)
                                s.c[e >> 3][(e >> 2) & 1][(e >> 1) & 1][e & 1] = at1(v.c[e >> 3][(e >> 2) & 1][(e >> 1) & 1][e & 1]);
#pragma unroll
                            for (int e = 0; e < 8; ++e) {
                                s.ik[e >> 2][(e >> 1) & 1][e & 1] = at1(v.ik[e >> 2][(e >> 1) & 1][e & 1]);
                                s.jk[e >> 2][(e >> 1) & 1][e & 1] = at1(v.jk[e >> 2][(e >> 1) & 1][e & 1]);
                            }
#pragma unroll
                            for (int e = 0; e < 4; ++e) s.kl[e >> 1][e & 1] = at1(v.kl[e >> 1][e & 1]);
                            every(l + u, want, [&](auto&& use) {
                                t4x_slices<float>(
                                    s, [&](int e) { return tl[e * kYL + u]; }, [&](int e) { return at1(tabk(e)); },
                                    [&](int sw, int c, float cell) {
                                        const uint32_t cu = __float2uint_rn(cell);
                                        use(sw, c, cu & wmask, cu >> pack);
                                    });
                            });
                        }
                        load(gi + 2);
                    }
                }
            }
            asm volatile("tcgen05.fence::before_thread_sync;");
            __syncwarp();
            if (lane == 0) {
                arrive_cl(cluster_addr(smem_u32(&acc_empty[SPLIT ? 1 : buf]), 0));
                asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(&tab_empty[buf])) : "memory");
            }
        }
    }
    if (!ok) *abort = 1;
    asm volatile("tcgen05.fence::before_thread_sync;");
    __syncthreads();
    // CTA 1: its epilogue has read the last accumulators, so the pair's final
    // commit to this CTA's `done` lands soon; it must land before the CTA exits
    if (rank == 1 && warp == 1 && lane == 0 && !t3_drain_cl(smem_u32(&done), 0)) *abort = 1;
    cluster_sync_all();  // the other CTA is done with this CTA's shared and tensor memory
    asm volatile("tcgen05.fence::after_thread_sync;");
    if (tid == 0 && abort_flag) atomicOr(status, 1);
    if (warp == 0) asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512));
}

std::vector<long long> t4_item_table(int n, std::vector<long long>& per) {
    std::vector<long long> begin((size_t)n + 1, 0);
    per.assign((size_t)std::max(n, 1), 0);
    for (int j = 0; j < n; ++j) {
        for (int k0 = j + 1; k0 <= n - 2; k0 += kP4K) per[j] += t4x_tiles(n, k0);
        begin[j + 1] = begin[j] + (long long)j * per[j];
    }
    return begin;
}

// Pair tables of a Distribution layer of an order-4 scan (host): the listed pairs (i, j) with at
// least one item, their first owned k and first item.  Returns the items; combos = combinations.
long long t4_layer_items(int n, int step, long long offset, std::vector<long long>& pbegin,
                         std::vector<int4>& pinfo, long long& combos) {
    pbegin.clear();
    pinfo.clear();
    combos = 0;
    long long total = 0;
    for (int i = 0; i + 3 < n; ++i)
        for (int j = i + 1; j + 2 < n; ++j) {
            const long long base = triple_index(i, j, j + 1, n), cnt = n - 1 - j;  // ranks base .. base + cnt - 1
            long long t = std::max(0ll, offset - base);
            t += ((offset - base - t) % step + step) % step;  // first t with base + t = offset (mod step)
            if (t >= cnt) continue;
            const int kf = j + 1 + (int)t;
            long long items = 0;
            for (long long k = kf; k <= n - 2; k += (long long)kP4K * step) items += t4x_tiles(n, (int)k);
            for (long long k = kf; k < n; k += step) combos += n - 1 - k;
            if (items == 0) continue;
            pbegin.push_back(total);
            pinfo.push_back(make_int4(i, j, kf, 0));
            total += items;
        }
    pbegin.push_back(total);
    return total;
}

cudaError_t f4_order4_maps(F4Plan& f, int snps) {
    cudaError_t e = tensor_map(&f.map_b4, f.planes, f.rows, 16 * f.wpr, kYRow, kYN / 2, true);
    if (e == cudaSuccess) e = tensor_map(&f.map_b4h, f.planes, f.rows, 16 * f.wpr, kYRow, 16 * kYHalfG, true);
    if (e == cudaSuccess) e = f4_bit_map(&f.map_k4, f, f.bits, 2 * snps, 2 * kYK);
    return e;
}

cudaError_t launch_tensor4x(const ScanWork& w, const F4Plan& f, const T4xRange& r, long long g0, long long g1,
                            const CandSink& sink, uint32_t* dump, const uint32_t* single, const uint4* pairs,
                            int* status, cudaStream_t s, int sms) {
    if (!f.tri || !pairs || !single || !r.begin || (!r.per && !r.pinfo)) return cudaErrorInvalidValue;
    using Fn = decltype(&tensor4x_kernel<false, false, false>);
    // bits of the index: layer, all, split
    static const Fn fns[8] = {tensor4x_kernel<false, false, false>, tensor4x_kernel<true, false, false>,
                              tensor4x_kernel<false, true, false>,  tensor4x_kernel<true, true, false>,
                              tensor4x_kernel<false, false, true>,  tensor4x_kernel<true, false, true>,
                              tensor4x_kernel<false, true, true>,   tensor4x_kernel<true, true, true>};
    // set once, by whichever host thread comes first (thread-safe static initialisation)
    static const cudaError_t attr = [] {
        cudaError_t e = cudaSuccess;
        for (int k = 0; k < 8 && e == cudaSuccess; ++k)
            e = cudaFuncSetAttribute(fns[k], cudaFuncAttributeMaxDynamicSharedMemorySize,
                                     (int)(k < 4 ? kYSmem<false> : kYSmem<true>));
        return e;
    }();
    if (attr != cudaSuccess) return attr;
    if (g1 <= g0) return cudaSuccess;
    static const int max_clusters = pair_clusters(tensor4x_kernel<false, false, false>, kYThreads, kYSmem<false>);
    const long long clusters = std::min<long long>(g1 - g0, max_clusters > 0 ? max_clusters : sms / 2);
    const unsigned grid = (unsigned)(2 * std::max(1ll, clusters));
    const double scale = 1.0 / (std::log(2.0) * 4294967296.0);
    LiveMap map{scale, -(double)w.base_key * scale - t4x_margin(w.d.n_cases + w.d.n_ctrls), 0, 0};
    const F4Quartic quart = f4_quartic(w.d.n_cases, w.d.n_ctrls, 81, map.bound_k, map.bound_c);
    map.bound_k *= scale;
    const bool all = dump || sink.digest || sink.thr == (long long)0x8000000000000000ull;
    fns[4 * !f.pack + 2 * all + (r.pinfo != nullptr)]<<<grid, kYThreads, f.pack ? kYSmem<false> : kYSmem<true>, s>>>(
        f.map_b4, f.map_b4h, *r.map_k, f.map_i, w, sink, r.begin, r.per, r.pinfo, r.n_pairs, g0, g1, f.nw_c, f.nw_t,
        f.pack, map, quart, dump, single, pairs, f.tri, f.pairf, f.row_p, f.row_q, status);
    count_launch();
    return cudaGetLastError();
}

}  // namespace fiu
