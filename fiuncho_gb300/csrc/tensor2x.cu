// Order-2 contingency tables on CTA pairs with 4-bit operands.
//
// The 4 core cells of a pair (i, j) are dot products of two plane rows: a work
// item (128 i, 120 j) is one GEMM
//     D[(i,x), (j,y)] = sum_s a_ix(s) a_jy(s)    (M 256, N 240)
// with tcgen05.mma.cta_group::2.kind::mxf4, both operands e2m1 plane rows by TMA
// (128-byte swizzle, 256 samples a stage, no producer warps).  CTA r stages its
// own 64 i (128 rows) and half r of the j rows; CTA 0 issues the MMAs.
//
// Classes that share an accumulator (cases + W controls, W = 2^p as the B scale)
// use two regions of 240 columns that alternate between items.  SPLIT: the cases
// accumulate in one region and the controls in the other; as soon as the case GEMM
// is done the epilogue packs its counts to 16 bits in shared memory, so the next
// item's case GEMM runs while this item's controls are evaluated.
//
// Rows are ordered (i / 8, x, i % 8) and columns (j / 8, y, j % 8): a 16x256b
// tensor-memory load gives a thread all 4 cores of (i, j) and (i, j + 1).  The 9
// cells of both follow from the single cores in two-wide single precision; the
// quadratic bound (F4Bound) rejects nearly all pairs, the others get the exact
// fixed-point key, so the kept set is the one of the exact key.
//
// Items are listed in bands of 512 i, j-tile by j-tile: the pairs at work share a
// band's i rows and, in part, each j tile in L2.  40 000 SNPs x 16 000 samples: planes
// of 640 MB, of which the 79 bands need the j above their first i, 25 GB in all; the
// largest launch reads 67 GB (5.0 TB/s), 2.7 times that.
//
// Bound by the MMAs at many samples (40 000 SNPs x 8 000/8 000: 41.6 -> 14.3 ms a
// search against e4m3 operands and one accumulator region per class, 94 % of 4 x
// the measured bf16 rate) and by the evaluation below about 8 000 samples (12 001
// SNPs x 3 999: 2.25 -> 0.77 ms).
//
// Reference semantics: GenotypeTable::combine_and_popcnt for order 2
// (src/base/gt_popcnt.cpp:4-35) over the pairs ThreadedSearch visits
// (include/fiuncho/ThreadedSearch.h:157-180) with one worker.
#include <algorithm>
#include <cmath>

#include "live.cuh"
#include "tensor2x.h"
#include "tensor_fp4.cuh"

namespace fiu {

constexpr int kZI = kP2I / 2;                       // i per CTA
constexpr int kZN = 2 * kP2J;                       // columns of an accumulator region
constexpr int kZG = kP2J / 8;                       // column groups of 8 j
constexpr int kZRow = kF4K / 2;                     // 128 bytes per operand row and stage
constexpr int kZSA = 2 * kZI * kZRow;               // 16 KB
constexpr int kZSB = kZN / 2 * kZRow;               // 15 KB
constexpr int kZStage = kZSA + kZSB;                // 31 KB
constexpr int kZColOne = 2 * kZN, kZColW = kZColOne + 16;
// Epilogue warps: three an SM quarter hide latencies better than two where the evaluation binds
// (counting kernels of 12 001 SNPs x 3 999 samples 0.714 -> 0.688 ms, of 1 000 x 4 000 0.117 -> 0.099);
// SPLIT holds both classes' cells (166 registers).
template <bool SPLIT>
constexpr int kZEpiWarps = SPLIT ? 8 : 12;
template <bool SPLIT>
constexpr int kZThreads = 32 * (4 + kZEpiWarps<SPLIT>);  // copies, MMAs, two staging warps; epilogue
// staged per item: single cores of the j (packed, or cases then controls), the threshold (key, bound)
constexpr int kZTabT = 4 * kP2J * 4, kZTab = kZTabT + 16;
constexpr int kZStash = kZEpiWarps<true> * ((kZG + 1) / 2) * 2 * 32 * 16;  // 64 KB: (warp, its group, lane block, lane), 8 counts
template <bool SPLIT>
constexpr int kZStages = SPLIT ? 5 : 7;
template <bool SPLIT>
constexpr size_t kZSmem = 1024 + (size_t)kZStages<SPLIT> * kZStage + (SPLIT ? kZStash : 0) + 2 * kZTab;
static_assert(kZSmem<false> <= 227 * 1024 - 512 && kZSmem<true> <= 227 * 1024 - 512, "order-2 pair kernel shared memory");
static_assert(kZStage % 1024 == 0 && kZSA % 1024 == 0, "operand tiles on swizzle atoms");
static_assert(kZColW + 16 <= 512, "tensor memory columns");

// Item g: position p0 of its first owned i, first j.
__device__ __forceinline__ void t2x_item(const long long* __restrict__ begin, int tiles, int first, int step,
                                         long long g, int& p0, int& j0) {
    int lo = 0, hi = (tiles + kP2Band - 1) / kP2Band - 1;
    while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (__ldg(begin + mid) <= g) lo = mid;
        else hi = mid - 1;
    }
    const int ca = min(kP2Band, tiles - kP2Band * lo);  // tiles in the band
    const unsigned idx = (unsigned)(g - __ldg(begin + lo)), b = idx / ca;
    p0 = kP2I * (kP2Band * lo + (int)(idx - b * ca));
    j0 = kP2J * ((layer_snp(first, step, kP2I * kP2Band * lo) + 1) / kP2J + (int)b);
}

// 9 cells of both classes (or packed) from cores c (x, y), singles of i (si: 0, 1, any left) and of j.
__device__ __forceinline__ f2 t2x_less(f2 a, f2 b, f2 c) { return f2_sub(f2_sub(a, b), c); }
__device__ __forceinline__ void t2x_cells(const f2 (&c)[2][2], const f2 (&si)[3], const f2 (&sj)[2], f2 (&t)[9]) {
#pragma unroll
    for (int x = 0; x < 2; ++x) {
        t[3 * x] = c[x][0];
        t[3 * x + 1] = c[x][1];
        t[3 * x + 2] = t2x_less(si[x], c[x][0], c[x][1]);
    }
#pragma unroll
    for (int y = 0; y < 2; ++y) t[6 + y] = t2x_less(sj[y], c[0][y], c[1][y]);
    t[8] = t2x_less(si[2], t[6], t[7]);
}

// SPLIT: one accumulator region per class.
template <bool SPLIT>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(kZThreads<SPLIT>, 1)
    tensor2x_kernel(const __grid_constant__ CUtensorMap map_a, const __grid_constant__ CUtensorMap map_b,
                    const __grid_constant__ ScanWork w, const __grid_constant__ CandSink sink,
                    const long long* __restrict__ begin, int tiles, int first, int istep, long long g0, long long g1,
                    int nw_c, int nw_t, int pack, const __grid_constant__ LiveMap map, uint32_t* dump,
                    const uint32_t* __restrict__ single, int* status) {
    constexpr int kStages = kZStages<SPLIT>;
    extern __shared__ uint8_t smraw[];
    __shared__ __align__(8) uint64_t full[kStages], empty[kStages];
    __shared__ __align__(8) uint64_t acc_full[2], acc_empty[2], tab_full[2], tab_empty[2], done;
    __shared__ uint32_t tmem_base;
    __shared__ int abort_flag;
    uint8_t* sm = (uint8_t*)(((uintptr_t)smraw + 1023) & ~(uintptr_t)1023);  // stages: A | B half
    uint8_t* tabs = sm + kStages * kZStage;
    uint4* stash = reinterpret_cast<uint4*>(tabs + 2 * kZTab);
    volatile int* abort = &abort_flag;
    const int n = w.d.snps;
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
            init(&full[s], 1);
            init(&empty[s], 1);
        }
        for (int b = 0; b < 2; ++b) {
            init(&acc_full[b], 1);
            init(&acc_empty[b], 2 * kZEpiWarps<SPLIT>);
            init(&tab_full[b], 2);
            init(&tab_empty[b], kZEpiWarps<SPLIT>);
        }
        init(&done, 1);
        asm volatile("fence.mbarrier_init.release.cluster;");
        abort_flag = 0;
    }
    asm volatile("tcgen05.fence::before_thread_sync;");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;");
    const uint32_t tmem = tmem_base;
    if (warp >= 4 && warp < 8) f4_fill_scales<16>(tmem, warp & 3, kZColOne, kZColW, pack);
    asm volatile("tcgen05.fence::before_thread_sync;");
    __syncthreads();
    cluster_sync_all();  // both CTAs' barriers and scales exist before either signals the other
    asm volatile("tcgen05.fence::after_thread_sync;");
    bool ok = true;

    if (warp == 0) {
        // ---------------------------------------------------------------- TMA producer (both CTAs)
        if (g0 + cid < g1 && elect_one()) {
            unsigned s = 0, par = 1, step = 0;  // stage, parity of its last release (first round: free)
            int p0, j0;
            t2x_item(begin, tiles, first, istep, g0 + cid, p0, j0);
            for (long long g = g0 + cid; g < g1 && ok; g += ncl) {
                const int arow = 2 * (p0 + kZI * (int)rank), brow = 2 * j0 + kP2J * (int)rank;
                for (int ks = 0; ks < ksteps; ++ks) {
                    if (!t3_wait_cl(smem_u32(&empty[s]), par, abort)) {
                        ok = false;
                        break;
                    }
                    // both CTAs' copies count on CTA 0's barrier, where the MMA issuer waits
                    const uint32_t st = smem_u32(sm + s * kZStage), bar = cluster_addr(smem_u32(&full[s]), 0);
                    if (rank == 0)
                        asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(&full[s])),
                                     "r"((uint32_t)(2 * kZStage))
                                     : "memory");
                    t3_tma_pair(st, &map_a, kZRow * ks, arow, bar);
                    t3_tma_pair(st + kZSA, &map_b, kZRow * ks, brow, bar);
                    if (step < kStages) ++step;
                    if (++s == kStages) {
                        s = 0;
                        par ^= 1;
                    }
                    // the next item's place is looked up while this item's copies are in flight
                    if (ks == 0 && g + ncl < g1) t2x_item(begin, tiles, first, istep, g + ncl, p0, j0);
                }
            }
            // copies in flight land before the pair is released: CTA 0 sees every copy of both CTAs
            // complete on its `full` barriers, CTA 1 sees its stages consumed.  Stage q was last filled in
            // the round before `par` names, or in this one when q < s.
            for (unsigned q = 0; q < step; ++q)
                if (!t3_drain_cl(smem_u32(rank == 0 ? &full[q] : &empty[q]), q < s ? par ^ 1 : par)) ok = false;
        }
        __syncwarp();
    } else if (warp == 1) {
        // ---------------------------------------------------------------- MMA issuer (CTA 0)
        if (rank == 0 && elect_one()) {
            ok = f4_pair_issue<SPLIT, kStages, kZStage, kStages, kZStage, kZN, kZColOne, kZColW>(
                (g1 - g0 - cid + ncl - 1) / ncl, smem_u32(sm), smem_u32(sm + kZSA), smem_u32(&full[0]),
                smem_u32(&empty[0]), smem_u32(&acc_full[0]), smem_u32(&acc_empty[0]), tmem, nw_c, nw_t, abort,
                [](unsigned) { return kZN; });
            commit_pair(smem_u32(&done));
            // neither CTA releases shared or tensor memory before the pair's MMAs are
            // done (CTA 1 waits once its own work is over, below)
            if (!t3_drain_cl(smem_u32(&done), 0)) ok = false;
        }
        __syncwarp();
    } else if (warp < 4) {
        // ---------------------------------------------------------------- table staging (both CTAs)
        const int t = tid - 64;  // 0 .. 63
        const float W = (float)(1u << pack);
        unsigned item = 0;
        for (long long g = g0 + cid; g < g1 && ok; g += ncl, ++item) {
            int p0, j0;
            t2x_item(begin, tiles, first, istep, g, p0, j0);
            const unsigned buf = item & 1;
            if (item >= 2 && !t3_wait(smem_u32(&tab_empty[buf]), ((item >> 1) - 1) & 1, abort)) {
                ok = false;
                break;
            }
            uint8_t* tab = tabs + buf * kZTab;
            float* tl = reinterpret_cast<float*>(tab);
            for (int ll = t; ll < kP2J; ll += 64) {
                const int j = j0 + ll;
                const uint4 v = j < n ? __ldg(reinterpret_cast<const uint4*>(single) + j) : make_uint4(0, 0, 0, 0);
                if (SPLIT) {
                    tl[ll] = u2f(v.x);
                    tl[kP2J + ll] = u2f(v.y);
                    tl[2 * kP2J + ll] = u2f(v.z);
                    tl[3 * kP2J + ll] = u2f(v.w);
                } else {
                    tl[ll] = fmaf(W, u2f(v.z), u2f(v.x));
                    tl[kP2J + ll] = fmaf(W, u2f(v.w), u2f(v.y));
                }
            }
            // the threshold of this item (the pairs take turns at raising the live one)
            if (sink.hist && rank == 0 && warp == 2 && item > 0 && (item < 3 || ((item + cid) & 7) == 0))
                live_update(sink, lane);
            if (t == 0) {
                const long long thr = sink.hist ? *(volatile long long*)sink.live : sink.thr;
                float est, bound;
                live_tests(map, thr, est, bound);
                *reinterpret_cast<long long*>(tab + kZTabT) = thr;
                *reinterpret_cast<float*>(tab + kZTabT + 8) = bound;
            }
            __syncwarp();
            if (lane == 0)
                asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(&tab_full[buf])) : "memory");
        }
    } else {
        // ---------------------------------------------------------------- epilogue (both CTAs)
        const int q = warp & 3, hh = (warp - 4) >> 2;  // lane quarter (16 i); its warps take groups in turn
        constexpr unsigned kShare = kZEpiWarps<SPLIT> / 4;
        const int il = lane >> 2, lc = 2 * (lane & 3);  // this thread's i of a block of 8, its two j of a group
        const float W = (float)(1u << pack);
        const uint32_t wmask = (1u << pack) - 1u;
        const uint32_t nc = (uint32_t)w.d.n_cases, nt = (uint32_t)w.d.n_ctrls;
        const bool all = dump != nullptr || sink.digest != nullptr;  // every pair takes the exact path
        const float m23 = 8388608.0f;
        uint4* mine = stash + (warp - 4) * ((kZG + 1) / 2) * 64 + lane;  // written and read by this warp only
        unsigned item = 0;
        for (long long g = g0 + cid; g < g1 && ok; g += ncl, ++item) {
            int p0, j0;
            t2x_item(begin, tiles, first, istep, g, p0, j0);
            const unsigned buf = item & 1, ph = (item >> 1) & 1;
            const unsigned gi0 = (hh + item) % kShare;  // the odd group of an item goes to each warp in turn
            // this thread's i and their single cores (0, 1, what is left), packed or per class
            int iv[2];
            f2 si[2][SPLIT ? 2 : 1][3];
#pragma unroll
            for (int u = 0; u < 2; ++u) {
                iv[u] = layer_snp(first, istep, p0 + kZI * (int)rank + 16 * q + 8 * u + il);
                const uint4 v = iv[u] < n ? __ldg(reinterpret_cast<const uint4*>(single) + iv[u]) : make_uint4(0, 0, 0, 0);
                const float a0 = u2f(v.x), a1 = u2f(v.y), b0 = u2f(v.z), b1 = u2f(v.w);
                const float ar = (float)nc - a0 - a1, br = (float)nt - b0 - b1;
                if constexpr (SPLIT) {
                    si[u][0][0] = f2_dup(a0);
                    si[u][0][1] = f2_dup(a1);
                    si[u][0][2] = f2_dup(ar);
                    si[u][1][0] = f2_dup(b0);
                    si[u][1][1] = f2_dup(b1);
                    si[u][1][2] = f2_dup(br);
                } else {
                    si[u][0][0] = f2_dup(fmaf(W, b0, a0));
                    si[u][0][1] = f2_dup(fmaf(W, b1, a1));
                    si[u][0][2] = f2_dup(fmaf(W, br, ar));
                }
            }
            // accumulators of lane block u, group gi: registers 4 y + 2 x (j) and + 1 (j + 1)
            auto ld = [&](int region, int u, unsigned gi, uint32_t (&r)[8]) {
                asm volatile(
                    "tcgen05.ld.sync.aligned.16x256b.x2.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
                    : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
                    : "r"(tmem + ((uint32_t)(32 * q + 16 * u) << 16) + (uint32_t)(kZN * region + 16 * gi)));
            };
            if (SPLIT) {
                // case counts -> 16 bits in shared memory (j | j + 1 << 16); their region is then free
                if (!t3_wait_cl(smem_u32(&acc_full[0]), item & 1, abort)) {
                    ok = false;
                    break;
                }
                asm volatile("tcgen05.fence::after_thread_sync;");
#pragma unroll 1
                for (unsigned gi = gi0; gi < kZG; gi += kShare) {
                    uint32_t r[2][8];
                    ld(0, 0, gi, r[0]);
                    ld(0, 1, gi, r[1]);
                    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
                    for (int u = 0; u < 2; ++u) {
                        uint32_t o[4];
#pragma unroll
                        for (int k = 0; k < 4; ++k)
                            o[k] = __byte_perm(__float_as_uint(__uint_as_float(r[u][2 * k]) + m23),
                                               __float_as_uint(__uint_as_float(r[u][2 * k + 1]) + m23), 0x5410);
                        mine[((gi >> 1) * 2 + u) * 32] = make_uint4(o[0], o[1], o[2], o[3]);
                    }
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
            const float* tl0 = reinterpret_cast<const float*>(tabs + buf * kZTab);
            const long long thr = *reinterpret_cast<const long long*>(tabs + buf * kZTab + kZTabT);
            const float thr_q = *reinterpret_cast<const float*>(tabs + buf * kZTab + kZTabT + 8);
#pragma unroll 1
            for (unsigned gi = gi0; gi < kZG; gi += kShare) {
                const int ll = 8 * gi + lc, j = j0 + ll;
                bool v[2][2];
                unsigned vm = 0, count = 0;
#pragma unroll
                for (int u = 0; u < 2; ++u)
#pragma unroll
                    for (int e = 0; e < 2; ++e) {
                        v[u][e] = iv[u] < n && j + e < n && j + e > iv[u];
                        const unsigned m = __ballot_sync(0xffffffffu, v[u][e]);
                        vm |= m;
                        count += __popc(m);
                    }
                if (!vm) continue;
                if (sink.evaluated && lane == 0) atomicAdd(sink.evaluated, (unsigned long long)count);
                uint32_t r[2][8];
                ld(SPLIT ? 1 : buf, 0, gi, r[0]);
                ld(SPLIT ? 1 : buf, 1, gi, r[1]);
                uint4 sv[2];
                if (SPLIT) {
                    sv[0] = mine[(gi >> 1) * 64];
                    sv[1] = mine[(gi >> 1) * 64 + 32];
                }
                const float* tl = tl0 + ll;
                f2 sj[SPLIT ? 2 : 1][2];
#pragma unroll
                for (int c = 0; c < (SPLIT ? 2 : 1); ++c)
#pragma unroll
                    for (int y = 0; y < 2; ++y) sj[c][y] = *reinterpret_cast<const f2*>(tl + (2 * c + y) * kP2J);
                asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
                for (int u = 0; u < 2; ++u) {
                    f2 t[SPLIT ? 2 : 1][9];  // packed cells, or cases and controls; (i, j) and (i, j + 1)
                    {
                        f2 c[2][2];
#pragma unroll
                        for (int x = 0; x < 2; ++x)
#pragma unroll
                            for (int y = 0; y < 2; ++y)
                                c[x][y] = f2_pack(__uint_as_float(r[u][4 * y + 2 * x]),
                                                  __uint_as_float(r[u][4 * y + 2 * x + 1]));
                        t2x_cells(c, si[u][SPLIT ? 1 : 0], sj[SPLIT ? 1 : 0], t[SPLIT ? 1 : 0]);
                    }
                    if constexpr (SPLIT) {
                        f2 c[2][2];
#pragma unroll
                        for (int x = 0; x < 2; ++x)
#pragma unroll
                            for (int y = 0; y < 2; ++y) {
                                const uint32_t o = (&sv[u].x)[2 * y + x];
                                c[x][y] = f2_add(f2_pack(__uint_as_float(__byte_perm(o, 0x4B000000u, 0x7610)),
                                                         __uint_as_float(__byte_perm(o, 0x4B000000u, 0x7632))),
                                                 f2_dup(-m23));
                            }
                        t2x_cells(c, si[u][0], sj[0], t[0]);
                    }
                    F4Bound bd(pack);
                    if constexpr (SPLIT) {
                        auto size = [&](int c) { return f2_add(f2_add(t[0][c], t[1][c]), bd.tiny); };
#pragma unroll
                        for (int c = 0; c < 8; c += 2) bd.two(t[1][c], size(c), t[1][c + 1], size(c + 1));
                        bd.acc = f2_fma(t[1][8], f2_mul(t[1][8], f2_rcp(size(8))), bd.acc);
                    } else {
#pragma unroll
                        for (int c = 0; c < 8; c += 2) bd.two(t[0][c], t[0][c + 1]);
                        bd.one(t[0][8]);
                    }
                    float b[2];
                    f2_unpack(bd.acc, b[0], b[1]);
                    if (!__any_sync(0xffffffffu, (v[u][0] && (all || b[0] >= thr_q)) || (v[u][1] && (all || b[1] >= thr_q))))
                        continue;
                    // the rare path: exact keys
#pragma unroll
                    for (int e = 0; e < 2; ++e) {
                        const bool want = v[u][e] && (all || b[e] >= thr_q);
                        unsigned long long dg = 0;
                        if (want) {
                            const int cmb[2] = {iv[u], j + e};
                            // owned prefix ordinal m of i: rank offset + m * step
                            uint32_t* o = dump ? dump + ((size_t)((iv[u] - w.dist_offset) / w.dist_step) * n + j + e) * 18
                                               : nullptr;
                            if (sink.digest) dg = dg_begin(cmb, 2, n);
                            long long key = w.base_key;
#pragma unroll
                            for (int c = 0; c < 9; ++c) {
                                float lo, hi;
                                f2_unpack(t[0][c], lo, hi);
                                uint32_t ca = __float2uint_rn(e ? hi : lo), cb;
                                if constexpr (SPLIT) {
                                    f2_unpack(t[1][c], lo, hi);
                                    cb = __float2uint_rn(e ? hi : lo);
                                } else {
                                    cb = ca >> pack;
                                    ca &= wmask;
                                }
                                if (o) {
                                    o[c] = ca;
                                    o[9 + c] = cb;
                                }
                                if (sink.digest) dg = dg_cell(dg, ca, cb);
                                const uint32_t a = min(ca, nc), bb = min(cb, nt);
                                key += __ldg(w.d.ftab + a) + __ldg(w.d.ftab + bb) - __ldg(w.d.ftab + a + bb);
                            }
                            if (key >= thr) live_append(sink, key, pack_code(cmb, 2, w.bits));
                        }
                        if (sink.digest) dg_warp_add(sink.digest, dg);
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

// One 16-byte chunk (32 samples) per thread.
__global__ void f4_ones_kernel(DevData d, uint4* planes, int wpr, int wc, int nc32, int nt32, int rows, int count,
                               int first, int step) {
    const size_t per_snp = 3 * (size_t)(d.cw + d.tw);
    const long long total = (long long)rows * wpr;
    for (long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x; e < total;
         e += (long long)gridDim.x * blockDim.x) {
        const int row = (int)(e / wpr), o = (int)(e - (long long)row * wpr);
        const int m = 8 * (row >> 4) + (row & 7), g = (row >> 3) & 1;
        const bool ctrl = o >= wc;
        const int k = ctrl ? o - wc : o;
        uint32_t v = 0;
        if (m < count && k < (ctrl ? nt32 : nc32)) {
            const size_t snp = (size_t)first + (size_t)step * m;
            const uint64_t word = __ldg(d.ref + snp * per_snp + (ctrl ? 3 * (size_t)d.cw : 0) +
                                        (size_t)g * (ctrl ? d.tw : d.cw) + (k >> 1));
            v = (uint32_t)(word >> (32 * (k & 1)));
        }
        planes[e] = f4_expand_ones(v);
    }
}

cudaError_t f4_ones_planes(const DevData& d, const F4Plan& f, int count, int first, int step, uint8_t*& planes,
                           cudaStream_t s) {
    const int rows = 16 * ((count + 7) / 8), wc = 8 * ((f.nw_c + 3) / 4);
    uint8_t* p = nullptr;
    cudaError_t e = cudaMalloc((void**)&p, std::max<size_t>(1, (size_t)rows * f.wpr * 16));
    if (e != cudaSuccess) return e;
    const long long total = (long long)rows * f.wpr;
    f4_ones_kernel<<<(unsigned)std::max<long long>(1, std::min<long long>((total + 255) / 256, 16384)), 256, 0, s>>>(
        d, reinterpret_cast<uint4*>(p), f.wpr, wc, 2 * f.nw_c, 2 * f.nw_t, rows, count, first, step);
    count_launch();
    e = cudaGetLastError();
    if (e != cudaSuccess) cudaFree(p);
    else planes = p;
    return e;
}

cudaError_t f4_map_a2(CUtensorMap* m, const F4Plan& f, const uint8_t* planes, int count) {
    return tensor_map(m, planes, 16 * std::max(1, (count + 7) / 8), 16 * f.wpr, kZRow, 2 * kZI, true);
}
cudaError_t f4_map_b2(CUtensorMap* m, const F4Plan& f, const uint8_t* planes, int count) {
    return tensor_map(m, planes, 16 * std::max(1, (count + 7) / 8), 16 * f.wpr, kZRow, kP2J, true);
}

std::vector<long long> t2x_items(int n, long long count, long long first, long long step, int& tiles) {
    tiles = (int)((count + kP2I - 1) / kP2I);
    const int bands = (tiles + kP2Band - 1) / kP2Band;
    const long long nb = (n + kP2J - 1) / kP2J;  // global j-tiles
    std::vector<long long> begin((size_t)bands + 1, 0);
    for (int r = 0; r < bands; ++r) {
        const long long i_first = first + step * (long long)kP2I * kP2Band * r;
        begin[r + 1] = begin[r] + std::min(kP2Band, tiles - kP2Band * r) * std::max(0ll, nb - (i_first + 1) / kP2J);
    }
    return begin;
}

cudaError_t launch_tensor2x(const ScanWork& w, const F4Plan& f, const T2xRange& r, long long g0, long long g1,
                            const CandSink& sink, uint32_t* dump, const uint32_t* single, int* status, cudaStream_t s,
                            int sms) {
    // set once, by whichever host thread comes first (thread-safe static initialisation)
    static const cudaError_t attr = [] {
        cudaError_t e = cudaFuncSetAttribute(tensor2x_kernel<false>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                             (int)kZSmem<false>);
        if (e == cudaSuccess)
            e = cudaFuncSetAttribute(tensor2x_kernel<true>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                     (int)kZSmem<true>);
        return e;
    }();
    if (attr != cudaSuccess) return attr;
    if (g1 <= g0) return cudaSuccess;
    static const int max_clusters = pair_clusters(tensor2x_kernel<false>, kZThreads<false>, kZSmem<false>);
    const long long clusters = std::min<long long>(g1 - g0, max_clusters > 0 ? max_clusters : sms / 2);
    const unsigned grid = (unsigned)(2 * std::max(1ll, clusters));
    LiveMap map{0, 0, 0, 0};
    f4_quadratic(w.d.n_cases, w.d.n_ctrls, 9, map.bound_k, map.bound_c);
    map.bound_k /= std::log(2.0) * 4294967296.0;
    if (f.pack)
        tensor2x_kernel<false><<<grid, kZThreads<false>, kZSmem<false>, s>>>(*r.map_a, *r.map_b, w, sink, r.item_begin, r.tiles,
                                                                      r.first, r.step, g0, g1, f.nw_c, f.nw_t, f.pack,
                                                                      map, dump, single, status);
    else
        tensor2x_kernel<true><<<grid, kZThreads<true>, kZSmem<true>, s>>>(*r.map_a, *r.map_b, w, sink, r.item_begin, r.tiles,
                                                                    r.first, r.step, g0, g1, f.nw_c, f.nw_t, 1, map,
                                                                    dump, single, status);
    count_launch();
    return cudaGetLastError();
}

}  // namespace fiu
