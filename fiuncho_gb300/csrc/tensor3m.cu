// Order-3 searches of data with missing calls on CTA pairs with 4-bit operands.
//
// A sample that lacks a call has no genotype at that SNP, so the cells of
// genotype 2 do not follow from the marginals and all 27 are counted:
//     cell[x][y][z] = sum_s a_ix(s) a_jy(s) a_lz(s),  x, y, z in {0, 1, 2}.
// A work item is (i, 64 j, up to 80 l) on a cluster of two CTAs, as in the
// complete-data kernel (tensor3x.cu: operand formats, roles, handover, scales).
// Its 9 genotypes (x, y) are three GEMMs over the samples, of four, four and one
// of them (M 256: 64 j, N <= 240: 80 l, 3 z); four rows a j keep all values of a
// thread's combinations in one tensor-memory lane quarter, without a transpose.
// Two accumulator regions alternate between the GEMMs.
//
// Epilogue.  The cells add up to the key whichever they are, so each GEMM's
// cells go into running sums of a thread's combinations: a single-precision
// estimate of the key with a proven error bound (the rows of an SNP share no
// sample: the cells of a combination sum to at most the class sizes, which is
// what the bound needs) rejects the combinations that cannot reach the threshold;
// the few others get the exact fixed-point key from the data set.  A search's
// first units, before a threshold, sum the exact key itself (ALL).
//
// Bound by the pace of the stages, as the complete-data kernel (its cost is three
// GEMMs where that one takes one, on tiles of 80 l instead of 120); the
// evaluation (81 logarithms a combination) takes 18 000 cycles an item.  400 SNPs x
// 4 000/4 000: 28.2 -> 1.9 ms a search (kernels 1.7) against the full-table kernel (27 AND, POPC and ADD a
// word of a combination, 16 POPC a cycle and SM).
//
// Reference semantics: GenotypeTable::combine_and_popcnt for order 3
// (src/base/gt_popcnt.cpp:4-35) and MutualInformation::compute
// (src/base/mi_compute.cpp:16-41).
#include <algorithm>
#include <cmath>

#include "exact_key.cuh"
#include "live.cuh"
#include "tensor3m.h"
#include "tensor_fp4.cuh"

namespace fiu {

constexpr int kMJ = kPmJ / 2;                       // j per CTA
constexpr int kMN = 48 * kPmG;                      // columns of an accumulator region
constexpr int kMRow = kF4K / 2;                     // 128 bytes per operand row and stage
constexpr int kMBitRow = kF4K / 8;                  // 32 bytes per bit row and stage
constexpr int kMHalfG = 2;                          // items of at most 2 groups bring 48 l rows a CTA, others 120
constexpr int kMStages = 8, kMAStages = 4;          // rings of the copies and of A, as in the complete-data kernel
constexpr int kMSA = 4 * kMJ * kMRow;               // 16 KB
constexpr int kMSB = kMN / 2 * kMRow;               // 15 KB: this CTA's half of the l rows
constexpr int kMSJ = 3 * kMJ * kMBitRow;            //  3 KB
constexpr int kMSI = 3 * kMBitRow;                  // 96 bytes
constexpr int kMBits = kMSJ + 128;                  // the bit rows of a stage, behind the A tiles
constexpr int kMColOne = 2 * kMN, kMColW = kMColOne + 16;
// 640 threads: copies, MMAs, two idle warps; two groups of four builders that take alternate stages; eight
// epilogue warps.  Registers a thread: 96 at launch, then 56 / 56 / 152.
constexpr int kMBuildWarps = 4, kMEpiWarps = 8;
constexpr int kMThreads = 32 * (4 + 2 * kMBuildWarps + kMEpiWarps);
constexpr int kMMeta = 16;                          // items in flight between the copies and the MMAs
constexpr size_t kMSmem = 1024 + (size_t)kMStages * (kMSB + kMBits) + (size_t)kMAStages * kMSA;
static_assert(kMSmem <= 227 * 1024 - 512, "shared memory");
static_assert(kMSA % 1024 == 0 && kMSB % 1024 == 0 && kMBits % 128 == 0, "operand tiles on swizzle atoms");
static_assert(kMColW + 16 <= 512, "tensor memory columns");

// One item: (i, j0 ..), l-tile of ng groups of 16 from l0.
struct T3mItem {
    int i, j0, l0, ng;
};

// Item g; i is the walker's position (the items of one walker ascend).
__device__ __forceinline__ T3mItem t3m_item(const long long* __restrict__ item_begin, int n, long long g, int& i) {
    if (i < 0) {
        int lo = 0, hi = n - 1;
        while (lo < hi) {
            const int mid = (lo + hi + 1) >> 1;
            if (__ldg(item_begin + mid) <= g) lo = mid;
            else hi = mid - 1;
        }
        i = lo;
    } else {
        while (__ldg(item_begin + i + 1) <= g) ++i;
    }
    int q = (int)(g - __ldg(item_begin + i));
    for (int j = i + 1;; j += kPmJ) {
        const int nl = t3m_tiles(n, j);
        if (q < nl) {
            const int G = t3m_groups(n, j), a = G * q / nl, b = G * (q + 1) / nl;
            return T3mItem{i, j, ((j + 1) & ~7) + 16 * a, b - a};
        }
        q -= nl;
    }
}

// Columns the MMAs of an item of ng groups multiply (at least 96).
__device__ __forceinline__ int t3m_n(int ng) { return 48 * max(ng, 2); }

template <bool ALL>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(kMThreads, 1)
    tensor3m_kernel(const __grid_constant__ CUtensorMap map_b, const __grid_constant__ CUtensorMap map_bh,
                    const __grid_constant__ CUtensorMap map_j, const __grid_constant__ CUtensorMap map_i,
                    const __grid_constant__ ScanWork w, const __grid_constant__ CandSink sink,
                    const long long* __restrict__ item_begin, long long g0, long long g1, int nw_c, int nw_t, int pack,
                    const __grid_constant__ LiveMap map, int* status) {
    extern __shared__ uint8_t smraw[];
    __shared__ __align__(8) uint64_t full_t[kMStages], empty[kMStages], full_a[kMAStages];
    __shared__ __align__(8) uint64_t acc_full[2], acc_empty[2], done;
    __shared__ uint32_t tmem_base;
    __shared__ int item_ng[kMMeta];  // groups of the items in flight, for the MMA issuer
    __shared__ int abort_flag;
    uint8_t* sm = (uint8_t*)(((uintptr_t)smraw + 1023) & ~(uintptr_t)1023);  // stages: B half; the A tiles; j | i
    uint8_t* sma = sm + kMStages * kMSB;
    uint8_t* smj = sma + kMAStages * kMSA;
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
        for (int s = 0; s < kMStages; ++s) {
            init(&full_t[s], 1);
            init(&empty[s], 1);
        }
        for (int s = 0; s < kMAStages; ++s) init(&full_a[s], 2 * kMBuildWarps);
        for (int b = 0; b < 2; ++b) {
            init(&acc_full[b], 1);
            init(&acc_empty[b], 2 * kMEpiWarps);
        }
        init(&done, 1);
        asm volatile("fence.mbarrier_init.release.cluster;");
        abort_flag = 0;
    }
    asm volatile("tcgen05.fence::before_thread_sync;");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;");
    const uint32_t tmem = tmem_base;
    if (warp >= 4 && warp < 8) f4_fill_scales<16>(tmem, warp & 3, kMColOne, kMColW, pack);
    asm volatile("tcgen05.fence::before_thread_sync;");
    __syncthreads();
    cluster_sync_all();  // both CTAs' barriers and scales exist before either signals the other
    asm volatile("tcgen05.fence::after_thread_sync;");
    bool ok = true;

    // (the register limits are set inside the branches, as in the complete-data kernel)
    if (warp < 4) {
        asm volatile("setmaxnreg.dec.sync.aligned.u32 56;");
        if (warp == 0) {
            // ---------------------------------------------------------------- TMA producer (both CTAs)
            if (g0 + cid < g1 && elect_one()) {
                unsigned s = 0, par = 1;  // stage and the parity its last release has (first round: free)
                unsigned step = 0, item = 0;
                int wi = -1;
                T3mItem it = t3m_item(item_begin, n, g0 + cid, wi);
                for (long long g = g0 + cid; g < g1 && ok; g += ncl) {
                    const int jrow = 3 * (it.j0 + kMJ * (int)rank), irow = 3 * it.i;
                    const int brow = 3 * it.l0 + t3m_n(it.ng) / 2 * (int)rank;
                    const bool half = it.ng <= kMHalfG;
                    item_ng[item++ % kMMeta] = it.ng;
                    T3mItem nx = it;
                    for (int ks = 0, left = 3 * ksteps; left > 0; --left) {
                        if (!t3_wait_cl(smem_u32(&empty[s]), par, abort)) {
                            ok = false;
                            break;
                        }
                        const uint32_t st = smem_u32(sm + s * kMSB), bar = smem_u32(&full_t[s]);
                        const uint32_t sj = smem_u32(smj + s * kMBits);
                        asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar),
                                     "r"((uint32_t)((half ? 24 * kMHalfG * kMRow : kMSB) + kMSJ + kMSI))
                                     : "memory");
                        t3_tma(sj, &map_j, kMBitRow * ks, jrow, bar);
                        t3_tma(sj + kMSJ, &map_i, kMBitRow * ks, irow, bar);
                        t3_tma(st, half ? &map_bh : &map_b, kMRow * ks, brow, bar);
                        if (step < kMStages) ++step;
                        if (++s == kMStages) {
                            s = 0;
                            par ^= 1;
                        }
                        // the next item's place is looked up while this item's copies are in flight
                        if (left == 3 * ksteps && g + ncl < g1) nx = t3m_item(item_begin, n, g + ncl, wi);
                        if (++ks == ksteps) ks = 0;
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
                ok = f4_pair_issue<false, kMAStages, kMSA, kMStages, kMSB, kMN, kMColOne, kMColW>(
                    3 * ((g1 - g0 - cid + ncl - 1) / ncl), smem_u32(sma), smem_u32(sm), smem_u32(&full_a[0]),
                    smem_u32(&empty[0]), smem_u32(&acc_full[0]), smem_u32(&acc_empty[0]), tmem, nw_c, nw_t, abort,
                    [&](unsigned gemm) { return t3m_n(item_ng[gemm / 3 % kMMeta]); });
                commit_pair(smem_u32(&done));
                // neither CTA releases shared or tensor memory before the pair's MMAs are
                // done (CTA 1 waits once its own work is over, below)
                if (!t3_drain_cl(smem_u32(&done), 0)) ok = false;
            }
            __syncwarp();
        }
    } else if (warp < 12) {
        asm volatile("setmaxnreg.dec.sync.aligned.u32 56;");
        // ---------------------------------------------------------------- A builders (both CTAs)
        // thread: 16-byte chunk c (32 samples) of j = rg and rg + 16 of every second stage; A row (j / 8, slot,
        // j % 8), slots (x, y) = (0,0) (0,1) (1,0) (1,1) | (0,2) (1,2) (2,0) (2,1) | (2,2) and none
        const int t = (tid - 128) & (32 * kMBuildWarps - 1), c = t & 7, rg = t >> 3;
        const uint32_t full0 = cluster_addr(smem_u32(&full_a[0]), 0);
        const int dst0 = (32 * (rg >> 3) + (rg & 7)) * kMRow + ((c ^ (rg & 7)) << 4);
        unsigned s = 0, par = 0, sa = 0;                // copy stage, A stage
        unsigned se = kMStages - kMAStages, pe = 1;     // the stage whose MMAs free this A stage
        bool mine = warp < 8;
        for (long long g = g0 + cid; g < g1 && ok; g += ncl) {
            for (int gemm = 0; gemm < 3 && ok; ++gemm)
                for (int ks = 0; ks < ksteps; ++ks, mine = !mine) {
                    if (mine) {
                        if (!t3_wait(smem_u32(&full_t[s]), par, abort)) {
                            ok = false;
                            break;
                        }
                        const uint32_t* sJ = reinterpret_cast<const uint32_t*>(smj + s * kMBits) + 24 * rg + c;
                        const uint32_t* sI = reinterpret_cast<const uint32_t*>(smj + s * kMBits + kMSJ) + c;
                        uint32_t jw[2][3], iw[3];
#pragma unroll
                        for (int v = 0; v < 3; ++v) {
                            jw[0][v] = sJ[8 * v];
                            jw[1][v] = sJ[24 * 16 + 8 * v];
                            iw[v] = sI[8 * v];
                        }
                        if (!t3_wait_cl(smem_u32(&empty[se]), pe, abort)) {
                            ok = false;
                            break;
                        }
                        uint8_t* dst = sma + sa * kMSA + dst0;
#pragma unroll
                        for (int u = 0; u < 2; ++u) {
                            const uint32_t* jv = jw[u];
                            const uint32_t i2 = gemm == 0 ? iw[1] : gemm == 1 ? iw[2] : 0u;  // of slots 2 and 3
                            const uint32_t v[4] = {gemm == 0 ? iw[0] & jv[0] : (gemm == 1 ? iw[0] : iw[2]) & jv[2],
                                                   gemm == 0 ? iw[0] & jv[1] : gemm == 1 ? iw[1] & jv[2] : 0u,
                                                   i2 & jv[0], i2 & jv[1]};
#pragma unroll
                            for (int k = 0; k < 4; ++k)
                                *reinterpret_cast<uint4*>(dst + (64 * u + 8 * k) * kMRow) = f4_expand_a(v[k], v[k]);
                        }
                        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
                        __syncwarp();
                        if (lane == 0) arrive_cl(full0 + 8 * sa);
                    }
                    if (++s == kMStages) {
                        s = 0;
                        par ^= 1;
                    }
                    if (++se == kMStages) {
                        se = 0;
                        pe ^= 1;
                    }
                    if (++sa == kMAStages) sa = 0;
                }
        }
    } else {
        asm volatile("setmaxnreg.inc.sync.aligned.u32 152;");
        // ---------------------------------------------------------------- epilogue (both CTAs)
        const int q = warp & 3, hh = (warp - 12) >> 2;  // lane quarter (8 j); its two warps take alternate 8 l
        const int lc = 2 * (lane & 3);
        const f2 inv_w = f2_dup(__uint_as_float((uint32_t)(127 - pack) << 23)), neg_w = f2_dup(-(float)(1 << pack));
        const f2 m23 = f2_dup(8388608.0f), neg_m23 = f2_dup(-8388608.0f);
        const f2 tiny = f2_dup(9.5367431640625e-07f);  // 2^-20: x lg2(x + tiny) = 0 at x = 0
        const uint32_t nc = (uint32_t)w.d.n_cases, nt = (uint32_t)w.d.n_ctrls;
        unsigned gemm = 0, item = 0;
        int wi = -1;
        for (long long g = g0 + cid; g < g1 && ok; g += ncl, ++item) {
            const T3mItem it = t3m_item(item_begin, n, g, wi);
            const int j = it.j0 + kMJ * (int)rank + 8 * q + (lane >> 2);
            long long thr = sink.thr;
            float thr_f = 0.f;
            if (sink.hist) thr = *(volatile long long*)sink.live;
            thr = __shfl_sync(0xffffffffu, thr, 0);
            if (!ALL) {
                float bound;
                live_tests(map, thr, thr_f, bound);
            }
            f2 kf[kPmG];                // estimates of the combinations (j, l) and (j, l + 1) of each group
            long long key[ALL ? kPmG : 1][2];
#pragma unroll
            for (int m = 0; m < kPmG; ++m) {
                kf[m] = 0;
                if (ALL) key[m][0] = key[m][1] = w.base_key;
            }
#pragma unroll 1
            for (int part = 0; part < 3 && ok; ++part, ++gemm) {
                const unsigned buf = gemm & 1, ph = (gemm >> 1) & 1;
                if (!t3_wait_cl(smem_u32(&acc_full[buf]), ph, abort)) {
                    ok = false;
                    break;
                }
                asm volatile("tcgen05.fence::after_thread_sync;");
#pragma unroll
                for (int m = 0; m < kPmG; ++m) {
                    if (m < it.ng) {
                        const int l = it.l0 + 8 * (2 * m + hh) + lc;
                        const bool v0 = j < n && l < n && l > j, v1 = j < n && l + 1 < n && l + 1 > j;
                        if (__any_sync(0xffffffffu, v0 || v1)) {
                            auto cell = [&](f2 D) {
                                const f2 b = f2_add(f2_fma_rz(D, inv_w, m23), neg_m23), a = f2_fma(neg_w, b, D);
                                if constexpr (ALL) {
                                    float x[2], y[2];
                                    f2_unpack(a, x[0], x[1]);
                                    f2_unpack(b, y[0], y[1]);
#pragma unroll
                                    for (int u = 0; u < 2; ++u)
                                        if (u ? v1 : v0) {
                                            const uint32_t ca = min(__float2uint_rn(x[u]), nc);
                                            const uint32_t cb = min(__float2uint_rn(y[u]), nt);
                                            key[m][u] += __ldg(w.d.ftab + ca) + __ldg(w.d.ftab + cb) -
                                                         __ldg(w.d.ftab + ca + cb);
                                        }
                                } else {
                                    auto lg = [](f2 v) {
                                        float x, y;
                                        f2_unpack(v, x, y);
                                        return f2_pack(t3_lg2(x), t3_lg2(y));
                                    };
                                    const f2 sab = f2_add(a, b);
                                    kf[m] = f2_fma(a, lg(f2_add(a, tiny)), kf[m]);
                                    kf[m] = f2_fma(b, lg(f2_add(b, tiny)), kf[m]);
                                    kf[m] = f2_sub(kf[m], f2_mul(sab, lg(f2_add(sab, tiny))));
                                }
                            };
#pragma unroll
                            for (int x = 0; x < 2; ++x) {
                                if (x && part == 2) break;
                                uint32_t r[12];  // 4 z + 2 (slot % 2) (l) and + 1 (l + 1)
                                const uint32_t at = tmem + ((uint32_t)(32 * q + 16 * x) << 16) +
                                                    (uint32_t)(kMN * buf + 24 * (2 * m + hh));
                                asm volatile(
                                    "tcgen05.ld.sync.aligned.16x256b.x2.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
                                    : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]),
                                      "=r"(r[6]), "=r"(r[7])
                                    : "r"(at));
                                asm volatile("tcgen05.ld.sync.aligned.16x256b.x1.b32 {%0,%1,%2,%3}, [%4];"
                                             : "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11])
                                             : "r"(at + 16));
                                asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
                                for (int e = 0; e < 6; ++e)
                                    if (!(e & 1) || part < 2)
                                        cell(f2_pack(__uint_as_float(r[2 * e]), __uint_as_float(r[2 * e + 1])));
                            }
                        }
                    }
                }
                asm volatile("tcgen05.fence::before_thread_sync;");
                __syncwarp();
                if (lane == 0) arrive_cl(cluster_addr(smem_u32(&acc_empty[buf]), 0));
            }
            if (!ok) break;
#pragma unroll
            for (int m = 0; m < kPmG; ++m) {
                const int l = it.l0 + 8 * (2 * m + hh) + lc;
                const bool v0 = m < it.ng && j < n && l < n && l > j, v1 = m < it.ng && j < n && l + 1 < n && l + 1 > j;
                const unsigned m0 = __ballot_sync(0xffffffffu, v0), m1 = __ballot_sync(0xffffffffu, v1);
                if (!(m0 | m1)) continue;
                if (sink.evaluated && lane == 0)
                    atomicAdd(sink.evaluated, (unsigned long long)(__popc(m0) + __popc(m1)));
                if constexpr (ALL) {
#pragma unroll
                    for (int u = 0; u < 2; ++u) {
                        const int cmb[3] = {it.i, j, l + u};
                        if ((u ? v1 : v0) && key[m][u] >= thr) live_append(sink, key[m][u], pack_code(cmb, 3, w.bits));
                    }
                } else {
                    float b0, b1;
                    f2_unpack(kf[m], b0, b1);
                    unsigned s0 = __ballot_sync(0xffffffffu, v0 && b0 >= thr_f);
                    unsigned s1 = __ballot_sync(0xffffffffu, v1 && b1 >= thr_f);
                    while (s0 | s1) {
                        const int u = s0 ? 0 : 1, src = __ffs(u ? s1 : s0) - 1;
                        if (u) s1 &= s1 - 1;
                        else s0 &= s0 - 1;
                        const int cmb[3] = {it.i, __shfl_sync(0xffffffffu, j, src), __shfl_sync(0xffffffffu, l, src) + u};
                        const long long ke = warp_exact_key<3>(&w.d, w.base_key, cmb[0], cmb[1], cmb[2], 0, sink.overflow);
                        if (lane == 0 && ke >= thr) live_append(sink, ke, pack_code(cmb, 3, w.bits));
                    }
                }
            }
            // the pairs take turns at raising the live threshold
            if (sink.hist && rank == 0 && warp == 12 && (item < 2 || ((item + cid) & 7) == 0)) live_update(sink, lane);
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

std::vector<long long> t3m_items(int n) {
    std::vector<long long> b((size_t)n + 1, 0);
    for (int i = 0; i < n; ++i) {
        long long c = 0;
        for (int j = i + 1; j < n - 1; j += kPmJ) c += t3m_tiles(n, j);
        b[i + 1] = b[i] + c;
    }
    return b;
}

cudaError_t f4_missing_maps(F4Plan& f, int snps) {
    cudaError_t e = tensor_map(&f.map_b, f.planes, f.rows, 16 * f.wpr, kMRow, kMN / 2, true);
    if (e == cudaSuccess) e = tensor_map(&f.map_b4h, f.planes, f.rows, 16 * f.wpr, kMRow, 24 * kMHalfG, true);
    if (e == cudaSuccess) e = f4_bit_map(&f.map_j, f, f.bits, 3 * snps, 3 * kMJ);
    if (e == cudaSuccess) e = f4_bit_map(&f.map_i, f, f.bits, 3 * snps, 3);
    return e;
}

cudaError_t launch_tensor3m(const ScanWork& w, const F4Plan& f, const long long* item_begin, long long g0, long long g1,
                            const CandSink& sink, double est_margin, int* status, cudaStream_t s, int sms) {
    if (!f.pack || !item_begin) return cudaErrorInvalidValue;
    // set once, by whichever host thread comes first (thread-safe static initialisation)
    static const cudaError_t attr = [] {
        cudaError_t e = cudaFuncSetAttribute(tensor3m_kernel<false>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                             (int)kMSmem);
        if (e == cudaSuccess)
            e = cudaFuncSetAttribute(tensor3m_kernel<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kMSmem);
        return e;
    }();
    if (attr != cudaSuccess) return attr;
    if (g1 <= g0) return cudaSuccess;
    static const int max_clusters = pair_clusters(tensor3m_kernel<false>, kMThreads, kMSmem);
    const long long clusters = std::min<long long>(g1 - g0, max_clusters > 0 ? max_clusters : sms / 2);
    const unsigned grid = (unsigned)(2 * std::max(1ll, clusters));
    const double scale = 1.0 / (std::log(2.0) * 4294967296.0);
    const LiveMap map{scale, -(double)w.base_key * scale - est_margin, 0, 0};
    const auto fn = sink.thr == (long long)0x8000000000000000ull ? tensor3m_kernel<true> : tensor3m_kernel<false>;
    fn<<<grid, kMThreads, kMSmem, s>>>(f.map_b, f.map_b4h, f.map_j, f.map_i, w, sink, item_begin, g0, g1, f.nw_c,
                                       f.nw_t, f.pack, map, status);
    count_launch();
    return cudaGetLastError();
}

}  // namespace fiu
