// Order-3 contingency tables on CTA pairs with 4-bit operands.
//
// For one-hot data the 8 core cells of a combination (i, j, l) -- genotypes
// x, y, z in {0, 1} -- are dot products over the samples of one class:
//     core[x][y][z] = sum_s a_ix(s) a_jy(s) a_lz(s),
// where a_gx(s) is 1 when sample s has genotype x at SNP g.
// A cluster of two CTAs (the two SMs of a TPC) runs one GEMM per work item
// (i, 64 j, up to 120 l):
//     D[(j,x,y), (l,z)] = sum_s A[(j,x,y), s] B[(l,z), s]    (M 256, N <= 240)
// with tcgen05.mma.cta_group::2.kind::mxf4, control samples weighted by W = 2^p
// through the B scale, so an accumulator holds cases + W controls of one core
// cell (classes too large to share one so: SPLIT, below).  CTA r builds the A rows of its 32 j and stages half r of the l rows;
// CTA 0 issues the MMAs; each CTA's 128 accumulator rows end up in its own
// tensor memory.  Two regions of 240 columns alternate between items, so the
// next item's GEMM runs while the epilogue evaluates the last one; the other 32
// columns hold the scales.
//
// Operands.  B rows are the data set's e2m1 planes (TMA, 128-byte swizzle, 256
// samples a stage).  A rows are built from bit rows (one bit a sample, a quarter
// of the planes' bytes): eight producer warps in two alternating groups AND the
// i and j words and spread the bits to nibbles straight into the swizzled A tile.
//
// Accumulator rows are ordered (j / 8, x, y, j % 8) and columns (l / 8, z, l % 8),
// so that two 16x256b tensor-memory loads give a thread all 8 cores of the
// combinations (j, l) and (j, l + 1), in neighbouring registers: no transpose
// through shared memory.
//
// Epilogue.  The 27 cells of both combinations follow from the packed cores and
// the packed marginals (pairs (i,j), (i,l), (j,l) and singles; every value an
// exact integer below 2^24) in two-wide single precision.  A quadratic bound on
// the MI (F4Bound) rejects nearly all of them; a warp with a survivor takes a
// logarithm estimate with a proven error bound and, for what passes that, the
// exact fixed-point key, so the kept set is the one of the exact key.
//
// What bounds it (2 000 SNPs x 4 000/4 000, one launch over the whole scan):
// 26.3 ms; without the evaluation 22.7, without the A build and the MMAs too
// 22.3 (about 540 cycles a stage; neither fewer bytes nor other copies a stage
// changed it); the MMAs alone are 18.6 (120 cycles per M 256 N 240 K 64).  Whole searches: 27.7 ms
// against 74.7 with e4m3 operands (128-byte rows of 128 samples: twice the shared-memory
// and L2 traffic, 82 KB a stage with LSU and tensor wavefronts at 83 % of peak;
// 81 logarithms a combination at 8 cycles a warp instruction and SM quarter where
// the bound takes about 21 reciprocals and 215 arithmetic cycles; a transpose
// through shared memory).  Tried on the way: A in tensor memory and B spread from
// bits by warps (5 KB a stage from L2, N 192): 45 ms, bound by issue slots.
//
// SPLIT (500 SNPs x 9 000/9 800): 5.6 -> 1.9 ms a search (kernels 1.6) against the e4m3 kernel, one CTA a
// tile, that counted classes apart before; 610 cycles a stage.
//
// Reference semantics: GenotypeTable::combine_and_popcnt for order 3
// (src/base/gt_popcnt.cpp:4-35) and MutualInformation::compute
// (src/base/mi_compute.cpp:16-41) over the combinations ThreadedSearch
// visits (include/fiuncho/ThreadedSearch.h:157-180) with one worker.
#include <algorithm>
#include <cmath>

#include "live.cuh"
#include "tensor3m.h"
#include "tensor_fp4.cuh"

namespace fiu {

constexpr int kXJ = kPxJ / 2;                       // j per CTA
constexpr int kXL = 8 * kPxG;                       // 120 l per item at most
constexpr int kXN = 2 * kXL;                        // columns of an accumulator region
constexpr int kXM = 4 * kXJ;                        // 128 accumulator rows per CTA
constexpr int kXRow = kF4K / 2;                     // 128 bytes per operand row and stage
constexpr int kXBitRow = kF4K / 8;                  // 32 bytes per bit row and stage
// Copies land in a ring of their own, deeper than the A ring (one ring of six
// stages, A beside what it is built from, kept the same pace: 27.1 against 26.9
// ms).  SPLIT has its stash in the space of the stages it lacks.
template <bool SPLIT>
constexpr int kXStages = SPLIT ? 5 : 8;
template <bool SPLIT>
constexpr int kXAStages = SPLIT ? 3 : 4;
constexpr int kXSA = kXM * kXRow;                   // 16 KB
constexpr int kXSB = kXN / 2 * kXRow;               // 15 KB: this CTA's half of the l rows
constexpr int kXSJ = 2 * kXJ * kXBitRow;            //  2 KB
constexpr int kXSI = 2 * kXBitRow;                  // 64 bytes
constexpr int kXStage = (kXSB + kXSJ + kXSI + 1023) / 1024 * 1024;  // 18 KB
constexpr int kXColOne = 2 * kXN, kXColW = kXColOne + 16;
// Builders in two groups that take alternate stages (a warp's chain of waits,
// loads, shifts, stores and arrival is longer than a stage's MMAs).
constexpr int kXBuildWarps = 4, kXEpiWarps = 8;     // builder warps per group
constexpr int kXThreads = 32 * (4 + 2 * kXBuildWarps + kXEpiWarps);  // 640: copies, MMAs, 2 staging, 8, 8
// registers a thread: 96 at launch, then 56 / 56 / 152 (3 x 56 + 2 x 152 <= 5 x 96)
constexpr int kXMeta = 16;                          // items in flight between the copies and the MMAs
// an item's staged tables: (i, l) marginals, one column per l; per j of this CTA (i, j) cores and j
// singles, each twice (both halves of a pair), and j; the threshold (key, estimate, bound).  SPLIT:
// cases and controls beside each other instead.
template <bool SPLIT>
constexpr int kXTabL = 9 * kXL * (SPLIT ? 8 : 4);
constexpr int kXTabJ = 6 * kXJ * 8;
template <bool SPLIT>
constexpr int kXTabT = kXTabL<SPLIT> + kXTabJ + 4 * kXJ;
template <bool SPLIT>
constexpr int kXTab = kXTabT<SPLIT> + 16;
constexpr int kXStash = kXEpiWarps * ((kPxG + 1) / 2) * 2 * 32 * 16;  // 64 KB: (warp, its group, x, lane), 8 counts
template <bool SPLIT>
constexpr size_t kXSmem = 1024 + (size_t)kXStages<SPLIT> * kXStage + (size_t)kXAStages<SPLIT> * kXSA +
                          2 * kXTab<SPLIT> + (SPLIT ? kXStash : 0);
static_assert(kXSmem<false> <= 227 * 1024 - 512 && kXSmem<true> <= 227 * 1024 - 512, "order-3 pair kernel shared memory");
static_assert(kXSA % 1024 == 0 && kXSB % 1024 == 0, "operand tiles on swizzle atoms");
static_assert(kXColW + 16 <= 512, "tensor memory columns");
static_assert(kXStages<false> < kXMeta, "an item has a stage at least");

// One item: (i, j0 ..), l-tile of ng groups of 8 from l0.  LIST (a Distribution
// layer): p0 is the first listed j instead of j0.
struct T3xItem {
    int i, j0, l0, ng;
    long long p0;
};

// Item g; i is the walker's position (the items of one walker ascend).
template <bool LIST>
__device__ __forceinline__ T3xItem t3x_item(const long long* __restrict__ item_begin,
                                            const long long* __restrict__ jl_begin, const int* __restrict__ jlist,
                                            int n, long long g, int& i) {
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
    T3xItem it;
    it.i = i;
    int q = (int)(g - __ldg(item_begin + i));
    long long p = LIST ? __ldg(jl_begin + i) : 0;
    for (int j = LIST ? __ldg(jlist + p) : i + 1;;) {
        const int nl = t3x_tiles(n, j);
        if (q < nl) {
            const int G = t3x_groups(n, j), a = G * q / nl, b = G * (q + 1) / nl;
            it.j0 = j;
            it.p0 = p;
            it.l0 = ((j + 1) & ~7) + 8 * a;
            it.ng = b - a;
            return it;
        }
        q -= nl;
        if (LIST) {
            p += kPxJ;
            j = __ldg(jlist + p);
        } else {
            j += kPxJ;
        }
    }
}

// Packed float c + W t of the counts of both classes.
__device__ __forceinline__ float t3x_pk(uint32_t c, uint32_t t, float W) { return fmaf(W, u2f(t), u2f(c)); }
// Entry (x, y) of the pair cores v, packed.
__device__ __forceinline__ float t3x_pair(const uint4& v, int x, int y, float W) {
    const uint32_t c = x ? v.y : v.x, t = x ? v.w : v.z;
    return t3x_pk(y ? c >> 16 : c & 0xffffu, y ? t >> 16 : t & 0xffffu, W);
}

// Both classes' counts of a pair core beside each other (SPLIT).
__device__ __forceinline__ f2 t3x_pair_ab(const uint4& v, int x, int y) {
    return f4_ab(x ? v.y : v.x, x ? v.w : v.z, y);
}

// Its inverse: cases | controls << 16.
__device__ __forceinline__ uint32_t t3x_word(f2 v) {
    float a, b;
    f2_unpack(f2_add(v, f2_dup(8388608.0f)), a, b);
    return __byte_perm(__float_as_uint(a), __float_as_uint(b), 0x5410);
}

// The 27 cells of a combination from its cores c (x, y, z), the (i, j) cores, the
// marginal table il(x, z) of (i, l), the (j, l) cores and the j singles; T is one
// value or two side by side.  use(e, q, cell): the e-th cell made, (x, y, z) at
// q = (x*3+y)*3+z.
__device__ __forceinline__ f2 t3x_less(f2 a, f2 b, f2 c) { return f2_sub(f2_sub(a, b), c); }
__device__ __forceinline__ float t3x_less(float a, float b, float c) { return a - b - c; }
template <class T, class IL, class Use>
__device__ __forceinline__ void t3x_cells(const T (&c)[2][2][2], const T (&ij)[2][2], IL&& il, const T (&jl)[2][2],
                                          const T (&sj)[2], Use&& use) {
    T a[2][2][3], y2[2][3];  // cells (x, y, z); cells (2, y, z)
#pragma unroll
    for (int x = 0; x < 2; ++x)
#pragma unroll
        for (int y = 0; y < 2; ++y) {
            a[x][y][0] = c[x][y][0];
            a[x][y][1] = c[x][y][1];
            a[x][y][2] = t3x_less(ij[x][y], c[x][y][0], c[x][y][1]);
#pragma unroll
            for (int z = 0; z < 3; ++z) use(6 * x + 3 * y + z, 9 * x + 3 * y + z, a[x][y][z]);
        }
#pragma unroll
    for (int x = 0; x < 2; ++x)
#pragma unroll
        for (int z = 0; z < 3; ++z) use(12 + 3 * x + z, 9 * x + 6 + z, t3x_less(il(x, z), a[x][0][z], a[x][1][z]));
#pragma unroll
    for (int y = 0; y < 2; ++y) {
        const T j2 = t3x_less(sj[y], jl[y][0], jl[y][1]);
#pragma unroll
        for (int z = 0; z < 3; ++z) {
            y2[y][z] = t3x_less(z < 2 ? jl[y][z & 1] : j2, a[0][y][z], a[1][y][z]);
            use(18 + 3 * y + z, 18 + 3 * y + z, y2[y][z]);
        }
    }
#pragma unroll
    for (int z = 0; z < 3; ++z) use(24 + z, 24 + z, t3x_less(il(2, z), y2[0][z], y2[1][z]));
}

// Counts of both classes of a cell: packed, or beside each other.
__device__ __forceinline__ void t3x_counts(float t, int pack, uint32_t& a, uint32_t& b) {
    const uint32_t u = __float2uint_rn(t);
    a = u & ((1u << pack) - 1u);
    b = u >> pack;
}
__device__ __forceinline__ void t3x_counts(f2 t, int, uint32_t& a, uint32_t& b) {
    float x, y;
    f2_unpack(t, x, y);
    a = __float2uint_rn(x);
    b = __float2uint_rn(y);
}

// The rare path (lanes with want): from the 27 cells t[(x*3+y)*3+z] of
// combination (i, j, l), the bounded single-precision estimate of the key
// (t3_margin), the exact fixed-point key for what passes it, and the
// warp-aggregated append of candidates.  Warp-synchronous.
template <class T>
__device__ __forceinline__ void t3x_survivor(const ScanWork& w, const CandSink& sink, long long thr, float thr_f,
                                             uint32_t* dump, const T (&t)[27], int pack, int i, int j, int l,
                                             bool want, int lane) {
    const int n = w.d.snps;
    bool cand = want;
    if (!dump && !sink.digest && thr != (long long)0x8000000000000000ull) {
        const float tiny = 9.5367431640625e-07f;  // 2^-20: x*lg2(x + tiny) = 0 at x = 0
        float kf = 0.f;
#pragma unroll
        for (int c = 0; c < 27; ++c) {
            uint32_t ua, ub;
            t3x_counts(t[c], pack, ua, ub);
            const float a = u2f(ua), b = u2f(ub), s = a + b;
            kf = fmaf(a, t3_lg2(a + tiny), kf);
            kf = fmaf(b, t3_lg2(b + tiny), kf);
            kf = fmaf(-s, t3_lg2(s + tiny), kf);
        }
        cand = want && kf >= thr_f;
    }
    if (!__any_sync(0xffffffffu, cand)) return;
    long long key = w.base_key;
    unsigned long long dg = 0;
    if (cand) {
        const uint32_t nc = (uint32_t)w.d.n_cases, nt = (uint32_t)w.d.n_ctrls;
        // owned prefix ordinal m of (i, j): rank offset + m * step
        uint32_t* o =
            dump ? dump + ((size_t)((pair_index(i, j, n) - w.dist_offset) / w.dist_step) * n + l) * 54 : nullptr;
        if (sink.digest) {
            const int cmb[3] = {i, j, l};
            dg = dg_begin(cmb, 3, n);
        }
#pragma unroll
        for (int c = 0; c < 27; ++c) {
            uint32_t ua, ub;
            t3x_counts(t[c], pack, ua, ub);
            const uint32_t a = min(ua, nc), b = min(ub, nt);
            key += __ldg(w.d.ftab + a) + __ldg(w.d.ftab + b) - __ldg(w.d.ftab + a + b);
            if (o) {
                o[c] = ua;
                o[27 + c] = ub;
            }
            if (sink.digest) dg = dg_cell(dg, ua, ub);
        }
    }
    if (sink.digest) dg_warp_add(sink.digest, dg);
    const bool pass = cand && key >= thr;
    const unsigned pm = __ballot_sync(0xffffffffu, pass);
    if (!pm) return;
    const int leader = __ffs(pm) - 1;
    unsigned base = 0;
    if (lane == leader) base = atomicAdd(sink.count, (unsigned)__popc(pm));
    base = __shfl_sync(0xffffffffu, base, leader);
    if (pass) {
        const unsigned idx = base + __popc(pm & ((1u << lane) - 1u));
        if (idx < sink.cap) {
            const int cmb[3] = {i, j, l};
            sink.buf[idx] = Cand{key, pack_code(cmb, 3, w.bits)};
            if (sink.hist) atomicAdd(sink.hist + live_bin(key), 1u);
        } else {
            atomicOr(sink.overflow, 1u);
        }
    }
}

// Columns the MMA of an item of ng groups multiplies (at least 64).
__device__ __forceinline__ int t3x_n(int ng) { return 16 * max(ng, 4); }

// What a launch does with the accumulators: search a data set or one Distribution layer of it, or
// store the cores of every triple (F4Plan::tri).
enum { kXScan, kXLayer, kXCores };

// SPLIT: classes that do not share an accumulator: the cases of an item accumulate in one region and
// its controls in the other; the epilogue packs the case counts to 16 bits in shared memory as soon as
// their GEMM is done, so the next item's case GEMM runs while this item's controls are evaluated.
template <int MODE, bool SPLIT>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(kXThreads, 1)
    tensor3x_kernel(const __grid_constant__ CUtensorMap map_b, const __grid_constant__ CUtensorMap map_j,
                    const __grid_constant__ CUtensorMap map_i, const __grid_constant__ ScanWork w,
                    const __grid_constant__ CandSink sink, const long long* __restrict__ item_begin, long long g0,
                    long long g1, int nw_c, int nw_t, int pack, const __grid_constant__ LiveMap map, uint32_t* dump,
                    const uint32_t* __restrict__ single, const uint4* __restrict__ pairs, int* status,
                    const long long* __restrict__ jl_begin, const int* __restrict__ jlist, float* tri,
                    const int* __restrict__ row_p, const int* __restrict__ row_q) {
    constexpr bool LIST = MODE == kXLayer;
    constexpr int kStages = kXStages<SPLIT>, kAStages = kXAStages<SPLIT>;
    extern __shared__ uint8_t smraw[];
    __shared__ __align__(8) uint64_t full_t[kStages], empty[kStages], full_a[kAStages];
    __shared__ __align__(8) uint64_t acc_full[2], acc_empty[2], tab_full[2], tab_empty[2], done;
    __shared__ uint32_t tmem_base;
    __shared__ int item_ng[kXMeta];  // groups of the items in flight, for the MMA issuer
    __shared__ int abort_flag;
    uint8_t* sm = (uint8_t*)(((uintptr_t)smraw + 1023) & ~(uintptr_t)1023);  // stages: B half | j | i; then the A tiles
    uint8_t* sma = sm + kStages * kXStage;
    uint8_t* tabs = sma + kAStages * kXSA;
    uint4* stash = reinterpret_cast<uint4*>(tabs + 2 * kXTab<SPLIT>);
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
            init(&full_t[s], 1);
            init(&empty[s], 1);
        }
        for (int s = 0; s < kAStages; ++s) init(&full_a[s], 2 * kXBuildWarps);
        for (int b = 0; b < 2; ++b) {
            init(&acc_full[b], 1);
            init(&acc_empty[b], 2 * kXEpiWarps);
            init(&tab_full[b], 2);
            init(&tab_empty[b], kXEpiWarps);
        }
        init(&done, 1);
        asm volatile("fence.mbarrier_init.release.cluster;");
        abort_flag = 0;
    }
    asm volatile("tcgen05.fence::before_thread_sync;");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;");
    const uint32_t tmem = tmem_base;
    if (warp >= 4 && warp < 8) f4_fill_scales<16>(tmem, warp & 3, kXColOne, kXColW, pack);
    asm volatile("tcgen05.fence::before_thread_sync;");
    __syncthreads();
    cluster_sync_all();  // both CTAs' barriers and scales exist before either signals the other
    asm volatile("tcgen05.fence::after_thread_sync;");
    bool ok = true;

    // (the register limits are set inside the branches: set before them, the
    // compiler would hold every branch to the smallest)
    if (warp < 4) {
        asm volatile("setmaxnreg.dec.sync.aligned.u32 56;");
        if (warp == 0) {
            // ---------------------------------------------------------------- TMA producer (both CTAs)
            if (g0 + cid < g1 && elect_one()) {
                unsigned s = 0, par = 1;  // stage and the parity its last release has (first round: free)
                unsigned step = 0, item = 0;
                int wi = -1;
                T3xItem it = t3x_item<LIST>(item_begin, jl_begin, jlist, n, g0 + cid, wi);
                for (long long g = g0 + cid; g < g1 && ok; g += ncl) {
                    int jr = it.j0 + kXJ * (int)rank;  // row (SNP position) of this CTA's first j
                    if (LIST) {
                        // 32 listed j are consecutive residue-ordered rows from the first one (rows past the
                        // end of i's list are loaded too and ignored by the epilogue)
                        const long long p = it.p0 + kXJ * (int)rank;
                        jr = p < __ldg(jl_begin + it.i + 1) ? residue_row(__ldg(jlist + p), layer_step(w.dist_step, n), n) : 0;
                    }
                    const int brow = 2 * it.l0 + t3x_n(it.ng) / 2 * (int)rank, irow = 2 * it.i;
                    item_ng[item++ % kXMeta] = it.ng;
                    T3xItem nx = it;
                    for (int ks = 0; ks < ksteps; ++ks) {
                        if (!t3_wait_cl(smem_u32(&empty[s]), par, abort)) {
                            ok = false;
                            break;
                        }
                        const uint32_t st = smem_u32(sm + s * kXStage), bar = smem_u32(&full_t[s]);
                        asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar),
                                     "r"((uint32_t)(kXSB + kXSJ + kXSI))
                                     : "memory");
                        t3_tma(st + kXSB, &map_j, kXBitRow * ks, 2 * jr, bar);
                        t3_tma(st + kXSB + kXSJ, &map_i, kXBitRow * ks, irow, bar);
                        t3_tma(st, &map_b, kXRow * ks, brow, bar);
                        if (step < kStages) ++step;
                        if (++s == kStages) {
                            s = 0;
                            par ^= 1;
                        }
                        // the next item's place is looked up while this item's copies are in flight
                        if (ks == 0 && g + ncl < g1) nx = t3x_item<LIST>(item_begin, jl_begin, jlist, n, g + ncl, wi);
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
                ok = f4_pair_issue<SPLIT, kAStages, kXSA, kStages, kXStage, kXN, kXColOne, kXColW>(
                    (g1 - g0 - cid + ncl - 1) / ncl, smem_u32(sma), smem_u32(sm), smem_u32(&full_a[0]),
                    smem_u32(&empty[0]), smem_u32(&acc_full[0]), smem_u32(&acc_empty[0]), tmem, nw_c, nw_t, abort,
                    [&](unsigned item) { return t3x_n(item_ng[item % kXMeta]); });
                commit_pair(smem_u32(&done));
                // neither CTA releases shared or tensor memory before the pair's MMAs are
                // done (CTA 1 waits once its own work is over, below: waiting here would
                // span its whole launch, longer than the bound on a single wait)
                if (!t3_drain_cl(smem_u32(&done), 0)) ok = false;
            }
            __syncwarp();
        } else if (MODE != kXCores) {
            // ---------------------------------------------------------------- table staging (both CTAs)
            const int t = tid - 64;  // 0 .. 63
            const float W = (float)(1u << pack);
            const float ntot = fmaf(W, (float)w.d.n_ctrls, (float)w.d.n_cases);
            const uint4* single4 = reinterpret_cast<const uint4*>(single);
            unsigned item = 0;
            int wi = -1;
            for (long long g = g0 + cid; g < g1 && ok; g += ncl, ++item) {
                const T3xItem it = t3x_item<LIST>(item_begin, jl_begin, jlist, n, g, wi);
                const unsigned buf = item & 1;
                if (item >= 2 && !t3_wait(smem_u32(&tab_empty[buf]), ((item >> 1) - 1) & 1, abort)) {
                    ok = false;
                    break;
                }
                uint8_t* tab = tabs + buf * kXTab<SPLIT>;
                const int i = it.i;
                const uint4 s1 = __ldg(single4 + i);
                // the threshold of this item (the pairs take turns at raising the live one)
                if (sink.hist && rank == 0 && warp == 2 && item > 0 && (item < 3 || ((item + cid) & 7) == 0))
                    live_update(sink, lane);
                if (t == 0) {
                    const long long thr = sink.hist ? *(volatile long long*)sink.live : sink.thr;
                    float est, bound;
                    live_tests(map, thr, est, bound);
                    *reinterpret_cast<long long*>(tab + kXTabT<SPLIT>) = thr;
                    *reinterpret_cast<float2*>(tab + kXTabT<SPLIT> + 8) = make_float2(est, bound);
                }
                for (int ll = t; ll < 8 * it.ng; ll += 64) {  // entries (x, z), x and z in {0, 1, any}
                    const int l = it.l0 + ll;
                    uint4 p = make_uint4(0, 0, 0, 0), sl = p;
                    if (l < n && l > i) {
                        p = __ldg(pairs + pair_index(i, l, n));
                        sl = __ldg(single4 + l);
                    }
                    if constexpr (SPLIT) {
                        f2* tl = reinterpret_cast<f2*>(tab);
                        f2 m[3][3];
#pragma unroll
                        for (int x = 0; x < 2; ++x) {
#pragma unroll
                            for (int z = 0; z < 2; ++z) m[x][z] = t3x_pair_ab(p, x, z);
                            m[x][2] = t3x_less(f4_ab(x ? s1.y : s1.x, x ? s1.w : s1.z, 0), m[x][0], m[x][1]);
                        }
#pragma unroll
                        for (int z = 0; z < 2; ++z)
                            m[2][z] = t3x_less(f4_ab(z ? sl.y : sl.x, z ? sl.w : sl.z, 0), m[0][z], m[1][z]);
                        m[2][2] = t3x_less(t3x_less(f2_pack((float)w.d.n_cases, (float)w.d.n_ctrls),
                                                    f4_ab(s1.x, s1.z, 0), f4_ab(s1.y, s1.w, 0)),
                                           m[2][0], m[2][1]);
#pragma unroll
                        for (int k = 0; k < 9; ++k) tl[k * kXL + ll] = m[k / 3][k % 3];
                    } else {
                        float* tl = reinterpret_cast<float*>(tab);
                        float m[3][3];
#pragma unroll
                        for (int x = 0; x < 2; ++x) {
#pragma unroll
                            for (int z = 0; z < 2; ++z) m[x][z] = t3x_pair(p, x, z, W);
                            m[x][2] = t3x_pk(x ? s1.y : s1.x, x ? s1.w : s1.z, W) - m[x][0] - m[x][1];
                        }
#pragma unroll
                        for (int z = 0; z < 2; ++z)
                            m[2][z] = t3x_pk(z ? sl.y : sl.x, z ? sl.w : sl.z, W) - m[0][z] - m[1][z];
                        m[2][2] = ntot - t3x_pk(s1.x, s1.z, W) - t3x_pk(s1.y, s1.w, W) - m[2][0] - m[2][1];
#pragma unroll
                        for (int k = 0; k < 9; ++k) tl[k * kXL + ll] = m[k / 3][k % 3];
                    }
                }
                if (t < kXJ) {
                    int j = n;
                    if (LIST) {
                        const long long p = it.p0 + kXJ * (int)rank + t;
                        if (p < __ldg(jl_begin + i + 1)) j = __ldg(jlist + p);
                    } else {
                        j = it.j0 + kXJ * (int)rank + t;
                    }
                    uint4 p = make_uint4(0, 0, 0, 0), sv = p;
                    if (j < n) {
                        p = __ldg(pairs + pair_index(i, j, n));
                        sv = __ldg(single4 + j);
                    }
                    f2* tj = reinterpret_cast<f2*>(tab + kXTabL<SPLIT>);
#pragma unroll
                    for (int k = 0; k < 6; ++k) {
                        if constexpr (SPLIT)
                            tj[k * kXJ + t] = k < 4 ? t3x_pair_ab(p, k >> 1, k & 1)
                                                    : f4_ab(k & 1 ? sv.y : sv.x, k & 1 ? sv.w : sv.z, 0);
                        else
                            tj[k * kXJ + t] = f2_dup(k < 4 ? t3x_pair(p, k >> 1, k & 1, W)
                                                           : t3x_pk(k & 1 ? sv.y : sv.x, k & 1 ? sv.w : sv.z, W));
                    }
                    reinterpret_cast<int*>(tab + kXTabL<SPLIT> + kXTabJ)[t] = j;
                }
                __syncwarp();
                if (lane == 0)
                    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(&tab_full[buf])) : "memory");
            }
        }
    } else if (warp < 12) {
        asm volatile("setmaxnreg.dec.sync.aligned.u32 56;");
        // ---------------------------------------------------------------- A builders (both CTAs)
        // thread: 16-byte chunk c (32 samples) of the j rows rg, rg + 16, .. of every second stage
        const int t = (tid - 128) & (32 * kXBuildWarps - 1), c = t & 7, rg = t >> 3;
        const uint32_t full0 = cluster_addr(smem_u32(&full_a[0]), 0);
        // A row (jj / 8, x, y, jj % 8) of staged row (jj, y) = rg + 16 u; x = 1 is 16 rows on, u + 1 32 rows
        const int jj = rg >> 1, y = rg & 1;
        const int dst0 = (8 * y + jj) * kXRow + ((c ^ jj) << 4);
        unsigned s = 0, par = 0, sa = 0;                  // copy stage, A stage
        unsigned se = kStages - kAStages, pe = 1;       // the stage whose MMAs free this A stage
        bool mine = warp < 8;
        for (long long g = g0 + cid; g < g1 && ok; g += ncl) {
            for (int ks = 0; ks < ksteps; ++ks, mine = !mine) {
                if (mine) {
                    if (!t3_wait(smem_u32(&full_t[s]), par, abort)) {
                        ok = false;
                        break;
                    }
                    const uint32_t* sJ = reinterpret_cast<const uint32_t*>(sm + s * kXStage + kXSB) + rg * 8 + c;
                    const uint32_t* sI = reinterpret_cast<const uint32_t*>(sm + s * kXStage + kXSB + kXSJ) + c;
                    uint32_t jw[4];
#pragma unroll
                    for (int u = 0; u < 4; ++u) jw[u] = sJ[128 * u];
                    const uint32_t i0 = sI[0], i1 = sI[8];
                    if (!t3_wait_cl(smem_u32(&empty[se]), pe, abort)) {
                        ok = false;
                        break;
                    }
                    uint8_t* dst = sma + sa * kXSA + dst0;
#pragma unroll
                    for (int u = 0; u < 4; ++u) {
                        *reinterpret_cast<uint4*>(dst + 32 * u * kXRow) = f4_expand_a(i0, jw[u]);
                        *reinterpret_cast<uint4*>(dst + (32 * u + 16) * kXRow) = f4_expand_a(i1, jw[u]);
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
        const int q = warp & 3, hh = (warp - 12) >> 2;  // lane quarter (8 j); the two warps of a quarter take alternate groups
        const int jl = lane >> 2, lc = 2 * (lane & 3);  // this thread's j and its two l of a group
        const float W = (float)(1u << pack);
        const bool all = dump != nullptr || sink.digest != nullptr;  // every combination takes the exact path
        uint4* mine = stash + (warp - 12) * ((kPxG + 1) / 2) * 64 + lane;  // written and read by this warp only
        unsigned item = 0;
        int wi = -1;
        for (long long g = g0 + cid; g < g1 && ok; g += ncl, ++item) {
            const T3xItem it = t3x_item<LIST>(item_begin, jl_begin, jlist, n, g, wi);
            const int i = it.i, l0 = it.l0, ng = it.ng;
            const unsigned buf = item & 1, ph = (item >> 1) & 1;
            const uint8_t* tab = tabs + buf * kXTab<SPLIT>;
            const int gi0 = (hh + item) & 1;  // the odd group of an item goes to either warp in turn
            // accumulators of one x: registers 4 z + 2 y (l) and + 1 (l + 1): lane block y, 8-column block z
            auto ld = [&](int region, int x, int gi, uint32_t (&r)[8]) {
                asm volatile(
                    "tcgen05.ld.sync.aligned.16x256b.x2.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
                    : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
                    : "r"(tmem + ((uint32_t)(32 * q + 16 * x) << 16) + (uint32_t)(kXN * region + 16 * gi)));
            };
            if (SPLIT) {
                // case counts -> 16 bits in shared memory (l | l + 1 << 16); their region is then free
                if (!t3_wait_cl(smem_u32(&acc_full[0]), item & 1, abort)) {
                    ok = false;
                    break;
                }
                asm volatile("tcgen05.fence::after_thread_sync;");
#pragma unroll 1
                for (int gi = gi0; gi < ng; gi += 2) {
                    uint32_t r[2][8];
                    ld(0, 0, gi, r[0]);
                    ld(0, 1, gi, r[1]);
                    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
                    for (int x = 0; x < 2; ++x) {
                        uint32_t o[4];  // 2 z + y
#pragma unroll
                        for (int k = 0; k < 4; ++k)
                            o[k] = __byte_perm(__float_as_uint(__uint_as_float(r[x][2 * k]) + 8388608.0f),
                                               __float_as_uint(__uint_as_float(r[x][2 * k + 1]) + 8388608.0f), 0x5410);
                        mine[((gi >> 1) * 2 + x) * 32] = make_uint4(o[0], o[1], o[2], o[3]);
                    }
                }
                asm volatile("tcgen05.fence::before_thread_sync;");
                __syncwarp();
                if (lane == 0) arrive_cl(cluster_addr(smem_u32(&acc_empty[0]), 0));
            }
            if (MODE != kXCores && !t3_wait(smem_u32(&tab_full[buf]), ph, abort)) {
                ok = false;
                break;
            }
            const int j = MODE == kXCores ? it.j0 + kXJ * (int)rank + 8 * q + jl
                                          : reinterpret_cast<const int*>(tab + kXTabL<SPLIT> + kXTabJ)[8 * q + jl];
            const bool j_ok = j < n;
            const f2* tj = reinterpret_cast<const f2*>(tab + kXTabL<SPLIT>) + 8 * q + jl;
            const f2 ij[2][2] = {{tj[0], tj[kXJ]}, {tj[2 * kXJ], tj[3 * kXJ]}}, sj[2] = {tj[4 * kXJ], tj[5 * kXJ]};
            const long long thr = *reinterpret_cast<const long long*>(tab + kXTabT<SPLIT>);
            const float thr_f = reinterpret_cast<const float*>(tab + kXTabT<SPLIT>)[2];
            const float thr_q = reinterpret_cast<const float*>(tab + kXTabT<SPLIT>)[3];
            const uint4* pj = j_ok ? pairs + pair_index(j, j + 1, n) - (j + 1) : pairs;  // + l: pair (j, l)
            const uint4 zero4 = make_uint4(0, 0, 0, 0);
            uint4 pa = zero4, pb = zero4;
            {
                const int l = l0 + 8 * gi0 + lc;
                if (MODE != kXCores && j_ok && gi0 < ng && l < n && l > j) pa = __ldg(pj + l);
                if (MODE != kXCores && j_ok && gi0 < ng && l + 1 < n && l + 1 > j) pb = __ldg(pj + l + 1);
            }
            if (!t3_wait_cl(smem_u32(&acc_full[SPLIT ? 1 : buf]), SPLIT ? item & 1 : ph, abort)) {
                ok = false;
                break;
            }
            asm volatile("tcgen05.fence::after_thread_sync;");
#pragma unroll 1
            for (int gi = gi0; gi < ng; gi += 2) {
                const int l = l0 + 8 * gi + lc;
                const bool v0 = j_ok && l < n && l > j, v1 = j_ok && l + 1 < n && l + 1 > j;
                const uint4 ca = pa, cb = pb;
                {  // the next group's (j, l) pairs, ahead of their use
                    const int ln = l + 16;
                    pa = pb = zero4;
                    if (MODE != kXCores && j_ok && gi + 2 < ng && ln < n && ln > j) pa = __ldg(pj + ln);
                    if (MODE != kXCores && j_ok && gi + 2 < ng && ln + 1 < n && ln + 1 > j) pb = __ldg(pj + ln + 1);
                }
                const unsigned m0 = __ballot_sync(0xffffffffu, v0), m1 = __ballot_sync(0xffffffffu, v1);
                if (!(m0 | m1)) continue;
                if (sink.evaluated && lane == 0)
                    atomicAdd(sink.evaluated, (unsigned long long)(__popc(m0) + __popc(m1)));
                uint32_t r[2][8];
                ld(SPLIT ? 1 : buf, 0, gi, r[0]);
                ld(SPLIT ? 1 : buf, 1, gi, r[1]);
                asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
                if constexpr (SPLIT) {
                    // one combination at a time, both classes side by side
#pragma unroll 1
                    for (int u = 0; u < 2; ++u) {
                        f2 c[2][2][2];
#pragma unroll
                        for (int x = 0; x < 2; ++x) {
                            const uint4 sv = mine[((gi >> 1) * 2 + x) * 32];
#pragma unroll
                            for (int y = 0; y < 2; ++y)
#pragma unroll
                                for (int z = 0; z < 2; ++z) {
                                    const uint32_t o = (&sv.x)[2 * z + y];
                                    c[x][y][z] = f2_pack(
                                        __uint_as_float(__byte_perm(o, 0x4B000000u, u ? 0x7632 : 0x7610)) - 8388608.0f,
                                        __uint_as_float(u ? r[x][4 * z + 2 * y + 1] : r[x][4 * z + 2 * y]));
                                }
                        }
                        const bool valid = u ? v1 : v0;
                        if constexpr (MODE == kXCores) {  // entries (x, y, z), cases | controls << 16: 32 bytes a triple
                            if (valid) {
                                uint4* o = reinterpret_cast<uint4*>(tri) +
                                           4 * (size_t)(__ldg(row_q + i) + __ldg(row_p + j) + (l >> 1)) + 2 * u;
#pragma unroll
                                for (int x = 0; x < 2; ++x)
                                    o[x] = make_uint4(t3x_word(c[x][0][0]), t3x_word(c[x][0][1]), t3x_word(c[x][1][0]),
                                                      t3x_word(c[x][1][1]));
                            }
                        } else {
                            const f2* tl = reinterpret_cast<const f2*>(tab) + 8 * gi + lc + u;
                            auto il = [&](int x, int z) { return tl[(3 * x + z) * kXL]; };
                            const uint4 cj = u ? cb : ca;
                            f2 jl2[2][2];
#pragma unroll
                            for (int y = 0; y < 2; ++y)
#pragma unroll
                                for (int z = 0; z < 2; ++z) jl2[y][z] = t3x_pair_ab(cj, y, z);
                            F4BoundAB bd;
                            t3x_cells<f2>(c, ij, il, jl2, sj, [&](int, int, f2 cell) { bd.one(cell); });
                            const bool want = valid && (all || bd.acc >= thr_q);
                            if (!__any_sync(0xffffffffu, want)) continue;
                            f2 t[27];
                            t3x_cells<f2>(c, ij, il, jl2, sj, [&](int, int k, f2 cell) { t[k] = cell; });
                            t3x_survivor(w, sink, thr, thr_f, dump, t, pack, i, j, l + u, want, lane);
                        }
                    }
                } else {
                    f2 c[2][2][2];  // [x][y][z], the two combinations side by side
#pragma unroll
                    for (int x = 0; x < 2; ++x)
#pragma unroll
                        for (int y = 0; y < 2; ++y)
#pragma unroll
                            for (int z = 0; z < 2; ++z)
                                c[x][y][z] = f2_pack(__uint_as_float(r[x][4 * z + 2 * y]),
                                                     __uint_as_float(r[x][4 * z + 2 * y + 1]));
                    if constexpr (MODE == kXCores) {  // entries (x, y, z) of l and l + 1 side by side, 64 bytes
                        if (v0 || v1) {
                            float4* o = reinterpret_cast<float4*>(tri) +
                                        4 * (size_t)(__ldg(row_q + i) + __ldg(row_p + j) + (l >> 1));
#pragma unroll
                            for (int k = 0; k < 4; ++k) {
                                float4 t;
                                f2_unpack(c[k >> 1][k & 1][0], t.x, t.y);
                                f2_unpack(c[k >> 1][k & 1][1], t.z, t.w);
                                o[k] = t;
                            }
                        }
                    } else {
                        const float* tl = reinterpret_cast<const float*>(tab) + 8 * gi + lc;
                        f2 jl2[2][2];
#pragma unroll
                        for (int y = 0; y < 2; ++y)
#pragma unroll
                            for (int z = 0; z < 2; ++z) jl2[y][z] = f2_pack(t3x_pair(ca, y, z, W), t3x_pair(cb, y, z, W));
                        F4Bound bd(pack);
                        f2 prev = 0;
                        t3x_cells<f2>(
                            c, ij, [&](int x, int z) { return *reinterpret_cast<const f2*>(tl + (3 * x + z) * kXL); },
                            jl2, sj, [&](int e, int, f2 cell) {  // the first twelve cells share reciprocals
                                if (e >= 12) bd.one(cell);
                                else if (e & 1) bd.two(prev, cell);
                                else prev = cell;
                            });
                        float b0, b1;
                        f2_unpack(bd.acc, b0, b1);
                        const bool w0 = v0 && (all || b0 >= thr_q), w1 = v1 && (all || b1 >= thr_q);
                        if (!__any_sync(0xffffffffu, w0 || w1)) continue;
#pragma unroll 1
                        for (int u = 0; u < 2; ++u) {
                            const bool want = u ? w1 : w0;
                            if (!__any_sync(0xffffffffu, want)) continue;
                            // the combination's cells again, one lane of each pair
                            auto at = [&](f2 v) {
                                float lo, hi;
                                f2_unpack(v, lo, hi);
                                return u ? hi : lo;
                            };
                            const uint4 cj = u ? cb : ca;
                            float c1[2][2][2], ij1[2][2], jl1[2][2], t[27];
#pragma unroll
                            for (int x = 0; x < 2; ++x)
#pragma unroll
                                for (int y = 0; y < 2; ++y) {
                                    c1[x][y][0] = at(c[x][y][0]);
                                    c1[x][y][1] = at(c[x][y][1]);
                                    ij1[x][y] = at(ij[x][y]);
                                    jl1[x][y] = t3x_pair(cj, x, y, W);
                                }
                            const float sj1[2] = {at(sj[0]), at(sj[1])};
                            t3x_cells<float>(
                                c1, ij1, [&](int x, int z) { return tl[(3 * x + z) * kXL + u]; }, jl1, sj1,
                                [&](int, int k, float cell) { t[k] = cell; });
                            t3x_survivor(w, sink, thr, thr_f, dump, t, pack, i, j, l + u, want, lane);
                        }
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

// ---------------------------------------------------------------------------
// Operand layout of a data set, 32 samples of an SNP's genotype row g < G per thread: the bit
// rows G snp + g hold the class's words of the reference layout, cases then controls, each class
// padded to a multiple of 256 samples; the planes hold the same bits spread to e2m1 in rows
// 8 G (snp / 8) + 8 g + snp % 8, SNPs past the last one zero.
template <int G>
__global__ void f4_layout_kernel(DevData d, uint32_t* bits, uint4* planes, int wpr, int wc, int nc32, int nt32,
                                 int rows) {
    const size_t per_snp = 3 * (size_t)(d.cw + d.tw);
    const long long total = (long long)rows * wpr;
    for (long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x; e < total;
         e += (long long)gridDim.x * blockDim.x) {
        const int row = (int)(e / wpr), o = (int)(e - (long long)row * wpr);
        const int snp = 8 * (row / (8 * G)) + (row & 7), g = (row >> 3) % G;
        const bool ctrl = o >= wc;
        const int k = ctrl ? o - wc : o;
        uint32_t v = 0;
        if (snp < d.snps) {
            if (k < (ctrl ? nt32 : nc32)) {
                const uint64_t word = __ldg(d.ref + snp * per_snp + (ctrl ? 3 * (size_t)d.cw : 0) +
                                            (size_t)g * (ctrl ? d.tw : d.cw) + (k >> 1));
                v = (uint32_t)(word >> (32 * (k & 1)));
            }
            bits[((size_t)G * snp + g) * wpr + o] = v;
        }
        planes[e] = f4_expand_b(v);
    }
}

int f4_pack(int n_cases, int n_ctrls) {
    for (int p = 1; p < 24; ++p) {
        const long long W = 1ll << p;
        if (W > n_cases && n_cases + W * (long long)n_ctrls < (1ll << 24)) return p;
    }
    return 0;
}

cudaError_t f4_bit_map(CUtensorMap* m, const F4Plan& f, const uint32_t* bits, int rows, int box_rows) {
    return tensor_map(m, bits, rows, 4 * f.wpr, kXBitRow, box_rows, false);
}

void f4_sizes(const DevData& d, F4Plan& f) {
    f.pack = f4_pack(d.n_cases, d.n_ctrls);
    f.nw_c = (d.n_cases + 63) / 64;
    f.nw_t = (d.n_ctrls + 63) / 64;
    f.wpr = 8 * ((f.nw_c + 3) / 4) + 8 * ((f.nw_t + 3) / 4);
}

cudaError_t f4_prepare(const DevData& d, F4Plan& f, int genotypes, cudaStream_t s) {
    const int wc = 8 * ((f.nw_c + 3) / 4);
    f.rows = 8 * genotypes * ((d.snps + 7) / 8);
    const size_t plane_bytes = (size_t)f.rows * f.wpr * 16;  // one allocation: planes, then bits
    cudaError_t e = cudaMalloc((void**)&f.planes, plane_bytes + (size_t)genotypes * d.snps * f.wpr * 4);
    if (e != cudaSuccess) return e;
    f.bits = reinterpret_cast<uint32_t*>(f.planes + plane_bytes);
    const long long total = (long long)f.rows * f.wpr;
    const unsigned grid = (unsigned)std::min<long long>((total + 255) / 256, 8192);
    (genotypes == 2 ? f4_layout_kernel<2> : f4_layout_kernel<3>)<<<grid, 256, 0, s>>>(
        d, f.bits, reinterpret_cast<uint4*>(f.planes), f.wpr, wc, 2 * f.nw_c, 2 * f.nw_t, f.rows);
    count_launch();
    if ((e = cudaGetLastError()) != cudaSuccess) return e;
    if (genotypes == 3) return f4_missing_maps(f, d.snps);
    if ((e = tensor_map(&f.map_b, f.planes, f.rows, 16 * f.wpr, kXRow, kXN / 2, true)) != cudaSuccess) return e;
    if ((e = f4_bit_map(&f.map_j, f, f.bits, 2 * d.snps, 2 * kXJ)) != cudaSuccess) return e;
    return f4_bit_map(&f.map_i, f, f.bits, 2 * d.snps, 2);
}

void f4_release(F4Plan& f) {
    cudaFree(f.planes);
    cudaFree(f.ones);
    cudaFree(f.tri);
    cudaFree(f.row_p);
    f.planes = f.ones = nullptr;
    f.bits = nullptr;
    f.tri = f.pairf = nullptr;
    f.row_p = f.row_q = nullptr;
}

std::vector<long long> t3x_items(int n) {
    std::vector<long long> b((size_t)n + 1, 0);
    for (int i = 0; i < n; ++i) {
        long long c = 0;
        for (int j = i + 1; j < n - 1; j += kPxJ) c += t3x_tiles(n, j);
        b[i + 1] = b[i] + c;
    }
    return b;
}

// Pair cores, entries (z, w) of (k, l) for l and l + 1 in 32 bytes: packed floats side by side, or (pack 0)
// words cases | controls << 16, the four of l first.
__global__ void f4_pairf_kernel(const uint4* __restrict__ pairs, uint32_t* out, const int* __restrict__ row_p, int n,
                                int pack) {
    const float W = (float)(1u << pack);
    const int k = blockIdx.x;
    for (int m = ((k + 1) >> 1) + threadIdx.x; m < (n + 1) / 2; m += blockDim.x) {
        uint32_t* o = out + 8 * (size_t)(row_p[k] + m);
        for (int u = 0; u < 2; ++u) {
            const int l = 2 * m + u;
            const uint4 p = l > k && l < n ? __ldg(pairs + pair_index(k, l, n)) : make_uint4(0, 0, 0, 0);
            for (int e = 0; e < 4; ++e) {
                const uint32_t c = e >> 1 ? p.y : p.x, t = e >> 1 ? p.w : p.z;
                if (pack) o[2 * e + u] = __float_as_uint(t3x_pair(p, e >> 1, e & 1, W));
                else o[4 * u + e] = e & 1 ? __byte_perm(c, t, 0x7632) : __byte_perm(c, t, 0x5410);
            }
        }
    }
}

// Rows of l pairs, row k from l = k + 1 rounded down to even: row_p (n), row_q (n), where F4Plan has them, and
// the entries of the pairs and of the triples.
struct F4Rows {
    std::vector<int> p;
    long long pairs = 0, triples = 0;
};
static F4Rows f4_rows(int n) {
    F4Rows r;
    r.p.resize((size_t)2 * n + 1);  // and the launch's status
    std::vector<long long> P((size_t)n + 1);
    for (int k = 0; k < n; ++k) {
        P[k] = r.pairs;
        r.p[k] = (int)(r.pairs - ((k + 1) >> 1));
        r.pairs += ((n + 1) >> 1) - ((k + 1) >> 1);
    }
    P[n] = r.pairs;
    for (int i = 0; i < n; ++i) {
        r.p[n + i] = (int)(r.triples - P[i + 1]);
        r.triples += P[n] - P[i + 1];
    }
    return r;
}

size_t f4_triples_bytes(int snps) {
    // row k has ceil(n / 2) - floor((k + 1) / 2) entries, and a triple's (i, k) one of row k for every i < k
    const unsigned long long n = snps, h = (n + 1) / 2;
    unsigned long long pairs = 0, triples = 0;
    if (n > 4096) return (size_t)std::min(5.34 * n * n * n, 4e18);  // (larger than any device)
    for (unsigned long long k = 0; k < n; ++k) {
        pairs += h - (k + 1) / 2;
        triples += k * (h - (k + 1) / 2);
    }
    return (size_t)triples * 64 + (size_t)pairs * 32;
}

cudaError_t f4_triples(const DevData& d, F4Plan& f, const long long* item_begin, long long items, const uint4* pairs,
                       cudaStream_t s, int sms) {
    const int n = d.snps;
    const F4Rows r4 = f4_rows(n);
    const std::vector<int>& p = r4.p;
    const long long B = r4.triples;
    int* rows = nullptr;
    char* tab = nullptr;  // triples, then pairs
    cudaError_t e = cudaMalloc((void**)&rows, p.size() * sizeof(int));
    if (e == cudaSuccess) e = cudaMalloc((void**)&tab, f4_triples_bytes(n));
    if (e == cudaSuccess) e = cudaMemcpyAsync(rows, p.data(), p.size() * sizeof(int), cudaMemcpyHostToDevice, s);
    if (e == cudaSuccess) {
        f.row_p = rows;
        f.row_q = rows + n;
        f.tri = reinterpret_cast<float*>(tab);
        f.pairf = reinterpret_cast<float*>(tab + (size_t)B * 64);
        f4_pairf_kernel<<<n, 128, 0, s>>>(pairs, reinterpret_cast<uint32_t*>(f.pairf), f.row_p, n, f.pack);
        count_launch();
        e = cudaGetLastError();
    }
    if (e == cudaSuccess) {
        ScanWork w{};
        w.d = d;
        w.order = 3;
        w.dist_n = n;
        w.dist_step = 1;
        const T3xRange r{item_begin, &f.map_j};
        e = launch_tensor3x(w, f, r, 0, items, CandSink{}, nullptr, nullptr, pairs, 0, rows + 2 * n, s, sms, true);
    }
    int gave_up = 0;
    if (e == cudaSuccess) e = cudaMemcpyAsync(&gave_up, rows + 2 * n, sizeof(int), cudaMemcpyDeviceToHost, s);
    if (e == cudaSuccess) e = cudaStreamSynchronize(s);
    if (e == cudaSuccess && gave_up) e = cudaErrorLaunchTimeout;
    if (e != cudaSuccess) {
        cudaFree(rows);
        cudaFree(tab);
        f.row_p = f.row_q = nullptr;
        f.tri = f.pairf = nullptr;
    }
    return e;
}

cudaError_t launch_tensor3x(const ScanWork& w, const F4Plan& f, const T3xRange& r, long long g0, long long g1,
                            const CandSink& sink, uint32_t* dump, const uint32_t* single, const uint4* pairs,
                            double est_margin, int* status, cudaStream_t s, int sms, bool cores) {
    using Fn = decltype(&tensor3x_kernel<kXScan, false>);
    static const Fn fns[6] = {tensor3x_kernel<kXScan, false>, tensor3x_kernel<kXLayer, false>,
                              tensor3x_kernel<kXCores, false>, tensor3x_kernel<kXScan, true>,
                              tensor3x_kernel<kXLayer, true>, tensor3x_kernel<kXCores, true>};
    // set once, by whichever host thread comes first (thread-safe static initialisation)
    static const cudaError_t attr = [] {
        cudaError_t e = cudaSuccess;
        for (int k = 0; k < 6 && e == cudaSuccess; ++k)
            e = cudaFuncSetAttribute(fns[k], cudaFuncAttributeMaxDynamicSharedMemorySize,
                                     (int)(k < 3 ? kXSmem<false> : kXSmem<true>));
        return e;
    }();
    if (attr != cudaSuccess) return attr;
    if (g1 <= g0) return cudaSuccess;
    static const int max_clusters = pair_clusters(tensor3x_kernel<kXScan, false>, kXThreads, kXSmem<false>);
    const long long clusters = std::min<long long>(g1 - g0, max_clusters > 0 ? max_clusters : sms / 2);
    const unsigned grid = (unsigned)(2 * std::max(1ll, clusters));
    const Fn fn = fns[(cores ? kXCores : r.jlist ? kXLayer : kXScan) + (f.pack ? 0 : 3)];
    const double scale = 1.0 / (std::log(2.0) * 4294967296.0);
    LiveMap map{scale, -(double)w.base_key * scale - est_margin, 0, 0};
    f4_quadratic(w.d.n_cases, w.d.n_ctrls, 27, map.bound_k, map.bound_c);
    map.bound_k *= scale;
    fn<<<grid, kXThreads, f.pack ? kXSmem<false> : kXSmem<true>, s>>>(
        f.map_b, *r.map_j, f.map_i, w, sink, r.item_begin, g0, g1, f.nw_c, f.nw_t, f.pack, map, dump, single, pairs,
        status, r.jl_begin, r.jlist, f.tri, f.row_p, f.row_q);
    count_launch();
    return cudaGetLastError();
}

}  // namespace fiu
