// Order-3 and order-2 contingency tables on the 5th-generation tensor cores
// (tcgen05).  Kernels: tensor3x_kernel (order 3, classes that pack into one
// accumulator, CTA pairs), tensor3_kernel (order 3, one accumulator per
// class, described first below), tensor2x_kernel (order 2, classes that
// pack, CTA pairs) and tensor2_kernel (order 2, per class).
//
// For one-hot data the 8 core cells of a combination (i, j, l) -- genotypes
// x, y, z in {0, 1} -- are dot products over the samples of one class:
//     core[x][y][z] = sum_s a_ix(s) a_jy(s) a_lz(s),
// where a_gx(s) is 1 when sample s has genotype x at SNP g.  A work item is
// (i, 32 consecutive j, 96 consecutive l); per class it is one GEMM
//     D[(j,x,y), (l,z)] = sum_s A[(j,x,y), s] B[(l,z), s]    (M 128, N 192),
// accumulated exactly in FP32 in tensor memory.
//
// Operands.  Each data set is expanded once into e4m3 operand planes in HBM:
// row 2*snp+g holds 0x38 (1.0) where the sample has genotype g, else 0; cases
// then controls, each class padded to a multiple of 128 samples.  B rows are
// plane rows 2l+z, loaded by TMA with 128-byte swizzle straight into the
// layout tcgen05 reads (K-major, SWIZZLE_128B descriptor).  A rows are the
// bytewise AND of the i and j plane rows (0x38 & 0x38 = 0x38): four producer
// warps read the TMA-staged j and i rows from shared memory, AND them in
// registers and write the result to tensor memory (tcgen05.st; one thread per
// row, 4 e4m3 per 32-bit column), where the MMA reads A from (the [a-tmem]
// form of tcgen05.mma): A never touches shared memory, whose bandwidth is the
// kernel's bound.
//
// Warp roles (448 threads, one CTA per SM): warp 0 issues the TMA copies,
// warp 1 issues tcgen05.mma (kind::f8f6f4, K 32 per instruction, 4 per
// 128-sample stage) and commits, warps 2-5 build A, warps 6-13 run the
// epilogue.  Four stages are handed over with mbarriers.  Tensor memory
// (512 columns): case accumulators in columns 0-191, control accumulators in
// 192-383, the A ring (4 stages x 32 columns) in 384-511.  As soon as an
// item's case GEMM is done the epilogue packs its counts to 16 bits in shared
// memory and frees columns 0-191, so the next item's case GEMM overlaps the
// current item's epilogue.
//
// Epilogue.  Each thread reads the accumulators of one row (j, x, y); a
// swizzled shared-memory transpose gives each thread the 16 core counts of one
// combination.  The full 27-cell tables are derived exactly from the pair and
// single cores (inclusion-exclusion, as the CUDA-core reduced-work kernel
// does).  A single-precision estimate of the fixed-point MI key (lg2.approx)
// with a proven error bound rejects the combinations that cannot reach the
// current threshold; the others get the exact 64-bit fixed-point key from the
// integer c*ln(c) table, so the kept set is exactly the one of the exact key.
//
// Reference semantics: GenotypeTable::combine_and_popcnt for order 3
// (src/base/gt_popcnt.cpp:4-35) and MutualInformation::compute
// (src/base/mi_compute.cpp:16-41) over the combinations ThreadedSearch
// visits (include/fiuncho/ThreadedSearch.h:157-180) with one worker.
#include <cudaTypedefs.h>

#include <algorithm>
#include <cmath>
#include <cstring>
#include <map>
#include <tuple>
#include <mutex>

#include "tensor3_eval.cuh"
#include "tensor2x.h"
#include "tensor3x.h"

namespace fiu {

constexpr int kT3J = 32, kT3L = 96;              // SNPs per tile
constexpr int kT3M = 4 * kT3J, kT3N = 2 * kT3L;  // 128 x 192 GEMM tile
constexpr int kT3Stages = 4;
constexpr int kT3SB = kT3N * kT3KB;              // 24 KB  l rows (1 KB multiple)
constexpr int kT3SJ = 2 * kT3J * kT3KB;          //  8 KB  staged j rows
constexpr int kT3SI = 1024;                      // i rows of a stage (2 x 128 B, 128-byte swizzle: the two
                                                 // rows' chunk c sit in different banks)
constexpr int kT3EpiWarps = 8, kT3BuildWarps = 4;
constexpr int kT3Threads = 32 * (2 + kT3BuildWarps + kT3EpiWarps);  // 448
constexpr int kT3Ebuf = 2048;                    // per epilogue warp: 256 transpose slots of 8 B
constexpr int kT3Stash = 32 * (kT3L / 2) * 4;    // per epilogue warp: 32 rows x 48 words (16-bit case pairs)
constexpr size_t kT3Smem = 1024 + (size_t)kT3Stages * (kT3SB + kT3SJ + kT3SI) +
                           (size_t)kT3EpiWarps * (kT3Ebuf + kT3Stash);
constexpr int kT3ColCtrl = kT3N, kT3ColA = 2 * kT3N;  // tensor-memory column bases
constexpr uint32_t kT3Idesc = (1u << 4) | ((uint32_t)(kT3N >> 3) << 17) | ((uint32_t)(kT3M >> 4) << 24);

static_assert(kT3Smem <= 227 * 1024 - 256, "tensor kernel shared memory");
static_assert(kT3ColA + 32 * kT3Stages <= 512, "tensor memory columns");

// Work items of one i: J-tile a starts at j0 = i+1+32a and has
// ceil((n-1-j0)/L) L-tiles starting at l0 = j0+1+L*b.
template <int L>
__device__ __forceinline__ void t3_decode(const long long* __restrict__ item_begin, int n, long long g, int& i,
                                          int& j0, int& l0) {
    int lo = 0, hi = n - 1;
    while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (item_begin[mid] <= g) lo = mid;
        else hi = mid - 1;
    }
    i = lo;
    long long q = g - item_begin[i];
    for (int a = 0;; ++a) {
        const int j = i + 1 + kT3J * a;
        const long long nl = (n - 1 - j + L - 1) / L;
        if (q < nl) {
            j0 = j;
            l0 = j + 1 + L * (int)q;
            return;
        }
        q -= nl;
    }
}

// List mode (a Distribution layer): the owned j of each i are listed in
// jlist[jl_begin[i] .. jl_begin[i+1]); an item takes J consecutive entries
// from p0 (= jl_begin[i] + J a) and an l-tile l0 = jlist[p0] + 1 + L b.
template <int J, int L>
__device__ __forceinline__ void t3l_decode(const long long* __restrict__ item_begin,
                                           const long long* __restrict__ jl_begin, const int* __restrict__ jlist,
                                           int n, long long g, int& i, long long& p0, int& l0) {
    int lo = 0, hi = n - 1;
    while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (item_begin[mid] <= g) lo = mid;
        else hi = mid - 1;
    }
    i = lo;
    long long q = g - item_begin[i];
    for (long long p = jl_begin[i];; p += J) {
        const int jf = jlist[p];
        const long long nl = (n - 1 - jf + L - 1) / L;
        if (q < nl) {
            p0 = p;
            l0 = jf + 1 + L * (int)q;
            return;
        }
        q -= nl;
    }
}

// The j of row jj (0..31) of a CTA's 32 j of an item: j0 + jj, or in list mode
// the listed entry p0 + jj (n when the list of i ends before it).
template <bool LIST>
__device__ __forceinline__ int t3x_j(int j0, long long p0, long long p_end, const int* __restrict__ jlist, int jj,
                                     int n) {
    if (!LIST) return j0 + jj;
    const long long p = p0 + jj;
    return p < p_end ? __ldg(jlist + p) : n;
}

// 8-byte slot of the order-3 epilogue transpose buffer holding the counts
// (cases z0 | z1 << 16, controls z0 | z1 << 16) of row (jl, xy) and column
// group k; the XOR makes both the row-wise writes (lanes (jl, xy), fixed k)
// and the combination-wise reads (lanes (jl, k / 2), fixed xy) cover the 32
// banks once per half-warp.
__device__ __forceinline__ int t3_slot(int jl, int k, int xy) {
    return ((jl * 8 + k) * 4 + xy) ^ ((jl & 3) | (((jl ^ (k >> 1)) & 3) << 2));
}

// Evaluates combination (i, j, l) whose 16 core counts (cases z0, z1, controls z0, z1 of each
// (x, y)) sit in column group k of this warp's transpose buffer (every lane calls it).
__device__ __forceinline__ void t3_eval(const ScanWork& w, const CandSink& sink, float thr_f, uint32_t* dump,
                                        const uint32_t* __restrict__ single, const uint4* __restrict__ pairs,
                                        const uint32_t* ebuf, int jl, int k, int i, int j, int l, bool j_ok,
                                        const uint4& pij, const float (&si)[2][2], const float (&sj)[2][2],
                                        int lane) {
    const bool valid = j_ok && l < w.d.snps && l > j;
    float core[2][8];
#pragma unroll
    for (int x4 = 0; x4 < 4; ++x4) {
        const uint2 c2 = *reinterpret_cast<const uint2*>(ebuf + 2 * t3_slot(jl, k, x4));
        core[0][2 * x4] = u2f(c2.x & 0xffffu);
        core[0][2 * x4 + 1] = u2f(c2.x >> 16);
        core[1][2 * x4] = u2f(c2.y & 0xffffu);
        core[1][2 * x4 + 1] = u2f(c2.y >> 16);
    }
    if (sink.evaluated) {
        const unsigned vmask = __ballot_sync(0xffffffffu, valid);
        if (lane == 0 && vmask) atomicAdd(sink.evaluated, (unsigned long long)__popc(vmask));
    }
    t3_eval_core(w, sink, thr_f, dump, single, pairs, core, i, j, l, valid, pij, si, sj, lane);
}

struct T3Maps {
    CUtensorMap l, j, i;
};

// LIST: a Distribution layer (t3l_decode; maps.j covers the residue-ordered planes, where the
// listed j of one i are consecutive rows).
template <bool LIST>
__global__ void __launch_bounds__(kT3Threads, 1)
    tensor3_kernel(const __grid_constant__ T3Maps maps, ScanWork w, const long long* __restrict__ item_begin,
                   long long g0, long long g1, int k_cases, CandSink sink, float thr_f, uint32_t* dump,
                   const uint32_t* __restrict__ single, const uint4* __restrict__ pairs, int* status,
                   const long long* __restrict__ jl_begin, const int* __restrict__ jlist) {
    extern __shared__ uint8_t smraw[];
    __shared__ __align__(8) uint64_t full_t[kT3Stages], full_a[kT3Stages], empty[kT3Stages];
    __shared__ __align__(8) uint64_t case_full, case_empty, ctrl_full, ctrl_empty, done;
    __shared__ uint32_t tmem_base;
    __shared__ int abort_flag;
    uint8_t* sm = (uint8_t*)(((uintptr_t)smraw + 1023) & ~(uintptr_t)1023);  // B ring
    uint8_t* sj_base = sm + kT3Stages * kT3SB;                                 // j ring
    uint8_t* si_base = sj_base + kT3Stages * kT3SJ;                            // i ring
    uint32_t* ebuf_all = reinterpret_cast<uint32_t*>(si_base + kT3Stages * kT3SI);
    uint4* stash_all = reinterpret_cast<uint4*>(ebuf_all + kT3EpiWarps * (kT3Ebuf / 4));
    volatile int* abort = &abort_flag;
    const DevData& d = w.d;
    const int n = d.snps;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int ks_c = k_cases / kT3KB;     // 128-sample steps of the case class
    const int ks_t = (d.tw + 1) / 2;      // ... of the control class
    const int ksteps = ks_c + ks_t;

    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_base)),
                     "r"(512));
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
    }
    if (tid == 0) {
        for (int s = 0; s < kT3Stages; ++s) {
            asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_u32(&full_t[s])));
            asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(&full_a[s])), "r"(kT3BuildWarps));
            asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_u32(&empty[s])));
        }
        asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_u32(&case_full)));
        asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(&case_empty)), "r"(kT3EpiWarps));
        asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_u32(&ctrl_full)));
        asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(&ctrl_empty)), "r"(kT3EpiWarps));
        asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_u32(&done)));
        asm volatile("fence.mbarrier_init.release.cluster;");
        abort_flag = 0;
    }
    asm volatile("tcgen05.fence::before_thread_sync;");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;");
    const uint32_t tmem = tmem_base;
    bool ok = true;

    if (warp == 0) {
        // ---------------------------------------------------------------- TMA producer
        if (lane == 0) {
            long long step = 0;
            for (long long g = g0 + blockIdx.x; g < g1 && ok; g += gridDim.x) {
                int i, j0, l0;  // LIST: j0 = the first listed j's row in the residue-ordered planes
                if (LIST) {
                    long long p0;
                    t3l_decode<kT3J, kT3L>(item_begin, jl_begin, jlist, n, g, i, p0, l0);
                    j0 = residue_row(jlist[p0], w.dist_step, n);
                } else {
                    t3_decode<kT3L>(item_begin, n, g, i, j0, l0);
                }
                for (int ks = 0; ks < ksteps; ++ks) {
                    const int s = (int)(step % kT3Stages);
                    const long long u = step / kT3Stages;
                    if (u > 0 && !t3_wait(smem_u32(&empty[s]), (uint32_t)((u - 1) & 1), abort)) {
                        ok = false;
                        break;
                    }
                    const int k0 = ks < ks_c ? ks * kT3KB : k_cases + (ks - ks_c) * kT3KB;
                    const uint32_t bar = smem_u32(&full_t[s]);
                    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar),
                                 "r"((uint32_t)(kT3SB + kT3SJ + 2 * kT3KB))
                                 : "memory");
                    t3_tma(smem_u32(sm + s * kT3SB), &maps.l, k0, 2 * l0, bar);
                    t3_tma(smem_u32(sj_base + s * kT3SJ), &maps.j, k0, 2 * j0, bar);
                    t3_tma(smem_u32(si_base + s * kT3SI), &maps.i, k0, 2 * i, bar);
                    ++step;
                }
            }
            // no copy may be in flight when the CTA exits: wait for the last use of every stage
            for (int s = 0; s < kT3Stages; ++s) {
                if (step <= s) continue;
                const long long last = s + ((step - 1 - s) / kT3Stages) * kT3Stages;
                if (!t3_drain(smem_u32(&full_t[s]), (uint32_t)((last / kT3Stages) & 1))) ok = false;
            }
        }
    } else if (warp == 1) {
        // ---------------------------------------------------------------- MMA issuer
        if (lane == 0) {
            long long step = 0, item = 0;
            for (long long g = g0 + blockIdx.x; g < g1 && ok; g += gridDim.x, ++item) {
                for (int ks = 0; ks < ksteps; ++ks, ++step) {
                    const int cls = ks >= ks_c;
                    if (item > 0 && (ks == 0 || ks == ks_c)) {  // accumulator columns free again?
                        if (!t3_wait(smem_u32(cls ? &ctrl_empty : &case_empty), (uint32_t)((item - 1) & 1), abort)) {
                            ok = false;
                            break;
                        }
                    }
                    const int s = (int)(step % kT3Stages);
                    if (!t3_wait(smem_u32(&full_a[s]), (uint32_t)((step / kT3Stages) & 1), abort)) {
                        ok = false;
                        break;
                    }
                    asm volatile("tcgen05.fence::after_thread_sync;");
                    const uint32_t sb = smem_u32(sm + s * kT3SB);
                    const uint32_t acol = tmem + (uint32_t)(kT3ColA + 32 * s);
                    const uint32_t dcol = tmem + (cls ? (uint32_t)kT3ColCtrl : 0u);
                    const bool first = ks == 0 || ks == ks_c;
#pragma unroll
                    for (int kk = 0; kk < 4; ++kk) {  // A: 8 columns (32 e4m3) per instruction
                        const uint64_t bd = t3_desc(sb + 32 * kk);
                        const uint32_t acc = (first && kk == 0) ? 0u : 1u;
                        asm volatile(
                            "{.reg .pred p; setp.ne.b32 p, %4, 0;\n"
                            "tcgen05.mma.cta_group::1.kind::f8f6f4 [%0], [%1], %2, %3, p;}\n" ::"r"(dcol),
                            "r"(acol + 8 * kk), "l"(bd), "r"(kT3Idesc), "r"(acc));
                    }
                    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(
                        smem_u32(&empty[s])));
                    if (ks == ks_c - 1 || ks == ksteps - 1)
                        asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(
                            smem_u32(ks == ks_c - 1 ? &case_full : &ctrl_full)));
                }
            }
            // every MMA of this thread complete before the tensor memory is released
            asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(
                smem_u32(&done)));
            if (!t3_drain(smem_u32(&done), 0)) ok = false;
        }
    } else if (warp < 2 + kT3BuildWarps) {
        // ---------------------------------------------------------------- A builders
        // thread = tensor-memory lane = A row m = (jj, x, y) of this warp's lane quarter
        const int m = 32 * (warp & 3) + lane;
        const int r = 2 * (m >> 2) + (m & 1), x = (m >> 1) & 1;  // staged j row (jj, y), i row x
        const uint32_t a_lane = tmem + ((uint32_t)(32 * (warp & 3)) << 16) + (uint32_t)kT3ColA;
        long long step = 0;
        for (long long g = g0 + blockIdx.x; g < g1 && ok; g += gridDim.x) {
            for (int ks = 0; ks < ksteps; ++ks, ++step) {
                const int s = (int)(step % kT3Stages);
                if (!t3_wait(smem_u32(&full_t[s]), (uint32_t)((step / kT3Stages) & 1), abort)) {
                    ok = false;
                    break;
                }
                const uint8_t* sJ = sj_base + s * kT3SJ + r * 128;
                const uint8_t* sI = si_base + s * kT3SI + x * 128;
                uint32_t a[32];
#pragma unroll
                for (int c = 0; c < 8; ++c) {
                    const uint4 jv = *reinterpret_cast<const uint4*>(sJ + ((c ^ (r & 7)) << 4));
                    const uint4 iv = *reinterpret_cast<const uint4*>(sI + ((c ^ x) << 4));
                    a[4 * c + 0] = jv.x & iv.x;
                    a[4 * c + 1] = jv.y & iv.y;
                    a[4 * c + 2] = jv.z & iv.z;
                    a[4 * c + 3] = jv.w & iv.w;
                }
                // slot s of the A ring is free: the TMA of this step waited for the MMAs of its last use
                asm volatile(
                    "tcgen05.st.sync.aligned.32x32b.x32.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%"
                    "16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31,%32};" ::"r"(a_lane +
                                                                                               (uint32_t)(32 * s)),
                    "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(a[4]), "r"(a[5]), "r"(a[6]), "r"(a[7]), "r"(a[8]),
                    "r"(a[9]), "r"(a[10]), "r"(a[11]), "r"(a[12]), "r"(a[13]), "r"(a[14]), "r"(a[15]), "r"(a[16]),
                    "r"(a[17]), "r"(a[18]), "r"(a[19]), "r"(a[20]), "r"(a[21]), "r"(a[22]), "r"(a[23]), "r"(a[24]),
                    "r"(a[25]), "r"(a[26]), "r"(a[27]), "r"(a[28]), "r"(a[29]), "r"(a[30]), "r"(a[31]));
                asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
                asm volatile("tcgen05.fence::before_thread_sync;");
                __syncwarp();
                if (lane == 0)
                    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(&full_a[s])) : "memory");
            }
        }
    } else {
        // ---------------------------------------------------------------- epilogue
        const int e = warp - (2 + kT3BuildWarps);  // 0..7
        const int q = warp & 3;                    // tensor-memory lane quarter this warp may access
        const int hh = e >> 2;                     // column groups 2 cc + hh: l offsets 16 cc + 8 hh + [0, 8)
        uint32_t* ebuf = ebuf_all + e * (kT3Ebuf / 4);
        uint4* stash = stash_all + e * (kT3Stash / 16);  // [word quad][lane]: conflict-free
        const uint32_t lane_base = tmem + ((uint32_t)(32 * q) << 16);
        // row (writer) view: jl = lane/4, xy = lane%4; combination (reader) view: jl = lane/4, kp = lane%4
        const int jl = lane >> 2, xy = lane & 3, kp = lane & 3;
        long long item = 0;
        for (long long g = g0 + blockIdx.x; g < g1 && ok; g += gridDim.x, ++item) {
            int i, j0 = 0, l0;
            long long p0 = 0, p_end = 0;
            if (LIST) {
                t3l_decode<kT3J, kT3L>(item_begin, jl_begin, jlist, n, g, i, p0, l0);
                p_end = jl_begin[i + 1];
            } else {
                t3_decode<kT3L>(item_begin, n, g, i, j0, l0);
            }
            // ---- phase 1: case counts -> 16-bit stash, case columns free for the next item
            if (!t3_wait(smem_u32(&case_full), (uint32_t)(item & 1), abort)) {
                ok = false;
                break;
            }
            asm volatile("tcgen05.fence::after_thread_sync;");
#pragma unroll 1
            for (int cc = 0; cc < 6; ++cc) {
                const uint32_t col = (uint32_t)(32 * cc + 16 * hh);
                uint32_t v[16], p[8];
                asm volatile(
                    "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, "
                    "[%16];"
                    : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]),
                      "=r"(v[8]), "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]),
                      "=r"(v[15])
                    : "r"(lane_base + col));
                asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
                for (int k = 0; k < 8; ++k)
                    p[k] = f2u(__uint_as_float(v[2 * k])) | (f2u(__uint_as_float(v[2 * k + 1])) << 16);
                stash[(2 * cc) * 32 + lane] = make_uint4(p[0], p[1], p[2], p[3]);
                stash[(2 * cc + 1) * 32 + lane] = make_uint4(p[4], p[5], p[6], p[7]);
            }
            asm volatile("tcgen05.fence::before_thread_sync;");
            __syncwarp();
            if (lane == 0)
                asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(&case_empty)) : "memory");
            // ---- per-item constants of this thread's j
            const int j = t3x_j<LIST>(j0, p0, p_end, jlist, 8 * q + jl, n);
            const bool j_ok = j < n;
            uint4 pij;
            float si[2][2], sj[2][2];
            t3_item_consts(single, pairs, i, j, n, j_ok, pij, si, sj);
            // ---- phase 2: control counts + stash -> transpose -> tables -> keys
            if (!t3_wait(smem_u32(&ctrl_full), (uint32_t)(item & 1), abort)) {
                ok = false;
                break;
            }
            asm volatile("tcgen05.fence::after_thread_sync;");
#pragma unroll 1
            for (int cc = 0; cc < 6; ++cc) {
                // a group without a valid combination for this warp is skipped (the two warps
                // of a lane quarter interleave over the l range); the columns are still released
                const int lg = l0 + 16 * cc + 8 * hh;
                if (!__any_sync(0xffffffffu, j_ok && lg + 7 > j && lg < n)) {
                    if (cc == 5) {
                        asm volatile("tcgen05.fence::before_thread_sync;");
                        __syncwarp();
                        if (lane == 0)
                            asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(&ctrl_empty))
                                         : "memory");
                    }
                    continue;
                }
                {
                    const uint32_t col = (uint32_t)(32 * cc + 16 * hh);
                    uint32_t vt[16];
                    asm volatile(
                        "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%"
                        "15}, [%16];"
                        : "=r"(vt[0]), "=r"(vt[1]), "=r"(vt[2]), "=r"(vt[3]), "=r"(vt[4]), "=r"(vt[5]), "=r"(vt[6]),
                          "=r"(vt[7]), "=r"(vt[8]), "=r"(vt[9]), "=r"(vt[10]), "=r"(vt[11]), "=r"(vt[12]),
                          "=r"(vt[13]), "=r"(vt[14]), "=r"(vt[15])
                        : "r"(lane_base + (uint32_t)kT3ColCtrl + col));
                    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
                    const uint4 s0 = stash[(2 * cc) * 32 + lane], s1 = stash[(2 * cc + 1) * 32 + lane];
                    const uint32_t su[8] = {s0.x, s0.y, s0.z, s0.w, s1.x, s1.y, s1.z, s1.w};
                    if (cc == 5) {  // last read of this item's accumulators: control columns free
                        asm volatile("tcgen05.fence::before_thread_sync;");
                        __syncwarp();
                        if (lane == 0)
                            asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(&ctrl_empty))
                                         : "memory");
                    }
#pragma unroll
                    for (int k = 0; k < 8; ++k) {
                        const uint32_t t0 = f2u(__uint_as_float(vt[2 * k]));
                        const uint32_t t1 = f2u(__uint_as_float(vt[2 * k + 1]));
                        *reinterpret_cast<uint2*>(ebuf + 2 * t3_slot(jl, k, xy)) = make_uint2(su[k], t0 | t1 << 16);
                    }
                }
                __syncwarp();
#pragma unroll 1
                for (int b = 0; b < 2; ++b)
                    t3_eval(w, sink, thr_f, dump, single, pairs, ebuf, jl, 2 * kp + b, i, j, lg + 2 * kp + b, j_ok,
                            pij, si, sj, lane);
                __syncwarp();
            }
        }
    }
    if (!ok) *abort = 1;
    asm volatile("tcgen05.fence::before_thread_sync;");
    __syncthreads();
    if (tid == 0 && abort_flag) atomicOr(status, 1);
    if (warp == 0) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512));
}

// Operand planes: one thread per 16 output bytes (16 samples of one row).
__global__ void t3_planes_kernel(DevData d, uint8_t* planes, int pitch, int k_cases) {
    const long long chunks = (long long)pitch / 16;
    const long long total = 2ll * d.snps * chunks;
    const size_t per_snp = 3 * (size_t)(d.cw + d.tw);
    for (long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x; e < total;
         e += (long long)gridDim.x * blockDim.x) {
        const long long row = e / chunks;
        const int ch = (int)(e - row * chunks);
        const int snp = (int)(row >> 1), g = (int)(row & 1);
        const int o = 16 * ch;
        const bool ctrl = o >= k_cases;
        const int k = ctrl ? o - k_cases : o;
        const int W = ctrl ? d.tw : d.cw;
        const int word = k >> 6;
        uint32_t bits = 0;
        if (word < W)
            bits = (uint32_t)(__ldg(d.ref + (size_t)snp * per_snp + (ctrl ? 3 * (size_t)d.cw : 0) + (size_t)g * W +
                                    word) >>
                              (k & 63)) &
                   0xffffu;
        uint4 v;
        uint32_t* pv = &v.x;
#pragma unroll
        for (int qd = 0; qd < 4; ++qd)
            pv[qd] = (((bits >> (4 * qd)) & 0xfu) * 0x00204081u & 0x01010101u) * 0x38u;
        *reinterpret_cast<uint4*>(planes + (size_t)row * pitch + o) = v;
    }
}

// Items per i of tensor3_kernel (host): prefix sums item_begin[0..n], item_begin[n] = total.
static long long t3_items(int n, int L, std::vector<long long>& item_begin) {
    item_begin.assign((size_t)n + 1, 0);
    long long total = 0;
    for (int i = 0; i < n; ++i) {
        item_begin[i] = total;
        for (int j = i + 1; j < n - 1; j += kT3J) total += (n - 1 - j + L - 1) / L;
    }
    item_begin[n] = total;
    return total;
}

static PFN_cuTensorMapEncodeTiled_v12000 t3_encoder() {
    static const PFN_cuTensorMapEncodeTiled_v12000 fn = [] {
        cudaDriverEntryPointQueryResult q;
        void* p = nullptr;
        if (cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &p, 12000, cudaEnableDefault, &q) ==
                cudaSuccess &&
            q == cudaDriverEntryPointSuccess)
            return (PFN_cuTensorMapEncodeTiled_v12000)p;
        return (PFN_cuTensorMapEncodeTiled_v12000) nullptr;
    }();
    return fn;
}

cudaError_t tensor_map(CUtensorMap* m, const void* base, int rows, int pitch, int box_bytes, int box_rows,
                       bool swizzle) {
    auto enc = t3_encoder();
    if (!enc) return cudaErrorNotSupported;
    cuuint64_t dims[2] = {(cuuint64_t)pitch, (cuuint64_t)rows};
    cuuint64_t strides[1] = {(cuuint64_t)pitch};
    cuuint32_t box[2] = {(cuuint32_t)box_bytes, (cuuint32_t)box_rows};
    cuuint32_t es[2] = {1, 1};
    const CUresult r = enc(m, CU_TENSOR_MAP_DATA_TYPE_UINT8, 2, const_cast<void*>(base), dims, strides, box, es,
                           CU_TENSOR_MAP_INTERLEAVE_NONE,
                           swizzle ? CU_TENSOR_MAP_SWIZZLE_128B : CU_TENSOR_MAP_SWIZZLE_NONE,
                           CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    return r == CUDA_SUCCESS ? cudaSuccess : cudaErrorInvalidValue;
}

static cudaError_t t3_map(CUtensorMap* m, uint8_t* base, int rows, int pitch, int box_rows, bool swizzle) {
    return tensor_map(m, base, rows, pitch, kT3KB, box_rows, swizzle);
}

// e4m3 planes (the per-class kernels of orders 3 and 4).
static cudaError_t e4m3_planes(T3Plan& plan, const DevData& d, cudaStream_t s) {
    if (plan.planes) return cudaSuccess;
    uint8_t* planes = nullptr;
    cudaError_t e = cudaMalloc((void**)&planes, (size_t)2 * d.snps * plan.pitch);
    if (e != cudaSuccess) return e;
    const long long total = 2ll * d.snps * (plan.pitch / 16);
    const int grid = (int)std::min<long long>((total + 255) / 256, 4096);
    t3_planes_kernel<<<grid, 256, 0, s>>>(d, planes, plan.pitch, plan.k_cases);
    count_launch();
    e = cudaGetLastError();
    if (e == cudaSuccess) e = cudaStreamSynchronize(s);
    const int rows = 2 * d.snps;
    if (e == cudaSuccess) e = t3_map(&plan.map_l, planes, rows, plan.pitch, kT3N, true);
    if (e == cudaSuccess) e = t3_map(&plan.map_j, planes, rows, plan.pitch, 2 * kT3J, true);
    if (e == cudaSuccess) e = t3_map(&plan.map_i, planes, rows, plan.pitch, 2, true);
    if (e == cudaSuccess) e = t3_map(&plan.map_l4, planes, rows, plan.pitch, 128, true);
    if (e != cudaSuccess) cudaFree(planes);
    else plan.planes = planes;
    return e;
}

void tensor3_prepare(const DevData& d, T3Plan& plan) {
    f4_sizes(d, plan.f4);
    plan.pair3 = plan.f4.pack != 0;
    plan.k_cases = kT3KB * ((d.cw + 1) / 2);
    plan.pitch = plan.k_cases + kT3KB * ((d.tw + 1) / 2);
}

// Copies a host item table to the device.
static cudaError_t upload(long long*& out, const std::vector<long long>& v) {
    long long* p = nullptr;
    cudaError_t e = cudaMalloc((void**)&p, v.size() * sizeof(long long));
    if (e == cudaSuccess) e = cudaMemcpy(p, v.data(), v.size() * sizeof(long long), cudaMemcpyHostToDevice);
    if (e != cudaSuccess) cudaFree(p);
    else out = p;
    return e;
}

// Order-3 items of the whole data set.
static cudaError_t order3_items(T3Plan& plan, const DevData& d) {
    if (plan.item_begin) return cudaSuccess;
    std::vector<long long> ib;
    if (plan.pair3) ib = t3x_items(d.snps);
    else t3_items(d.snps, kT3L, ib);
    plan.total = ib.back();
    const double n = d.snps;
    plan.item_combos = n * (n - 1) * (n - 2) / 6.0 / std::max(1ll, plan.total);
    return upload(plan.item_begin, ib);
}

// The operands of an order, made on its first search (items_mu held): e4m3 planes, or the 4-bit
// layout and at order 4 the packed cores of the triples.
static cudaError_t order_planes(T3Plan& plan, const DevData& d, int order, const uint4* pairs, cudaStream_t s,
                                int sms) {
    cudaError_t e = cudaSuccess;
    if (order == 2) {
        if (plan.f4.ones) return e;
        e = f4_ones_planes(d, plan.f4, d.snps, 0, 1, plan.f4.ones, s);
        if (e == cudaSuccess) e = cudaStreamSynchronize(s);
        if (e == cudaSuccess) e = f4_map_a2(&plan.f4.map_a2, plan.f4, plan.f4.ones, d.snps);
        if (e == cudaSuccess) e = f4_map_b2(&plan.f4.map_b2, plan.f4, plan.f4.ones, d.snps);
        return e;
    }
    if (!plan.pair3) return e4m3_planes(plan, d, s);
    if (!plan.f4.bits) {
        e = f4_prepare(d, plan.f4, s);
        if (e == cudaSuccess) e = cudaStreamSynchronize(s);
        if (e != cudaSuccess) f4_release(plan.f4);
    }
    if (e == cudaSuccess && order == 4 && !plan.f4.tri) {
        e = order3_items(plan, d);
        if (e == cudaSuccess) e = f4_order4_maps(plan.f4, d.snps);
        if (e == cudaSuccess) e = f4_triples(d, plan.f4, plan.item_begin, plan.total, pairs, s, sms);
    }
    return e;
}

// The work items of the whole data set at order 3 or 4, made on the first
// search of that order (the host enumeration grows as n^2 / 16 at order 4:
// about 0.1 s at 40 000 SNPs, which a search of another order need not pay).
cudaError_t tensor3_order_items(T3Plan& plan, const DevData& d, int order, const uint4* pairs, cudaStream_t s,
                                int sms) {
    std::lock_guard<std::mutex> g(plan.items_mu);
    cudaError_t e = order_planes(plan, d, order, pairs, s, sms);
    if (e == cudaSuccess && order == 3) e = order3_items(plan, d);
    if (e == cudaSuccess && order == 2 && !plan.item2_begin) {
        const std::vector<long long> ib = t2x_items(d.snps, d.snps - 1, 0, 1, plan.n_itiles);
        plan.total2 = ib.back();
        plan.item2_combos = (double)d.snps * (d.snps - 1) / 2 / std::max(1ll, plan.total2);
        e = upload(plan.item2_begin, ib);
    }
    if (e == cudaSuccess && order == 4 && !plan.item4_begin && d.snps >= 4) {
        std::vector<long long> per4;
        const std::vector<long long> ib4 = t4_item_table(d.snps, plan.pair3, per4);
        if (!plan.pair3) e = t3_map(&plan.map_k4, plan.planes, 2 * d.snps, plan.pitch, 32, true);
        if (e == cudaSuccess) e = upload(plan.item4_per, per4);
        if (e != cudaSuccess) return e;
        plan.total4 = ib4.back();
        const double n = d.snps;
        plan.item4_combos = n * (n - 1) * (n - 2) * (n - 3) / 24.0 / std::max(1ll, plan.total4);
        e = upload(plan.item4_begin, ib4);
    }
    return e;
}

// Work items of Distribution layers of order-3 scans (the pair kernel's list
// mode), one entry per (step, offset) used on the data set.  The owned j of
// one i are the j > i of one residue mod step (pair ranks base(i) + j - i - 1
// step through the layer's offset class), so in a copy of the operand planes
// ordered by residue -- SNPs r, r + step, r + 2 step, .. for r = 0, 1, .. --
// they are consecutive rows, and one tiled TMA copy per stage loads an item's
// j rows as in the scan of all prefixes.
struct T3Layer {
    long long* item_begin = nullptr;  // order 3: [n + 1] first item of each i; order 2: [tiles + 1] of each tile
    long long* jl_begin = nullptr;    // order 3: [n + 1] first listed j of each i
    int* jlist = nullptr;             // order 3: owned j of each i, ascending
    long long total = 0;
    double item_combos = 0;
    int n_tiles = 0;                  // order 2: tiles of owned i; order 4: listed pairs
    int4* pinfo = nullptr;            // order 4: (i, j, first owned k) of each listed pair
    CUtensorMap map_jr;               // order 3: 64 rows of the residue-ordered planes (pair kernel: bit rows)
    uint8_t* planes = nullptr;        // order 2: the owned SNPs' planes
    CUtensorMap map_ar;               // order 2: box 128 B x 128 rows over them
    CUtensorMap map_kr;               // order 4: 32 rows of the residue-ordered planes (pair kernel: bit rows)
};
struct T3Layers {
    std::mutex mu;
    std::map<std::tuple<int, int, int>, T3Layer> by;  // (order, step, offset)
    // residue-ordered operand planes, and bit rows (pair kernels of orders 3 and 4), per step
    std::map<int, uint8_t*> by_residue, bits_by_residue;
};

// The rows of every SNP (row_bytes each, SNP-major in src) ordered by residue mod step, made on first use.
static cudaError_t residue_copy(std::map<int, uint8_t*>& by, const uint8_t* src, size_t row_bytes, int n, int step,
                                cudaStream_t s) {
    if (by.count(step)) return cudaSuccess;
    uint8_t* perm = nullptr;
    cudaError_t e = cudaMalloc((void**)&perm, (size_t)n * row_bytes);
    // residue class r holds SNPs r + step m, m < ceil((n - r) / step)
    for (int r = 0; r < step && r < n && e == cudaSuccess; ++r)
        e = cudaMemcpy2DAsync(perm + (size_t)residue_row(r, step, n) * row_bytes, row_bytes,
                              src + (size_t)r * row_bytes, (size_t)step * row_bytes, row_bytes,
                              (size_t)((n - r + step - 1) / step), cudaMemcpyDeviceToDevice, s);
    if (e == cudaSuccess) e = cudaStreamSynchronize(s);
    if (e != cudaSuccess) cudaFree(perm);
    else by[step] = perm;
    return e;
}


static bool is_layer(const ScanWork& w) { return w.dist_step != 1 || w.dist_offset != 0; }

bool tensor_layer_ok(const T3Plan& plan, const ScanWork& w) {
    return (w.order == 2 || w.order == 3 || (w.order == 4 && w.d.snps >= 4)) && w.dist_n == w.d.snps;
}

static const T3Layer* find_layer(const T3Plan& plan, const ScanWork& w) {
    if (!plan.layers) return nullptr;
    std::lock_guard<std::mutex> g(plan.layers->mu);
    auto it = plan.layers->by.find(std::make_tuple(w.order, w.dist_step, w.dist_offset));
    return it == plan.layers->by.end() ? nullptr : &it->second;
}

cudaError_t tensor3_layer(T3Plan& plan, const ScanWork& w, const uint4* pairs, cudaStream_t s, int sms) {
    if (!tensor_layer_ok(plan, w)) return cudaErrorInvalidValue;
    if (!plan.layers) plan.layers = new T3Layers;
    std::lock_guard<std::mutex> g(plan.layers->mu);
    const auto key = std::make_tuple(w.order, w.dist_step, w.dist_offset);
    if (plan.layers->by.count(key)) return cudaSuccess;
    const bool px = w.order != 2 && plan.pair3;  // the pair kernels' j or k operand: bit rows
    cudaError_t pe;
    {
        std::lock_guard<std::mutex> gp(plan.items_mu);
        pe = order_planes(plan, w.d, w.order, pairs, s, sms);
    }
    if (pe == cudaSuccess && w.order != 2)
        pe = px ? residue_copy(plan.layers->bits_by_residue, (const uint8_t*)plan.f4.bits, (size_t)8 * plan.f4.wpr,
                               w.d.snps, w.dist_step, s)
                : residue_copy(plan.layers->by_residue, plan.planes, (size_t)2 * plan.pitch, w.d.snps, w.dist_step, s);
    if (pe != cudaSuccess) return pe;
    uint8_t* perm = px || w.order == 2 ? nullptr : plan.layers->by_residue[w.dist_step];
    const int n = w.d.snps;
    const long long step = w.dist_step, offset = w.dist_offset;
    if (w.order == 4) {
        std::vector<long long> pb;
        std::vector<int4> pi;
        long long combos = 0;
        const long long total = t4_layer_items(n, (int)step, offset, px, pb, pi, combos);
        T3Layer L;
        L.total = total;
        L.n_tiles = (int)pi.size();
        L.item_combos = (double)combos / std::max(1ll, total);
        cudaError_t e = px ? f4_bit_map(&L.map_kr, plan.f4,
                                        (const uint32_t*)plan.layers->bits_by_residue[w.dist_step], 2 * n, 32)
                           : t3_map(&L.map_kr, perm, 2 * n, plan.pitch, 32, true);
        if (e == cudaSuccess) e = cudaMalloc((void**)&L.item_begin, pb.size() * sizeof(long long));
        if (e == cudaSuccess) e = cudaMalloc((void**)&L.pinfo, std::max<size_t>(1, pi.size()) * sizeof(int4));
        if (e == cudaSuccess)
            e = cudaMemcpy(L.item_begin, pb.data(), pb.size() * sizeof(long long), cudaMemcpyHostToDevice);
        if (e == cudaSuccess && !pi.empty())
            e = cudaMemcpy(L.pinfo, pi.data(), pi.size() * sizeof(int4), cudaMemcpyHostToDevice);
        if (e != cudaSuccess) {
            cudaFree(L.item_begin);
            cudaFree(L.pinfo);
            return e;
        }
        plan.layers->by[key] = L;
        return cudaSuccess;
    }
    if (w.order == 2) {
        // owned prefixes: SNPs i = offset + m step, in planes of their own
        const int count = offset < n ? (int)((n - offset + step - 1) / step) : 0;
        long long combos = 0;
        for (long long i = offset; i < n; i += step) combos += n - 1 - i;
        T3Layer L;
        const std::vector<long long> tb = t2x_items(n, count, offset, step, L.n_tiles);
        L.total = tb.back();
        L.item_combos = (double)combos / std::max(1ll, L.total);
        cudaError_t e = f4_ones_planes(w.d, plan.f4, count, (int)offset, (int)step, L.planes, s);
        if (e == cudaSuccess) e = cudaStreamSynchronize(s);
        if (e == cudaSuccess) e = f4_map_a2(&L.map_ar, plan.f4, L.planes, count);
        if (e == cudaSuccess) e = upload(L.item_begin, tb);
        if (e != cudaSuccess) {
            cudaFree(L.planes);
            return e;
        }
        plan.layers->by[key] = L;
        return cudaSuccess;
    }
    // order 3: owned prefixes (i, j): lexicographic ranks offset + m * step; the pairs
    // (i, j > i) have ranks base(i) + (j - i - 1), base(i) = i (n-1) - i (i-1) / 2
    std::vector<long long> ib((size_t)n + 1), jb((size_t)n + 1);
    std::vector<int> jl;
    long long total = 0, combos = 0;
    for (int i = 0; i < n; ++i) {
        ib[i] = total;
        jb[i] = (long long)jl.size();
        const long long base = (long long)i * (n - 1) - (long long)i * (i - 1) / 2, cnt = n - 1 - i;
        long long t = std::max(0ll, offset - base);
        t += ((offset - base - t) % step + step) % step;  // first t with base + t = offset (mod step)
        for (; t < cnt; t += step) {
            jl.push_back(i + 1 + (int)t);
            combos += n - 2 - i - t;
        }
        // the pair kernel's items, or the per-class kernel's of 32 listed j and 96 l
        for (size_t a = (size_t)jb[i]; a < jl.size(); a += px ? kPxJ : kT3J)
            total += px ? t3x_tiles(n, jl[a]) : (n - 1 - jl[a] + kT3L - 1) / kT3L;
    }
    ib[n] = total;
    jb[n] = (long long)jl.size();
    T3Layer L;
    L.total = total;
    L.item_combos = (double)combos / std::max(1ll, total);
    cudaError_t e = px ? f4_bit_map(&L.map_jr, plan.f4, (const uint32_t*)plan.layers->bits_by_residue[w.dist_step],
                                    2 * n, 2 * kT3J)
                       : t3_map(&L.map_jr, perm, 2 * n, plan.pitch, 2 * kT3J, true);
    if (e == cudaSuccess) e = cudaMalloc((void**)&L.item_begin, ib.size() * sizeof(long long));
    if (e == cudaSuccess) e = cudaMalloc((void**)&L.jl_begin, jb.size() * sizeof(long long));
    if (e == cudaSuccess) e = cudaMalloc((void**)&L.jlist, std::max<size_t>(1, jl.size()) * sizeof(int));
    if (e == cudaSuccess) e = cudaMemcpy(L.item_begin, ib.data(), ib.size() * sizeof(long long), cudaMemcpyHostToDevice);
    if (e == cudaSuccess) e = cudaMemcpy(L.jl_begin, jb.data(), jb.size() * sizeof(long long), cudaMemcpyHostToDevice);
    if (e == cudaSuccess && !jl.empty())
        e = cudaMemcpy(L.jlist, jl.data(), jl.size() * sizeof(int), cudaMemcpyHostToDevice);
    if (e != cudaSuccess) {
        cudaFree(L.item_begin);
        cudaFree(L.jl_begin);
        cudaFree(L.jlist);
        return e;
    }
    plan.layers->by[key] = L;
    return cudaSuccess;
}

bool tensor_live(const T3Plan& plan, const ScanWork& w) { return w.order == 2 || plan.pair3; }

long long tensor_units(const T3Plan& plan, const ScanWork& w) {
    if (is_layer(w)) {
        const T3Layer* L = find_layer(plan, w);
        return L ? L->total : 0;
    }
    return w.order == 2 ? plan.total2 : w.order == 4 ? plan.total4 : plan.total;
}
double tensor_item_combos(const T3Plan& plan, const ScanWork& w) {
    if (is_layer(w)) {
        const T3Layer* L = find_layer(plan, w);
        return L ? L->item_combos : 1.0;
    }
    return w.order == 2 ? plan.item2_combos : w.order == 4 ? plan.item4_combos : plan.item_combos;
}

void tensor3_release(T3Plan& plan) {
    if (plan.layers) {
        for (auto& kv : plan.layers->by) {
            cudaFree(kv.second.item_begin);
            cudaFree(kv.second.jl_begin);
            cudaFree(kv.second.jlist);
            cudaFree(kv.second.pinfo);
            cudaFree(kv.second.planes);
        }
        for (auto& kv : plan.layers->by_residue) cudaFree(kv.second);
        for (auto& kv : plan.layers->bits_by_residue) cudaFree(kv.second);
        delete plan.layers;
        plan.layers = nullptr;
    }
    f4_release(plan.f4);
    cudaFree(plan.planes);
    cudaFree(plan.item_begin);
    cudaFree(plan.item2_begin);
    cudaFree(plan.item4_begin);
    cudaFree(plan.item4_per);
    plan.planes = nullptr;
    plan.item_begin = nullptr;
    plan.item2_begin = nullptr;
    plan.item4_begin = nullptr;
    plan.item4_per = nullptr;
}

// Bound on |single-precision estimate - exact key / (ln2 * 2^32)| over the 81
// terms of one combination: with N the number of samples every partial sum is
// at most 2 N lg2 N (81 roundings of at most 2^-24 of it), lg2.approx is
// within 2^-18 of log2 on every input the kernel can see (measured worst case
// 1.93e-6, checked exhaustively against FP64 by fiu_probe_lg2_error), the
// x + 2^-20 shift moves each term by at most 2^-20 / ln 2 (counts below 16)
// or one rounding of the count, and the integer table rounds each term by
// 1/2.  Doubled.
static double t3_margin(int n_samples) {
    const double N = n_samples, lgN = std::log2(std::max(2.0, N)), B = 2 * N * lgN;
    const double u = std::ldexp(1.0, -24), e20 = std::ldexp(1.0, -20), e_lg2 = std::ldexp(1.0, -18);
    const double err = 81 * u * B + 2 * N * (18 * u + e_lg2) + 81 * e20 / std::log(2.0) +
                       2 * N * std::ldexp(1.0, -23) / std::log(2.0) + 81 * 0.5 / (std::log(2.0) * 4294967296.0);
    return 2 * err + 1e-3;
}

// Self-check of the bounded mbarrier wait the tensor kernels use: one thread
// initialises an mbarrier (one arrival expected), arrives on it first when
// `arrive` is set, then waits for phase 0 with the given limit in the same
// try-wait loop as t3_wait.  Without the arrival nothing completes the phase
// and the wait must give up after the limit; out[0] = 1 if it completed,
// out[1] = elapsed ns.
__global__ void t3_wait_probe_kernel(unsigned long long limit_ns, int arrive, unsigned long long* out) {
    __shared__ __align__(8) uint64_t bar;
    if (threadIdx.x != 0) return;
    asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_u32(&bar)));
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    if (arrive) asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(&bar)) : "memory");
    const unsigned long long t0 = t3_now();
    bool done = false;
    for (;;) {
        if (t3_try(smem_u32(&bar), 0)) {
            done = true;
            break;
        }
        if (t3_now() - t0 > limit_ns) break;
    }
    out[0] = done ? 1 : 0;
    out[1] = t3_now() - t0;
    asm volatile("mbarrier.inval.shared::cta.b64 [%0];" ::"r"(smem_u32(&bar)) : "memory");
}

cudaError_t probe_wait_limit(unsigned limit_us, int arrive, int* completed, double* elapsed_ms, cudaStream_t s) {
    unsigned long long* d = nullptr;
    cudaError_t e = cudaMallocAsync((void**)&d, 2 * sizeof(unsigned long long), s);
    if (e != cudaSuccess) return e;
    unsigned long long h[2] = {0, 0};
    t3_wait_probe_kernel<<<1, 32, 0, s>>>((unsigned long long)limit_us * 1000ull, arrive, d);
    count_launch();
    e = cudaGetLastError();
    if (e == cudaSuccess) e = cudaMemcpyAsync(h, d, sizeof(h), cudaMemcpyDeviceToHost, s);
    cudaFreeAsync(d, s);
    if (e == cudaSuccess) e = cudaStreamSynchronize(s);
    *completed = (int)h[0];
    *elapsed_ms = (double)h[1] / 1e6;
    return e;
}

// Every input of t3_lg2 in the kernel is x = (float)(c + 2^-20) for an integer
// count c in [0, max_c]; largest |t3_lg2(x) - log2(x)| over them, log2 in FP64.
__global__ void t3_lg2_probe_kernel(unsigned max_c, unsigned long long* worst_bits) {
    double worst = 0;
    for (unsigned c = blockIdx.x * blockDim.x + threadIdx.x; c <= max_c; c += gridDim.x * blockDim.x) {
        const float x = (float)c + 9.5367431640625e-07f;
        const double err = fabs((double)t3_lg2(x) - log2((double)x));
        worst = fmax(worst, err);
    }
    atomicMax(worst_bits, (unsigned long long)__double_as_longlong(worst));  // non-negative doubles order as integers
}

cudaError_t probe_lg2_error(unsigned max_c, double* max_abs_err, cudaStream_t s) {
    unsigned long long* d = nullptr;
    cudaError_t e = cudaMallocAsync((void**)&d, sizeof(unsigned long long), s);
    if (e != cudaSuccess) return e;
    unsigned long long h = 0;
    e = cudaMemsetAsync(d, 0, sizeof(unsigned long long), s);
    if (e == cudaSuccess) {
        t3_lg2_probe_kernel<<<256, 256, 0, s>>>(max_c, d);
        count_launch();
        e = cudaGetLastError();
    }
    if (e == cudaSuccess) e = cudaMemcpyAsync(&h, d, sizeof(h), cudaMemcpyDeviceToHost, s);
    cudaFreeAsync(d, s);
    if (e == cudaSuccess) e = cudaStreamSynchronize(s);
    double v;
    memcpy(&v, &h, sizeof(v));
    *max_abs_err = v;
    return e;
}

cudaError_t launch_tensor3(const ScanWork& w, const T3Plan& plan, long long g0, long long g1, const CandSink& sink,
                           uint32_t* dump, const uint32_t* single, const uint4* pairs, const uint4* triples,
                           int* status, cudaStream_t s, int sms) {
    if (w.order == 2) {
        const T3Layer* L = is_layer(w) ? find_layer(plan, w) : nullptr;
        if (is_layer(w) && (!L || !tensor_layer_ok(plan, w))) return cudaErrorInvalidValue;
        const T2xRange r{L ? L->item_begin : plan.item2_begin, L ? L->n_tiles : plan.n_itiles,
                         L ? &L->map_ar : &plan.f4.map_a2, &plan.f4.map_b2, L ? w.dist_offset : 0,
                         L ? w.dist_step : 1};
        return launch_tensor2x(w, plan.f4, r, g0, g1, sink, dump, single, status, s, sms);
    }
    if (w.order == 4) {
        const T3Layer* L = is_layer(w) ? find_layer(plan, w) : nullptr;
        if (is_layer(w) && (!L || !tensor_layer_ok(plan, w))) return cudaErrorInvalidValue;
        if (plan.pair3) {
            const T4xRange r = L ? T4xRange{L->item_begin, nullptr, &L->map_kr, L->pinfo, L->n_tiles}
                                 : T4xRange{plan.item4_begin, plan.item4_per, &plan.f4.map_k4};
            return launch_tensor4x(w, plan.f4, r, g0, g1, sink, dump, single, pairs, status, s, sms);
        }
        return launch_tensor4(w, plan.map_l4, L ? L->map_kr : plan.map_k4, plan.map_i,
                              L ? L->item_begin : plan.item4_begin, L ? nullptr : plan.item4_per, plan.k_cases, g0, g1,
                              sink, dump, single, pairs, triples, status, s, sms, L ? L->pinfo : nullptr,
                              L ? L->n_tiles : 0);
    }
    // set once, by whichever host thread comes first (thread-safe static initialisation)
    static const cudaError_t attr = [] {
        cudaError_t e = cudaFuncSetAttribute(tensor3_kernel<false>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                             (int)kT3Smem);
        if (e == cudaSuccess)
            e = cudaFuncSetAttribute(tensor3_kernel<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kT3Smem);
        return e;
    }();
    if (attr != cudaSuccess) return attr;
    const long long items = g1 - g0;
    if (items <= 0) return cudaSuccess;
    const double scale = 1.0 / (std::log(2.0) * 4294967296.0);
    const double thr = ((double)sink.thr - (double)w.base_key) * scale - t3_margin(w.d.n_cases + w.d.n_ctrls);
    const float thr_f = (float)std::max(-3.0e38, std::min(3.0e38, thr));
    const unsigned grid = (unsigned)(items < sms ? items : sms);
    T3Maps maps{plan.map_l, plan.map_j, plan.map_i};
    if (plan.pair3) {
        const T3Layer* L = is_layer(w) ? find_layer(plan, w) : nullptr;
        if (is_layer(w) && (!L || !tensor_layer_ok(plan, w))) return cudaErrorInvalidValue;
        const T3xRange r = L ? T3xRange{L->item_begin, &L->map_jr, L->jl_begin, L->jlist}
                             : T3xRange{plan.item_begin, &plan.f4.map_j};
        return launch_tensor3x(w, plan.f4, r, g0, g1, sink, dump, single, pairs,
                               t3_margin(w.d.n_cases + w.d.n_ctrls), status, s, sms);
    }
    if (is_layer(w)) {
        const T3Layer* L = find_layer(plan, w);
        if (!L || !tensor_layer_ok(plan, w)) return cudaErrorInvalidValue;
        const T3Maps lmaps{plan.map_l, L->map_jr, plan.map_i};
        tensor3_kernel<true><<<grid, kT3Threads, kT3Smem, s>>>(lmaps, w, L->item_begin, g0, g1, plan.k_cases, sink,
                                                               thr_f, dump, single, pairs, status, L->jl_begin,
                                                               L->jlist);
    } else {
        tensor3_kernel<false><<<grid, kT3Threads, kT3Smem, s>>>(maps, w, plan.item_begin, g0, g1, plan.k_cases, sink,
                                                                thr_f, dump, single, pairs, status, nullptr, nullptr);
    }
    count_launch();
    return cudaGetLastError();
}

}  // namespace fiu
