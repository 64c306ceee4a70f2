// Device helpers of the tcgen05 kernels on 4-bit operands (kind::mxf4).
//
// Operands are genotype indicators, 0 or 1 (or 0 and a power of two, with the
// other operand's the inverse): e2m1 holds them exactly and tcgen05.mma kind::mxf4 sums their products in FP32, exactly
// up to 2^24, at twice the samples per instruction of e4m3 (M 128 x N 256:
// 64 samples in 128 cycles against 32; measured, every sum equal to the
// integer one up to 1.67e7).  The block scales (ue8m0, one per 32 samples of a
// row) are the same for every row and block of an instruction, so their layout
// in tensor memory does not matter: a region of 8 columns filled with 2^0 and
// one filled with 2^p, written once per launch.  The second is used as the B
// scale of control samples when both classes share an accumulator, which then
// holds cases + 2^p * controls.
#pragma once

#include <algorithm>
#include <cmath>

#include "tensor_bounds.h"
#include "tensor_common.cuh"

namespace fiu {

constexpr int kF4K = 256;                        // samples per 128-byte operand row and pipeline stage

// Instruction descriptor: e2m1 x e2m1 (format 1 at bits 7 and 10), ue8m0 scales (bit 23), N / 8, M / 16.
__host__ __device__ constexpr uint32_t f4_idesc(int M, int N) {
    return (1u << 7) | (1u << 10) | ((uint32_t)(N >> 3) << 17) | (1u << 23) | ((uint32_t)(M >> 4) << 24);
}

__device__ __forceinline__ void f4_mma(uint32_t d, uint64_t a, uint64_t b, uint32_t idesc, uint32_t sfa, uint32_t sfb,
                                       uint32_t acc) {
    asm volatile(
        "{.reg .pred p; setp.ne.b32 p, %6, 0;\n"
        "tcgen05.mma.cta_group::2.kind::mxf4.block_scale.block32 [%0], %1, %2, %3, [%4], [%5], p;}\n" ::"r"(d),
        "l"(a), "l"(b), "r"(idesc), "r"(sfa), "r"(sfb), "r"(acc));
}

// The MMA issuer of a CTA-pair kernel (one elected thread of CTA 0): for each of
// `items` items the GEMM of M 256 x n_of(item) columns over the class's 64-sample
// steps.  A tiles come from a ring of kA stages of kAStage bytes at a0 (full0), B
// tiles from a ring of kB stages of kBStage bytes at b0, released by empty0 (kB
// barriers); accumulator regions of kRegion columns alternate by acc_full0 /
// acc_empty0.  SPLIT (classes that do not share an accumulator): the cases of an
// item, then its controls, are two GEMMs, each into a region of its own.
// Returns false after a wait that gave up.  Its own time per stage
// counts (about 230 cycles alone on an SM quarter, up to twice that beside other
// warps, against 480 of MMA at N 240), so the loop holds what it must and decodes
// no items.
template <bool SPLIT, int kA, int kAStage, int kB, int kBStage, int kRegion, int kOne, int kW, class NOf>
__device__ __forceinline__ bool f4_pair_issue(long long items, uint32_t a0, uint32_t b0, uint32_t full0,
                                              uint32_t empty0, uint32_t acc_full0, uint32_t acc_empty0, uint32_t tmem,
                                              int nw_c, int nw_t, volatile int* abort, NOf&& n_of) {
    const uint32_t desc_hi = (uint32_t)(t3_desc(0) >> 32), desc_a = (uint32_t)t3_desc(a0), desc_b = (uint32_t)t3_desc(b0);
    const uint32_t one = tmem + (uint32_t)kOne;
    uint32_t fbar = 0, ad = desc_a, par = 0;  // A stage: barrier offset, descriptor, parity
    uint32_t ebar = 0, bd = desc_b;           // B stage
    for (unsigned item = 0; item < (SPLIT ? 2 : 1) * items; ++item) {
        const unsigned buf = item & 1;
        if (item >= 2 && !t3_wait_cl(acc_empty0 + 8 * buf, ((item >> 1) - 1) & 1, abort)) return false;
        const uint32_t dcol = tmem + (uint32_t)(kRegion * buf);
        uint32_t acc = 0, idesc = 0;
        for (int cls = SPLIT ? (int)buf : 0; cls < (SPLIT ? (int)buf + 1 : 2); ++cls) {
            const uint32_t sfb = tmem + (uint32_t)(cls && !SPLIT ? kW : kOne);
            for (int left = cls ? nw_t : nw_c; left > 0; left -= 4) {
                if (!t3_wait_cl(full0 + fbar, par, abort)) return false;  // both CTAs' A and B are in place
                asm volatile("tcgen05.fence::after_thread_sync;");
                if (!acc) idesc = f4_idesc(256, n_of(SPLIT ? item >> 1 : item));
                auto mma = [&](int k) {
                    f4_mma(dcol, (uint64_t)desc_hi << 32 | (ad + 2 * k), (uint64_t)desc_hi << 32 | (bd + 2 * k), idesc,
                           one, sfb, acc);
                    acc = 1;
                };
                mma(0);
                if (left >= 4) {
                    mma(1);
                    mma(2);
                    mma(3);
                } else {  // the class's last steps
                    for (int k = 1; k < left; ++k) mma(k);
                }
                commit_pair(empty0 + ebar);
                fbar += 8;
                ad += kAStage >> 4;
                if (fbar == 8 * kA) {
                    fbar = 0;
                    ad = desc_a;
                    par ^= 1;
                }
                ebar += 8;
                bd += kBStage >> 4;
                if (ebar == 8 * kB) {
                    ebar = 0;
                    bd = desc_b;
                }
            }
        }
        commit_pair(acc_full0 + 8 * buf);
    }
    return true;
}

// Fills this warp's 32 tensor-memory lanes of both scale regions, `cols` (a
// multiple of 8) columns each: 8 hold the scales of 256 rows.  Every lane
// quarter has to be filled by one warp whose index is the quarter mod 4.
template <int cols>
__device__ __forceinline__ void f4_fill_scales(uint32_t tmem, int q, int col_one, int col_w, int p) {
    const uint32_t base = tmem + ((uint32_t)(32 * q) << 16);
    const uint32_t one = 0x7F7F7F7Fu, w = (uint32_t)(0x7F + p) * 0x01010101u;
#pragma unroll
    for (int c = 0; c < cols; c += 4) {
        asm volatile("tcgen05.st.sync.aligned.32x32b.x4.b32 [%0], {%1, %1, %1, %1};" ::"r"(base + col_one + c),
                     "r"(one));
        asm volatile("tcgen05.st.sync.aligned.32x32b.x4.b32 [%0], {%1, %1, %1, %1};" ::"r"(base + col_w + c),
                     "r"(w));
    }
    asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
}

// Operand bytes of 32 samples, one bit each: nibble u of word t belongs to bit
// 4 u + t.  A bit is used where it stands or after one shift, so A has it as
// 0.5, 1, 2 and 1 in words 0 to 3 and B as 2, 1, 0.5 and 1: the products of
// two set bits are 1.  A is the AND of two (the shift and mask of a word are
// then 6 operations, against 8 with 1.0 everywhere).
__device__ __forceinline__ uint4 f4_expand_a(uint32_t i, uint32_t j) {
    const uint32_t v = i & j;
    return make_uint4(i & j & 0x11111111u, i & j & 0x22222222u, i & j & 0x44444444u, (v >> 2) & 0x22222222u);
}
__device__ __forceinline__ uint4 f4_expand_b(uint32_t w) {
    const uint32_t v = w >> 2;
    return make_uint4((w << 2) & 0x44444444u, w & 0x22222222u, v & 0x11111111u, v & 0x22222222u);
}

// 1.0 wherever a bit is set: planes that both operands of an MMA are read from.
__device__ __forceinline__ uint4 f4_expand_ones(uint32_t w) {
    return make_uint4((w << 1) & 0x22222222u, w & 0x22222222u, (w >> 1) & 0x22222222u, (w >> 2) & 0x22222222u);
}

// Row of SNP l, genotype z in the operand planes: SNPs in groups of 8, the
// eight rows of genotype 0 before the eight of genotype 1, so that a thread
// reading 16x256b accumulator columns finds two neighbouring SNPs in a
// register pair and the two genotypes in successive 8-column blocks.
__host__ __device__ __forceinline__ int f4_row(int l, int z) { return 16 * (l >> 3) + 8 * z + (l & 7); }

// ---- two single-precision values per operation (f32x2) -----------------------
// Same arithmetic rate as the scalar forms (measured: 2 cycles against 1 per
// warp instruction) at half the issue slots.
using f2 = unsigned long long;
__device__ __forceinline__ f2 f2_pack(float a, float b) {
    f2 r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
    return r;
}
__device__ __forceinline__ void f2_unpack(f2 v, float& a, float& b) {
    asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(v));
}
__device__ __forceinline__ f2 f2_dup(float a) { return f2_pack(a, a); }
__device__ __forceinline__ f2 f2_add(f2 a, f2 b) {
    f2 r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ f2 f2_sub(f2 a, f2 b) {
    f2 r;
    asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ f2 f2_mul(f2 a, f2 b) {
    f2 r;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ f2 f2_fma(f2 a, f2 b, f2 c) {
    f2 r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
    return r;
}
__device__ __forceinline__ f2 f2_fma_rz(f2 a, f2 b, f2 c) {
    f2 r;
    asm("fma.rz.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
    return r;
}
__device__ __forceinline__ f2 f2_rcp(f2 v) {
    float a, b;
    f2_unpack(v, a, b);
    asm("rcp.approx.ftz.f32 %0, %0;" : "+f"(a));
    asm("rcp.approx.ftz.f32 %0, %0;" : "+f"(b));
    return f2_pack(a, b);
}

// ---- the quadratic bound on the mutual information (tensor_bounds.h) -------------
// One reciprocal a cell instead of three logarithms.  For q = 1/2 the bound is at
// most 4 / (2 / ln2) = 1.39 times the value, so nearly every combination falls
// below a top-N threshold and its logarithms are never taken.
//
// Cells arrive packed, D = cases + W controls (exact in FP32): controls =
// floor(D / W) by a fused multiply-add that rounds toward zero at 2^23.
struct F4Bound {
    f2 inv_w, m23, neg_m23, neg_w1, tiny, acc;
    __device__ __forceinline__ explicit F4Bound(int p) {
        inv_w = f2_dup(__uint_as_float((uint32_t)(127 - p) << 23));
        m23 = f2_dup(8388608.0f);
        neg_m23 = f2_dup(-8388608.0f);
        neg_w1 = f2_dup(1.0f - (float)(1 << p));
        tiny = f2_dup(9.5367431640625e-07f);  // 2^-20
        acc = 0;
    }
    // controls b and size s (+ 2^-20, so that an empty cell divides by no zero) of packed cells D
    __device__ __forceinline__ void split(f2 D, f2& b, f2& s) const {
        b = f2_add(f2_fma_rz(D, inv_w, m23), neg_m23);
        s = f2_add(f2_fma(neg_w1, b, D), tiny);
    }
    __device__ __forceinline__ void one(f2 D) {
        f2 b, s;
        split(D, b, s);
        acc = f2_fma(b, f2_mul(b, f2_rcp(s)), acc);
    }
    // two cells with one reciprocal: (b1^2 s2 + b2^2 s1) / (s1 s2)
    __device__ __forceinline__ void two(f2 b1, f2 s1, f2 b2, f2 s2) {
        const f2 r = f2_rcp(f2_mul(s1, s2));
        const f2 num = f2_fma(f2_mul(b1, b1), s2, f2_mul(f2_mul(b2, b2), s1));
        acc = f2_fma(num, r, acc);
    }
    __device__ __forceinline__ void two(f2 D1, f2 D2) {
        f2 b1, s1, b2, s2;
        split(D1, b1, s1);
        split(D2, b2, s2);
        two(b1, s1, b2, s2);
    }
};

// Both classes' counts beside each other, from 16-bit halves of the words c and t.
__device__ __forceinline__ f2 f4_ab(uint32_t c, uint32_t t, int hi) {
    const uint32_t sel = hi ? 0x7632 : 0x7610;
    return f2_add(f2_pack(__uint_as_float(__byte_perm(c, 0x4B000000u, sel)),
                          __uint_as_float(__byte_perm(t, 0x4B000000u, sel))),
                  f2_dup(-8388608.0f));
}
// The same of a word cases | controls << 16.
__device__ __forceinline__ f2 f4_ab(uint32_t w) {
    return f2_add(f2_pack(__uint_as_float(__byte_perm(w, 0x4B000000u, 0x7610)),
                          __uint_as_float(__byte_perm(w, 0x4B000000u, 0x7632))),
                  f2_dup(-8388608.0f));
}
// The quadratic bound with the cases and controls of one combination's cells side by side.
struct F4BoundAB {
    float acc = 0.f;
    __device__ __forceinline__ void one(f2 ab) {
        float a, b, r;
        f2_unpack(ab, a, b);
        asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"((a + b) + 9.5367431640625e-07f));
        acc = fmaf(b, b * r, acc);
    }
};

// A closer bound (tensor_bounds.h), for tables of many cells: at order 4 the
// quadratic one leaves a third of the warps a survivor.
struct F4Bound4 : F4Bound {
    f2 a2, a3, a4;
    __device__ __forceinline__ F4Bound4(int p, const F4Quartic& k) : F4Bound(p) {
        a2 = f2_dup(k.a2);
        a3 = f2_dup(k.a3);
        a4 = f2_dup(k.a4);
    }
    __device__ __forceinline__ void one(f2 D) {
        f2 b, s;
        split(D, b, s);
        const f2 pr = f2_mul(b, f2_rcp(s));
        acc = f2_fma(f2_mul(b, pr), f2_fma(pr, f2_fma(pr, a4, a3), a2), acc);
    }
};
struct F4Bound4AB {
    F4Quartic k;
    float acc = 0.f;
    __device__ __forceinline__ explicit F4Bound4AB(const F4Quartic& q) : k(q) {}
    __device__ __forceinline__ void one(f2 ab) {
        float a, b, r;
        f2_unpack(ab, a, b);
        asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"((a + b) + 9.5367431640625e-07f));
        const float pr = b * r;
        acc = fmaf(b * pr, fmaf(pr, fmaf(pr, k.a4, k.a3), k.a2), acc);
    }
};
// A threshold key as the kernels' tests, rounded down (device).
__device__ __forceinline__ void live_tests(const LiveMap& m, long long thr, float& est, float& bound) {
    est = __double2float_rd(fma((double)thr, m.est_k, m.est_c));
    bound = __double2float_rd(fma((double)thr, m.bound_k, m.bound_c));
}

}  // namespace fiu
