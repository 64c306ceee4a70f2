// Evaluation of one order-3 combination on the per-class kernel's core counts (tensor3.cu).
#pragma once

#include "tensor_common.cuh"

namespace fiu {

// Float view of the packed 16-bit pair cores [class][x][y].
__device__ __forceinline__ float pcf(const uint4& v, int k) {
    const uint32_t w = (&v.x)[k >> 1];
    return u2f((k & 1) ? (w >> 16) : (w & 0xffffu));
}

// Full 27-cell table of one class in single precision (every value an exact
// integer), the derivation of expand3: core[(x*2+y)*2+z], pair cores of
// (i,j), (i,l), (j,l), singles of i, j, l, class size.
__device__ __forceinline__ void expand3f(const float* core, const uint4& pij, const uint4& pil, const uint4& pjl,
                                         const float* si, const float* sj, const float* sl, float ncls, int cls,
                                         float* t) {
    const int o = 4 * cls;
#pragma unroll
    for (int x = 0; x < 2; ++x)
#pragma unroll
        for (int y = 0; y < 2; ++y) {
            t[(x * 3 + y) * 3 + 0] = core[(x * 2 + y) * 2 + 0];
            t[(x * 3 + y) * 3 + 1] = core[(x * 2 + y) * 2 + 1];
            t[(x * 3 + y) * 3 + 2] = pcf(pij, o + x * 2 + y);
        }
#pragma unroll
    for (int x = 0; x < 2; ++x) {
#pragma unroll
        for (int z = 0; z < 2; ++z) t[(x * 3 + 2) * 3 + z] = pcf(pil, o + x * 2 + z);
        t[(x * 3 + 2) * 3 + 2] = si[x];
    }
#pragma unroll
    for (int y = 0; y < 2; ++y) {
#pragma unroll
        for (int z = 0; z < 2; ++z) t[(2 * 3 + y) * 3 + z] = pcf(pjl, o + y * 2 + z);
        t[(2 * 3 + y) * 3 + 2] = sj[y];
    }
    t[24] = sl[0];
    t[25] = sl[1];
    t[26] = ncls;
#pragma unroll
    for (int xy = 0; xy < 9; ++xy) t[xy * 3 + 2] -= t[xy * 3 + 0] + t[xy * 3 + 1];
#pragma unroll
    for (int x = 0; x < 3; ++x)
#pragma unroll
        for (int z = 0; z < 3; ++z) t[(x * 3 + 2) * 3 + z] -= t[(x * 3 + 0) * 3 + z] + t[(x * 3 + 1) * 3 + z];
#pragma unroll
    for (int yz = 0; yz < 9; ++yz) t[18 + yz] -= t[yz] + t[9 + yz];
}

// Evaluates combination (i, j, l) from its 16 core counts (core[class][(x*2+y)*2+z]): exact 27-cell
// tables, the bounded single-precision prefilter, the exact fixed-point key for survivors, and the
// warp-aggregated append of candidates (warp-synchronous: every lane calls it).
__device__ __forceinline__ void t3_eval_core(const ScanWork& w, const CandSink& sink, float thr_f, uint32_t* dump,
                                             const uint32_t* __restrict__ single, const uint4* __restrict__ pairs,
                                             const float (&core)[2][8], int i, int j, int l, bool valid,
                                             const uint4& pij, const float (&si)[2][2], const float (&sj)[2][2],
                                             int lane) {
    const DevData& d = w.d;
    const int n = d.snps;
    const uint32_t ncls[2] = {(uint32_t)d.n_cases, (uint32_t)d.n_ctrls};
    const float ncf[2] = {(float)d.n_cases, (float)d.n_ctrls};
    const float tiny = 9.5367431640625e-07f;  // 2^-20: x*lg2(x + tiny) = 0 at x = 0
    uint4 pil = make_uint4(0, 0, 0, 0), pjl = pil, sl4 = pil;
    if (valid) {
        pjl = __ldg(pairs + pair_index(j, l, n));
        pil = __ldg(pairs + pair_index(i, l, n));
        sl4 = __ldg(reinterpret_cast<const uint4*>(single) + l);
    }
    const float sl[2][2] = {{u2f(sl4.x), u2f(sl4.y)}, {u2f(sl4.z), u2f(sl4.w)}};
    float t[2][27];
#pragma unroll
    for (int cls = 0; cls < 2; ++cls)
        expand3f(core[cls], pij, pil, pjl, si[cls], sj[cls], sl[cls], ncf[cls], cls, t[cls]);
    // single-precision estimate of sum over cells of T[a] + T[b] - T[a+b], in units of ln2 * 2^32
    float kf = 0.f;
#pragma unroll
    for (int c = 0; c < 27; ++c) {
        const float a = t[0][c], bb = t[1][c], s = a + bb;
        kf = fmaf(a, t3_lg2(a + tiny), kf);
        kf = fmaf(bb, t3_lg2(bb + tiny), kf);
        kf = fmaf(-s, t3_lg2(s + tiny), kf);
    }
    const bool cand = valid && (dump != nullptr || sink.digest != nullptr || kf >= thr_f);
    long long key = w.base_key;
    bool pass = false;
    unsigned long long dg = 0;
    if (cand) {
#pragma unroll
        for (int c = 0; c < 27; ++c) {
            const uint32_t a = min(f2u(fmaxf(t[0][c], 0.f)), ncls[0]);
            const uint32_t bb = min(f2u(fmaxf(t[1][c], 0.f)), ncls[1]);
            key += __ldg(d.ftab + a) + __ldg(d.ftab + bb) - __ldg(d.ftab + a + bb);
        }
        pass = key >= sink.thr;
        if (dump) {
            // owned prefix ordinal m of (i, j): rank offset + m * step
            const size_t m = (size_t)((pair_index(i, j, n) - w.dist_offset) / w.dist_step);
            uint32_t* o = dump + (m * n + l) * 54;
#pragma unroll
            for (int c = 0; c < 27; ++c) {
                o[c] = f2u(t[0][c]);
                o[27 + c] = f2u(t[1][c]);
            }
        }
        if (sink.digest) {
            const int cmb[3] = {i, j, l};
            dg = dg_begin(cmb, 3, n);
#pragma unroll
            for (int c = 0; c < 27; ++c) dg = dg_cell(dg, f2u(t[0][c]), f2u(t[1][c]));
        }
    }
    if (sink.digest) dg_warp_add(sink.digest, dg);
    const unsigned mask = __ballot_sync(0xffffffffu, pass);
    if (mask) {
        const int leader = __ffs(mask) - 1;
        unsigned base = 0;
        if (lane == leader) base = atomicAdd(sink.count, (unsigned)__popc(mask));
        base = __shfl_sync(0xffffffffu, base, leader);
        if (pass) {
            const unsigned idx = base + __popc(mask & ((1u << lane) - 1u));
            if (idx < sink.cap) {
                const int cmb[3] = {i, j, l};
                sink.buf[idx] = Cand{key, pack_code(cmb, 3, w.bits)};
            } else {
                atomicOr(sink.overflow, 1u);
            }
        }
    }
}

// Per-item constants of one j: the pair cores of (i, j) and the single cores of i and j as floats.
__device__ __forceinline__ void t3_item_consts(const uint32_t* __restrict__ single, const uint4* __restrict__ pairs,
                                               int i, int j, int n, bool j_ok, uint4& pij, float (&si)[2][2],
                                               float (&sj)[2][2]) {
    const uint4 a = __ldg(reinterpret_cast<const uint4*>(single) + i);
    uint4 b = make_uint4(0, 0, 0, 0);
    pij = make_uint4(0, 0, 0, 0);
    if (j_ok) {
        b = __ldg(reinterpret_cast<const uint4*>(single) + j);
        pij = __ldg(pairs + pair_index(i, j, n));
    }
    si[0][0] = u2f(a.x);
    si[0][1] = u2f(a.y);
    si[1][0] = u2f(a.z);
    si[1][1] = u2f(a.w);
    sj[0][0] = u2f(b.x);
    sj[0][1] = u2f(b.y);
    sj[1][0] = u2f(b.z);
    sj[1][1] = u2f(b.w);
}

}  // namespace fiu
