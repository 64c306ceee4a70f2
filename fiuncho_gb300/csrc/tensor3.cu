// Host side of the tensor-core kernels (tcgen05, 4-bit operands, CTA pairs):
// tensor2x.cu, tensor3x.cu and tensor4x.cu hold the kernels of orders 2, 3 and 4;
// here are a data set's plan (operand planes, work-item tables, the items of
// Distribution layers), the dispatch to them and two self-checks.
//
// Reference semantics: the combinations ThreadedSearch visits
// (include/fiuncho/ThreadedSearch.h:157-180), with one worker or with a
// Distribution layer's.
#include <cudaTypedefs.h>

#include <algorithm>
#include <cmath>
#include <cstring>
#include <map>
#include <tuple>
#include <mutex>

#include "tensor2x.h"
#include "tensor3m.h"
#include "tensor_bounds.h"
#include "tensor_common.cuh"

namespace fiu {

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

void tensor3_prepare(const DevData& d, T3Plan& plan) { f4_sizes(d, plan.f4); }

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
    const std::vector<long long> ib = plan.missing ? t3m_items(d.snps) : t3x_items(d.snps);
    plan.total = ib.back();
    const double n = d.snps;
    plan.item_combos = n * (n - 1) * (n - 2) / 6.0 / std::max(1ll, plan.total);
    return upload(plan.item_begin, ib);
}

// The operands of an order, made on its first search (items_mu held): the 4-bit layout and at order 4
// the cores of the triples.
static cudaError_t order_planes(T3Plan& plan, const DevData& d, int order, const uint4* pairs, cudaStream_t s,
                                int sms) {
    cudaError_t e = cudaSuccess;
    if (order == 2) {
        if (plan.f4.ones) return e;
        uint8_t* ones = nullptr;
        e = f4_ones_planes(d, plan.f4, d.snps, 0, 1, ones, s);
        if (e == cudaSuccess) e = cudaStreamSynchronize(s);
        if (e == cudaSuccess) e = f4_map_a2(&plan.f4.map_a2, plan.f4, ones, d.snps);
        if (e == cudaSuccess) e = f4_map_b2(&plan.f4.map_b2, plan.f4, ones, d.snps);
        if (e == cudaSuccess) plan.f4.ones = ones;  // (what is named here is complete)
        else cudaFree(ones);
        return e;
    }
    if (!plan.f4.bits) {
        // made apart: searches of order 2 may be reading what the plan holds
        F4Plan made = plan.f4;
        e = f4_prepare(d, made, plan.missing ? 3 : 2, s);
        if (e == cudaSuccess) e = cudaStreamSynchronize(s);
        if (e != cudaSuccess) {
            cudaFree(made.planes);
            return e;
        }
        plan.f4.map_b = made.map_b;
        plan.f4.map_j = made.map_j;
        plan.f4.map_i = made.map_i;
        plan.f4.map_b4h = made.map_b4h;
        plan.f4.rows = made.rows;
        plan.f4.planes = made.planes;
        plan.f4.bits = made.bits;
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
        const std::vector<long long> ib4 = t4_item_table(d.snps, per4);
        plan.total4 = ib4.back();
        const double n = d.snps;
        plan.item4_combos = n * (n - 1) * (n - 2) * (n - 3) / 24.0 / std::max(1ll, plan.total4);
        if (!plan.item4_per) e = upload(plan.item4_per, per4);
        if (e == cudaSuccess) e = upload(plan.item4_begin, ib4);
    }
    return e;
}

// Work items of Distribution layers of order-3 scans (the pair kernel's list
// mode), one entry per (step, offset) used on the data set.  The owned j of
// one i are the j > i of one residue mod step (pair ranks base(i) + j - i - 1
// step through the layer's offset class), so in a copy of the bit rows
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
    CUtensorMap map_jr;               // order 3: 64 residue-ordered bit rows
    uint8_t* planes = nullptr;        // order 2: the owned SNPs' planes
    CUtensorMap map_ar;               // order 2: box 128 B x 128 rows over them
    CUtensorMap map_kr;               // order 4: 32 residue-ordered bit rows
};
struct T3Layers {
    std::mutex mu;
    std::map<std::tuple<int, int, int>, T3Layer> by;  // (order, step, offset)
    std::map<int, uint8_t*> bits_by_residue;  // residue-ordered bit rows (orders 3 and 4), per layer_step
};

// Bit rows (2 an SNP, wpr words each) ordered by residue, 16 bytes a thread.
__global__ void residue_rows_kernel(const uint4* __restrict__ src, uint4* __restrict__ dst, int n, int step,
                                    int per_snp) {
    const long long total = (long long)n * per_snp;
    for (long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x; e < total;
         e += (long long)gridDim.x * blockDim.x) {
        const int row = (int)(e / per_snp), o = (int)(e - (long long)row * per_snp);
        dst[e] = __ldg(src + (long long)residue_snp(row, step, n) * per_snp + o);
    }
}

// The bit rows ordered by residue mod step (layer_step's), made on first use.  (A kernel: a copy with
// the step as its pitch is refused from 2 GB on, which a step of a few hundred thousand SNPs reaches.)
static cudaError_t residue_copy(std::map<int, uint8_t*>& by, const F4Plan& f, int n, int step, cudaStream_t s) {
    if (by.count(step)) return cudaSuccess;
    const int per_snp = f.wpr / 2;  // 2 rows of wpr words; wpr is a multiple of 8
    uint8_t* perm = nullptr;
    cudaError_t e = cudaMalloc((void**)&perm, (size_t)n * per_snp * 16);
    if (e != cudaSuccess) return e;
    const long long total = (long long)n * per_snp;
    residue_rows_kernel<<<(unsigned)std::min<long long>((total + 255) / 256, 8192), 256, 0, s>>>(
        reinterpret_cast<const uint4*>(f.bits), reinterpret_cast<uint4*>(perm), n, step, per_snp);
    count_launch();
    e = cudaGetLastError();
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
    {
        std::lock_guard<std::mutex> gp(plan.items_mu);
        if (!plan.layers) plan.layers = new T3Layers;
    }
    std::lock_guard<std::mutex> g(plan.layers->mu);
    const auto key = std::make_tuple(w.order, w.dist_step, w.dist_offset);
    if (plan.layers->by.count(key)) return cudaSuccess;
    cudaError_t pe;
    {
        std::lock_guard<std::mutex> gp(plan.items_mu);
        pe = order_planes(plan, w.d, w.order, pairs, s, sms);
    }
    if (pe == cudaSuccess && w.order != 2)
        pe = residue_copy(plan.layers->bits_by_residue, plan.f4, w.d.snps, layer_step(w.dist_step, w.d.snps), s);
    if (pe != cudaSuccess) return pe;
    const int n = w.d.snps, pstep = layer_step(w.dist_step, n);
    const long long step = w.dist_step, offset = w.dist_offset;
    if (w.order == 4) {
        std::vector<long long> pb;
        std::vector<int4> pi;
        long long combos = 0;
        const long long total = t4_layer_items(n, (int)step, offset, pb, pi, combos);
        T3Layer L;
        L.total = total;
        L.n_tiles = (int)pi.size();
        L.item_combos = (double)combos / std::max(1ll, total);
        cudaError_t e = f4_bit_map(&L.map_kr, plan.f4, (const uint32_t*)plan.layers->bits_by_residue[pstep],
                                   2 * n, 32);
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
        for (size_t a = (size_t)jb[i]; a < jl.size(); a += kPxJ) total += t3x_tiles(n, jl[a]);
    }
    ib[n] = total;
    jb[n] = (long long)jl.size();
    T3Layer L;
    L.total = total;
    L.item_combos = (double)combos / std::max(1ll, total);
    cudaError_t e = f4_bit_map(&L.map_jr, plan.f4, (const uint32_t*)plan.layers->bits_by_residue[pstep], 2 * n,
                               kPxJ);
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
        for (auto& kv : plan.layers->bits_by_residue) cudaFree(kv.second);
        delete plan.layers;
        plan.layers = nullptr;
    }
    f4_release(plan.f4);
    cudaFree(plan.item_begin);
    cudaFree(plan.item2_begin);
    cudaFree(plan.item4_begin);
    cudaFree(plan.item4_per);
    plan.item_begin = nullptr;
    plan.item2_begin = nullptr;
    plan.item4_begin = nullptr;
    plan.item4_per = nullptr;
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
                           uint32_t* dump, const uint32_t* single, const uint4* pairs, int* status, cudaStream_t s,
                           int sms) {
    const T3Layer* L = is_layer(w) ? find_layer(plan, w) : nullptr;
    if (is_layer(w) && (!L || !tensor_layer_ok(plan, w))) return cudaErrorInvalidValue;
    if (w.order == 2) {
        const T2xRange r{L ? L->item_begin : plan.item2_begin, L ? L->n_tiles : plan.n_itiles,
                         L ? &L->map_ar : &plan.f4.map_a2, &plan.f4.map_b2, L ? w.dist_offset : 0,
                         L ? layer_step(w.dist_step, w.d.snps) : 1};
        return launch_tensor2x(w, plan.f4, r, g0, g1, sink, dump, single, status, s, sms);
    }
    if (w.order == 4) {
        const T4xRange r = L ? T4xRange{L->item_begin, nullptr, &L->map_kr, L->pinfo, L->n_tiles}
                             : T4xRange{plan.item4_begin, plan.item4_per, &plan.f4.map_k4};
        return launch_tensor4x(w, plan.f4, r, g0, g1, sink, dump, single, pairs, status, s, sms);
    }
    const double margin = t3_margin(w.d.n_cases + w.d.n_ctrls);
    if (plan.missing) return launch_tensor3m(w, plan.f4, plan.item_begin, g0, g1, sink, margin, status, s, sms);
    const T3xRange r = L ? T3xRange{L->item_begin, &L->map_jr, L->jl_begin, L->jlist}
                         : T3xRange{plan.item_begin, &plan.f4.map_j};
    return launch_tensor3x(w, plan.f4, r, g0, g1, sink, dump, single, pairs, margin, status, s, sms);
}

}  // namespace fiu
