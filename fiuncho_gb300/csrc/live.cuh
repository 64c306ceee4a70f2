// Device side of the live threshold (CandSink::hist, live).
#pragma once

#include "internal.h"

namespace fiu {

__device__ __forceinline__ int live_bin(long long key) {
    if (key < (1ll << 30)) return 0;
    const int e = 63 - __clzll(key);
    return e > 47 ? kLiveBins - 1 : (e - 30) * 128 + (int)((key >> (e - 7)) & 127);
}
__device__ __forceinline__ long long live_edge(int bin) {
    const int e = bin / 128 + 30;
    return (128ll + bin % 128) << (e - 7);
}

// One warp: the lower edge of the highest bin at which `keep` candidates lie in it or above (the
// least key if there are fewer, or only with bin 0).  Every lane returns it.
__device__ __forceinline__ long long live_scan(const unsigned* hist, unsigned keep, int lane) {
    constexpr int kPer = kLiveBins / 32;
    static_assert(kLiveBins % 32 == 0, "bins per lane");
    const int top = kLiveBins - 1 - kPer * lane;  // lane 0 has the highest bins
    unsigned sum = 0;
#pragma unroll 8
    for (int b = 0; b < kPer; ++b) sum += __ldcg(hist + top - b);
    unsigned upto = sum;  // inclusive over the lanes
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
        const unsigned o = __shfl_up_sync(0xffffffffu, upto, d);
        if (lane >= d) upto += o;
    }
    const unsigned hit = __ballot_sync(0xffffffffu, upto >= keep);
    long long thr = (long long)0x8000000000000000ull;
    if (hit) {
        const int src = __ffs(hit) - 1;
        if (lane == src) {
            unsigned above = upto - sum;
            int b = top;
            for (int k = 0; k < kPer; ++k, --b) {
                above += __ldcg(hist + b);
                if (above >= keep) break;
            }
            if (b > 0 && b > top - kPer) thr = live_edge(b);
        }
        thr = __shfl_sync(0xffffffffu, thr, src);
    }
    return thr;
}

// One warp raises the launch's live threshold (nothing when it has risen past this already).
__device__ __forceinline__ void live_update(const CandSink& sink, int lane) {
    const long long thr = live_scan(sink.hist, sink.keep, lane);
    if (lane == 0 && thr > *(volatile long long*)sink.live) atomicMax(sink.live, thr);
}

// One lane's candidate: into the buffer and the histogram.
__device__ __forceinline__ void live_append(const CandSink& sink, long long key, unsigned long long code) {
    const unsigned idx = atomicAdd(sink.count, 1u);
    if (idx < sink.cap) {
        sink.buf[idx] = Cand{key, code};
        if (sink.hist) atomicAdd(sink.hist + live_bin(key), 1u);
    } else {
        atomicOr(sink.overflow, 1u);
    }
}

}  // namespace fiu
