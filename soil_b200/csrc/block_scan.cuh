// block_scan.cuh — CTA-wide exclusive scan of one u32 per thread (kBlock threads).
#pragma once

#include "soil_internal.cuh"

namespace soil {

// Exclusive block scan of one value per thread; returns the prefix of this
// thread and writes the block total to *total.
__device__ __forceinline__ uint32_t block_exclusive_scan(uint32_t v, uint32_t* total) {
    __shared__ uint32_t warp_tot[kBlock / 32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    uint32_t inc = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        uint32_t t = __shfl_up_sync(0xffffffffu, inc, o);
        if (lane >= o) inc += t;
    }
    if (lane == 31) warp_tot[warp] = inc;
    __syncthreads();
    if (warp == 0) {
        uint32_t w = lane < kBlock / 32 ? warp_tot[lane] : 0;
        uint32_t wi = w;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            uint32_t t = __shfl_up_sync(0xffffffffu, wi, o);
            if (lane >= o) wi += t;
        }
        if (lane < kBlock / 32) warp_tot[lane] = wi - w;  // exclusive warp offsets
        if (lane == kBlock / 32 - 1) *total = wi;
    }
    __syncthreads();
    const uint32_t res = warp_tot[warp] + inc - v;
    __syncthreads();
    return res;
}

// One CTA scans n values: out[t] (and out2[t] when given) = exclusive prefix
// of in over [0, n); returns the total.  ITEMS consecutive values per thread
// per pass, so a pass covers kBlock * ITEMS values.
template <int ITEMS>
__device__ __forceinline__ uint32_t cta_scan_array(const uint32_t* in, uint32_t* out,
                                                   uint32_t* out2, uint64_t n) {
    __shared__ uint32_t tot;
    uint32_t carry = 0;
    for (uint64_t b0 = 0; b0 < n; b0 += (uint64_t)kBlock * ITEMS) {
        const uint64_t t0 = b0 + (uint64_t)threadIdx.x * ITEMS;
        uint32_t v[ITEMS];
        uint32_t sum = 0;
#pragma unroll
        for (int j = 0; j < ITEMS; ++j) {
            v[j] = t0 + j < n ? in[t0 + j] : 0u;
            sum += v[j];
        }
        uint32_t run = block_exclusive_scan(sum, &tot) + carry;
#pragma unroll
        for (int j = 0; j < ITEMS; ++j) {
            if (t0 + j < n) {
                out[t0 + j] = run;
                if (out2) out2[t0 + j] = run;
            }
            run += v[j];
        }
        carry += tot;
        __syncthreads();
    }
    return carry;
}

constexpr int kScanItems = 8;  // consecutive counts per thread
constexpr int kScanTile = kBlock * kScanItems;

// A thread's 8 consecutive items [base, base + 8) (zero past n): two 16-byte
// loads when the group is whole and aligned, else one by one.
__device__ __forceinline__ void load8(const uint32_t* in, uint64_t base, uint64_t n,
                                      uint32_t (&v)[kScanItems]) {
    if (base + kScanItems <= n && (reinterpret_cast<uintptr_t>(in + base) & 15u) == 0) {
        const uint4 a = *reinterpret_cast<const uint4*>(in + base);
        const uint4 b = *reinterpret_cast<const uint4*>(in + base + 4);
        v[0] = a.x; v[1] = a.y; v[2] = a.z; v[3] = a.w;
        v[4] = b.x; v[5] = b.y; v[6] = b.z; v[7] = b.w;
        return;
    }
#pragma unroll
    for (int k = 0; k < kScanItems; ++k) v[k] = (base + k < n) ? in[base + k] : 0u;
}

// out[base + k] = pre + v[0] + ... + v[k - 1] for the items below n.
// With add, plus add[base + k].
__device__ __forceinline__ void store8_scan(uint32_t* out, uint64_t base, uint64_t n,
                                            const uint32_t (&v)[kScanItems], uint32_t pre,
                                            const uint32_t* add = nullptr) {
    uint32_t o[kScanItems];
    if (add) load8(add, base, n, o);
#pragma unroll
    for (int k = 0; k < kScanItems; ++k) {
        o[k] = add ? o[k] + pre : pre;
        pre += v[k];
    }
    if (base + kScanItems <= n && (reinterpret_cast<uintptr_t>(out + base) & 15u) == 0) {
        *reinterpret_cast<uint4*>(out + base) = make_uint4(o[0], o[1], o[2], o[3]);
        *reinterpret_cast<uint4*>(out + base + 4) = make_uint4(o[4], o[5], o[6], o[7]);
        return;
    }
#pragma unroll
    for (int k = 0; k < kScanItems; ++k)
        if (base + k < n) out[base + k] = o[k];
}

// A tile of the scan without waits between CTAs (k_scan.cu): 8,192 counts.
constexpr int kDirectThreads = 1024;
constexpr uint64_t kDirectTile = (uint64_t)kDirectThreads * kScanItems;

__device__ __forceinline__ uint32_t cta_exclusive_1024(uint32_t v, uint32_t* total) {
    __shared__ uint32_t w[32];
    static_assert(kDirectThreads == 32 * 32, "one warp scans the warps' sums");
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    uint32_t inc = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t t = __shfl_up_sync(0xffffffffu, inc, o);
        if (lane >= o) inc += t;
    }
    if (lane == 31) w[warp] = inc;
    __syncthreads();
    uint32_t x = w[lane], xi = x;  // every warp scans the sums: one barrier fewer
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t t = __shfl_up_sync(0xffffffffu, xi, o);
        if (lane >= o) xi += t;
    }
    *total = __shfl_sync(0xffffffffu, xi, 31);
    return __shfl_sync(0xffffffffu, xi - x, warp) + inc - v;
}

// This CTA's tile of the scan of in[0, n) (plus add[0, n] when given) into
// out[0, n]; returns the total on the threads of the last tile's CTA (else a
// prefix).
__device__ __forceinline__ uint32_t scan_direct_tile(const uint32_t* in, uint32_t* out, uint64_t n,
                                                     uint64_t tile, uint64_t ntiles,
                                                     const uint32_t* add) {
    __shared__ uint32_t before[32];
    const uint64_t base = tile * kDirectTile + (uint64_t)threadIdx.x * kScanItems;
    uint32_t v[kScanItems];
    load8(in, base, n, v);
    uint32_t c = 0;  // this thread's share of the counts before the tile
    const uint64_t first = tile * kDirectTile;
    if ((reinterpret_cast<uintptr_t>(in) & 15u) == 0) {
        const uint4* in4 = reinterpret_cast<const uint4*>(in);
#pragma unroll 8
        for (uint64_t k = threadIdx.x; k < first / 4; k += kDirectThreads) {
            const uint4 a = in4[k];
            c += a.x + a.y + a.z + a.w;
        }
    } else {
        for (uint64_t k = threadIdx.x; k < first; k += kDirectThreads) c += in[k];
    }
    c = __reduce_add_sync(0xffffffffu, c);
    if ((threadIdx.x & 31) == 0) before[threadIdx.x >> 5] = c;
    uint32_t s = 0, tot;
#pragma unroll
    for (int k = 0; k < kScanItems; ++k) s += v[k];
    const uint32_t in_tile = cta_exclusive_1024(s, &tot);  // its barrier covers `before`
    const uint32_t carry = __reduce_add_sync(0xffffffffu, before[threadIdx.x & 31]);
    store8_scan(out, base, n, v, carry + in_tile, add);
    if (tile + 1 == ntiles && threadIdx.x == 0) out[n] = carry + tot + (add ? add[n] : 0u);
    return carry + tot;
}

}  // namespace soil
