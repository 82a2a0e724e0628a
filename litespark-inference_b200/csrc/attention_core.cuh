// Device building blocks shared by the attention kernels: cache elements, rows of a cache, maxima by the integer reduction.
#pragma once
#include "common.cuh"

namespace lspk {

template <typename KVT> __device__ __forceinline__ float kv_load(const KVT* p);
template <> __device__ __forceinline__ float kv_load<float>(const float* p) { return *p; }
template <> __device__ __forceinline__ float kv_load<__half>(const __half* p) { return __half2float(*p); }
template <typename KVT> __device__ __forceinline__ KVT kv_make(float v);
template <> __device__ __forceinline__ float kv_make<float>(float v) { return v; }
template <> __device__ __forceinline__ __half kv_make<__half>(float v) { return __float2half_rn(v); }
template <typename KVT> __device__ __forceinline__ float kv_round(float v);
template <> __device__ __forceinline__ float kv_round<float>(float v) { return v; }
template <> __device__ __forceinline__ float kv_round<__half>(float v) { return __half2float(__float2half_rn(v)); }

// 16 bytes of cache row -> fp32 values (8 halves or 4 floats).
template <typename KVT> struct KvVec;
template <> struct KvVec<__half> {
    static constexpr int N = 8;
    static __device__ __forceinline__ void unpack(const uint4& c, float* f) {
        const __half2* h = reinterpret_cast<const __half2*>(&c);
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const float2 v = __half22float2(h[i]);
            f[2 * i] = v.x;
            f[2 * i + 1] = v.y;
        }
    }
};
template <> struct KvVec<float> {
    static constexpr int N = 4;
    static __device__ __forceinline__ void unpack(const uint4& c, float* f) {
        f[0] = __uint_as_float(c.x);
        f[1] = __uint_as_float(c.y);
        f[2] = __uint_as_float(c.z);
        f[3] = __uint_as_float(c.w);
    }
};

// Order-preserving map float -> uint32 (and back), so that a maximum over possibly negative floats
// can use the integer warp reduction.
__device__ __forceinline__ uint32_t float_to_ordered(float f) {
    const uint32_t u = __float_as_uint(f);
    return (u & 0x80000000u) ? ~u : (u | 0x80000000u);
}
__device__ __forceinline__ float ordered_to_float(uint32_t u) {
    return __uint_as_float((u & 0x80000000u) ? (u & 0x7fffffffu) : ~u);
}

}  // namespace lspk
