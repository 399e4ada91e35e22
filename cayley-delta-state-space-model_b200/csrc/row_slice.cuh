// A row of head_dim values over the lanes of a group: kCols contiguous columns per lane, 16-byte accesses where the row is
// exactly kCols x lanes long.
#pragma once
#include "cdssm_common.cuh"

namespace cdssm {

template <int kLanes = 8>
__device__ __forceinline__ float group_sum(float v) {   // sum over the kLanes (8 or 16) lanes of a unit
    v += __shfl_xor_sync(0xffffffffu, v, 1);
    v += __shfl_xor_sync(0xffffffffu, v, 2);
    v += __shfl_xor_sync(0xffffffffu, v, 4);
    if (kLanes == 16) v += __shfl_xor_sync(0xffffffffu, v, 8);
    return v;
}

// Raw (storage-typed) slice of one row: kCols contiguous columns starting at g*kCols.  (Plain loads: kernels that start
// before their predecessor has finished must not move them above the wait, which __ldg would allow.)
template <typename T, int kCols> struct RowSlice;
template <int kCols> struct RowSlice<__nv_bfloat16, kCols> {
    uint4 v[kCols / 8];
    __device__ __forceinline__ void load(const __nv_bfloat16* row, int g, int D, bool vec) {
        if (vec) {
            const uint4* p = reinterpret_cast<const uint4*>(row + g * kCols);
#pragma unroll
            for (int i = 0; i < kCols / 8; i++) v[i] = p[i];
        } else {
            unsigned short* s = reinterpret_cast<unsigned short*>(v);
#pragma unroll
            for (int i = 0; i < kCols; i++) {
                const int d = g * kCols + i;
                s[i] = d < D ? reinterpret_cast<const unsigned short*>(row)[d] : (unsigned short)0;
            }
        }
    }
    __device__ __forceinline__ void zero() {
#pragma unroll
        for (int i = 0; i < kCols / 8; i++) v[i] = make_uint4(0, 0, 0, 0);
    }
    __device__ __forceinline__ void get(float* f) const {
#pragma unroll
        for (int i = 0; i < kCols / 8; i++) unpack8(v[i], f + 8 * i);
    }
    static __device__ __forceinline__ void store(__nv_bfloat16* row, int g, int D, bool vec, const float* f) {
        if (vec) {
#pragma unroll
            for (int i = 0; i < kCols / 8; i++) Vec8<__nv_bfloat16>::st(row + g * kCols + 8 * i, f + 8 * i);
        } else {
#pragma unroll
            for (int i = 0; i < kCols; i++)
                if (g * kCols + i < D) IO<__nv_bfloat16>::st(row + g * kCols + i, f[i]);
        }
    }
};
template <int kCols> struct RowSlice<float, kCols> {
    float4 v[kCols / 4];
    __device__ __forceinline__ void load(const float* row, int g, int D, bool vec) {
        if (vec) {
            const float4* p = reinterpret_cast<const float4*>(row + g * kCols);
#pragma unroll
            for (int i = 0; i < kCols / 4; i++) v[i] = p[i];
        } else {
            float* s = reinterpret_cast<float*>(v);
#pragma unroll
            for (int i = 0; i < kCols; i++) {
                const int d = g * kCols + i;
                s[i] = d < D ? row[d] : 0.f;
            }
        }
    }
    __device__ __forceinline__ void zero() {
#pragma unroll
        for (int i = 0; i < kCols / 4; i++) v[i] = make_float4(0.f, 0.f, 0.f, 0.f);
    }
    __device__ __forceinline__ void get(float* f) const {
        const float* s = reinterpret_cast<const float*>(v);
#pragma unroll
        for (int i = 0; i < kCols; i++) f[i] = s[i];
    }
    static __device__ __forceinline__ void store(float* row, int g, int D, bool vec, const float* f) {
        if (vec) {
#pragma unroll
            for (int i = 0; i < kCols / 4; i++)
                *reinterpret_cast<float4*>(row + g * kCols + 4 * i) = make_float4(f[4 * i], f[4 * i + 1], f[4 * i + 2], f[4 * i + 3]);
        } else {
#pragma unroll
            for (int i = 0; i < kCols; i++)
                if (g * kCols + i < D) row[g * kCols + i] = f[i];
        }
    }
};

}  // namespace cdssm
