// epilogue.cuh -- results of a u8 x s8 product from its accumulators (offset included), for the kernels that store
// rows with plain vector stores.
#pragma once
#include "common.cuh"

namespace b200 {

// conversion factor of column n (without per-row scales), in the order of the other kernels
__device__ __forceinline__ float column_factor(const GemmEpilogue &ep, uint32_t n)
{
    if (ep.col_factor != nullptr) {
        return ep.col_factor[n];
    }
    if (!ep.per_channel) {
        return ep.factor;
    }
    const float sb = ep.col_scale ? ep.col_scale[n] : ep.sB;
    if (ep.row_scale != nullptr) {
        return sb;   // divided per element
    }
    return __fdiv_rn(ep.num, __fmul_rn(ep.sA_dev ? *ep.sA_dev : ep.sA, sb));
}

// what C holds in V consecutive columns of row m
template <int V>
__device__ __forceinline__ void read_c(uint32_t N, const void *C, uint32_t m, uint32_t n, int (&acc)[V])
{
    const int32_t *cin = reinterpret_cast<const int32_t *>(C) + (size_t)m * N + n;
    if (V == 4) {
        const int4 v = *reinterpret_cast<const int4 *>(cin);
        acc[0] = v.x;
        acc[1 % V] = v.y;
        acc[2 % V] = v.z;
        acc[3 % V] = v.w;
    } else {
        acc[0] = cin[0];
    }
}
// V consecutive results of row m, columns n .. n+V-1
template <int V>
__device__ __forceinline__ void finish(const GemmEpilogue &ep, uint32_t N, void *C, uint32_t m, uint32_t n, const int (&acc)[V], const float (&cf)[V])
{
    const size_t o = (size_t)m * N + n;
    if (ep.out_kind == 0) {
        int32_t *out = reinterpret_cast<int32_t *>(C) + o;
        if (V == 4) {
            *reinterpret_cast<int4 *>(out) = make_int4(acc[0], acc[1 % V], acc[2 % V], acc[3 % V]);
        } else {
            out[0] = acc[0];
        }
        return;
    }
    float f[V];
#pragma unroll
    for (int j = 0; j < V; ++j) {
        f[j] = cf[j];
        if (ep.per_channel && ep.row_scale != nullptr) {
            f[j] = __fdiv_rn(ep.num, __fmul_rn(ep.row_scale[m], cf[j]));
        }
    }
    if (ep.out_kind == 1) {
        float *out = reinterpret_cast<float *>(C) + o;
        if (V == 4) {
            *reinterpret_cast<float4 *>(out) = make_float4(acc_to_f32(acc[0], f[0]), acc_to_f32(acc[1 % V], f[1 % V]),
                acc_to_f32(acc[2 % V], f[2 % V]), acc_to_f32(acc[3 % V], f[3 % V]));
        } else {
            out[0] = acc_to_f32(acc[0], f[0]);
        }
    } else {
        uint8_t *out = reinterpret_cast<uint8_t *>(C) + o;
        if (V == 4) {
            *reinterpret_cast<uint32_t *>(out) = acc_to_u8(acc[0], f[0]) | (acc_to_u8(acc[1 % V], f[1 % V]) << 8) |
                (acc_to_u8(acc[2 % V], f[2 % V]) << 16) | (acc_to_u8(acc[3 % V], f[3 % V]) << 24);
        } else {
            out[0] = (uint8_t)acc_to_u8(acc[0], f[0]);
        }
    }
}

}  // namespace b200
