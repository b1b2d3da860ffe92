// quantize.cu -- dynamic-range scale finding, quantize, requantize, dequantize.
//
// Replaces compute/tensor/src/cpu/x86/int8/avx512/quantize.cpp:21-416 and dequantize.cpp:18-101.
// All kernels are one or two streaming passes with 128-bit loads, bound by memory; short calls by the host's wait for
// the scale.  The maximum reaches the host through mapped memory (MaxMail) instead of memset, copy and
// synchronisation, and the conversion runs backwards over what the maximum's pass left in L2.  Measured: 98304 fp32 ->
// u8 as part of a 128 x 768 x 768 linear call 41.4 -> 29.8 us; 50.3 M elements, fp32 -> u8, int32 -> u8 and int32 -> fp32
// 250.8 -> 221.8 us (1.31 GB moved).
#include <cstring>

#include "common.cuh"

namespace b200 {
namespace {

constexpr int TPB = 256;

inline uint32_t grid_for(uint64_t n_vec, int sms)
{
    uint64_t blocks = (n_vec + TPB - 1) / TPB;
    const uint64_t cap = (uint64_t)sms * 16;
    if (blocks > cap) {
        blocks = cap;
    }
    return (uint32_t)(blocks ? blocks : 1);
}

// max |x| of binary32 or int32 data (quantize.cpp:36-108) into m.words[0]; with a mail, reported to the host.  Streams
// forwards: what was read last is still in L2 when the conversion pass starts from the end.
constexpr int MAX_TPB = 512;
template <typename T>
__global__ void __launch_bounds__(MAX_TPB) absmax_kernel(const T *__restrict__ x, uint64_t n, const MaxMail m)
{
    struct alignas(16) V4 {
        T a, b, c, d;
    };
    int mx = 0;
    const uint64_t tid = (uint64_t)blockIdx.x * MAX_TPB + threadIdx.x;
    const uint64_t stride = (uint64_t)gridDim.x * MAX_TPB;
    const uint64_t n4 = (reinterpret_cast<uintptr_t>(x) & 15) == 0 ? n / 4 : 0;
    const V4 *x4 = reinterpret_cast<const V4 *>(x);
    auto top = [](const V4 &v) { return max(max(magnitude(v.a), magnitude(v.b)), max(magnitude(v.c), magnitude(v.d))); };
    uint64_t i = tid;
    for (; i + 3 * stride < n4; i += 4 * stride) {  // four independent 128-bit loads in flight per thread
        const V4 a = x4[i], b = x4[i + stride], c = x4[i + 2 * stride], d = x4[i + 3 * stride];
        mx = max(mx, max(max(top(a), top(b)), max(top(c), top(d))));
    }
    for (; i < n4; i += stride) {
        mx = max(mx, top(x4[i]));
    }
    for (uint64_t j = n4 * 4 + tid; j < n; j += stride) {
        mx = max(mx, magnitude(x[j]));
    }
    mx = __reduce_max_sync(0xffffffffu, mx);
    // one atomic per CTA: thousands of warps hitting one address serialise in L2
    __shared__ int warp_max[MAX_TPB / 32];
    if ((threadIdx.x & 31) == 0) {
        warp_max[threadIdx.x >> 5] = mx;
    }
    __syncthreads();
    if (threadIdx.x < 32) {
        mx = __reduce_max_sync(0xffffffffu, threadIdx.x < MAX_TPB / 32 ? warp_max[threadIdx.x] : 0);
        if (threadIdx.x == 0) {
            if (mx != 0) {
                atomicMax(m.words, (unsigned)mx);
            }
            if (m.d_mail != nullptr) {
                report_maximum(m, gridDim.x);
            }
        }
    }
}
// A launch judged by its own status, not by the thread's last error: that may be an earlier call's.
template <typename... P, typename... A>
cudaError_t launch(uint32_t grid, uint32_t block, cudaStream_t st, void (*kernel)(P...), A... args)
{
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(grid);
    cfg.blockDim = dim3(block);
    cfg.stream = st;
    count_launch();
    return cudaLaunchKernelEx(&cfg, kernel, args...);
}
template <typename T>
cudaError_t launch_absmax(DeviceCtx *c, const T *x, uint64_t n, const MaxMail &m, cudaStream_t st)
{
    // a block takes 16 KiB at least; four blocks per SM at most (all resident)
    const uint64_t blocks = (n + 8 * MAX_TPB - 1) / (8 * MAX_TPB), cap = 4 * (uint64_t)c->sm_count;
    return launch((uint32_t)(blocks < cap ? blocks : cap), MAX_TPB, st, absmax_kernel<T>, x, n, m);
}

// the absmax at *scale becomes 127 / absmax (quantize.cpp:63-67), for pipelines that never leave the stream
__global__ void finalize_scale_kernel(float *scale)
{
    const float mx = *scale;
    *scale = (mx == 0.f) ? 1.0f : __fdiv_rn(127.0f, mx);
}

// ---- element functions ------------------------------------------------------------------------
struct F32ToU8 {  // quantize.cpp:135-178: vmulps, vaddps 128, vcvtps2dq{rn}, max 1, min 255
    float s;
    __device__ uint32_t operator()(float x) const
    {
        const int r = cvt_rne_x86(__fadd_rn(__fmul_rn(x, s), 128.0f));
        return (uint32_t)min(255, max(1, r));
    }
};
struct F32ToI8 {  // quantize.cpp:195-233: vmulps, vcvtps2dq, max -127, min 127
    float s;
    __device__ uint32_t operator()(float x) const
    {
        const int r = cvt_rne_x86(__fmul_rn(x, s));
        return (uint32_t)(min(127, max(-127, r)) & 0xFF);
    }
};
struct I32ToU8 {  // quantize.cpp:377-414: vcvtdq2ps, vmulps, vaddps 128, vcvtps2dq, vpmovusdb
    float s;
    __device__ uint32_t operator()(int x) const
    {
        return usat8_x86(cvt_rne_x86(__fadd_rn(__fmul_rn(__int2float_rn(x), s), 128.0f)));
    }
};
struct I32ToI8 {  // quantize.cpp:328-359: vcvtdq2ps, vmulps, vcvtps2dq, vpmovsdb
    float s;
    __device__ uint32_t operator()(int x) const
    {
        return (uint32_t)(ssat8_x86(cvt_rne_x86(__fmul_rn(__int2float_rn(x), s))) & 0xFF);
    }
};

struct F32ToU8Dev {  // same arithmetic, scale read from device memory
    const float *s;
    __device__ uint32_t operator()(float x) const
    {
        const int r = cvt_rne_x86(__fadd_rn(__fmul_rn(x, *s), 128.0f));
        return (uint32_t)min(255, max(1, r));
    }
};

// 32-bit source -> 8-bit destination.  A block converts 4096 elements, four 16-byte loads in flight per thread,
// neighbouring lanes on neighbouring vectors; blocks run from the end of the tensor to its start, so that what the
// maximum's pass read last comes from L2.
constexpr uint32_t TO8_BLOCK = TPB * 16;
template <typename SrcT, typename Op>
__global__ void __launch_bounds__(TPB) to8_kernel(const SrcT *__restrict__ x, uint64_t n, uint8_t *__restrict__ q, Op op)
{
    struct alignas(16) V4 {
        SrcT a, b, c, d;
    };
    const uint64_t first = (uint64_t)(gridDim.x - 1 - blockIdx.x) * TO8_BLOCK;
    const uint64_t last = min(n, first + TO8_BLOCK);
    const bool aligned = (reinterpret_cast<uintptr_t>(x) & 15) == 0 && (reinterpret_cast<uintptr_t>(q) & 3) == 0;
    if (aligned && last - first == TO8_BLOCK) {
        const V4 *xv = reinterpret_cast<const V4 *>(x + first) + threadIdx.x;
        uint32_t *qv = reinterpret_cast<uint32_t *>(q + first) + threadIdx.x;
        V4 v[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            v[j] = xv[j * TPB];
        }
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            qv[j * TPB] = op(v[j].a) | (op(v[j].b) << 8) | (op(v[j].c) << 16) | (op(v[j].d) << 24);
        }
        return;
    }
    for (uint64_t i = first + threadIdx.x; i < last; i += TPB) {
        q[i] = (uint8_t)op(x[i]);
    }
}
template <typename SrcT, typename Op>
EE launch_to8(const SrcT *x, uint64_t n, uint8_t *q, Op op, cudaStream_t st)
{
    const uint64_t blocks = (n + TO8_BLOCK - 1) / TO8_BLOCK;
    if (blocks > 0x7FFFFFFFull) {
        return NOT_SUPPORTED;
    }
    B200_CUDA(launch((uint32_t)blocks, TPB, st, to8_kernel<SrcT, Op>, x, n, q, op));
    return SUCCESS;
}

// quantize.cpp:271-313: byte-wise + 0x80
__global__ void u8_to_i8_kernel(const uint8_t *__restrict__ x, uint64_t n, uint8_t *__restrict__ q)
{
    const uint64_t tid = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
    const bool aligned = ((reinterpret_cast<uintptr_t>(x) | reinterpret_cast<uintptr_t>(q)) & 15) == 0;
    const uint64_t n16 = aligned ? n / 16 : 0;
    for (uint64_t i = tid; i < n16; i += stride) {
        uint4 v = reinterpret_cast<const uint4 *>(x)[i];
        v.x ^= 0x80808080u;
        v.y ^= 0x80808080u;
        v.z ^= 0x80808080u;
        v.w ^= 0x80808080u;
        reinterpret_cast<uint4 *>(q)[i] = v;
    }
    for (uint64_t i = n16 * 16 + tid; i < n; i += stride) {
        q[i] = x[i] ^ 0x80u;
    }
}

// dequantize.cpp:18-52: (float)q * (1/scale)
__global__ void dequant_i32_kernel(const int32_t *__restrict__ q, uint64_t n, float factor, float *__restrict__ out)
{
    const uint64_t tid = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
    const bool aligned = ((reinterpret_cast<uintptr_t>(q) | reinterpret_cast<uintptr_t>(out)) & 15) == 0;
    const uint64_t n4 = aligned ? n / 4 : 0;
    const int4 *q4 = reinterpret_cast<const int4 *>(q);
    float4 *o4 = reinterpret_cast<float4 *>(out);
    auto one = [factor](int4 v) {
        return make_float4(acc_to_f32(v.x, factor), acc_to_f32(v.y, factor), acc_to_f32(v.z, factor), acc_to_f32(v.w, factor));
    };
    uint64_t i = tid;
    for (; i + 3 * stride < n4; i += 4 * stride) {
        const int4 a = q4[i], b = q4[i + stride], c = q4[i + 2 * stride], d = q4[i + 3 * stride];
        o4[i] = one(a);
        o4[i + stride] = one(b);
        o4[i + 2 * stride] = one(c);
        o4[i + 3 * stride] = one(d);
    }
    for (; i < n4; i += stride) {
        o4[i] = one(q4[i]);
    }
    for (uint64_t i = n4 * 4 + tid; i < n; i += stride) {
        out[i] = acc_to_f32(q[i], factor);
    }
}

// dequantize.cpp:54-101: (float)((int)q - 128) * (1.0f/scale)
__global__ void dequant_u8_kernel(const uint8_t *__restrict__ q, uint64_t n, float factor, float *__restrict__ out)
{
    const uint64_t tid = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
    const bool aligned = ((reinterpret_cast<uintptr_t>(q) | reinterpret_cast<uintptr_t>(out)) & 15) == 0;
    const uint64_t n16 = aligned ? n / 16 : 0;
    for (uint64_t i = tid; i < n16; i += stride) {
        const uint4 v = reinterpret_cast<const uint4 *>(q)[i];
        const uint32_t w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            reinterpret_cast<float4 *>(out)[i * 4 + j] =
                make_float4(acc_to_f32((int)(w[j] & 0xFF) - 128, factor), acc_to_f32((int)((w[j] >> 8) & 0xFF) - 128, factor),
                    acc_to_f32((int)((w[j] >> 16) & 0xFF) - 128, factor), acc_to_f32((int)(w[j] >> 24) - 128, factor));
        }
    }
    for (uint64_t i = n16 * 16 + tid; i < n; i += stride) {
        out[i] = acc_to_f32((int)q[i] - 128, factor);
    }
}

// quantize.cpp:236-269: round() = half away from zero on the fp32 product
__global__ void bias_offsetc_kernel(const float *bias, const int32_t *offsetC, uint32_t n, float scale, int32_t *out)
{
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) {
        int b = 0;
        if (bias != nullptr) {
            b = (int)roundf(__fmul_rn(bias[i], scale));
        }
        out[i] = b + (offsetC ? offsetC[i] : 0);
    }
}
__global__ void bias_i32_offsetc_kernel(const int32_t *bias, const int32_t *offsetC, uint32_t n, int32_t *out)
{
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) {
        out[i] = bias[i] + (offsetC ? offsetC[i] : 0);
    }
}

uint64_t desc_elems(const TensorDesc *d)
{
    if (d->nDims == 0) {
        return 0;
    }
    uint64_t n = 1;
    for (uint32_t i = 0; i < d->nDims && i < 20; ++i) {
        n *= d->dims[i];
    }
    return n;
}

// absmax of device data, result to host
template <typename T>
EE absmax_host(const T *d_x, uint64_t n, int *mx)
{
    DeviceCtx *c = ctx();
    cudaStream_t st = tls().stream;
    *mx = 0;
    if (capturing(st)) {
        return UNKNOWN;   // the scale has to reach the host
    }
    if (n == 0) {
        return SUCCESS;
    }
    MaxLease lease(c);
    if (!lease.ok()) {
        return UNKNOWN;
    }
    B200_CUDA(launch_absmax(c, d_x, n, lease.mail(), st));
    lease.launched(st);
    return lease.wait(mx);
}
EE absmax_f32_host(const float *d_x, uint64_t n, float *mx)
{
    int bits = 0;
    B200_EE(absmax_host(d_x, n, &bits));
    std::memcpy(mx, &bits, 4);
    return SUCCESS;
}

// factor[n] = num / (sA * sB[n]): fp32 multiply, fp32 divide -- the order in which Bolt forms the
// factor of a layer (fully_connected.cpp:396,409; mmm_avx512_vnni.cpp:1805)
__global__ void col_factor_kernel(float num, float sA, const float *d_sA, float sB, const float *col_scale, uint32_t N,
    float *out)
{
    const uint32_t n = blockIdx.x * blockDim.x + threadIdx.x;
    if (n < N) {
        const float sa = d_sA ? *d_sA : sA;
        const float sb = col_scale ? col_scale[n] : sB;
        out[n] = __fdiv_rn(num, __fmul_rn(sa, sb));
    }
}

}  // namespace

// int32 (device) whose maximum is known -> u8 (device) with the reference's scale protocol; the convolution's u8
// output (convolution_direct.cpp:2798-2806).  scale2 is a host array of two floats.
EE quantize_i32_u8_device(const int32_t *d_src, uint64_t n, int mx, uint8_t *d_q, F32 *scale2)
{
    float raw = 0;
    if (scale2[0] < 0 && scale2[1] > 0) {
        raw = (mx == 0) ? 1.0f : 127.0f / (float)mx;
        scale2[0] = scale2[1] * raw;
    } else if (scale2[0] > 0 && scale2[1] > 0) {
        raw = scale2[0] / scale2[1];
    }
    if (n == 0) {
        return SUCCESS;
    }
    return launch_to8<int32_t, I32ToU8>(d_src, n, d_q, I32ToU8{raw}, tls().stream);
}

// F32 -> U8_Q on device pointers, scale handling of quantize_x86 (cpu/x86/quantize.cpp:33-41,
// avx512/quantize.cpp:129-133): the dynamic scale 127 / max|x| unless mode != 0 and a positive scale is given
EE quantize_f32_u8_device(const float *d_src, uint64_t n, uint8_t *d_q, F32 *scale, int mode)
{
    DeviceCtx *c = ctx();
    if (c == nullptr) {
        return UNKNOWN;
    }
    if (!mode || *scale <= 0) {
        float mx = 0;
        B200_EE(absmax_f32_host(d_src, n, &mx));
        const float s = (mx == 0) ? 1.0f : 127 / mx;
        *scale = (*scale > s) ? *scale : s;
    }
    if (n == 0) {
        return SUCCESS;
    }
    return launch_to8<float, F32ToU8>(d_src, n, d_q, F32ToU8{*scale}, tls().stream);
}

}  // namespace b200

using namespace b200;

extern "C" {

EE quantize_cuda_b200(const TensorDesc *dDesc, const void *data, TensorDesc *qDesc, void *qData, F32 *scale,
    int mode)
{
    if (dDesc == nullptr || qDesc == nullptr) {
        return NULL_POINTER;
    }
    DeviceCtx *c = ctx();
    if (c == nullptr) {
        return UNKNOWN;
    }
    const uint64_t n = desc_elems(dDesc);
    const DataType sdt = dDesc->dt, qdt = qDesc->dt;
    const bool f32 = (sdt == DT_F32 || sdt == DT_F32_8Q);
    const bool known = (f32 && (qdt == DT_I8 || qdt == DT_U8_Q)) || (sdt == DT_U8_Q && qdt == DT_I8) ||
        (sdt == DT_I32 && (qdt == DT_I8 || qdt == DT_U8_Q));
    if (!known) {
        return NOT_SUPPORTED;
    }
    if (sdt != DT_U8_Q && scale == nullptr) {
        return NOT_MATCH;  // quantize.cpp:123-125
    }
    if (n == 0) {
        return SUCCESS;
    }
    if (data == nullptr || qData == nullptr) {
        return NULL_POINTER;
    }
    cudaStream_t st = tls().stream;
    Stage sg;
    const size_t src_bytes = n * (sdt == DT_U8_Q ? 1 : 4);
    const void *d_src = sg.in(data, src_bytes);
    uint8_t *d_q = reinterpret_cast<uint8_t *>(sg.out(qData, n));
    if (d_src == nullptr || d_q == nullptr) {
        return ALLOC_FAILED;
    }
    const uint32_t grid = grid_for((n + 15) / 16, c->sm_count);
    if (f32) {
        if (!mode || *scale <= 0) {  // quantize.cpp:129-133
            float mx = 0;
            B200_EE(absmax_f32_host(reinterpret_cast<const float *>(d_src), n, &mx));
            const float s = (mx == 0) ? 1.0f : 127 / mx;
            *scale = (*scale > s) ? *scale : s;
        }
        if (qdt == DT_U8_Q) {
            B200_EE((launch_to8<float, F32ToU8>(reinterpret_cast<const float *>(d_src), n, d_q, F32ToU8{*scale}, st)));
        } else {
            B200_EE((launch_to8<float, F32ToI8>(reinterpret_cast<const float *>(d_src), n, d_q, F32ToI8{*scale}, st)));
        }
    } else if (sdt == DT_U8_Q) {
        u8_to_i8_kernel<<<grid, TPB, 0, st>>>(reinterpret_cast<const uint8_t *>(d_src), n, d_q);
        count_launch();
        B200_CUDA(cudaGetLastError());
    } else {
        float raw = 0;  // quantize.cpp:320-326 / 369-375
        if (scale[0] < 0 && scale[1] > 0) {
            int mx = 0;
            B200_EE(absmax_host(reinterpret_cast<const int32_t *>(d_src), n, &mx));
            raw = (mx == 0) ? 1.0f : 127.0f / (float)mx;
            scale[0] = scale[1] * raw;
        } else if (scale[0] > 0 && scale[1] > 0) {
            raw = scale[0] / scale[1];
        }
        if (qdt == DT_U8_Q) {
            B200_EE((launch_to8<int32_t, I32ToU8>(reinterpret_cast<const int32_t *>(d_src), n, d_q, I32ToU8{raw}, st)));
        } else {
            B200_EE((launch_to8<int32_t, I32ToI8>(reinterpret_cast<const int32_t *>(d_src), n, d_q, I32ToI8{raw}, st)));
        }
    }
    return sg.finish();
}

EE bolt_b200_absmax_scale_f32(const F32 *data, uint64_t n, F32 *d_scale)
{
    DeviceCtx *c = ctx();
    if (c == nullptr) {
        return UNKNOWN;
    }
    if (data == nullptr || d_scale == nullptr) {
        return NULL_POINTER;
    }
    cudaStream_t st = tls().stream;
    // the maximum is found in the caller's own word: a shared one would mix calls on several streams
    unsigned *bits = reinterpret_cast<unsigned *>(d_scale);
    B200_CUDA(cudaMemsetAsync(bits, 0, 4, st));
    if (n > 0) {
        B200_CUDA(launch_absmax(c, data, n, MaxMail{bits, nullptr, nullptr, 0}, st));
    }
    B200_CUDA(launch(1, 1, st, finalize_scale_kernel, d_scale));
    return SUCCESS;
}

EE bolt_b200_col_factor(F32 num, F32 sA, const F32 *d_sA, F32 sB, const F32 *col_scale, U32 N, F32 *factor)
{
    if (ctx() == nullptr) {
        return UNKNOWN;
    }
    if (factor == nullptr) {
        return NULL_POINTER;
    }
    if (N == 0) {
        return SUCCESS;
    }
    col_factor_kernel<<<(N + 255) / 256, 256, 0, tls().stream>>>(num, sA, d_sA, sB, col_scale, N, factor);
    count_launch();
    B200_CUDA(cudaGetLastError());
    return SUCCESS;
}

EE bolt_b200_quantize_f32_u8_dev(const F32 *data, uint64_t n, UINT8 *q, const F32 *d_scale)
{
    DeviceCtx *c = ctx();
    if (c == nullptr) {
        return UNKNOWN;
    }
    if (data == nullptr || q == nullptr || d_scale == nullptr) {
        return NULL_POINTER;
    }
    if (n == 0) {
        return SUCCESS;
    }
    return launch_to8<float, F32ToU8Dev>(data, n, q, F32ToU8Dev{d_scale}, tls().stream);
}

EE quantize_bias_offsetC_cuda_b200(const void *bias, const TensorDesc *biasDesc, DataType qType,
    const void *filter, const TensorDesc *filterDesc, const F32 *scale, void *offsetCBias)
{
    if (biasDesc == nullptr || filterDesc == nullptr) {
        return NULL_POINTER;
    }
    if (qType != DT_I32) {
        return NOT_SUPPORTED;
    }
    if (ctx() == nullptr) {
        return UNKNOWN;
    }
    if (bias == nullptr && filter == nullptr) {
        return SUCCESS;
    }
    // "native" formats carry no packed offset (quantize.cpp:244-259)
    const DataFormat fdf = filterDesc->df;
    const bool native = fdf == DF_NCHW || fdf == 24 /*DF_NHWC*/ || fdf == 15 /*DF_MTK*/ || fdf == DF_NORMAL ||
        fdf == DF_TRANSPOSE;
    uint32_t n = (uint32_t)desc_elems(biasDesc);
    const bool no_bias = (bias == nullptr) || n == 0;
    if (no_bias) {
        n = filterDesc->dims[0] > filterDesc->dims[1] ? filterDesc->dims[0] : filterDesc->dims[1];
    } else if (biasDesc->dt != DT_F32 && biasDesc->dt != DT_I32) {
        return NOT_SUPPORTED;
    }
    if (n == 0) {
        return SUCCESS;
    }
    if (offsetCBias == nullptr) {
        return NULL_POINTER;
    }
    cudaStream_t st = tls().stream;
    Stage sg;
    const bool i32_bias = !no_bias && biasDesc->dt == DT_I32;
    // fp32 bias (or none): the packed offset is read only from non-native filter formats;
    // int32 bias: `filter` is an offset array whenever it is given (quantize.cpp:100-111)
    const bool use_off = (filter != nullptr) && (i32_bias || !native);
    const int32_t *d_off = use_off ? reinterpret_cast<const int32_t *>(sg.in(filter, (size_t)n * 4)) : nullptr;
    const void *d_bias = no_bias ? nullptr : sg.in(bias, (size_t)n * 4);
    int32_t *d_out = reinterpret_cast<int32_t *>(sg.out(offsetCBias, (size_t)n * 4));
    if (d_out == nullptr || (use_off && d_off == nullptr) || (!no_bias && d_bias == nullptr)) {
        return ALLOC_FAILED;
    }
    if (i32_bias) {
        bias_i32_offsetc_kernel<<<(n + 255) / 256, 256, 0, st>>>(reinterpret_cast<const int32_t *>(d_bias), d_off, n,
            d_out);
    } else {
        if (!no_bias && scale == nullptr) {
            return NULL_POINTER;
        }
        bias_offsetc_kernel<<<(n + 255) / 256, 256, 0, st>>>(reinterpret_cast<const float *>(d_bias), d_off, n,
            no_bias ? 0.f : scale[0], d_out);
    }
    count_launch();
    B200_CUDA(cudaGetLastError());
    return sg.finish();
}

EE dequantize_cuda_b200(const TensorDesc *qDesc, const void *qData, const F32 *scale, const TensorDesc *bDesc,
    const void *bData, const TensorDesc *dDesc, void *dData)
{
    (void)bDesc;
    (void)bData;  // ignored, as on x86 (cpu/x86/dequantize.cpp:19-48)
    if (qDesc == nullptr || dDesc == nullptr || scale == nullptr) {
        return NULL_POINTER;
    }
    if (dDesc->dt != DT_F32 || (qDesc->dt != DT_I32 && qDesc->dt != DT_U8_Q)) {
        return NOT_SUPPORTED;
    }
    DeviceCtx *c = ctx();
    if (c == nullptr) {
        return UNKNOWN;
    }
    const uint64_t n = desc_elems(dDesc);
    if (n == 0) {
        return SUCCESS;
    }
    if (qData == nullptr || dData == nullptr) {
        return NULL_POINTER;
    }
    cudaStream_t st = tls().stream;
    Stage sg;
    const bool i32 = qDesc->dt == DT_I32;
    const void *d_q = sg.in(qData, n * (i32 ? 4 : 1));
    float *d_out = reinterpret_cast<float *>(sg.out(dData, n * 4));
    if (d_q == nullptr || d_out == nullptr) {
        return ALLOC_FAILED;
    }
    const float factor = i32 ? (1 / *scale) : (1.0f / scale[0]);
    if (i32) {
        dequant_i32_kernel<<<grid_for((n + 3) / 4, c->sm_count), TPB, 0, st>>>(
            reinterpret_cast<const int32_t *>(d_q), n, factor, d_out);
    } else {
        dequant_u8_kernel<<<grid_for((n + 15) / 16, c->sm_count), TPB, 0, st>>>(
            reinterpret_cast<const uint8_t *>(d_q), n, factor, d_out);
    }
    count_launch();
    B200_CUDA(cudaGetLastError());
    return sg.finish();
}

}  // extern "C"
