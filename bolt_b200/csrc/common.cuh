// common.cuh -- internal declarations shared by the .cu files of libbolt_b200.so.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#include <atomic>
#include <condition_variable>
#include <map>
#include <mutex>
#include <vector>

#include "bolt_b200.h"

namespace b200 {

#define B200_ALIGN(x, a) ((((x) + (a)-1) / (a)) * (a))

// ---- device-side exact arithmetic ----------------------------------------------------------
// The reference computes every float step as a separate IEEE binary32 instruction (vcvtdq2ps,
// vmulps, vaddps, vcvtps2dq); the helpers below use the _rn intrinsics so that nvcc cannot
// contract a multiply and an add into one fused operation.

// vcvtps2dq: round to nearest even; NaN and |f| >= 2^31 give 0x80000000.
__device__ __forceinline__ int cvt_rne_x86(float f)
{
    return (f >= -2147483648.0f && f < 2147483648.0f) ? __float2int_rn(f) : (int)0x80000000;
}
// vpmovusdb: the dword is read as unsigned, then clamped to 255.
__device__ __forceinline__ uint32_t usat8_x86(int v)
{
    return min((uint32_t)v, 255u);
}
// vpmovsdb
__device__ __forceinline__ int ssat8_x86(int v)
{
    return max(-128, min(127, v));
}
// GEMM / GEMV / conv u8 epilogue: vcvtdq2ps, vmulps, vcvtps2dq, vpaddd 128, vpmovusdb.
__device__ __forceinline__ uint32_t acc_to_u8(int acc, float factor)
{
    float f = __fmul_rn(__int2float_rn(acc), factor);
    // __float2int_rn saturates where vcvtps2dq returns 0x80000000; after +128 both land above
    // 255 as unsigned, except NaN (0 here), which is mapped by hand.
    int r = (f != f) ? (int)0x80000000 : __float2int_rn(f);
    return usat8_x86((int)((uint32_t)r + 128u));
}
__device__ __forceinline__ float acc_to_f32(int acc, float factor)
{
    return __fmul_rn(__int2float_rn(acc), factor);
}

// 32 bytes per lane (32-byte aligned): lanes on different rows then write whole sectors.  4096 x 768 x 3072 -> fp32 with
// its quantization 89.2 -> 62.0 us per call together with the mapped scale (which alone took the u8 result from 54.9 to
// 36.4); 2048 x 4096 x 16384 -> fp32 147.5 -> 116.8 us.
__device__ __forceinline__ void store_v8(void *p, const uint32_t (&v)[8])
{
    asm volatile("st.global.v8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"l"(p), "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]),
                 "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7])
                 : "memory");
}
__device__ __forceinline__ void load_v8(const void *p, uint32_t (&v)[8])
{
    asm volatile("ld.global.v8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
                 : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7])
                 : "l"(p)
                 : "memory");
}
// the same in 16-byte pieces where only those are aligned
__device__ __forceinline__ void store_8(void *p, const uint32_t (&v)[8], bool aligned32)
{
    if (aligned32) {
        store_v8(p, v);
    } else {
        reinterpret_cast<uint4 *>(p)[0] = make_uint4(v[0], v[1], v[2], v[3]);
        reinterpret_cast<uint4 *>(p)[1] = make_uint4(v[4], v[5], v[6], v[7]);
    }
}
__device__ __forceinline__ void load_8(const void *p, uint32_t (&v)[8], bool aligned32)
{
    if (aligned32) {
        load_v8(p, v);
    } else {
        const uint4 a = reinterpret_cast<const uint4 *>(p)[0], b = reinterpret_cast<const uint4 *>(p)[1];
        v[0] = a.x;
        v[1] = a.y;
        v[2] = a.z;
        v[3] = a.w;
        v[4] = b.x;
        v[5] = b.y;
        v[6] = b.z;
        v[7] = b.w;
    }
}

// ---- per-device state ------------------------------------------------------------------------
struct WeightTwin {
    void *dev;
    size_t bytes;
};

// kernel families whose dynamic shared-memory limit has to be raised above 48 KiB; the attribute
// belongs to the device that is current when it is set, so it is remembered per device context
enum KernelFamily { KF_GEMM = 0, KF_CONV, KF_CONV_HALF, KF_GEMV, KF_GEMV_ROW, KF_BNN, KF_GATHER, KF_MATMUL, KF_MATMUL_ROW, KF_PROBE, KF_COUNT };

// A maximum that a kernel finds and the host waits for.  Device words {running maximum, finished blocks}, both zero
// between uses (the last block rewinds them); it then stores sequence number and maximum, as one 8-byte word, into
// mapped host memory, where the host polls: no memset, no copy, no stream synchronisation, and later work of the
// stream need not be waited for.
struct MaxMail {
    unsigned *words;
    unsigned long long *d_mail;
    volatile unsigned long long *h_mail;
    uint32_t seq;
};
constexpr int MAX_MAILS = 64;   // as many calls at a time; more wait for one

struct DeviceCtx {
    int device = 0;
    bool smem_raised[KF_COUNT] = {};
    std::mutex attr_mu;
    int max_pairs = -1;  // co-resident 2-CTA clusters of the tensor-core GEMM (-1: not queried yet)
    int sm_count = 148;
    int *d_status = nullptr;      // device-side error word
    void *d_scatter_maps = nullptr;  // 8 tensor maps of a scatter GEMM (allocated on first use)
    unsigned *d_scratch_u = nullptr;   // the words of the MaxMails
    std::mutex mu;       // guards the staging workspace (one staged call at a time)
    std::mutex twin_mu;  // guards twins
    std::mutex mail_mu;     // guards mail_free and mails
    std::condition_variable mail_cv;
    std::vector<MaxMail *> mail_free;
    int mails = 0;          // in the pool or in use
    std::map<const void *, WeightTwin> twins;  // host packed weight -> device copy
    // growable staging workspace for host-pointer calls
    char *ws = nullptr;
    size_t ws_bytes = 0;
    size_t ws_used = 0;
};

struct ThreadState {
    int device = -1;  // -1: not chosen through bolt_b200_set_device -- follow the thread's current CUDA device
    cudaStream_t stream = nullptr;
    bool device_only = false;
    int last_gemm_tc = 0;
};

DeviceCtx *ctx();          // context of the calling thread's device (created on first use)
ThreadState &tls();
extern std::atomic<uint64_t> g_launches;
inline void count_launch(int n = 1)
{
    g_launches.fetch_add((uint64_t)n, std::memory_order_relaxed);
}

// One MaxMail for the duration of a call (found on a stream that is not being captured: the host has to wait):
// ok(), launch a kernel with mail(), launched() if that succeeded, wait().
class MaxLease {
public:
    explicit MaxLease(DeviceCtx *c);
    ~MaxLease();
    MaxLease(const MaxLease &) = delete;
    MaxLease &operator=(const MaxLease &) = delete;
    bool ok() const
    {
        return m_ != nullptr;
    }
    const MaxMail &mail() const
    {
        return *m_;
    }
    // from here on the mail belongs to a kernel on `st`, until that is seen to have reported
    void launched(cudaStream_t st)
    {
        in_flight_ = true;
        st_ = st;
    }
    // the maximum that the kernel reports
    EE wait(int *maximum);

private:
    DeviceCtx *c_;
    MaxMail *m_ = nullptr;
    cudaStream_t st_ = nullptr;
    bool in_flight_ = false;
};
bool capturing(cudaStream_t st);

#ifdef __CUDACC__
// by one thread of a block, after a block barrier behind the block's last atomicMax on words[0]
__device__ __forceinline__ void report_maximum(const MaxMail &m, unsigned blocks)
{
    __threadfence();
    if (atomicInc(m.words + 1, blocks - 1) == blocks - 1) {   // wraps to 0
        __threadfence();
        const unsigned mx = atomicExch(m.words, 0u);
        *reinterpret_cast<volatile unsigned long long *>(m.d_mail) = ((unsigned long long)m.seq << 32) | mx;
        __threadfence_system();
    }
}
// |x| as a non-negative integer that orders like it: the bits of a binary32, or vpabsd of an int32 (|INT_MIN| stays
// negative and never wins)
__device__ __forceinline__ int magnitude(float x)
{
    return (int)(__float_as_uint(x) & 0x7FFFFFFFu);
}
__device__ __forceinline__ int magnitude(int x)
{
    return (int)(x < 0 ? 0u - (unsigned)x : (unsigned)x);
}
#endif

#ifdef __CUDACC__
// Programmatic stream serialization (a kernel's set-up runs beside the end of the kernel in front of it): on unless
// BOLT_B200_NO_PDL is set in the environment, or the runtime has refused it where it took the plain launch.
bool programmatic_launches();
void refuse_programmatic_launches();
template <typename... P, typename... A>
cudaError_t launch_programmatic(const cudaLaunchConfig_t &plain, void (*kernel)(P...), const A &...args)
{
    if (!programmatic_launches()) {
        return cudaLaunchKernelEx(&plain, kernel, args...);
    }
    cudaLaunchAttribute at[2];
    unsigned n = 0;
    for (; n < plain.numAttrs && n < 1; ++n) {
        at[n] = plain.attrs[n];
    }
    at[n].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[n].val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t cfg = plain;
    cfg.attrs = at;
    cfg.numAttrs = n + 1;
    cudaError_t e = cudaLaunchKernelEx(&cfg, kernel, args...);
    if (e != cudaSuccess && !capturing(plain.stream)) {
        cudaGetLastError();
        e = cudaLaunchKernelEx(&plain, kernel, args...);
        if (e == cudaSuccess) {
            refuse_programmatic_launches();
        }
    }
    return e;
}
#endif

// cudaFuncAttributeMaxDynamicSharedMemorySize for every kernel of a family, once per device
// (the calling thread's device must be current, which ctx() guarantees)
EE raise_smem_limit(DeviceCtx *c, KernelFamily f, const void *const *kernels, int n, size_t bytes);

// true if p is memory the GPU can dereference (device or managed)
bool is_device_ptr(const void *p);
// true if p is plain device memory of a GPU other than the one this thread's calls run on
bool on_other_device(const void *p);

// Staging helper for one call: maps caller pointers to device pointers.  Host inputs are
// copied into the workspace; host outputs get a workspace buffer that finish() copies back.
class Stage {
public:
    Stage();
    ~Stage();
    // input: returns a device pointer holding `bytes` bytes of p
    const void *in(const void *p, size_t bytes);
    // output (optionally preloaded with the host content when `also_in`)
    void *out(void *p, size_t bytes, bool also_in = false);
    // device scratch that lives until finish()
    void *scratch(size_t bytes);
    // copy outputs back; synchronises the stream if anything was staged
    EE finish();
    bool any_host() const
    {
        return any_host_;
    }

private:
    struct Out {
        void *host;
        void *dev;
        size_t bytes;
    };
    std::vector<Out> outs_;
    std::vector<void *> big_;  // direct allocations that did not fit the workspace
    bool any_host_ = false;
    bool locked_ = false;
    void *alloc(size_t bytes);
};

EE cuda_ee(cudaError_t e);
#define B200_CUDA(call)                    \
    do {                                   \
        cudaError_t _e = (call);           \
        if (_e != cudaSuccess) {           \
            return ::b200::cuda_ee(_e);    \
        }                                  \
    } while (0)
#define B200_EE(call)          \
    do {                       \
        EE _s = (call);        \
        if (_s != SUCCESS) {   \
            return _s;         \
        }                      \
    } while (0)

// cuTensorMapEncodeTiled (found through the runtime's driver entry point) for byte tensors of
// rank <= 5; zero fill out of range.  `map` points at a CUtensorMap.
bool tensor_map_encoder_available();
bool encode_tiled_u8(void *map, uint32_t rank, const void *base, const uint64_t *dims, const uint64_t *strides,
    const uint32_t *box, const uint32_t *elem_strides, int swizzle_bytes /* 0, 32, 64 or 128 */);

// ---- kernel launchers (device pointers only) ----------------------------------------------
struct GemmEpilogue {
    int out_kind;              // 0 int32, 1 fp32, 2 u8
    int accumulate;            // add incoming int32 bits of C (kinds 0, 1)
    const int32_t *offsetC;    // [N] or null
    float factor;              // used when per_channel == 0
    int per_channel;           // 1: factor = num / (sA[m] * sB[n])
    float num, sA, sB;
    const float *sA_dev;       // device scalar overriding sA, or null
    const float *row_scale;    // [M] or null
    const float *col_scale;    // [N] or null
    const float *col_factor;   // [N] or null: ready-made per-column factors (then nothing is divided in the kernel)
    const void *prefetch;      // device memory a later call will read (the next layer's weight), or null:
    size_t prefetch_bytes;     // brought into L2 while this GEMM runs
    // u8 output stored into scatter_n matrices [M][scatter_ld] (this GPU's and its peers') at column scatter_col0
    void *scatter_dst[8];
    uint32_t scatter_n, scatter_ld, scatter_col0;
};

// B: ALIGN(N,16) rows, pitch Kp = ALIGN(K,8) bytes, K contiguous, zero padded.
EE launch_gemm_tcgen05(uint32_t M, uint32_t N, uint32_t K, const uint8_t *A, const int8_t *B,
    uint32_t Kp, void *C, const GemmEpilogue &ep, cudaStream_t st);
bool gemm_tcgen05_eligible(uint32_t M, uint32_t N, uint32_t K, const void *A, const void *B,
    uint32_t Kp, bool a_transposed);
bool gemm_skinny_preferred(uint32_t M, uint32_t N, uint32_t K, int sms);
EE launch_gemm_skinny(uint32_t M, uint32_t N, uint32_t K, const uint8_t *A, const int8_t *B, uint32_t Kp, void *C,
    const GemmEpilogue &ep, bool preload, cudaStream_t st);
EE launch_gemm_gather(uint32_t M, uint32_t N, uint32_t K, const uint8_t *A, bool a_transposed,
    const int8_t *B, uint32_t Kp, void *C, const GemmEpilogue &ep, cudaStream_t st);

// The products of one matmul call, C[i] = A[ia(i)] * B[ib(i)]
struct MatmulOperand {
    const void *p;
    uint64_t elems;        // of all its products
    int f32;               // binary32, quantized by the call (else u8 A / s8 B; M = 1: s8 A / u8 B)
    int transposed;        // A: stored [K][M]; B: stored [N][K]
    float scale;           // f32: lower bound of the dynamic scale, else the scale
    uint32_t dims[4];      // batch extents
    int direct;            // as many products as C has
    unsigned *slots;       // f32: scratch for the partial maxima
    uint64_t max_slots;
};
struct MatmulBatch {
    uint32_t M, N, K;
    uint64_t batches;
    uint32_t c_dims[4];
    MatmulOperand a, b;
    void *C;
    int out_kind;          // 1 fp32, 2 u8 with the scale c_scale
    int accumulate;
    float c_scale;
};
EE launch_matmul_batch(const MatmulBatch &mb, cudaStream_t st);
uint32_t gather_block_n(uint64_t tiles_m, uint32_t N, int sms);   // column block of its tiles
EE launch_pack_rhs(const int8_t *src, bool src_is_nk, uint32_t N, uint32_t K, int8_t *dst,
    uint32_t Kp, uint32_t Np, int32_t *offsetC, cudaStream_t st);
EE launch_gemv_row(uint32_t N, uint32_t K, const uint8_t *Mx, bool transposed, const int8_t *v, void *y, int out_kind,
    float factor, cudaStream_t st);
EE launch_gemv(uint32_t N, uint32_t K, const int8_t *W, uint32_t Kp, const uint8_t *x,
    const int32_t *offsetC, void *y, int out_kind, float factor, cudaStream_t st);

}  // namespace b200
