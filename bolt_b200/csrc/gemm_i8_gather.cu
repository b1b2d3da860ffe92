// gemm_i8_gather.cu -- u8 x s8 products on the sm_100a tensor cores whose operands TMA cannot fetch.
//
// The TMA kernel (gemm_i8_tcgen05.cu) needs 16-byte aligned rows and an untransposed A.  Here the CTA's threads
// bring the operands into the swizzled shared-memory layout of tcgen05.mma themselves, so any K, any alignment and
// a transposed A run on the tensor cores.  Shapes: frames x features against classes (333 x 515 x 1001), the
// 1..33-sized products of Bolt's cover test (compute/blas_enhance/tests/test_mmm.cpp:165-171).
//
// One tile is 128 rows x block_n columns; a CTA is 256 threads, all of which load, convert and store; one of them
// issues the MMAs.  Two 128-byte K blocks are in flight (block k+1 is fetched and stored while the MMAs of block k
// run) and two or three CTAs share an SM: nothing here is specialised by warp, because these products are bound by
// latency and by the load / store instructions, not by the tensor pipe.
//
// Measured, 333 x 515 x 1001 u8 x s8 -> fp32 behind its dynamic quantization, whole calls: 111 us with the 16 x 16
// CUDA-core kernel that stood here, 37 us with this one (about 30 us of it are the quantization and the host).
#include <cuda.h>

#include <algorithm>
#include <cstring>

#include "common.cuh"
#include "epilogue.cuh"
#include "tcgen05.cuh"

namespace b200 {
namespace {

using namespace tc;

constexpr int THREADS = 256;
constexpr int MAX_BN = 128;
constexpr int STAGE_A = BLOCK_M * BLOCK_K;     // 16 KiB
constexpr int EPI_PITCH = 36;                  // words per staged row: 16-byte aligned, conflict-free for 8-lane phases

struct Ctl {
    uint64_t done[2];       // the MMAs reading a stage have completed
    uint32_t tmem_base;
    float scale[2];         // of the two operands (batched products)
};
constexpr size_t SMEM_BYTES = 1024 + 2 * (size_t)(STAGE_A + MAX_BN * BLOCK_K) + sizeof(Ctl);
static_assert(8 * 32 * EPI_PITCH * 4 <= 2 * (STAGE_A + 32 * BLOCK_K), "the epilogue staging reuses the operand stages");

// where an operand lies: element (row, k)
enum Layout {
    ROWS_K = 0,       // bytes p[row * ld + k]
    K_ROWS = 1,       // bytes p[k * ld + row]
    F32_ROWS_K = 2,   // the same two in binary32, quantized while they are loaded
    F32_K_ROWS = 3
};
// Byte operands are fetched a K block ahead into registers, which two CTAs per SM leave room for; binary32 ones are not
__host__ __device__ constexpr bool fetched_ahead(int la, int lb)
{
    return la < F32_ROWS_K && lb < F32_ROWS_K;
}
__host__ __device__ constexpr int ctas_per_sm(int la, int lb)
{
    return fetched_ahead(la, lb) ? 2 : 3;
}
struct Operand {
    const uint8_t *p;
    uint64_t ld;       // in elements
    uint32_t rows;     // rows that exist
    uint32_t k;        // elements of K that may be read; zeros beyond
    int vec;           // ROWS_K: 16, 8 or 1 (alignment of every row); K_ROWS: 4 or 1; F32_*: 1 if float4 loads are aligned
};

struct GatherParams {
    uint32_t M, N, K, block_n, tiles_m, tiles_n, tmem_cols;
    Operand a, b;
    void *C;
    GemmEpilogue ep;
    int vec_c;         // 4-element vectors of C are aligned
    int *status;
};

// The products of Bolt's matmul operator: one per batch index, operands quantized on the way in.
struct BatchParams {
    uint64_t batches;
    uint32_t c_dims[4], a_dims[4], b_dims[4];   // batch extents, innermost first; an operand's may be smaller (broadcast)
    int a_direct, b_direct;                     // as many products of the operand as of C: same index
    uint64_t a_bytes, b_bytes, c_bytes;         // one product's operands and result
    const unsigned *a_max, *b_max;              // partial maxima of |a|, |b| (float bits); null: the scale is a_scale, b_scale
    uint32_t a_slots, b_slots;
    float a_scale, b_scale, c_scale;
};

// 16 bytes from any address, of which the first n (0..16) exist: the aligned words that hold at least one of
// them ...
__device__ __forceinline__ void load_words(const uint8_t *p, uint32_t n, uint32_t (&v)[5])
{
    const uintptr_t a = reinterpret_cast<uintptr_t>(p);
    const uint32_t *w = reinterpret_cast<const uint32_t *>(a & ~(uintptr_t)3);
    const uint32_t end = n ? (uint32_t)(a & 3) + n : 0u;
#pragma unroll
    for (int j = 0; j < 5; ++j) {
        v[j] = (4u * j < end) ? __ldg(w + j) : 0u;
    }
}
// ... shifted into place
__device__ __forceinline__ uint4 shift_words(const uint8_t *p, uint32_t n, const uint32_t (&v)[5])
{
    const uint32_t lead = (uint32_t)(reinterpret_cast<uintptr_t>(p) & 3);
    uint32_t r[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        r[j] = __funnelshift_r(v[j], v[j + 1], lead * 8);
        const int left = (int)n - 4 * j;
        if (left < 4) {
            r[j] = left <= 0 ? 0u : r[j] & ((1u << (8 * left)) - 1u);
        }
    }
    return make_uint4(r[0], r[1], r[2], r[3]);
}

// quantizeF32ToU8 (avx512/quantize.cpp:135-178) with the zero point taken off again, and quantizeF32ToI8 (:195-233)
// The low byte of the result holds it.  vcvtps2dq gives 0x80000000 for NaN and from 2^31 on, which the clamp turns
// into the lower bound; below that, clamping before rounding is the same as after it, and adding 1.5 * 2^23 rounds
// (to nearest even) and leaves the integer in the low mantissa bits.
template <bool ZERO_POINT>
__device__ __forceinline__ uint32_t quantize_bits(float x, float s)
{
    constexpr float lo = ZERO_POINT ? 1.0f : -127.0f, hi = ZERO_POINT ? 255.0f : 127.0f;
    float f = __fmul_rn(x, s);
    if (ZERO_POINT) {
        f = __fadd_rn(f, 128.0f);
    }
    f = f < 2147483648.0f ? f : lo;
    return __float_as_uint(__fadd_rn(fminf(fmaxf(f, lo), hi), 12582912.0f));
}
template <bool ZERO_POINT>
__device__ __forceinline__ uint32_t quantize1(float x, float s)
{
    return (quantize_bits<ZERO_POINT>(x, s) ^ (ZERO_POINT ? 0x80u : 0u)) & 0xFFu;
}
template <bool ZERO_POINT>
__device__ __forceinline__ uint32_t quantize4(float4 v, float s)
{
    const uint32_t lo = __byte_perm(quantize_bits<ZERO_POINT>(v.x, s), quantize_bits<ZERO_POINT>(v.y, s), 0x0040);
    const uint32_t hi = __byte_perm(quantize_bits<ZERO_POINT>(v.z, s), quantize_bits<ZERO_POINT>(v.w, s), 0x0040);
    return __byte_perm(lo, hi, 0x5410) ^ (ZERO_POINT ? 0x80808080u : 0u);
}
// the first n (0..4) of four floats; with aligned vectors the extents are multiples of 4
__device__ __forceinline__ float4 load4f(const float *p, uint32_t n, int vec)
{
    if (vec) {   // n is 0 or 4
        return n ? __ldg(reinterpret_cast<const float4 *>(p)) : make_float4(0.f, 0.f, 0.f, 0.f);
    }
    float4 v;
    v.x = n > 0 ? __ldg(p) : 0.f;
    v.y = n > 1 ? __ldg(p + 1) : 0.f;
    v.z = n > 2 ? __ldg(p + 2) : 0.f;
    v.w = n > 3 ? __ldg(p + 3) : 0.f;
    return v;
}
__device__ __forceinline__ uint32_t first_bytes(uint32_t w, uint32_t n)
{
    return n >= 4 ? w : (n == 0 ? 0u : w & ((1u << (8 * n)) - 1u));
}

// The same tile from binary32.  Bytes beyond K are zeros (not quantized zeros).
template <int LAYOUT, bool ZERO_POINT>
__device__ __forceinline__ void load_tile_f32(const Operand &o, uint32_t r0, uint32_t rows_tile, uint32_t kb, uint8_t *dst, float s)
{
    const float *base = reinterpret_cast<const float *>(o.p);
    const uint32_t k0 = kb * BLOCK_K;
    const uint32_t left = o.k - k0;
    const uint32_t sh = left <= 32 ? 3u : (left <= 64 ? 4u : 5u);   // words of 4 k per row: 8, 16 or 32
    // eight float4 per thread are on their way before the first is used
    if (LAYOUT == F32_ROWS_K) {
        // lanes along K: a thread makes one 4-byte word of a float4
        const uint32_t total = rows_tile << sh;
        for (uint32_t i0 = threadIdx.x; i0 < total; i0 += 8 * THREADS) {
            float4 v[8];
#pragma unroll
            for (int u = 0; u < 8; ++u) {
                const uint32_t i = i0 + u * THREADS, row = i >> sh, k = k0 + (i & ((1u << sh) - 1u)) * 4;
                const uint32_t n = (i < total && r0 + row < o.rows && k < o.k) ? min(4u, o.k - k) : 0u;
                v[u] = load4f(base + (uint64_t)(r0 + row) * o.ld + k, n, o.vec);
            }
#pragma unroll
            for (int u = 0; u < 8; ++u) {
                const uint32_t i = i0 + u * THREADS, row = i >> sh, q = i & ((1u << sh) - 1u), k = k0 + q * 4;
                if (i < total) {
                    const uint32_t n = k < o.k ? min(4u, o.k - k) : 0u;
                    *reinterpret_cast<uint32_t *>(dst + row * 128 + (((q >> 2) ^ (row & 7)) << 4) + (q & 3) * 4) =
                        first_bytes(quantize4<ZERO_POINT>(v[u], s), n);
                }
            }
        }
    } else {
        // 4 rows x 4 k, transposed in registers; a warp covers 16 rows (64 bytes of each k) x 32 k
        const uint32_t total = (rows_tile << sh) / 4;
        auto place = [&](uint32_t i, uint32_t &q, uint32_t &row) {
            const uint32_t rest = i >> 5;
            q = (i & 7) + ((rest & ((1u << (sh - 3)) - 1u)) << 3);
            row = (((i >> 3) & 3) + ((rest >> (sh - 3)) << 2)) * 4;
        };
        for (uint32_t i0 = threadIdx.x; i0 < total; i0 += 2 * THREADS) {
            float4 v[2][4];
#pragma unroll
            for (int u = 0; u < 2; ++u) {
                const uint32_t i = i0 + u * THREADS;
                uint32_t q, row;
                place(i, q, row);
                const uint32_t k = k0 + q * 4, have = (i < total && r0 + row < o.rows) ? min(4u, o.rows - (r0 + row)) : 0u;
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    v[u][j] = load4f(base + (uint64_t)(k + j) * o.ld + r0 + row, k + j < o.k ? have : 0u, o.vec);
                }
            }
#pragma unroll
            for (int u = 0; u < 2; ++u) {
                const uint32_t i = i0 + u * THREADS;
                uint32_t q, row;
                place(i, q, row);
                if (i < total) {
                    const uint32_t k = k0 + q * 4;
                    uint32_t w[4];
#pragma unroll
                    for (int j = 0; j < 4; ++j) {
                        w[j] = k + j < o.k ? quantize4<ZERO_POINT>(v[u][j], s) : 0u;
                    }
                    const uint32_t a = __byte_perm(w[0], w[1], 0x5140), b = __byte_perm(w[2], w[3], 0x5140);
                    const uint32_t d = __byte_perm(w[0], w[1], 0x7362), e = __byte_perm(w[2], w[3], 0x7362);
                    const uint32_t t[4] = {__byte_perm(a, b, 0x5410), __byte_perm(a, b, 0x7632), __byte_perm(d, e, 0x5410), __byte_perm(d, e, 0x7632)};
#pragma unroll
                    for (int j = 0; j < 4; ++j) {
                        *reinterpret_cast<uint32_t *>(dst + (row + j) * 128 + (((q >> 2) ^ ((row + j) & 7)) << 4) + (q & 3) * 4) = t[j];
                    }
                }
            }
        }
    }
}

// K block `kb` of rows [r0, r0 + rows_tile) into the 128-byte swizzled tile at `dst`: the 16-byte chunk c of row r
// lies at r * 128 + ((c ^ (r & 7)) << 4).  Rows and bytes that do not exist become zeros; then every byte is XORed.
// In two steps: fetch() issues all of a thread's loads, put() shifts or transposes and stores, so that the loads of
// the next K block run beside the MMAs of this one.
constexpr int CHUNKS = BLOCK_M * 8 / THREADS;   // ROWS_K: a thread moves four 16-byte chunks at most
struct Fragment {
    uint32_t w[CHUNKS][5];
};
template <int LAYOUT>
__device__ __forceinline__ void fetch(const Operand &o, uint32_t r0, uint32_t rows_tile, uint32_t kb, Fragment &f)
{
    if (LAYOUT == ROWS_K) {
        // eight neighbouring lanes cover one row's 128 bytes
        const uint32_t c = threadIdx.x & 7, row0 = threadIdx.x >> 3, k = kb * BLOCK_K + c * 16;
        const uint8_t *p0 = o.p + (uint64_t)(r0 + row0) * o.ld + k;
        const uint64_t step = (uint64_t)(THREADS / 8) * o.ld;
        const uint32_t bytes = k < o.k ? min(16u, o.k - k) : 0u;
        auto count = [&](int i) {
            const uint32_t row = row0 + i * (THREADS / 8);
            return (row < rows_tile && r0 + row < o.rows) ? bytes : 0u;
        };
        if (o.vec == 16) {
#pragma unroll
            for (int i = 0; i < CHUNKS; ++i) {
                const uint4 v = count(i) ? __ldg(reinterpret_cast<const uint4 *>(p0 + i * step)) : make_uint4(0, 0, 0, 0);
                f.w[i][0] = v.x;
                f.w[i][1] = v.y;
                f.w[i][2] = v.z;
                f.w[i][3] = v.w;
            }
        } else if (o.vec == 8) {
#pragma unroll
            for (int i = 0; i < CHUNKS; ++i) {
                const uint2 *p = reinterpret_cast<const uint2 *>(p0 + i * step);
                const uint32_t n = count(i);
                const uint2 lo = n ? __ldg(p) : make_uint2(0, 0);
                const uint2 hi = n == 16 ? __ldg(p + 1) : make_uint2(0, 0);
                f.w[i][0] = lo.x;
                f.w[i][1] = lo.y;
                f.w[i][2] = hi.x;
                f.w[i][3] = hi.y;
            }
        } else {
#pragma unroll
            for (int i = 0; i < CHUNKS; ++i) {
                load_words(p0 + i * step, count(i), f.w[i]);
            }
        }
    } else {
        // 4 rows x 16 k per thread: sixteen 4-byte loads, lanes along the rows
        const uint32_t quads = rows_tile >> 2, c = threadIdx.x / quads, row = (threadIdx.x - c * quads) * 4, k = kb * BLOCK_K + c * 16;
        const uint32_t left = (c < 8 && r0 + row < o.rows) ? o.rows - (r0 + row) : 0u;
        const uint8_t *p = o.p + (uint64_t)k * o.ld + r0 + row;
        if (o.vec == 4) {   // (then the number of rows is a multiple of 4 too)
#pragma unroll
            for (int j = 0; j < 16; ++j) {
                f.w[j >> 2][j & 3] = (k + j < o.k && left != 0) ? __ldg(reinterpret_cast<const uint32_t *>(p + (uint64_t)j * o.ld)) : 0u;
            }
        } else {
#pragma unroll
            for (int j = 0; j < 16; ++j) {
                uint32_t w = 0;
#pragma unroll
                for (uint32_t t = 0; t < 4; ++t) {
                    w |= (k + j < o.k && t < left) ? (uint32_t)__ldg(p + (uint64_t)j * o.ld + t) << (8 * t) : 0u;
                }
                f.w[j >> 2][j & 3] = w;
            }
        }
    }
}
template <int LAYOUT, uint32_t XOR>
__device__ __forceinline__ void put(const Operand &o, uint32_t r0, uint32_t rows_tile, uint32_t kb, const Fragment &f, uint8_t *dst)
{
    if (LAYOUT == ROWS_K) {
        const uint32_t c = threadIdx.x & 7, row0 = threadIdx.x >> 3, k = kb * BLOCK_K + c * 16;
        const uint32_t bytes = k < o.k ? min(16u, o.k - k) : 0u;
        const uint8_t *p0 = o.p + (uint64_t)(r0 + row0) * o.ld + k;
        const uint64_t step = (uint64_t)(THREADS / 8) * o.ld;
#pragma unroll
        for (int i = 0; i < CHUNKS; ++i) {
            const uint32_t row = row0 + i * (THREADS / 8);
            if (row < rows_tile) {
                uint4 v = make_uint4(f.w[i][0], f.w[i][1], f.w[i][2], f.w[i][3]);
                if (o.vec < 8) {
                    v = shift_words(p0 + i * step, r0 + row < o.rows ? bytes : 0u, f.w[i]);
                }
                *reinterpret_cast<uint4 *>(dst + row * 128 + ((c ^ (row & 7)) << 4)) = make_uint4(v.x ^ XOR, v.y ^ XOR, v.z ^ XOR, v.w ^ XOR);
            }
        }
    } else {
        const uint32_t quads = rows_tile >> 2, c = threadIdx.x / quads, row = (threadIdx.x - c * quads) * 4;
        if (c < 8) {
            uint32_t t[4][4];   // [row][word of 4 k]
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                const uint32_t a = __byte_perm(f.w[q][0], f.w[q][1], 0x5140), b = __byte_perm(f.w[q][2], f.w[q][3], 0x5140);
                const uint32_t d = __byte_perm(f.w[q][0], f.w[q][1], 0x7362), e = __byte_perm(f.w[q][2], f.w[q][3], 0x7362);
                t[0][q] = __byte_perm(a, b, 0x5410);
                t[1][q] = __byte_perm(a, b, 0x7632);
                t[2][q] = __byte_perm(d, e, 0x5410);
                t[3][q] = __byte_perm(d, e, 0x7632);
            }
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                *reinterpret_cast<uint4 *>(dst + (row + j) * 128 + ((c ^ ((row + j) & 7)) << 4)) =
                    make_uint4(t[j][0] ^ XOR, t[j][1] ^ XOR, t[j][2] ^ XOR, t[j][3] ^ XOR);
            }
        }
    }
}

// scale = max(given, 127 / max|x|), the dynamic scale of quantize (avx512/quantize.cpp:129-133), from the partial
// maxima that absmax_pair_kernel left; called by a whole warp
__device__ __forceinline__ float dynamic_scale(const unsigned *slots, uint32_t n, float given, uint32_t lane)
{
    unsigned m = 0;
    for (uint32_t i = lane; i < n; i += 8 * 32) {   // (the loads of a round go out together)
        unsigned v[8];
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            v[j] = i + 32 * j < n ? slots[i + 32 * j] : 0u;
        }
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            m = max(m, v[j]);
        }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        m = max(m, __shfl_xor_sync(0xffffffffu, m, o));
    }
    const float mx = __uint_as_float(m);
    const float s = (mx == 0.f) ? 1.0f : __fdiv_rn(127.0f, mx);
    return (given > s) ? given : s;
}
// which of the operand's products goes with C's product `ic`
__device__ __forceinline__ uint64_t batch_index(uint64_t ic, const uint32_t (&c)[4], const uint32_t (&x)[4], int direct)
{
    if (direct) {
        return ic;
    }
    uint32_t idx[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        idx[i] = (uint32_t)(ic % c[i]);
        ic /= c[i];
    }
    uint64_t g = 0;
#pragma unroll
    for (int i = 3; i >= 0; --i) {
        g = g * x[i] + (idx[i] < x[i] ? idx[i] : 0u);
    }
    return g;
}

// BATCH: A arrives as (or is made) signed by taking the zero point off, so that sum (a - 128) b needs no column sums:
// it equals sum a b - 128 sum b in 32-bit arithmetic.
template <int LA, int LB, bool BATCH>
__global__ void __launch_bounds__(THREADS, ctas_per_sm(LA, LB))
gemm_gather_kernel(const __grid_constant__ GatherParams p, const __grid_constant__ BatchParams bp)
{
    extern __shared__ uint8_t smem_raw[];
    uint8_t *smem = align_1024(smem_raw);
    const uint32_t stage_bytes = STAGE_A + p.block_n * BLOCK_K;   // both tiles stay 1024-byte aligned
    Ctl *ctl = reinterpret_cast<Ctl *>(smem + 2 * (size_t)(STAGE_A + MAX_BN * BLOCK_K));
    const uint32_t warp = warp_index(), lane = threadIdx.x & 31;

    if (threadIdx.x == 0) {
        mbar_init(&ctl->done[0], 1);
        mbar_init(&ctl->done[1], 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&ctl->tmem_base)),
                     "r"(p.tmem_cols)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    tcgen05_fence_before();
    __syncthreads();
    tcgen05_fence_after();
    const uint32_t tmem_base = ctl->tmem_base;
    const uint32_t idesc = make_idesc_i8(p.block_n) | (BATCH ? 1u << 7 : 0u);   // bit 7: A is s8
    const uint32_t num_kb = (p.K + BLOCK_K - 1) / BLOCK_K;
    const uint64_t per_batch = (uint64_t)p.tiles_m * p.tiles_n;
    const uint64_t tiles = BATCH ? per_batch * bp.batches : per_batch;
    Operand oa = p.a, ob = p.b;
    void *C = p.C;
    float scale_a = 0.f, scale_b = 0.f, factor = 0.f;
    if (BATCH) {
        asm volatile("griddepcontrol.wait;" ::: "memory");   // the partial maxima (and everything before them) are there
        if (warp < 2) {
            const bool a = warp == 0;
            const float given = a ? bp.a_scale : bp.b_scale;
            const unsigned *slots = a ? bp.a_max : bp.b_max;
            const float s = slots ? dynamic_scale(slots, a ? bp.a_slots : bp.b_slots, given, lane) : given;
            if (lane == 0) {
                ctl->scale[warp] = s;
            }
        }
        __syncthreads();
        scale_a = ctl->scale[0];
        scale_b = ctl->scale[1];
        factor = __fdiv_rn(p.ep.out_kind == 2 ? bp.c_scale : 1.0f, __fmul_rn(scale_a, scale_b));
    }
    uint32_t issued = 0;   // K blocks handed to the tensor core so far: stage = issued & 1, parity from issued >> 1
    bool dead = false;

    for (uint64_t tile = blockIdx.x; tile < tiles && !dead; tile += gridDim.x) {
        const uint64_t batch = BATCH ? tile / per_batch : 0u;
        const uint64_t in_batch = tile - batch * per_batch;
        const uint32_t m0 = (uint32_t)(in_batch % p.tiles_m) * BLOCK_M, n0 = (uint32_t)(in_batch / p.tiles_m) * p.block_n;
        if (BATCH) {
            oa.p = p.a.p + batch_index(batch, bp.c_dims, bp.a_dims, bp.a_direct) * bp.a_bytes;
            ob.p = p.b.p + batch_index(batch, bp.c_dims, bp.b_dims, bp.b_direct) * bp.b_bytes;
            C = reinterpret_cast<uint8_t *>(p.C) + batch * bp.c_bytes;
        }
        constexpr bool AHEAD = fetched_ahead(LA, LB);
        Fragment fa, fb;
        if (AHEAD && num_kb != 0) {
            fetch<LA>(oa, m0, BLOCK_M, 0, fa);
            fetch<LB>(ob, n0, p.block_n, 0, fb);
        }
        for (uint32_t kb = 0; kb < num_kb; ++kb, ++issued) {
            const uint32_t s = issued & 1;
            uint8_t *sa = smem + s * stage_bytes, *sb = sa + STAGE_A;
            // the MMAs that read this stage two K blocks ago are done
            bool ok = issued < 2 || mbar_wait(&ctl->done[s], ((issued >> 1) + 1) & 1);
            if (ok) {
                if constexpr (LA >= F32_ROWS_K) {
                    load_tile_f32<LA, true>(oa, m0, BLOCK_M, kb, sa, scale_a);
                } else {
                    if (!AHEAD) {
                        fetch<LA>(oa, m0, BLOCK_M, kb, fa);
                    }
                    put<LA, BATCH ? 0x80808080u : 0u>(oa, m0, BLOCK_M, kb, fa, sa);
                }
                if constexpr (LB >= F32_ROWS_K) {
                    load_tile_f32<LB, false>(ob, n0, p.block_n, kb, sb, scale_b);
                } else {
                    if (!AHEAD) {
                        fetch<LB>(ob, n0, p.block_n, kb, fb);
                    }
                    put<LB, 0u>(ob, n0, p.block_n, kb, fb, sb);
                }
                if (AHEAD && kb + 1 < num_kb) {
                    fetch<LA>(oa, m0, BLOCK_M, kb + 1, fa);
                    fetch<LB>(ob, n0, p.block_n, kb + 1, fb);
                }
                fence_proxy_async_smem();
            }
            if (__syncthreads_or(!ok)) {
                dead = true;
                break;
            }
            if (warp == 0) {
                const bool leader = elect_one();   // the same lane every time
                tcgen05_fence_after();
                const uint64_t da = make_desc_sw128(smem_u32(sa)), db = make_desc_sw128(smem_u32(sb));
                const uint32_t steps = (min((uint32_t)BLOCK_K, p.K - kb * BLOCK_K) + UMMA_K - 1) / UMMA_K;
                for (uint32_t k = 0; k < steps; ++k) {
                    if (leader) {
                        umma_i8(tmem_base, da + 2 * k, db + 2 * k, idesc, (kb | k) != 0 ? 1u : 0u);
                    }
                }
                if (leader) {
                    tcgen05_commit(&ctl->done[s]);
                }
            }
            __syncwarp();
        }
        if (dead) {
            break;
        }
        if (num_kb != 0) {
            const uint32_t last = issued - 1;
            const bool ok = mbar_wait(&ctl->done[last & 1], (last >> 1) & 1);
            if (__syncthreads_or(!ok)) {
                dead = true;
                break;
            }
        }
        tcgen05_fence_after();
        // Epilogue: warp = lane quadrant x half of the 32-column chunks.  The accumulators go through shared memory
        // (the operand stages, which nothing reads any more) so that C is read and written along its rows.
        const uint32_t quad = warp & 3, half = warp >> 2, nch = p.block_n >> 5;
        const uint32_t c_begin = half ? (nch + 1) / 2 : 0u, c_end = half ? nch : (nch + 1) / 2;
        int32_t *stg = reinterpret_cast<int32_t *>(smem) + warp * 32 * EPI_PITCH;
        const bool add_c = p.ep.out_kind != 2 && p.ep.accumulate;   // its reads go out together, before the first store
        for (uint32_t c = c_begin; c < c_end; ++c) {
            uint32_t r[32];
            if (num_kb != 0) {
                tmem_ld32(tmem_base + ((quad * 32u) << 16) + c * 32, r);
                tmem_ld_wait(r);
            } else {
#pragma unroll
                for (int j = 0; j < 32; ++j) {
                    r[j] = 0;
                }
            }
            __syncwarp();
#pragma unroll
            for (int j = 0; j < 32; j += 4) {
                *reinterpret_cast<uint4 *>(stg + lane * EPI_PITCH + j) = make_uint4(r[j], r[j + 1], r[j + 2], r[j + 3]);
            }
            __syncwarp();
            const uint32_t mq = m0 + quad * 32, nc = n0 + c * 32;
            if (p.vec_c) {
                // N is a multiple of 4: eight lanes per row, four columns each
                const uint32_t n = nc + (lane & 7) * 4;
                if (n < p.N) {
                    int off[4];
                    float cf[4];
#pragma unroll
                    for (int j = 0; j < 4; ++j) {
                        off[j] = p.ep.offsetC ? __ldg(p.ep.offsetC + n + j) : 0;
                        cf[j] = BATCH ? factor : (p.ep.out_kind ? column_factor(p.ep, n + j) : 0.f);
                    }
                    for (uint32_t i0 = lane >> 3; i0 < 32; i0 += 16) {
                        int acc[4][4] = {};
                        if (add_c) {
#pragma unroll
                            for (int u = 0; u < 4; ++u) {
                                if (mq + i0 + 4 * u < p.M) {
                                    read_c<4>(p.N, C, mq + i0 + 4 * u, n, acc[u]);
                                }
                            }
                        }
#pragma unroll
                        for (int u = 0; u < 4; ++u) {
                            const uint32_t i = i0 + 4 * u;
                            if (mq + i < p.M) {
                                const int4 v = *reinterpret_cast<const int4 *>(stg + i * EPI_PITCH + (lane & 7) * 4);
                                acc[u][0] += v.x + off[0];
                                acc[u][1] += v.y + off[1];
                                acc[u][2] += v.z + off[2];
                                acc[u][3] += v.w + off[3];
                                finish<4>(p.ep, p.N, C, mq + i, n, acc[u], cf);
                            }
                        }
                    }
                }
            } else {
                const uint32_t n = nc + lane;
                if (n < p.N) {
                    const int off = p.ep.offsetC ? __ldg(p.ep.offsetC + n) : 0;
                    const float cf[1] = {BATCH ? factor : (p.ep.out_kind ? column_factor(p.ep, n) : 0.f)};
                    for (uint32_t i0 = 0; i0 < 32; i0 += 16) {
                        int acc[16][1] = {};
                        if (add_c) {
#pragma unroll
                            for (int u = 0; u < 16; ++u) {
                                if (mq + i0 + u < p.M) {
                                    read_c<1>(p.N, C, mq + i0 + u, n, acc[u]);
                                }
                            }
                        }
#pragma unroll
                        for (int u = 0; u < 16; ++u) {
                            if (mq + i0 + u < p.M) {
                                acc[u][0] += stg[(i0 + u) * EPI_PITCH + lane] + off;
                                finish<1>(p.ep, p.N, C, mq + i0 + u, n, acc[u], cf);
                            }
                        }
                    }
                }
            }
        }
        // the next tile's operands overwrite the staging, its MMAs the accumulators
        tcgen05_fence_before();
        __syncthreads();
        tcgen05_fence_after();
    }
    if (dead && threadIdx.x == 0) {
        atomicExch(p.status, 31);
    }
    tcgen05_fence_before();
    __syncthreads();
    if (warp == 0) {
        tcgen05_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(p.tmem_cols) : "memory");
    }
}

// Partial maxima of |a| and |b| (float bits): the first ga blocks take a, the others b; block i of an operand writes
// slot i.  No initial value and no atomic: whoever needs the scale reduces the few hundred slots itself.
constexpr int MAX_THREADS = 512;
constexpr uint32_t MAX_BLOCK = MAX_THREADS * 32;   // elements a block takes at a time: 64 KiB
__device__ __forceinline__ unsigned abs4(float4 v)
{
    return max(max(__float_as_uint(v.x) & 0x7FFFFFFFu, __float_as_uint(v.y) & 0x7FFFFFFFu),
        max(__float_as_uint(v.z) & 0x7FFFFFFFu, __float_as_uint(v.w) & 0x7FFFFFFFu));
}
__global__ void __launch_bounds__(MAX_THREADS)
absmax_pair_kernel(const float *a, uint64_t na, unsigned *a_slots, uint32_t ga, const float *b, uint64_t nb, unsigned *b_slots, uint32_t gb)
{
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    const bool first = blockIdx.x < ga;
    const float *x = first ? a : b;
    const uint64_t n = first ? na : nb;
    const uint32_t blk = first ? blockIdx.x : blockIdx.x - ga;
    const uint32_t blocks = first ? ga : gb;
    const bool aligned = (reinterpret_cast<uintptr_t>(x) & 15) == 0;
    unsigned m = 0;
    // eight 16-byte loads per thread in flight
    for (uint64_t i0 = (uint64_t)blk * MAX_BLOCK; i0 < n; i0 += (uint64_t)blocks * MAX_BLOCK) {
        const uint64_t i1 = min(n, i0 + MAX_BLOCK);
        if (aligned && i1 - i0 == MAX_BLOCK) {
            const float4 *x4 = reinterpret_cast<const float4 *>(x + i0) + threadIdx.x;
            float4 v[8];
#pragma unroll
            for (int j = 0; j < 8; ++j) {
                v[j] = __ldg(x4 + j * MAX_THREADS);
            }
#pragma unroll
            for (int j = 0; j < 8; ++j) {
                m = max(m, abs4(v[j]));
            }
        } else {
#pragma unroll 8
            for (uint64_t i = i0 + threadIdx.x; i < i1; i += MAX_THREADS) {
                m = max(m, __float_as_uint(__ldg(x + i)) & 0x7FFFFFFFu);
            }
        }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        m = max(m, __shfl_xor_sync(0xffffffffu, m, o));
    }
    __shared__ unsigned warp_max[MAX_THREADS / 32];
    if ((threadIdx.x & 31) == 0) {
        warp_max[threadIdx.x >> 5] = m;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
#pragma unroll
        for (int w = 1; w < MAX_THREADS / 32; ++w) {
            m = max(m, warp_max[w]);
        }
        (first ? a_slots : b_slots)[blk] = m;
    }
}

__device__ __forceinline__ int dp4a_s8s8(uint32_t a, uint32_t b, int acc)
{
    int d;
    asm("dp4a.s32.s32 %0, %1, %2, %3;" : "=r"(d) : "r"(a), "r"(b), "r"(acc));
    return d;
}
// u8 results of the row GEMV: all but the last N % 4 rows through vpmovusdb, those add 128, compare signed with 255
// and keep the low byte (mvm_avx512_vnni_row.cpp:384-406, 884-900)
__device__ __forceinline__ void store_mvm(void *y, uint32_t n, uint32_t N, int acc, int out_kind, float factor)
{
    if (out_kind == 1) {
        reinterpret_cast<float *>(y)[n] = acc_to_f32(acc, factor);
    } else if (n >= N - (N % 4)) {
        const int t = (int)((uint32_t)cvt_rne_x86(__fmul_rn(__int2float_rn(acc), factor)) + 128u);
        reinterpret_cast<uint8_t *>(y)[n] = (t < 255) ? (uint8_t)t : (uint8_t)255;
    } else {
        reinterpret_cast<uint8_t *>(y)[n] = (uint8_t)acc_to_u8(acc, factor);
    }
}

// A decoding step's attention is bound by reading the matrix; one query against 384 keys of 64 takes one block of
// 32 keys x 64 per 8 KiB.
// One row of C per product: y[n] = sum_k (m_u8[n, k] - 128) v_s8[k], the vector being A and the matrix B, both
// quantized on the way in.  Blocks of 256 threads take MVM_ROWS rows n of one product at a time.
// LB ROWS_K: 2^k lanes share a row, four k each, dp4a; LB K_ROWS: lanes along n, the warps split K.
constexpr uint32_t MVM_ROWS = 32;
template <int LB>
__global__ void __launch_bounds__(THREADS)
mvm_batch_kernel(const __grid_constant__ GatherParams p, const __grid_constant__ BatchParams bp, int a_f32)
{
    extern __shared__ __align__(16) uint8_t sv[];   // the vector as s8, zero padded to a multiple of 128
    __shared__ float scales[2];
    __shared__ int part[THREADS / 32][32];
    const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    asm volatile("griddepcontrol.wait;" ::: "memory");
    if (warp < 2) {
        const float given = warp == 0 ? bp.a_scale : bp.b_scale;
        const unsigned *slots = warp == 0 ? bp.a_max : bp.b_max;
        const float s = slots ? dynamic_scale(slots, warp == 0 ? bp.a_slots : bp.b_slots, given, lane) : given;
        if (lane == 0) {
            scales[warp] = s;
        }
    }
    __syncthreads();
    const float sa = scales[0], sb = scales[1];
    const float factor = __fdiv_rn(p.ep.out_kind == 2 ? bp.c_scale : 1.0f, __fmul_rn(sa, sb));
    const uint32_t blocks_n = (p.N + MVM_ROWS - 1) / MVM_ROWS;
    const uint32_t k_pad = (p.K + 127) & ~127u;
    for (uint64_t t = blockIdx.x; t < blocks_n * bp.batches; t += gridDim.x) {
        const uint64_t batch = t / blocks_n;
        const uint32_t n0 = (uint32_t)(t - batch * blocks_n) * MVM_ROWS;
        const uint8_t *pa = p.a.p + batch_index(batch, bp.c_dims, bp.a_dims, bp.a_direct) * bp.a_bytes;
        const uint8_t *pb = p.b.p + batch_index(batch, bp.c_dims, bp.b_dims, bp.b_direct) * bp.b_bytes;
        uint8_t *y = reinterpret_cast<uint8_t *>(p.C) + batch * bp.c_bytes;
        __syncthreads();   // the previous product's vector and partial sums have been read
        for (uint32_t k = threadIdx.x; k < k_pad; k += THREADS) {
            uint32_t v = 0;
            if (k < p.K) {
                v = a_f32 ? quantize1<false>(__ldg(reinterpret_cast<const float *>(pa) + k), sa) : (uint32_t)__ldg(pa + k);
            }
            sv[k] = (uint8_t)v;
        }
        __syncthreads();
        if (LB == ROWS_K || LB == F32_ROWS_K) {
            const uint32_t words = (p.K + 3) / 4;
            uint32_t sh = 0;                       // 2^sh lanes per row
            while (sh < 5 && (1u << sh) < words) {
                ++sh;
            }
            const uint32_t per_warp = 32u >> sh, sub = lane & ((1u << sh) - 1u);
            for (uint32_t r = warp * per_warp; r < MVM_ROWS; r += (THREADS / 32) * per_warp) {
                const uint32_t n = n0 + r + (lane >> sh);
                int acc = 0;
                if (n < p.N && r + (lane >> sh) < MVM_ROWS) {
                    for (uint32_t q = sub; q < words; q += 1u << sh) {
                        const uint32_t have = min(4u, p.K - q * 4);
                        uint32_t w;
                        if (LB == F32_ROWS_K) {
                            w = quantize4<true>(load4f(reinterpret_cast<const float *>(pb) + (uint64_t)n * p.K + q * 4, have, p.b.vec), sb);
                        } else {
                            const uint8_t *e = pb + (uint64_t)n * p.K + q * 4;
                            if (p.b.vec >= 8 && have == 4) {
                                w = __ldg(reinterpret_cast<const uint32_t *>(e));
                            } else {
                                w = 0;
                                for (uint32_t j = 0; j < have; ++j) {
                                    w |= (uint32_t)__ldg(e + j) << (8 * j);
                                }
                            }
                            w ^= 0x80808080u;
                        }
                        // (beyond K the vector is zero)
                        acc = dp4a_s8s8(w, *reinterpret_cast<const uint32_t *>(sv + q * 4), acc);
                    }
                }
                for (uint32_t o = (1u << sh) >> 1; o > 0; o >>= 1) {
                    acc += __shfl_xor_sync(0xffffffffu, acc, o);
                }
                if (sub == 0 && n < p.N && r + (lane >> sh) < MVM_ROWS) {
                    store_mvm(y, n, p.N, acc, p.ep.out_kind, factor);
                }
            }
        } else {
            const uint32_t n = n0 + lane;
            int acc = 0;
            if (n < p.N) {
#pragma unroll 8
                for (uint32_t k = warp; k < p.K; k += THREADS / 32) {
                    const uint64_t e = (uint64_t)k * p.N + n;
                    const uint32_t q = LB == F32_K_ROWS ? quantize1<true>(__ldg(reinterpret_cast<const float *>(pb) + e), sb) : ((uint32_t)__ldg(pb + e) ^ 0x80u);
                    acc += (int)(int8_t)q * (int)(int8_t)sv[k];
                }
            }
            part[warp][lane] = acc;
            __syncthreads();
            if (warp == 0 && n < p.N) {
#pragma unroll
                for (int w = 1; w < THREADS / 32; ++w) {
                    acc += part[w][lane];
                }
                store_mvm(y, n, p.N, acc, p.ep.out_kind, factor);
            }
        }
    }
}

int row_alignment(const void *p, uint64_t ld)
{
    const uint64_t a = reinterpret_cast<uintptr_t>(p) | ld;
    return a % 16 == 0 ? 16 : (a % 8 == 0 ? 8 : 1);
}

}  // namespace

// Tile width: as few column blocks of at most 128 as cover N, narrower while there are fewer tiles than SMs.
uint32_t gather_block_n(uint64_t tiles_m, uint32_t N, int sms)
{
    const uint32_t blocks = (N + MAX_BN - 1) / MAX_BN;
    uint32_t bn = (uint32_t)B200_ALIGN((N + blocks - 1) / blocks, 32);
    while (bn > 32 && tiles_m * ((N + bn - 1) / bn) < (uint64_t)sms) {
        bn -= 32;
    }
    return bn;
}

// A u8 [M][K] (or [K][M] when a_transposed), B the packed weight [ALIGN(N,16)][Kp], zero padded.
EE launch_gemm_gather(uint32_t M, uint32_t N, uint32_t K, const uint8_t *A, bool a_transposed, const int8_t *B,
    uint32_t Kp, void *C, const GemmEpilogue &ep, cudaStream_t st)
{
    if (M == 0 || N == 0) {
        return SUCCESS;
    }
    if ((M + 15) / 16 > 65535) {
        return NOT_SUPPORTED;   // (a million rows of such operands have never been taken; the kernel itself has no such limit)
    }
    DeviceCtx *c = ctx();
    if (c == nullptr) {
        return UNKNOWN;
    }
    {
        const void *ks[2] = {(const void *)gemm_gather_kernel<ROWS_K, ROWS_K, false>, (const void *)gemm_gather_kernel<K_ROWS, ROWS_K, false>};
        B200_EE(raise_smem_limit(c, KF_GATHER, ks, 2, SMEM_BYTES));
    }
    GatherParams p;
    p.M = M;
    p.N = N;
    p.K = K;
    p.tiles_m = (M + BLOCK_M - 1) / BLOCK_M;
    p.block_n = gather_block_n(p.tiles_m, N, c->sm_count);
    p.tiles_n = (N + p.block_n - 1) / p.block_n;
    p.tmem_cols = p.block_n > 64 ? 128u : p.block_n;
    p.a.p = A;
    p.a.rows = M;
    p.a.k = K;
    p.a.ld = a_transposed ? M : K;
    p.a.vec = a_transposed ? (((reinterpret_cast<uintptr_t>(A) | M) % 4 == 0) ? 4 : 1) : row_alignment(A, K);
    p.b.p = reinterpret_cast<const uint8_t *>(B);
    p.b.rows = N;
    p.b.k = Kp;   // zeros between K and Kp
    p.b.ld = Kp;
    p.b.vec = row_alignment(B, Kp);
    p.C = C;
    p.ep = ep;
    p.status = c->d_status;
    const uintptr_t c_align = ep.out_kind == 2 ? 4 : 16;
    p.vec_c = (N % 4 == 0) && (reinterpret_cast<uintptr_t>(C) % c_align == 0);
    const uint64_t tiles = (uint64_t)p.tiles_m * p.tiles_n, slots = (uint64_t)c->sm_count * ctas_per_sm(ROWS_K, ROWS_K);
    const uint32_t grid = (uint32_t)(tiles < slots ? tiles : slots);
    if (a_transposed) {
        gemm_gather_kernel<K_ROWS, ROWS_K, false><<<grid, THREADS, SMEM_BYTES, st>>>(p, BatchParams());
    } else {
        gemm_gather_kernel<ROWS_K, ROWS_K, false><<<grid, THREADS, SMEM_BYTES, st>>>(p, BatchParams());
    }
    count_launch();
    B200_CUDA(cudaGetLastError());
    return SUCCESS;
}

namespace {

// its set-up runs beside the reduction in front of it, if there is one
template <typename... P, typename... A>
cudaError_t launch_behind(bool reduction, const cudaLaunchConfig_t &cfg, void (*kernel)(P...), const A &...args)
{
    return reduction ? launch_programmatic(cfg, kernel, args...) : cudaLaunchKernelEx(&cfg, kernel, args...);
}
template <int LA>
cudaError_t launch_batch(int lb, bool reduction, const cudaLaunchConfig_t &cfg, const GatherParams &p, const BatchParams &bp)
{
    switch (lb) {
        case ROWS_K:
            return launch_behind(reduction, cfg, gemm_gather_kernel<LA, ROWS_K, true>, p, bp);
        case K_ROWS:
            return launch_behind(reduction, cfg, gemm_gather_kernel<LA, K_ROWS, true>, p, bp);
        case F32_ROWS_K:
            return launch_behind(reduction, cfg, gemm_gather_kernel<LA, F32_ROWS_K, true>, p, bp);
        default:
            return launch_behind(reduction, cfg, gemm_gather_kernel<LA, F32_K_ROWS, true>, p, bp);
    }
}
template <int LA>
void batch_kernels(const void **ks)
{
    ks[0] = (const void *)gemm_gather_kernel<LA, ROWS_K, true>;
    ks[1] = (const void *)gemm_gather_kernel<LA, K_ROWS, true>;
    ks[2] = (const void *)gemm_gather_kernel<LA, F32_ROWS_K, true>;
    ks[3] = (const void *)gemm_gather_kernel<LA, F32_K_ROWS, true>;
}
Operand operand(const MatmulOperand &o, uint32_t rows, uint32_t K, bool rows_contiguous)
{
    Operand r;
    r.p = reinterpret_cast<const uint8_t *>(o.p);
    r.ld = rows_contiguous ? rows : K;
    r.rows = rows;
    r.k = K;
    const uint64_t a = reinterpret_cast<uintptr_t>(o.p);
    if (o.f32) {
        r.vec = (a % 16 == 0) && (r.ld % 4 == 0);
    } else if (rows_contiguous) {
        r.vec = ((a | r.ld) % 4 == 0) ? 4 : 1;
    } else {
        r.vec = row_alignment(o.p, r.ld);
    }
    return r;
}

}  // namespace

// All products of a matmul call: at most one pass over the binary32 operands for their scales, then one kernel that
// quantizes, multiplies and converts.  BERT-base attention of 32 x 128 tokens, scores and context (384 products of
// 128 x 64 x 128 and of 128 x 128 x 64): 47 us against 8.0 ms for a pack and a GEMM launch per product.  Its memory
// floor is 15 us (each operand and result once); the operands are read a second time for their scales.
EE launch_matmul_batch(const MatmulBatch &mb, cudaStream_t st)
{
    DeviceCtx *c = ctx();
    if (c == nullptr) {
        return UNKNOWN;
    }
    const size_t mvm_smem = B200_ALIGN((size_t)mb.K, 128);
    if (mb.M == 1 && mvm_smem > 200 * 1024) {
        return NOT_SUPPORTED;
    }
    {
        const void *ks[16];
        batch_kernels<ROWS_K>(ks);
        batch_kernels<K_ROWS>(ks + 4);
        batch_kernels<F32_ROWS_K>(ks + 8);
        batch_kernels<F32_K_ROWS>(ks + 12);
        B200_EE(raise_smem_limit(c, KF_MATMUL, ks, 16, SMEM_BYTES));
        const void *kv[4] = {(const void *)mvm_batch_kernel<ROWS_K>, (const void *)mvm_batch_kernel<K_ROWS>,
            (const void *)mvm_batch_kernel<F32_ROWS_K>, (const void *)mvm_batch_kernel<F32_K_ROWS>};
        B200_EE(raise_smem_limit(c, KF_MATMUL_ROW, kv, 4, 200 * 1024));
    }
    GatherParams p;
    std::memset(&p, 0, sizeof(p));
    BatchParams bp;
    std::memset(&bp, 0, sizeof(bp));
    p.M = mb.M;
    p.N = mb.N;
    p.K = mb.K;
    p.a = operand(mb.a, mb.M, mb.K, mb.a.transposed);
    p.b = operand(mb.b, mb.N, mb.K, !mb.b.transposed);
    p.C = mb.C;
    p.ep.out_kind = mb.out_kind;
    p.ep.accumulate = mb.accumulate;
    p.status = c->d_status;
    bp.batches = mb.batches;
    for (int i = 0; i < 4; ++i) {
        bp.c_dims[i] = mb.c_dims[i];
        bp.a_dims[i] = mb.a.dims[i];
        bp.b_dims[i] = mb.b.dims[i];
    }
    bp.a_direct = mb.a.direct;
    bp.b_direct = mb.b.direct;
    bp.a_bytes = (uint64_t)mb.M * mb.K * (mb.a.f32 ? 4 : 1);
    bp.b_bytes = (uint64_t)mb.N * mb.K * (mb.b.f32 ? 4 : 1);
    const uint32_t esz = mb.out_kind == 2 ? 1 : 4;
    bp.c_bytes = (uint64_t)mb.M * mb.N * esz;
    bp.a_scale = mb.a.scale;
    bp.b_scale = mb.b.scale;
    bp.c_scale = mb.c_scale;
    // every product starts at a multiple of its size, so the vectors' alignment has to hold for that too
    auto all_batches = [&](Operand &o, const MatmulOperand &m, uint64_t bytes) {
        if (m.f32) {
            o.vec = o.vec && (bytes % 16 == 0 || mb.batches == 1);
        } else if (m.transposed != (&m == &mb.b)) {
            o.vec = (bytes % 4 == 0 || mb.batches == 1) ? o.vec : 1;
        } else if (mb.batches != 1 && bytes % 16 != 0) {
            o.vec = (bytes % 8 == 0 && o.vec >= 8) ? 8 : 1;
        }
    };
    all_batches(p.a, mb.a, bp.a_bytes);
    all_batches(p.b, mb.b, bp.b_bytes);
    p.vec_c = (mb.N % 4 == 0) && ((reinterpret_cast<uintptr_t>(mb.C) | (mb.batches == 1 ? 0 : bp.c_bytes)) % (4 * esz) == 0);

    // partial maxima: a block per 64 KiB of an operand, four blocks per SM at most, and no more slots than given
    auto blocks_for = [&](const MatmulOperand &o) -> uint32_t {
        if (!o.f32) {
            return 0;
        }
        uint64_t g = (o.elems + MAX_BLOCK - 1) / MAX_BLOCK;
        g = std::min<uint64_t>(g, 4 * (uint64_t)c->sm_count);
        return (uint32_t)std::min<uint64_t>(g, o.max_slots);
    };
    const uint32_t ga = blocks_for(mb.a), gb = blocks_for(mb.b);
    bp.a_max = ga ? mb.a.slots : nullptr;
    bp.b_max = gb ? mb.b.slots : nullptr;
    bp.a_slots = ga;
    bp.b_slots = gb;
    if (ga + gb) {
        absmax_pair_kernel<<<ga + gb, MAX_THREADS, 0, st>>>(reinterpret_cast<const float *>(mb.a.p), mb.a.elems, mb.a.slots, ga,
            reinterpret_cast<const float *>(mb.b.p), mb.b.elems, mb.b.slots, gb);
        count_launch();
        B200_CUDA(cudaGetLastError());
    }
    cudaLaunchConfig_t cfg = {};
    cfg.blockDim = dim3(THREADS);
    cfg.stream = st;
    const bool reduction = ga + gb != 0;
    const int la = (mb.a.f32 ? 2 : 0) + (mb.a.transposed ? 1 : 0);
    const int lb = (mb.b.f32 ? 2 : 0) + (mb.b.transposed ? 0 : 1);
    cudaError_t e;
    if (mb.M == 1) {
        const uint64_t work = (uint64_t)((mb.N + MVM_ROWS - 1) / MVM_ROWS) * mb.batches;
        cfg.gridDim = dim3((uint32_t)std::min<uint64_t>(work, 8 * (uint64_t)c->sm_count));
        cfg.dynamicSmemBytes = mvm_smem;
        const int af = mb.a.f32 ? 1 : 0;
        tls().last_gemm_tc = 0;
        e = lb == ROWS_K ? launch_behind(reduction, cfg, mvm_batch_kernel<ROWS_K>, p, bp, af)
            : lb == K_ROWS ? launch_behind(reduction, cfg, mvm_batch_kernel<K_ROWS>, p, bp, af)
            : lb == F32_ROWS_K ? launch_behind(reduction, cfg, mvm_batch_kernel<F32_ROWS_K>, p, bp, af)
                               : launch_behind(reduction, cfg, mvm_batch_kernel<F32_K_ROWS>, p, bp, af);
    } else {
        p.tiles_m = (mb.M + BLOCK_M - 1) / BLOCK_M;
        p.block_n = gather_block_n((uint64_t)p.tiles_m * mb.batches, mb.N, c->sm_count);
        p.tiles_n = (mb.N + p.block_n - 1) / p.block_n;
        p.tmem_cols = p.block_n > 64 ? 128u : p.block_n;
        cfg.dynamicSmemBytes = SMEM_BYTES;
        const uint64_t tiles = (uint64_t)p.tiles_m * p.tiles_n * mb.batches;
        cfg.gridDim = dim3((uint32_t)std::min<uint64_t>(tiles, (uint64_t)c->sm_count * ctas_per_sm(la, lb)));
        e = la == ROWS_K ? launch_batch<ROWS_K>(lb, reduction, cfg, p, bp)
            : la == K_ROWS ? launch_batch<K_ROWS>(lb, reduction, cfg, p, bp)
            : la == F32_ROWS_K ? launch_batch<F32_ROWS_K>(lb, reduction, cfg, p, bp)
                               : launch_batch<F32_K_ROWS>(lb, reduction, cfg, p, bp);
        tls().last_gemm_tc = 1;
    }
    count_launch();
    B200_CUDA(e);
    return SUCCESS;
}

}  // namespace b200
