// gemm_i8_gather.cu -- u8 x s8 products on the sm_100a tensor cores whose operands TMA cannot fetch.
//
// The TMA kernel (gemm_i8_tcgen05.cu) needs 16-byte aligned rows and an untransposed A.  Here the CTA's threads
// bring the operands into the swizzled shared-memory layout of tcgen05.mma themselves, so any K, any alignment and
// a transposed A run on the tensor cores.  Shapes: frames x features against classes (333 x 515 x 1001), the
// 1..33-sized products of Bolt's cover test (compute/blas_enhance/tests/test_mmm.cpp:165-171).
//
// One tile is 128 rows x block_n columns; a CTA is 256 threads, all of which load, convert and store; one of them
// issues the MMAs.  Two 128-byte K blocks are in flight (the loads of block k+1 run while the MMAs of block k do)
// and three CTAs share an SM, which is what hides the load latency: nothing here is specialised by warp, because
// these products are bound by latency and by the load / store instructions, not by the tensor pipe.
//
// Measured, 333 x 515 x 1001 u8 x s8 -> fp32 behind its dynamic quantization, whole calls: 111 us with the 16 x 16
// CUDA-core kernel that stood here, 61 us with this one (about 40 us of both are the quantization and the host).
#include <cuda.h>

#include "common.cuh"
#include "tcgen05.cuh"

namespace b200 {
namespace {

using namespace tc;

constexpr int THREADS = 256;
constexpr int MAX_BN = 128;
constexpr int STAGE_A = BLOCK_M * BLOCK_K;     // 16 KiB
constexpr int EPI_PITCH = 36;                  // words per staged row: 16-byte aligned, conflict-free for 8-lane phases
constexpr int CTAS_PER_SM = 3;

struct Ctl {
    uint64_t done[2];       // the MMAs reading a stage have completed
    uint32_t tmem_base;
};
constexpr size_t SMEM_BYTES = 1024 + 2 * (size_t)(STAGE_A + MAX_BN * BLOCK_K) + sizeof(Ctl);
static_assert(8 * 32 * EPI_PITCH * 4 <= 2 * (STAGE_A + 32 * BLOCK_K), "the epilogue staging reuses the operand stages");

// where an operand lies: element (row, k)
enum Layout {
    ROWS_K = 0,   // p[row * ld + k]
    K_ROWS = 1    // p[k * ld + row]
};
struct Operand {
    const uint8_t *p;
    uint64_t ld;
    uint32_t rows;     // rows that exist
    uint32_t k;        // bytes of K that may be read; zeros beyond
    int vec;           // ROWS_K: 16, 8 or 1 (alignment of every row); K_ROWS: 4 or 1
};

struct GatherParams {
    uint32_t M, N, K, block_n, tiles_m, tiles_n, tmem_cols;
    Operand a, b;
    void *C;
    GemmEpilogue ep;
    int vec_c;         // 4-element vectors of C are aligned
    int *status;
};

// 16 bytes from any address, of which the first n (>= 1) exist: aligned words that hold at least one of
// them, shifted into place
__device__ __forceinline__ uint4 load16_any(const uint8_t *p, uint32_t n)
{
    const uintptr_t a = reinterpret_cast<uintptr_t>(p);
    const uint32_t *w = reinterpret_cast<const uint32_t *>(a & ~(uintptr_t)3);
    const uint32_t lead = (uint32_t)(a & 3);
    const uint32_t end = lead + n;
    uint32_t v[5];
#pragma unroll
    for (int j = 0; j < 5; ++j) {
        v[j] = (4u * j < end) ? __ldg(w + j) : 0u;
    }
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

// K block `kb` of rows [r0, r0 + rows_tile) into the 128-byte swizzled tile at `dst`: the 16-byte chunk c of row r
// lies at r * 128 + ((c ^ (r & 7)) << 4).  Rows and bytes that do not exist become zeros.
template <int LAYOUT>
__device__ __forceinline__ void load_tile(const Operand &o, uint32_t r0, uint32_t rows_tile, uint32_t kb, uint8_t *dst)
{
    const uint32_t k0 = kb * BLOCK_K;
    if (LAYOUT == ROWS_K) {
        // a thread moves 16-byte chunks; eight neighbouring lanes cover one row's 128 bytes
#pragma unroll 4
        for (uint32_t i = threadIdx.x; i < rows_tile * 8; i += THREADS) {
            const uint32_t row = i >> 3, c = i & 7, k = k0 + c * 16;
            uint4 v = make_uint4(0, 0, 0, 0);
            if (r0 + row < o.rows && k < o.k) {
                const uint8_t *p = o.p + (uint64_t)(r0 + row) * o.ld + k;
                const uint32_t n = min(16u, o.k - k);
                if (o.vec == 16 && n == 16) {
                    v = __ldg(reinterpret_cast<const uint4 *>(p));
                } else if (o.vec >= 8 && (n & 7) == 0) {
                    const uint2 lo = __ldg(reinterpret_cast<const uint2 *>(p));
                    const uint2 hi = n == 16 ? __ldg(reinterpret_cast<const uint2 *>(p) + 1) : make_uint2(0, 0);
                    v = make_uint4(lo.x, lo.y, hi.x, hi.y);
                } else {
                    v = load16_any(p, n);
                }
            }
            *reinterpret_cast<uint4 *>(dst + row * 128 + ((c ^ (row & 7)) << 4)) = v;
        }
    } else {
        // a thread takes 4 rows x 16 k (sixteen 4-byte loads, lanes along the rows) and transposes in registers
        for (uint32_t i = threadIdx.x; i < rows_tile * 2; i += THREADS) {
            const uint32_t quads = rows_tile >> 2;
            const uint32_t c = i / quads, row = (i - c * quads) * 4, k = k0 + c * 16;
            const uint32_t left = r0 + row < o.rows ? o.rows - (r0 + row) : 0u;
            const uint8_t *p = o.p + (uint64_t)k * o.ld + r0 + row;
            uint32_t w[16];
#pragma unroll
            for (int j = 0; j < 16; ++j) {
                w[j] = 0;
                if (k + j < o.k && left != 0) {
                    const uint8_t *q = p + (uint64_t)j * o.ld;
                    if (o.vec == 4 && left >= 4) {
                        w[j] = __ldg(reinterpret_cast<const uint32_t *>(q));
                    } else {
                        for (uint32_t t = 0; t < min(left, 4u); ++t) {
                            w[j] |= (uint32_t)__ldg(q + t) << (8 * t);
                        }
                    }
                }
            }
            uint32_t t[4][4];   // [row][word of 4 k]
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                const uint32_t a = __byte_perm(w[4 * q], w[4 * q + 1], 0x5140), b = __byte_perm(w[4 * q + 2], w[4 * q + 3], 0x5140);
                const uint32_t d = __byte_perm(w[4 * q], w[4 * q + 1], 0x7362), e = __byte_perm(w[4 * q + 2], w[4 * q + 3], 0x7362);
                t[0][q] = __byte_perm(a, b, 0x5410);
                t[1][q] = __byte_perm(a, b, 0x7632);
                t[2][q] = __byte_perm(d, e, 0x5410);
                t[3][q] = __byte_perm(d, e, 0x7632);
            }
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                *reinterpret_cast<uint4 *>(dst + (row + j) * 128 + ((c ^ ((row + j) & 7)) << 4)) =
                    make_uint4(t[j][0], t[j][1], t[j][2], t[j][3]);
            }
        }
    }
}

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

// V consecutive results of row m, columns n .. n+V-1
template <int V>
__device__ __forceinline__ void finish(const GatherParams &p, void *C, uint32_t m, uint32_t n, int (&acc)[V], const float (&cf)[V])
{
    const GemmEpilogue &ep = p.ep;
    const size_t o = (size_t)m * p.N + n;
    if (ep.out_kind != 2 && ep.accumulate) {
        const int32_t *cin = reinterpret_cast<const int32_t *>(C) + o;
        if (V == 4) {
            const int4 v = *reinterpret_cast<const int4 *>(cin);
            acc[0] += v.x;
            acc[1 % V] += v.y;
            acc[2 % V] += v.z;
            acc[3 % V] += v.w;
        } else {
            acc[0] += cin[0];
        }
    }
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

template <int LA>
__global__ void __launch_bounds__(THREADS, CTAS_PER_SM) gemm_gather_kernel(const __grid_constant__ GatherParams p)
{
    extern __shared__ uint8_t smem_raw[];
    uint8_t *smem = reinterpret_cast<uint8_t *>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
    const uint32_t stage_bytes = STAGE_A + p.block_n * BLOCK_K;   // both tiles stay 1024-byte aligned
    Ctl *ctl = reinterpret_cast<Ctl *>(smem + 2 * (size_t)(STAGE_A + MAX_BN * BLOCK_K));
    const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31;

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
    const uint32_t idesc = make_idesc_i8(p.block_n);
    const uint32_t num_kb = (p.K + BLOCK_K - 1) / BLOCK_K;
    const uint64_t tiles = (uint64_t)p.tiles_m * p.tiles_n;
    uint32_t issued = 0;   // K blocks handed to the tensor core so far: stage = issued & 1, parity from issued >> 1
    bool dead = false;

    for (uint64_t tile = blockIdx.x; tile < tiles && !dead; tile += gridDim.x) {
        const uint32_t m0 = (uint32_t)(tile % p.tiles_m) * BLOCK_M, n0 = (uint32_t)(tile / p.tiles_m) * p.block_n;
        for (uint32_t kb = 0; kb < num_kb; ++kb, ++issued) {
            const uint32_t s = issued & 1;
            uint8_t *sa = smem + s * stage_bytes, *sb = sa + STAGE_A;
            // the MMAs that read this stage two K blocks ago are done
            bool ok = issued < 2 || mbar_wait(&ctl->done[s], ((issued >> 1) + 1) & 1);
            if (ok) {
                load_tile<LA>(p.a, m0, BLOCK_M, kb, sa);
                load_tile<ROWS_K>(p.b, n0, p.block_n, kb, sb);
                fence_proxy_async_smem();
            }
            if (__syncthreads_or(!ok)) {
                dead = true;
                break;
            }
            if (threadIdx.x == 0) {
                tcgen05_fence_after();
                const uint64_t da = make_desc_sw128(smem_u32(sa)), db = make_desc_sw128(smem_u32(sb));
                const uint32_t steps = (min((uint32_t)BLOCK_K, p.K - kb * BLOCK_K) + UMMA_K - 1) / UMMA_K;
                for (uint32_t k = 0; k < steps; ++k) {
                    umma_i8(tmem_base, da + 2 * k, db + 2 * k, idesc, (kb | k) != 0 ? 1u : 0u);
                }
                tcgen05_commit(&ctl->done[s]);
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
                        cf[j] = p.ep.out_kind ? column_factor(p.ep, n + j) : 0.f;
                    }
#pragma unroll 4
                    for (uint32_t i = lane >> 3; i < 32; i += 4) {
                        if (mq + i < p.M) {
                            const int4 v = *reinterpret_cast<const int4 *>(stg + i * EPI_PITCH + (lane & 7) * 4);
                            int acc[4] = {v.x + off[0], v.y + off[1], v.z + off[2], v.w + off[3]};
                            finish<4>(p, p.C, mq + i, n, acc, cf);
                        }
                    }
                }
            } else {
                const uint32_t n = nc + lane;
                if (n < p.N) {
                    const int off = p.ep.offsetC ? __ldg(p.ep.offsetC + n) : 0;
                    const float cf[1] = {p.ep.out_kind ? column_factor(p.ep, n) : 0.f};
#pragma unroll 4
                    for (uint32_t i = 0; i < 32; ++i) {
                        if (mq + i < p.M) {
                            int acc[1] = {stg[i * EPI_PITCH + lane] + off};
                            finish<1>(p, p.C, mq + i, n, acc, cf);
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

// Tile width: as few column blocks of at most 128 as cover N, narrower while there are fewer tiles than SMs.
uint32_t pick_bn(uint32_t tiles_m, uint32_t N, int sms)
{
    const uint32_t blocks = (N + MAX_BN - 1) / MAX_BN;
    uint32_t bn = (uint32_t)B200_ALIGN((N + blocks - 1) / blocks, 32);
    while (bn > 32 && (uint64_t)tiles_m * ((N + bn - 1) / bn) < (uint64_t)sms) {
        bn -= 32;
    }
    return bn;
}

int row_alignment(const void *p, uint64_t ld)
{
    const uint64_t a = reinterpret_cast<uintptr_t>(p) | ld;
    return a % 16 == 0 ? 16 : (a % 8 == 0 ? 8 : 1);
}

}  // namespace

// A u8 [M][K] (or [K][M] when a_transposed), B the packed weight [ALIGN(N,16)][Kp], zero padded.
EE launch_gemm_gather(uint32_t M, uint32_t N, uint32_t K, const uint8_t *A, bool a_transposed, const int8_t *B,
    uint32_t Kp, void *C, const GemmEpilogue &ep, cudaStream_t st)
{
    if (M == 0 || N == 0) {
        return SUCCESS;
    }
    if ((M + 15) / 16 > 65535) {
        return NOT_SUPPORTED;
    }
    DeviceCtx *c = ctx();
    if (c == nullptr) {
        return UNKNOWN;
    }
    {
        const void *ks[2] = {(const void *)gemm_gather_kernel<ROWS_K>, (const void *)gemm_gather_kernel<K_ROWS>};
        B200_EE(raise_smem_limit(c, KF_GATHER, ks, 2, SMEM_BYTES));
    }
    GatherParams p;
    p.M = M;
    p.N = N;
    p.K = K;
    p.tiles_m = (M + BLOCK_M - 1) / BLOCK_M;
    p.block_n = pick_bn(p.tiles_m, N, c->sm_count);
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
    const uint64_t tiles = (uint64_t)p.tiles_m * p.tiles_n, slots = (uint64_t)c->sm_count * CTAS_PER_SM;
    const uint32_t grid = (uint32_t)(tiles < slots ? tiles : slots);
    if (a_transposed) {
        gemm_gather_kernel<K_ROWS><<<grid, THREADS, SMEM_BYTES, st>>>(p);
    } else {
        gemm_gather_kernel<ROWS_K><<<grid, THREADS, SMEM_BYTES, st>>>(p);
    }
    count_launch();
    B200_CUDA(cudaGetLastError());
    return SUCCESS;
}

}  // namespace b200
