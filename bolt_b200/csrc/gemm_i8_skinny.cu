// gemm_i8_skinny.cu -- u8 x s8 products of few rows and a weight that fits L2: a short query through a layer.
//
// Such a product is latency from end to end: about 2 MB of weight over 148 SMs is 16 KB each, and the 128-row tensor
// tile of gemm_i8_tcgen05.cu costs barriers, descriptors, tensor memory and a store through staging for a handful of
// rows.  Here a CTA owns 8 or 16 columns, its warps split K, every lane loads 16 contiguous bytes of a weight row and
// of the activation rows straight into the fragments of mma.m16n8k32 (the order of K inside a 64-byte unit is free as
// long as both operands use the same one, so no shuffles and no shared memory on the way in), and the warps' partial
// sums meet once in shared memory.
//
// 24 layers of 768 x 3072 and 3072 x 768 at 16 tokens, the whole pass: 183 us with a TMA kernel launch and a Python call
// per layer, 95 us with this (9.1 us are the weights' share of the memory rate; the rest is 24 times a latency).
//
// In a chain of layers (bolt_b200_gemm_u8s8_chain) the kernel of layer i+1 starts while layer i runs and has its weight
// fragments, offsets and factors in registers when layer i's result arrives.  That is safe because this kernel lets
// its successor start only after its own wait: whoever starts then knows that everything before layer i is complete,
// and the chain's weights are constant.  A layer with its input scale in device memory waits first.
#include "common.cuh"
#include "epilogue.cuh"

namespace b200 {
namespace {

constexpr int MAX_WARPS = 16;

struct SkinnyParams {
    uint32_t M, N, K, Kp;
    const uint8_t *A;
    const int8_t *B;
    void *C;
    GemmEpilogue ep;
    int vec_c;
    int preload;   // the weight, offsets and column factors may be read before the previous kernel has finished
};

__device__ __forceinline__ void mma_u8s8(int (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1)
{
    asm volatile("mma.sync.aligned.m16n8k32.row.col.s32.u8.s8.s32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
                 : "+r"(c[0]), "+r"(c[1]), "+r"(c[2]), "+r"(c[3])
                 : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}
__device__ __forceinline__ uint4 load16(const void *p)
{
    uint4 v;
    asm volatile("ld.global.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(p) : "memory");
    return v;
}

// MT blocks of 16 rows, NT blocks of 8 columns, UNITS 64-byte units of K in flight per warp
template <int MT, int NT, int UNITS>
__global__ void __launch_bounds__(MAX_WARPS * 32, MT == 1 ? 2 : 1) gemm_skinny_kernel(const __grid_constant__ SkinnyParams p)
{
    extern __shared__ __align__(16) int part[];   // [warp][NT][MT * 16 rows][8]
    const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31, warps = blockDim.x >> 5;
    const uint32_t g = lane >> 2, t = lane & 3;
    const uint32_t n0 = blockIdx.x * (8 * NT);
    const uint32_t units = (p.K + 63) / 64;
    const uint4 zero = make_uint4(0, 0, 0, 0);
    // weight rows n0 + 8 j + g (the packed weight has a multiple of 16 of them); K is a multiple of 16
    const int8_t *brow = p.B + (size_t)(n0 + g) * p.Kp + t * 16;
    uint4 b[UNITS][NT];
    auto load_b = [&](uint32_t u0) {
#pragma unroll
        for (int i = 0; i < UNITS; ++i) {
            const uint32_t k = (u0 + i * warps) * 64;
#pragma unroll
            for (int j = 0; j < NT; ++j) {
                b[i][j] = (k + t * 16 < p.K && n0 + 8 * j < p.N) ? load16(brow + (size_t)(8 * j) * p.Kp + k) : zero;
            }
        }
    };
    // what this thread will convert: four columns of rows threadIdx.x / (2 NT), ...
    const uint32_t q = threadIdx.x % (2 * NT), n = n0 + q * 4;
    int off[4];
    float cf[4];
    auto load_columns = [&] {
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const bool in = n + j < p.N;
            off[j] = (in && p.ep.offsetC) ? p.ep.offsetC[n + j] : 0;
            cf[j] = (in && p.ep.out_kind) ? column_factor(p.ep, n + j) : 0.f;
        }
    };
    if (p.preload) {
        load_b(warp);
        load_columns();
    }
    asm volatile("griddepcontrol.wait;" ::: "memory");
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");   // not earlier: see the head of this file
    if (!p.preload) {
        load_b(warp);
    }
    int acc[MT][NT][4] = {};
    for (uint32_t u0 = warp; u0 < units; u0 += UNITS * warps) {
        uint4 a[UNITS][MT][2];
#pragma unroll
        for (int i = 0; i < UNITS; ++i) {
            const uint32_t k = (u0 + i * warps) * 64 + t * 16;
#pragma unroll
            for (int m = 0; m < MT; ++m) {
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    const uint32_t row = m * 16 + h * 8 + g;
                    a[i][m][h] = (k < p.K && row < p.M) ? load16(p.A + (size_t)row * p.K + k) : zero;
                }
            }
        }
        if (u0 != warp) {
            load_b(u0);
        }
#pragma unroll
        for (int i = 0; i < UNITS; ++i) {
#pragma unroll
            for (int m = 0; m < MT; ++m) {
#pragma unroll
                for (int j = 0; j < NT; ++j) {
                    mma_u8s8(acc[m][j], a[i][m][0].x, a[i][m][1].x, a[i][m][0].y, a[i][m][1].y, b[i][j].x, b[i][j].y);
                    mma_u8s8(acc[m][j], a[i][m][0].z, a[i][m][1].z, a[i][m][0].w, a[i][m][1].w, b[i][j].z, b[i][j].w);
                }
            }
        }
    }
    if (!p.preload) {
        load_columns();
    }
#pragma unroll
    for (int j = 0; j < NT; ++j) {
#pragma unroll
        for (int m = 0; m < MT; ++m) {
            int *dst = part + ((warp * NT + j) * (MT * 16) + m * 16 + g) * 8 + t * 2;
            *reinterpret_cast<int2 *>(dst) = make_int2(acc[m][j][0], acc[m][j][1]);
            *reinterpret_cast<int2 *>(dst + 64) = make_int2(acc[m][j][2], acc[m][j][3]);
        }
    }
    __syncthreads();
    const uint32_t rows_per_pass = blockDim.x / (2 * NT);
    for (uint32_t m = threadIdx.x / (2 * NT); m < p.M && n < p.N; m += rows_per_pass) {
        int v[4] = {off[0], off[1], off[2], off[3]};
        const int *src = part + ((q >> 1) * (MT * 16) + m) * 8 + (q & 1) * 4;
        for (uint32_t w = 0; w < warps; ++w) {
            const int4 x = *reinterpret_cast<const int4 *>(src + w * (NT * MT * 128));
            v[0] += x.x;
            v[1] += x.y;
            v[2] += x.z;
            v[3] += x.w;
        }
        const bool add_c = p.ep.out_kind != 2 && p.ep.accumulate;
        if (p.vec_c) {
            if (add_c) {
                int old[4];
                read_c<4>(p.N, p.C, m, n, old);
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    v[j] += old[j];
                }
            }
            finish<4>(p.ep, p.N, p.C, m, n, v, cf);
        } else {
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                if (n + j < p.N) {
                    int one[1] = {0};
                    if (add_c) {
                        read_c<1>(p.N, p.C, m, n + j, one);
                    }
                    one[0] += v[j];
                    const float f[1] = {cf[j]};
                    finish<1>(p.ep, p.N, p.C, m, n + j, one, f);
                }
            }
        }
    }
}

template <int MT, int NT, int UNITS>
cudaError_t launch(const SkinnyParams &p, cudaStream_t st)
{
    const uint32_t units = (p.K + 63) / 64;
    uint32_t warps = (units + UNITS - 1) / UNITS;   // one batch of loads per warp, if sixteen warps can do it
    warps = warps < 4 ? 4 : (warps > MAX_WARPS ? MAX_WARPS : warps);
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((p.N + 8 * NT - 1) / (8 * NT));
    cfg.blockDim = dim3(warps * 32);
    cfg.dynamicSmemBytes = warps * NT * MT * 128 * sizeof(int);
    cfg.stream = st;
    return launch_programmatic(cfg, gemm_skinny_kernel<MT, NT, UNITS>, p);
}

}  // namespace

// Few rows, and a weight of at most 32 MiB and 6144 columns: beyond that the TMA kernel streams as fast.  Measured, us per
// product in a graph of forty, this kernel against that one (whose time does not depend on so few rows): 16 rows x 768 x
// 3072 3.0 / 4.0, 3072 x 768 3.2 / 7.1, 4096 x 4096 5.6 / 8.9, 8192 x 4096 10.9 / 15.1, 1024 x 16384 7.0 / 5.8, 4096 x 12288
// 17.9 / 12.2.  With 32 rows 768 x 3072 3.4 / 4.0, 1024 x 4096 3.6 / 4.4, 8192 x 2048 7.8 / 14.6, but 4096 x 4096 9.3 / 8.9,
// 8192 x 4096 17.7 / 15.1.  From 33 rows on it only pays with 8 columns per CTA: 48 x 3072 x 768 5.1 / 7.1, 64 x 256 x 1024
// 2.7 / 3.2, but 64 x 768 x 3072 6.1 / 4.0.
bool gemm_skinny_preferred(uint32_t M, uint32_t N, uint32_t K, int sms)
{
    const uint64_t weight = (uint64_t)N * K;
    if (M <= 16) {
        return N <= 6144 && weight <= (32ull << 20);
    }
    if (M <= 32) {
        return weight <= (12ull << 20) ? N <= 6144 : (N <= 2048 && weight <= (32ull << 20));
    }
    return M <= 64 && N <= 8 * (uint32_t)sms && weight <= (32ull << 20);
}

// The operands satisfy gemm_tcgen05_eligible.  preload: see SkinnyParams.
EE launch_gemm_skinny(uint32_t M, uint32_t N, uint32_t K, const uint8_t *A, const int8_t *B, uint32_t Kp, void *C,
    const GemmEpilogue &ep, bool preload, cudaStream_t st)
{
    DeviceCtx *c = ctx();
    if (c == nullptr) {
        return UNKNOWN;
    }
    SkinnyParams p;
    p.M = M;
    p.N = N;
    p.K = K;
    p.Kp = Kp;
    p.A = A;
    p.B = B;
    p.C = C;
    p.ep = ep;
    const uintptr_t c_align = ep.out_kind == 2 ? 4 : 16;
    p.vec_c = (N % 4 == 0) && (reinterpret_cast<uintptr_t>(C) % c_align == 0);
    // (d_sA is no constant of the chain: an earlier layer may just be writing it)
    p.preload = preload && ep.sA_dev == nullptr ? 1 : 0;
    // 8 columns per CTA, 16 where that makes more CTAs than SMs
    const bool wide = (N + 7) / 8 > (uint32_t)c->sm_count;
    cudaError_t e;
    if (M <= 16) {
        e = wide ? launch<1, 2, 2>(p, st) : launch<1, 1, 3>(p, st);
    } else if (M <= 32) {
        e = wide ? launch<2, 2, 2>(p, st) : launch<2, 1, 3>(p, st);
    } else {
        e = launch<4, 1, 2>(p, st);   // (narrow: gemm_skinny_preferred)
    }
    count_launch();
    B200_CUDA(e);
    return SUCCESS;
}

}  // namespace b200
