// bnn.cu -- 1-bit convolution (XNOR-Net: DT_BIN11, DoReFa: DT_BIN01) on packed 32-bit words.
//
// Replaces Bolt's ARMv8.2 kernels (compute/tensor/src/cpu/arm/bnn/convolution_xnor_A76.cpp:17-724,
// convolution_dorefa_A76.cpp:17-715), the filter bit repack (convolution_transform_bnn.h:32-86) and
// the input binarisation (common/uni/include/data_type.h:197-233):
//   bit(x)  = x >= 0 (BIN11) or x >= 0.5 (BIN01); padding is a zero bit in both modes
//   XNOR    : sum = fh*fw*ic - 2 * popcount(x XOR w)       (zero bit = -1)
//   DoReFa  : sum = popcount(x AND w)
//   output  = fma_fp16( (fp16)(int16)sum, scale[oc], bias[oc] ), fp16 NCHWc8
//
// Three kernels: binarise + zero-pad the fp16 NCHWc8 input into bit words [N][C/32][Hp][Wp] (one streaming pass, 16x
// smaller than the input), repack the filter bits into [OC][tap][C/32] words (once), and the convolution: an implicit
// GEMM on the tensor cores (kind::i8), pixels x output channels x (tap, word, bit).  Only the bits travel through
// memory; a CTA's threads widen them to bytes while they fill the operand stages -- activations to 0 / 1, weights to
// -1 / +1 (XNOR) or 0 / 1 (DoReFa) -- and with
//     acc = sum_valid x * (2w - 1),   fh*fw*ic - 2 popcount(x XOR w) = 2 acc + fh*fw*ic - 2 popcount(w)
// the padding (x = 0) needs no treatment.  The order of the 32 bits of a word inside its 32 bytes of K is free as
// long as both operands use the same one: word j of 8 takes bits j, j+8, j+16, j+24, one shift and one mask.
//
// Measured, 256 -> 256 channels, 3 x 3 on 28 x 28, batch 128, whole call: 519 us with XOR + popcount (16 per clock and
// SM: 411 us of popcounts alone), 86 us with this; 26 us is the tensor pipe's share, 15 us the bytes.
#include <cuda_fp16.h>

#include <cstring>

#include "common.cuh"
#include "tcgen05.cuh"

namespace b200 {
namespace {

using namespace tc;

constexpr int WIDEN_THREADS = 256;                // widen, and convert the results
constexpr int THREADS = WIDEN_THREADS + 32;       // + the warp that issues the MMAs
constexpr int MAX_BN = 128;                       // output channels of a tile
constexpr int STAGE_A = 2 * BLOCK_M * BLOCK_K;    // two row blocks: 256 pixels
constexpr int STAGE = STAGE_A + MAX_BN * BLOCK_K; // 48 KiB; two stages, two CTAs per SM
constexpr uint32_t MAX_WORDS = 800;               // (tap, word) pairs of a filter: its sums, of 25600 bits at most, stay int16

struct B4d {
    DataType dt;
    DataFormat df;
    uint32_t n, c, h, w;
};
bool get4(const TensorDesc *d, B4d *o)
{
    if (d == nullptr || d->nDims != 4) {
        return false;
    }
    o->dt = d->dt;
    o->df = d->df;
    o->w = d->dims[0];
    o->h = d->dims[1];
    o->c = d->dims[2];
    o->n = d->dims[3];
    return true;
}

// filter bits NCHW, MSB first in each byte (cpu/general/convolution.cpp:161-179) -> words [OC][tap][Cw],
// bit (c % 32) of word c / 32
__global__ void bnn_pack_filter_kernel(const uint8_t *__restrict__ src, uint32_t OC, uint32_t IC, uint32_t taps,
    uint32_t Cw, uint32_t *__restrict__ dst)
{
    const size_t total = (size_t)OC * taps * Cw;
    for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += (size_t)gridDim.x * blockDim.x) {
        const uint32_t cw = (uint32_t)(i % Cw);
        const uint32_t tap = (uint32_t)((i / Cw) % taps);
        const uint32_t oc = (uint32_t)(i / ((size_t)Cw * taps));
        uint32_t word = 0;
        for (uint32_t b = 0; b < 32; ++b) {
            const uint32_t c = cw * 32 + b;
            if (c < IC) {
                const size_t pos = ((size_t)oc * IC + c) * taps + tap;
                word |= (uint32_t)((src[pos >> 3] >> (7 - (pos & 7))) & 1u) << b;
            }
        }
        dst[i] = word;
    }
}

// fp16 NCHWc8 -> bit words [N][Cw][Hp][Wp], zero words in the padding ring.  Lanes run along the row, so that both
// the 16-byte reads of a channel block and the 4-byte writes are contiguous.
__global__ void bnn_binarize_pad_kernel(const __half *__restrict__ in, uint32_t N, uint32_t IC, uint32_t IH, uint32_t IW,
    uint32_t Hp, uint32_t Wp, uint32_t pt, uint32_t pl, uint32_t Cw, float threshold, uint32_t *__restrict__ out)
{
    const uint32_t total = N * Hp * Wp * Cw;   // the scratch is smaller than 4 GiB, so words count in 32 bits
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < total; i += gridDim.x * blockDim.x) {
        const uint32_t row = i / Wp, x = i - row * Wp;
        const uint32_t pl_ = row / Hp, y = row - pl_ * Hp;
        const uint32_t n = pl_ / Cw, cw = pl_ - n * Cw;
        uint32_t word = 0;
        const int iy = (int)y - (int)pt, ix = (int)x - (int)pl;
        if (iy >= 0 && iy < (int)IH && ix >= 0 && ix < (int)IW) {
            const size_t pix = (size_t)iy * IW + ix;
#pragma unroll
            for (uint32_t blk = 0; blk < 4; ++blk) {
                const uint32_t c0 = cw * 32 + blk * 8;
                if (c0 < IC) {
                    const uint4 v = *reinterpret_cast<const uint4 *>(
                        in + ((size_t)n * IC + c0) * IH * IW + pix * 8);
                    const uint32_t h[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
                    for (int j = 0; j < 4; ++j) {
                        const float lo = __half2float(__ushort_as_half((unsigned short)(h[j] & 0xFFFFu)));
                        const float hi = __half2float(__ushort_as_half((unsigned short)(h[j] >> 16)));
                        word |= (lo >= threshold ? 1u : 0u) << (blk * 8 + 2 * j);
                        word |= (hi >= threshold ? 1u : 0u) << (blk * 8 + 2 * j + 1);
                    }
                }
            }
        }
        out[i] = word;
    }
}

struct BnnParams {
    uint32_t N, OH, OW, OC, Hp, Wp, Cw, FH, FW, sH, sW;
    uint32_t kbits;     // fh * fw * ic
    uint32_t kw_words;  // fh * fw * Cw
    uint32_t row_blocks, block_n, tiles_m, tiles_n, tmem_cols;   // tile: row_blocks (1 or 2) x 128 pixels, block_n channels
    const uint32_t *xb;
    const uint32_t *wb;
    const __half *scale;
    const __half *bias;
    __half *out;
    int *status;
};

struct BnnCtl {
    uint64_t full[2];       // a stage is widened (one arrival per warp)
    uint64_t done[2];       // the MMAs reading a stage have completed
    uint64_t drained;       // the accumulators have been read (one arrival per warp)
    uint32_t tmem_base;
    __align__(16) int corr[MAX_BN];      // XNOR: kbits - 2 popcount(w) of every channel of the tile
    __half2 scale[MAX_BN / 2], bias[MAX_BN / 2];
};
constexpr size_t BNN_SMEM = 1024 + 2 * (size_t)STAGE + sizeof(BnnCtl);

// 32 bits -> 32 bytes: the bit t becomes the byte t * mul + add.  (1, 0) leaves 0 / 1; (-254, -1) gives -1 / +1: the
// complement of 254 t, which never carries into the next byte.
struct Widen {
    uint32_t mul, add;
};
template <bool PLAIN>
__device__ __forceinline__ void store_word(uint8_t *tile, uint32_t row, uint32_t word, uint32_t w, const Widen &m)
{
    uint32_t v[8];
#pragma unroll
    for (int j = 0; j < 8; ++j) {
        const uint32_t t = (w >> j) & 0x01010101u;
        v[j] = PLAIN ? t : t * m.mul + m.add;
    }
    uint8_t *r = tile + row * 128;
    *reinterpret_cast<uint4 *>(r + (((2 * word) ^ (row & 7)) << 4)) = make_uint4(v[0], v[1], v[2], v[3]);
    *reinterpret_cast<uint4 *>(r + (((2 * word + 1) ^ (row & 7)) << 4)) = make_uint4(v[4], v[5], v[6], v[7]);
}

// Tile = up to 256 pixels x up to 128 channels; K in blocks of 4 words = 128 bytes.  256 threads widen: each the word
// (threadIdx & 3) of rows threadIdx / 4, + 64, + 128, + 192 of the pixels and of rows + 0, + 64 of the weights; the
// words of K block k+1 are fetched while block k is widened.  A ninth warp issues the MMAs, so that the widening warps
// wait for nobody but the stage they need.  Two stages, and two CTAs share an SM: one's epilogue runs beside the
// other's MMAs.
template <bool XNOR>
__global__ void __launch_bounds__(THREADS, 2) bnn_conv_kernel(const __grid_constant__ BnnParams p)
{
    extern __shared__ uint8_t smem_raw[];
    uint8_t *smem = align_1024(smem_raw);
    BnnCtl *ctl = reinterpret_cast<BnnCtl *>(smem + 2 * STAGE);
    const uint32_t warp = warp_index(), lane = threadIdx.x & 31;
    if (threadIdx.x == 0) {
        for (int i = 0; i < 2; ++i) {
            mbar_init(&ctl->full[i], WIDEN_THREADS / 32);
            mbar_init(&ctl->done[i], 1);
        }
        mbar_init(&ctl->drained, WIDEN_THREADS / 32);
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
    const uint32_t num_kb = (p.kw_words + 3) / 4;
    const uint32_t tiles = p.tiles_m * p.tiles_n;
    bool dead = false;

    if (warp == WIDEN_THREADS / 32) {
        // ------------------------------- MMA issuer ---------------------------------------------
        {
            const bool leader = elect_one();   // (commits follow the MMAs of the thread that issues them)
            const uint32_t idesc = make_idesc_i8(p.block_n);
            uint32_t issued = 0, it = 0;
            for (uint32_t tile = blockIdx.x; !dead && tile < tiles; tile += gridDim.x, ++it) {
                if (it != 0 && !mbar_wait_warp(&ctl->drained, (it - 1) & 1)) {
                    dead = true;
                    break;
                }
                for (uint32_t kb = 0; kb < num_kb; ++kb, ++issued) {
                    const uint32_t s = issued & 1;
                    if (!mbar_wait_warp(&ctl->full[s], (issued >> 1) & 1)) {
                        dead = true;
                        break;
                    }
                    tcgen05_fence_after();
                    uint8_t *sa = smem + s * STAGE;
                    const uint64_t db = make_desc_sw128(smem_u32(sa + STAGE_A));
                    for (uint32_t r = 0; r < p.row_blocks; ++r) {
                        const uint64_t da = make_desc_sw128(smem_u32(sa + r * BLOCK_M * BLOCK_K));
#pragma unroll
                        for (uint32_t q = 0; q < 4; ++q) {
                            if (leader) {
                                umma_i8(tmem_base + r * MAX_BN, da + 2 * q, db + 2 * q, idesc, (kb | q) != 0 ? 1u : 0u);
                            }
                        }
                    }
                    if (leader) {
                        tcgen05_commit(&ctl->done[s]);
                    }
                    __syncwarp();
                }
            }
        }
        __syncwarp();
    } else {
        // ------------------------------- widening and epilogue ------------------------------------
        const uint32_t npix = p.N * p.OH * p.OW;
        const uint32_t plane = p.Hp * p.Wp;
        const uint32_t word = threadIdx.x & 3, row0 = threadIdx.x >> 2;
        const uint32_t a_rows = 2 * p.row_blocks;   // rows of 64 this thread serves
        uint32_t issued = 0, staged_n0 = 0xFFFFFFFFu;
        for (uint32_t tile = blockIdx.x; tile < tiles; tile += gridDim.x) {
            const uint32_t m0 = (tile % p.tiles_m) * p.row_blocks * BLOCK_M, n0 = (tile / p.tiles_m) * p.block_n;
            if (n0 != staged_n0) {
                // constants of the tile's channels (the previous tile's epilogue is over: it ended with a barrier)
                if (threadIdx.x < p.block_n) {
                    const uint32_t o = threadIdx.x;
                    const bool in = n0 + o < p.OC;
                    reinterpret_cast<__half *>(ctl->scale)[o] = in ? p.scale[n0 + o] : __half(0.f);
                    reinterpret_cast<__half *>(ctl->bias)[o] = in ? p.bias[n0 + o] : __half(0.f);
                }
                staged_n0 = n0;
            }
            // first word of this thread's pixels (tap 0, word 0) and weights.  Rows that do not exist read some other
            // words: their accumulators are never stored.
            const uint32_t *xp[4], *wp[2];
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const uint32_t pix = m0 + row0 + 64 * i;
                xp[i] = p.xb;
                if ((uint32_t)i < a_rows && pix < npix) {
                    const uint32_t ow = pix % p.OW, t = pix / p.OW, oh = t % p.OH, n = t / p.OH;
                    xp[i] += (n * p.Cw * p.Hp + oh * p.sH) * p.Wp + ow * p.sW;
                }
            }
#pragma unroll
            for (int i = 0; i < 2; ++i) {
                const uint32_t o = row0 + 64 * i;
                wp[i] = p.wb + ((o < p.block_n && n0 + o < p.OC) ? (n0 + o) * p.kw_words : 0u);
            }
            // this thread's word of K block kb is k = 4 kb + word = (kh, kw, cw)
            uint32_t k = word, cw = word % p.Cw, tap = word / p.Cw, kw = tap % p.FW, kh = tap / p.FW;
            int ones[2] = {0, 0};   // set bits of this thread's words of its two channels
            // The words of a K block.  Two sets: a block's words are asked for two blocks ahead, and nothing looks at them
            // before they are widened.
            struct Words {
                uint32_t x[4], w[2];
                Widen m;          // of the weights: zeros beyond K (there the activations are any words)
            };
            auto fetch = [&](Words &f) {
                const bool valid = k < p.kw_words;
                const uint32_t off = valid ? cw * plane + kh * p.Wp + kw : 0u, wk = valid ? k : 0u;
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    f.x[i] = __ldg(xp[i] + off);
                }
#pragma unroll
                for (int i = 0; i < 2; ++i) {
                    f.w[i] = __ldg(wp[i] + wk);
                }
                f.m.mul = valid ? (XNOR ? (uint32_t)-254 : 1u) : 0u;
                f.m.add = valid && XNOR ? 0xFFFFFFFFu : 0u;
                k += 4;
                cw += 4;
                while (cw >= p.Cw) {
                    cw -= p.Cw;
                    if (++kw == p.FW) {
                        kw = 0;
                        ++kh;
                    }
                }
            };
            auto block = [&](Words &f) {
                const uint32_t s = issued & 1;
                uint8_t *sa = smem + s * STAGE, *sb = sa + STAGE_A;
                if (!dead && issued >= 2 && !mbar_wait(&ctl->done[s], ((issued >> 1) + 1) & 1)) {
                    dead = true;
                }
                dead = __any_sync(0xffffffffu, dead);
                ++issued;
                if (dead) {
                    return;   // keeps meeting the barriers below without touching anything
                }
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    if ((uint32_t)i < a_rows) {
                        store_word<true>(sa, row0 + 64 * i, word, f.x[i], f.m);
                    }
                }
#pragma unroll
                for (int i = 0; i < 2; ++i) {
                    if (row0 + 64 * i < p.block_n) {
                        store_word<false>(sb, row0 + 64 * i, word, f.w[i], f.m);
                        if (XNOR) {
                            ones[i] += f.m.mul != 0 ? __popc(f.w[i]) : 0;
                        }
                    }
                }
                fence_proxy_async_smem();
                __syncwarp();
                if (lane == 0) {
                    mbar_arrive(&ctl->full[s]);
                }
                fetch(f);
            };
            Words f0, f1;
            fetch(f0);
            fetch(f1);
            for (uint32_t kb = 0; kb < num_kb; kb += 2) {
                block(f0);
                if (kb + 1 < num_kb) {
                    block(f1);
                }
            }
            if (XNOR) {
                // four neighbouring lanes hold a channel's words
#pragma unroll
                for (int i = 0; i < 2; ++i) {
                    int t = ones[i] + __shfl_xor_sync(0xffffffffu, ones[i], 1);
                    t += __shfl_xor_sync(0xffffffffu, t, 2);
                    if (word == 0 && row0 + 64 * i < p.block_n) {
                        ctl->corr[row0 + 64 * i] = (int)p.kbits - 2 * t;
                    }
                }
            }
            if (!dead) {
                const uint32_t last = issued - 1;
                dead = !mbar_wait(&ctl->done[last & 1], (last >> 1) & 1);
            }
            dead = __any_sync(0xffffffffu, dead);
            asm volatile("bar.sync 1, %0;" ::"n"(WIDEN_THREADS) : "memory");   // the constants are there
            if (!dead) {
                tcgen05_fence_after();
                // int16 sum -> fp16 (round to nearest even), one fused multiply-add, 8 channels = 16 bytes; a lane is a
                // pixel, so 32 lanes write 512 contiguous bytes.  Warp = lane quadrant x (row block, or half of the channels).
                const uint32_t quad = warp & 3, half = warp >> 2, nch = p.block_n >> 5;
                const uint32_t r = p.row_blocks == 2 ? half : 0u;
                const uint32_t c_begin = p.row_blocks == 2 ? 0u : (half ? (nch + 1) / 2 : 0u);
                const uint32_t c_end = p.row_blocks == 2 ? nch : (half ? nch : (nch + 1) / 2);
                const uint32_t pix = m0 + r * BLOCK_M + quad * 32 + lane;
                const uint32_t n = pix / (p.OH * p.OW);
                const size_t oplane = (size_t)p.OH * p.OW;
                __half *dst = p.out + (size_t)n * p.OC * oplane + (size_t)(pix - n * (uint32_t)oplane) * 8;
                for (uint32_t c = c_begin; c < c_end; ++c) {
                    uint32_t acc[32];
                    tmem_ld32(tmem_base + ((quad * 32u) << 16) + r * MAX_BN + c * 32, acc);
                    tmem_ld_wait(acc);
                    if (pix < npix) {
#pragma unroll
                        for (int ob = 0; ob < 32; ob += 8) {
                            const uint32_t oc = n0 + c * 32 + ob;
                            if (oc < p.OC) {
                                uint32_t h[4];
#pragma unroll
                                for (int j = 0; j < 8; j += 2) {
                                    const uint32_t o = c * 32 + ob + j;
                                    int s0 = (int)acc[ob + j], s1 = (int)acc[ob + j + 1];
                                    if (XNOR) {
                                        const int2 co = *reinterpret_cast<const int2 *>(ctl->corr + o);
                                        s0 = 2 * s0 + co.x;
                                        s1 = 2 * s1 + co.y;
                                    }
                                    // int16 -> fp16 by way of binary32, which holds every int16 exactly
                                    const __half2 hs = __floats2half2_rn((float)(short)s0, (float)(short)s1);
                                    const __half2 v = __hfma2(hs, ctl->scale[o >> 1], ctl->bias[o >> 1]);
                                    h[j >> 1] = *reinterpret_cast<const uint32_t *>(&v);
                                }
                                *reinterpret_cast<uint4 *>(dst + (size_t)oc * oplane) = make_uint4(h[0], h[1], h[2], h[3]);
                            }
                        }
                    }
                }
                tcgen05_fence_before();
                __syncwarp();
                if (lane == 0) {
                    mbar_arrive(&ctl->drained);
                }
            }
            asm volatile("bar.sync 1, %0;" ::"n"(WIDEN_THREADS) : "memory");   // the constants have been read
        }
    }
    if (dead && lane == 0) {
        atomicExch(p.status, 41);
    }
    tcgen05_fence_before();
    __syncthreads();
    if (warp == 0) {
        tcgen05_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(p.tmem_cols) : "memory");
    }
}

// Tile: 256 pixels x 128 channels where that leaves every SM its two CTAs; with fewer tiles than that, one row block
// of 128 pixels and then narrower channel blocks.
void pick_tile(uint64_t npix, uint32_t OC, int sms, BnnParams *p)
{
    const uint32_t blocks = (OC + MAX_BN - 1) / MAX_BN;
    uint32_t bn = (uint32_t)B200_ALIGN((OC + blocks - 1) / blocks, 32), rb = 2;
    auto tiles = [&] { return ((npix + rb * BLOCK_M - 1) / (rb * BLOCK_M)) * ((OC + bn - 1) / bn); };
    if (tiles() < 2 * (uint64_t)sms) {
        rb = 1;
    }
    while (bn > 32 && tiles() < (uint64_t)sms) {
        bn -= 32;
    }
    p->row_blocks = rb;
    p->block_n = bn;
    p->tiles_m = (uint32_t)((npix + rb * BLOCK_M - 1) / (rb * BLOCK_M));
    p->tiles_n = (OC + bn - 1) / bn;
    p->tmem_cols = rb == 2 ? 256u : (bn > 64 ? 128u : bn);
}

struct BnnGeom {
    B4d in, f, out;
    uint32_t sH, sW, pt, pb, pl, pr, Hp, Wp, Cw, taps;
    size_t xb_bytes;
};

EE bnn_geometry(const TensorDesc *inputDesc, const TensorDesc *filterDesc, const TensorDesc *outputDesc,
    const ConvolutionParamSpec *cp, BnnGeom *g)
{
    if (!get4(inputDesc, &g->in) || !get4(filterDesc, &g->f) || !get4(outputDesc, &g->out) || cp == nullptr) {
        return NOT_MATCH;
    }
    if (cp->group > 1 || cp->dilatedRate_h > 1 || cp->dilatedRate_w > 1) {
        return NOT_SUPPORTED;
    }
    g->sH = cp->stride_h ? cp->stride_h : 1;
    g->sW = cp->stride_w ? cp->stride_w : 1;
    g->pt = cp->pad_top;
    g->pb = cp->pad_bottom;
    g->pl = cp->pad_left;
    g->pr = cp->pad_right;
    g->Hp = g->in.h + g->pt + g->pb;
    g->Wp = g->in.w + g->pl + g->pr;
    g->Cw = (g->f.c + 31) / 32;
    g->taps = g->f.h * g->f.w;
    g->xb_bytes = (size_t)g->in.n * g->Hp * g->Wp * g->Cw * 4;
    // the output geometry must be the one the input, filter and padding give: the kernel reads the padded
    // bit tensor at (oh * stride + kh, ow * stride + kw) without further checks
    if (g->f.h == 0 || g->f.w == 0 || g->Hp < g->f.h || g->Wp < g->f.w || g->out.n != g->in.n ||
        g->out.h != (g->Hp - g->f.h) / g->sH + 1 || g->out.w != (g->Wp - g->f.w) / g->sW + 1) {
        return NOT_MATCH;
    }
    return SUCCESS;
}

}  // namespace

EE bnn_transform_filter_bytes(const TensorDesc *filterDesc, U32 *bytes)
{
    B4d f;
    if (!get4(filterDesc, &f) || bytes == nullptr) {
        return NOT_MATCH;
    }
    *bytes = f.n * f.h * f.w * ((f.c + 31) / 32) * 4 + 32;
    return SUCCESS;
}

EE bnn_transform_filter(const TensorDesc *filterDesc, const void *filter, TensorDesc *ftmDesc, void *dst)
{
    B4d f;
    if (!get4(filterDesc, &f) || ftmDesc == nullptr) {
        return NOT_MATCH;
    }
    if (f.df == DF_NCHWN16C8) {
        *ftmDesc = *filterDesc;  // already transformed (convolution_transform_bnn.h:47-50)
        return SUCCESS;
    }
    if (f.df != DF_NCHW) {
        return NOT_MATCH;
    }
    if (filter == nullptr || dst == nullptr) {
        return NULL_POINTER;
    }
    DeviceCtx *c = ctx();
    if (c == nullptr) {
        return UNKNOWN;
    }
    cudaStream_t st = tls().stream;
    const uint32_t Cw = (f.c + 31) / 32, taps = f.h * f.w;
    const size_t words = (size_t)f.n * taps * Cw;
    Stage sg;
    const uint8_t *d_src = reinterpret_cast<const uint8_t *>(sg.in(filter, ((size_t)f.n * f.c * taps + 7) / 8));
    uint32_t *d_dst = reinterpret_cast<uint32_t *>(sg.out(dst, words * 4));
    if (d_src == nullptr || d_dst == nullptr) {
        return ALLOC_FAILED;
    }
    bnn_pack_filter_kernel<<<(uint32_t)((words + 255) / 256), 256, 0, st>>>(d_src, f.n, f.c, taps, Cw, d_dst);
    count_launch();
    B200_CUDA(cudaGetLastError());
    *ftmDesc = *filterDesc;
    ftmDesc->df = DF_NCHWN16C8;
    return sg.finish();
}

EE bnn_tmp_bytes(const TensorDesc *inputDesc, const TensorDesc *filterDesc, const TensorDesc *outputDesc,
    const ConvolutionParamSpec *cp, U32 *bytes)
{
    if (bytes == nullptr) {
        return NULL_POINTER;
    }
    BnnGeom g;
    B200_EE(bnn_geometry(inputDesc, filterDesc, outputDesc, cp, &g));
    const size_t b = g.xb_bytes + 512;
    if (b > 0xFFFFFFFFull) {
        return NOT_SUPPORTED;
    }
    *bytes = (U32)b;
    return SUCCESS;
}

EE bnn_run(const TensorDesc *inputDesc, const void *input, const TensorDesc *filterDesc, const void *filter,
    const ConvolutionParamSpec *cp, const void *scale, const void *bias, U32 tmpBytes, void *tmp,
    const TensorDesc *outputDesc, void *output)
{
    BnnGeom g;
    B200_EE(bnn_geometry(inputDesc, filterDesc, outputDesc, cp, &g));
    if (input == nullptr || filter == nullptr || output == nullptr || scale == nullptr || bias == nullptr ||
        tmp == nullptr) {
        return NULL_POINTER;  // cpu/arm/bnn/convolution.cpp:32-35
    }
    if (g.in.dt != DT_F16 || g.out.dt != DT_F16) {
        return NOT_MATCH;  // :46-51
    }
    if (g.in.df != DF_NCHWC8 || g.out.df != DF_NCHWC8 || g.f.df != DF_NCHWN16C8) {
        return NOT_MATCH;  // :52-54, convolution_xnor_A76.cpp:53-55
    }
    if (g.in.c != g.f.c || g.out.c != g.f.n || (g.in.c % 8) != 0 || (g.out.c % 8) != 0) {
        return NOT_MATCH;
    }
    U32 need = 0;
    B200_EE(bnn_tmp_bytes(inputDesc, filterDesc, outputDesc, cp, &need));
    if (tmpBytes < need) {
        return NOT_MATCH;
    }
    const size_t in_elems = (size_t)g.in.n * g.in.c * g.in.h * g.in.w;
    const size_t out_elems = (size_t)g.out.n * g.out.c * g.out.h * g.out.w;
    if (in_elems == 0 || out_elems == 0) {
        return NOT_SUPPORTED;  // pick_tile divides by the channel blocks, and the kernel's walk over K by the words of a tap
    }
    DeviceCtx *c = ctx();
    if (c == nullptr) {
        return UNKNOWN;
    }
    cudaStream_t st = tls().stream;
    const bool xnor = g.f.dt == DT_BIN11;
    const size_t w_words = (size_t)g.f.n * g.taps * g.Cw;
    Stage sg;
    const __half *d_in = reinterpret_cast<const __half *>(sg.in(input, in_elems * 2));
    const uint32_t *d_w = reinterpret_cast<const uint32_t *>(sg.in(filter, w_words * 4));
    const __half *d_scale = reinterpret_cast<const __half *>(sg.in(scale, (size_t)g.out.c * 2));
    const __half *d_bias = reinterpret_cast<const __half *>(sg.in(bias, (size_t)g.out.c * 2));
    __half *d_out = reinterpret_cast<__half *>(sg.out(output, out_elems * 2));
    char *d_tmp = is_device_ptr(tmp) ? reinterpret_cast<char *>(tmp) : reinterpret_cast<char *>(sg.scratch(need));
    if (d_in == nullptr || d_w == nullptr || d_scale == nullptr || d_bias == nullptr || d_out == nullptr ||
        d_tmp == nullptr) {
        return ALLOC_FAILED;
    }
    const size_t npix = (size_t)g.out.n * g.out.h * g.out.w;
    if (((g.taps * g.Cw + 3) & ~3u) > MAX_WORDS) {
        return NOT_SUPPORTED;
    }
    uint32_t *d_xb = reinterpret_cast<uint32_t *>(B200_ALIGN(reinterpret_cast<uintptr_t>(d_tmp), 256));
    {
        const size_t words = g.xb_bytes / 4;
        size_t blocks = (words + 255) / 256;
        if (blocks > (size_t)c->sm_count * 64) {   // (16 made one round and a half of the 28 x 28 x 256 batch)
            blocks = (size_t)c->sm_count * 64;
        }
        bnn_binarize_pad_kernel<<<(uint32_t)blocks, 256, 0, st>>>(d_in, g.in.n, g.in.c, g.in.h, g.in.w, g.Hp, g.Wp, g.pt,
            g.pl, g.Cw, xnor ? 0.0f : 0.5f, d_xb);
        count_launch();
    }
    BnnParams p;
    p.N = g.in.n;
    p.OH = g.out.h;
    p.OW = g.out.w;
    p.OC = g.out.c;
    p.Hp = g.Hp;
    p.Wp = g.Wp;
    p.Cw = g.Cw;
    p.FH = g.f.h;
    p.FW = g.f.w;
    p.sH = g.sH;
    p.sW = g.sW;
    p.kbits = g.f.h * g.f.w * g.f.c;
    p.kw_words = g.taps * g.Cw;
    p.xb = d_xb;
    p.wb = d_w;
    p.scale = d_scale;
    p.bias = d_bias;
    p.out = d_out;
    p.status = c->d_status;
    pick_tile(npix, p.OC, c->sm_count, &p);
    {
        const void *ks[2] = {(const void *)bnn_conv_kernel<true>, (const void *)bnn_conv_kernel<false>};
        B200_EE(raise_smem_limit(c, KF_BNN, ks, 2, BNN_SMEM));
    }
    const uint64_t tiles = (uint64_t)p.tiles_m * p.tiles_n;
    const uint32_t grid = (uint32_t)(tiles < 2 * (uint64_t)c->sm_count ? tiles : 2 * (uint64_t)c->sm_count);
    if (xnor) {
        bnn_conv_kernel<true><<<grid, THREADS, BNN_SMEM, st>>>(p);
    } else {
        bnn_conv_kernel<false><<<grid, THREADS, BNN_SMEM, st>>>(p);
    }
    count_launch();
    B200_CUDA(cudaGetLastError());
    return sg.finish();
}

}  // namespace b200
