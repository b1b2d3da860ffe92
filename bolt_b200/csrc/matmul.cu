// matmul.cu -- the int8 branch of Bolt's `matmul` operator (compute/tensor/src/matmul.cpp:303-557) for
// CUDA_B200: both operands may arrive as fp32 and are quantized per call (dynamic scale 127 / absmax, or the
// scale the tensor carries), and the result is written as fp32 (accumulator / (scaleA * scaleB)) or requantized
// to u8.  All products of a call run in one launch that quantizes its operands while it loads them
// (launch_matmul_batch); where that is slower (few tiles and a long K, large products), for a result of one column and for
// one that lies over its operands, the quantize / pack / multiply kernels run one after the other.
//
// The x86 convention applies (matmul.cpp:373-398): u8 activations with zero point 128 times s8, except
// when the result is a vector, where A becomes s8 and B u8.  Leading (batch) dimensions broadcast as in
// matmul.cpp:489-517.  All work is enqueued on the thread's stream; the scale of a dynamically requantized u8 result
// comes back to the host, which is what the operator's interface (Tensor::get_scale) requires.
#include <algorithm>
#include <cmath>

#include "common.cuh"

namespace b200 {
namespace {

inline size_t bytes_of(DataType dt)
{
    return (dt == DT_F32 || dt == DT_I32 || dt == DT_U32 || dt == DT_F32_8Q) ? 4 : (dt == DT_F16 ? 2 : 1);
}
inline uint64_t elems(const TensorDesc &d)
{
    uint64_t n = d.nDims ? 1 : 0;
    for (U32 i = 0; i < d.nDims; ++i) {
        n *= d.dims[i];
    }
    return n;
}
inline bool use_int8(DataType a, DataType b, DataType c, F32 cScale)
{
    // matmul.cpp:205-209; the scale is read through an I32 parameter, so |scale| < 1 does not count
    return a == DT_I8 || b == DT_I8 || a == DT_U8_Q || b == DT_U8_Q || c == DT_U8_Q || c == DT_I8 || (I32)cScale != 0;
}
void align_descs(TensorDesc *a, TensorDesc *b)
{
    while (a->nDims < b->nDims) {
        a->dims[a->nDims++] = 1;
    }
    while (b->nDims < a->nDims) {
        b->dims[b->nDims++] = 1;
    }
}
TensorDesc desc2d(DataType dt, DataFormat df, U32 rows, U32 cols)
{
    TensorDesc d;
    d.dt = dt;
    d.df = df;
    d.nDims = 2;
    d.dims[0] = cols;
    d.dims[1] = rows;
    return d;
}
TensorDesc desc1d(DataType dt, U32 len)
{
    TensorDesc d;
    d.dt = dt;
    d.df = DF_NORMAL;
    d.nDims = 1;
    d.dims[0] = len;
    return d;
}

// what the operator decides before touching data
struct Plan {
    TensorDesc a, b, c;          // a and b aligned to the same rank; c as the caller gave it
    bool is_mvm;
    DataType qa, qb, qc;         // operand types of the product, type the product writes
    bool quantA, quantB, stageC;
    bool static_u8;              // u8 output requantized inside the product with the caller's scale
    U32 kDimA, kDimB;
    DataFormat dfA, dfB;
    U32 mmm_bytes;
    uint64_t loopsA, loopsB, loopsC;
};

EE inner_tmp_bytes(const Plan &p, U32 *bytes)
{
    // matmul.cpp:211-243
    const TensorDesc &A = p.a, &B = p.b;
    if (A.dims[1 - p.kDimA] == 1) {
        return b200_matrix_vector_multiply_tmp_bytes(
            desc2d(p.qb, p.dfB == DF_TRANSPOSE ? DF_NORMAL : DF_TRANSPOSE, B.dims[1], B.dims[0]),
            desc1d(p.qa, A.dims[p.kDimA]), bytes, CUDA_B200);
    }
    if (B.dims[1 - p.kDimB] == 1) {
        return b200_matrix_vector_multiply_tmp_bytes(
            desc2d(p.qa, p.dfA, A.dims[1], A.dims[0]), desc1d(p.qb, B.dims[p.kDimB]), bytes, CUDA_B200);
    }
    return b200_matrix_matrix_multiply_tmp_bytes(
        desc2d(p.qa, p.dfA, A.dims[1], A.dims[0]), desc2d(p.qb, p.dfB, B.dims[1], B.dims[0]), bytes, CUDA_B200);
}

EE make_plan(const TensorDesc *aDesc, int tA, const TensorDesc *bDesc, int tB, const TensorDesc *cDesc, F32 cScale, Plan *p)
{
    if (aDesc == nullptr || bDesc == nullptr || cDesc == nullptr) {
        return NULL_POINTER;
    }
    p->a = *aDesc;
    p->b = *bDesc;
    p->c = *cDesc;
    if (p->a.nDims < 1 || p->b.nDims < 2 || p->a.nDims > 6 || p->b.nDims > 6 || p->c.nDims > 6) {
        return NOT_SUPPORTED;
    }
    if (!use_int8(p->a.dt, p->b.dt, p->c.dt, cScale)) {
        return NOT_SUPPORTED;  // the floating-point matmul is not part of this library
    }
    if (p->c.dt != DT_F32 && p->c.dt != DT_U8_Q) {
        return NOT_SUPPORTED;
    }
    if (p->a.nDims == 1) {  // matmul.cpp:360-365
        p->a.nDims = 2;
        p->a.dims[1] = 1;
        p->c.nDims = 2;
        p->c.dims[1] = 1;
    }
    p->is_mvm = (p->c.dims[0] == 1) || (p->c.dims[1] == 1);
    p->qa = p->is_mvm ? DT_I8 : DT_U8_Q;
    p->qb = p->is_mvm ? DT_U8_Q : DT_I8;
    p->qc = DT_F32;
    p->static_u8 = false;
    if (p->c.dt == DT_U8_Q && cScale > 0) {
        p->qc = DT_U8_Q;
        p->static_u8 = true;
    }
    p->quantA = p->a.dt != p->qa;
    p->quantB = p->b.dt != p->qb;
    p->stageC = p->c.dt != p->qc;
    // an operand is either fp32 (quantized here) or already of the type the product wants
    if ((p->quantA && p->a.dt != DT_F32) || (p->quantB && p->b.dt != DT_F32)) {
        return NOT_SUPPORTED;
    }
    p->kDimA = tA ? 1 : 0;
    p->dfA = tA ? DF_TRANSPOSE : DF_NORMAL;
    p->kDimB = tB ? 0 : 1;
    p->dfB = tB ? DF_TRANSPOSE : DF_NORMAL;
    align_descs(&p->a, &p->b);
    if (p->a.dims[p->kDimA] != p->b.dims[p->kDimB]) {
        return NOT_MATCH;
    }
    if (p->c.dims[0] != p->b.dims[1 - p->kDimB] || p->c.dims[1] != p->a.dims[1 - p->kDimA]) {
        return NOT_MATCH;
    }
    const uint64_t a2 = (uint64_t)p->a.dims[0] * p->a.dims[1], b2 = (uint64_t)p->b.dims[0] * p->b.dims[1];
    const uint64_t c2 = (uint64_t)p->c.dims[0] * p->c.dims[1];
    if (a2 == 0 || b2 == 0 || c2 == 0) {
        return NOT_MATCH;
    }
    p->loopsA = elems(p->a) / a2;
    p->loopsB = elems(p->b) / b2;
    p->loopsC = elems(p->c) / c2;
    return inner_tmp_bytes(*p, &p->mmm_bytes);
}

__global__ void fill_rows_kernel(uint8_t *dst, uint64_t total, const uint8_t *row, uint32_t row_bytes)
{
    // dst = the bias bytes repeated (matmul.cpp:457-466); a zero fill when row == nullptr
    for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += (uint64_t)gridDim.x * blockDim.x) {
        dst[i] = row ? row[i % row_bytes] : (uint8_t)0;
    }
}

U32 global_index(uint64_t ic, const TensorDesc &c, const TensorDesc &x)
{
    // matmul.cpp:494-517: the batch coordinates of C, each folded to 0 where the operand's extent is smaller
    U32 idx[8];
    for (U32 i = 2; i < c.nDims; ++i) {
        idx[i] = (U32)(ic % c.dims[i]);
        ic /= c.dims[i];
    }
    U32 g = 0;
    for (int i = (int)x.nDims - 1; i >= 2; --i) {
        U32 v = (U32)i < c.nDims ? idx[i] : 0;
        if (v >= x.dims[i]) {
            v = 0;
        }
        g = g * x.dims[i] + v;
    }
    return g;
}

// One launch for all products, or one product after the other through quantize, pack and the TMA GEMM (GEMV)?  The batched
// kernels never pack and keep the host out of it, but they convert an fp32 operand again for every tile row / column of
// the other one, fill the tensor pipe a quarter as well, and one CTA walks all of a tile's K.  So the two are estimated,
// in us; the constants are fitted to the figures behind, us per call, one launch against one by one:
//   fp32 in and out: 128 x 128 with K = 512 22 / 38, 1024 37 / 39, 2048 66 / 43, 16384 466 / 101; 1024 x 1024 with K = 256
//   18 / 39, 1024 68 / 43; 4 x (128 x 128) with K = 4096 123 / 131, 8192 240 / 189; 12 x (16 x 64) with K = 16384
//   449 / 648; 4 x 1024^3 86 / 89; 384 x (128 x 64 x 128 and 128 x 128 x 64) 47 / 8000 for the pair
//   u8 x s8: 128 x 128 with K = 1024 12 / 14, 2048 19 / 14, 65536 427 / 214; 16 x 16384 with K = 4096 39 / 72; 1024^3
//   14 / 16; 4 x (256 x 256) with K = 16384 115 / 241
//   K off the 16-byte grid, or A stored [K][M]: fp32 136 x 36 x 25084 719 / 363, 3 x (12 x 7 x 5708) 156 / 274, [K][M]
//   87 x 9 x 20897 735 / 1047; fp32 x s8, [K][M] 2 x (1860 x 4 x 7664) 381 / 272
//   a row, matrix stored [N][K]: fp32 768 x 768 14 / 32, 768 x 3072 63 / 38, 1024 x 16384 340 / 70, 4 x (2048 x 2048)
//   57 / 68; u8 1024 x 1024 12 / 9, 8192 x 8192 68 / 21, 2 x (1024 x 1024) 12 / 13, 96 x (2048 x 64) 25 / 396
//   a row, matrix stored [K][N]: one launch is faster throughout (1 x 65536 x 64 8 / 10 ... 96 x 64 x 2048 18 / 5318)
// Over 504 random shapes, types and storage orders it takes the faster way within 10 % in all but seven (at worst 1.8 times:
// fp32, [K][M] 3 x (1796 x 12 x 12753) 1106 / 609).
// Products of more than 2^30 multiply-adds always go one by one (1 x 2048^3 209 / 112, 4 x 2048^3 903 / 272).
struct Product {
    double M, N, K, batches, elems;   // elems: of the fp32 operands
    bool f32_a, f32_b, a_cols, b_rows;   // a_cols: A is stored [K][M]; b_rows: B [N][K]
    bool tma;                            // TMA can fetch the (quantized) A
};
bool one_launch_is_faster(const Product &q, int sms)
{
    const double quantize = 12.0 * (q.f32_a + q.f32_b);   // two launches and a wait of the host
    if (q.M == 1) {
        if (!q.b_rows) {
            return true;
        }
        // 32 rows per block, eight blocks per SM: a warp's loads one behind the other, each a latency (twice that for an fp32
        // matrix of more than 8 MB; bytes off the 8-byte grid are read one at a time)
        const double rounds = std::ceil(std::ceil(q.N / 32) * q.batches / (8.0 * sms));
        const double loads = std::ceil(std::min(q.N, 32.0) / 8) * std::ceil(q.K / 128);
        const double load = q.f32_b ? (q.N * q.K * q.batches > (double)(2 << 20) ? 0.58 : 0.27) : ((uint64_t)q.K % 8 == 0 ? 0.235 : 0.45);
        const double batched = 5 + 1.5 * (q.f32_a + q.f32_b) + rounds * loads * load + 0.8e-6 * q.elems;
        const double row = ((uint64_t)q.K % 16 == 0 ? 0.9e-3 : 1.8e-3) * q.K;
        const double singly = 9 + quantize + 4.3 * (q.batches - 1) + q.batches * row + 1.5e-6 * q.elems;
        return batched <= singly;
    }
    if (q.M * q.N * q.K > (double)(1ull << 30)) {
        return false;
    }
    // K blocks of 128 bytes; the tiles of launch_matmul_batch
    const double kb = std::ceil(q.K / 128), tiles_m = q.batches * std::ceil(q.M / 128);
    const double bn = gather_block_n((uint64_t)tiles_m, (uint32_t)q.N, sms), tiles = tiles_m * std::ceil(q.N / bn);
    const bool f32 = q.f32_a || q.f32_b;   // (binary32 keeps an SM busy; bytes are fetched ahead, and CTAs share the SM)
    const double rounds = f32 ? std::ceil(tiles / sms) : std::max(1.0, tiles / (2.5 * sms));
    // (bytes stored across K in rows off the 4-byte grid are loaded one at a time)
    const double block_a = q.f32_a ? (q.a_cols ? 4.0 : 2.4) : (q.a_cols && (uint64_t)q.M % 4 != 0 ? 3.0 : 0.0);
    const double block_b = q.f32_b ? 0.4 * (bn / 32) : (!q.b_rows && (uint64_t)q.N % 4 != 0 ? 3.0 : 0.0);
    const double batched = (f32 ? 8 : 5.5) + rounds * kb * (0.83 + block_a + block_b) + 0.8e-6 * q.elems;
    // Singly, B is packed and C is cleared, read and written; a K block costs 0.4 where TMA can fetch A, else its bytes are
    // gathered, one by one from unaligned columns.
    const double block = q.tma ? 0.4 : (q.a_cols && (uint64_t)q.M % 4 != 0 ? 6.2 : 1.8);
    const double singly = std::max(14.0, 8 + block * kb) + quantize + (q.batches - 1) * std::max(10.0, 6 + block * kb) + 1.5e-6 * q.elems +
        (0.6e-6 * q.K + 2.4e-6 * q.M) * q.N * q.batches;
    return batched <= singly;
}
bool one_launch(const Plan &p, const void *A, int sms, cudaStream_t st)
{
    Product q;
    q.M = p.a.dims[1 - p.kDimA];
    q.N = p.b.dims[1 - p.kDimB];
    q.K = p.a.dims[p.kDimA];
    q.batches = (double)p.loopsC;
    q.f32_a = p.quantA;
    q.f32_b = p.quantB;
    q.elems = (p.quantA ? (double)elems(p.a) : 0) + (p.quantB ? (double)elems(p.b) : 0);
    q.a_cols = p.dfA == DF_TRANSPOSE;
    q.b_rows = p.dfB == DF_TRANSPOSE;
    q.tma = !q.a_cols && p.a.dims[p.kDimA] % 16 == 0 && (p.quantA || reinterpret_cast<uintptr_t>(A) % 16 == 0);
    if (q.M != 1 && q.N == 1) {
        return false;   // a result of one column has no batched kernel
    }
    if (one_launch_is_faster(q, sms)) {
        return true;
    }
    // The scales of separately quantized operands have to reach the host, which a stream that is being captured cannot wait
    // for: there the batched kernels take what they can.
    return (p.quantA || p.quantB) && (q.M == 1 || q.M * q.N * q.K <= (double)(1ull << 30)) && capturing(st);
}

bool overlap(const void *a, size_t na, const void *b, size_t nb)
{
    const uintptr_t x = reinterpret_cast<uintptr_t>(a), y = reinterpret_cast<uintptr_t>(b);
    return x < y + nb && y < x + na;
}

// the scratch of the batched kernel: an operand's partial maxima lie where its quantized copy would
MatmulOperand batch_operand(const void *data, const TensorDesc &d, bool f32, int transposed, F32 scale, uint64_t loops, uint64_t loopsC, char *scratch)
{
    MatmulOperand o;
    o.p = data;
    o.elems = elems(d);
    o.f32 = f32 ? 1 : 0;
    o.transposed = transposed;
    o.scale = scale;
    for (U32 i = 0; i < 4; ++i) {
        o.dims[i] = i + 2 < d.nDims ? d.dims[i + 2] : 1;
    }
    o.direct = loops == loopsC;
    o.slots = reinterpret_cast<unsigned *>(scratch);
    o.max_slots = B200_ALIGN(o.elems, 256) / 4;
    return o;
}

}  // namespace
}  // namespace b200

using namespace b200;

extern "C" {

// matmul.cpp:42-99
EE matmul_infer_output_size_cuda_b200(const TensorDesc *aDesc, int transposeA, const TensorDesc *bDesc, int transposeB,
    TensorDesc *cDesc)
{
    if (aDesc == nullptr || bDesc == nullptr || cDesc == nullptr) {
        return NULL_POINTER;
    }
    TensorDesc a = *aDesc, b = *bDesc;
    if (a.nDims < 2 || b.nDims < 2 || a.nDims > 6 || b.nDims > 6) {
        return NOT_SUPPORTED;
    }
    if (transposeA) {
        std::swap(a.dims[0], a.dims[1]);
    }
    if (transposeB) {
        std::swap(b.dims[0], b.dims[1]);
    }
    if (a.dims[0] != b.dims[1]) {
        return NOT_MATCH;
    }
    align_descs(&a, &b);
    *cDesc = a;
    cDesc->dims[0] = b.dims[0];
    for (U32 i = 2; i < a.nDims; ++i) {
        const U32 x = a.dims[i], y = b.dims[i];
        if (x != y && x != 1 && y != 1) {
            return NOT_MATCH;
        }
        cDesc->dims[i] = x > y ? x : y;
    }
    return SUCCESS;
}

// matmul.cpp:245-301
EE matmul_infer_forward_tmp_bytes_cuda_b200(const TensorDesc *aDesc, int transposeA, const TensorDesc *bDesc,
    int transposeB, const TensorDesc *cDesc, F32 cScale, U32 *bytes)
{
    if (bytes == nullptr) {
        return NULL_POINTER;
    }
    Plan p;
    B200_EE(make_plan(aDesc, transposeA, bDesc, transposeB, cDesc, cScale, &p));
    uint64_t total = B200_ALIGN((uint64_t)p.mmm_bytes, 256) + 1024;
    if (p.quantA) {
        total += B200_ALIGN(elems(p.a), 256);
    }
    if (p.quantB) {
        total += B200_ALIGN(elems(p.b), 256);
    }
    if (p.stageC) {
        total += B200_ALIGN(elems(p.c) * 4, 256);
    }
    if (total > 0xffffffffull) {
        return NOT_SUPPORTED;
    }
    *bytes = (U32)total;
    return SUCCESS;
}

EE matmul_cuda_b200(const TensorDesc *aDesc, int transposeA, const void *A, F32 aScale, const TensorDesc *bDesc,
    int transposeB, const void *B, F32 bScale, const TensorDesc *biasDesc, const void *bias, U32 tmpBytes, void *tmp,
    const TensorDesc *cDesc, void *C, F32 *cScale)
{
    if (A == nullptr || B == nullptr || C == nullptr || cScale == nullptr) {
        return NULL_POINTER;
    }
    DeviceCtx *c = ctx();
    if (c == nullptr) {
        return UNKNOWN;
    }
    Plan p;
    B200_EE(make_plan(aDesc, transposeA, bDesc, transposeB, cDesc, *cScale, &p));
    U32 need = 0;
    B200_EE(matmul_infer_forward_tmp_bytes_cuda_b200(aDesc, transposeA, bDesc, transposeB, cDesc, *cScale, &need));
    if (tmp == nullptr || tmpBytes < need) {
        return NOT_MATCH;
    }
    if (p.loopsC == 0) {
        return SUCCESS;  // an empty batch
    }
    if (p.loopsA == 0 || p.loopsB == 0) {
        return NOT_MATCH;  // products of operands that do not exist
    }
    const uint64_t nA = elems(p.a), nB = elems(p.b), nC = elems(p.c);
    const size_t bias_bytes = (bias != nullptr && biasDesc != nullptr) ? (size_t)elems(*biasDesc) * bytes_of(biasDesc->dt) : 0;
    cudaStream_t st = tls().stream;

    // host pointers: the whole operator runs on device copies made for this call
    const bool host = !is_device_ptr(A) || !is_device_ptr(B) || !is_device_ptr(C) || !is_device_ptr(tmp) ||
        (bias_bytes && !is_device_ptr(bias));
    std::vector<void *> owned;
    struct Free {
        std::vector<void *> &v;
        ~Free()
        {
            for (void *q : v) {
                cudaFree(q);
            }
        }
    } guard{owned};
    const size_t c_bytes = (size_t)nC * bytes_of(p.c.dt);
    void *hostC = nullptr;
    if (host) {
        if (tls().device_only) {
            return NOT_MATCH;
        }
        auto dev_copy = [&](const void *src, size_t bytes, bool copy) -> void * {
            if (is_device_ptr(src)) {
                return const_cast<void *>(src);
            }
            void *d = nullptr;
            if (cudaMalloc(&d, bytes ? bytes : 16) != cudaSuccess) {
                cudaGetLastError();
                return nullptr;
            }
            owned.push_back(d);
            if (copy && cudaMemcpyAsync(d, src, bytes, cudaMemcpyHostToDevice, st) != cudaSuccess) {
                return nullptr;
            }
            return d;
        };
        A = dev_copy(A, (size_t)nA * bytes_of(p.a.dt), true);
        B = dev_copy(B, (size_t)nB * bytes_of(p.b.dt), true);
        if (bias_bytes) {
            bias = dev_copy(bias, bias_bytes, true);
        }
        tmp = dev_copy(tmp, tmpBytes, false);
        if (!is_device_ptr(C)) {
            hostC = C;
        }
        C = dev_copy(C, c_bytes, false);
        if (A == nullptr || B == nullptr || tmp == nullptr || C == nullptr || (bias_bytes && bias == nullptr)) {
            return ALLOC_FAILED;
        }
    }
    if (on_other_device(A) || on_other_device(B) || on_other_device(C) || on_other_device(tmp)) {
        return NOT_MATCH;
    }

    // The batched kernel reads A and B while it writes C.  A result over its own operands (fp32 in, fp32 out) needs the
    // quantized copies of the other way.
    const bool in_place = !p.stageC && (overlap(C, c_bytes, A, (size_t)nA * bytes_of(p.a.dt)) || overlap(C, c_bytes, B, (size_t)nB * bytes_of(p.b.dt)));
    const bool fused = !in_place && one_launch(p, A, c->sm_count, st);
    // (the tmp bytes count 1 KiB more than what is laid out in it)
    char *t = fused ? reinterpret_cast<char *>(B200_ALIGN(reinterpret_cast<uintptr_t>(tmp), 16)) : reinterpret_cast<char *>(tmp);
    char *slotsA = t, *slotsB = t + (p.quantA ? B200_ALIGN(nA, 256) : 0);
    F32 scaleO = 1;
    // operands: quantize into tmp, or take the caller's quantized bytes and scale (matmul.cpp:401-421)
    if (fused) {
        t = slotsB + (p.quantB ? B200_ALIGN(nB, 256) : 0);
    } else if (p.quantA) {
        F32 s = aScale;
        TensorDesc q = p.a;
        q.dt = p.qa;
        B200_EE(quantize_cuda_b200(&p.a, A, &q, t, &s, 0));
        scaleO *= s;
        A = t;
        t += B200_ALIGN(nA, 256);
    } else {
        scaleO *= aScale;
    }
    if (fused) {
        // the scales are found and used on the device
    } else if (p.quantB) {
        F32 s = bScale;
        TensorDesc q = p.b;
        q.dt = p.qb;
        B200_EE(quantize_cuda_b200(&p.b, B, &q, t, &s, 0));
        scaleO *= s;
        B = t;
        t += B200_ALIGN(nB, 256);
    } else {
        scaleO *= bScale;
    }
    void *prod = C;
    if (p.stageC) {
        prod = t;
        t += B200_ALIGN(nC * 4, 256);
    }
    F32 scaleArray[2] = {-1, -1};
    const F32 *scalePtr = &scaleO;
    if (p.static_u8) {
        scaleArray[1] = *cScale / scaleO;  // matmul.cpp:383-386,429-431
        scalePtr = scaleArray;
    }
    // the product accumulates on top of C: zero, or the bias bytes repeated (matmul.cpp:453-476)
    const size_t prod_bytes = (size_t)nC * bytes_of(p.qc);
    if (bias_bytes) {
        if (prod_bytes % bias_bytes != 0) {
            return NOT_MATCH;
        }
        const uint32_t grid = (uint32_t)std::min<uint64_t>((prod_bytes + 255) / 256, (uint64_t)c->sm_count * 8);
        fill_rows_kernel<<<grid, 256, 0, st>>>(reinterpret_cast<uint8_t *>(prod), prod_bytes,
            reinterpret_cast<const uint8_t *>(bias), (uint32_t)bias_bytes);
        count_launch();
    } else if (!fused) {
        B200_CUDA(cudaMemsetAsync(prod, 0, prod_bytes, st));
    }

    if (fused) {
        MatmulBatch mb;
        mb.M = p.a.dims[1 - p.kDimA];
        mb.N = p.b.dims[1 - p.kDimB];
        mb.K = p.a.dims[p.kDimA];
        mb.batches = p.loopsC;
        for (U32 i = 0; i < 4; ++i) {
            mb.c_dims[i] = i + 2 < p.c.nDims ? p.c.dims[i + 2] : 1;
        }
        mb.a = batch_operand(A, p.a, p.quantA, p.dfA == DF_TRANSPOSE, aScale, p.loopsA, p.loopsC, slotsA);
        mb.b = batch_operand(B, p.b, p.quantB, p.dfB == DF_TRANSPOSE, bScale, p.loopsB, p.loopsC, slotsB);
        mb.C = prod;
        mb.out_kind = p.static_u8 ? 2 : 1;
        mb.accumulate = bias_bytes && !p.static_u8 ? 1 : 0;
        mb.c_scale = *cScale;
        B200_EE(launch_matmul_batch(mb, st));
    }
    const size_t a2 = (size_t)p.a.dims[0] * p.a.dims[1], b2 = (size_t)p.b.dims[0] * p.b.dims[1];
    const size_t c2 = (size_t)p.c.dims[0] * p.c.dims[1] * bytes_of(p.qc);
    for (uint64_t ic = 0; !fused && ic < p.loopsC; ++ic) {
        const uint64_t ia = p.loopsA == p.loopsC ? ic : global_index(ic, p.c, p.a);
        const uint64_t ib = p.loopsB == p.loopsC ? ic : global_index(ic, p.c, p.b);
        const char *pa = reinterpret_cast<const char *>(A) + ia * a2;
        const char *pb = reinterpret_cast<const char *>(B) + ib * b2;
        char *pc = reinterpret_cast<char *>(prod) + ic * c2;
        EE ret;
        tls().last_gemm_tc = 0;   // (the GEMM sets it)
        if (p.a.dims[1 - p.kDimA] == 1) {
            ret = b200_matrix_vector_multiply(
                desc2d(p.qb, p.dfB == DF_TRANSPOSE ? DF_NORMAL : DF_TRANSPOSE, p.b.dims[1], p.b.dims[0]), pb,
                desc1d(p.qa, p.a.dims[p.kDimA]), pa, p.mmm_bytes, t, desc1d(p.qc, p.c.dims[0]), pc, scalePtr, CUDA_B200);
        } else if (p.b.dims[1 - p.kDimB] == 1) {
            ret = b200_matrix_vector_multiply(desc2d(p.qa, p.dfA, p.a.dims[1], p.a.dims[0]), pa,
                desc1d(p.qb, p.b.dims[p.kDimB]), pb, p.mmm_bytes, t, desc1d(p.qc, p.c.dims[1]), pc, scalePtr, CUDA_B200);
        } else {
            ret = b200_matrix_matrix_multiply(desc2d(p.qa, p.dfA, p.a.dims[1], p.a.dims[0]), pa,
                desc2d(p.qb, p.dfB, p.b.dims[1], p.b.dims[0]), pb, p.mmm_bytes, t,
                desc2d(p.qc, DF_NORMAL, p.c.dims[1], p.c.dims[0]), pc, scalePtr, CUDA_B200);
        }
        B200_EE(ret);
    }
    // matmul.cpp:535-554: a u8 output without a given scale is quantized from the fp32 product
    if (p.stageC) {
        F32 scales[2] = {*cScale, scaleO};   // (of an fp32 source only the first is read)
        TensorDesc src = p.c;
        src.dt = p.qc;
        B200_EE(quantize_cuda_b200(&src, prod, &p.c, C, scales, 0));
        *cScale = scales[0];
    }
    if (hostC != nullptr) {
        B200_CUDA(cudaMemcpyAsync(hostC, C, c_bytes, cudaMemcpyDeviceToHost, st));
    }
    if (host) {
        B200_CUDA(cudaStreamSynchronize(st));
    }
    return SUCCESS;
}

}  // extern "C"
