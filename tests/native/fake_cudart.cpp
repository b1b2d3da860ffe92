// A CUDA runtime without a device, linked in the place of the real one: memory is the host's, launches are recorded and run
// nothing.  Two users: max_mail_harness.cu, which answers the stream calls itself, and fake_gpu.py, which drives the whole
// library through its C ABI.
#include <cuda.h>
#include <cuda_runtime_api.h>

#include <cstdint>
#include <cstdlib>
#include <cstring>
#include <map>
#include <string>
#include <vector>

int (*on_query)(void) = nullptr;
int (*on_synchronize)(void) = nullptr;

namespace {

cudaError_t last = cudaSuccess;
cudaError_t fail(cudaError_t e)
{
    return last = e;
}
struct Names {
    std::map<const void *, std::string> of;   // kernel -> mangled name
    static Names &get()
    {
        static Names n;
        return n;
    }
};
std::vector<std::string> launched;
void *max_words = nullptr;   // where the last absmax_kernel was to count
int refused = 0;
bool captured = false, refuse_programmatic = false, refuse_fills = false;
struct Call {
    dim3 grid, block;
    size_t smem;
    void *stream;
} pushed;
struct Fill {
    void *p;
    int v;
    size_t n;
};
std::vector<Fill> fills;   // cudaMemset does not wait: they happen when somebody waits for the stream
void run_fills()
{
    for (const Fill &f : fills) {
        std::memset(f.p, f.v, f.n);
    }
    fills.clear();
}

// struct MaxMail of common.cuh, and what the kernels that get one report
struct Mail {
    unsigned *words;
    unsigned long long *d_mail;
    volatile unsigned long long *h_mail;
    uint32_t seq;
};
cudaError_t run(const void *f, dim3 grid, dim3 block, void **args)
{
    if (grid.x == 0 || block.x == 0) {
        return fail(cudaErrorInvalidConfiguration);
    }
    const std::string &name = Names::get().of[f];
    launched.push_back(name);
    if (name.find("absmax_kernel") != std::string::npos) {
        const Mail *m = reinterpret_cast<const Mail *>(args[2]);
        max_words = m->words;
        if (m->d_mail != nullptr) {
            *m->d_mail = ((unsigned long long)m->seq << 32) | 0x40000000u;   // 2.0
        }
    }
    return cudaSuccess;
}
CUresult encode(CUtensorMap *m, CUtensorMapDataType, cuuint32_t, void *, const cuuint64_t *, const cuuint64_t *, const cuuint32_t *,
    const cuuint32_t *, CUtensorMapInterleave, CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill)
{
    std::memset(m, 0, sizeof(*m));
    return CUDA_SUCCESS;
}

}  // namespace

extern "C" {

// ---- for the tests ----
int fake_launches(void)
{
    return (int)launched.size();
}
const char *fake_launch_name(int i)
{
    return launched[i].c_str();
}
void fake_forget_launches(void)
{
    launched.clear();
}
void *fake_max_words(void)
{
    return max_words;
}
void fake_capture(int on)   // streams are being captured
{
    captured = on != 0;
}
void fake_refuse_programmatic(int on)
{
    refuse_programmatic = on != 0;
}
int fake_refused(void)
{
    return refused;
}
void fake_refuse_fills(int on)
{
    refuse_fills = on != 0;
}
void fake_set_last_error(int e)
{
    last = (cudaError_t)e;
}
int fake_last_error(void)
{
    return (int)last;
}
int fake_unordered_fills(void)
{
    return (int)fills.size();
}

// ---- memory ----
cudaError_t cudaMalloc(void **p, size_t n)
{
    *p = std::aligned_alloc(4096, (n + 4095) / 4096 * 4096);
    std::memset(*p, 0xA5, n);
    return cudaSuccess;
}
cudaError_t cudaFree(void *p)
{
    std::free(p);
    return cudaSuccess;
}
cudaError_t cudaFreeHost(void *p)
{
    return cudaFree(p);
}
cudaError_t cudaHostAlloc(void **p, size_t n, unsigned)
{
    return cudaMalloc(p, n);
}
cudaError_t cudaHostGetDevicePointer(void **d, void *h, unsigned)
{
    *d = h;
    return cudaSuccess;
}
cudaError_t cudaMemset(void *p, int v, size_t n)
{
    if (refuse_fills && n > 1024) {   // (the words of the maxima, not the smaller status)
        return fail(cudaErrorNotSupported);
    }
    fills.push_back(Fill{p, v, n});
    return cudaSuccess;
}
cudaError_t cudaMemsetAsync(void *p, int v, size_t n, cudaStream_t)
{
    std::memset(p, v, n);
    return cudaSuccess;
}
cudaError_t cudaMemcpy(void *d, const void *s, size_t n, cudaMemcpyKind)
{
    run_fills();
    std::memcpy(d, s, n);
    return cudaSuccess;
}
cudaError_t cudaMemcpyAsync(void *d, const void *s, size_t n, cudaMemcpyKind, cudaStream_t)
{
    std::memcpy(d, s, n);
    return cudaSuccess;
}
cudaError_t cudaPointerGetAttributes(cudaPointerAttributes *a, const void *)
{
    std::memset(a, 0, sizeof(*a));
    a->type = cudaMemoryTypeDevice;
    return cudaSuccess;
}
cudaError_t cudaIpcGetMemHandle(cudaIpcMemHandle_t *, void *)
{
    return fail(cudaErrorNotSupported);
}
cudaError_t cudaIpcOpenMemHandle(void **, cudaIpcMemHandle_t, unsigned)
{
    return fail(cudaErrorNotSupported);
}
cudaError_t cudaIpcCloseMemHandle(void *)
{
    return fail(cudaErrorNotSupported);
}

// ---- device, streams, events ----
cudaError_t cudaGetDevice(int *d)
{
    *d = 0;
    return cudaSuccess;
}
cudaError_t cudaSetDevice(int)
{
    return cudaSuccess;
}
cudaError_t cudaGetDeviceCount(int *n)
{
    *n = 1;
    return cudaSuccess;
}
cudaError_t cudaGetDeviceProperties_v2(cudaDeviceProp *p, int)
{
    std::memset(p, 0, sizeof(*p));
    p->multiProcessorCount = 148;
    return cudaSuccess;
}
cudaError_t cudaGetLastError(void)
{
    const cudaError_t e = last;
    last = cudaSuccess;
    return e;
}
cudaError_t cudaStreamQuery(cudaStream_t)
{
    return on_query ? (cudaError_t)on_query() : cudaSuccess;
}
cudaError_t cudaStreamSynchronize(cudaStream_t)
{
    run_fills();
    return on_synchronize ? (cudaError_t)on_synchronize() : cudaSuccess;
}
cudaError_t cudaDeviceSynchronize(void)
{
    return cudaStreamSynchronize(nullptr);
}
cudaError_t cudaStreamIsCapturing(cudaStream_t, cudaStreamCaptureStatus *s)
{
    *s = captured ? cudaStreamCaptureStatusActive : cudaStreamCaptureStatusNone;
    return cudaSuccess;
}
cudaError_t cudaEventCreate(cudaEvent_t *)
{
    return fail(cudaErrorNotSupported);
}
cudaError_t cudaEventDestroy(cudaEvent_t)
{
    return fail(cudaErrorNotSupported);
}
cudaError_t cudaEventElapsedTime(float *, cudaEvent_t, cudaEvent_t)
{
    return fail(cudaErrorNotSupported);
}
cudaError_t cudaEventRecord(cudaEvent_t, cudaStream_t)
{
    return fail(cudaErrorNotSupported);
}
cudaError_t cudaEventSynchronize(cudaEvent_t)
{
    return fail(cudaErrorNotSupported);
}

// ---- kernels ----
cudaError_t cudaFuncSetAttribute(const void *, cudaFuncAttribute, int)
{
    return cudaSuccess;
}
cudaError_t cudaOccupancyMaxActiveClusters(int *n, const void *, const cudaLaunchConfig_t *)
{
    *n = 74;
    return cudaSuccess;
}
cudaError_t cudaLaunchKernel(const void *f, dim3 grid, dim3 block, void **args, size_t, cudaStream_t)
{
    return run(f, grid, block, args);
}
cudaError_t cudaLaunchKernelExC(const cudaLaunchConfig_t *c, const void *f, void **args)
{
    for (unsigned i = 0; i < c->numAttrs; ++i) {
        if (refuse_programmatic && c->attrs[i].id == cudaLaunchAttributeProgrammaticStreamSerialization) {
            ++refused;
            return fail(cudaErrorNotSupported);
        }
    }
    return run(f, c->gridDim, c->blockDim, args);
}
cudaError_t cudaGetDriverEntryPoint(const char *name, void **p, unsigned long long, cudaDriverEntryPointQueryResult *r)
{
    const bool known = std::strcmp(name, "cuTensorMapEncodeTiled") == 0;
    *p = known ? reinterpret_cast<void *>(encode) : nullptr;
    if (r != nullptr) {
        *r = known ? cudaDriverEntryPointSuccess : cudaDriverEntryPointSymbolNotFound;
    }
    return known ? cudaSuccess : fail(cudaErrorNotSupported);
}
cudaError_t cudaGetSymbolAddress(void **, const void *)
{
    return fail(cudaErrorNotSupported);
}
unsigned __cudaPushCallConfiguration(dim3 grid, dim3 block, size_t smem, void *stream)
{
    pushed = Call{grid, block, smem, stream};
    return 0;
}
cudaError_t __cudaPopCallConfiguration(dim3 *grid, dim3 *block, size_t *smem, void *stream)
{
    *grid = pushed.grid;
    *block = pushed.block;
    *smem = pushed.smem;
    *reinterpret_cast<void **>(stream) = pushed.stream;
    return cudaSuccess;
}
void **__cudaRegisterFatBinary(void *)
{
    return nullptr;
}
void __cudaRegisterFatBinaryEnd(void **) {}
void __cudaUnregisterFatBinary(void **) {}
void __cudaRegisterFunction(void **, const char *host, char *, const char *name, int, void *, void *, void *, void *, int *)
{
    Names::get().of[host] = name;
}
void __cudaRegisterVar(void **, char *, char *, const char *, int, size_t, int, int) {}

}  // extern "C"
