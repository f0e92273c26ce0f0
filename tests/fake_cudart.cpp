// A CUDA runtime for the library's host code on a machine without a GPU: nothing runs, and a launch
// is refused as the device would refuse it, for more than 48 KB of dynamic shared memory or a
// cluster of more than eight CTAs that the kernel has not opted in to on the current device.
#include <cuda_runtime_api.h>

#include <map>
#include <utility>

namespace {
struct Allowed {
    size_t smem = 48 * 1024;
    bool wide = false;
};
std::map<std::pair<int, const void *>, Allowed> g_allowed;
int g_device = 0, g_launches = 0;
cudaError_t g_error = cudaSuccess;
dim3 g_grid, g_block;
size_t g_smem;

cudaError_t launch(const void *fn, size_t smem, unsigned cluster)
{
    const Allowed a = g_allowed[{g_device, fn}];
    ++g_launches;
    if (smem > a.smem) return g_error = cudaErrorInvalidValue;
    if (cluster > 8 && !a.wide) return g_error = cudaErrorInvalidClusterSize;
    return cudaSuccess;
}
}  // namespace

extern "C" {
void fake_set_device(int d) { g_device = d; }
int fake_launches() { return g_launches; }

void **__cudaRegisterFatBinary(void *) { return nullptr; }
void __cudaRegisterFatBinaryEnd(void **) {}
void __cudaUnregisterFatBinary(void **) {}
void __cudaRegisterFunction(void **, const char *, char *, const char *, int, uint3 *, uint3 *, dim3 *, dim3 *, int *) {}
void __cudaRegisterVar(void **, char *, char *, const char *, int, size_t, int, int) {}
unsigned __cudaPushCallConfiguration(dim3 grid, dim3 block, size_t smem, void *)
{
    g_grid = grid, g_block = block, g_smem = smem;
    return 0;
}
cudaError_t __cudaPopCallConfiguration(dim3 *grid, dim3 *block, size_t *smem, void *stream)
{
    *grid = g_grid, *block = g_block, *smem = g_smem;
    *(void **)stream = nullptr;
    return cudaSuccess;
}
cudaError_t cudaLaunchKernel(const void *fn, dim3, dim3, void **, size_t smem, cudaStream_t) { return launch(fn, smem, 1); }
cudaError_t cudaLaunchKernelExC(const cudaLaunchConfig_t *c, const void *fn, void **)
{
    unsigned cluster = 1;
    for (unsigned i = 0; i < c->numAttrs; ++i)
        if (c->attrs[i].id == cudaLaunchAttributeClusterDimension) cluster = c->attrs[i].val.clusterDim.x;
    return launch(fn, c->dynamicSmemBytes, cluster);
}
cudaError_t cudaFuncSetAttribute(const void *fn, cudaFuncAttribute what, int value)
{
    Allowed &a = g_allowed[{g_device, fn}];
    if (what == cudaFuncAttributeMaxDynamicSharedMemorySize) a.smem = (size_t)value;
    if (what == cudaFuncAttributeNonPortableClusterSizeAllowed) a.wide = value != 0;
    return cudaSuccess;
}
cudaError_t cudaOccupancyMaxPotentialClusterSize(int *n, const void *, const cudaLaunchConfig_t *)
{
    *n = 16;
    return cudaSuccess;
}
cudaError_t cudaOccupancyMaxActiveBlocksPerMultiprocessor(int *n, const void *, int, size_t)
{
    *n = 1;
    return cudaSuccess;
}
cudaError_t cudaOccupancyMaxActiveBlocksPerMultiprocessorWithFlags(int *n, const void *, int, size_t, unsigned)
{
    *n = 1;
    return cudaSuccess;
}
cudaError_t cudaDeviceGetAttribute(int *v, cudaDeviceAttr, int)
{
    *v = 148;
    return cudaSuccess;
}
cudaError_t cudaGetDevice(int *d)
{
    *d = g_device;
    return cudaSuccess;
}
cudaError_t cudaGetLastError()
{
    const cudaError_t e = g_error;
    g_error = cudaSuccess;
    return e;
}
const char *cudaGetErrorString(cudaError_t e)
{
    return e == cudaErrorInvalidValue ? "shared memory above the opt-in" : e == cudaErrorInvalidClusterSize
        ? "cluster above the opt-in" : "no error";
}
cudaError_t cudaMemsetAsync(void *, int, size_t, cudaStream_t) { return cudaSuccess; }
}
