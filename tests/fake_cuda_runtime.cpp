// A stand-in for the CUDA runtime calls that liblutgemm_b200.so makes, for tests of its host code without a GPU: the
// library's object files are linked with this file (tests/host_dispatch.py).  Launches, memsets and attribute calls are
// recorded and nothing runs; every pointer is only a number.  fake_* is what the tests call.
#include <cuda_runtime_api.h>
#include <stdio.h>

#include <map>
#include <string>
#include <vector>

namespace {

struct Call {
    std::string name;  // kernel name (mangled) or "memset"
    unsigned long long size[4];  // grid x, y, z and dynamic shared memory; for a memset its bytes
};
std::vector<Call> g_calls;
// (filled by the constructors of the other object files, so not a global with a constructor of its own)
std::map<const void *, std::string> &kernels() {
    static std::map<const void *, std::string> m;
    return m;
}
struct {
    dim3 grid, block;
    size_t smem;
    cudaStream_t stream;
} g_config;
alignas(256) char g_symbol[256];  // the address of every device variable

}  // namespace

extern "C" {

void fake_reset() { g_calls.clear(); }
int fake_calls() { return (int)g_calls.size(); }
const char *fake_name(int i) { return g_calls[i].name.c_str(); }
unsigned long long fake_size(int i, int j) { return g_calls[i].size[j]; }

// ---- what the compiler's host stubs call ------------------------------------------------------------------------
void **__cudaRegisterFatBinary(void *) {
    static void *handle;
    return &handle;
}
void __cudaRegisterFatBinaryEnd(void **) {}
void __cudaUnregisterFatBinary(void **) {}
void __cudaRegisterVar(void **, char *, char *, const char *, int, size_t, int, int) {}
void __cudaRegisterFunction(void **, const char *host, char *, const char *name, int, void *, void *, void *, void *, int *) {
    kernels()[host] = name;
}
unsigned __cudaPushCallConfiguration(dim3 grid, dim3 block, size_t smem, void *stream) {
    g_config = {grid, block, smem, (cudaStream_t)stream};
    return 0;
}
cudaError_t __cudaPopCallConfiguration(dim3 *grid, dim3 *block, size_t *smem, void *stream) {
    *grid = g_config.grid;
    *block = g_config.block;
    *smem = g_config.smem;
    *(cudaStream_t *)stream = g_config.stream;
    return cudaSuccess;
}

// ---- runtime API ------------------------------------------------------------------------------------------------
cudaError_t cudaLaunchKernel(const void *func, dim3 grid, dim3 block, void **, size_t smem, cudaStream_t) {
    // the limits that a device would refuse a launch for
    if (!grid.x || !grid.y || !grid.z || grid.x > 0x7fffffffu || grid.y > 65535u || grid.z > 65535u ||
        block.x * block.y * block.z > 1024u)
        return cudaErrorInvalidConfiguration;
    g_calls.push_back({kernels()[func], {grid.x, grid.y, grid.z, smem}});
    return cudaSuccess;
}
cudaError_t cudaMemsetAsync(void *, int, size_t bytes, cudaStream_t) {
    g_calls.push_back({"memset", {bytes, 0, 0, 0}});
    return cudaSuccess;
}
cudaError_t cudaGetDevice(int *dev) {
    *dev = 0;
    return cudaSuccess;
}
cudaError_t cudaDeviceGetAttribute(int *value, cudaDeviceAttr attr, int) {
    *value = attr == cudaDevAttrMultiProcessorCount ? 148 : 0;
    return cudaSuccess;
}
cudaError_t cudaFuncSetAttribute(const void *, cudaFuncAttribute, int) { return cudaSuccess; }
cudaError_t cudaOccupancyMaxActiveBlocksPerMultiprocessorWithFlags(int *blocks, const void *, int, size_t, unsigned) {
    *blocks = 1;
    return cudaSuccess;
}
cudaError_t cudaGetSymbolAddress(void **ptr, const void *) {
    *ptr = g_symbol;
    return cudaSuccess;
}
cudaError_t cudaMemcpyFromSymbol(void *, const void *, size_t, size_t, cudaMemcpyKind) { return cudaErrorNotSupported; }
cudaError_t cudaMemcpyToSymbol(const void *, const void *, size_t, size_t, cudaMemcpyKind) { return cudaErrorNotSupported; }
cudaError_t cudaGetLastError() { return cudaSuccess; }
const char *cudaGetErrorString(cudaError_t) { return "error of the stand-in runtime"; }
cudaError_t cudaGetDriverEntryPoint(const char *, void **fn, unsigned long long, cudaDriverEntryPointQueryResult *q) {
    *fn = nullptr;  // no tensor maps: the kernels without bulk copies are chosen
    *q = cudaDriverEntryPointSymbolNotFound;
    return cudaSuccess;
}

}  // extern "C"
