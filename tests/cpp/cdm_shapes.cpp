// Launch decisions of the CDM passes without a device: linked with the compiled passes and
// with the runtime calls below in place of the CUDA runtime's.
//
//   cdm_shapes probe <call>           the n-th runtime call of the cluster check fails (0: none);
//                                     prints whether clusters are used, and the error left behind
//   cdm_shapes dims <w> <h> <d>       a level's layout and launch shapes: ppitch pplane nblk pnb
//                                     pdz tnb each shallow
#include <atomic>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include "kernels.h"
#include "stats.h"

namespace regb {
std::atomic<long long> g_launches{0};
}

namespace {
int g_calls = 0, g_fail = 0;
cudaError_t g_last = cudaSuccess;
cudaError_t call()
{
    if (++g_calls != g_fail)
        return cudaSuccess;
    return g_last = cudaErrorInvalidValue;
}
}  // namespace

extern "C" {
cudaError_t cudaGetDevice(int* d)
{
    *d = 0;
    return call();
}
cudaError_t cudaFuncSetAttribute(const void*, cudaFuncAttribute, int) { return call(); }
cudaError_t cudaOccupancyMaxActiveClusters(int* n, const void*, const cudaLaunchConfig_t*)
{
    *n = 1;
    return call();
}
cudaError_t cudaGetLastError()
{
    const cudaError_t e = g_last;
    g_last = cudaSuccess;
    return e;
}
cudaError_t cudaLaunchKernel(const void*, dim3, dim3, void**, size_t, cudaStream_t) { return call(); }
cudaError_t cudaLaunchKernelExC(const cudaLaunchConfig_t*, const void*, void**) { return call(); }
cudaError_t cudaMemsetAsync(void*, int, size_t, cudaStream_t) { return call(); }
void** __cudaRegisterFatBinary(void*)
{
    static void* handle;
    return &handle;
}
void __cudaRegisterFatBinaryEnd(void**) {}
void __cudaUnregisterFatBinary(void**) {}
void __cudaRegisterFunction(void**, const char*, char*, const char*, int, uint3*, uint3*, dim3*, dim3*, int*) {}
unsigned __cudaPushCallConfiguration(dim3, dim3, size_t, CUstream_st*) { return 0; }
cudaError_t __cudaPopCallConfiguration(dim3*, dim3*, size_t*, void*) { return cudaSuccess; }
}

int main(int argc, char** argv)
{
    if (argc == 3 && !std::strcmp(argv[1], "probe")) {
        g_fail = std::atoi(argv[2]);
        regb::CdmSeg s{};
        regb::cdm_set_dims(s, 32, 32, 32);
        const bool small = regb::cdm_poisson_small(s);
        std::printf("%d %d %d\n", (int)small, (int)g_last, g_calls);
        return 0;
    }
    if (argc == 5 && !std::strcmp(argv[1], "dims")) {
        regb::CdmSeg s{};
        regb::cdm_set_dims(s, std::atoi(argv[2]), std::atoi(argv[3]), std::atoi(argv[4]));
        std::printf("%lld %lld %d %d %d %d %d %d\n", s.ppitch, s.pplane, s.nblk, s.pnb, s.pdz, s.tnb, s.each,
                    s.shallow);
        return 0;
    }
    return 2;
}
