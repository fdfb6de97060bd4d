// Test infrastructure: the cluster kernel's object file (rcpg_small.o) on a
// stand-in for the few runtime calls it makes, to test without a GPU what it
// does on a device that cannot place its cluster.
#include <cuda_runtime.h>

#include "rcpg_device.h"

namespace {
int fit = 1;                           // clusters that fit at once
cudaError_t set_error = cudaSuccess;   // of cudaFuncSetAttribute
cudaError_t ask_error = cudaSuccess;   // of cudaOccupancyMaxActiveClusters
cudaError_t run_error = cudaSuccess;   // of the launch
cudaError_t last = cudaSuccess;
int launches = 0;
unsigned cluster = 0;
cudaError_t set_last(cudaError_t e) {
    if (e != cudaSuccess) last = e;
    return e;
}
}  // namespace

extern "C" {
unsigned __cudaPopCallConfiguration(dim3*, dim3*, size_t*, void*) { return 0; }
void** __cudaRegisterFatBinary(void*) { return nullptr; }
void __cudaRegisterFatBinaryEnd(void**) {}
void __cudaUnregisterFatBinary(void**) {}
void __cudaRegisterFunction(void**, const char*, char*, const char*, int, uint3*, uint3*, dim3*, dim3*, int*) {}
cudaError_t cudaLaunchKernel(const void*, dim3, dim3, void**, size_t, cudaStream_t) { return cudaErrorUnknown; }
cudaError_t cudaFuncSetAttribute(const void*, cudaFuncAttribute, int) { return set_last(set_error); }
cudaError_t cudaGetLastError() {
    const cudaError_t e = last;
    last = cudaSuccess;
    return e;
}
cudaError_t cudaOccupancyMaxActiveClusters(int* n, const void*, const cudaLaunchConfig_t* cfg) {
    cluster = cfg->attrs[0].val.clusterDim.x;
    *n = fit;
    return set_last(ask_error);
}
cudaError_t cudaLaunchKernelExC(const cudaLaunchConfig_t*, const void*, void**) {
    ++launches;
    return set_last(run_error);
}

// small_steps_ok for N particles; -1 where it leaves an error behind
int sf_ok(unsigned long long N, int ndim, unsigned cells, int clusters, int set, int ask) {
    fit = clusters;
    set_error = static_cast<cudaError_t>(set);
    ask_error = static_cast<cudaError_t>(ask);
    rcpg::DevArrays a{};
    a.N = N;
    a.ndim = ndim;
    a.permute = 1;
    a.C_alloc = cells;
    const bool ok = rcpg::small_steps_ok(a);
    return last != cudaSuccess ? -1 : (ok ? 1 : 0);
}
unsigned sf_cluster() { return cluster; }
// what a launch reports
int sf_run(int ndim, int set, int run) {
    set_error = static_cast<cudaError_t>(set);
    run_error = static_cast<cudaError_t>(run);
    rcpg::DevArrays a{};
    a.N = 100;
    a.ndim = ndim;
    launches = 0;
    const int e = static_cast<int>(rcpg::launch_small_steps(a, 1, nullptr));
    cudaGetLastError();
    return e;
}
}
