// Test infrastructure: the engine's host code (rcpg_engine.cu, compiled as
// plain C++) on a stand-in for the CUDA runtime and for the kernels. Device
// memory is host memory, launches act on the control block at once, and two
// devices exist, each with its own current setting per thread: a launch or an
// allocation with another device current than the engine's fails or is
// counted, as on a machine. What the host decides -- how many steps it asks
// for, when it resumes after a row overflow, which path and which graph it
// takes, which device it leaves current -- is tested here without a GPU.
#include <cuda_runtime.h>

#include <cstdint>
#include <cstdlib>
#include <cstring>
#include <map>
#include <stdexcept>
#include <vector>

#include "rcpg_engine.h"

namespace {

struct Stream {
    int device;
};

struct Fake {
    // scenario
    int small_clusters = 0;                    // clusters of the small-packing kernel that fit the device
    std::vector<std::uint64_t> overflow_steps; // steps whose build finds a row beyond the capacity
    std::vector<std::uint32_t> overflow_need;
    std::uint64_t build_every = 1;             // steps that rebuild
    std::uint64_t reorder_every = 0;           // steps that open with a reorder stop the loop
    // records
    int observer_device = -1;                  // device that was current in every observer call (-2: several)
    std::uint64_t wrong_device = 0;            // launches and allocations on a device that is not the engine's
    std::uint64_t graph_launches = 0, small_launches = 0;
    int captured = 0;                          // steps of the graph captured last
    cudaStream_t capturing = nullptr;          // the stream whose launches are captured
    rcpg::DevArrays graph_arrays{};
};
Fake fk;
thread_local int current_device = 0;
thread_local cudaError_t last_error = cudaSuccess;
std::map<void*, int> memory;  // allocation -> device

int device_of(cudaStream_t st) { return st ? reinterpret_cast<Stream*>(st)->device : 0; }

// Whether a launch on st takes place.
bool launched(cudaStream_t st) {
    if (current_device == device_of(st)) return true;
    if (++fk.wrong_device > 1000) throw std::runtime_error("a loop whose launches all fail");
    last_error = cudaErrorInvalidResourceHandle;
    return false;
}

// The row length that the build of the open step reports.
std::uint32_t need_of(const rcpg::DevCtl& k) {
    for (std::size_t i = 0; i < fk.overflow_steps.size(); ++i)
        if (k.c.steps == fk.overflow_steps[i]) return fk.overflow_need[i];
    return 8;
}

// The controller: closes the open step and opens the next, or halts.
void controller(const rcpg::DevArrays& a) {
    rcpg::DevCtl& k = *a.ctl;
    if (k.stopped | k.halted) return;
    if (k.row_need > a.S) {
        k.halted = 1u;
        return;
    }
    k.c.hist_filled = k.c.steps;
    k.c.reorder = 0;
    if (k.c.steps + 1 > k.c.step_cap) {
        k.stopped = 1u;
        return;
    }
    k.c.steps += 1;
    if (fk.reorder_every && k.c.steps % fk.reorder_every == 0) k.c.reorder = k.stopped = 1u;
}

void step(const rcpg::DevArrays& a) {
    if (!(a.ctl->stopped | a.ctl->halted)) {
        a.ctl->row_need = need_of(*a.ctl);
        if (a.ctl->c.steps % fk.build_every == 0) a.ctl->nbuilds += 1;
    }
    controller(a);
}

}  // namespace

// ---- the CUDA runtime ------------------------------------------------------
extern "C" {
cudaError_t cudaGetDevice(int* d) { *d = current_device; return cudaSuccess; }
cudaError_t cudaSetDevice(int d) { current_device = d; return cudaSuccess; }
cudaError_t cudaGetLastError() { const cudaError_t e = last_error; last_error = cudaSuccess; return e; }
const char* cudaGetErrorString(cudaError_t) { return "stand-in error"; }
cudaError_t cudaMemPoolCreate(cudaMemPool_t* p, const cudaMemPoolProps* props) {
    *p = reinterpret_cast<cudaMemPool_t>(new int(props->location.id));
    return cudaSuccess;
}
cudaError_t cudaMemPoolSetAttribute(cudaMemPool_t, cudaMemPoolAttr, void*) { return cudaSuccess; }
cudaError_t cudaMallocFromPoolAsync(void** p, size_t n, cudaMemPool_t pool, cudaStream_t st) {
    *p = std::calloc(1, n);
    memory[*p] = *reinterpret_cast<int*>(pool);
    if (memory[*p] != device_of(st)) ++fk.wrong_device;
    return cudaSuccess;
}
cudaError_t cudaFreeAsync(void* p, cudaStream_t) { memory.erase(p); std::free(p); return cudaSuccess; }
cudaError_t cudaMallocHost(void** p, size_t n) { *p = std::calloc(1, n); return cudaSuccess; }
cudaError_t cudaMemcpyAsync(void* d, const void* s, size_t n, cudaMemcpyKind, cudaStream_t) {
    std::memmove(d, s, n);
    return cudaSuccess;
}
cudaError_t cudaMemsetAsync(void* p, int v, size_t n, cudaStream_t) { std::memset(p, v, n); return cudaSuccess; }
cudaError_t cudaStreamCreateWithFlags(cudaStream_t* st, unsigned) {
    *st = reinterpret_cast<cudaStream_t>(new Stream{current_device});
    return cudaSuccess;
}
cudaError_t cudaStreamDestroy(cudaStream_t st) { delete reinterpret_cast<Stream*>(st); return cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaEventCreate(cudaEvent_t* e) { *e = nullptr; return cudaSuccess; }
cudaError_t cudaEventCreateWithFlags(cudaEvent_t* e, unsigned) { *e = nullptr; return cudaSuccess; }
cudaError_t cudaEventDestroy(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaEventSynchronize(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventElapsedTime(float* ms, cudaEvent_t, cudaEvent_t) { *ms = 1.0f; return cudaSuccess; }
cudaError_t cudaStreamBeginCapture(cudaStream_t st, cudaStreamCaptureMode) {
    fk.capturing = st;
    fk.captured = 0;
    return cudaSuccess;
}
cudaError_t cudaStreamEndCapture(cudaStream_t st, cudaGraph_t* g) {
    if (st == fk.capturing) fk.capturing = nullptr;  // else the body of a conditional node
    *g = reinterpret_cast<cudaGraph_t>(&fk);
    return cudaSuccess;
}
cudaError_t cudaStreamBeginCaptureToGraph(cudaStream_t, cudaGraph_t, const cudaGraphNode_t*, const cudaGraphEdgeData*,
                                          size_t, cudaStreamCaptureMode) {
    return cudaSuccess;
}
cudaError_t cudaStreamGetCaptureInfo_v2(cudaStream_t, cudaStreamCaptureStatus* s, unsigned long long*, cudaGraph_t* g,
                                        const cudaGraphNode_t** deps, size_t* n) {
    *s = cudaStreamCaptureStatusActive;
    if (g) *g = reinterpret_cast<cudaGraph_t>(&fk);
    if (deps) *deps = nullptr;
    if (n) *n = 0;
    return cudaSuccess;
}
cudaError_t cudaStreamUpdateCaptureDependencies(cudaStream_t, cudaGraphNode_t*, size_t, unsigned) { return cudaSuccess; }
cudaError_t cudaGraphConditionalHandleCreate(cudaGraphConditionalHandle* h, cudaGraph_t, unsigned, unsigned) {
    *h = 1;
    return cudaSuccess;
}
cudaError_t cudaGraphAddNode(cudaGraphNode_t* node, cudaGraph_t, const cudaGraphNode_t*, size_t, cudaGraphNodeParams* p) {
    static cudaGraph_t bodies[4] = {};
    p->conditional.phGraph_out = bodies;
    *node = nullptr;
    return cudaSuccess;
}
cudaError_t cudaGraphInstantiate(cudaGraphExec_t* e, cudaGraph_t, unsigned long long) {
    *e = reinterpret_cast<cudaGraphExec_t>(&fk);
    return cudaSuccess;
}
cudaError_t cudaGraphGetNodes(cudaGraph_t, cudaGraphNode_t*, size_t* n) { *n = 4; return cudaSuccess; }
cudaError_t cudaGraphDestroy(cudaGraph_t) { return cudaSuccess; }
cudaError_t cudaGraphExecDestroy(cudaGraphExec_t) { return cudaSuccess; }
cudaError_t cudaGraphLaunch(cudaGraphExec_t, cudaStream_t st) {
    if (!launched(st)) return cudaErrorInvalidResourceHandle;
    ++fk.graph_launches;
    for (int k = 0; k < fk.captured; ++k) step(fk.graph_arrays);
    return cudaSuccess;
}
}

// ---- the kernels -------------------------------------------------------------
namespace rcpg {

void launch_rebuild(const DevArrays& a, cudaStream_t st, bool) {
    if (fk.capturing || !launched(st) || (a.ctl->stopped | a.ctl->halted)) return;
    a.ctl->row_need = need_of(*a.ctl);
    if (a.ctl->c.steps % fk.build_every == 0) a.ctl->nbuilds += 1;
}
void launch_rebuild_timed(const DevArrays& a, cudaStream_t st, cudaEvent_t, cudaEvent_t) { launch_rebuild(a, st, false); }
void launch_forces(const DevArrays&, int, cudaStream_t st) { launched(st); }
void launch_forces_variant(const DevArrays&, int, cudaStream_t) {}
void launch_step_gate(const DevArrays& a, unsigned long long, cudaStream_t) {
    fk.graph_arrays = a;
    ++fk.captured;
}
void launch_reduce_exact(const DevArrays&, cudaStream_t st) { launched(st); }
void launch_reduce_fast(const DevArrays&, cudaStream_t st) { launched(st); }
void launch_diff_max(const double*, const double*, std::uint64_t, unsigned long long*, cudaStream_t st) { launched(st); }
void launch_controller(const DevArrays& a, int open_only, cudaStream_t st) {
    if (fk.capturing || !launched(st)) return;
    if (open_only) a.ctl->c.steps = 1;
    else controller(a);
}
// an ADAM pass adds one to the first coordinate
void launch_adam_refresh(const DevArrays& a, int do_adam, int, cudaStream_t st) {
    if (fk.capturing || !launched(st)) return;
    if (do_adam && a.ctl->adam_go) a.pos[0] += 1.0;
}
void launch_reorder(const DevArrays&, cudaStream_t st) { launched(st); }
void launch_fix_height(const DevArrays&, cudaStream_t st) { launched(st); }
void launch_pack(std::uint64_t N, int ndim, const double* x, const double* D, double* pos, cudaStream_t st) {
    if (!launched(st)) return;
    const int P = pos_stride(ndim);
    for (std::uint64_t i = 0; i < N; ++i) {
        for (int d = 0; d < ndim; ++d) pos[i * P + d] = x[i * ndim + d];
        pos[i * P + ndim] = D[i];
    }
}
void launch_identity(std::uint64_t, std::uint64_t*, std::uint32_t*, cudaStream_t st) { launched(st); }
void launch_collect(const DevArrays& a, double kd, bool fixed, double* x, double* D, std::uint64_t*, cudaStream_t st) {
    if (!launched(st)) return;
    const int P = pos_stride(a.ndim);
    for (std::uint64_t i = 0; i < a.N; ++i) {
        for (int d = 0; d < a.ndim; ++d) x[i * a.ndim + d] = a.pos[i * P + d];
        D[i] = fixed ? a.pos[i * P + a.ndim] : a.pos[i * P + a.ndim] * kd;
    }
}
bool small_steps_ok(const DevArrays&) { return fk.small_clusters > 0; }
cudaError_t launch_small_steps(const DevArrays& a, std::uint32_t steps, cudaStream_t st) {
    if (!launched(st)) return cudaErrorInvalidResourceHandle;
    ++fk.small_launches;
    for (std::uint32_t k = 0; k < steps; ++k) step(a);
    return cudaSuccess;
}

}  // namespace rcpg

// ---- what the tests call -------------------------------------------------------
extern "C" {

void hf_reset(int small_clusters) {
    fk = Fake{};
    fk.small_clusters = small_clusters;
}
void hf_overflow(std::uint64_t step, std::uint32_t need) {
    fk.overflow_steps.push_back(step);
    fk.overflow_need.push_back(need);
}
void hf_build_every(std::uint64_t steps) { fk.build_every = steps; }
void hf_engines(void* e, std::uint64_t n) { static_cast<rcpg::Engine*>(e)->set_engines(n); }
void hf_reorder_every(std::uint64_t steps) { fk.reorder_every = steps; }
void hf_set_device(int d) { current_device = d; }
void hf_leave_error() { last_error = cudaErrorInvalidValue; }
int hf_get_device() { return current_device; }
int hf_observer_device() { return fk.observer_device; }
// wrong-device launches and allocations, graph launches, steps of the graph, small-packing launches
void hf_counts(std::uint64_t* out) {
    out[0] = fk.wrong_device;
    out[1] = fk.graph_launches;
    out[2] = static_cast<std::uint64_t>(fk.captured);
    out[3] = fk.small_launches;
}
void* hf_engine(std::uint64_t N, int ndim, double wide, int exact, int mixed, int graph_steps, std::uint64_t max_steps,
                int device) {
    rcpg::EngineInput in;
    in.N = N;
    in.ndim = ndim;
    in.positions.assign(ndim * N, 0.5);
    in.diameters.assign(N, 0.01);
    in.diameters[0] *= wide;
    in.fix_diameter = true;
    in.max_steps = max_steps;
    in.reorder_interval = 0;
    in.exact = exact != 0;
    in.pair_precision = mixed;
    in.graph_steps = graph_steps;
    in.device = device;
    try {
        return new rcpg::Engine(std::move(in));
    } catch (const std::exception&) {
        return nullptr;
    }
}
void hf_free(void* e) { delete static_cast<rcpg::Engine*>(e); }
int hf_advance(void* e, std::uint64_t k) {
    try {
        return static_cast<rcpg::Engine*>(e)->advance(k) ? 1 : 0;
    } catch (const std::exception&) {
        return -1;
    }
}
std::uint64_t hf_steps(void* e) { return static_cast<rcpg::Engine*>(e)->steps_done(); }
// the steps that a run's observer sees; their number
std::uint64_t hf_run(void* e, std::uint64_t interval, std::uint64_t* steps, std::uint64_t cap) {
    std::uint64_t n = 0;
    std::vector<rcpg::TraceSample> trace;
    try {
        static_cast<rcpg::Engine*>(e)->run(
            interval, true, interval,
            [&](const rcpg::Observation& o, const std::vector<double>*) {
                if (n < cap) steps[n] = o.step;
                ++n;
                fk.observer_device = fk.observer_device == -1 || fk.observer_device == current_device ? current_device : -2;
            },
            &trace);
    } catch (const std::exception&) {
        return 0;
    }
    if (trace.size() != n) return 0;
    return n;
}
int hf_result(void* e, double* x0) {
    try {
        rcpg::EngineResult r = static_cast<rcpg::Engine*>(e)->result();
        *x0 = r.positions[0];
        return 0;
    } catch (const std::exception&) {
        return -1;
    }
}
}
