// Host driver of one packing on one GPU.
#pragma once

#include <cuda_runtime.h>

#include <cstdint>
#include <cstdlib>
#include <functional>
#include <new>
#include <stdexcept>
#include <string>
#include <utility>
#include <vector>

#include "rcpg_device.h"
#include "rcpg_setup.h"

namespace rcpg {

struct Observation {
    std::uint64_t step;
    double phi, force_magnitude, energy, max_min_dist;
};

// A malloc'd array that a result can hand over (release) instead of copying.
template <typename T>
class HostArray {
public:
    HostArray() = default;
    HostArray(HostArray&& o) noexcept : p_(o.p_), n_(o.n_) { o.p_ = nullptr; o.n_ = 0; }
    HostArray& operator=(HostArray&& o) noexcept {
        std::swap(p_, o.p_);
        std::swap(n_, o.n_);
        return *this;
    }
    ~HostArray() { std::free(p_); }
    // n elements, not initialised
    void resize(std::size_t n) {
        std::free(p_);
        n_ = 0;
        p_ = static_cast<T*>(std::malloc(n * sizeof(T) + 1));
        if (!p_) throw std::bad_alloc();
        n_ = n;
    }
    T* data() { return p_; }
    const T* data() const { return p_; }
    std::size_t size() const { return n_; }
    T& operator[](std::size_t i) { return p_[i]; }
    const T* begin() const { return p_; }
    const T* end() const { return p_ + n_; }
    // the array, to be freed with std::free()
    T* release() {
        T* p = p_;
        p_ = nullptr;
        n_ = 0;
        return p;
    }

private:
    T* p_ = nullptr;
    std::size_t n_ = 0;
};

// PackingResult (rcp_generator.hpp:35-90) minus the research-only fields.
struct EngineResult {
    HostArray<double> positions;  // [N*ndim]
    HostArray<double> diameters;
    std::vector<double> box;
    std::vector<std::int8_t> walls;
    std::vector<double> phi_history, force_history, energy_history, max_overlap_history,
        mu_history, alpha_history;
    std::vector<std::int8_t> mu_flag_history;
    std::uint64_t steps = 0;
    double phi = 0.0, max_min_dist = 0.0, force_magnitude = 0.0;
    HostArray<std::uint64_t> particle_origin;
    // engine statistics
    std::uint64_t builds = 0;
    std::uint32_t row_capacity = 0;
    // mixed precision: step after which the pair terms were FP64 (0: never
    // switched), and the relative error of the final state's energy sum and
    // forces with FP32 pair terms against FP64 ones (NaN when not mixed)
    std::uint64_t fp64_switch_step = 0;
    double pair_energy_rel_error = 0.0, pair_force_rel_error = 0.0;
};

struct TraceSample {
    std::uint64_t step;
    std::vector<double> positions;  // [N*ndim]
    std::vector<double> diameters;
    double phi, force, energy, max_min_dist;
};

using ObserverFn = std::function<void(const Observation&, const std::vector<double>* positions)>;

struct DevCtl;
// pinned host copies of the control block, recycled across engines
// Stream-ordered device allocation from this library's pool of the current
// device (freed memory stays reserved for the next engine; free with cudaFreeAsync).
cudaError_t pool_alloc_async(void** p, std::size_t bytes, cudaStream_t st);
DevCtl* pinned_ctl_acquire();
void pinned_ctl_release(DevCtl* p);

// Size classes of the cell grids (one grid per doubling of D0 when
// max/min D0 > 2.5, else one grid) into h.nclass, class_d0, class_d0max.
void set_size_classes(const std::vector<double>& D0, DevCtl& h);

class EngineError : public std::runtime_error {
   public:
    EngineError(int code, const std::string& msg) : std::runtime_error(msg), code_(code) {}
    int code() const { return code_; }

   private:
    int code_;
};

// Makes a device current for its scope. Launches, allocations and events go to
// the current device, whatever the stream; an engine may be used from any
// thread, and its caller may have selected another device since.
class DeviceGuard {
   public:
    explicit DeviceGuard(int device) {
        cudaGetLastError();  // what the caller's own calls left is not the engine's error
        cudaError_t e = cudaGetDevice(&before_);
        if (e == cudaSuccess && before_ != device) {
            e = cudaSetDevice(device);
            switched_ = e == cudaSuccess;
        }
        if (e != cudaSuccess)
            throw EngineError(-2, std::string("rcpgenerator_b200: cannot select the engine's device: ") +
                                      cudaGetErrorString(e));
    }
    ~DeviceGuard() {
        if (switched_) cudaSetDevice(before_);
    }
    DeviceGuard(const DeviceGuard&) = delete;
    DeviceGuard& operator=(const DeviceGuard&) = delete;

   private:
    int before_ = 0;
    bool switched_ = false;
};

class Engine {
   public:
    explicit Engine(EngineInput in, cudaStream_t stream = nullptr);
    ~Engine();
    Engine(const Engine&) = delete;
    Engine& operator=(const Engine&) = delete;

    // Advance by at most max_new_steps steps (0 = to completion). Returns
    // true once the run is finished (converged or step cap).
    bool advance(std::uint64_t max_new_steps);
    // Run to completion with optional observation / trajectory capture.
    void run(std::uint64_t progress_interval, bool capture_positions,
             std::uint64_t trajectory_interval, const ObserverFn& observer,
             std::vector<TraceSample>* trace);
    EngineResult result();
    std::uint64_t steps_done() const { return host_c_.hist_filled; }
    bool finished() const { return finished_; }
    cudaStream_t stream() const { return st_; }
    std::uint64_t N() const { return N_; }
    int ndim() const { return ndim_; }
    // Kernel launches issued so far by this engine (the graph counts per node).
    std::uint64_t launches() const { return launches_; }
    std::uint64_t builds();
    // Times `reps` back-to-back launches of the pair-force kernel on the
    // current state (CUDA events on the engine stream); returns the average
    // duration and the kernel's algorithmic bytes per launch.
    void profile_pair_kernel(std::uint32_t reps, double* avg_ms, double* alg_bytes,
                             double* mean_row);
    // The same for the neighbour build's search (graph mode: the tiled build
    // with the step's forces fused), each launch after the binning stages of a
    // full rebuild of the current state and a cold L2. Leaves the rows rebuilt
    // for the current positions; the control block is restored.
    void profile_build_kernel(std::uint32_t reps, double* avg_ms, double* alg_bytes);
    // Mixed precision: the final state's forces evaluated with FP32 and with
    // FP64 pair terms on the same rows; relative difference of the pair
    // energy sum and max |F32 - F64| / max |F64|. Leaves the state unchanged.
    void pair_precision_error(double* energy_rel, double* force_rel);
    // Waits for the device by sleeping on a blocking event instead of spinning
    // (for many engines driven by more host threads than cores: a batch).
    void set_blocking_sync(bool on);
    // How many engines run at the same time (a batch): among many, what counts
    // is the share of the GPU that a step takes.
    void set_engines(std::uint64_t n) { engines_ = n; }
    // Later steps by the step graph also where the cluster kernel applies
    // (diagnostic: both give the same results bit for bit).
    void prefer_step_graph(bool on) { step_graph_ = on; }
    // Which way the step graph's later builds bring the particles into cell
    // order (diagnostic: the same state either way).
    void gather_builds(bool on) {
        a_.gather = on ? 1 : 0;
        destroy_graph();
    }

   private:
    void setup_host(EngineInput in);
    void alloc_device();
    void free_device();
    void upload_initial();
    void ensure_row_capacity(std::uint32_t need);
    void push_ctl();
    void pull_ctl();
    void publish_step_params();
    void do_reorder_and_rebuild();
    void do_target_lock(std::uint64_t step);
    void forces_and_reduce(bool exact_reduce);
    void finish_step_host();
    bool step_host();
    bool advance_graph(std::uint64_t max_new_steps);
    bool by_cluster(std::uint64_t always);
    void capture_graph();
    // steps of the captured graph: the largest divisor of graph_steps_ from 8 down
    // to 4, else the smallest one above 8 (fewer than 4 steps: all of them)
    int captured_steps() const;
    // one step of the step graph: gate, conditional build, pair-kernel switch,
    // controller, ADAM (kernels run only where the step needs them)
    void capture_step();
    template <typename Body>
    void add_conditional(int type, unsigned long long handle, unsigned size, Body body);
    std::uint64_t kernels_per_build() const;
    void destroy_graph();
    void handle_overflow_and_resume();
    // exact mode: the ADAM pass of the last finished step, if it is still due
    void apply_pending_adam();
    void after_stop();
    void observe(std::uint64_t step, bool capture, const ObserverFn& observer,
                 std::vector<TraceSample>* trace);
    void sample(Observation& ob, bool capture, std::vector<double>& xs, std::vector<TraceSample>* trace);
    void download_histories();
    // the current state in the reference's order: x [N*ndim], diameters D0 * kd
    // (D0 when fixed) [N], particle_origin [N] (optional)
    void download_particles(double kd, bool fixed, double* x, double* D, std::uint64_t* origin);
    void check(cudaError_t e, const char* what);

    // configuration
    std::uint64_t N_ = 0;
    int ndim_ = 0;
    int P_ = 0;
    bool exact_ = false;
    bool mixed_ = false;          // FP32 pair terms until the max overlap falls below mixed_switch_
    double mixed_switch_ = 1e-5;
    int graph_steps_ = 32;
    int device_ = 0;
    cudaStream_t st_ = nullptr;
    bool own_stream_ = false;
    std::uint32_t neighbor_max_ = 0;

    // host copies
    std::vector<double> x0_;          // initial positions (after setup scaling)
    std::vector<double> D0_;          // D0 after setup
    std::vector<std::uint32_t> caps_;
    std::vector<std::int8_t> walls_;
    Controller host_c_{};
    DevCtl hctl_{};
    std::vector<double> h_phi_, h_force_, h_energy_, h_maxov_, h_mu_, h_alpha_;
    std::vector<std::int8_t> h_muflag_;
    Histories hh_{};
    std::uint64_t hist_size_ = 0;
    bool histories_on_device_ = false;
    bool finished_ = false;
    bool adam_pending_ = false;   // exact mode: ADAM pass of the last finished step not yet applied
    std::uint64_t launches_ = 0;
    double initial_U_ = 0.0, initial_maxov_ = 0.0;

    // device
    DevArrays a_{};
    void* d_block_ = nullptr;
    std::vector<void*> allocs_;
    cudaGraphExec_t graph_exec_ = nullptr;
    cudaGraph_t graph_ = nullptr;
    bool small_ = false;       // graph mode: the cluster kernel can run the steps (small_steps_ok)
    bool step_graph_ = false;  // ... but is not asked to
    // by_cluster(): steps and builds since the last choice, and that choice
    std::uint64_t engines_ = 1, steps_seen_ = 0, builds_seen_ = 0;
    bool chosen_ = false, few_builds_ = false;
    std::uint64_t graph_nodes_per_step_ = 0;
    cudaStream_t body_st_ = nullptr;  // captures the bodies of the step graph's conditional nodes
    std::uint32_t* pinned_ = nullptr;
    DevCtl* hctl_pinned_ = nullptr;
    cudaEvent_t sync_ev_ = nullptr;  // blocking-sync event (set_blocking_sync)
};

}  // namespace rcpg
