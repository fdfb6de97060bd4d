// Steps of a small packing in one launch (graph mode): one thread-block
// cluster runs the whole loop -- build when triggered, forces, controller, ADAM
// + refresh trigger -- for up to a given number of steps, its phases separated
// by the hardware's cluster barriers instead of kernel launches.
//
// What it replaces: a step of the captured graph is four dependent kernels
// and two conditional nodes (37 us at N = 64 on one B200) and nine kernels
// more when it rebuilds (70 us at N = 2,000), each of which finds a
// handful of busy blocks, loads its parameters from memory again and waits
// for the last one to drain. The particles' arithmetic is a few microseconds of
// that. Here the control block and the cell offsets stay in shared memory
// (every block of the cluster keeps its own copy and runs the controller
// itself, on the same inputs, so no block waits for another one's result), and
// a step without a build has two cluster barriers.
//
// The results are the step graph's, bit for bit: the same device code
// computes grid, rows, pair terms and schedule (rcpg_step.cuh), and the sums
// are combined in the graph's order -- a warp's 32 particles by the shuffle
// tree, the eight warps of each 256 particles in order, those blocks by the
// controller's tree -- whichever block of the cluster computed them.
//
// Bound by latency: two barriers, the chain partner index -> record -> square
// root -> division of the longest row, and the controller's serial divisions;
// what is known earlier (bias corrections, boost) is computed beside them.
// Per step on one B200, set-up included, against the step graph of that time:
// N = 64 2-D 39.6 -> 9.3 us; N = 2,000 3-D, builds in three steps of four, 75 ->
// 33 us; a batch of 96 packings of up to 4,096 particles 2.7 times as fast.
// Where it runs: small_steps_ok, small_always, Engine::by_cluster.
//
// Work is dealt out by warps of 32 consecutive particles: warp w of the
// packing belongs to block w mod C. N <= kSmallN, so that a thread has at most
// one particle.
#include <cooperative_groups.h>
#include <cuda_runtime.h>

#include <cstdint>
#include <type_traits>

#include "rcpg_device.h"
#include "rcpg_devutil.cuh"
#include "rcpg_step.cuh"

namespace rcpg {

namespace cg = cooperative_groups;

namespace {

constexpr int kSmallThreads = 512;
constexpr int kSmallWarps = kSmallThreads / 32;
constexpr int kSmallBlocks = 16;                                  // most blocks of the cluster
constexpr int kSmallN = kSmallBlocks * kSmallThreads;             // 8,192 particles
constexpr int kSmallUnits = kSmallN / 32;                         // warps of particles
constexpr int kSmallSums = 9;                                     // sums per warp of particles
constexpr std::uint32_t kSmallCells = 12288;                      // cell offsets held in shared memory

// per pair: the force (up to 8 components), U, Lc, dk, Fm
constexpr int kTermFields = kMaxDim + 4;

struct SmallShared {
    DevCtl ctl;                               // this block's copy of the control block
    ForceSums total;
    StepPre ahead;                            // for the step being computed
    double hred[(kCtlThreads / 32) * 6];
    HistStats stats;
    std::uint32_t trigger[2];                 // some particle asks for a build (written by any block)
    std::uint32_t scan[kSmallWarps];
    std::uint32_t row_need, cap_error;        // as the last build left them
    int go, have_stats;
    // pair terms of a round (one column per lane), then each particle's sums
    double terms[kSmallWarps][kTermFields][33];
    double maxov[kSmallWarps][32];
    std::uint32_t npair[kSmallWarps][32];
    std::uint32_t list[kSmallWarps][32 * (kRowList + 1)];
    std::uint32_t sq[kSmallWarps][64], send[kSmallWarps][64];
    std::uint32_t cell_start[kSmallCells];
};

// Exclusive scan of the cell counts into this block's cell_start[0 .. n - 1].
__device__ void scan_cells(const std::uint32_t* count, std::uint32_t n, SmallShared& sh) {
    const std::uint32_t per = (n + kSmallThreads - 1) / kSmallThreads;
    const std::uint32_t c0 = threadIdx.x * per;
    for (std::uint32_t c = threadIdx.x; c < n; c += kSmallThreads) sh.cell_start[c] = __ldcg(count + c);
    __syncthreads();
    std::uint32_t sum = 0;
    for (std::uint32_t k = 0; k < per; ++k)
        if (c0 + k < n) sum += sh.cell_start[c0 + k];
    std::uint32_t total;
    std::uint32_t run = block_exclusive_scan<std::uint32_t>(sum, sh.scan, total);
    for (std::uint32_t k = 0; k < per; ++k)
        if (c0 + k < n) {
            const std::uint32_t v = sh.cell_start[c0 + k];
            sh.cell_start[c0 + k] = run;
            run += v;
        }
    __syncthreads();
}

__device__ __forceinline__ unsigned long long bits_of(double v) {
    return static_cast<unsigned long long>(__double_as_longlong(v));
}

// The pair sums of this block's particles (row_pairs, with `lanes` threads per
// particle and the same order of every sum): the force components, U, Lc, dk
// and Fm in sh.terms, sh.maxov, sh.npair at [warp of the particle][field][lane].
template <int ND, bool MX>
__device__ __forceinline__ void pair_sums(const DevArrays& b, const DevCtl* ctl, SmallShared& sh, int lanes,
                                          std::uint32_t rank, std::uint32_t C, std::uint32_t units) {
    using T = std::conditional_t<MX, float, double>;
    constexpr int NF = ND + 4;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int s = lane & (lanes - 1), first = lane & ~(lanes - 1);
    const std::uint32_t N = static_cast<std::uint32_t>(b.N);
    const std::uint32_t p = threadIdx.x / static_cast<std::uint32_t>(lanes);  // particle of the block
    const std::uint32_t t = (rank + (p >> 5) * C) * 32u + (p & 31u);
    const bool live = rank + (p >> 5) * C < units && t < N;
    double xi[ND], D0i = 0.0, bx[ND], ibx[ND];
    float hbf[ND];
    std::uint32_t n = 0;
    RCPG_UNROLL
    for (int d = 0; d < ND; ++d) {
        bx[d] = ctl->g.box[d];
        ibx[d] = ctl->g.inv_box[d];
        hbf[d] = static_cast<float>(0.5 * bx[d]);
        xi[d] = 0.0;
    }
    if (live) {
        load_pos<ND>(b.pos, t, xi, D0i);
        n = min(b.nbr_cnt[t], b.S);
    }
    const double kap = ctl->force_kappa;
    const double Di = xmul(D0i, kap);
    const float kapf = static_cast<float>(kap);
    const float Dif = static_cast<float>(D0i) * kapf;
    T sum[NF];  // sums s, s + lanes, s + 2 lanes, ... of the list (force, U, Lc, dk, Fm)
    RCPG_UNROLL
    for (int f = 0; f < NF; ++f) sum[f] = T(0);
    T maxov = T(0);
    std::uint32_t npair = 0;
    T* const out = reinterpret_cast<T*>(&sh.terms[warp][0][0]);
    auto row_id = [&](std::uint32_t k) -> std::uint32_t {
        return k < n ? b.nbr[static_cast<std::uint64_t>(k) * N + t] : 0xffffffffu;
    };
    const std::uint32_t most = __reduce_max_sync(0xffffffffu, n);
    // the next round's record and the row id after it are on their way while a round computes
    double xn[ND], D0n = 0.0;
    std::uint32_t jn = row_id(s), jnn = row_id(lanes + s);
    RCPG_UNROLL
    for (int d = 0; d < ND; ++d) xn[d] = xi[d];
    if (jn < N) load_pos<ND>(b.pos, jn, xn, D0n);
    for (std::uint32_t k0 = 0; k0 < most; k0 += lanes) {
        const std::uint32_t j = jn;
        const bool in = j < N;
        double xj[ND];
        const double D0j = D0n;
        RCPG_UNROLL
        for (int d = 0; d < ND; ++d) xj[d] = xn[d];
        jn = jnn;
        jnn = row_id(k0 + 2 * lanes + s);
        if (jn < N) load_pos<ND>(b.pos, jn, xn, D0n);
        T dx[ND], d2, r;
        if constexpr (MX) {
            d2 = mixed_disp<ND>(xi, xj, bx, hbf, dx);
            r = mixed_rij(Dif, static_cast<float>(D0j), kapf);
        } else {
            r = xmul(0.5, xadd(Di, xmul(D0j, kap)));
            d2 = pair_disp<ND>(xi, xj, bx, ibx, dx);
        }
        bool ov;
        if constexpr (MX) ov = in && d2 < r * r;
        else ov = in && d2 < xmul(r, r);
        const unsigned hits = __ballot_sync(0xffffffffu, ov);
        if (hits == 0u) continue;
        const unsigned upper = __ballot_sync(0xffffffffu, ov && j > t);
        if (ov) {
            // fields as T in columns of 33
            if constexpr (MX) {
                PairTermsF pf;
                float none[ND];
                RCPG_UNROLL
                for (int d = 0; d < ND; ++d) none[d] = 0.0f;
                pair_terms_mixed_f<ND>(dx, d2, r, none, pf);
                RCPG_UNROLL
                for (int d = 0; d < ND; ++d) out[33 * d + lane] = dx[d];
                out[33 * ND + lane] = pf.U;
                out[33 * (ND + 1) + lane] = pf.Lc;
                out[33 * (ND + 2) + lane] = pf.gap;
                out[33 * (ND + 3) + lane] = pf.Fm;
            } else {
                PairTerms pt;
                pair_scalars_f64(d2, r, pt);
                RCPG_UNROLL
                for (int d = 0; d < ND; ++d) out[33 * d + lane] = xmul(pt.Fm, dx[d]);
                out[33 * ND + lane] = pt.U;
                out[33 * (ND + 1) + lane] = pt.Lc;
                out[33 * (ND + 2) + lane] = pt.dk;
                out[33 * (ND + 3) + lane] = pt.Fm;
            }
        }
        __syncwarp();
        // the group's overlapping pairs in order, each lane its sums
        unsigned todo = (hits >> first) & (0xffffffffu >> (32 - lanes));
        while (todo) {
            const int q = first + __ffs(todo) - 1;
            todo &= todo - 1u;
            const bool up = ((upper >> q) & 1u) != 0u;
            RCPG_UNROLL
            for (int f = 0; f < NF; ++f) {
                if ((f & (lanes - 1)) != s || (f >= ND && !up)) continue;
                const T v = out[33 * f + q];
                if constexpr (MX) {
                    if (f < ND) sum[f] = __fmaf_rn(out[33 * (ND + 3) + q], v, sum[f]);
                    else if (f == ND + 2) sum[f] = mixed_add_dk(sum[f], out[33 * (ND + 1) + q], v);
                    else sum[f] += v;
                } else {
                    sum[f] = xadd(sum[f], v);
                }
            }
            if (up && s == 0) {
                const T u = out[33 * ND + q];
                maxov = MX ? static_cast<T>(fmaxf(static_cast<float>(maxov), static_cast<float>(u)))
                           : static_cast<T>(fmax(static_cast<double>(maxov), static_cast<double>(u)));
                ++npair;
            }
        }
        __syncwarp();
    }
    __syncthreads();  // sh.terms now takes the particles' sums
    if (live) {
        const int pw = static_cast<int>(p >> 5), pl = static_cast<int>(p & 31u);
        RCPG_UNROLL
        for (int f = 0; f < NF; ++f)
            if ((f & (lanes - 1)) == s) sh.terms[pw][f][pl] = static_cast<double>(sum[f]);
        if (s == 0) {
            sh.maxov[pw][pl] = static_cast<double>(maxov);
            sh.npair[pw][pl] = npair;
        }
    }
}

template <int ND>
__global__ void __launch_bounds__(kSmallThreads, 1) k_small_steps(DevArrays a, std::uint32_t steps, int lanes) {
    extern __shared__ __align__(16) unsigned char small_smem[];
    SmallShared& sh = *reinterpret_cast<SmallShared*>(small_smem);
    cg::cluster_group cluster = cg::this_cluster();
    const std::uint32_t C = cluster.num_blocks(), rank = cluster.block_rank();
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const std::uint32_t N = static_cast<std::uint32_t>(a.N);
    const std::uint32_t units = (N + 31) / 32;
    // the particle of this thread in the forces and the ADAM step: warp w of
    // this block holds particles 32 u .. 32 u + 31, u = rank + w C
    const std::uint32_t unit = rank + static_cast<std::uint32_t>(warp) * C;
    const std::uint32_t i = unit * 32u + static_cast<std::uint32_t>(lane);
    const bool mine = unit < units && i < N;
    DevCtl* const g = a.ctl;
    DevCtl* const ctl = &sh.ctl;
    // the warps' sums of a step, [sum][warp of the packing] (through L2: eight
    // times as fast here as loads from the other blocks' shared memory)
    unsigned long long* const sums = reinterpret_cast<unsigned long long*>(a.block_sums);
    static_assert(kSmallSums * kSmallUnits * 8 <= 4096 * sizeof(ForceSums), "room in the block sums");
    static_assert(sizeof(DevCtl) % 8 == 0, "control block copied by 8-byte words");
    {
        const unsigned long long* src = reinterpret_cast<const unsigned long long*>(g);
        unsigned long long* dst = reinterpret_cast<unsigned long long*>(ctl);
        for (int w = tid; w < static_cast<int>(sizeof(DevCtl) / 8); w += kSmallThreads) dst[w] = src[w];
    }
    if (tid == 0) {
        sh.trigger[0] = sh.trigger[1] = 0u;
        sums_zero(sh.total);  // the wall terms join the pair sums: their own stay zero
    }
    __syncthreads();
    if (lane == 0) prepare_ahead(ctl->c.t, ctl->c.steps, a.hist, sh.ahead, kSmallWarps - 1 - warp);
    if (ctl->stopped | ctl->halted) return;  // the same in every block
    cluster.sync();             // every block has read the control block and cleared its flags
    for (std::uint32_t it = 0; it < steps; ++it) {
        DevArrays b = bound_arrays(a, ctl->buf);
        const bool build = ctl->rebuild_flag != 0u;
        if (build) {
            // ---- neighbour build (k_build_prepare .. k_build_rows) ----------
            if (tid == 0) {
                double c0;
                plan_grid(ctl, ND, a.C_alloc, c0);
                ctl->forces_done = 0u;
                if (rank == 0) {
                    g->row_need = 0u;
                    g->stray = 0u;
                }
            }
            __syncthreads();
            const std::uint32_t ncells = ctl->ncells;
            double x[ND], D0 = 0.0;
            std::uint32_t cell = 0, arrival = 0;
            if (mine) {
                load_pos<ND>(b.pos, i, x, D0);
                cell = bin_cell<ND>(ctl, x, D0);
                arrival = atomicAdd(&a.cell_count[cell], 1u);
            }
            cluster.sync();
            scan_cells(a.cell_count, ncells + 1, sh);
            double ms[ND], vs[ND];
            std::uint64_t origin = 0;
            std::uint32_t cap = 0, ref = 0;
            if (mine) {
                a.cell_list[sh.cell_start[cell] + arrival] = i;
                RCPG_UNROLL
                for (int d = 0; d < ND; ++d) {
                    ms[d] = b.m[static_cast<std::uint64_t>(i) * ND + d];
                    vs[d] = b.v[static_cast<std::uint64_t>(i) * ND + d];
                }
                origin = b.origin[i];
                cap = b.caps[i];
                ref = b.ref_rank[i];
            }
            cluster.sync();
            // the particle's place in cell order: its cell's members in
            // ascending order of their present index. The state moves to the
            // other buffer set, the search record is written.
            {
                const DevArrays dst = bound_arrays(a, ctl->buf ^ 1u);
                if (mine) {
                    const std::uint32_t q0 = sh.cell_start[cell], q1 = sh.cell_start[cell + 1];
                    std::uint32_t q = q0;
                    for (std::uint32_t k = q0; k < q1; ++k) q += __ldcg(a.cell_list + k) < i;
                    store_pos<ND>(dst.pos, q, x, D0);
                    RCPG_UNROLL
                    for (int d = 0; d < ND; ++d) {
                        a.x_last[static_cast<std::uint64_t>(q) * ND + d] = x[d];
                        dst.m[static_cast<std::uint64_t>(q) * ND + d] = ms[d];
                        dst.v[static_cast<std::uint64_t>(q) * ND + d] = vs[d];
                    }
                    dst.origin[q] = origin;
                    dst.caps[q] = cap;
                    dst.ref_rank[q] = ref;
                    store_search_record<ND>(a.fpos, ctl, &g->stray, q, x, D0);
                }
                // the counts clear again for the next build
                for (std::uint32_t c = rank * kSmallThreads + tid; c <= ncells; c += C * kSmallThreads)
                    a.cell_count[c] = 0u;
            }
            cluster.sync();
            if (tid == 0) {
                ctl->buf ^= 1u;
                ctl->rebuild_flag = 1u;
            }
            __syncthreads();
            b = bound_arrays(a, ctl->buf);
            // rows of this block's particles, `lanes` threads each
            {
                SearchParams<ND> sp;
                sp.read(ctl, *reinterpret_cast<volatile std::uint32_t*>(&g->stray) == 0u);
                const std::uint32_t own = ((units + C - 1 - rank) / C) * 32u;  // particles of this block's warps
                const std::uint32_t per = kSmallThreads / static_cast<std::uint32_t>(lanes);
                std::uint32_t need = 0;
                for (std::uint32_t p0 = 0; p0 < own; p0 += per) {
                    __syncwarp();
                    const std::uint32_t p = p0 + static_cast<std::uint32_t>(tid / lanes);
                    const std::uint32_t t = (rank + (p >> 5) * C) * 32u + (p & 31u);
                    const bool live = p < own && t < N;
                    if (lanes == 1) {
                        if (!live) continue;
                        const std::uint32_t n =
                            search_row_one<ND, false>(b, ctl, sp, sh.cell_start, t, sh.list[warp] + lane * (kRowList + 1));
                        close_row<ND>(b, g, t, n);
                        need = max(need, n);
                    } else {
                        const std::uint32_t n = search_row_group<ND, false>(b, ctl, sp, sh.cell_start, t, live, lanes,
                                                                            sh.list[warp], sh.sq[warp], sh.send[warp]);
                        if (live && (lane & (lanes - 1)) == 0) close_row<ND>(b, g, t, n);
                        need = max(need, n);
                    }
                }
                need = __reduce_max_sync(0xffffffffu, need);
                if (lane == 0 && need) atomicMax(&g->row_need, need);
            }
            __syncthreads();
        }
        // ---- forces (k_forces) ---------------------------------------------
        // `lanes` threads per particle: each computes the terms of every
        // lanes-th partner (an FP64 square root and two divisions, about 350
        // cycles that nothing in the thread can overlap) and adds up some of
        // the sums over all partners, in row order, from the terms that the
        // group's lanes leave in shared memory
        if (ctl->pair_fp32) pair_sums<ND, true>(b, ctl, sh, lanes, rank, C, units);
        else pair_sums<ND, false>(b, ctl, sh, lanes, rank, C, units);
        double xi[ND], D0i = 0.0, fi[ND], mi[ND], vi[ND], xl[ND];
        if (mine) {
            load_pos<ND>(b.pos, i, xi, D0i);
            RCPG_UNROLL
            for (int d = 0; d < ND; ++d) {  // for the ADAM step
                mi[d] = b.m[static_cast<std::uint64_t>(i) * ND + d];
                vi[d] = b.v[static_cast<std::uint64_t>(i) * ND + d];
                xl[d] = a.x_last[static_cast<std::uint64_t>(i) * ND + d];
            }
        }
        __syncthreads();
        {
            ForceSums s;
            sums_zero(s);
            if (mine) {
                const double* col = &sh.terms[warp][0][lane];
                RCPG_UNROLL
                for (int d = 0; d < ND; ++d) fi[d] = col[33 * d];
                // (adding to zero, as k_forces adds to its running sums: -0 becomes 0)
                s.pair_U = xadd(0.0, col[33 * ND]);
                s.pair_Lc = xadd(0.0, col[33 * (ND + 1)]);
                s.pair_dk = xadd(0.0, col[33 * (ND + 2)]);
                s.pair_Fm = xadd(0.0, col[33 * (ND + 3)]);
                s.pair_maxov = sh.maxov[warp][lane];
                const double Di = xmul(D0i, ctl->force_kappa);
                std::uint32_t wc = 0;
                wall_forces<ND>(xi, Di, ctl->g, fi, s.pair_U, s.pair_dk, s.pair_Fm, wc);
                s.pair_count = sh.npair[warp][lane] + wc;
                const double f2 = force_norm2<ND>(fi);
                if (f2 > 1.0E-16) {
                    s.sum_mag = xsqrt(f2);
                    s.mag_count = 1ull;
                }
                s.sum_D = Di;
                RCPG_UNROLL
                for (int d = 0; d < ND; ++d) a.F[static_cast<std::uint64_t>(i) * ND + d] = fi[d];
            }
            if (unit < units) {
                warp_reduce_sums(s);
                if (lane == 0) {
                    unsigned long long* w = sums + unit;
                    w[0 * kSmallUnits] = bits_of(s.pair_U);
                    w[1 * kSmallUnits] = bits_of(s.pair_Lc);
                    w[2 * kSmallUnits] = bits_of(s.pair_dk);
                    w[3 * kSmallUnits] = bits_of(s.pair_Fm);
                    w[4 * kSmallUnits] = bits_of(s.pair_maxov);
                    w[5 * kSmallUnits] = bits_of(s.sum_mag);
                    w[6 * kSmallUnits] = bits_of(s.sum_D);
                    w[7 * kSmallUnits] = s.pair_count;
                    w[8 * kSmallUnits] = s.mag_count;
                }
            }
        }
        cluster.sync();
        // ---- controller (k_controller), in every block ----------------------
        {
            if (tid == kSmallThreads - 1) {
                sh.row_need = build ? *reinterpret_cast<volatile std::uint32_t*>(&g->row_need) : ctl->row_need;
                sh.cap_error = build ? *reinterpret_cast<volatile std::uint32_t*>(&g->cap_error) : ctl->cap_error;
            }
            // one warp per sum: lane k takes the eight warps of the particles
            // 256 k .. 256 k + 255 in order, then the controller's tree over
            // the lanes (absent warps and blocks add zero)
            if (warp < kSmallSums) {
                unsigned long long w[8];
                RCPG_UNROLL
                for (std::uint32_t k = 0; k < 8; ++k)
                    w[k] = 8u * lane + k < units ? __ldcg(sums + warp * kSmallUnits + 8 * lane + k) : 0ull;
                // members of ForceSums: pair_U, Lc, dk, Fm, maxov, sum_mag, sum_D, pair_count, mag_count
                const int f = warp < 5 ? warp : (warp < 7 ? warp + 3 : (warp == 7 ? 10 : 12));
                if (f >= 10) {
                    unsigned long long n = 0;
                    RCPG_UNROLL
                    for (int k = 0; k < 8; ++k) n += w[k];
                    RCPG_UNROLL
                    for (int o = 16; o > 0; o >>= 1) n += __shfl_down_sync(0xffffffffu, n, o);
                    if (lane == 0) reinterpret_cast<unsigned long long*>(&sh.total)[f] = n;
                } else {
                    double v = __longlong_as_double(static_cast<long long>(w[0]));
                    RCPG_UNROLL
                    for (int k = 1; k < 8; ++k) {
                        const double z = __longlong_as_double(static_cast<long long>(w[k]));
                        v = f == 4 ? fmax(v, z) : xadd(v, z);
                    }
                    v = f == 4 ? fmax(0.0, v) : xadd(0.0, v);  // the controller adds the block sums to zero
                    RCPG_UNROLL
                    for (int o = 16; o > 0; o >>= 1) {
                        const double z = shfl_down_d(v, o);
                        v = f == 4 ? fmax(v, z) : xadd(v, z);
                    }
                    v = f == 4 ? v : xadd(v, 0.0);
                    if (lane == 0) reinterpret_cast<double*>(&sh.total)[f] = v;
                }
            }
            __syncthreads();
            if (tid == 0) {
                Controller& c = ctl->c;
                bool go = true;
                ctl->sums = sh.total;
                ctl->nsum_blocks = (units + 7) / 8;
                ctl->pair_kernel_runs += 1ull;
                ctl->row_need = sh.row_need;
                ctl->cap_error = sh.cap_error;
                if (sh.row_need > a.S || sh.cap_error) {
                    ctl->halted = 1u;
                    ctl->adam_go = 0u;
                    go = false;
                } else {
                    StepScalars& sc = ctl->scal;
                    finalize_schedule(sh.total, ctl->force_mu, sc);
                    end_step(c, a.hist, sc, &sh.ahead);
                    if (ctl->pair_fp32 && sc.max_overlap > 0.0 && sc.max_overlap < ctl->mixed_switch) {
                        ctl->pair_fp32 = 0u;
                        ctl->fp64_switch_step = c.steps;
                    }
                    ctl->graph_steps += 1ull;
                    for (int d = 0; d < ND; ++d) ctl->adam_box[d] = c.box[d];
                    ctl->adam_alpha = c.adam_alpha;
                    ctl->adam_inv_b1 = c.inv_b1;
                    ctl->adam_inv_b2 = c.inv_b2;
                    ctl->adam_go = 1u;
                    ctl->fix_height_scale = 1.0;
                    if (c.steps + 1 > c.step_cap) {
                        ctl->stopped = 1u;
                        go = false;
                    }
                }
                sh.go = go ? 1 : 0;
            } else if (tid == 32) {
                // what is only reported (not after a halt, whose step is redone)
                if (!(sh.row_need > a.S || sh.cap_error)) {
                    finalize_report(sh.total, ND, ctl->scal);
                    end_step_report(ctl->c, a.hist, ctl->scal);
                }
            }
            __syncthreads();
            const std::uint64_t next = ctl->c.steps + 1;
            const bool stats = sh.go && need_hist_stats(ctl->c, a.hist, next, &sh.ahead);
            if (stats) hist_stats_block<kCtlThreads>(a.hist, next, sh.stats, sh.hred);
            if (tid == 0) sh.have_stats = stats ? 1 : 0;
            __syncthreads();
        }
        if (ctl->halted) break;
        // ---- ADAM step (k_adam_refresh); the last thread opens the next step
        // meanwhile (with fix_height first: the step's stretch comes from it)
        auto open_next = [&]() {
            if (tid != kSmallThreads - 1 || !sh.go) return;
            Controller& c = ctl->c;
            begin_step(c, a.hist, c.steps + 1, sh.have_stats ? &sh.stats : nullptr, &sh.ahead);
            ctl->fix_height_scale = c.reorder ? 1.0 : c.fix_height_scale;
            if (c.done || c.reorder || c.lock_now) ctl->stopped = 1u;
            else publish_step(ctl, c, ND, ctl->g.box, ctl->kappa_min);
        };
        const bool stretch = ctl->c.fix_height != 0;
        if (stretch) {
            open_next();
            __syncthreads();
        }
        if (mine) {
            RCPG_UNROLL
            for (int d = 0; d < ND; ++d) {
                const std::uint64_t e = static_cast<std::uint64_t>(i) * ND + d;
                xi[d] = adam_coord(fi[d], mi[d], vi[d], xi[d], ctl->adam_alpha, ctl->adam_inv_b1, ctl->adam_inv_b2,
                                   ctl->adam_box[d]);
                b.m[e] = mi[d];
                b.v[e] = vi[d];
            }
            if (stretch && ctl->fix_height_scale != 1.0) xi[ND - 1] = xmul(xi[ND - 1], ctl->fix_height_scale);
            store_pos<ND>(b.pos, i, xi, D0i);
        }
        if (!stretch) open_next();
        __syncthreads();
        // ---- refresh trigger -------------------------------------------------
        bool trig = false;
        if (mine && !ctl->stopped && ctl->c.rebuild_mode == REBUILD_CHECK) {
            double d2 = 0.0;
            RCPG_UNROLL
            for (int d = 0; d < ND; ++d) {
                const double dd = xsub(xi[d], xl[d]);
                d2 = xadd(d2, xmul(dd, dd));
            }
            trig = refresh_trigger(d2, xmul(D0i, ctl->refresh_kappa), xmul(D0i, ctl->kappa_min), ctl->theta);
        }
        // meanwhile, the parts of the next step's schedule that are known now
        if (lane == 0) prepare_ahead(ctl->c.t, ctl->c.steps, a.hist, sh.ahead, kSmallWarps - 1 - warp);
        const std::uint32_t par = it & 1u;
        if (__syncthreads_or(trig) && static_cast<std::uint32_t>(tid) < C)
            *cluster.map_shared_rank(&sh.trigger[par], tid) = 1u;
        cluster.sync();
        if (tid == 0) {
            if (sh.trigger[par]) ctl->rebuild_flag = 1u;
            sh.trigger[par] = 0u;  // next written two steps on, after two more barriers
        }
        __syncthreads();
        if (ctl->stopped) break;
    }
    cluster.sync();  // no block leaves while another reads its shared memory
    if (rank == 0) {
        if (tid == 0) {
            ctl->cap_error = *reinterpret_cast<volatile std::uint32_t*>(&g->cap_error);
            ctl->cap_error_key = *reinterpret_cast<volatile unsigned long long*>(&g->cap_error_key);
            ctl->stray = *reinterpret_cast<volatile std::uint32_t*>(&g->stray);
        }
        __syncthreads();
        const unsigned long long* src = reinterpret_cast<const unsigned long long*>(ctl);
        unsigned long long* dst = reinterpret_cast<unsigned long long*>(g);
        for (int w = tid; w < static_cast<int>(sizeof(DevCtl) / 8); w += kSmallThreads) dst[w] = src[w];
    }
}

// Blocks of the cluster: four warps of particles each as long as the cluster
// may grow, so that the build has several threads per particle.
int small_blocks(std::uint64_t N) {
    const std::uint64_t units = (N + 31) / 32;
    int C = 1;
    while (C < kSmallBlocks && static_cast<std::uint64_t>(C) * 4 < units) C *= 2;
    return C;
}

// Clusters of this packing's kernel that the device can hold at once (none
// where it has no room for one: a partitioned GPU, fewer multiprocessors or
// less shared memory); without `clusters`, up to `steps` steps launched.
template <int ND>
cudaError_t small_nd(const DevArrays& a, std::uint32_t steps, cudaStream_t st, int* clusters) {
    const int C = small_blocks(a.N);
    const std::uint64_t own = ((a.N + 31) / 32 + C - 1) / C * 32;  // particles per block
    int lanes = 1;
    while (lanes < 32 && own * static_cast<std::uint64_t>(lanes) * 2 <= kSmallThreads) lanes *= 2;
    cudaError_t e = cudaFuncSetAttribute(k_small_steps<ND>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         static_cast<int>(sizeof(SmallShared)));
    if (e == cudaSuccess) e = cudaFuncSetAttribute(k_small_steps<ND>, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
    if (e != cudaSuccess) return e;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(static_cast<unsigned>(C));
    cfg.blockDim = dim3(kSmallThreads);
    cfg.dynamicSmemBytes = sizeof(SmallShared);
    cfg.stream = st;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = static_cast<unsigned>(C);
    attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    if (clusters) return cudaOccupancyMaxActiveClusters(clusters, k_small_steps<ND>, &cfg);
    return cudaLaunchKernelEx(&cfg, k_small_steps<ND>, a, steps, lanes);
}

cudaError_t small_any(const DevArrays& a, std::uint32_t steps, cudaStream_t st, int* clusters) {
    switch (a.ndim) {
        case 2: return small_nd<2>(a, steps, st, clusters);
        case 3: return small_nd<3>(a, steps, st, clusters);
        case 4: return small_nd<4>(a, steps, st, clusters);
        case 5: return small_nd<5>(a, steps, st, clusters);
        case 6: return small_nd<6>(a, steps, st, clusters);
        case 7: return small_nd<7>(a, steps, st, clusters);
        case 8: return small_nd<8>(a, steps, st, clusters);
        default: return cudaErrorInvalidValue;
    }
}

}  // namespace

bool small_steps_ok(const DevArrays& a) {
    if (!a.permute || a.sorted_rows || a.N > static_cast<std::uint64_t>(kSmallN) || a.C_alloc + 1 > kSmallCells)
        return false;
    int clusters = 0;
    const cudaError_t e = small_any(a, 0, nullptr, &clusters);
    if (e != cudaSuccess) cudaGetLastError();  // the step graph runs instead
    return e == cudaSuccess && clusters > 0;
}

cudaError_t launch_small_steps(const DevArrays& a, std::uint32_t steps, cudaStream_t st) {
    return small_any(a, steps, st, nullptr);
}

}  // namespace rcpg
