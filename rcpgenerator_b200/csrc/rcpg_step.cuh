// Device code of one packing step shared by the kernels of the step graph
// (rcpg_kernels.cu) and the cluster kernel of small packings (rcpg_small.cu):
// the cell grid of a build, the row search, the pair terms of a row, the
// history windows of the controller.
#pragma once

#include <cuda_runtime.h>

#include <cstdint>
#include <type_traits>

#include "rcpg_device.h"
#include "rcpg_devutil.cuh"

namespace rcpg {
namespace {

// The cell grids of a build (one thread): per size class as many cells as fit
// with at least one largest-member cutoff each, coarsened until all fit
// C_alloc; resets what a build reports. c0 = cells of class 0's grid.
__device__ inline void plan_grid(DevCtl* ctl, int nd, std::uint32_t C_alloc, double& c0) {
    const int K = ctl->nclass > 1 ? ctl->nclass : 1;
    // per class: cells at least one largest-member cutoff wide
    long long nc[kMaxClass][kMaxDim];
    double cells_k[kMaxClass];
    double total = 0.0;
    for (int k = 0; k < K; ++k) {
        const double dmax = K > 1 ? xmul(ctl->class_d0max[k], ctl->build_kappa) : ctl->build_Dmax;
        const double cutoff = (dmax + ctl->build_t_shell) * (1.0 + 1e-6);
        cells_k[k] = 1.0;
        for (int d = 0; d < nd; ++d) {
            double q = floor(ctl->g.box[d] / cutoff);
            if (!(q >= 1.0)) q = 1.0;
            if (q > 1048576.0) q = 1048576.0;
            nc[k][d] = static_cast<long long>(q);
            cells_k[k] *= q;
        }
        total += cells_k[k];
    }
    // coarsen the class with the most cells until all fit
    while (total > static_cast<double>(C_alloc)) {
        int km = 0;
        for (int k = 1; k < K; ++k)
            if (cells_k[k] > cells_k[km]) km = k;
        int dm = 0;
        for (int d = 1; d < nd; ++d)
            if (nc[km][d] > nc[km][dm]) dm = d;
        const long long nn = (nc[km][dm] * 3) / 4;
        total -= cells_k[km];
        cells_k[km] = cells_k[km] / static_cast<double>(nc[km][dm]) * static_cast<double>(nn < 1 ? 1 : nn);
        total += cells_k[km];
        nc[km][dm] = nn < 1 ? 1 : nn;
        if (cells_k[km] <= 1.0 && total > static_cast<double>(C_alloc)) break;
    }
    std::uint32_t cells = 0;
    for (int k = 0; k < K; ++k) {
        ctl->cls_base[k] = cells;
        std::uint32_t ck = 1;
        for (int d = 0; d < nd; ++d) {
            ctl->cls_ncell[k][d] = static_cast<int>(nc[k][d]);
            ctl->cls_scale[k][d] = static_cast<double>(nc[k][d]) / ctl->g.box[d];
            ck *= static_cast<std::uint32_t>(nc[k][d]);
        }
        cells += ck;
    }
    ctl->cls_base[K] = cells;
    for (int d = 0; d < nd; ++d) {
        ctl->ncell[d] = ctl->cls_ncell[0][d];
        ctl->cell_scale[d] = ctl->cls_scale[0][d];
    }
    ctl->ncells = cells;
    c0 = cells_k[0];
    // every build re-anchors every particle
    ctl->kappa_min = ctl->build_kappa;
    ctl->row_need = 0u;
    ctl->stray = 0u;
    ctl->nbuilds += 1u;
}

// Cell of a particle in its size class's grid.
template <int ND>
__device__ __forceinline__ std::uint32_t bin_cell(const DevCtl* ctl, const double* x, double D0) {
    int k = 0;  // size class
    while (k + 1 < ctl->nclass && D0 >= ctl->class_d0[k + 1]) ++k;
    std::uint32_t c = ctl->cls_base[k], mul = 1;
    RCPG_UNROLL
    for (int d = 0; d < ND; ++d) {
        const int cd = cell_coord(x[d], ctl->cls_scale[k][d], ctl->cls_ncell[k][d]);
        c += static_cast<std::uint32_t>(cd) * mul;
        mul *= static_cast<std::uint32_t>(ctl->cls_ncell[k][d]);
    }
    return c;
}

// FP32 search record of particle q (DevArrays::fpos). A coordinate outside the
// box (by more than a millionth of it) becomes NaN, which fails no FP32 test of
// k_build_rows, and DevCtl::stray keeps its geometric pruning off: such a
// particle sits in a boundary cell that its position does not belong to.
template <int ND>
__device__ __forceinline__ void store_search_record(float* fpos, const DevCtl* ctl, std::uint32_t* stray,
                                                    std::uint64_t q, const double* x, double D0) {
    constexpr int FP = search_stride(ND);
    float r[FP];
    RCPG_UNROLL
    for (int d = 0; d < FP; ++d) r[d] = 0.0f;
    bool inside = true;
    RCPG_UNROLL
    for (int d = 0; d < ND; ++d) {
        const double L = ctl->g.box[d];
        const bool in = x[d] >= -1e-6 * L && x[d] <= (1.0 + 1e-6) * L;
        r[d] = in ? static_cast<float>(x[d]) : __int_as_float(0x7fffffff);
        inside = inside && in;
    }
    if (!inside) *stray = 1u;
    r[ND] = static_cast<float>(xmul(D0, ctl->build_kappa));
    float4* dst = reinterpret_cast<float4*>(fpos + q * FP);
    RCPG_UNROLL
    for (int h = 0; h < FP / 4; ++h) dst[h] = make_float4(r[4 * h], r[4 * h + 1], r[4 * h + 2], r[4 * h + 3]);
}

// Row search of the graph engine (cell-order storage, rows in scan order):
// every build the cell-unit search does not take (ndim > 3, several size
// classes, small packings, narrow grids). Along axis 0 the neighbour cells of
// a particle are consecutive, so in cell-order storage their members are one
// contiguous range of particles (two where the range wraps): a particle scans
// nn_1 * nn_2 * ... such ranges per size class instead of nn_0 times as many
// cells.
//
// Two tests keep candidates away from the FP64 predicate. (1) A range whose
// cells lie farther from the particle than the largest cutoff to a member of
// their class is not visited, and the others are shortened to the cells within
// that cutoff (a ball touches a third to two thirds of the cells of its
// bounding cube in 3 and 4 dimensions, fewer where the particle is smaller
// than the grid's). (2) A candidate is tested in FP32 on its search record
// with the minimum image min(|t|, L - |t|): four instructions per axis, no
// branch and no round, where the FP64 predicate takes seven at half the rate.
// Both are widened past every rounding (kSearchRel, kSearchAbs), so neither
// drops a partner; the candidates left are listed in scan order in shared
// memory and tested by the FP64 predicate, densely.
//
// G lanes share a particle. G = 1: one thread walks the ranges in order
// (consecutive threads are neighbours in space, so their ranges overlap and
// stay in L1). G > 1: search_row_group(). The scan
// order -- size classes, then the cells with axis 0 fastest, then the
// members -- does not depend on G, so neither do the rows. row_lanes() picks G
// per size class: the particles of a class are consecutive, and those of a
// larger class have several times the candidates (one G for all classes left
// the few large particles of a power law running alone: 404 us against 212).
//
// Bound by instruction issue (about 20 ranges of 1 to 2 candidates per particle
// where cells hold half a particle) and, for small packings, by the latency of
// cell start -> record -> test. One B200, per build, against the
// warp-per-particle search over single cells in FP64 that it replaces: 3-D
// power law N = 300,007 790 -> 212 us; 4-D log-normal N = 12,001 255 -> 74 us
// early in the run.
constexpr int kRowThreads = 128;
constexpr int kRowList = 24;          // listed candidates per lane
constexpr int kSliceLanes = 8;        // groups up to this size deal out ranges, larger ones candidates
// In box sides: the FP32 rounding of a position, of t and of L - |t| is at most
// 1.2e-7 per axis (3.4e-7 in 8 dimensions), and positions may lie 1e-6 outside
// the box; relative: the sum of squares and the cutoff round by less than 1e-6.
constexpr float kSearchAbs = 3e-6f, kSearchRel = 1.000004f;
// In a box whose longest side is below this the FP32 squares may leave FP32's
// normal range: the absolute widening is worth at least 9e-12 of the squared
// side, 9e-42 here, and the squares' subnormal steps are 1.4e-45. An infinite
// side in the widening then lets every candidate and every range through.
constexpr float kSearchMinSide = 1e-15f;

template <int ND>
struct SearchRecord {
    float x[ND], D;
};

// NC: the records are not written by the running kernel (read-only loads)
template <int ND, bool NC>
__device__ __forceinline__ SearchRecord<ND> load_search_record(const float* fpos, std::uint32_t q) {
    constexpr int FP = search_stride(ND);
    float w[FP];
    const float4* p = reinterpret_cast<const float4*>(fpos + static_cast<std::uint64_t>(q) * FP);
    RCPG_UNROLL
    for (int h = 0; h < FP / 4; ++h) {
        const float4 v = NC ? __ldg(p + h) : p[h];
        w[4 * h] = v.x;
        w[4 * h + 1] = v.y;
        w[4 * h + 2] = v.z;
        w[4 * h + 3] = v.w;
    }
    SearchRecord<ND> r;
    RCPG_UNROLL
    for (int d = 0; d < ND; ++d) r.x[d] = w[d];
    r.D = w[ND];
    return r;
}

// FP32 test of candidate j for particle i: false only for a pair outside the
// shell. half_i = widened Di/2 + t.
template <int ND>
__device__ __forceinline__ bool maybe_partner(const SearchRecord<ND>& i, float half_i, const SearchRecord<ND>& j,
                                              const float* side) {
    float d2 = 0.0f;
    RCPG_UNROLL
    for (int d = 0; d < ND; ++d) {
        const float t = fabsf(j.x[d] - i.x[d]);
        const float m = fminf(t, side[d] - t);
        d2 = __fmaf_rn(m, m, d2);
    }
    const float rc = __fmaf_rn(j.D, 0.5f * kSearchRel, half_i);
    return !(d2 > rc * rc);
}

// The neighbourhood of particle (xi, Di) in the grid of size class kc: cells
// lo .. lo + nn - 1 per axis (periodic), nn_1 * nn_2 * ... ranges along axis 0.
template <int ND>
struct RowScan {
    int nc[ND], nn[ND], lo[ND];
    std::uint32_t base;
    int rows;
    float x[ND], cell[ND];  // position, cell width
    float rcut, rcut2;      // widened largest cutoff; infinite: no pruning

    __device__ __forceinline__ void open(const DevCtl* ctl, int kc, int K, double kap, double t_shell,
                                         const double* xi, double Di, const float* side, float widest, bool prune) {
        const double dmax = K > 1 ? xmul(ctl->class_d0max[kc], kap) : ctl->build_Dmax;
        const double rc = (Di + dmax) * 0.5 + t_shell;
        rows = 1;
        RCPG_UNROLL
        for (int d = 0; d < ND; ++d) {
            const double scale = ctl->cls_scale[kc][d];
            nc[d] = ctl->cls_ncell[kc][d];
            // cells per cutoff on this axis: 1 with one grid (cells are at
            // least one cutoff wide), computed per class otherwise
            double mm = 1.0;
            if (K > 1) {
                mm = ceil(rc * scale * (1.0 + 1e-6));
                if (!(mm >= 1.0)) mm = 1.0;
            }
            if (!(2.0 * mm + 1.0 <= static_cast<double>(nc[d]))) {
                nn[d] = nc[d];  // every cell of the axis, once
                lo[d] = 0;
            } else {
                const int m = static_cast<int>(mm);
                nn[d] = 2 * m + 1;
                lo[d] = cell_coord(xi[d], scale, nc[d]) - m;
            }
            if (d > 0) rows *= nn[d];
            x[d] = static_cast<float>(xi[d]);
            cell[d] = __fdividef(side[d], static_cast<float>(nc[d]));
        }
        base = ctl->cls_base[kc];
        rcut = prune ? __fmaf_rn(static_cast<float>(rc), kSearchRel * kSearchRel, 2.0f * kSearchAbs * widest) : HUGE_VALF;
        rcut2 = rcut * rcut;
    }
    // Cell k of axis d: its periodic index, and far2 plus its squared distance
    // on that axis from the particle.
    __device__ __forceinline__ float axis(int d, int k, const float* side, float far2, int& c) const {
        c = lo[d] + k;
        if (c < 0) c += nc[d];
        else if (c >= nc[d]) c -= nc[d];
        float t = fabsf(__fmaf_rn(static_cast<float>(c) + 0.5f, cell[d], -x[d]));
        t = fmaxf(fminf(t, side[d] - t) - 0.5f * cell[d], 0.0f);
        return __fmaf_rn(t, t, far2);
    }
    // The particle ranges [q0, q1), then [q2, q3), of the grid row that starts
    // at cell `row` and lies far2 away over the other axes (far2 <= rcut2); the
    // cells beyond the rest of the cutoff are left out.
    __device__ __forceinline__ void ranges(const std::uint32_t* cell_start, std::uint32_t row, float far2,
                                           const float* side, std::uint32_t& q0, std::uint32_t& q1,
                                           std::uint32_t& q2, std::uint32_t& q3) const {
        q0 = q1 = q2 = q3 = 0u;
        int b = lo[0], e = lo[0] + nn[0];
        if (nn[0] < nc[0] && rcut2 < HUGE_VALF) {
            const float r = sqrtf(rcut2 - far2);
            const float inv = __fdividef(static_cast<float>(nc[0]), side[0]);
            b = max(b, __float2int_rd((x[0] - r) * inv));
            e = min(e, __float2int_rd((x[0] + r) * inv) + 1);
            if (b >= e) return;
        }
        const std::uint32_t* cs = cell_start + base + row;
        if (b < 0 || e > nc[0]) {
            if (b >= nc[0] || e <= 0) {  // wholly beyond one end
                const int shift = e <= 0 ? nc[0] : -nc[0];
                b += shift;
                e += shift;
            } else {
                q2 = cs[0];
                q3 = cs[b < 0 ? e : e - nc[0]];
                if (b < 0) b += nc[0];
                e = nc[0];
            }
        }
        q0 = cs[b];
        q1 = cs[e];
    }
    // body(q0, q1, q2, q3) for every grid row within the cutoff, in order (axis 1 fastest)
    template <int D = ND - 1, typename Body>
    __device__ __forceinline__ void each_row(const std::uint32_t* cell_start, const float* side, const Body& body,
                                             std::uint32_t part = 0, float far2 = 0.0f) const {
        for (int k = 0; k < nn[D]; ++k) {
            int c;
            const float f = axis(D, k, side, far2, c);
            if (f > rcut2) continue;
            const std::uint32_t row = (part + static_cast<std::uint32_t>(c)) * static_cast<std::uint32_t>(nc[D - 1]);
            if constexpr (D == 1) {
                std::uint32_t q0, q1, q2, q3;
                ranges(cell_start, row, f, side, q0, q1, q2, q3);
                body(q0, q1, q2, q3);
            } else {
                each_row<D - 1>(cell_start, side, body, row, f);
            }
        }
    }
    // the ranges of row number r in that order (empty beyond the cutoff)
    __device__ __forceinline__ void row_ranges(int r, const std::uint32_t* cell_start, const float* side,
                                               std::uint32_t& q0, std::uint32_t& q1, std::uint32_t& q2,
                                               std::uint32_t& q3) const {
        int off[ND];
        RCPG_UNROLL
        for (int d = 1; d < ND; ++d) {
            const int up = static_cast<int>((static_cast<float>(r) + 0.5f) * __frcp_rn(static_cast<float>(nn[d])));
            off[d] = r - up * nn[d];
            r = up;
        }
        std::uint32_t row = 0;
        float f = 0.0f;
        RCPG_UNROLL
        for (int d = ND - 1; d > 0; --d) {
            int c;
            f = axis(d, off[d], side, f, c);
            row = (row + static_cast<std::uint32_t>(c)) * static_cast<std::uint32_t>(nc[d - 1]);
        }
        q0 = q1 = q2 = q3 = 0u;
        if (!(f > rcut2)) ranges(cell_start, row, f, side, q0, q1, q2, q3);
    }
};

// The row's end: capacity checks and the published length (as in k_cells).
template <int ND>
__device__ __forceinline__ void close_row(const DevArrays& a, DevCtl* ctl, std::uint32_t t, std::uint32_t n) {
    const std::uint64_t N = a.N;
    const std::uint32_t cap = a.caps[t];
    if (n > cap && n <= a.S) {
        // the reference's capacity check counts the partners after t in its own
        // order; a row that fits the capacity in full needs no count
        const std::uint32_t rt = a.ref_rank[t];
        std::uint32_t n_half = 0;
        for (std::uint32_t k = 0; k < n; ++k)
            n_half += a.ref_rank[a.nbr[static_cast<std::uint64_t>(k) * N + t]] > rt;
        if (n_half > cap) report_cap_error(ctl, rt, cap);
    }
    a.nbr_cnt[t] = n > a.S ? 0u : n;  // overflow: empty row, rebuilt after the capacity grows
}

// Lanes per particle of size class k, g0 those of the two smallest classes (for
// the second a thread per particle still measured faster: 212 us against 247).
__device__ __forceinline__ int row_lanes(int g0, int k) {
    const int g = k <= 1 ? g0 : (2 * g0) << (k < 6 ? k - 1 : 5);
    return g < 32 ? g : 32;
}

// One particle's search state.
template <int ND, bool NC>
struct RowSearch {
    std::uint32_t t, n, listed;  // particle; row length and listed candidates so far
    double xi[ND], Di;
    SearchRecord<ND> ri;
    float half_i;

    __device__ __forceinline__ void begin(const DevArrays& a, std::uint32_t p, double kap, double t_shell, float widest) {
        t = p;
        n = listed = 0;
        double D0;
        load_pos<ND>(a.pos, t, xi, D0);
        Di = xmul(D0, kap);
        ri = load_search_record<ND, NC>(a.fpos, t);
        half_i = __fmaf_rn(__fmaf_rn(ri.D, 0.5f, static_cast<float>(t_shell)), kSearchRel, kSearchAbs * widest);
    }
    // FP64 predicate of listed candidate q
    __device__ __forceinline__ bool partner(const DevArrays& a, const DevCtl* ctl, std::uint32_t q, double kap,
                                            double t_shell) const {
        double xj[ND], D0j;
        if constexpr (NC) load_pos_g<ND>(a.pos, q, xj, D0j, 1);
        else load_pos<ND>(a.pos, q, xj, D0j);
        const double Dj = xmul(D0j, kap);
        return q != t && ((ND <= 3 || q > t) ? in_shell<ND>(xi, xj, Di, Dj, ctl->g.box, ctl->g.inv_box, t_shell)
                                             : in_shell<ND>(xi, xj, Dj, Di, ctl->g.box, ctl->g.inv_box, t_shell));
    }
};

// What every particle's search of one build shares.
template <int ND>
struct SearchParams {
    double kap, t_shell;
    int K;       // size classes
    bool prune;  // no particle lies outside the box
    float side[ND], widest;  // box sides; the longest, for the widening

    __device__ __forceinline__ void read(const DevCtl* ctl, bool in_box) {
        kap = ctl->build_kappa;
        t_shell = ctl->build_t_shell;
        K = ctl->nclass > 1 ? ctl->nclass : 1;
        prune = in_box;
        widest = 0.0f;
        RCPG_UNROLL
        for (int d = 0; d < ND; ++d) {
            side[d] = static_cast<float>(ctl->g.box[d]);
            widest = fmaxf(widest, side[d]);
        }
        if (widest < kSearchMinSide) widest = HUGE_VALF;
    }
};

// The row of particle t by one thread; list holds kRowList entries. Returns
// the row length (entries beyond a.S are counted, not stored).
template <int ND, bool NC>
__device__ __forceinline__ std::uint32_t search_row_one(const DevArrays& a, const DevCtl* ctl, const SearchParams<ND>& sp,
                                                        const std::uint32_t* cell_start, std::uint32_t t,
                                                        std::uint32_t* list) {
    const std::uint64_t N = a.N;
    const std::uint32_t S = a.S;
    const float* const fpos = a.fpos;
    RowSearch<ND, NC> rs;
    rs.begin(a, t, sp.kap, sp.t_shell, sp.widest);
    auto flush = [&]() {
        for (std::uint32_t k = 0; k < rs.listed; ++k) {
            const std::uint32_t q = list[k];
            if (rs.partner(a, ctl, q, sp.kap, sp.t_shell)) {
                if (rs.n < S) a.nbr[static_cast<std::uint64_t>(rs.n) * N + t] = q;
                ++rs.n;
            }
        }
        rs.listed = 0;
    };
    for (int kc = 0; kc < sp.K; ++kc) {
        RowScan<ND> sc;
        sc.open(ctl, kc, sp.K, sp.kap, sp.t_shell, rs.xi, rs.Di, sp.side, sp.widest, sp.prune);
        sc.each_row(cell_start, sp.side, [&](std::uint32_t q, std::uint32_t qe, std::uint32_t q2, std::uint32_t q3) {
            for (;;) {
                if (q >= qe) {  // the wrapped part of the range, then done
                    if (q2 >= q3) break;
                    q = q2;
                    qe = q3;
                    q2 = q3;
                }
                constexpr std::uint32_t U = 2;  // candidates in flight
                bool hit[U];
                RCPG_UNROLL
                for (std::uint32_t u = 0; u < U; ++u)
                    hit[u] = maybe_partner<ND>(rs.ri, rs.half_i,
                                               load_search_record<ND, NC>(fpos, min(q + u, qe - 1)), sp.side) &&
                             q + u < qe;
                RCPG_UNROLL
                for (std::uint32_t u = 0; u < U; ++u)
                    if (hit[u]) list[rs.listed++] = q + u;
                q += U;
                if (rs.listed > static_cast<std::uint32_t>(kRowList) - U) flush();
            }
        });
    }
    flush();
    return rs.n;
}

// Rows by the G lanes of a particle's group (a power of two, 2 to 32, aligned
// in the warp). All 32 lanes enter, groups without a particle with live =
// false: the loops run to the longest group of the warp and every vote and
// shuffle has the full mask, since votes on per-group masks run one group
// after the other. The three arrays are the warp's: 32 * (kRowList + 1) listed
// candidates, 64 range starts and 64 range ends.
//
// One size class by candidates: the ranges of G grid rows at a time are
// numbered by a scan over the lanes, each round tests G consecutive candidates.
template <int ND, bool NC>
__device__ __forceinline__ void search_class_group(const DevArrays& a, const DevCtl* ctl, const SearchParams<ND>& sp,
                                                   const std::uint32_t* cell_start, const RowScan<ND>& sc,
                                                   RowSearch<ND, NC>& rs, int G, std::uint32_t* s_list,
                                                   std::uint32_t* s_q, std::uint32_t* s_end) {
    constexpr unsigned kAll = 0xffffffffu;
    const std::uint64_t N = a.N;
    const std::uint32_t S = a.S;
    const float* const fpos = a.fpos;
    const int lane = threadIdx.x & 31;
    const int s = lane & (G - 1), first = lane & ~(G - 1);
    const unsigned group = kAll >> (32 - G), below = (1u << s) - 1u;
    const std::uint32_t L = static_cast<std::uint32_t>(kRowList * G);
    std::uint32_t* const list = s_list + first * kRowList;
    std::uint32_t* const sq = s_q + 2 * first;
    std::uint32_t* const se = s_end + 2 * first;
    rs.listed = 0;
    // partners among the listed candidates, appended to the row in order
    auto flush = [&]() {
        __syncwarp();
        const std::uint32_t most = __reduce_max_sync(kAll, rs.listed);
        for (std::uint32_t k0 = 0; k0 < most; k0 += 2 * G) {
            std::uint32_t q[2];
            bool ok[2];
            RCPG_UNROLL
            for (int u = 0; u < 2; ++u) {
                const std::uint32_t k = k0 + static_cast<std::uint32_t>(u * G + s);
                ok[u] = k < rs.listed;
                q[u] = ok[u] ? list[k] : rs.t;
            }
            RCPG_UNROLL
            for (int u = 0; u < 2; ++u) ok[u] = rs.partner(a, ctl, q[u], sp.kap, sp.t_shell) && ok[u];
            RCPG_UNROLL
            for (int u = 0; u < 2; ++u) {
                const unsigned hits = (__ballot_sync(kAll, ok[u]) >> first) & group;
                const std::uint32_t slot = rs.n + __popc(hits & below);
                if (ok[u] && slot < S) a.nbr[static_cast<std::uint64_t>(slot) * N + rs.t] = q[u];
                rs.n += static_cast<std::uint32_t>(__popc(hits));
            }
        }
        rs.listed = 0;
        __syncwarp();
    };
    const int most_rows = __reduce_max_sync(kAll, sc.rows);
    for (int r0 = 0; r0 < most_rows; r0 += G) {
        // the ranges of row r0 + s; numbers of the non-empty ranges and of their candidates
        std::uint32_t q0 = 0, q1 = 0, q2 = 0, q3 = 0;
        if (r0 + s < sc.rows) sc.row_ranges(r0 + s, cell_start, sp.side, q0, q1, q2, q3);
        const std::uint32_t n0 = q1 - q0, n1 = q3 - q2;
        std::uint32_t ci = n0 + n1, ei = (n0 != 0u) + (n1 != 0u);
        for (int o = 1; o < G; o <<= 1) {
            const std::uint32_t cv = __shfl_up_sync(kAll, ci, o, G), ev = __shfl_up_sync(kAll, ei, o, G);
            if (s >= o) {
                ci += cv;
                ei += ev;
            }
        }
        const std::uint32_t T = __shfl_sync(kAll, ci, G - 1, G);
        const std::uint32_t most = __reduce_max_sync(kAll, T);
        if (most == 0) continue;
        ci -= n0 + n1;
        ei -= (n0 != 0u) + (n1 != 0u);
        __syncwarp();  // the previous ranges are no longer read
        if (n0) {
            sq[ei] = q0 - ci;
            ci += n0;
            se[ei++] = ci;
        }
        if (n1) {
            sq[ei] = q2 - ci;
            se[ei] = ci + n1;
        }
        __syncwarp();
        // G consecutive candidates per round, U rounds in flight
        constexpr int U = 4;
        int e = 0;
        for (std::uint32_t k0 = 0; k0 < most; k0 += U * G) {
            if (__any_sync(kAll, rs.listed > L - U * G)) flush();
            std::uint32_t q[U];
            bool hit[U];
            RCPG_UNROLL
            for (int u = 0; u < U; ++u) {
                const std::uint32_t k = k0 + static_cast<std::uint32_t>(u * G + s);
                hit[u] = k < T;
                if (hit[u])
                    while (k >= se[e]) ++e;
                q[u] = hit[u] ? k + sq[e] : rs.t;
            }
            SearchRecord<ND> r[U];
            RCPG_UNROLL
            for (int u = 0; u < U; ++u) r[u] = load_search_record<ND, NC>(fpos, q[u]);
            RCPG_UNROLL
            for (int u = 0; u < U; ++u) {
                const unsigned hits =
                    (__ballot_sync(kAll, maybe_partner<ND>(rs.ri, rs.half_i, r[u], sp.side) && hit[u]) >> first) & group;
                if ((hits >> s) & 1u) list[rs.listed + __popc(hits & below)] = q[u];
                rs.listed += static_cast<std::uint32_t>(__popc(hits));
            }
        }
    }
    flush();
}

// The row of particle t by its group, each size class in one of two ways. Few
// ranges per lane (small groups): each lane walks its own slice of the class's
// ranges and keeps its partners in its own list, and the lists are appended in
// lane order; a list that overflows makes the warp repeat the class by
// candidates. Many lanes for few ranges: by candidates at once. Returns the
// row length in every lane of the group.
template <int ND, bool NC>
__device__ __forceinline__ std::uint32_t search_row_group(const DevArrays& a, const DevCtl* ctl,
                                                          const SearchParams<ND>& sp, const std::uint32_t* cell_start,
                                                          std::uint32_t t, bool live, int G, std::uint32_t* s_list,
                                                          std::uint32_t* s_q, std::uint32_t* s_end) {
    constexpr unsigned kAll = 0xffffffffu;
    const std::uint64_t N = a.N;
    const std::uint32_t S = a.S;
    const float* const fpos = a.fpos;
    const int lane = threadIdx.x & 31, s = lane & (G - 1);
    RowSearch<ND, NC> rs;
    rs.begin(a, live ? t : 0u, sp.kap, sp.t_shell, sp.widest);
    for (int kc = 0; kc < sp.K; ++kc) {
        RowScan<ND> sc;
        sc.open(ctl, kc, sp.K, sp.kap, sp.t_shell, rs.xi, rs.Di, sp.side, sp.widest, sp.prune);
        if (!live) sc.rows = 0;
        bool by_candidates = G > kSliceLanes;
        if (!by_candidates) {
            std::uint32_t* const list = s_list + lane * (kRowList + 1);
            std::uint32_t cnt = 0;
            const int r1 = sc.rows * (s + 1) / G;
            for (int r = sc.rows * s / G; r < r1; ++r) {
                std::uint32_t q, qe, q2, q3;
                sc.row_ranges(r, cell_start, sp.side, q, qe, q2, q3);
                for (;;) {
                    if (q >= qe) {  // the wrapped part of the range, then done
                        if (q2 >= q3) break;
                        q = q2;
                        qe = q3;
                        q2 = q3;
                    }
                    constexpr std::uint32_t U = 4;  // candidates in flight
                    SearchRecord<ND> rec[U];
                    RCPG_UNROLL
                    for (std::uint32_t u = 0; u < U; ++u) rec[u] = load_search_record<ND, NC>(fpos, min(q + u, qe - 1));
                    RCPG_UNROLL
                    for (std::uint32_t u = 0; u < U; ++u) {
                        if (q + u < qe && maybe_partner<ND>(rs.ri, rs.half_i, rec[u], sp.side)) {
                            if (cnt < static_cast<std::uint32_t>(kRowList)) list[cnt] = q + u;
                            ++cnt;
                        }
                    }
                    q += U;
                }
            }
            by_candidates = __any_sync(kAll, cnt > static_cast<std::uint32_t>(kRowList));
            if (!by_candidates) {
                std::uint32_t m = 0;  // partners kept
                for (std::uint32_t k = 0; k < cnt; k += 2) {
                    const std::uint32_t qa = list[k], qb = k + 1 < cnt ? list[k + 1] : qa;
                    const bool oa = rs.partner(a, ctl, qa, sp.kap, sp.t_shell);
                    const bool ob = rs.partner(a, ctl, qb, sp.kap, sp.t_shell) && k + 1 < cnt;
                    if (oa) list[m++] = qa;
                    if (ob) list[m++] = qb;
                }
                __syncwarp();
                std::uint32_t incl = m;
                for (int o = 1; o < G; o <<= 1) {
                    const std::uint32_t v = __shfl_up_sync(kAll, incl, o, G);
                    if (s >= o) incl += v;
                }
                for (std::uint32_t k = 0; k < m; ++k) {
                    const std::uint32_t slot = rs.n + incl - m + k;
                    if (slot < S) a.nbr[static_cast<std::uint64_t>(slot) * N + rs.t] = list[k];
                }
                rs.n += __shfl_sync(kAll, incl, G - 1, G);
            }
        }
        if (by_candidates) {
            __syncwarp();  // the lanes' lists are no longer read
            search_class_group<ND, NC>(a, ctl, sp, cell_start, sc, rs, G, s_list, s_q, s_end);
        }
    }
    __syncwarp();  // the group's first lane reads the row that all its lanes have stored (close_row)
    return rs.n;
}

// The pair terms of row slot t, particle (xi, D0i; Di = D0i * kap), over its n
// partners: the force in fi, summed in row order, and counted(j, terms) for
// every overlapping partner j. Partners in chunks of kChunk: the row ids and
// then the partner positions of a chunk are loaded before any of its
// arithmetic, so a thread keeps kChunk gathers in flight; the chunk's
// displacements and overlap tests come first (independent work), then the
// overlapping pairs' terms in row order. MX: FP32 terms, the force summed in
// FP32.
template <int ND, bool MX, typename Counted>
__device__ __forceinline__ void row_pairs(const DevArrays& a, std::uint64_t t, std::uint32_t n, const double* xi,
                                          double D0i, double Di, double kap, const double* bx, const double* inv_box,
                                          double* fi, Counted&& counted) {
    constexpr std::uint32_t kChunk = 4;
    const std::uint64_t N = a.N;
    float fif[ND], hbf[ND];
    double ibx[ND];
    RCPG_UNROLL
    for (int d = 0; d < ND; ++d) {
        fi[d] = 0.0;
        fif[d] = 0.0f;
        hbf[d] = static_cast<float>(0.5 * bx[d]);
        if constexpr (!MX) ibx[d] = inv_box[d];
    }
    const float kapf = static_cast<float>(kap);
    const float Dif = static_cast<float>(D0i) * kapf;
    for (std::uint32_t k0 = 0; k0 < n; k0 += kChunk) {
        std::uint32_t jj[kChunk];
        double xj[kChunk][ND], D0j[kChunk];
        RCPG_UNROLL
        for (std::uint32_t u = 0; u < kChunk; ++u)
            jj[u] = (k0 + u < n) ? __ldg(a.nbr + static_cast<std::uint64_t>(k0 + u) * N + t) : 0u;
        RCPG_UNROLL
        for (std::uint32_t u = 0; u < kChunk; ++u)
            if (k0 + u < n && jj[u] < N) load_pos_g<ND>(a.pos, jj[u], xj[u], D0j[u], 1);
        using PT = std::conditional_t<MX, float, double>;
        PT pdx[kChunk][ND], pd2[kChunk], pr[kChunk];
        bool pov[kChunk];
        RCPG_UNROLL
        for (std::uint32_t u = 0; u < kChunk; ++u) {
            const bool live = k0 + u < n && jj[u] < N;
            if (!live) {  // a defined record for the unused slots
                RCPG_UNROLL
                for (int d = 0; d < ND; ++d) xj[u][d] = xi[d];
                D0j[u] = 0.0;
            }
            if constexpr (MX) {
                pd2[u] = mixed_disp<ND>(xi, xj[u], bx, hbf, pdx[u]);
                pr[u] = mixed_rij(Dif, static_cast<float>(D0j[u]), kapf);
                pov[u] = live && pd2[u] < pr[u] * pr[u];
            } else {
                pr[u] = xmul(0.5, xadd(Di, xmul(D0j[u], kap)));
                pd2[u] = pair_disp<ND>(xi, xj[u], bx, ibx, pdx[u]);
                pov[u] = live && pd2[u] < xmul(pr[u], pr[u]);
            }
        }
        RCPG_UNROLL
        for (std::uint32_t u = 0; u < kChunk; ++u) {
            if (!pov[u]) continue;
            if constexpr (MX) {
                PairTermsF pf;
                pair_terms_mixed_f<ND>(pdx[u], pd2[u], pr[u], fif, pf);
                counted(jj[u], pf);
            } else {
                PairTerms pt;
                pair_terms_f64<ND>(pdx[u], pd2[u], pr[u], fi, pt);
                counted(jj[u], pt);
            }
        }
    }
    if constexpr (MX) {
        RCPG_UNROLL
        for (int d = 0; d < ND; ++d) fi[d] = static_cast<double>(fif[d]);
    }
}

// Window statistics of the histories for begin_step(step), computed by the
// whole block: sums in a fixed tree (graph mode; the host sums in order).
constexpr int kCtlThreads = 256;

// StepPre of the open step (time t, number steps), parts 0..2 by one thread each.
__device__ __forceinline__ void prepare_ahead(double t, std::uint64_t steps, const Histories& h, StepPre& p, int part) {
    if (part == 0) {
        p.pb1 = pow(0.9, t);
        p.inv_b1 = xdiv(1.0, xsub(1.0, p.pb1));
    } else if (part == 1) {
        p.pb2 = pow(0.999, t);
        p.inv_b2 = xdiv(1.0, xsub(1.0, p.pb2));
    } else if (part == 2) {
        const std::uint64_t step = steps + 1;
        p.boost = exp(xdiv(-static_cast<double>(step), 350.0));
        p.phi_250 = step > 251 ? h.phi[step - 250] : 0.0;
    }
}

// Whether begin_step(step) may read window statistics: the phi range while mu
// decays or the final oscillation phase waits for its tick, the force means
// where the learning-rate rule's other conditions hold (they read no windows).
__device__ __forceinline__ bool need_hist_stats(const Controller& c, const Histories& h, std::uint64_t step,
                                                const StepPre* ahead = nullptr) {
    if (step <= 250) return false;
    if (step >= c.mu_decay_next_tick && (c.mu_decay_active || c.osc_phase == OSC_FINAL)) return true;
    return step > 2500 && step - c.last_alpha_update > 500 && static_cast<double>(step) > xadd(c.mu_change, 500.0) &&
           xsub(c.phi, ahead ? ahead->phi_250 : h.phi[step - 250]) < 5e-4;
}

// by the first T threads of the block (which all threads enter)
template <int T>
__device__ void hist_stats_block(const Histories& h, std::uint64_t step, HistStats& out, double* red) {
    // (lo, hi) inclusive index ranges of the four force means
    const long long S = static_cast<long long>(step);
    const long long lo[4] = {S - 450, S - 75, S - 200, S - 3000};
    const long long hi[4] = {S - 250, S - 1, S - 1, S - 2500};
    double sum[4] = {0.0, 0.0, 0.0, 0.0};
    // a window whose start precedes step 1 wraps in the unsigned step
    // arithmetic of hist_mean, which then sums nothing: the same here
    RCPG_UNROLL
    for (int w = 0; w < 4; ++w)
        if (lo[w] >= 0 && threadIdx.x < T)
            for (long long k = lo[w] + threadIdx.x; k <= hi[w]; k += T) sum[w] = xadd(sum[w], h.force[k]);
    // phi range over [step - 250, step - 1)
    double mn = HUGE_VAL, mx = -HUGE_VAL;
    for (long long k = S - 250 + threadIdx.x; k < S - 1; k += T)
        if (k >= 0 && threadIdx.x < T) {
            mn = fmin(mn, h.phi[k]);
            mx = fmax(mx, h.phi[k]);
        }
    RCPG_UNROLL
    for (int o = 16; o > 0; o >>= 1) {
        RCPG_UNROLL
        for (int w = 0; w < 4; ++w) sum[w] = xadd(sum[w], __shfl_down_sync(0xffffffffu, sum[w], o));
        mn = fmin(mn, __shfl_down_sync(0xffffffffu, mn, o));
        mx = fmax(mx, __shfl_down_sync(0xffffffffu, mx, o));
    }
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = T / 32;
    if (lane == 0 && warp < nw) {
        RCPG_UNROLL
        for (int w = 0; w < 4; ++w) red[warp * 6 + w] = sum[w];
        red[warp * 6 + 4] = mn;
        red[warp * 6 + 5] = mx;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        for (int k = 1; k < nw; ++k) {
            RCPG_UNROLL
            for (int w = 0; w < 4; ++w) red[w] = xadd(red[w], red[k * 6 + w]);
            red[4] = fmin(red[4], red[k * 6 + 4]);
            red[5] = fmax(red[5], red[k * 6 + 5]);
        }
        // the divisors of hist_mean: end - start + 1 in unsigned step arithmetic
        const std::uint64_t u = step;
        out.f_450_250 = xdiv(red[0], static_cast<double>((u - 250) - (u - 450) + 1));
        out.f_75_1 = xdiv(red[1], static_cast<double>((u - 1) - (u - 75) + 1));
        out.f_200_1 = xdiv(red[2], static_cast<double>((u - 1) - (u - 200) + 1));
        out.f_3000_2500 = xdiv(red[3], static_cast<double>((u - 2500) - (u - 3000) + 1));
        out.phi_range_250 = xsub(red[5], red[4]);
    }
}

}  // namespace
}  // namespace rcpg
