// Overlap report of a packed state on the GPU: the pair-overlap diagnostic of
// the reference's analysis package (rcptools/overlap.py:7-113) -- candidate
// pairs i < j within 2 * R_max (its KD-tree query radius, overlap.py:53),
// minimum image by round-half-even of pos[i] - pos[j] over every axis when a
// box is given (overlap.py:63-65), overlap (r_i + r_j) - |d| > 0, fractions
// in the "sum" and "min" conventions (overlap.py:71-75).
//
// Cells at least 2 R_max wide (one grid). The state goes to the GPU once; the
// binning, the scans and the cell-order copy of the records run there (on the
// host, and twice, to size the output first, they were most of the call: 19.2
// -> 4.9 ms for a report of 200,003 particles with 583,000 overlapping pairs on
// one B200; what is left is bound by the copies of the state and of the result
// and by widening the result to the report's types). Then one thread per particle over the
// contiguous member ranges of its neighbour cells along axis 0, two passes:
// counts, then the pairs of each particle at its offset, sorted by j. Which
// arrival order a cell's members have does not matter to either.
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstdint>
#include <cstdio>
#include <string>
#include <vector>

#include "../../include/rcpg.h"
#include "rcpg_core.h"
#include "rcpg_engine.h"

namespace {

using rcpg::xadd;
using rcpg::xmul;
using rcpg::xsub;

constexpr int kOvMaxDim = 8;

struct OvGrid {
    int ndim;
    int periodic;
    int ncell[kOvMaxDim];
    double lo[kOvMaxDim], width[kOvMaxDim], box[kOvMaxDim];
    double near[kOvMaxDim];  // up to this difference a pair needs no image; -1: every pair takes the quotient
    double rq;               // candidate radius 2 R_max
};

// |x_i - x_j|^2 with the image removed, in the operation order of the
// reference's NumPy expression (no fused multiply-adds). Below 0.49 box
// lengths the rounded quotient is zero: no division (129 cycles in FP64). A
// zero or infinite side has no such range: 0 / 0 and 0 * inf are not numbers,
// which drops the pair.
template <int ND>
__device__ __forceinline__ double pair_dist2(const double* xi, const double* __restrict__ x, std::uint64_t q,
                                             const OvGrid& g) {
    double s = 0.0;
    RCPG_UNROLL
    for (int d = 0; d < ND; ++d) {
        double dd = xsub(xi[d], x[q * ND + d]);
        if (g.periodic && !(fabs(dd) <= g.near[d])) dd = xsub(dd, xmul(nearbyint(dd / g.box[d]), g.box[d]));
        s = xadd(s, xmul(dd, dd));
    }
    return s;
}

// cell of each particle and its arrival rank there
__global__ void __launch_bounds__(256) k_ov_bin(const double* __restrict__ x, std::uint64_t N, OvGrid g,
                                                std::uint32_t* __restrict__ cell_of, std::uint32_t* __restrict__ rank,
                                                std::uint32_t* __restrict__ count) {
    const std::uint64_t i = blockIdx.x * 256ull + threadIdx.x;
    if (i >= N) return;
    std::uint32_t c = 0, mul = 1;
    for (int d = 0; d < g.ndim; ++d) {
        double v = x[i * g.ndim + d] - g.lo[d];
        if (g.periodic) v -= floor(v / g.box[d]) * g.box[d];
        // cell index, clamped (a NaN from a zero box side goes to cell 0)
        const double q = floor(v / g.width[d]);
        long long k = 0;
        if (q >= static_cast<double>(g.ncell[d] - 1)) k = g.ncell[d] - 1;
        else if (q > 0.0) k = static_cast<long long>(q);
        c += static_cast<std::uint32_t>(k) * mul;
        mul *= static_cast<std::uint32_t>(g.ncell[d]);
    }
    cell_of[i] = c;
    rank[i] = atomicAdd(&count[c], 1u);
}

// the records in cell order
__global__ void __launch_bounds__(256) k_ov_scatter(const double* __restrict__ x, const double* __restrict__ D,
                                                    std::uint64_t N, int ndim, const std::uint32_t* __restrict__ cell_of,
                                                    const std::uint32_t* __restrict__ rank,
                                                    const std::uint32_t* __restrict__ start, double* __restrict__ sx,
                                                    double* __restrict__ sR, std::uint32_t* __restrict__ sid) {
    const std::uint64_t i = blockIdx.x * 256ull + threadIdx.x;
    if (i >= N) return;
    const std::uint64_t q = start[cell_of[i]] + rank[i];
    for (int d = 0; d < ndim; ++d) sx[q * ndim + d] = x[i * ndim + d];
    sR[q] = D[i] / 2.0;
    sid[q] = static_cast<std::uint32_t>(i);
}

// Exclusive scan in tiles of 2048; sums[tile] = the tile's total.
constexpr int kOvScanThreads = 256, kOvScanItems = 8, kOvTile = kOvScanThreads * kOvScanItems;

template <typename In, typename Out>
__global__ void __launch_bounds__(kOvScanThreads) k_ov_scan(const In* in, Out* out,
                                                            std::uint64_t n, Out* __restrict__ sums) {
    __shared__ Out s_warp[kOvScanThreads / 32];
    const std::uint64_t base = blockIdx.x * static_cast<std::uint64_t>(kOvTile) + threadIdx.x * kOvScanItems;
    Out v[kOvScanItems], sum = 0;
    RCPG_UNROLL
    for (int k = 0; k < kOvScanItems; ++k) {
        v[k] = base + k < n ? static_cast<Out>(in[base + k]) : Out(0);
        sum += v[k];
    }
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    Out incl = sum;
    RCPG_UNROLL
    for (int o = 1; o < 32; o <<= 1) {
        const Out y = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += y;
    }
    if (lane == 31) s_warp[warp] = incl;
    __syncthreads();
    Out off = incl - sum, total = 0;
    for (int w = 0; w < kOvScanThreads / 32; ++w) {
        off += w < warp ? s_warp[w] : Out(0);
        total += s_warp[w];
    }
    RCPG_UNROLL
    for (int k = 0; k < kOvScanItems; ++k) {
        if (base + k < n) out[base + k] = off;
        off += v[k];
    }
    if (threadIdx.x == 0 && sums) sums[blockIdx.x] = total;
}

template <typename Out>
__global__ void __launch_bounds__(kOvScanThreads) k_ov_scan_add(Out* __restrict__ out, std::uint64_t n,
                                                                const Out* __restrict__ offsets) {
    const Out add = offsets[blockIdx.x];
    const std::uint64_t base = blockIdx.x * static_cast<std::uint64_t>(kOvTile) + threadIdx.x;
    RCPG_UNROLL
    for (int k = 0; k < kOvScanItems; ++k) {
        const std::uint64_t e = base + static_cast<std::uint64_t>(k) * kOvScanThreads;
        if (e < n) out[e] += add;
    }
}

// elements of scratch that scan() needs for n values (all levels)
std::uint64_t scan_scratch(std::uint64_t n) {
    std::uint64_t t = 0;
    while (n > static_cast<std::uint64_t>(kOvTile)) {
        n = (n + kOvTile - 1) / kOvTile;
        t += n;
    }
    return t + 1;
}

// out = exclusive scan of in (n values); in may be out when the types agree
template <typename In, typename Out>
void scan(const In* in, Out* out, std::uint64_t n, Out* tmp, cudaStream_t st) {
    const std::uint64_t tiles = (n + kOvTile - 1) / kOvTile;
    k_ov_scan<In, Out><<<static_cast<unsigned>(tiles), kOvScanThreads, 0, st>>>(in, out, n, tiles > 1 ? tmp : nullptr);
    if (tiles <= 1) return;
    scan<Out, Out>(tmp, tmp, tiles, tmp + tiles, st);
    k_ov_scan_add<Out><<<static_cast<unsigned>(tiles), kOvScanThreads, 0, st>>>(out, n, tmp);
}

// PASS 0: counts (candidates into *ncand, overlaps per particle); PASS 1:
// writes the overlaps of i at off[i]. One thread per particle in cell order.
template <int ND, int PASS>
__global__ void __launch_bounds__(128) k_overlap(const double* __restrict__ sx, const double* __restrict__ sR,
                                                 const std::uint32_t* __restrict__ sid, std::uint64_t N, OvGrid g,
                                                 const std::uint32_t* __restrict__ cell_of,
                                                 const std::uint32_t* __restrict__ cell_start,
                                                 unsigned long long* __restrict__ ncand,
                                                 std::uint32_t* __restrict__ nov,
                                                 const unsigned long long* __restrict__ off,
                                                 std::uint32_t* __restrict__ pairs, double* __restrict__ fsum,
                                                 double* __restrict__ fmin_, unsigned long long capacity) {
    const std::uint64_t t = blockIdx.x * 128ull + threadIdx.x;
    unsigned long long cand = 0;
    if (t < N) {
        const std::uint32_t i = sid[t];
        double xi[ND];
        RCPG_UNROLL
        for (int d = 0; d < ND; ++d) xi[d] = sx[t * ND + d];
        const double Ri = sR[t];
        // the distinct neighbour cells: 1, 2 or 3 per axis
        int first[ND], span[ND], odo[ND];
        {
            std::uint32_t c = cell_of[i];
            RCPG_UNROLL
            for (int d = 0; d < ND; ++d) {
                const int n = g.ncell[d];
                const int ci = static_cast<int>(c % static_cast<std::uint32_t>(n));
                c /= static_cast<std::uint32_t>(n);
                odo[d] = 0;
                if (g.periodic) {
                    span[d] = n >= 3 ? 3 : n;
                    first[d] = n >= 3 ? ci - 1 : 0;
                } else {
                    first[d] = ci > 0 ? ci - 1 : 0;
                    span[d] = min(ci + 1, n - 1) - first[d] + 1;
                }
            }
        }
        // squared distances above this are beyond g.rq whatever the root's rounding
        const double far2 = g.rq * g.rq * (1.0 + 1e-14);
        std::uint32_t cnt = 0;
        const unsigned long long base = PASS ? off[i] : 0ull;
        auto range = [&](std::uint32_t q, std::uint32_t qe) {
            for (; q < qe; ++q) {
                const std::uint32_t j = sid[q];
                if (j <= i) continue;
                const double d2 = pair_dist2<ND>(xi, sx, q, g);
                if (d2 > far2) continue;
                const double dist = sqrt(d2);
                if (!(dist <= g.rq)) continue;
                ++cand;
                const double Rj = sR[q];
                const double rsum = xadd(Ri, Rj);
                const double ov = xsub(rsum, dist);
                if (!(ov > 0.0)) continue;
                if (PASS) {
                    const unsigned long long w = base + cnt;
                    if (w < capacity) {
                        // insertion by j: the pairs of i end sorted
                        unsigned long long p2 = w;
                        while (p2 > base && pairs[2 * (p2 - 1) + 1] > j) {
                            pairs[2 * p2] = pairs[2 * (p2 - 1)];
                            pairs[2 * p2 + 1] = pairs[2 * (p2 - 1) + 1];
                            fsum[p2] = fsum[p2 - 1];
                            fmin_[p2] = fmin_[p2 - 1];
                            --p2;
                        }
                        pairs[2 * p2] = i;
                        pairs[2 * p2 + 1] = j;
                        fsum[p2] = ov / rsum;
                        fmin_[p2] = ov / fmin(Ri, Rj);
                    }
                }
                ++cnt;
            }
        };
        while (true) {
            std::uint32_t row = 0;  // first cell of the grid row
            RCPG_UNROLL
            for (int d = ND - 1; d > 0; --d) {
                int c = first[d] + odo[d];
                if (c < 0) c += g.ncell[d];
                else if (c >= g.ncell[d]) c -= g.ncell[d];
                row = (row + static_cast<std::uint32_t>(c)) * static_cast<std::uint32_t>(g.ncell[d - 1]);
            }
            const std::uint32_t* cs = cell_start + row;
            const int b = first[0], e = first[0] + span[0], n = g.ncell[0];
            if (b < 0) {
                range(cs[b + n], cs[n]);
                range(cs[0], cs[e]);
            } else if (e > n) {
                range(cs[b], cs[n]);
                range(cs[0], cs[e - n]);
            } else {
                range(cs[b], cs[e]);
            }
            int d = 1;
            RCPG_UNROLL
            for (int k = 1; k < ND; ++k) {
                if (d == k) {
                    if (++odo[k] == span[k]) {
                        odo[k] = 0;
                        ++d;
                    }
                }
            }
            if (d >= ND) break;
        }
        if (!PASS) nov[i] = cnt;
    }
    if (!PASS) {
        RCPG_UNROLL
        for (int o = 16; o > 0; o >>= 1) cand += __shfl_down_sync(0xffffffffu, cand, o);
        if ((threadIdx.x & 31) == 0 && cand) atomicAdd(ncand, cand);
    }
}

template <int PASS, typename... Args>
void launch_overlap(int ndim, unsigned blocks, cudaStream_t st, Args... args) {
    switch (ndim) {
        case 1: k_overlap<1, PASS><<<blocks, 128, 0, st>>>(args...); break;
        case 2: k_overlap<2, PASS><<<blocks, 128, 0, st>>>(args...); break;
        case 3: k_overlap<3, PASS><<<blocks, 128, 0, st>>>(args...); break;
        case 4: k_overlap<4, PASS><<<blocks, 128, 0, st>>>(args...); break;
        case 5: k_overlap<5, PASS><<<blocks, 128, 0, st>>>(args...); break;
        case 6: k_overlap<6, PASS><<<blocks, 128, 0, st>>>(args...); break;
        case 7: k_overlap<7, PASS><<<blocks, 128, 0, st>>>(args...); break;
        case 8: k_overlap<8, PASS><<<blocks, 128, 0, st>>>(args...); break;
        default: break;
    }
}

int32_t fail(char* err, std::size_t errlen, int32_t code, const std::string& msg) {
    if (err && errlen) std::snprintf(err, errlen, "%s", msg.c_str());
    return code;
}

struct DevBuf {
    std::vector<void*> ptrs;
    cudaStream_t st;
    explicit DevBuf(cudaStream_t s) : st(s) {}
    template <typename T>
    T* get(std::size_t n) {
        void* p = nullptr;
        if (rcpg::pool_alloc_async(&p, n * sizeof(T) + 16, st) != cudaSuccess)
            throw std::runtime_error("rcpgenerator_b200: device allocation failed");
        ptrs.push_back(p);
        return static_cast<T*>(p);
    }
    ~DevBuf() {
        for (void* p : ptrs) cudaFreeAsync(p, st);
        cudaStreamSynchronize(st);
    }
};

}  // namespace

extern "C" int32_t rcpg_overlap_report(uint64_t N, int32_t ndim, const double* positions, const double* diameters,
                                       const double* box, uint64_t* n_candidate_out, uint64_t* n_overlap_out,
                                       uint64_t capacity, uint32_t* pairs_out, double* frac_sum_out,
                                       double* frac_min_out, int32_t device, char* err, size_t errlen) {
    if (n_candidate_out) *n_candidate_out = 0;
    if (n_overlap_out) *n_overlap_out = 0;
    if (ndim < 1 || ndim > kOvMaxDim || (N && (!positions || !diameters)) ||
        (capacity && (!pairs_out || !frac_sum_out || !frac_min_out)))
        return fail(err, errlen, RCPG_EINVAL, "rcpgenerator_b200: bad arguments to rcpg_overlap_report");
    if (N < 2) return RCPG_OK;
    if (N >= 0xFFFFFFF0ull) return fail(err, errlen, RCPG_EINVAL, "rcpgenerator_b200: N too large");
    int ndev = 0;
    if (cudaGetDeviceCount(&ndev) != cudaSuccess || ndev <= 0) {
        cudaGetLastError();
        return fail(err, errlen, RCPG_ECUDA, "rcpgenerator_b200: no CUDA device available (this engine has no CPU path)");
    }
    try {
        if (cudaSetDevice(device) != cudaSuccess) throw std::runtime_error("cudaSetDevice failed");
        // grid: cells at least 2 R_max wide, at most about 2N + 64 cells
        OvGrid g{};
        g.ndim = ndim;
        g.periodic = box ? 1 : 0;
        double dmax = 0.0;
        for (uint64_t i = 0; i < N; ++i) dmax = std::max(dmax, diameters[i]);
        const double rq = 2.0 * (dmax / 2.0);
        g.rq = rq;
        const double cell_min = rq * (1.0 + 1e-6);  // binning slack: a pair within rq never skips a cell
        double cells = 1.0;
        for (int d = 0; d < ndim; ++d) {
            double lo, hi;
            if (box) {
                lo = 0.0;
                hi = box[d];
            } else {
                lo = hi = positions[d];
                for (uint64_t i = 1; i < N; ++i) {
                    lo = std::min(lo, positions[i * ndim + d]);
                    hi = std::max(hi, positions[i * ndim + d]);
                }
                hi = std::max(hi, lo + 1e-300);
            }
            const double L = hi - lo;
            double n = rq > 0.0 ? std::floor(L / cell_min) : 1.0;
            if (!(n >= 1.0)) n = 1.0;
            if (n > 1048576.0) n = 1048576.0;
            g.lo[d] = lo;
            g.box[d] = box ? box[d] : L;
            g.near[d] = g.box[d] > 0.0 && std::isfinite(g.box[d]) ? 0.49 * g.box[d] : -1.0;
            g.ncell[d] = static_cast<int>(n);
            cells *= n;
        }
        const double cap_cells = 2.0 * static_cast<double>(N) + 64.0;
        while (cells > cap_cells) {
            int dm = 0;
            for (int d = 1; d < ndim; ++d)
                if (g.ncell[d] > g.ncell[dm]) dm = d;
            const int nn = std::max(1, (g.ncell[dm] * 3) / 4);
            cells = cells / g.ncell[dm] * nn;
            g.ncell[dm] = nn;
        }
        for (int d = 0; d < ndim; ++d) g.width[d] = (box ? box[d] : (g.box[d])) / g.ncell[d];
        const std::uint64_t C = static_cast<std::uint64_t>(cells);
        cudaStream_t st = nullptr;
        if (cudaStreamCreateWithFlags(&st, cudaStreamNonBlocking) != cudaSuccess)
            throw std::runtime_error("cudaStreamCreate failed");
        std::uint64_t total_ov = 0, total_cand = 0;
        {
            DevBuf B(st);
            double* dx = B.get<double>(N * ndim);
            double* dD = B.get<double>(N);
            std::uint32_t* dcell = B.get<std::uint32_t>(N);
            std::uint32_t* drank = B.get<std::uint32_t>(N);
            std::uint32_t* dstart = B.get<std::uint32_t>(C + 1);
            double* sx = B.get<double>(N * ndim);
            double* sR = B.get<double>(N);
            std::uint32_t* sid = B.get<std::uint32_t>(N);
            std::uint32_t* dnov = B.get<std::uint32_t>(N + 1);
            unsigned long long* doff = B.get<unsigned long long>(N + 1);
            unsigned long long* dcand = B.get<unsigned long long>(1);
            std::uint32_t* tmp32 = B.get<std::uint32_t>(scan_scratch(C + 1));
            unsigned long long* tmp64 = B.get<unsigned long long>(scan_scratch(N + 1));
            auto ok = [&](cudaError_t e, const char* what) {
                if (e != cudaSuccess)
                    throw std::runtime_error(std::string("rcpgenerator_b200: CUDA error in ") + what + ": " +
                                             cudaGetErrorString(e));
            };
            ok(cudaMemcpyAsync(dx, positions, N * ndim * 8, cudaMemcpyHostToDevice, st), "H2D");
            ok(cudaMemcpyAsync(dD, diameters, N * 8, cudaMemcpyHostToDevice, st), "H2D");
            ok(cudaMemsetAsync(dstart, 0, (C + 1) * 4, st), "memset");
            ok(cudaMemsetAsync(dnov, 0, (N + 1) * 4, st), "memset");
            ok(cudaMemsetAsync(dcand, 0, 8, st), "memset");
            const unsigned b256 = static_cast<unsigned>((N + 255) / 256);
            k_ov_bin<<<b256, 256, 0, st>>>(dx, N, g, dcell, drank, dstart);
            scan<std::uint32_t, std::uint32_t>(dstart, dstart, C + 1, tmp32, st);
            k_ov_scatter<<<b256, 256, 0, st>>>(dx, dD, N, ndim, dcell, drank, dstart, sx, sR, sid);
            const unsigned blocks = static_cast<unsigned>((N + 127) / 128);
            launch_overlap<0>(ndim, blocks, st, sx, sR, sid, N, g, dcell, dstart, dcand, dnov,
                              static_cast<const unsigned long long*>(nullptr), static_cast<std::uint32_t*>(nullptr),
                              static_cast<double*>(nullptr), static_cast<double*>(nullptr), 0ull);
            ok(cudaGetLastError(), "k_overlap count");
            // offsets of the particles' pairs; the last one is the total
            scan<std::uint32_t, unsigned long long>(dnov, doff, N + 1, tmp64, st);
            unsigned long long totals[2];
            ok(cudaMemcpyAsync(&totals[0], doff + N, 8, cudaMemcpyDeviceToHost, st), "D2H");
            ok(cudaMemcpyAsync(&totals[1], dcand, 8, cudaMemcpyDeviceToHost, st), "D2H");
            ok(cudaStreamSynchronize(st), "sync");
            total_ov = totals[0];
            total_cand = totals[1];
            const std::uint64_t m = std::min<std::uint64_t>(total_ov, capacity);
            if (m > 0) {
                std::uint32_t* dpairs = B.get<std::uint32_t>(2 * m);
                double* dfs = B.get<double>(m);
                double* dfm = B.get<double>(m);
                launch_overlap<1>(ndim, blocks, st, sx, sR, sid, N, g, dcell, dstart,
                                  static_cast<unsigned long long*>(nullptr), static_cast<std::uint32_t*>(nullptr), doff,
                                  dpairs, dfs, dfm, static_cast<unsigned long long>(m));
                ok(cudaGetLastError(), "k_overlap write");
                ok(cudaMemcpyAsync(pairs_out, dpairs, 2 * m * 4, cudaMemcpyDeviceToHost, st), "D2H");
                ok(cudaMemcpyAsync(frac_sum_out, dfs, m * 8, cudaMemcpyDeviceToHost, st), "D2H");
                ok(cudaMemcpyAsync(frac_min_out, dfm, m * 8, cudaMemcpyDeviceToHost, st), "D2H");
                ok(cudaStreamSynchronize(st), "sync");
            }
        }
        cudaStreamDestroy(st);
        if (n_candidate_out) *n_candidate_out = total_cand;
        if (n_overlap_out) *n_overlap_out = total_ov;
        if (total_ov > capacity)
            return fail(err, errlen, RCPG_ENOSPC, "rcpgenerator_b200: more overlapping pairs than the output capacity");
        return RCPG_OK;
    } catch (const std::exception& e) {
        return fail(err, errlen, RCPG_ECUDA, e.what());
    }
}
