// nl.cu — cylinder neighbor list and boundary neighbor list on the device,
// with on-device re-vectorization of the excluded-volume and boundary force
// fields.
//
// Pair rule (HybridCylinderCylinderNL::updateNeighborsbin,
// src/Structure/HybridNeighborListImpl.cpp:332-471): a pair (c, n) is stored
// under the key cylinder c when c.id > n.id, the two are not on the same
// filament within |dposition| <= 2, and rmin^2 <= d^2 <= rmax^2, where d^2 is
// the squared distance of the midpoints 0.5*(b1 + b2) (Cylinder.cpp:48)
// summed x, y, z (Util/Math/Vec.hpp:378-384) and rmax^2, rmin^2 are float
// products (HybridNeighborListImpl.h:88-89). The bin grid is the reference's
// (bins of 1.125*sqrt(float rmax^2), HybridNeighborListImpl.cpp:176-240), so a
// midpoint outside it is the same error (getBin throws, :243-262). d^2 is
// rounded without contraction (__dmul_rn/__dadd_rn) so the pair set is the
// oracle's bit for bit.
//
// Passes: midpoints + bin index and boundary counts -> scan of the bins ->
// scatter -> each bin's records in cylinder order -> per-key neighbor counts
// (27-bin stencil) -> scan of both lists' counts -> excluded-volume and boundary
// records. Eight stream operations and one wait: the records go to the buffers
// of the last build while they hold them (a rebuild of 40,000 cylinders with
// scans of three kernels, the boundary list apart and the records after a wait
// for the totals: 143 us; now 72).
#include <algorithm>
#include <climits>
#include <cstring>
#include <vector>

#include "device_math.cuh"
#include "handle.h"

namespace mb {

namespace {

constexpr int kScanThreads = 256, kScanPer = 8, kScanShift = 11;
constexpr int kScanTile = 1 << kScanShift;
static_assert(kScanTile == kScanThreads * kScanPer, "a thread scans kScanPer counts");
constexpr int kFound = 16;  // neighbors of a key that counting keeps for the writing
constexpr int kLaneBin = 4; // cylinders of a bin that one lane takes (walk_key)
constexpr int kKeyLanes = 4;  // threads that write a key's records

struct Grid {
    double bin;
    int g[3];
    double lim[3];  // bin * g, the exclusive upper bound of the grid
};

Grid make_grid(const medyan_nl_params& p) {
    Grid G{};
    const float rmaxsq = p.rmax * p.rmax;
    G.bin = 1.125 * (double)std::sqrt(rmaxsq);
    for (int d = 0; d < 3; ++d) {
        int size = (int)(p.grid_size[d]);
        int ib = (int)G.bin;
        G.g[d] = (ib != 0 && size % ib == 0) ? (int)(size / G.bin) : (int)(size / G.bin + 1);
        if (G.g[d] < 1) G.g[d] = 1;
        G.lim[d] = G.bin * G.g[d];
    }
    return G;
}

struct CylDev {
    int n;
    const int* b1;
    const int* b2;
    const int* id;
    const int* fil;
    const int* pos;
    const int* type;
    const int* branching;
    const int* minus_end;
    const double* eqlen;
    const double* exclk;
};

// An exclusive scan: entry i is local[i] plus the counts before its tile.
struct Scan {
    const int* local;
    const int* base;
    __device__ __forceinline__ int operator[](int i) const { return __ldg(local + i) + __ldg(base + (i >> kScanShift)); }
};

// A binned cylinder, in bin order.
struct Item {
    double m[3];
    int id, fil, pos, cyl;
};

// Boundary list of a build: its planes and the counts per plane and cylinder.
struct BoundaryDev {
    const double4* planes;
    int n_planes;
    float cutoff;
};

// Boundary NL: number of terms of cylinder i against plane p (0, 1 or 2).
__device__ __forceinline__ int boundary_terms(const CylDev& c, const double* __restrict__ x, const double4& pl,
                                              float cutoff, int i) {
    const double* p1 = x + 3 * (size_t)c.b1[i];
    const double* p2 = x + 3 * (size_t)c.b2[i];
    // Cylinder::coordinate = midPointCoordinate(b1, b2, 0.5) (Cylinder.cpp:46)
    double m[3];
    for (int d = 0; d < 3; ++d) m[d] = p1[d] * (1.0 - 0.5) + 0.5 * p2[d];
    double dist = (pl.x * m[0] + pl.y * m[1] + pl.z * m[2] + pl.w) / sqrt(pl.x * pl.x + pl.y * pl.y + pl.z * pl.z);
    if (!(dist < (double)cutoff)) return 0;
    return (c.minus_end && c.minus_end[i]) ? 2 : 1;
}

// Thread t < n: midpoint and bin of cylinder t, and its place among the bin's
// arrivals. Thread n + p n + i: the count of plane p and cylinder i.
__global__ void k_midpoints(CylDev c, const double* __restrict__ x, Grid G, BoundaryDev B, double* __restrict__ mid,
                            int* __restrict__ cell, int* __restrict__ slot, int* __restrict__ bin_count,
                            int* __restrict__ err, int* __restrict__ count) {
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= c.n) {
        const int p = t / c.n - 1;
        if (p < B.n_planes) count[t] = boundary_terms(c, x, B.planes[p], B.cutoff, t % c.n);
        return;
    }
    const int i = t;
    const double* p1 = x + 3 * (size_t)c.b1[i];
    const double* p2 = x + 3 * (size_t)c.b2[i];
    long long idx = 0, stride = 1;
    bool bad = false;
    for (int d = 0; d < 3; ++d) {
        double m = 0.5 * (p1[d] + p2[d]);
        mid[3 * (size_t)i + d] = m;
        if (!(m >= 0.0) || m >= G.lim[d]) bad = true;
        int q = bad ? 0 : (int)(m / G.bin);
        idx += (long long)q * stride;
        stride *= G.g[d];
    }
    if (bad) {
        atomicOr(err, 1);
        cell[i] = -1;
        return;
    }
    cell[i] = (int)idx;
    slot[i] = atomicAdd(bin_count + idx, 1);
}

// Sum of v over the block's threads before this one; total: over all.
__device__ __forceinline__ int block_before(int v, int* warp_sum, int& total) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    int s = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int u = __shfl_up_sync(0xffffffffu, s, o);
        if (lane >= o) s += u;
    }
    __syncthreads();  // the sums of the call before have been read
    if (lane == 31) warp_sum[warp] = s;
    __syncthreads();
    int before = s - v;
    total = 0;
#pragma unroll
    for (int w = 0; w < kScanThreads / 32; ++w) {
        if (w < warp) before += warp_sum[w];
        total += warp_sum[w];
    }
    return before;
}

// Exclusive scan of in[0..n) to entries 0..n, the last one the total, in one
// kernel: each block scans a tile, the last one to end (ticket) the tiles' sums;
// readers add the two (Scan). No block waits for another.
__global__ void __launch_bounds__(kScanThreads) k_scan(const int* __restrict__ in, int n, int* __restrict__ local,
                                                       int* __restrict__ base, unsigned* __restrict__ ticket) {
    __shared__ int warp_sum[kScanThreads / 32];
    __shared__ bool last;
    const int i0 = blockIdx.x * kScanTile + threadIdx.x * kScanPer;
    int v[kScanPer], sum = 0, total;
#pragma unroll
    for (int k = 0; k < kScanPer; ++k) v[k] = 0;
    if (i0 + kScanPer <= n) {  // tiles begin on 16-byte boundaries
        const int4 a = *reinterpret_cast<const int4*>(in + i0), b = *reinterpret_cast<const int4*>(in + i0 + 4);
        v[0] = a.x, v[1] = a.y, v[2] = a.z, v[3] = a.w, v[4] = b.x, v[5] = b.y, v[6] = b.z, v[7] = b.w;
    } else {
#pragma unroll
        for (int k = 0; k < kScanPer; ++k)
            if (i0 + k < n) v[k] = in[i0 + k];
    }
#pragma unroll
    for (int k = 0; k < kScanPer; ++k) {
        const int u = v[k];
        v[k] = sum;
        sum += u;
    }
    const int before = block_before(sum, warp_sum, total);
#pragma unroll
    for (int k = 0; k < kScanPer; ++k)
        if (i0 + k <= n) local[i0 + k] = before + v[k];
    if (threadIdx.x == 0) {
        base[blockIdx.x] = total;
        last = ticket_add(ticket, 1u) == gridDim.x - 1;
    }
    __syncthreads();
    if (!last) return;
    int carry = 0;
    for (int t0 = 0; t0 < (int)gridDim.x; t0 += kScanThreads) {
        const int t = t0 + threadIdx.x;
        const int u = t < (int)gridDim.x ? __ldcg(base + t) : 0;
        const int b = block_before(u, warp_sum, total);
        if (t < (int)gridDim.x) base[t] = carry + b;
        carry += total;
    }
}

__global__ void k_scatter(int n, const int* __restrict__ cell, const int* __restrict__ slot, Scan start,
                          int* __restrict__ order) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n && cell[i] >= 0) order[start[cell[i]] + slot[i]] = i;
}

// Deterministic bin contents: the first arrival's thread sorts its bin by
// cylinder index and writes the bin's records.
__global__ void k_fill_bins(CylDev c, const int* __restrict__ cell, const int* __restrict__ slot, Scan start,
                            const double* __restrict__ mid, int* __restrict__ order, Item* __restrict__ items) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= c.n || cell[i] < 0 || slot[i] != 0) return;
    const int s0 = start[cell[i]], s1 = start[cell[i] + 1];
    for (int a = s0 + 1; a < s1; ++a) {
        int v = order[a], q = a - 1;
        while (q >= s0 && order[q] > v) {
            order[q + 1] = order[q];
            --q;
        }
        order[q + 1] = v;
    }
    for (int a = s0; a < s1; ++a) {
        const int j = order[a];
        const double* m = mid + 3 * (size_t)j;
        items[a] = Item{{m[0], m[1], m[2]}, c.id[j], c.fil[j], c.pos[j], j};
    }
}

// Neighbors of key i, found by a warp whose lanes read the 27 bins of the stencil
// side by side: the bins hold a tenth of a cylinder on average, so one thread per
// key spent its time on 27 dependent loads in a row (40,000 cylinders: 48 us; a
// warp 19). Then each lane takes a bin's cylinders, or, where a bin holds more
// than kLaneBin, all lanes take the bins' cylinders one after another, 32 at a
// time: in a bundle a few bins hold all of them (rebuild of 2,000 cylinders with
// 35,500 pairs: a lane per bin 510 us, now 147; 400,000 spread cylinders: a
// lane per bin 271 us, all lanes 302). A key's pairs are in bin order, dx
// outermost, then the bin's order, either way. put(k, j): neighbor number k of the
// key is j; returns their number. All 32 lanes call.
template <class Put>
__device__ __forceinline__ int walk_key(const CylDev& c, const Grid& G, int ci, int i, const Scan& start,
                                        const Item* __restrict__ items, const double* __restrict__ mid, double rmaxsq,
                                        double rminsq, int skip_branch, Put put) {
    const int lane = threadIdx.x & 31;
    const int ix = ci % G.g[0], iy = (ci / G.g[0]) % G.g[1], iz = ci / (G.g[0] * G.g[1]);
    const int jx = ix + lane / 9 - 1, jy = iy + lane / 3 % 3 - 1, jz = iz + lane % 3 - 1;
    int q0 = 0, q1 = 0;
    if (lane < 27 && jx >= 0 && jx < G.g[0] && jy >= 0 && jy < G.g[1] && jz >= 0 && jz < G.g[2]) {
        const int cj = jx + G.g[0] * (jy + G.g[1] * jz);
        q0 = start[cj];
        q1 = start[cj + 1];
    }
    const int idi = c.id[i], fi = c.fil[i], pi = c.pos[i];
    const double mx = mid[3 * (size_t)i], my = mid[3 * (size_t)i + 1], mz = mid[3 * (size_t)i + 2];
    auto is_pair = [&](const Item& o) {
        if (idi <= o.id) return false;
        if (fi == o.fil) {
            const int ds = pi - o.pos;
            if ((ds < 0 ? -ds : ds) <= 2) return false;
        }
        // d^2 of the midpoints, rounded as written: ((dx*dx + dy*dy) + dz*dz)
        const double dx = __dadd_rn(o.m[0], -mx), dy = __dadd_rn(o.m[1], -my), dz = __dadd_rn(o.m[2], -mz);
        const double d2 = __dadd_rn(__dadd_rn(__dmul_rn(dx, dx), __dmul_rn(dy, dy)), __dmul_rn(dz, dz));
        if (d2 > rmaxsq || d2 < rminsq) return false;
        return !(skip_branch && c.branching[o.cyl] == i);
    };
    // v of the lanes up to this one
    auto upto = [&](int v) {
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int u = __shfl_up_sync(0xffffffffu, v, o);
            if (lane >= o) v += u;
        }
        return v;
    };
    if (!__any_sync(0xffffffffu, q1 - q0 > kLaneBin)) {
        int n = 0;
        for (int q = q0; q < q1; ++q) n += is_pair(items[q]) ? 1 : 0;
        if (!__any_sync(0xffffffffu, n)) return 0;
        int before = upto(n);  // pairs of the bins before this lane's
        const int total = __shfl_sync(0xffffffffu, before, 31);
        before -= n;
        for (int q = q0; q < q1 && n > 0; ++q) {
            if (!is_pair(items[q])) continue;
            put(before, items[q].cyl);
            ++before;
            --n;
        }
        return total;
    }
    const int end = upto(q1 - q0);  // cylinders of the bins up to this lane's
    const int total = __shfl_sync(0xffffffffu, end, 31), base = q1 - end;
    int found = 0;
    for (int t0 = 0; t0 < total; t0 += 32) {
        const int t = t0 + lane;
        int b = 0;  // the bin of number t: the bins that end at or before it
#pragma unroll
        for (int s = 16; s > 0; s >>= 1)
            if (__shfl_sync(0xffffffffu, end, b + s - 1) <= t) b += s;
        const int q = __shfl_sync(0xffffffffu, base, b) + t;
        const int j = t < total && is_pair(items[q]) ? items[q].cyl : -1;
        const unsigned hits = __ballot_sync(0xffffffffu, j >= 0);
        if (j >= 0) put(found + __popc(hits & ((1u << lane) - 1u)), j);
        found += __popc(hits);
    }
    return found;
}

// Counts the pairs of each key, a warp per key, and keeps its first neighbors.
__global__ void k_count_pairs(CylDev c, Grid G, const double* __restrict__ mid, const int* __restrict__ cell, Scan start,
                              const Item* __restrict__ items, double rmaxsq, double rminsq, int skip_branch,
                              int* __restrict__ count, int* __restrict__ found) {
    const int i = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5), lane = threadIdx.x & 31;
    if (i >= c.n) return;
    const int ci = cell[i];
    int n = 0;
    if (ci >= 0)
        n = walk_key(c, G, ci, i, start, items, mid, rmaxsq, rminsq, skip_branch, [&](int k, int j) {
            if (k < kFound) found[(size_t)i * kFound + k] = j;
        });
    if (lane == 0) count[i] = n;
}

// Where the records of a build go: pairs (key, neighbor) of the standalone
// build, or excluded-volume records (branch-parent pairs skipped,
// CylinderExclVolume.cpp:85) and boundary records. room: what the buffers hold;
// lists that do not fit, or of a build with a midpoint outside the grid, are
// not written. totals (pinned, may be null): pairs, the error flag, boundary
// terms.
struct Records {
    int2* pairs;
    int4* ex_bs;
    double* ex_krs;
    int* b_bs;
    double2* b_p;
    int* b_plane;
    double4* planes;
    int room, b_room;
    double b_k, b_slen;
    int* totals;
};

// Writes them: kKeyLanes threads per key its pairs, from what counting found (all
// again by the warp when it found more than it kept: with a thread per key a
// warp walked 32 such keys one after another, half the time of a bundle's rebuild),
// then a thread per plane p and cylinder i its terms.
template <bool PAIRS>
__global__ void __launch_bounds__(256) k_write_records(CylDev c, Grid G, BoundaryDev B, const double* __restrict__ mid,
                                                       const int* __restrict__ cell, Scan start,
                                                       const Item* __restrict__ items, double rmaxsq, double rminsq,
                                                       int skip_branch, Scan off, const int* __restrict__ found,
                                                       const int* __restrict__ err, Records R) {
    const int m = c.n * (1 + B.n_planes), u = blockIdx.x * blockDim.x + threadIdx.x, sub = u % kKeyLanes;
    const bool key = u < kKeyLanes * c.n;
    const int t = key ? u / kKeyLanes : u - (kKeyLanes - 1) * c.n;  // the count's index
    const int n_pairs = off[c.n], n_terms = off[m] - n_pairs, bad = *err;
    if (u == 0 && R.totals) {
        R.totals[0] = n_pairs;
        R.totals[1] = bad;
        R.totals[2] = n_terms;
    }
    if (bad || n_pairs > R.room || n_terms > R.b_room) return;
    const int o = t < m ? off[t] : 0, n = t < m ? off[t + 1] - o : 0;
    auto put = [&](int i, int at, int j) {
        if constexpr (PAIRS) {
            R.pairs[at] = make_int2(i, j);
        } else {
            R.ex_bs[at] = make_int4(3 * c.b1[i], 3 * c.b2[i], 3 * c.b1[j], 3 * c.b2[j]);
            double k = c.exclk[i];
            if (c.type[i] != c.type[j]) k = k < c.exclk[j] ? c.exclk[j] : k;
            R.ex_krs[at] = k * c.eqlen[i] * c.eqlen[j];
        }
    };
    if (key && n <= kFound)
        for (int k = sub; k < n; k += kKeyLanes) put(t, o + k, found[(size_t)t * kFound + k]);
    unsigned many = __ballot_sync(0xffffffffu, key && sub == 0 && n > kFound);
    for (; many; many &= many - 1u) {
        const int l = __ffs(many) - 1, i = __shfl_sync(0xffffffffu, t, l), at = __shfl_sync(0xffffffffu, o, l);
        walk_key(c, G, cell[i], i, start, items, mid, rmaxsq, rminsq, skip_branch,
                 [&](int k, int j) { put(i, at + k, j); });
    }
    if constexpr (!PAIRS) {
        if (u < B.n_planes) R.planes[u] = B.planes[u];
        if (key || n == 0) return;
        const int p = t / c.n - 1, i = t % c.n;
        int at = o - n_pairs;
        if (n == 2) {
            R.b_bs[at] = 3 * c.b1[i];
            R.b_p[at] = make_double2(R.b_k, R.b_slen);
            R.b_plane[at] = p;
            ++at;
        }
        R.b_bs[at] = 3 * c.b2[i];
        R.b_p[at] = make_double2(R.b_k, R.b_slen);
        R.b_plane[at] = p;
    }
}

// Canonical order for the standalone build: each key's neighbors ascending.
__global__ void k_sort_pairs(int n, Scan offset, int2* __restrict__ pairs) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const int s0 = offset[i], s1 = offset[i + 1];
    for (int a = s0 + 1; a < s1; ++a) {
        int2 v = pairs[a];
        int q = a - 1;
        while (q >= s0 && pairs[q].y > v.y) {
            pairs[q + 1] = pairs[q];
            --q;
        }
        pairs[q + 1] = v;
    }
}

// BoundaryCylinderRepulsion::computeLoadForces with the exponential
// repulsion (BoundaryCylinderRepulsion.cpp:125-196, BoundaryCylinderRepulsionExp.cpp:113-118):
// one block per tip, threads over the tip's monomer positions; planes in
// order, each plane whose neighbor list (member[p*n + cyl] > 0, from the last
// build) holds the tip's cylinder adds its term.
__global__ void k_boundary_load(CylDev c, const double* __restrict__ x, const double4* __restrict__ planes,
                                int n_planes, const int* __restrict__ member, double k, double slen, int n_tips,
                                const int* __restrict__ tip_cyl, const int* __restrict__ tip_plus,
                                const int* __restrict__ tip_nmon, const double* __restrict__ tip_mon,
                                const long long* __restrict__ tip_off, double* __restrict__ out) {
    for (int t = blockIdx.x; t < n_tips; t += gridDim.x) {
        const int ci = tip_cyl[t];
        const bool plus = tip_plus[t] != 0;
        const double* bo = x + 3 * (size_t)(plus ? c.b1[ci] : c.b2[ci]);
        const double* bd = x + 3 * (size_t)(plus ? c.b2[ci] : c.b1[ci]);
        // normalizedVector(bd - bo)
        const double vx = bd[0] - bo[0], vy = bd[1] - bo[1], vz = bd[2] - bo[2];
        const double m = sqrt(vx * vx + vy * vy + vz * vz);
        const double dir[3] = {vx / m, vy / m, vz / m};
        const int nmon = tip_nmon[t];
        const double mon = tip_mon[t];
        double* o = out + tip_off[t];
        for (int i = threadIdx.x; i < nmon; i += blockDim.x) {
            const double s = i * mon;
            const double p[3] = {bd[0] + s * dir[0], bd[1] + s * dir[1], bd[2] + s * dir[2]};
            double load = 0.0;
            for (int q = 0; q < n_planes; ++q) {
                if (member[(size_t)q * c.n + ci] <= 0) continue;
                const double4 pl = planes[q];
                const double proj0 = -(pl.x * dir[0] + pl.y * dir[1] + pl.z * dir[2]);
                const double proj = proj0 < 0.0 ? 0.0 : proj0;  // std::max(.., 0.0)
                const double dist =
                    (pl.x * p[0] + pl.y * p[1] + pl.z * p[2] + pl.w) / sqrt(pl.x * pl.x + pl.y * pl.y + pl.z * pl.z);
                const double R = -dist / slen;
                load += proj * (k * exp(R) / slen);
            }
            o[i] = load;
        }
    }
}

}  // namespace

// Device buffers of one neighbor-list builder (grow-only).
struct NLBuilder {
    DevBuf<int> b1, b2, id, fil, pos, type, branching, minus_end;
    DevBuf<double> eqlen, exclk;
    DevBuf<double> mid;
    DevBuf<int> cell, slot, bins, bin_start, bin_base, order, off, off_base, found;
    DevBuf<Item> items;
    // pairs per key, then boundary terms per plane and cylinder; the load forces read
    // the boundary membership of the last build that gave the handle its records
    DevBuf<int> counts, counts_built;
    DevBuf<int2> pairs;
    DevBuf<double4> planes;
    medyan_nl_params nl{};
    medyan_boundary_params bp{};
    std::vector<double> plane_host;
    bool has_boundary = false;
    bool boundary_built = false;  // counts_built holds the last build's plane membership
    int n = 0;

    CylDev view() const {
        return CylDev{n, b1.raw(), b2.raw(), id.raw(), fil.raw(), pos.raw(), type.raw(), branching.raw(),
                      minus_end.raw(), eqlen.raw(), exclk.raw()};
    }

    cudaError_t set(const medyan_cylinders* c, cudaStream_t s) {
        n = c->n_cyl;
        boundary_built = false;
        std::vector<int> zeros(n, 0), neg(n, -1);
        std::vector<double> dz(n, 0.0);
        cudaError_t e;
#define SETI(buf, ptr, dflt)                                                \
    e = (buf).assign((ptr) ? (ptr) : dflt.data(), (size_t)n, s);           \
    if (e != cudaSuccess) return e;
        SETI(b1, c->bead1, zeros);
        SETI(b2, c->bead2, zeros);
        SETI(id, c->id, zeros);
        SETI(fil, c->filament_id, zeros);
        SETI(pos, c->position_on_filament, zeros);
        SETI(type, c->type, zeros);
        SETI(branching, c->branching_cylinder, neg);
        SETI(minus_end, c->is_minus_end, zeros);
        SETI(eqlen, c->eq_length, dz);
        SETI(exclk, c->excl_k, dz);
#undef SETI
        return cudaSuccess;
    }

    int planes_on() const { return has_boundary && bp.n_planes > 0 ? bp.n_planes : 0; }
    BoundaryDev boundary(bool on) const { return BoundaryDev{planes.raw(), on ? planes_on() : 0, bp.cutoff}; }
    Scan starts() const { return Scan{bin_start.raw(), bin_base.raw()}; }
    Scan offsets() const { return Scan{off.raw(), off_base.raw()}; }
    long long n_bins() const {
        const Grid G = make_grid(nl);
        return (long long)G.g[0] * G.g[1] * G.g[2];
    }
    int* error() const { return bins.raw() + n_bins(); }

    cudaError_t scan(const int* cnt, int m, DevBuf<int>& local, DevBuf<int>& base, int* ticket, cudaStream_t s) {
        const int tiles = m / kScanTile + 1;  // of the m + 1 entries
        cudaError_t e = local.reserve((size_t)m + 1);
        if (e == cudaSuccess) e = base.reserve(tiles);
        if (e != cudaSuccess) return e;
        k_scan<<<tiles, kScanThreads, 0, s>>>(cnt, m, local.raw(), base.raw(), reinterpret_cast<unsigned*>(ticket));
        return cudaGetLastError();
    }

    static int blocks_of(long long threads) { return (int)((threads + 255) / 256); }

    // Bins the midpoints, counts pairs per key and (boundary) terms per plane and
    // cylinder, and scans the counts. Nothing is waited for.
    medyan_status enqueue_count(const double* x, int skip_branch, bool with_boundary, cudaStream_t s) {
        const Grid G = make_grid(nl);
        const long long nbins = n_bins();
        if (nbins > (1LL << 30)) return MEDYAN_ERR_INVALID_ARG;
        const BoundaryDev B = boundary(with_boundary);
        const int m = n * (1 + B.n_planes);
        const size_t n1 = n > 0 ? n : 1;
        cudaError_t e = mid.reserve(3 * n1);
        if (e == cudaSuccess) e = cell.reserve(n1);
        if (e == cudaSuccess) e = slot.reserve(n1);
        if (e == cudaSuccess) e = order.reserve(n1);
        if (e == cudaSuccess) e = items.reserve(n1);
        if (e == cudaSuccess) e = found.reserve(kFound * n1);
        if (e == cudaSuccess) e = counts.reserve((size_t)m + 1);
        // the other one too, so that no later build has to allocate
        if (e == cudaSuccess && with_boundary && !boundary_built) e = counts_built.reserve((size_t)m + 1);
        if (e == cudaSuccess) e = bins.reserve(nbins + 3);  // then the error flag and the scans' tickets
        if (e == cudaSuccess) e = cudaMemsetAsync(bins.raw(), 0, sizeof(int) * (nbins + 3), s);
        if (e != cudaSuccess) return cuda_status(e);
        if (n > 0)
            k_midpoints<<<blocks_of(m), 256, 0, s>>>(view(), x, G, B, mid.raw(), cell.raw(), slot.raw(), bins.raw(),
                                                     error(), counts.raw());
        e = scan(bins.raw(), (int)nbins, bin_start, bin_base, error() + 1, s);
        if (e != cudaSuccess) return cuda_status(e);
        if (n > 0) {
            k_scatter<<<blocks_of(n), 256, 0, s>>>(n, cell.raw(), slot.raw(), starts(), order.raw());
            k_fill_bins<<<blocks_of(n), 256, 0, s>>>(view(), cell.raw(), slot.raw(), starts(), mid.raw(), order.raw(),
                                                     items.raw());
            const float rmaxsq = nl.rmax * nl.rmax, rminsq = nl.rmin * nl.rmin;
            k_count_pairs<<<blocks_of(32LL * n), 256, 0, s>>>(view(), G, mid.raw(), cell.raw(), starts(), items.raw(),
                                                              (double)rmaxsq, (double)rminsq, skip_branch, counts.raw(),
                                                              found.raw());
        }
        return cuda_status(scan(counts.raw(), m, off, off_base, error() + 2, s));
    }

    template <bool PAIRS>
    cudaError_t enqueue_write(int skip_branch, const Records& R, cudaStream_t s) {
        const BoundaryDev B = boundary(!PAIRS);
        const float rmaxsq = nl.rmax * nl.rmax, rminsq = nl.rmin * nl.rmin;
        const long long threads = (long long)n * (kKeyLanes + B.n_planes);  // at least one block copies the planes
        k_write_records<PAIRS><<<blocks_of(threads > B.n_planes ? threads : B.n_planes + 1), 256, 0, s>>>(
            view(), make_grid(nl), B, mid.raw(), cell.raw(), starts(), items.raw(), (double)rmaxsq, (double)rminsq,
            skip_branch, offsets(), found.raw(), error(), R);
        return cudaGetLastError();
    }

    // The count, waited for; returns the pair total.
    medyan_status count_pairs(const double* x, int skip_branch, cudaStream_t s, long long* total) {
        const medyan_status st = enqueue_count(x, skip_branch, false, s);
        if (st != MEDYAN_OK) return st;
        int h[3] = {0, 0, 0};
        cudaError_t e = cudaMemcpyAsync(&h[0], off.raw() + n, sizeof(int), cudaMemcpyDeviceToHost, s);
        if (e == cudaSuccess)
            e = cudaMemcpyAsync(&h[1], off_base.raw() + (n >> kScanShift), sizeof(int), cudaMemcpyDeviceToHost, s);
        if (e == cudaSuccess) e = cudaMemcpyAsync(&h[2], error(), sizeof(int), cudaMemcpyDeviceToHost, s);
        if (e == cudaSuccess) e = cudaStreamSynchronize(s);
        if (e != cudaSuccess) return cuda_status(e);
        if (h[2]) return MEDYAN_ERR_OUT_OF_GRID;
        *total = h[0] + h[1];
        return MEDYAN_OK;
    }

    std::vector<double4> planes_host4() const {
        std::vector<double4> v(bp.n_planes);
        for (int p = 0; p < bp.n_planes; ++p)
            v[p] = make_double4(plane_host[4 * p], plane_host[4 * p + 1], plane_host[4 * p + 2], plane_host[4 * p + 3]);
        return v;
    }
};

void destroy_nl(medyan_mech* h) {
    delete reinterpret_cast<NLBuilder*>(h->nl);
    h->nl = nullptr;
}

}  // namespace mb

using namespace mb;

extern "C" {

medyan_status medyan_nl_build(const medyan_cylinders* cyl, const double* coord, int32_t n_beads,
                              const medyan_nl_params* p, int32_t* pairs_out, int64_t capacity, int64_t* n_pairs) {
    if (!cyl || !p || !n_pairs || cyl->n_cyl < 0 || n_beads < 0 || (!coord && n_beads)) return MEDYAN_ERR_INVALID_ARG;
    if (!(p->rmax > 0) || p->rmin < 0) return MEDYAN_ERR_INVALID_ARG;
    for (int i = 0; i < cyl->n_cyl; ++i) {
        if (!cyl->bead1 || !cyl->bead2 || !cyl->id || !cyl->filament_id || !cyl->position_on_filament)
            return MEDYAN_ERR_INVALID_ARG;
        if (cyl->bead1[i] < 0 || cyl->bead1[i] >= n_beads || cyl->bead2[i] < 0 || cyl->bead2[i] >= n_beads)
            return MEDYAN_ERR_INDEX_RANGE;
    }
    cudaStream_t s;
    cudaError_t e = cudaStreamCreateWithFlags(&s, cudaStreamNonBlocking);
    if (e != cudaSuccess) return cuda_status(e);
    medyan_status st = MEDYAN_OK;
    {
        NLBuilder b;
        b.nl = *p;
        DevBuf<double> x;
        e = b.set(cyl, s);
        if (e == cudaSuccess) e = x.assign(coord, 3 * (size_t)n_beads, s);
        if (e != cudaSuccess) st = cuda_status(e);
        long long total = 0;
        if (st == MEDYAN_OK) st = b.count_pairs(x.raw(), 0, s, &total);
        if (st == MEDYAN_OK) {
            *n_pairs = total;
            if (pairs_out) {
                if (total > capacity) st = MEDYAN_ERR_CAPACITY;
                else if (total > 0) {
                    e = b.pairs.reserve(total);
                    if (e == cudaSuccess) {
                        Records R{};
                        R.pairs = b.pairs.raw();
                        R.room = (int)total;
                        e = b.enqueue_write<true>(0, R, s);
                        if (e == cudaSuccess) {
                            k_sort_pairs<<<NLBuilder::blocks_of(b.n), 256, 0, s>>>(b.n, b.offsets(), b.pairs.raw());
                            e = cudaGetLastError();
                        }
                        if (e == cudaSuccess) e = cudaMemcpyAsync(pairs_out, b.pairs.raw(), sizeof(int2) * total, cudaMemcpyDeviceToHost, s);
                    }
                    if (e == cudaSuccess) e = cudaStreamSynchronize(s);
                    if (e != cudaSuccess) st = cuda_status(e);
                }
            }
        } else {
            *n_pairs = 0;
        }
        cudaStreamSynchronize(s);
    }
    cudaStreamDestroy(s);
    return st;
}

medyan_status medyan_mech_set_cylinders(medyan_mech* h, const medyan_cylinders* cyl, const medyan_nl_params* nl,
                                        const medyan_boundary_params* boundary) {
    if (!h || !cyl || !nl || cyl->n_cyl < 0 || !(nl->rmax > 0) || nl->rmin < 0) return MEDYAN_ERR_INVALID_ARG;
    if (!cyl->bead1 || !cyl->bead2 || !cyl->id || !cyl->filament_id || !cyl->position_on_filament || !cyl->eq_length ||
        !cyl->excl_k)
        return MEDYAN_ERR_INVALID_ARG;
    for (int i = 0; i < cyl->n_cyl; ++i) {
        if (cyl->bead1[i] < 0 || cyl->bead1[i] >= h->n_beads || cyl->bead2[i] < 0 || cyl->bead2[i] >= h->n_beads)
            return MEDYAN_ERR_INDEX_RANGE;
        if (cyl->branching_cylinder && (cyl->branching_cylinder[i] < -1 || cyl->branching_cylinder[i] >= cyl->n_cyl))
            return MEDYAN_ERR_INDEX_RANGE;
    }
    if (boundary && boundary->n_planes > 0 && !boundary->plane_eq) return MEDYAN_ERR_INVALID_ARG;
    if (!h->nl) h->nl = reinterpret_cast<medyan_mech::NL*>(new NLBuilder());
    NLBuilder* b = reinterpret_cast<NLBuilder*>(h->nl);
    b->nl = *nl;
    b->has_boundary = boundary && boundary->n_planes > 0;
    if (b->has_boundary) {
        b->bp = *boundary;
        b->plane_host.assign(boundary->plane_eq, boundary->plane_eq + 4 * boundary->n_planes);
        b->bp.plane_eq = b->plane_host.data();
        cudaError_t e = b->planes.assign(b->planes_host4().data(), boundary->n_planes, h->stream);
        if (e != cudaSuccess) return cuda_status(e);
    }
    // bead indices into the handle's internal order
    std::vector<int32_t> b1(cyl->n_cyl), b2(cyl->n_cyl);
    for (int i = 0; i < cyl->n_cyl; ++i) {
        b1[i] = h->pos_host.empty() ? cyl->bead1[i] : h->pos_host[cyl->bead1[i]];
        b2[i] = h->pos_host.empty() ? cyl->bead2[i] : h->pos_host[cyl->bead2[i]];
    }
    medyan_cylinders ci = *cyl;
    ci.bead1 = b1.data();
    ci.bead2 = b2.data();
    cudaError_t e = b->set(&ci, h->stream);
    return cuda_status(e);
}

medyan_status medyan_mech_rebuild_neighbors(medyan_mech* h, int64_t* n_excl_out, int64_t* n_boundary_out) {
    if (!h || !h->nl) return MEDYAN_ERR_INVALID_ARG;
    NLBuilder* b = reinterpret_cast<NLBuilder*>(h->nl);
    cudaStream_t s = h->stream;
    bool written = false;
    // both lists' counts and, where the handle's buffers have room, the records; one
    // wait for the totals. The records come again when they did not fit.
    int* tot = h->small->nl_totals;  // pairs, outside the grid, boundary terms
    tot[0] = tot[1] = tot[2] = 0;
    medyan_status st = b->enqueue_count(h->x.raw(), 1, true, s);
    if (st != MEDYAN_OK) return st;
    const int np = b->planes_on();
    auto write = [&] {
        Records R{};
        R.ex_bs = h->excl_bs.raw();
        R.ex_krs = h->excl_krs.raw();
        R.room = (int)std::min({h->excl_bs.cap, h->excl_krs.cap, (size_t)INT_MAX});
        R.b_bs = h->boundary_bs.raw();
        R.b_p = h->boundary_p.raw();
        R.b_plane = h->boundary_plane.raw();
        R.planes = h->planes.raw();
        R.b_room = (int)std::min({h->boundary_bs.cap, h->boundary_p.cap, h->boundary_plane.cap, (size_t)INT_MAX});
        if (h->planes.cap < (size_t)np) R.b_room = -1;
        R.b_k = b->bp.k;
        R.b_slen = b->bp.screen_length;
        R.totals = tot;
        cudaError_t e = b->enqueue_write<false>(1, R, s);
        if (e == cudaSuccess) e = cudaStreamSynchronize(s);
        written = e == cudaSuccess && !tot[1] && tot[0] <= R.room && tot[2] <= R.b_room;
        return e;
    };
    cudaError_t e = write();
    if (e != cudaSuccess) return cuda_status(e);
    if (tot[1]) return MEDYAN_ERR_OUT_OF_GRID;
    // a list that outgrows its buffer gets an eighth more: moving beads change it a little each time
    auto fit = [](auto& buf, size_t count) {
        cudaError_t e = count <= buf.cap && buf.raw() ? cudaSuccess : buf.reserve(buf.cap > 1 ? count + count / 8 : count);
        return e == cudaSuccess ? buf.reserve(count) : e;
    };
    e = fit(h->excl_bs, tot[0]);
    if (e == cudaSuccess) e = fit(h->excl_krs, tot[0]);
    if (e == cudaSuccess && np > 0) e = fit(h->boundary_bs, tot[2]);
    if (e == cudaSuccess && np > 0) e = fit(h->boundary_p, tot[2]);
    if (e == cudaSuccess && np > 0) e = fit(h->boundary_plane, tot[2]);
    if (e == cudaSuccess && np > 0) e = h->planes.reserve(np);
    if (e == cudaSuccess && !written) e = write();
    if (e != cudaSuccess) return cuda_status(e);
    h->ff.n_excl = tot[0];
    const int nb = tot[2];
    if (np > 0) {
        h->ff.n_boundary = nb;
        h->ff.n_planes = np;
        b->counts.swap(b->counts_built);
        b->boundary_built = true;
    }
    st = refresh_device_ff(h);
    if (st != MEDYAN_OK) return st;
    if (n_excl_out) *n_excl_out = tot[0];
    if (n_boundary_out) *n_boundary_out = nb;
    return sync_status(h);
}

medyan_status medyan_mech_get_excl_volume(medyan_mech* h, int32_t* beads_out, double* k_out, double* eqlen_out,
                                          int64_t capacity, int64_t* n_out) {
    if (!h || !n_out) return MEDYAN_ERR_INVALID_ARG;
    const int64_t n = h->ff.n_excl;
    *n_out = n;
    if (!beads_out) return MEDYAN_OK;
    if (n > capacity) return MEDYAN_ERR_CAPACITY;
    if (n == 0) return MEDYAN_OK;
    std::vector<int4> bs(n);
    std::vector<double> krs(n);
    cudaError_t e = cudaMemcpyAsync(bs.data(), h->excl_bs.raw(), sizeof(int4) * n, cudaMemcpyDeviceToHost, h->stream);
    if (e == cudaSuccess)
        e = cudaMemcpyAsync(krs.data(), h->excl_krs.raw(), sizeof(double) * n, cudaMemcpyDeviceToHost, h->stream);
    if (e == cudaSuccess) e = cudaStreamSynchronize(h->stream);
    if (e != cudaSuccess) return cuda_status(e);
    // internal offsets back to the caller's bead order
    auto ext = [&](int off) { return h->order_host.empty() ? off : 3 * h->order_host[off / 3]; };
    for (int64_t i = 0; i < n; ++i) {
        beads_out[4 * i] = ext(bs[i].x);
        beads_out[4 * i + 1] = ext(bs[i].y);
        beads_out[4 * i + 2] = ext(bs[i].z);
        beads_out[4 * i + 3] = ext(bs[i].w);
        // the device keeps krep*L1*L2; report it with unit lengths
        if (k_out) k_out[i] = krs[i];
        if (eqlen_out) {
            eqlen_out[2 * i] = 1.0;
            eqlen_out[2 * i + 1] = 1.0;
        }
    }
    return MEDYAN_OK;
}

}  // extern "C"

extern "C" medyan_status medyan_mech_boundary_load_forces(medyan_mech* h, const medyan_load_tips* tips,
                                                          double* load_out, int64_t capacity) {
    if (!h || !tips || tips->n_tips < 0) return MEDYAN_ERR_INVALID_ARG;
    const int nt = tips->n_tips;
    if (nt == 0) return MEDYAN_OK;
    if (!tips->cylinder || !tips->plus_end || !tips->n_mon || !tips->mon_size || !load_out)
        return MEDYAN_ERR_INVALID_ARG;
    NLBuilder* b = reinterpret_cast<NLBuilder*>(h->nl);
    if (!b) return MEDYAN_ERR_INVALID_ARG;  // no cylinder list: medyan_mech_set_cylinders first
    std::vector<long long> off(nt);
    long long tot = 0;
    for (int t = 0; t < nt; ++t) {
        if (tips->n_mon[t] < 0 || tips->cylinder[t] < 0 || tips->cylinder[t] >= b->n) return MEDYAN_ERR_INVALID_ARG;
        off[t] = tot;
        tot += tips->n_mon[t];
    }
    if (tot > capacity) return MEDYAN_ERR_CAPACITY;
    if (!b->has_boundary || b->bp.n_planes <= 0) {
        std::fill(load_out, load_out + tot, 0.0);
        return MEDYAN_OK;
    }
    if (!b->boundary_built) return MEDYAN_ERR_INVALID_ARG;  // medyan_mech_rebuild_neighbors first
    if (tot == 0) return MEDYAN_OK;
    cudaError_t e = cudaSetDevice(h->device);
    cudaStream_t s = h->stream;
    DevBuf<int> cyl, plus, nmon;
    DevBuf<double> mon, out;
    DevBuf<long long> doff;
    if (e == cudaSuccess) e = cyl.assign(tips->cylinder, nt, s);
    if (e == cudaSuccess) e = plus.assign(tips->plus_end, nt, s);
    if (e == cudaSuccess) e = nmon.assign(tips->n_mon, nt, s);
    if (e == cudaSuccess) e = mon.assign(tips->mon_size, nt, s);
    if (e == cudaSuccess) e = doff.assign(off.data(), nt, s);
    if (e == cudaSuccess) e = out.reserve(tot);
    if (e != cudaSuccess) return cuda_status(e);
    const int g = nt < 148 * 8 ? nt : 148 * 8;
    k_boundary_load<<<g, 128, 0, s>>>(b->view(), h->x.raw(), b->planes.raw(), b->bp.n_planes, b->counts_built.raw() + b->n,
                                      b->bp.k, b->bp.screen_length, nt, cyl.raw(), plus.raw(), nmon.raw(),
                                      mon.raw(), doff.raw(), out.raw());
    e = cudaGetLastError();
    if (e == cudaSuccess) e = cudaMemcpyAsync(load_out, out.raw(), sizeof(double) * tot, cudaMemcpyDeviceToHost, s);
    if (e == cudaSuccess) e = cudaStreamSynchronize(s);
    return cuda_status(e);
}
