// neigh.cu -- cell list and neighbour lists on the device.
//
// Replaces the host CSR flatten of LAMMPS neighbour lists plus the selection
// kernels get_environment_Steinhardt_Q (src/cvs/CVs_Steinhardt.cu:1324-1406),
// get_environment_Steinhardt_LocalQ (src/cvs/CVs_Steinhardt_Local.cu:1210-1285)
// and get_environment_Strufactor (src/cvs/CVs_Strufactor.cu:1014-1080).
//
// Per step: bin atoms to cells (counting sort: histogram, scan, scatter in
// atomic arrival order, then every atom moves to its rank by caller index
// within its cell, so the order is deterministic), then
// one thread per sorted atom walks its 9 neighbour-cell columns (z-adjacent
// cells are contiguous in the sorted order).  A candidate is decided by its
// FP32 cell-relative distance unless it lies within ~1e-5 of the bound, where
// the FP64 test on the caller's raw coordinates (the FP64 oracle's operation
// order) decides -- the neighbour sets are exact.
//
// With skin lists (NEIGH_SKIN) the cell list and candidate lists (cutoff +
// skin) are rebuilt only when k_refresh finds an atom that moved more than
// skin / 2 since the last rebuild (or NEIGH_EVERY steps have passed); every
// step the candidates are filtered to the exact lists at the current
// positions, so the neighbour sets are exact either way.  This is the model
// of the reference, which reads LAMMPS's skin lists and filters them by
// r < cutoff_r every step (src/cvs/CVs_Steinhardt.cu:135-147,
// src/core/neigh_hub.cu:191-222).
#include "persist.cuh"

#include <cooperative_groups.h>
#include <math_constants.h>

#include <atomic>

namespace mtd {

namespace {

namespace cg = cooperative_groups;


// The rebuild kernels return at once while the skin gate is closed (the
// gate is written by k_refresh, complete before pdl_entry returns).
__device__ __forceinline__ bool gate_closed(const SkinState *sk) {
    return sk && *(volatile const unsigned *)&sk->gate == 0u;
}


__global__ void k_bin(CellGrid g, SysDev s) {
    pdl_entry();
    if (gate_closed(s.skin)) return;
    bin_body(g, s, blockIdx.x);
}

// Exclusive block scan of one value per thread (blockDim.x == kScanBlock).
constexpr int kScanBlock = 1024;
__device__ __forceinline__ int block_excl_scan(int v, int &total) {
    __shared__ int warp_tot[32];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    int x = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        int y = __shfl_up_sync(0xffffffffu, x, o);
        if (lane >= o) x += y;
    }
    if (lane == 31) warp_tot[warp] = x;
    __syncthreads();
    if (warp == 0) {
        int t = warp_tot[lane];
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            int y = __shfl_up_sync(0xffffffffu, t, o);
            if (lane >= o) t += y;
        }
        warp_tot[lane] = t;
    }
    __syncthreads();
    total = warp_tot[31];
    const int excl = (warp > 0 ? warp_tot[warp - 1] : 0) + x - v;
    __syncthreads();
    return excl;
}

// Three-pass exclusive scan of the cell histogram: per-block scan, scan of the
// block totals, add-back.  The totals live in start[ncell + 1 ...].
__global__ void __launch_bounds__(kScanBlock) k_scan_blocks(const int *__restrict__ count, int *__restrict__ start,
                                                            int *__restrict__ bsum, int ncell, const SkinState *skin) {
    pdl_entry();
    if (gate_closed(skin)) return;
    const int i = blockIdx.x * kScanBlock + threadIdx.x;
    int total;
    const int e = block_excl_scan(i < ncell ? count[i] : 0, total);
    if (i < ncell) start[i] = e;
    if (threadIdx.x == 0) bsum[blockIdx.x] = total;
}

__global__ void __launch_bounds__(kScanBlock) k_scan_top(int *__restrict__ bsum, int nb, int *__restrict__ start,
                                                         int ncell, const SkinState *skin) {
    pdl_entry();
    if (gate_closed(skin)) return;
    int carry = 0;
    for (int base = 0; base < nb; base += kScanBlock) {
        const int i = base + threadIdx.x;
        int total;
        const int e = block_excl_scan(i < nb ? bsum[i] : 0, total);
        if (i < nb) bsum[i] = carry + e;
        carry += total;
    }
    if (threadIdx.x == 0) start[ncell] = carry;
}

__global__ void __launch_bounds__(kScanBlock) k_scan_add(int *__restrict__ start, const int *__restrict__ bsum,
                                                         int ncell, const SkinState *skin) {
    pdl_entry();
    if (gate_closed(skin)) return;
    const int i = blockIdx.x * kScanBlock + threadIdx.x;
    if (i < ncell) start[i] += bsum[blockIdx.x];
}

// Single-kernel add-back when the block totals fit one block: each block sums
// the totals of the blocks before it (the last block also writes the total).
__global__ void __launch_bounds__(kScanBlock) k_scan_add_fused(int *__restrict__ start, const int *__restrict__ bsum,
                                                               int ncell, int nb, const SkinState *skin) {
    pdl_entry();
    if (gate_closed(skin)) return;
    __shared__ int red[32];
    const int b = blockIdx.x, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    int v = threadIdx.x < b ? bsum[threadIdx.x] : 0;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
    if (lane == 0) red[warp] = v;
    __syncthreads();
    int off = 0;
#pragma unroll 1
    for (int w = 0; w < (kScanBlock >> 5); ++w) off += red[w];
    const int i = b * kScanBlock + threadIdx.x;
    if (i < ncell) start[i] += off;
    if (b == nb - 1 && threadIdx.x == 0) start[ncell] = off + bsum[b];
}



// Also zeroes the cell counts for the next build (the scan has consumed them).
__global__ void k_scatter(SysDev s, int ncell) {
    pdl_entry();
    if (gate_closed(s.skin)) return;
    scatter_body(s, ncell, blockIdx.x, gridDim.x);
}

// One thread per sorted slot: the atom that arrived there takes the place of
// its rank by caller index among its cell's members (removes the atomic
// arrival order), and its sorted per-atom arrays are written there.
__global__ void k_place(CellGrid g, SysDev s) {
    pdl_entry();
    if (gate_closed(s.skin)) return;
    place_body(g, s, blockIdx.x);
}

// The whole cell list in one launch of one cluster (16 SMs), its phases apart
// by cluster barriers instead of launches: bin, scan (a chunk of cells per
// block, the blocks' totals read from each other's shared memory; the counts
// are zeroed for the next build as they are read), scatter, place.  The same
// per-atom work and the same order as the five kernels, for up to an atom and
// 16 cells a thread (a sparse system's empty cells are work for the whole GPU).
// A small system's kernels are all latency, and five launches cost more than
// 16 SMs do: a step of local Q4 + Q6, three contexts in turn, 21.8 us at 4,000
// atoms and 29.2 with the five kernels, 24.9 and 29.3 at 8,000, 32.6 and 32.7 at
// 16,000, but 39.7 and 37.5 at 20,000, 59.1 and 45.9 at 42,000, 76.7 and 59.6 at
// 65,000 (a step alone 56 and 61, 62 and 63, 78 and 76, 97 and 96, 116 and 105,
// 147 and 127).
constexpr int kClusterBlocks = 16, kClusterAtoms = 1, kClusterCells = 16;   // per thread
__global__ void __launch_bounds__(kScanBlock) k_cells_cluster(CellGrid g, SysDev s) {
    pdl_entry();
    __shared__ int sum;
    if (gate_closed(s.skin)) return;
    cg::cluster_group cl = cg::this_cluster();
    const int rank = cl.block_rank();
    for (int v = rank; v * kScanBlock < s.n; v += kClusterBlocks) bin_body(g, s, v);
    cl.sync();
    const int per = (g.ncell + kClusterBlocks * kScanBlock - 1) / (kClusterBlocks * kScanBlock);
    const int c0 = (rank * kScanBlock + threadIdx.x) * per, c1 = min(c0 + per, g.ncell);
    int mine = 0;
    for (int c = c0; c < c1; ++c) mine += s.count[c];
    int total;
    int at = block_excl_scan(mine, total);
    if (threadIdx.x == 0) sum = total;
    cl.sync();
    for (int r = 0; r < rank; ++r) at += *cl.map_shared_rank(&sum, r);
    for (int c = c0; c < c1; ++c) {
        const int v = s.count[c];
        s.count[c] = 0;
        s.start[c] = at;
        at += v;
    }
    if (rank == kClusterBlocks - 1 && threadIdx.x == kScanBlock - 1) s.start[g.ncell] = s.n;
    cl.sync();   // also: no block leaves while another reads its total
    for (int v = rank; v * kScanBlock < s.n; v += kClusterBlocks) {
        const int i = v * kScanBlock + threadIdx.x;
        if (i < s.n) s.arrival[s.start[s.cellof[i]] + s.slot[i]] = i;
    }
    cl.sync();
    for (int v = rank; v * kScanBlock < s.n; v += kClusterBlocks) place_body(g, s, v);
}

template <int KIND>
__global__ void __launch_bounds__(kBlock) k_neighbors(CellGrid g, SysDev s, NeighSpec ns, NeighDev nd,
                                                      DevStatus *status) {
    pdl_entry();
    if (gate_closed(s.skin)) return;
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= s.n) return;
    const GeoF gf = geo_f(g, s.pf);
    const GeoD gd = geo_d(g, s.xs);
    const float4 a = s.pf[k];
    const int w = __float_as_int(a.w);
    const int cx = w & 1023, cy = (w >> 10) & 1023, cz = w >> 20;
    const int nz = g.nc[2];
    int cnt = 0;
    for (int ox = -1; ox <= 1; ++ox) {
        int x = cx + ox;
        if (g.periodic[0]) {
            if (g.nc[0] < 3 && ox != 0 && (g.nc[0] == 1 || ox == -1)) continue;
            x = (x + g.nc[0]) % g.nc[0];
        } else if (x < 0 || x >= g.nc[0]) continue;
        for (int oy = -1; oy <= 1; ++oy) {
            int y = cy + oy;
            if (g.periodic[1]) {
                if (g.nc[1] < 3 && oy != 0 && (g.nc[1] == 1 || oy == -1)) continue;
                y = (y + g.nc[1]) % g.nc[1];
            } else if (y < 0 || y >= g.nc[1]) continue;
            const int col = (x * g.nc[1] + y) * nz;
            // z cells of the column: one contiguous range unless the stencil wraps
            int zr[3][2], nr = 0;
            if (nz >= 3 && cz >= 1 && cz <= nz - 2) {
                zr[0][0] = cz - 1;
                zr[0][1] = cz + 1;
                nr = 1;
            } else if (nz >= 3 && g.periodic[2]) {
                if (cz == 0) {
                    zr[0][0] = 0; zr[0][1] = 1; zr[1][0] = nz - 1; zr[1][1] = nz - 1; nr = 2;
                } else {
                    zr[0][0] = nz - 2; zr[0][1] = nz - 1; zr[1][0] = 0; zr[1][1] = 0; nr = 2;
                }
            } else {
                zr[0][0] = max(cz - 1, 0);
                zr[0][1] = min(cz + 1, nz - 1);
                nr = 1;
            }
            for (int r = 0; r < nr; ++r) {
                const int jb = s.start[col + zr[r][0]], je = s.start[col + zr[r][1] + 1];
                for (int j = jb; j < je; ++j) {
                    if (j == k) continue;
                    const float4 b = s.pf[j];
                    float dx, dy, dz;
                    disp_f(gf, a, b, dx, dy, dz);
                    const float r2f = dx * dx + dy * dy + dz * dz;
                    if (!decide<KIND>(gd, ns, s.xs, k, j, r2f)) continue;
                    if (cnt < nd.M) nd.list[(size_t)cnt * s.npad + k] = j;
                    ++cnt;
                }
            }
        }
    }
    nd.count[k] = cnt;
    if (cnt > nd.M) note_overflow<KIND>(status, ns, cnt);
}


// Fast path, valid when every periodic dimension has at least three cells
// (neighbors_fast_body).
template <int KIND>
__global__ void __launch_bounds__(kBlock) k_neighbors_fast(CellGrid g, SysDev s, NeighSpec ns, NeighDev nd,
                                                           DevStatus *status) {
    pdl_entry();
    if (gate_closed(s.skin)) return;
    neighbors_fast_body<KIND>(g, s, ns, nd, status, blockIdx.x);
}

// Same lists as k_neighbors_fast, one warp per atom: lanes 0..26 read the
// stencil cells' ranges at once, the candidates of all cells are dealt to the
// lanes in list order, and a ballot packs the survivors.  Bound by latency
// where it is used: a thread per atom goes through some 50 (STEP) to 180
// candidates one after another with a few warps per SM, a warp per atom
// through two to six rounds of them (a lane per stencil cell in place of the
// dealing measured the same for STEP and a quarter longer for switches).  A
// smooth switch is evaluated for 32 candidates in range at a time.  With the
// cap of STEINH Q the warp also ranks its list (k_select_cap), from shared
// memory.
// (A candidate's cell is found by a bit mask of the cells that begin in its
// round; a binary search by shuffles cost 30 instructions more a round, 33 us
// against 27 at 32,000 atoms.)  Event intervals, before and now: 4,000 atoms,
// cutoff 3.9 with the cap 58 us (search 35, ranking 23) and 10; 32,000 atoms,
// cutoff 6.0 with the cap 101 and 37, without 54 and 27; 61,111 atoms, FERMI
// 125 and 53.
constexpr int kWarpAtoms = kBlock / 32;
template <int KIND, bool CAP>
__global__ void __launch_bounds__(kBlock) k_neighbors_warp(CellGrid g, SysDev s, NeighSpec ns, NeighDev nd,
                                                           DevStatus *status) {
    pdl_entry();
    __shared__ int held[CAP || KIND == NK_SWITCH ? kWarpAtoms : 1][kMaxCapList];
    __shared__ float held_r2[KIND == NK_SWITCH ? kWarpAtoms : 1][kMaxCapList];
    __shared__ float4 cells[kWarpAtoms][27];
    if (gate_closed(s.skin)) return;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, k = blockIdx.x * kWarpAtoms + warp;
    if (k >= s.n) return;   // whole warps; no block-wide synchronisation below
    const unsigned all = 0xffffffffu, below = (1u << lane) - 1;
    const GeoD gd = geo_d(g, s.xs);
    const float4 a = s.pf[k];
    const int w = __float_as_int(a.w);
    const int ox = lane / 9 - 1, oy = lane / 3 % 3 - 1, oz = lane % 3 - 1;
    int x = (w & 1023) + ox, y = ((w >> 10) & 1023) + oy, z = (w >> 20) + oz;
    bool cell = lane < 27;
    if (x < 0 || x >= g.nc[0]) {
        cell = cell && g.periodic[0];
        x += x < 0 ? g.nc[0] : -g.nc[0];
    }
    if (y < 0 || y >= g.nc[1]) {
        cell = cell && g.periodic[1];
        y += y < 0 ? g.nc[1] : -g.nc[1];
    }
    if (z < 0 || z >= g.nc[2]) {
        cell = cell && g.periodic[2];
        z += z < 0 ? g.nc[2] : -g.nc[2];
    }
    int first = 0, len = 0;
    if (cell) {
        const int key = cell_key(g, x, y, z);
        first = __ldg(s.start + key);
        len = __ldg(s.start + key + 1) - first;
    }
    int end = len;   // candidates up to and with this lane's cell
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int v = __shfl_up_sync(all, end, o);
        if (lane >= o) end += v;
    }
    const int begin = end - len, total = __shfl_sync(all, end, 31);
    // the non-empty cells in order: where candidate t lies (first - begin + t), the cell's shift
    const unsigned full = __ballot_sync(all, len > 0);
    if (len > 0)
        cells[warp][__popc(full & below)] = make_float4(__int_as_float(first - begin), (float)ox * g.hf[0] - a.x,
                                                        (float)oy * g.hf[1] - a.y, (float)oz * g.hf[2] - a.z);
    __syncwarp();
    int cnt = 0, wait = 0, opened = -1;   // opened: the last cell begun before this round
    const int most = min(nd.M, kMaxCapList);   // entries of a capped list; more are an overflow
    auto keep = [&](bool in, int j) {
        const unsigned hits = __ballot_sync(all, in);
        const int at = cnt + __popc(hits & below);
        if (CAP && in && at < most) held[warp][at] = j;
        if (!CAP && in && at < nd.M) nd.list[(size_t)at * s.npad + k] = j;
        cnt += __popc(hits);
    };
    // NK_SWITCH: the switch is evaluated for full warps of candidates in range
    auto decide_held = [&](int n) {
        __syncwarp();
        const int j = lane < n ? held[warp][lane] : k;
        const float r2f = lane < n ? held_r2[warp][lane] : 0.f;
        keep(lane < n && decide<KIND>(gd, ns, s.xs, k, j, r2f), j);
    };
    for (int t0 = 0; t0 < total; t0 += 32) {
        const int t = t0 + lane;
        const unsigned starts = __reduce_or_sync(all, len > 0 && (unsigned)(begin - t0) < 32u ? 1u << (begin - t0) : 0u);
        const float4 c = cells[warp][opened + __popc(starts & (below | 1u << lane))];
        opened += __popc(starts);
        const int j = __float_as_int(c.x) + t;
        float r2f = INFINITY;
        if (t < total && j != k) {
            const float4 b = __ldg(s.pf + j);
            const float dx = b.x + c.y, dy = b.y + c.z, dz = b.z + c.w;
            r2f = dx * dx + dy * dy + dz * dz;
        }
        if (KIND != NK_SWITCH) {
            keep(r2f < INFINITY && decide<KIND>(gd, ns, s.xs, k, j, r2f), j);
            continue;
        }
        // NaN fails, as in decide
        const bool in = r2f <= ns.hi2;
        const unsigned hits = __ballot_sync(all, in);
        const int at = wait + __popc(hits & below);
        if (in) {
            held[warp][at] = j;
            held_r2[warp][at] = r2f;
        }
        wait += __popc(hits);
        if (wait >= 32) {
            decide_held(32);
            const int j2 = held[warp][32 + lane];
            const float q2 = held_r2[warp][32 + lane];
            __syncwarp();
            held[warp][lane] = j2;
            held_r2[warp][lane] = q2;
            wait -= 32;
        }
    }
    if (KIND == NK_SWITCH && wait > 0) decide_held(wait);
    if (lane == 0) {
        nd.count[k] = cnt;
        if (cnt > (CAP ? most : nd.M)) note_overflow<KIND>(status, ns, cnt);
    }
    if (!CAP) return;
    __syncwarp();
    const int c = min(cnt, most);
    const double xk[3] = {s.xs[3 * k], s.xs[3 * k + 1], s.xs[3 * k + 2]};
    double r2[2];
    int id[2], jj[2], rank[2] = {0, 0};
#pragma unroll
    for (int e = 0; e < 2; ++e) {
        const int t = lane + 32 * e;
        r2[e] = CUDART_INF;
        id[e] = 0x7fffffff;
        jj[e] = 0;
        if (t < c) {
            jj[e] = held[warp][t];
            const double xj[3] = {s.xs[3 * jj[e]], s.xs[3 * jj[e] + 1], s.xs[3 * jj[e] + 2]};
            double d[3];
            r2[e] = exact_disp(gd, xk, xj, d);
            id[e] = s.perm[jj[e]];
        }
    }
    if (c <= 32) {
        for (int u = 0; u < c; ++u) {
            const double ru = __shfl_sync(all, r2[0], u);
            const int iu = __shfl_sync(all, id[0], u);
            rank[0] += ru < r2[0] || (ru == r2[0] && iu < id[0]);
        }
    } else {
        for (int u = 0; u < c; ++u) {
            const double ru = __shfl_sync(all, u < 32 ? r2[0] : r2[1], u);
            const int iu = __shfl_sync(all, u < 32 ? id[0] : id[1], u);
#pragma unroll
            for (int e = 0; e < 2; ++e) rank[e] += ru < r2[e] || (ru == r2[e] && iu < id[e]);
        }
    }
    double kr2 = CUDART_INF;
    int kid = 0x7fffffff;
    unsigned owner = 0;
#pragma unroll
    for (int e = 0; e < 2; ++e) {
        const bool mine = lane + 32 * e < c;
        if (mine) nd.list[(size_t)(lane + 32 * e) * s.npad + k] = jj[e] | (rank[e] < ns.cap ? 1 << kFlagBit : 0);
        const bool key = mine && c > ns.cap && rank[e] == ns.cap - 1;
        if (key) {
            kr2 = r2[e];
            kid = id[e];
        }
        owner |= __ballot_sync(all, key);
    }
    if (lane == (owner ? __ffs(owner) - 1 : 0)) {
        nd.key_r2[k] = kr2;
        nd.key_id[k] = kid;
        nd.nkept[k] = c < ns.cap ? c : ns.cap;
    }
}

// Same lists as k_neighbors_fast (same cells in the same order, same tests),
// with the warp's divergence taken out of the cell loop: each thread first
// records the non-empty cells of its 27-cell stencil in shared memory (a
// uniform pass), then walks all its candidates in one flat loop, moving to the
// next recorded cell when one runs out.  A warp then runs as many trips as
// its busiest lane has candidates, instead of, for each of 27 cells, as many
// as the fullest lane's cell holds.
constexpr int kFlatBlock = 128;
template <int KIND>
__global__ void __launch_bounds__(kFlatBlock) k_neighbors_flat(CellGrid g, SysDev s, NeighSpec ns, NeighDev nd,
                                                               DevStatus *status) {
    pdl_entry();
    // [cell][thread]: a lane's entry sits in the same bank whatever cell it reads
    __shared__ int2 rng[27][kFlatBlock];
    if (gate_closed(s.skin)) return;
    const int tid = threadIdx.x;
    const int k = blockIdx.x * blockDim.x + tid;
    if (k >= s.n) return;   // no block-wide synchronisation below
    const GeoD gd = geo_d(g, s.xs);
    const float4 a = s.pf[k];
    const int w = __float_as_int(a.w);
    const int cx = w & 1023, cy = (w >> 10) & 1023, cz = w >> 20;
    const int nx = g.nc[0], ny = g.nc[1], nz = g.nc[2];
    // the cell shift o h - offset for o = -1, 0, 1 per dimension (as k_neighbors_fast forms it)
    const float shx[3] = {-g.hf[0] - a.x, 0.f * g.hf[0] - a.x, g.hf[0] - a.x};
    const float shy[3] = {-g.hf[1] - a.y, 0.f * g.hf[1] - a.y, g.hf[1] - a.y};
    const float shz[3] = {-g.hf[2] - a.z, 0.f * g.hf[2] - a.z, g.hf[2] - a.z};
    int nr = 0;
#pragma unroll 1
    for (int ox = 0; ox < 3; ++ox) {
        int x = cx + ox - 1;
        if (x < 0 || x >= nx) {
            if (!g.periodic[0]) continue;
            x += x < 0 ? nx : -nx;
        }
#pragma unroll 1
        for (int oy = 0; oy < 3; ++oy) {
            int y = cy + oy - 1;
            if (y < 0 || y >= ny) {
                if (!g.periodic[1]) continue;
                y += y < 0 ? ny : -ny;
            }
#pragma unroll
            for (int oz = 0; oz < 3; ++oz) {
                int z = cz + oz - 1;
                if (z < 0 || z >= nz) {
                    if (!g.periodic[2]) continue;
                    z += z < 0 ? nz : -nz;
                }
                const int key = cell_key(g, x, y, z);
                const int b0 = __ldg(s.start + key), b1 = __ldg(s.start + key + 1);
                // end < 2^26, the stencil offsets (2 bits each) above it
                const unsigned code = (unsigned)ox | ((unsigned)oy << 2) | ((unsigned)oz << 4);
                if (b0 < b1) rng[nr++][tid] = make_int2(b0, (int)((unsigned)b1 | (code << 26)));
            }
        }
    }
    int cnt = 0;
    int r = 0, j = 0, je = 0;
    float sx = 0.f, sy = 0.f, sz = 0.f;
    auto open = [&]() {
        const int2 e = rng[r++][tid];
        const unsigned code = (unsigned)e.y >> 26;
        j = e.x;
        je = e.y & ((1 << 26) - 1);
        const unsigned qx = code & 3u, qy = (code >> 2) & 3u, qz = code >> 4;
        sx = qx == 0 ? shx[0] : (qx == 1 ? shx[1] : shx[2]);
        sy = qy == 0 ? shy[0] : (qy == 1 ? shy[1] : shy[2]);
        sz = qz == 0 ? shz[0] : (qz == 1 ? shz[1] : shz[2]);
    };
    bool live = nr > 0;
    float4 nxt = make_float4(0.f, 0.f, 0.f, 0.f);
    if (live) {
        open();
        nxt = __ldg(s.pf + j);
    }
    while (live) {
        const float4 b = nxt;
        const int jj = j;
        const float dx = b.x + sx, dy = b.y + sy, dz = b.z + sz;
        if (++j == je) {
            live = r < nr;
            if (live) open();
        }
        if (live) nxt = __ldg(s.pf + j);
        const float r2f = dx * dx + dy * dy + dz * dz;
        if (r2f > ns.hi2 || jj == k) continue;
        if (KIND != NK_CAND && !decide<KIND>(gd, ns, s.xs, k, jj, r2f)) continue;
        if (cnt < nd.M) nd.list[(size_t)cnt * s.npad + k] = jj;
        ++cnt;
    }
    nd.count[k] = cnt;
    if (cnt > nd.M) {
        if (KIND == NK_CAND) atomicMax(&status->cand_overflow, (unsigned)cnt);
        else note_overflow<KIND>(status, ns, cnt);
    }
}

// STEINH Q cap: keep the `cap` nearest by (r2, caller index), the order of the
// reference's strict-'>' insertion with ties resolved canonically.
__global__ void __launch_bounds__(kBlock) k_select_cap(CellGrid g, SysDev s, NeighSpec ns, NeighDev nd) {
    pdl_entry();
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= s.n) return;
    const GeoD gd = geo_d(g, s.xs);
    const int c = min(nd.count[k], min(nd.M, kMaxCapList));
    double r2[kMaxCapList];
    int id[kMaxCapList];
    const double xk[3] = {s.xs[3 * k], s.xs[3 * k + 1], s.xs[3 * k + 2]};
    for (int t = 0; t < c; ++t) {
        const int j = nd.list[(size_t)t * s.npad + k];
        const double xj[3] = {s.xs[3 * j], s.xs[3 * j + 1], s.xs[3 * j + 2]};
        double d[3];
        r2[t] = exact_disp(gd, xk, xj, d);
        id[t] = s.perm[j];
    }
    double kr2 = CUDART_INF;
    int kid = 0x7fffffff;
    for (int t = 0; t < c; ++t) {
        int rank = 0;
        for (int u = 0; u < c; ++u)
            if (r2[u] < r2[t] || (r2[u] == r2[t] && id[u] < id[t])) ++rank;
        if (rank < ns.cap) nd.list[(size_t)t * s.npad + k] |= (1 << kFlagBit);
        if (c > ns.cap && rank == ns.cap - 1) {
            kr2 = r2[t];
            kid = id[t];
        }
    }
    nd.key_r2[k] = kr2;
    nd.key_id[k] = kid;
    nd.nkept[k] = c < ns.cap ? c : ns.cap;
}

// Skin lists, every step: one thread per sorted slot of the last rebuild.
// Repacks the caller's positions into that order (xs, and pf as FP32 offsets
// from the slot's build cell, which stays within half a cell of it while the
// lists are valid), refreshes the group mask, and opens the gate when a
// rebuild is due: an atom moved more than skin / 2 (minimum image) since the
// build, a non-finite position, NEIGH_EVERY reached, or force (the sorted
// order is not valid yet, or the last rebuild gave up: nothing else is read).
__global__ void k_refresh(CellGrid g, SysDev s, int every, double half2, int force) {
    pdl_entry();
    SkinState *sk = s.skin;
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    // a rebuild that gave up leaves the sorted order and lists unusable: rebuild as if forced
    if (*(volatile const unsigned *)&sk->invalid) force = 1;
    if (k == 0 && (force || (every > 0 && sk->age >= (unsigned)every))) atomicOr(&sk->gate, 1u);
    if (force || k >= s.n) return;
    const int i = s.perm[k];
    const double x[3] = {s.x[3 * (size_t)i], s.x[3 * (size_t)i + 1], s.x[3 * (size_t)i + 2]};
    const bool finite = isfinite(x[0]) && isfinite(x[1]) && isfinite(x[2]);
    if (!finite && s.status) atomicOr(&s.status->bad_pos, 1u);
    double d2 = 0.0;
    const float4 p = s.pf[k];
    const int w = __float_as_int(p.w);
    const int cc[3] = {w & 1023, (w >> 10) & 1023, w >> 20};
    float off[3];
#pragma unroll
    for (int c = 0; c < 3; ++c) {
        double t = x[c] - s.xref[3 * (size_t)k + c];
        double o = (x[c] - g.lo[c]) - cc[c] * g.h[c];
        if (g.periodic[c]) {
            t -= g.L[c] * rint(t * g.invL[c]);
            o -= g.L[c] * rint((o - 0.5 * g.h[c]) * g.invL[c]);
        }
        d2 += t * t;
        off[c] = (float)o;
    }
    const unsigned moved = !(finite && d2 <= half2);
    const unsigned ballot = __ballot_sync(__activemask(), moved);   // one atomic per warp
    if (ballot && (threadIdx.x & 31) == __ffs(ballot) - 1) atomicOr(&sk->gate, 1u);
    s.xs[3 * (size_t)k] = x[0];
    s.xs[3 * (size_t)k + 1] = x[1];
    s.xs[3 * (size_t)k + 2] = x[2];
    s.pf[k] = make_float4(off[0], off[1], off[2], p.w);
    s.smask[k] = i < s.nown ? (s.mask ? s.mask[i] : -1) : 0;
}

// Skin lists, every step: the exact lists of one environment from its
// candidates.  reset (the first kernel after the gated rebuild kernels)
// records the step in the skin state and closes the gate.
template <int KIND>
__global__ void __launch_bounds__(kBlock) k_filter(CellGrid g, SysDev s, NeighSpec ns, NeighDev nd, NeighDev cand,
                                                   DevStatus *status, SkinState *reset) {
    pdl_entry();
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (reset && k == 0) {
        if (reset->gate) {
            reset->age = 1;
            reset->builds += 1;
        } else {
            reset->age += 1;
        }
        reset->gate = 0;
    }
    if (k >= s.n) return;
    filter_atom<KIND>(geo_f(g, s.pf), geo_d(g, s.xs), s.xs, ns, cand, nd, s.npad, k, status);
}

// Skin lists, the whole rebuild as one cooperative launch: while the gate is
// closed every block returns at once (one launch instead of six that each
// return at once); when it is open the phases run with grid barriers between
// them: cell counts zeroed, bin, chunk scan, chunk offsets, scatter, place,
// candidates.  The same per-thread bodies and 256-atom blocks as the separate
// kernels, so the sorted order and the candidate lists are the same.  A
// barrier wait that runs out marks the step (status->timeout, no deposit, no
// bias force) and the skin state invalid (the next step rebuilds from scratch).
__global__ void __launch_bounds__(kPersistBlock, 8) k_rebuild(CellGrid g, SysDev s, NeighSpec ns, NeighDev cd,
                                                           DevStatus *status, GridBar *bar, int limit, int stall) {
    pdl_entry();
    if (gate_closed(s.skin)) return;
    const int G = gridDim.x;
    const int nb = (s.n + kPersistBlock - 1) / kPersistBlock;
    const int nchunk = (g.ncell + kPersistBlock - 1) / kPersistBlock;
    int *bsum = s.start + g.ncell + 1;
    auto fail = [&]() {
        if (threadIdx.x == 0) {
            atomicOr(&status->timeout, 1u);
            atomicExch(&s.skin->invalid, 1u);
        }
    };
    // counts are zero after every complete build; a build that gave up may
    // have left some, so the rebuild starts from zero
    for (int c = blockIdx.x * kPersistBlock + threadIdx.x; c < g.ncell; c += G * kPersistBlock) s.count[c] = 0;
    if (!grid_barrier(bar, limit, stall && blockIdx.x == 0)) return fail();
    for (int v = blockIdx.x; v < nb; v += G) bin_body(g, s, v);
    if (!grid_barrier(bar, limit, false)) return fail();
    for (int v = blockIdx.x; v < nchunk; v += G) scan_chunk(s, g.ncell, v, bsum);
    if (!grid_barrier(bar, limit, false)) return fail();
    for (int v = blockIdx.x; v < nchunk; v += G) scan_offset(s, g.ncell, v, nchunk, bsum);
    if (!grid_barrier(bar, limit, false)) return fail();
    for (int v = blockIdx.x; v < nb; v += G) scatter_body(s, g.ncell, v, nb);
    if (!grid_barrier(bar, limit, false)) return fail();
    for (int v = blockIdx.x; v < nb; v += G) place_body(g, s, v);
    if (!grid_barrier(bar, limit, false)) return fail();
    if (blockIdx.x == 0 && threadIdx.x == 0) s.skin->invalid = 0u;
    for (int v = blockIdx.x; v < nb; v += G) neighbors_fast_body<NK_CAND>(g, s, ns, cd, status, v);
}

}  // namespace

int rebuild_blocks() {
    static int blocks[64] = {};
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return 0;
    if (blocks[dev] == 0) {
        int sms = 0, per = 0;
        if (cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess) return 0;
        if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, k_rebuild, kPersistBlock, 0) != cudaSuccess) return 0;
        blocks[dev] = per * sms > 0 ? per * sms : -1;
    }
    return blocks[dev] > 0 ? blocks[dev] : 0;
}

cudaError_t launch_rebuild(const CellGrid &g, const SysDev &s, const NeighSpec &ns, NeighDev cd, DevStatus *status,
                           GridBar *bar, int limit, int stall, cudaStream_t st) {
    const int blocks = rebuild_blocks();
    if (blocks < 1) return cudaErrorInvalidConfiguration;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(blocks);
    cfg.blockDim = dim3(kPersistBlock);
    cfg.stream = st;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeCooperative;
    at[0].val.cooperative = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    const cudaError_t e = cudaLaunchKernelEx(&cfg, k_rebuild, g, s, ns, cd, status, bar, limit, stall);
    prof_mark("skin_rebuild", st);
    return e;
}

// Whether k_cells_cluster can run on the current device (asked once).
static bool cells_cluster_ok() {
    static std::atomic<int> known[64];
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return false;
    int k = known[dev].load();
    if (k == 0) {
        cudaLaunchConfig_t cfg = {};
        cfg.gridDim = dim3(kClusterBlocks);
        cfg.blockDim = dim3(kScanBlock);
        cudaLaunchAttribute at[1];
        at[0].id = cudaLaunchAttributeClusterDimension;
        at[0].val.clusterDim.x = kClusterBlocks;
        at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
        cfg.attrs = at;
        cfg.numAttrs = 1;
        int fit = 0;
        k = cudaFuncSetAttribute(k_cells_cluster, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) == cudaSuccess &&
                    cudaOccupancyMaxActiveClusters(&fit, k_cells_cluster, &cfg) == cudaSuccess && fit > 0
                ? 1
                : -1;
        cudaGetLastError();
        known[dev].store(k);
    }
    return k > 0;
}

int launch_build_cells(const CellGrid &g, SysDev &s, cudaStream_t st) {
    const int nb = (s.n + kBlock - 1) / kBlock;
    const SkinState *sk = s.skin;
    constexpr int kThreads = kClusterBlocks * kScanBlock;
    if (s.n > 0 && s.n <= kThreads * kClusterAtoms && g.ncell <= kThreads * kClusterCells && cells_cluster_ok()) {
        launch_k_cluster(k_cells_cluster, kClusterBlocks, kClusterBlocks, kScanBlock, st, g, s);
        prof_mark("cell_list", st);
        return 1;
    }
    if (s.n > 0) launch_k(k_bin, nb, kBlock, 0, st, g, s);
    prof_mark("cell_bin", st);
    {
        const int sb = (g.ncell + kScanBlock - 1) / kScanBlock;
        int *bsum = s.start + g.ncell + 1;   // scratch after the ncell + 1 starts
        launch_k(k_scan_blocks, sb, kScanBlock, 0, st, s.count, s.start, bsum, g.ncell, sk);
        if (sb <= kScanBlock) {
            launch_k(k_scan_add_fused, sb, kScanBlock, 0, st, s.start, bsum, g.ncell, sb, sk);
        } else {
            launch_k(k_scan_top, 1, kScanBlock, 0, st, bsum, sb, s.start, g.ncell, sk);
            launch_k(k_scan_add, sb, kScanBlock, 0, st, s.start, bsum, g.ncell, sk);
        }
    }
    prof_mark("cell_scan", st);
    if (s.n > 0) {
        launch_k(k_scatter, nb, kBlock, 0, st, s, g.ncell);
        prof_mark("cell_scatter", st);
        launch_k(k_place, nb, kBlock, 0, st, g, s);
        prof_mark("cell_sort", st);
    }
    const int sb = (g.ncell + kScanBlock - 1) / kScanBlock;
    return (s.n > 0 ? 3 : 0) + (sb <= kScanBlock ? 2 : 3);
}

// One warp per atom up to 65,536 atoms, 131,072 for a smooth switch: there a
// thread per atom has the warps to hide its loads and runs fewer instructions
// (STEP at 64,000 atoms 38 us and 29 with a warp per atom, at 100,000 39 and
// 41, at 200,000 68 and 74; cutoff 6.0 at 32,000 54 and 27, at 87,000 57 and
// 60; FERMI at 64,000 110 and 55).
constexpr int kWarpMax = 65536;

int launch_neighbors(const CellGrid &g, const SysDev &s, const NeighSpec &ns, NeighDev nd, DevStatus *status,
                     cudaStream_t st) {
    if (s.n == 0) return 0;
    const int nb = (s.n + kBlock - 1) / kBlock;
    bool fast = true;
    for (int c = 0; c < 3; ++c)
        if (g.periodic[c] && g.nc[c] < 3) fast = false;
    // the fast path has three interchangeable shapes (identical lists): 256- or
    // 128-thread blocks of k_neighbors_fast, or k_neighbors_flat (autotuned)
    // skin-list candidates need the fast path (the context builds them only where it applies)
    bool capped = ns.cap > 0 && ns.kind != NK_CAND;
    if (fast && ns.variant == 0 && ns.kind != NK_CAND && s.n <= (ns.kind == NK_SWITCH ? 2 : 1) * kWarpMax) {
        const int wb = (s.n + kWarpAtoms - 1) / kWarpAtoms;
        if (ns.kind == NK_RANGE && capped) launch_k(k_neighbors_warp<NK_RANGE, true>, wb, kBlock, 0, st, g, s, ns, nd, status);
        else if (ns.kind == NK_RANGE) launch_k(k_neighbors_warp<NK_RANGE, false>, wb, kBlock, 0, st, g, s, ns, nd, status);
        else if (ns.kind == NK_STEP) launch_k(k_neighbors_warp<NK_STEP, false>, wb, kBlock, 0, st, g, s, ns, nd, status);
        else launch_k(k_neighbors_warp<NK_SWITCH, false>, wb, kBlock, 0, st, g, s, ns, nd, status);
        capped = false;   // ranked by the same kernel
    } else if (fast && ns.variant == 2 && s.n < (1 << 26)) {
        const int fb = (s.n + kFlatBlock - 1) / kFlatBlock;
        if (ns.kind == NK_RANGE) launch_k(k_neighbors_flat<NK_RANGE>, fb, kFlatBlock, 0, st, g, s, ns, nd, status);
        else if (ns.kind == NK_STEP) launch_k(k_neighbors_flat<NK_STEP>, fb, kFlatBlock, 0, st, g, s, ns, nd, status);
        else if (ns.kind == NK_CAND) launch_k(k_neighbors_flat<NK_CAND>, fb, kFlatBlock, 0, st, g, s, ns, nd, status);
        else launch_k(k_neighbors_flat<NK_SWITCH>, fb, kFlatBlock, 0, st, g, s, ns, nd, status);
    } else if (fast) {
        const int tb = ns.variant == 1 ? 128 : kBlock;
        const int gb = (s.n + tb - 1) / tb;
        if (ns.kind == NK_RANGE) launch_k(k_neighbors_fast<NK_RANGE>, gb, tb, 0, st, g, s, ns, nd, status);
        else if (ns.kind == NK_STEP) launch_k(k_neighbors_fast<NK_STEP>, gb, tb, 0, st, g, s, ns, nd, status);
        else if (ns.kind == NK_CAND) launch_k(k_neighbors_fast<NK_CAND>, gb, tb, 0, st, g, s, ns, nd, status);
        else launch_k(k_neighbors_fast<NK_SWITCH>, gb, tb, 0, st, g, s, ns, nd, status);
    } else if (ns.kind == NK_RANGE) launch_k(k_neighbors<NK_RANGE>, nb, kBlock, 0, st, g, s, ns, nd, status);
    else if (ns.kind == NK_STEP) launch_k(k_neighbors<NK_STEP>, nb, kBlock, 0, st, g, s, ns, nd, status);
    else launch_k(k_neighbors<NK_SWITCH>, nb, kBlock, 0, st, g, s, ns, nd, status);
    prof_mark(ns.kind == NK_CAND ? "neighbor_candidates" : "neighbors", st);
    if (capped) launch_select_cap(g, s, ns, nd, st);
    return capped ? 2 : 1;
}

void launch_select_cap(const CellGrid &g, const SysDev &s, const NeighSpec &ns, NeighDev nd, cudaStream_t st) {
    if (s.n == 0) return;
    const int nb = (s.n + kBlock - 1) / kBlock;
    launch_k(k_select_cap, nb, kBlock, 0, st, g, s, ns, nd);
    prof_mark("select_cap", st);
}

void launch_refresh(const CellGrid &g, const SysDev &s, int every, double half_skin, int force, cudaStream_t st) {
    const int nb = s.n > 0 ? (s.n + kBlock - 1) / kBlock : 1;
    launch_k(k_refresh, nb, kBlock, 0, st, g, s, every, half_skin * half_skin, force);
    prof_mark("skin_refresh", st);
}

void launch_filter(const CellGrid &g, const SysDev &s, const NeighSpec &ns, NeighDev nd, NeighDev cand,
                   DevStatus *status, SkinState *reset, cudaStream_t st) {
    const int nb = s.n > 0 ? (s.n + kBlock - 1) / kBlock : 1;
    if (ns.kind == NK_RANGE) launch_k(k_filter<NK_RANGE>, nb, kBlock, 0, st, g, s, ns, nd, cand, status, reset);
    else if (ns.kind == NK_STEP) launch_k(k_filter<NK_STEP>, nb, kBlock, 0, st, g, s, ns, nd, cand, status, reset);
    else launch_k(k_filter<NK_SWITCH>, nb, kBlock, 0, st, g, s, ns, nd, cand, status, reset);
    prof_mark("skin_filter", st);
}

}  // namespace mtd
