// hillsum.cu -- V(s) = sum_h w_h exp(-|s - c_h|^2 / (2 sigma_h^2)) and its
// gradient in FP64 over a batch of CV points.  No counterpart in the reference
// (its grids are its only bias representation).
//
// What bounds it: the FP64 pipe (64 lanes per SM and clock).  One thread per
// point over every hill costs about 40 FP64 operations per (point, hill) pair,
// most of them in the exponential, although 88 % of the pairs of a 4D bias lie
// beyond the 8.9 sigma where a hill counts.  So:
//   * the points are put in cells of the CV box (a counting sort of their
//     indices), and a block takes 32 consecutive ones, a compact piece of the
//     box.  A point's sum runs over its hills in the same order whatever its
//     neighbours in the block, so the order of the sort (atomics) does not
//     reach the result;
//   * the block's warps split the hills, 32 Q consecutive ones at a time in
//     deposit order, every Q-th for one split (a metadynamics run deposits
//     along a trajectory, so the 32 are close together and every split gets the
//     same share of the near ones; with 32 consecutive hills a split a quarter
//     of the warps waited at the block's end).  A warp tests 32 such groups at
//     once by their bounding boxes, one per lane, then the 32 hills of a
//     surviving group against its points' box, and gathers the survivors in
//     shared memory in order.  Hills in random order cost the box tests (under
//     a tenth of the pair work) and lose nothing;
//   * a pair is 24 FP64 operations: 2^(-x/32) for x = 32 log2(e) r^2 / (2 s^2)
//     from a 32-entry table and a degree-5 polynomial on |f| <= 1/2 (the
//     degree-6 Taylor polynomial with its last term folded into the lower ones
//     by the Chebyshev polynomial T6: error 7e-17), with x's integer part taken
//     by the 1.5 * 2^52 addition and no separate reduction of the argument.
//     The table is one entry per lane, read by shuffles (a table in shared
//     memory took 7 of the 11 wavefronts of a pair).
// 65,536 uniform points in a 4D box, 20,000 hills (27 % of the pairs are near
// a block's box): 5,274 us before, 990 now, with the FP64 pipe 60 % busy while
// blocks run; error against 64-bit torch 6.5e-16 (5.4e-15 before).  Sums of few
// hills or few pairs go without the sorting, or without the blocks (few_hills,
// few_pairs).
#include "hillsum.h"

#include <cooperative_groups.h>

#include <algorithm>
#include <cmath>

namespace mtd {

namespace {

namespace cg = cooperative_groups;

constexpr int kIn = 4;
constexpr int kTab = 32;             // table entries per octave, one per lane
constexpr int kWarps = 8;            // warps per block
constexpr int kMaxSplit = 8;         // blocks per cluster
constexpr int kBuf = 64;             // gathered hills per warp
constexpr int kBoxRec = 9;           // rows of group boxes: lo[4], hi[4], largest cut
constexpr int kMaxCells = 16384;

struct Cells {
    int nb[kIn];
    double lo[kIn], sc[kIn];         // bin = (s - lo) * sc
};

__device__ __forceinline__ int cell_of(const Cells &c, int D, const double *__restrict__ p) {
    int key = 0;
    for (int k = 0; k < D; ++k) {
        // NaN and values outside land in an edge bin
        const double u = fmin(fmax((p[k] - c.lo[k]) * c.sc[k], 0.0), (double)(c.nb[k] - 1));
        key = key * c.nb[k] + (int)u;
    }
    return key;
}

// Hill h packed for pair_add; past nh a cut of 0, which reaches no point.
__device__ __forceinline__ void load_hill(const double *__restrict__ hills, int h, int nh, double2 (&r)[4]) {
#pragma unroll
    for (int e = 0; e < 4; ++e) r[e] = make_double2(0.0, 0.0);
    if (h < nh) {
        const double2 *src = reinterpret_cast<const double2 *>(hills + (size_t)h * kHillRec);
#pragma unroll
        for (int e = 0; e < 4; ++e) r[e] = src[e];
        // 32 log2(e) / (2 sigma^2); finite, so that a hill on the point itself has the exponent 0
        r[2].y = fmin(r[2].y * (1.4426950408889634074 * kTab), 1.7976931348623157e308);
        if (!isfinite(r[3].x)) r[3].y = 0.0;      // a width whose 1 / sigma^2 overflows reaches no point
    }
}

// Blocks below `npb` count the points of each cell; the others, one warp per
// group of 32 hills (hills q, q + Q, ... of a run of 32 Q, for split q), write the groups' bounding boxes (rows of ng) and the
// hills as four rows of pairs (c0 c1, c2 c3, w x/r^2, 1/sigma^2 cut), which a
// warp reads 512 contiguous bytes at a time.
__global__ void __launch_bounds__(256) k_hs_count(Cells c, int D, int npts, const double *__restrict__ pts, int ps,
                                                  int npb, int *__restrict__ count, int nh, int ng, int Q,
                                                  const double *__restrict__ hills, double *__restrict__ boxes,
                                                  double2 *__restrict__ rows) {
    if ((int)blockIdx.x < npb) {
        const int i = blockIdx.x * blockDim.x + threadIdx.x;
        if (i < npts) atomicAdd(count + cell_of(c, D, pts + (size_t)i * ps), 1);
        return;
    }
    const int lane = threadIdx.x & 31, g = ((int)blockIdx.x - npb) * 8 + (threadIdx.x >> 5);
    const int h = g / Q * 32 * Q + lane * Q + g % Q;
    if (g >= ng) return;
    double2 r[4];
    load_hill(hills, h, nh, r);
#pragma unroll
    for (int e = 0; e < 4; ++e) rows[((size_t)e * ng + g) * 32 + lane] = r[e];
    const double cen[kIn] = {r[0].x, r[0].y, r[1].x, r[1].y};
    double cut = r[3].y;
    for (int o = 16; o > 0; o >>= 1) cut = fmax(cut, __shfl_xor_sync(0xffffffffu, cut, o));
    if (lane == 0) boxes[(size_t)8 * ng + g] = cut;
#pragma unroll
    for (int k = 0; k < kIn; ++k) {
        double lo = h < nh ? cen[k] : INFINITY, hi = h < nh ? cen[k] : -INFINITY;
        for (int o = 16; o > 0; o >>= 1) {
            lo = fmin(lo, __shfl_xor_sync(0xffffffffu, lo, o));
            hi = fmax(hi, __shfl_xor_sync(0xffffffffu, hi, o));
        }
        if (lane == 0) {
            boxes[(size_t)k * ng + g] = lo;
            boxes[(size_t)(kIn + k) * ng + g] = hi;
        }
    }
}

// Exclusive scan of the cell counts in place (one block).
__global__ void __launch_bounds__(1024) k_hs_scan(int ncell, int *count) {
    __shared__ int wsum[32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int per = (ncell + 1023) / 1024, a = min(ncell, (int)threadIdx.x * per), b = min(ncell, a + per);
    int s = 0;
    for (int e = a; e < b; ++e) s += count[e];
    int inc = s;
    for (int o = 1; o < 32; o <<= 1) {
        const int v = __shfl_up_sync(0xffffffffu, inc, o);
        if (lane >= o) inc += v;
    }
    if (lane == 31) wsum[warp] = inc;
    __syncthreads();
    if (warp == 0) {
        int w = wsum[lane];
        for (int o = 1; o < 32; o <<= 1) {
            const int v = __shfl_up_sync(0xffffffffu, w, o);
            if (lane >= o) w += v;
        }
        wsum[lane] = w;
    }
    __syncthreads();
    int run = inc - s + (warp ? wsum[warp - 1] : 0);
    for (int e = a; e < b; ++e) {
        const int v = count[e];
        count[e] = run;
        run += v;
    }
}

__global__ void __launch_bounds__(256) k_hs_place(Cells c, int D, int npts, const double *__restrict__ pts, int ps,
                                                  int *__restrict__ cursor, int *__restrict__ perm) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < npts) perm[atomicAdd(cursor + cell_of(c, D, pts + (size_t)i * ps), 1)] = i;
}

struct Acc {
    double v, g[kIn];
};

// One gathered hill at one point.  A pair beyond the cut adds zeros (its r^2
// is replaced by 0 so that the exponential stays finite).
__device__ __forceinline__ void pair_add(const double2 *__restrict__ rec, const double (&s)[kIn], double tab,
                                         Acc &acc) {
    constexpr double kMagic = 6755399441055744.0;   // 1.5 * 2^52
    // exp(-kL f): f^6 / 720 on |f| <= 1/2 is 1.5 f^4 / 4 - 9 f^2 / 256 + 1 / 2048 + T6(2 f) / 2048
    constexpr double kL = 0.69314718055994530942 / kTab, k6 = kL * kL * kL * kL * kL * kL / 720;
    constexpr double c1 = -kL, c2 = kL * kL / 2 - k6 * 9 / 256, c3 = -kL * kL * kL / 6,
                     c4 = kL * kL * kL * kL / 24 + k6 * 3 / 8, c5 = -kL * kL * kL * kL * kL / 120;
    const double2 a = rec[0], b = rec[kBuf], wq = rec[2 * kBuf], ic = rec[3 * kBuf];
    const double d0 = s[0] - a.x, d1 = s[1] - a.y, d2 = s[2] - b.x, d3 = s[3] - b.y;
    double r2 = fma(d3, d3, fma(d2, d2, fma(d1, d1, d0 * d0)));
    // r2 >= 0: it compares as an integer, off the FP64 pipe (a NaN is above every cut)
    const bool in = (unsigned long long)__double_as_longlong(r2) < (unsigned long long)__double_as_longlong(ic.y);
    r2 = in ? r2 : 0.0;
    const double t = fma(r2, wq.y, kMagic);
    const int n = __double2loint(t);
    const double f = fma(r2, wq.y, kMagic - t);
    const double T = __shfl_sync(0xffffffffu, tab, n);   // lane n & 31
    const double Ts = __hiloint2double(__double2hiint(T) - ((n >> 5) << 20), __double2loint(T));
    double p = fma(f, c5, c4);
    p = fma(p, f, c3);
    p = fma(p, f, c2);
    p = fma(p, f, c1);
    p = fma(p, f, 1.0);
    double e = (wq.x * Ts) * p;
    e = in ? e : 0.0;
    acc.v += e;
    const double ec = e * ic.x;
    acc.g[0] = fma(-ec, d0, acc.g[0]);
    acc.g[1] = fma(-ec, d1, acc.g[1]);
    acc.g[2] = fma(-ec, d2, acc.g[2]);
    acc.g[3] = fma(-ec, d3, acc.g[3]);
}

// A point's coordinates; one that is not finite stands at 1e150 and is written as zeros.
__device__ __forceinline__ bool load_point(const double *__restrict__ pts, int ps, int D, int i, double (&s)[kIn]) {
    bool fin = i >= 0;
#pragma unroll
    for (int k = 0; k < kIn; ++k) {
        s[k] = i >= 0 && k < D ? pts[(size_t)i * ps + k] : 0.0;
        fin = fin && isfinite(s[k]);
    }
#pragma unroll
    for (int k = 0; k < kIn; ++k)
        if (!fin) s[k] = 1e150;
    return fin;
}

// A thread per point over all hills in deposit order: for few hills, where a
// block's box tests and the sum of its splits cost more than the pairs.
constexpr int kPlainBlock = 128;
__global__ void __launch_bounds__(kPlainBlock)
    k_hillsum_plain(int D, int npts, const double *__restrict__ pts, int ps, int nh, const double *__restrict__ hills,
                    double *__restrict__ V, double *__restrict__ dV, int gs) {
    __shared__ double2 tile[4][kBuf];
    const int slot = blockIdx.x * kPlainBlock + threadIdx.x, i = slot < npts ? slot : -1;
    const double tab = exp2(-(double)(threadIdx.x & 31) / kTab);
    double s[kIn];
    const bool fin = load_point(pts, ps, D, i, s);
    Acc acc{};
    for (int h0 = 0; h0 < nh; h0 += kBuf) {
        const int c = min(kBuf, nh - h0);
        __syncthreads();
        if (threadIdx.x < kBuf) {
            double2 r[4];
            load_hill(hills, h0 + threadIdx.x, nh, r);
#pragma unroll
            for (int e = 0; e < 4; ++e) tile[e][threadIdx.x] = r[e];
        }
        __syncthreads();
#pragma unroll 4
        for (int e = 0; e < c; ++e) pair_add(tile[0] + e, s, tab, acc);
    }
    if (i < 0) return;
    V[i] = fin ? acc.v : 0.0;
    if (dV)
#pragma unroll
        for (int k = 0; k < kIn; ++k)
            if (k < gs && (k < D || gs == kIn)) dV[(size_t)i * gs + k] = fin ? acc.g[k] : 0.0;
}

// Squared distance between two boxes (a point is a box of no size); NaN bounds
// give NaN, which is below no cut.
__device__ __forceinline__ double gap2(double plo, double phi, double lo, double hi) {
    double d = plo - hi;
    if (!(d > lo - phi)) d = lo - phi;
    if (d <= 0.0) d = 0.0;
    return d * d;
}

// A block's warps share 32 points and split the hills, and so do the blocks of
// a cluster: split q of Q takes groups q, q + Q, ...; the splits' sums are
// added in split order.  (Warps with points of their own finish apart, by their
// share of the hills: 2.5 warps per issue waited at the block's end.)
// RAW: the hills as they are, without the rows and boxes of a scratch, each group
// tested hill by hill; the same sums bit for bit (a hill left out adds zeros).
template <bool RAW>
__global__ void __launch_bounds__(kWarps * 32, 2)
    k_hillsum(int D, int npts, const double *__restrict__ pts, int ps, const int *__restrict__ perm, int nh,
              const double *__restrict__ hills, int ng, const double2 *__restrict__ rows,
              const double *__restrict__ boxes, double *__restrict__ V, double *__restrict__ dV, int gs) {
    __shared__ double2 buf[kWarps][4][kBuf];
    cg::cluster_group cl = cg::this_cluster();
    const int nsplit = cl.num_blocks(), rank = cl.block_rank();
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int Q = kWarps * nsplit, q = warp + kWarps * rank;
    const int slot = (int)blockIdx.x / nsplit * 32 + lane;
    const int i = slot < npts ? (perm ? perm[slot] : slot) : -1;
    const double tab = exp2(-(double)lane / kTab);
    double s[kIn], plo[kIn], phi[kIn];
    const bool fin = load_point(pts, ps, D, i, s);
    // a point that is not finite is within reach of no hill: its box is empty
#pragma unroll
    for (int k = 0; k < kIn; ++k) {
        plo[k] = fin ? s[k] : INFINITY;
        phi[k] = fin ? s[k] : -INFINITY;
    }
#pragma unroll
    for (int k = 0; k < kIn; ++k)
        for (int o = 16; o > 0; o >>= 1) {
            plo[k] = fmin(plo[k], __shfl_xor_sync(0xffffffffu, plo[k], o));
            phi[k] = fmax(phi[k], __shfl_xor_sync(0xffffffffu, phi[k], o));
        }
    Acc acc{};
    int held = 0;
    double2 *mine = buf[warp][0];
    for (int g0 = q; g0 < ng; g0 += 32 * Q) {
        const int gl = g0 + lane * Q;
        bool near = RAW && gl < ng;
        if (!RAW && gl < ng) {
            const double *bx = boxes + gl;
            double r2 = 0.0;
#pragma unroll
            for (int k = 0; k < kIn; ++k) r2 += gap2(plo[k], phi[k], bx[(size_t)k * ng], bx[(size_t)(kIn + k) * ng]);
            near = r2 < bx[(size_t)8 * ng];
        }
        unsigned todo = __ballot_sync(0xffffffffu, near);
        while (todo) {
            const int t = __ffs(todo) - 1;
            todo &= todo - 1;
            const int g = g0 + t * Q;
            double2 r[4];
            if (RAW) {
                load_hill(hills, g / Q * 32 * Q + lane * Q + g % Q, nh, r);
            } else {
                const double2 *src = rows + (size_t)g * 32 + lane;
#pragma unroll
                for (int e = 0; e < 4; ++e) r[e] = src[(size_t)e * ng * 32];
            }
            const double d2 = gap2(plo[0], phi[0], r[0].x, r[0].x) + gap2(plo[1], phi[1], r[0].y, r[0].y) +
                              gap2(plo[2], phi[2], r[1].x, r[1].x) + gap2(plo[3], phi[3], r[1].y, r[1].y);
            const bool hit = d2 < r[3].y;
            const unsigned hits = __ballot_sync(0xffffffffu, hit);
            if (hit) {
                double2 *dst = mine + held + __popc(hits & ((1u << lane) - 1));
#pragma unroll
                for (int e = 0; e < 4; ++e) dst[e * kBuf] = r[e];
            }
            held += __popc(hits);
            if (held > kBuf - 32) {
                __syncwarp();
#pragma unroll 4
                for (int e = 0; e < held; ++e) pair_add(mine + e, s, tab, acc);
                held = 0;
                __syncwarp();
            }
        }
    }
    __syncwarp();
    for (int e = 0; e < held; ++e) pair_add(mine + e, s, tab, acc);
    // the warps' sums, [5][warp][lane] over the hill buffers, by five warps in warp
    // order; then the blocks' of the cluster, [5][lane] behind them, in block order
    constexpr int kT = kWarps * 32;
    static_assert(sizeof(buf) >= (1 + kIn) * (kT + 32) * sizeof(double) && kWarps > kIn, "room and warps for the sums");
    __syncthreads();
    double *red = &buf[0][0][0].x, *tot = red + (1 + kIn) * kT;
    red[threadIdx.x] = acc.v;
#pragma unroll
    for (int k = 0; k < kIn; ++k) red[(1 + k) * kT + threadIdx.x] = acc.g[k];
    __syncthreads();
    double o = 0.0;
    if (warp <= kIn) {
#pragma unroll
        for (int w = 0; w < kWarps; ++w) o += red[warp * kT + w * 32 + lane];
    }
    if (nsplit > 1) {
        if (warp <= kIn) tot[warp * 32 + lane] = o;
        cl.sync();
        if (rank == 0 && warp <= kIn) {
            o = 0.0;
            for (int b = 0; b < nsplit; ++b) o += cl.map_shared_rank(tot, b)[warp * 32 + lane];
        }
        cl.sync();   // no block leaves while another reads its sums
    }
    if (rank == 0 && i >= 0) {
        if (!fin) o = 0.0;
        if (warp == 0) V[i] = o;
        else if (dV && warp <= gs && (warp <= D || gs == kIn)) dV[(size_t)i * gs + warp - 1] = o;
    }
}

}  // namespace

namespace {
// Cells of about 32 points: the widest bins are halved until there are enough.
int make_cells(Cells &c, int D, const double *lo, const double *hi, int npts) {
    int ncell = 1;
    for (int k = 0; k < D; ++k) c.nb[k] = 1;
    while (ncell * 32 < npts && ncell < kMaxCells) {
        int w = 0;
        for (int k = 1; k < D; ++k)
            if ((hi[k] - lo[k]) / c.nb[k] > (hi[w] - lo[w]) / c.nb[w]) w = k;
        c.nb[w] *= 2;
        ncell *= 2;
    }
    for (int k = 0; k < D; ++k) {
        c.lo[k] = lo[k];
        c.sc[k] = c.nb[k] / (hi[k] - lo[k]);
    }
    return ncell;
}
}  // namespace

// The routes, by measurement (4D, 1 to 20,000 hills, 500 to 65,536 points; us):
// Few hills on many points: a thread per point.  Blocks of 32 points cost 3 to 5 us
// a round (two blocks an SM: 9,472 points) whatever the hills.  More than two
// rounds: 100 hills, 37,000 points 15 and 21 in blocks, 65,536 points 21 and 35;
// 300 hills 37 and 39, 54 and 57; but 600 hills on 65,536 points 101 and 70.  More
// than one: 16,000 points 6.0 and 9.2 with 10 hills, 8.7 and 10.7 with 50, but 14
// and 13 with 100.  8,000 points 8.6 and 6.7 with 50.
static bool few_hills(int npts, int nh) {
    constexpr int round = 32 * 2 * 148;
    return (nh <= 300 && npts > 2 * round) || (nh <= 64 && npts > round);
}

// Few pairs: no sorting and no group boxes, whose kernels cost about 18 us.  1,000
// hills, 4,000 points 19 and 33 sorted, 8,000 points 29 and 41, 16,000 points 54
// and 48; 2,500 hills, 4,000 points 36 and 44, 8,000 points 64 and 56; 10,000
// hills, 1,000 points 36 and 48; but 20,000 hills, 500 points 64 and 54: every
// pair of an unsorted block is computed, 3.2 us per 1,000 hills at least.
static bool few_pairs(int npts, int nh) { return nh <= 12000 && (long long)npts * nh <= 12000000; }

// Blocks of a cluster that split the hills: as many as are resident (two an SM),
// times a wave for each 2,500 hills up to eight, since the points' shares of the
// hills are unequal.  A split costs each block its box tests, half-full buffers and
// the sum over the cluster: 20,000 hills, 65,536 points 1,024 in one block each,
// 989 in two, 1,076 in four, 4,000 points 269, 222, 154 and 144 in eight; 1,000
// hills, 16,000 points 48, 53, 65 and 99, 500 points 33, 27, 24 and 23.
static int splits(int npts, int nh) {
    const double blocks = 148 * 2 * std::min(8.0, nh / 2500.0);
    int split = 1;
    while (split < kMaxSplit && (npts + 31) / 32 * split < blocks) split *= 2;
    return split;
}

size_t hillsum_scratch(int npts, int nh) {
    if (few_hills(npts, nh) || few_pairs(npts, nh)) return 0;
    const size_t run = 32 * kWarps * kMaxSplit, ng = (nh + run - 1) / run * (run / 32);
    return sizeof(double2) * 4 * 32 * ng + sizeof(double) * kBoxRec * ng + sizeof(int) * ((size_t)kMaxCells + npts);
}

cudaError_t hillsum_batch(int D, const double *lo, const double *hi, int npts, const double *pts, int ps, int nh,
                          const double *hills, double *V, double *dV, int gs, void *scratch, cudaStream_t st) {
    if (npts <= 0) return cudaSuccess;
    const int nsplit = splits(npts, nh);
    if (few_hills(npts, nh)) {
        k_hillsum_plain<<<(npts + kPlainBlock - 1) / kPlainBlock, kPlainBlock, 0, st>>>(D, npts, pts, ps, nh, hills, V, dV,
                                                                                       gs);
        return cudaGetLastError();
    }
    Cells c{};
    const int ncell = make_cells(c, D, lo, hi, npts);
    const int Q = kWarps * nsplit, ng = (nh + 32 * Q - 1) / (32 * Q) * Q;
    const bool raw = !scratch, sorted = !raw && ncell > 1;
    double2 *rows = static_cast<double2 *>(scratch);
    double *boxes = reinterpret_cast<double *>(rows + (size_t)4 * 32 * ng);
    int *count = reinterpret_cast<int *>(boxes + (size_t)kBoxRec * ng), *perm = count + ncell;
    const int npb = sorted ? (npts + 255) / 256 : 0;
    if (sorted) cudaMemsetAsync(count, 0, sizeof(int) * ncell, st);
    if (!raw && npb + ng > 0)
        k_hs_count<<<npb + (ng + 7) / 8, 256, 0, st>>>(c, D, npts, pts, ps, npb, count, nh, ng, Q, hills, boxes, rows);
    if (sorted) {
        k_hs_scan<<<1, 1024, 0, st>>>(ncell, count);
        k_hs_place<<<npb, 256, 0, st>>>(c, D, npts, pts, ps, count, perm);
    }
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3((unsigned)((npts + 31) / 32 * nsplit));
    cfg.blockDim = dim3(kWarps * 32);
    cfg.stream = st;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = (unsigned)nsplit;
    at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    const cudaError_t e =
        cudaLaunchKernelEx(&cfg, raw ? k_hillsum<true> : k_hillsum<false>, D, npts, pts, ps,
                           (const int *)(sorted ? perm : nullptr), nh, hills, ng, (const double2 *)rows,
                           (const double *)boxes, V, dV, gs);
    return e != cudaSuccess ? e : cudaGetLastError();
}

}  // namespace mtd
