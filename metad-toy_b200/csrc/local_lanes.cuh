// local_lanes.cuh -- the STEINH L passes with kLanes lanes per atom, for systems
// too small to fill the GPU with a thread per atom (local_body.cuh, whose
// definitions these share).  Each lane takes every kLanes-th neighbour; the
// lanes' record sums are added by a butterfly that leaves each lane a slice of
// the record, so norms, scaling and stores go on in slices.
// Bound by latency: a thread per atom waits for its 8 to 20 neighbours' records
// one after another, with a fifth of the GPU's warps.  Event intervals at 4,000
// atoms, thread and lanes: STEP in FP64 q 14 us and 9, LQ 19 and 11, lambda 18
// and 10, forces 27 and 10; FERMI in mixed precision 19 and 10, 25 and 13, 24
// and 11, 51 and 14.
#pragma once

#include "local_body.cuh"

namespace mtd {

// A record padded to a whole number of slices: lane `sub` of an atom holds
// elements [sub * W, sub * W + W) after spread().
template <int LA, int LB, typename T> struct LSlice {
    using S = LSet<LA, LB, T>;
    static constexpr int P = (S::SQ + kLanes - 1) / kLanes * kLanes, W = P / kLanes;
    T v[P];

    __device__ __forceinline__ LSlice() {
#pragma unroll
        for (int e = 0; e < P; ++e) v[e] = T(0);
    }
    // Adds the lanes' records; v[0 .. W) is then this lane's slice.
    __device__ __forceinline__ void spread(int sub) {
        static_assert(kLanes == 8, "three halving steps");
#pragma unroll
        for (int st = 0; st < 3; ++st) {
            const int o = kLanes >> (st + 1), h = P >> (st + 1);
            const bool up = (sub & o) != 0;
#pragma unroll
            for (int e = 0; e < h; ++e) {
                const T send = up ? v[e] : v[e + h], keep = up ? v[e + h] : v[e];
                v[e] = keep + __shfl_xor_sync(0xffffffffu, send, o);
            }
        }
    }
    // Element e of the slice in the record, and whether it belongs to order B.
    static __device__ __forceinline__ int at(int sub, int e) { return sub * W + e; }
    static __device__ __forceinline__ bool in_b(int sub, int e) { return at(sub, e) >= S::SA; }
    __device__ __forceinline__ void load(const T *__restrict__ rec, int sub) {
#pragma unroll
        for (int e = 0; e < W; ++e) v[e] = at(sub, e) < S::SQ ? rec[at(sub, e)] : T(0);
    }
    __device__ __forceinline__ void store(T *__restrict__ rec, int sub) const {
#pragma unroll
        for (int e = 0; e < W; ++e)
            if (at(sub, e) < S::SQ) rec[at(sub, e)] = v[e];
    }
};

// w_m of element i of a record of one order: 1 for m = 0, 2 above.
__device__ __forceinline__ int lane_weight(int i) { return i < 2 ? 1 : 2; }

template <int LA, int LB, typename T, bool STEP>
__device__ __forceinline__ void local_q_lanes(const LocalDev<T> &d) {
    using S = LSet<LA, LB, T>;
    const int k = blockIdx.x * (kBlock / kLanes) + threadIdx.x / kLanes, sub = threadIdx.x % kLanes;
    LSlice<LA, LB, T> acc;
    T nf = T(0);
    int c = 0;
    if (k < d.n) {
        const auto a = d.geo.load(k);
        c = min(d.nb.count[k], d.nb.M);
        for (int t = sub; t < c; t += kLanes) {
            T ux, uy, uz, rinv, sg, dsg;
            pair_geom<T, STEP>(d, a, nb_index(d.nb, d.npad, t, k), ux, uy, uz, rinv, sg, dsg);
            nf += sg;
            ylm_accum<LA, T>(ux, uy, uz, sg, acc.v);
            if constexpr (LB > 0) ylm_accum<LB, T>(ux, uy, uz, sg, acc.v + S::SA);
        }
    }
    nf = lanes_total<kLanes>(nf);
    acc.spread(sub);
    if (k >= d.n) return;
    const bool active = c > 0 && nf >= T(1e-12);
    const T inv = active ? T(1) / nf : T(0);
#pragma unroll
    for (int e = 0; e < acc.W; ++e) acc.v[e] *= inv;
    acc.store(d.q + (size_t)k * S::SQ, sub);
    if (sub == 0) d.nf[k] = active ? nf : T(0);
}

template <int LA, int LB, typename T, bool STEP>
__device__ __forceinline__ void local_lq_lanes(const LocalDev<T> &d) {
    using S = LSet<LA, LB, T>;
    using R = LSlice<LA, LB, T>;
    __shared__ double smem[8 * 32];
    const int k = blockIdx.x * (kBlock / kLanes) + threadIdx.x / kLanes, sub = threadIdx.x % kLanes;
    const bool valid = k < d.n, ing = valid && (d.smask[k] & d.groupbit) != 0;
    const T nfk = valid ? d.nf[k] : T(0);
    const bool on = ing && nfk > T(0);
    R A, qk;
    if (on) {
        const auto a = d.geo.load(k);
        const int c = min(d.nb.count[k], d.nb.M);
        qk.load(d.q + (size_t)k * S::SQ, sub);
        for (int t = sub; t < c; t += kLanes) {
            const int j = nb_index(d.nb, d.npad, t, k);
            const T sg = pair_sigma<T, STEP>(d, a, j);
            T qj[S::SQ];
            load_rec32(d.q + (size_t)j * S::SQ, qj);
#pragma unroll
            for (int s = 0; s < S::SQ; ++s) A.v[s] += sg * qj[s];
        }
    }
    A.spread(sub);
    const T inv = on ? T(1) / (nfk + T(1)) : T(0);
    T nA = T(0), nB = T(0);
#pragma unroll
    for (int e = 0; e < R::W; ++e) {
        const T v = (qk.v[e] + A.v[e]) * inv;
        A.v[e] = v;
        const bool b = R::in_b(sub, e);
        const int i = R::at(sub, e) - (b ? S::SA : 0);
        (b ? nB : nA) += T(lane_weight(i)) * v * v;
    }
    nA = lanes_total<kLanes>(nA);
    if (LB > 0) nB = lanes_total<kLanes>(nB);
    double part[5] = {0, 0, 0, 0, 0};
    if (valid) {
        const T lqA = on ? t_sqrt<T>(nA * T(4.0 * kPi / (2 * LA + 1))) : T(0);
        const T lqB = on && LB > 0 ? t_sqrt<T>(nB * T(4.0 * kPi / (2 * LB + 1))) : T(0);
        T e[4] = {T(0), T(0), T(0), T(0)};
        if (ing) {
            const double fA = sw_f<double>(d.sw_cvA, (double)lqA);
            part[0] = (double)lqA * fA;
            part[1] = fA;
            part[4] = 1.0;
            if (nfk > T(0)) {
                const double dfA = sw_df<double>(d.sw_cvA, (double)lqA);
                const double den = fmax((double)lqA, 1e-12) * ((double)nfk + 1.0);
                const double C = 4.0 * kPi / (2 * LA + 1);
                e[0] = (T)((dfA * lqA + fA) * C / den);
                e[1] = (T)(dfA * C / den);
            }
            if constexpr (LB > 0) {
                const double fB = sw_f<double>(d.sw_cvB, (double)lqB);
                part[2] = (double)lqB * fB;
                part[3] = fB;
                if (nfk > T(0)) {
                    const double dfB = sw_df<double>(d.sw_cvB, (double)lqB);
                    const double den = fmax((double)lqB, 1e-12) * ((double)nfk + 1.0);
                    const double C = 4.0 * kPi / (2 * LB + 1);
                    e[2] = (T)((dfB * lqB + fB) * C / den);
                    e[3] = (T)(dfB * C / den);
                }
            }
        }
        // e1 of each order in the record's m = 0 imaginary slots (local_lq_body)
#pragma unroll
        for (int w = 0; w < R::W; ++w) {
            if (R::at(sub, w) == 1) A.v[w] = e[0];
            if (LB > 0 && R::at(sub, w) == S::SA + 1) A.v[w] = e[2];
        }
        A.store(d.lq + (size_t)k * S::SQ, sub);
        if (sub == 0) {
            d.lqs[2 * k] = lqA;
            d.lqs[2 * k + 1] = lqB;
#pragma unroll
            for (int t = 0; t < 4; ++t) d.e12[4 * k + t] = e[t];
        } else {
#pragma unroll
            for (int t = 0; t < 5; ++t) part[t] = 0.0;
        }
    }
    double p8[8] = {part[0], part[1], part[2], part[3], part[4], 0.0, 0.0, 0.0};
    const double tot = block_sum_spread<8>(p8, smem);
    if (threadIdx.x < 20 && (threadIdx.x & 3) == 0) d.partials[blockIdx.x * 8 + (threadIdx.x >> 2)] = tot;
}

// The adjoint (local_lambda_body).  FLAT: a step pair switch and flat CV
// switches, whose gather needs no coefficient and runs before the wait for the
// bias kernel.
template <int LA, int LB, typename T, bool STEP, bool FLAT>
__device__ __forceinline__ void local_lambda_lanes(const LocalDev<T> &d) {
    using S = LSet<LA, LB, T>;
    using R = LSlice<LA, LB, T>;
    constexpr bool DSIG = !STEP;
    if (FLAT) pdl_release();
    else pdl_entry();
    const int k = blockIdx.x * (kBlock / kLanes) + threadIdx.x / kLanes, sub = threadIdx.x % kLanes;
    const bool valid = k < d.n;
    const T nfk = valid ? d.nf[k] : T(0);
    const bool on = nfk > T(0);
    T c1A = T(1), c2A = T(0), c1B = T(1), c2B = T(0);
    if (!FLAT) {
        c1A = (T)d.coef[0];
        c2A = (T)d.coef[1];
        c1B = (T)d.coef[2];
        c2B = (T)d.coef[3];
    }
    R lam;
    if (on) {
        const auto a = d.geo.load(k);
        const int c = min(d.nb.count[k], d.nb.M);
        for (int t = sub; t < c; t += kLanes) {
            const int j = nb_index(d.nb, d.npad, t, k);
            T lqj[S::SQ];
            load_rec32(d.lq + (size_t)j * S::SQ, lqj);
            T wjA, wjB;
            if (FLAT) {
                wjA = lqj[1];
                wjB = LB > 0 ? lqj[S::SA + 1] : T(0);
            } else {
                T ej[4];
                load_rec(d.e12 + 4 * (size_t)j, ej);
                wjA = c1A * ej[0] + c2A * ej[1];
                wjB = c1B * ej[2] + c2B * ej[3];
            }
            if (wjA == T(0) && wjB == T(0)) continue;
            const T sg = pair_sigma<T, STEP>(d, a, j);
            add_g<LA, T>(lam.v, lqj, wjA, sg);
            if constexpr (LB > 0) add_g<LB, T>(lam.v + S::SA, lqj + S::SA, wjB, sg);
        }
    }
    lam.spread(sub);
    // this atom's own G, in slices; the m = 0 imaginary slot holds e1, not LQ
    R lqk, G;
    if (on) {
        lqk.load(d.lq + (size_t)k * S::SQ, sub);
        const T wA = c1A * d.e12[4 * k] + c2A * d.e12[4 * k + 1];
        const T wB = c1B * d.e12[4 * k + 2] + c2B * d.e12[4 * k + 3];
#pragma unroll
        for (int e = 0; e < R::W; ++e) {
            const bool b = R::in_b(sub, e);
            const int i = R::at(sub, e) - (b ? S::SA : 0);
            if (i == 1) lqk.v[e] = T(0);
            G.v[e] = T(lane_weight(i)) * (b ? wB : wA) * lqk.v[e];
            lam.v[e] += G.v[e];
        }
    }
    T sA = T(0), sB = T(0);
    if (FLAT) {
        pdl_wait();
        if (on) {
            const T inv = T(1) / nfk;
            sA = (T)d.coef[0] * inv;
            sB = (T)d.coef[2] * inv;
        }
    } else {
        sA = sB = on ? T(1) / nfk : T(0);
    }
    if constexpr (DSIG) {
        R qk;
        if (on) qk.load(d.q + (size_t)k * S::SQ, sub);
        T tA = T(0), tB = T(0), uA = T(0), uB = T(0);
#pragma unroll
        for (int e = 0; e < R::W; ++e) {
            const bool b = R::in_b(sub, e);
            (b ? tB : tA) += lam.v[e] * qk.v[e];
            (b ? uB : uA) += G.v[e] * lqk.v[e];
        }
        tA = lanes_total<kLanes>(tA);
        tB = lanes_total<kLanes>(tB);
        uA = lanes_total<kLanes>(uA);
        uB = lanes_total<kLanes>(uB);
        if (valid) {
            if (sub == 0) {
                d.tu[4 * k] = tA * sA;
                d.tu[4 * k + 1] = uA;
                d.tu[4 * k + 2] = tB * sA;
                d.tu[4 * k + 3] = uB;
            }
            G.store(d.g + (size_t)k * S::SQ, sub);
        }
    }
    if (!valid) return;
#pragma unroll
    for (int e = 0; e < R::W; ++e) lam.v[e] *= R::in_b(sub, e) ? sB : sA;
    lam.store(d.lam + (size_t)k * S::SQ, sub);
}

// Forces of 32 atoms per block (local_force_body); in caller order the block's
// stretch of f goes through shared memory as there.
template <int LA, int LB, typename T, bool STEP, bool CALLER>
__device__ __forceinline__ void local_force_lanes(const LocalDev<T> &d, const double *__restrict__ f_src,
                                                  double *__restrict__ f_dst, const SysDev &s, const CellGrid &g,
                                                  double *vpart, DevStatus *status) {
    constexpr int AB = kBlock / kLanes;
    __shared__ double smem[6 * 32];
    __shared__ double fstage[CALLER ? 3 * AB : 1];
    const int local = threadIdx.x / kLanes, sub = threadIdx.x % kLanes;
    int k = blockIdx.x * AB + local, ib0 = 0, cnt = 0;
    bool valid = k < d.n;
    if constexpr (CALLER) {
        ib0 = d.i0 + blockIdx.x * AB;
        cnt = max(0, min(AB, d.i1 - ib0));
        for (int e = threadIdx.x; e < 3 * cnt; e += blockDim.x) fstage[e] = f_src[3 * (size_t)ib0 + e];
        __syncthreads();
        valid = local < cnt;
        k = valid ? d.iperm[ib0 + local] : 0;
        valid = valid && (unsigned)k < (unsigned)d.n;
    }
    T gx = T(0), gy = T(0), gz = T(0);
    if (valid) local_force_sum<LA, LB, T, STEP>(d, k, sub, kLanes, gx, gy, gz);
    gx = lanes_total<kLanes>(gx);
    gy = lanes_total<kLanes>(gy);
    gz = lanes_total<kLanes>(gz);
    double vir[6] = {0, 0, 0, 0, 0, 0};
    if (valid && sub == 0) {
        const int i = CALLER ? ib0 + local : d.perm[k];
        const double fx = -(double)gx, fy = -(double)gy, fz = -(double)gz;   // delta f = -dV/dx
        if constexpr (CALLER) {
            fstage[3 * local] += fx;
            fstage[3 * local + 1] += fy;
            fstage[3 * local + 2] += fz;
        } else if ((unsigned)i < (unsigned)d.n) {   // a sorted order left by a rebuild that gave up is not trusted
            f_dst[3 * i] = f_src[3 * i] + fx;
            f_dst[3 * i + 1] = f_src[3 * i + 1] + fy;
            f_dst[3 * i + 2] = f_src[3 * i + 2] + fz;
        }
        if (!(isfinite(fx) && isfinite(fy) && isfinite(fz))) atomicOr(&status->nan_force, 1u);
        if (vpart && (unsigned)i < (unsigned)d.n) force_virial(s, g, k, i, fx, fy, fz, vir);
    }
    if constexpr (CALLER) {
        __syncthreads();
        for (int e = threadIdx.x; e < 3 * cnt; e += blockDim.x) f_dst[3 * (size_t)ib0 + e] = fstage[e];
    }
    if (vpart) {
        block_sum<6>(vir, smem);
        if (threadIdx.x == 0)
            for (int t = 0; t < 6; ++t) vpart[blockIdx.x * 8 + t] = vir[t];
    }
}

}  // namespace mtd
