// sf.cu -- structure-factor CVs.
//
// STRU_FACTOR (Debye form) replaces structure_factor_cv_kernel and the AVE /
// COUNT gradient kernels (src/cvs/CVs_Strufactor.cu:1082-1271):
//   S_i = 1 + sum_{j: 1e-12 <= r2 <= rc2} sin(q r)/(q r) s(r),
//   s = 1 - ((r2 - 0.8 rc2)/(0.2 rc2))^3 above 0.8 rc2,
//   dCV/dx_a = - sum_j (a_a + a_j) g'(r_aj) dhat_aj,  a_i = dCV/dS_i.
// STRU_FACTOR_K (no reference counterpart): rho_k = sum_j exp(i k.x_j) over the
// group, S(k) = |rho_k|^2/N, CV = mean_k S(k),
//   dCV/dx_j = 2/(N K) sum_k k (-Re rho_k sin(k.x_j) + Im rho_k cos(k.x_j)).
// Phases are formed in FP64 in half turns and reduced before the FP32 (or FP64)
// polynomials; the sums over atoms are FP64 block partials reduced in a fixed
// order.
#include "kernels.h"

#include <algorithm>
#include <type_traits>

namespace mtd {

namespace {

template <typename T> __device__ __forceinline__ void t_sincos(T x, T *s, T *c);
template <> __device__ __forceinline__ void t_sincos<float>(float x, float *s, float *c) { sincosf(x, s, c); }
template <> __device__ __forceinline__ void t_sincos<double>(double x, double *s, double *c) { sincos(x, s, c); }

template <typename T> __device__ __forceinline__ void debye_g(T r2, T rc2, T qf, T &gv, T &dg) {
    const T r = t_sqrt<T>(r2), th = qf * r;
    T s = T(1), ds = T(0);
    const T r_on = T(0.8) * rc2;
    if (r2 > r_on) {
        const T t = (r2 - r_on) / (rc2 - r_on);
        s = T(1) - t * t * t;
        ds = T(-3) * t * t * (T(2) * r) / (rc2 - r_on);
    }
    if (qf == T(0)) {   // WEIGHT_CHEM: the taper alone is the pair term
        gv = s;
        dg = ds;
        return;
    }
    T sn, cs;
    t_sincos<T>(th, &sn, &cs);
    gv = sn / th * s;
    dg = (cs / th - sn / (th * th)) * s * qf + ds * sn / th;
}

// STRU_FACTOR Chemical: the type weight of every sorted atom (types outside
// the table weigh 0, as type 0 does).
template <typename T> __global__ void k_chem_weights(DebyeDev<T> d) {
    pdl_entry();
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= d.n) return;
    const int i = d.perm[k];
    const int t = (unsigned)i < (unsigned)d.n ? d.types[i] : 0;
    d.w[k] = (T)(t >= 0 && t < d.ntab ? d.wtab[t] : 0.0);
}

template <typename T, int G> __global__ void __launch_bounds__(kBlock) k_debye_values(DebyeDev<T> d) {
    pdl_entry();
    __shared__ double smem[4 * 32];
    const int k = blockIdx.x * (kBlock / G) + threadIdx.x / G, sub = threadIdx.x % G;
    double part[4] = {0, 0, 0, 0};
    const bool on = k < d.n && (d.smask[k] & d.groupbit);
    T S = T(0);
    if (on) {
        const int c = min(d.nb.count[k], d.nb.M);
        const T rc2 = (T)d.rc2, qf = (T)d.qf;
        const auto a = d.geo.load(k);
        const T wk = d.w ? d.w[k] : T(1);
        for (int t = sub; t < c; t += G) {
            const int j = d.nb.list[(size_t)t * d.npad + k];
            T dx, dy, dz;
            d.geo.disp(a, d.geo.load(j), dx, dy, dz);
            T gv, dg;
            debye_g<T>(dx * dx + dy * dy + dz * dz, rc2, qf, gv, dg);
            S += d.w ? wk * d.w[j] * gv : gv;
        }
    }
    if (G > 1) S = lanes_total<G>(S);
    if (on) S += T(1);
    if (on && sub == 0) {
        part[0] = (double)S;
        part[1] = sw_f<double>(d.sw, (double)S);
        part[2] = 1.0;
    }
    if (k < d.n && sub == 0) d.S[k] = S;
    block_sum<4>(part, smem);
    if (threadIdx.x == 0)
        for (int t = 0; t < 4; ++t) d.partials[blockIdx.x * 8 + t] = part[t];
}

template <typename T>
__device__ __forceinline__ T debye_a(const DebyeDev<T> &d, int k, double c0, double c1) {
    if (!(d.smask[k] & d.groupbit)) return T(0);
    double a = c0;
    if (c1 != 0.0) a += c1 * sw_df<double>(d.sw, (double)d.S[k]);
    return (T)a;
}

template <typename T, int G>
__global__ void __launch_bounds__(kBlock) k_debye_force(DebyeDev<T> d, const double *__restrict__ f_src,
                                                        double *__restrict__ f_dst, SysDev s, CellGrid g,
                                                        double *vpart, DevStatus *status) {
    pdl_entry();
    __shared__ double smem[6 * 32];
    const int k = blockIdx.x * (kBlock / G) + threadIdx.x / G, sub = threadIdx.x % G;
    double vir[6] = {0, 0, 0, 0, 0, 0};
    const double c0 = d.coef[0], c1 = d.coef[1];
    T gx = T(0), gy = T(0), gz = T(0);
    if (k < d.n) {
        const T ak = debye_a<T>(d, k, c0, c1);
        const T rc2 = (T)d.rc2, qf = (T)d.qf;
        const int c = min(d.nb.count[k], d.nb.M);
        const auto a = d.geo.load(k);
        const T wk = d.w ? d.w[k] : T(1);
        for (int t = sub; t < c; t += G) {
            const int j = d.nb.list[(size_t)t * d.npad + k];
            T w = ak + debye_a<T>(d, j, c0, c1);
            if (d.w) w *= wk * d.w[j];
            if (w == T(0)) continue;
            T dx, dy, dz;
            d.geo.disp(a, d.geo.load(j), dx, dy, dz);
            const T r2 = dx * dx + dy * dy + dz * dz;
            T gv, dg;
            debye_g<T>(r2, rc2, qf, gv, dg);
            const T f = w * dg * t_rsqrt<T>(r2);
            gx -= f * dx;
            gy -= f * dy;
            gz -= f * dz;
        }
    }
    if (G > 1) {
        gx = lanes_total<G>(gx);
        gy = lanes_total<G>(gy);
        gz = lanes_total<G>(gz);
    }
    if (k < d.n && sub == 0) {
        const int i = d.perm[k];
        const double fx = -(double)gx, fy = -(double)gy, fz = -(double)gz;
        if ((unsigned)i < (unsigned)d.n) {   // a sorted order left by a rebuild that gave up is not trusted
            f_dst[3 * i] = f_src[3 * i] + fx;
            f_dst[3 * i + 1] = f_src[3 * i + 1] + fy;
            f_dst[3 * i + 2] = f_src[3 * i + 2] + fz;
        }
        if (!(isfinite(fx) && isfinite(fy) && isfinite(fz))) atomicOr(&status->nan_force, 1u);
        if (vpart && (unsigned)i < (unsigned)d.n) {
            double ux = s.xs[3 * k], uy = s.xs[3 * k + 1], uz = s.xs[3 * k + 2];
            if (s.image) {
                int ix, iy, iz;
                unpack_image(s.image[i], ix, iy, iz);
                ux += ix * g.L[0];
                uy += iy * g.L[1];
                uz += iz * g.L[2];
            }
            vir[0] = fx * ux; vir[1] = fy * uy; vir[2] = fz * uz;
            vir[3] = fx * uy; vir[4] = fx * uz; vir[5] = fy * uz;
        }
    }
    if (vpart) {
        block_sum<6>(vir, smem);
        if (threadIdx.x == 0)
            for (int t = 0; t < 6; ++t) vpart[blockIdx.x * 8 + t] = vir[t];
    }
}

// ------------------------------------------------------------------ S(k)
// The value pass sums exp(i k.x) with the k-vectors over the threads: a thread
// keeps a pair of them and its sums in registers and goes through atoms staged
// in shared memory, so nothing is summed across lanes until its block is done.
// (With the atoms over the threads, and every k's sums reduced over the block
// in FP64, those reductions were 10 of 26 instructions per atom-k pair.)
// In mixed precision the phase (k / pi).x is formed in FP64 (B200 runs FP64 at
// half the FP32 rate) with its fraction left in the low word (kTurnBase), and
// finished with FP32 polynomials on the pair of k-vectors (turn_sincos2); FP64
// mode keeps the phase in radians (phase_sincos_f64).  A
// per-dimension FP32 phase-table variant (three shared-memory loads and an
// FP32 reduction per pair) measured 2.2x slower and was removed.
// The shapes the autotuner picks (SkDev::qv: 2, 4 or 8 atoms in flight per
// thread in the value pass; SkDev::qf: the unroll depth of the force pass's
// loop over k) leave every sum's order as it is.
constexpr int kSkBlocks = 148 * 4;   // resident blocks of both passes
constexpr int kSkChunk = 512;        // atoms staged at a time in the value pass
constexpr int kSkFlush = 8;          // most atoms summed in FP32 before they join the FP64 sums

// sin(pi f), cos(pi f) (unsigned) and the sign masks of one atom's phases with
// a pair of k-vectors (/ pi); far: beyond the base's range or not finite, the
// phase is then rounded in FP64.
__device__ __forceinline__ void sk_pair(bool far, double2 kx, double2 ky, double2 kz, double x, double y, double z,
                                        float2 &s0, float2 &c0, unsigned &ga, unsigned &gb) {
    if (!far) {
        const double ta = fma(kz.x, z, fma(ky.x, y, fma(kx.x, x, kTurnBase)));
        const double tb = fma(kz.y, z, fma(ky.y, y, fma(kx.y, x, kTurnBase)));
        turn_sincos2(ta, tb, s0, c0);
        ga = turn_sign(ta);
        gb = turn_sign(tb);
    } else {
        ga = halfturn_sincos_f32_parts(kx.x * x + ky.x * y + kz.x * z, s0.x, c0.x);
        gb = halfturn_sincos_f32_parts(kx.y * x + ky.y * y + kz.y * z, s0.y, c0.y);
    }
}

// Phases beyond kPhaseMax, out of the passes' way: sin and cos, and sin(ph - shift).
// There the last bit of a phase is a quarter radian and more, so the rounding of
// ph / pi adds nothing (sincos() has a stack frame, 1.3 us on a 20 us kernel).
__device__ __noinline__ double2 far_sincos(double ph) {
    double2 v;
    sincospi(ph * kInvPi, &v.x, &v.y);
    return v;
}
__device__ __noinline__ double far_sin(double ph, double shift) {
    const double2 a = far_sincos(ph), b = far_sincos(shift);
    return a.x * b.y - a.y * b.x;
}

// Threads are streams of np (a tile's pairs of k) each: stream s of S takes
// staged atoms s, s + S, ....  Block b sums atoms b * per .. (b + 1) * per - 1.
// Bound by the SM's dispatch: 21 instructions per atom-k pair, of which the 3
// FP64 and 7 paired FP32 ones take two cycles each (38 cycles a pair are
// measured, the FMA pipe is 46 % busy).  1,048,576 atoms x 96 k: 147 us before
// (26 instructions with 6 FP64 and the slow conversion, atoms over the
// threads), 114 now; FP64 at 108,000 x 24: 22 us (sincos()), 19 now, 157,216 x 90:
// 80 and 44.
template <bool FP64, int U, int F>
__global__ void __launch_bounds__(256, FP64 ? 2 : 4) k_sk_partial(SkDev d, int per) {
    pdl_entry();
    __shared__ double2 xy[kSkChunk];
    __shared__ double zz[kSkChunk];
    __shared__ int wcount[2][8];
    const int np = (d.K + 1) / 2, ntile = (np + 63) / 64, TP = (np + ntile - 1) / ntile, S = (int)blockDim.x / TP;
    const int st = threadIdx.x / TP, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int a0 = min(blockIdx.x * per, d.nown), a1 = min(a0 + per, d.nown);
    const double reach = d.reach;
    int total = 0;
    for (int tile = 0; tile < ntile; ++tile) {
        const int p = tile * TP + (int)threadIdx.x % TP;
        const bool active = st < S && p < np;
        constexpr double unit = FP64 ? 1.0 : kInvPi;
        double2 kv[3];
#pragma unroll
        for (int c = 0; c < 3; ++c)   // an odd K is filled up with a zero vector, whose sums are not written
            kv[c] = make_double2(active ? d.k[6 * p + c] * unit : 0.0,
                                 active && 2 * p + 1 < d.K ? d.k[6 * p + 3 + c] * unit : 0.0);
        double c64[2] = {0.0, 0.0}, s64[2] = {0.0, 0.0};
        for (int c0 = a0; c0 < a1; c0 += kSkChunk) {
            // the group's atoms of the chunk, in order
            double px[2], py[2], pz[2];
            bool keep[2], is_far = false;
            unsigned ball[2];
            __syncthreads();
#pragma unroll
            for (int r = 0; r < 2; ++r) {
                const int i = c0 + (int)threadIdx.x + 256 * r;
                keep[r] = i < a1 && (!d.mask || (d.mask[i] & d.groupbit));
                ball[r] = __ballot_sync(0xffffffffu, keep[r]);
                if (lane == 0) wcount[r][warp] = __popc(ball[r]);
                if (keep[r]) {
                    px[r] = d.x[3 * i];
                    py[r] = d.x[3 * i + 1];
                    pz[r] = d.x[3 * i + 2];
                    is_far = is_far || !(fabs(px[r]) + fabs(py[r]) + fabs(pz[r]) < reach);
                }
            }
            __syncthreads();
            int m = 0;
#pragma unroll
            for (int r = 0; r < 2; ++r) {
                int at = m + __popc(ball[r] & ((1u << lane) - 1));
                for (int w = 0; w < 8; ++w) {
                    if (w < warp) at += wcount[r][w];
                    m += wcount[r][w];
                }
                if (keep[r]) {
                    xy[at] = make_double2(px[r], py[r]);
                    zz[at] = pz[r];
                }
            }
            const bool any_far = __syncthreads_or(is_far);
            total += m;
            if (!active) continue;
            int j = st;
            if constexpr (FP64) {
                auto sum = [&](double ph, bool far, int e) {
                    double s, c;
                    if (far) {
                        const double2 v = far_sincos(ph);
                        s = v.x;
                        c = v.y;
                    } else {
                        phase_sincos_f64(ph, s, c);
                    }
                    c64[e] += c;
                    s64[e] += s;
                };
                auto add = [&](bool far) {
                    const double2 q = xy[j];
                    const double z = zz[j];
                    sum(fma(kv[2].x, z, fma(kv[1].x, q.y, kv[0].x * q.x)), far, 0);
                    sum(fma(kv[2].y, z, fma(kv[1].y, q.y, kv[0].y * q.x)), far, 1);
                };
                if (!any_far) {
#pragma unroll U
                    for (; j < m; j += S) add(false);
                } else {
#pragma unroll 1
                    for (; j < m; j += S) add(!(fabs(xy[j].x) + fabs(xy[j].y) + fabs(zz[j]) < reach));
                }
            } else {
                constexpr int kOuter = U > F ? U / F : 1, kInner = U < F ? U : F;
                float2 fc, fs;
                auto add = [&](int e, bool far) {
                    const double2 q = xy[e];
                    float2 s0, c0f;
                    unsigned ga, gb;
                    sk_pair(far, kv[0], kv[1], kv[2], q.x, q.y, zz[e], s0, c0f, ga, gb);
                    // the sign (-1)^n as a factor of exact FMAs: the same sums
                    // as adding the signed sin and cos
                    const float2 sg = make_float2(__uint_as_float(0x3f800000u | ga), __uint_as_float(0x3f800000u | gb));
                    fc = __ffma2_rn(sg, c0f, fc);
                    fs = __ffma2_rn(sg, s0, fs);
                };
                auto flush = [&] {
                    c64[0] += (double)fc.x;
                    c64[1] += (double)fc.y;
                    s64[0] += (double)fs.x;
                    s64[1] += (double)fs.y;
                };
                for (; j < m; j += kSkFlush * S) {
                    if (!any_far && j + (kSkFlush - 1) * S < m) {
#pragma unroll kOuter
                        for (int e = 0; e < kSkFlush; e += F) {
                            fc = fs = make_float2(0.f, 0.f);
#pragma unroll kInner
                            for (int t = 0; t < F; ++t) add(j + (e + t) * S, false);
                            flush();
                        }
                    } else {
#pragma unroll 1
                        for (int e = j; e < min(m, j + kSkFlush * S);) {
                            fc = fs = make_float2(0.f, 0.f);
#pragma unroll 1
                            for (int t = 0; t < F && e < m; ++t, e += S) {
                                const double2 q = xy[e];
                                add(e, !(fabs(q.x) + fabs(q.y) + fabs(zz[e]) < reach));
                            }
                            flush();
                        }
                    }
                }
            }
        }
        // the streams' sums in stream order; partials are one row of blocks per value
        __syncthreads();
        static_assert(sizeof(xy) >= 4 * 256 * sizeof(double), "the sums fit over the staged atoms");
        double *red = &xy[0].x;
        red[threadIdx.x] = c64[0];
        red[256 + threadIdx.x] = s64[0];
        red[512 + threadIdx.x] = c64[1];
        red[768 + threadIdx.x] = s64[1];
        __syncthreads();
        for (int e = threadIdx.x; e < 4 * TP; e += blockDim.x) {
            const int v = 4 * (tile * TP + e % TP) + e / TP;
            if (v >= 2 * d.K) continue;
            double sum = 0.0;
            for (int q = 0; q < S; ++q) sum += red[e / TP * 256 + q * TP + e % TP];
            d.partials[(size_t)v * d.nblocks + blockIdx.x] = sum;
        }
    }
    if (threadIdx.x == 0) d.partials[(size_t)(2 * d.K) * d.nblocks + blockIdx.x] = (double)(total / ntile);
}

// One warp per output value (2K rho components + the group count).
__global__ void __launch_bounds__(256) k_sk_reduce(SkDev d) {
    pdl_entry();
    const int v = blockIdx.x * 8 + (threadIdx.x >> 5), lane = threadIdx.x & 31;
    if (v > 2 * d.K) return;
    double acc = 0.0;
    for (int b = lane; b < d.nblocks; b += 32) acc += d.partials[(size_t)v * d.nblocks + b];
    for (int o = 16; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
    if (lane == 0) {
        if (v < 2 * d.K) d.rho[v] = acc;
        else *d.ngroup = acc;
    }
}

// f_dst = f_src + (gx, gy, gz) of atom i and its virial term.
__device__ __forceinline__ void sk_apply(const SkDev &d, const SysDev &s, const CellGrid &g, int i, double gx,
                                         double gy, double gz, const double *__restrict__ f_src,
                                         double *__restrict__ f_dst, bool virial, double (&vir)[6]) {
    f_dst[3 * i] = f_src[3 * i] + gx;
    f_dst[3 * i + 1] = f_src[3 * i + 1] + gy;
    f_dst[3 * i + 2] = f_src[3 * i + 2] + gz;
    if (virial) {
        double ux = d.x[3 * i], uy = d.x[3 * i + 1], uz = d.x[3 * i + 2];
        if (s.image) {
            int ix, iy, iz;
            unpack_image(s.image[i], ix, iy, iz);
            ux += ix * g.L[0];
            uy += iy * g.L[1];
            uz += iz * g.L[2];
        }
        vir[0] = gx * ux; vir[1] = gy * uy; vir[2] = gz * uz;
        vir[3] = gx * uy; vir[4] = gx * uz; vir[5] = gy * uz;
    }
}

// Force pass, AT atoms per thread and tile (atoms tile * 256 * AT + a * 256 +
// threadIdx.x), tiles over a grid of resident blocks.  One sine per pair:
// Im rho cos(k.x) - Re rho sin(k.x) = -|rho| sin(k.x - arg rho), with the
// phase of rho(k) set off the phase sum's start (FP64: taken off its remainder) and
// |rho| multiplied into k (FP64: the sine), both formed once per block; phases in
// half turns in mixed precision.  k-vectors go in pairs, with
// the sums over the even and the odd k kept apart and added at the end, so the
// forces do not depend on U, AT or the grid.
// Bound by dispatch as the value pass (16 instructions a pair, 27 cycles).
// 1,048,576 atoms x 96 k: 119 us before (sine and cosine, 3 more FP64
// additions), 82 now; FP64 at 108,000 x 24: 16 us, 15 now, 157,216 x 90: 60 and 39.
template <bool FP64, int U, int AT>
__global__ void __launch_bounds__(256, FP64 ? 2 : 4)
    k_sk_force(SkDev d, const double *__restrict__ f_src, double *__restrict__ f_dst, SysDev s, CellGrid g,
               double *vpart) {
    pdl_entry();
    __shared__ double smem[6 * 32];
    extern __shared__ double2 skf_raw[];   // per pair of k: 4 double2; 1 double2 (FP64) or 3 float2
    const int np = (d.K + 1) / 2;
    double2 *kp = skf_raw, *wd = kp + 4 * np;
    float2 *wf = reinterpret_cast<float2 *>(wd);
    const double a = d.coef[0];
    for (int q = threadIdx.x; q < 2 * np; q += blockDim.x) {
        const bool real = q < d.K;   // an odd K is filled up with a zero vector
        const double re = real ? d.rho[2 * q] : 0.0, im = real ? d.rho[2 * q + 1] : 0.0;
        const double amp = -sqrt(re * re + im * im), ph = atan2(im, re);
        double *kd = reinterpret_cast<double *>(kp) + q / 2 * 8 + q % 2;
        for (int c = 0; c < 3; ++c) {
            const double kc = real ? d.k[3 * q + c] : 0.0;
            kd[2 * c] = FP64 ? kc : kc * kInvPi;
            if (!FP64) reinterpret_cast<float *>(wf)[q / 2 * 6 + 2 * c + q % 2] = (float)(amp * kc);
        }
        if (FP64) reinterpret_cast<double *>(wd)[q] = amp;
        kd[6] = FP64 ? ph : kTurnBase - ph * kInvPi;
    }
    const double reach = d.reach;
    __syncthreads();
    for (int tile = blockIdx.x; tile * 256 * AT < d.n; tile += gridDim.x) {
        using R2 = typename std::conditional<FP64, double2, float2>::type;
        double x[AT], y[AT], z[AT];
        R2 fx[AT], fy[AT], fz[AT];
        bool on[AT], far[AT], any = false, any_far = false;
#pragma unroll
        for (int t = 0; t < AT; ++t) {
            const int i = (tile * AT + t) * 256 + threadIdx.x;
            on[t] = i < d.nown && (!d.mask || (d.mask[i] & d.groupbit));
            x[t] = on[t] ? d.x[3 * i] : 0.0;
            y[t] = on[t] ? d.x[3 * i + 1] : 0.0;
            z[t] = on[t] ? d.x[3 * i + 2] : 0.0;
            fx[t].x = fy[t].x = fz[t].x = fx[t].y = fy[t].y = fz[t].y = 0;
            far[t] = !(fabs(x[t]) + fabs(y[t]) + fabs(z[t]) < reach);
            any = any || on[t];
            any_far = any_far || far[t];
        }
        auto add_pair = [&](int q, int t, bool is_far) {
            const double2 kx = kp[4 * q], ky = kp[4 * q + 1], kz = kp[4 * q + 2], base = kp[4 * q + 3];
            double ua = fma(kz.x, z[t], fma(ky.x, y[t], FP64 ? kx.x * x[t] : fma(kx.x, x[t], base.x)));
            double ub = fma(kz.y, z[t], fma(ky.y, y[t], FP64 ? kx.y * x[t] : fma(kx.y, x[t], base.y)));
            if constexpr (FP64) {
                const double sa = (is_far ? far_sin(ua, base.x) : phase_sin_f64(ua, base.x)) * wd[q].x;
                const double sb = (is_far ? far_sin(ub, base.y) : phase_sin_f64(ub, base.y)) * wd[q].y;
                fx[t] = make_double2(fma(sa, kx.x, fx[t].x), fma(sb, kx.y, fx[t].y));
                fy[t] = make_double2(fma(sa, ky.x, fy[t].x), fma(sb, ky.y, fy[t].y));
                fz[t] = make_double2(fma(sa, kz.x, fz[t].x), fma(sb, kz.y, fz[t].y));
            } else {
                float2 s0, c0;
                unsigned ga, gb;
                if (!is_far) {
                    turn_sin2(ua, ub, s0);
                    ga = turn_sign(ua);
                    gb = turn_sign(ub);
                } else {
                    // the phase without the base, its sum rounded as the phase is
                    ua = fma(kz.x, z[t], fma(ky.x, y[t], kx.x * x[t])) + (base.x - kTurnBase);
                    ub = fma(kz.y, z[t], fma(ky.y, y[t], kx.y * x[t])) + (base.y - kTurnBase);
                    ga = halfturn_sincos_f32_parts(ua, s0.x, c0.x);
                    gb = halfturn_sincos_f32_parts(ub, s0.y, c0.y);
                }
                // the sign (-1)^n on the sine: exact
                s0.x = __uint_as_float(__float_as_uint(s0.x) ^ ga);
                s0.y = __uint_as_float(__float_as_uint(s0.y) ^ gb);
                fx[t] = __ffma2_rn(s0, wf[3 * q], fx[t]);
                fy[t] = __ffma2_rn(s0, wf[3 * q + 1], fy[t]);
                fz[t] = __ffma2_rn(s0, wf[3 * q + 2], fz[t]);
            }
        };
        if (any && !any_far) {
#pragma unroll U
            for (int q = 0; q < np; ++q)
#pragma unroll
                for (int t = 0; t < AT; ++t) add_pair(q, t, false);
        } else if (any) {
            for (int q = 0; q < np; ++q)
#pragma unroll
                for (int t = 0; t < AT; ++t) add_pair(q, t, far[t]);
        }
#pragma unroll
        for (int t = 0; t < AT; ++t) {
            const int vb = tile * AT + t, i = vb * 256 + threadIdx.x;
            double vir[6] = {0, 0, 0, 0, 0, 0};
            if (i < d.n)
                sk_apply(d, s, g, i, on[t] ? -a * ((double)fx[t].x + (double)fx[t].y) : 0.0,
                         on[t] ? -a * ((double)fy[t].x + (double)fy[t].y) : 0.0,
                         on[t] ? -a * ((double)fz[t].x + (double)fz[t].y) : 0.0, f_src, f_dst, vpart != nullptr, vir);
            // one virial partial per 256 atoms, as the other units write
            if (vpart && vb * 256 < d.n) {
                block_sum<6>(vir, smem);
                if (threadIdx.x == 0)
                    for (int c = 0; c < 6; ++c) vpart[vb * 8 + c] = vir[c];
                __syncthreads();
            }
        }
    }
}

}  // namespace

template <typename T> void launch_debye_values(const DebyeDev<T> &d, cudaStream_t st) {
    if (d.n == 0) return;
    if (d.w) launch_k(k_chem_weights<T>, (d.n + kBlock - 1) / kBlock, kBlock, 0, st, d);
    const int ab = d.lanes ? kBlock / kLanes : kBlock, nb = (d.n + ab - 1) / ab;
    if (d.lanes) launch_k(k_debye_values<T, kLanes>, nb, kBlock, 0, st, d);
    else launch_k(k_debye_values<T, 1>, nb, kBlock, 0, st, d);
    prof_mark("debye_values", st);
}
template <typename T>
void launch_debye_forces(const DebyeDev<T> &d, const double *f_src, double *f_dst, const SysDev &s, const CellGrid &g,
                         double *vpart, DevStatus *status, cudaStream_t st) {
    if (d.n == 0) return;
    const int ab = d.lanes ? kBlock / kLanes : kBlock, nb = (d.n + ab - 1) / ab;
    if (d.lanes) launch_k(k_debye_force<T, kLanes>, nb, kBlock, 0, st, d, f_src, f_dst, s, g, vpart, status);
    else launch_k(k_debye_force<T, 1>, nb, kBlock, 0, st, d, f_src, f_dst, s, g, vpart, status);
    prof_mark("debye_force", st);
}
template void launch_debye_values<float>(const DebyeDev<float> &, cudaStream_t);
template void launch_debye_values<double>(const DebyeDev<double> &, cudaStream_t);
template void launch_debye_forces<float>(const DebyeDev<float> &, const double *, double *, const SysDev &,
                                         const CellGrid &, double *, DevStatus *, cudaStream_t);
template void launch_debye_forces<double>(const DebyeDev<double> &, const double *, double *, const SysDev &,
                                          const CellGrid &, double *, DevStatus *, cudaStream_t);

// Blocks of the value pass: 64 atoms each give a small system the whole GPU.
int sk_blocks(int n) {
    const int b = (n + 63) / 64;
    return b < kSkBlocks ? (b < 1 ? 1 : b) : kSkBlocks;
}

// Atoms summed in FP32 before they join the FP64 sums: as many as a thread of a
// grid-wide loop of 256 threads a block has, rounded down to a power of two, so one
// (every term goes into an FP64 sum) up to 303,104 atoms and four at 1,048,576.
// Value pass with one and with eight throughout: 42.6 us and 38.1 at 296,352 atoms x
// 90, 16.3 and 15.7 at 108,000 x 24; with four and eight 113.6 and 111.3 at
// 1,048,576 x 96.
template <int U> static void launch_sk_partial_u(const SkDev &d, cudaStream_t st) {
    const int per = (d.nown + d.nblocks - 1) / d.nblocks;
    if (d.fp64) launch_k(k_sk_partial<true, U, 1>, d.nblocks, 256, 0, st, d, per);
    else if (per < 2 * 256) launch_k(k_sk_partial<false, U, 1>, d.nblocks, 256, 0, st, d, per);
    else if (per < 4 * 256) launch_k(k_sk_partial<false, U, 2>, d.nblocks, 256, 0, st, d, per);
    else if (per < 8 * 256) launch_k(k_sk_partial<false, U, 4>, d.nblocks, 256, 0, st, d, per);
    else launch_k(k_sk_partial<false, U, kSkFlush>, d.nblocks, 256, 0, st, d, per);
}

template <int U>
static void launch_sk_force_u(const SkDev &d, const double *f_src, double *f_dst, const SysDev &s, const CellGrid &g,
                              double *vpart, size_t sm, int nb, cudaStream_t st) {
    if (d.fp64) {
        launch_k(k_sk_force<true, U, 1>, std::min(nb, kSkBlocks / 2), 256, sm, st, d, f_src, f_dst, s, g, vpart);
    } else if (nb <= kSkBlocks) {   // one atom a thread until the resident blocks are full
        launch_k(k_sk_force<false, U, 1>, nb, 256, sm, st, d, f_src, f_dst, s, g, vpart);
    } else {
        launch_k(k_sk_force<false, U, 2>, std::min((nb + 1) / 2, kSkBlocks), 256, sm, st, d, f_src, f_dst, s, g, vpart);
    }
}

void launch_sk_values(const SkDev &d, cudaStream_t st) {
    if (d.qv == 4) launch_sk_partial_u<2>(d, st);
    else if (d.qv == 16) launch_sk_partial_u<8>(d, st);
    else launch_sk_partial_u<4>(d, st);
    prof_mark("sk_partial", st);
    launch_k(k_sk_reduce, (2 * d.K + 8) / 8, 256, 0, st, d);
    prof_mark("sk_reduce", st);
}

void launch_sk_forces(const SkDev &d, const double *f_src, double *f_dst, const SysDev &s, const CellGrid &g,
                      double *vpart, cudaStream_t st) {
    if (d.n == 0) return;
    const int nb = (d.n + 255) / 256;
    // per pair of k: 4 double2, then 1 double2 or 3 float2 (40,960 and 45,056 bytes at 1,024 k)
    const size_t sm = (size_t)((d.K + 1) / 2) * (4 * sizeof(double2) + (d.fp64 ? sizeof(double2) : 3 * sizeof(float2)));
    if (d.qf == 1) launch_sk_force_u<1>(d, f_src, f_dst, s, g, vpart, sm, nb, st);
    else if (d.qf == 4) launch_sk_force_u<4>(d, f_src, f_dst, s, g, vpart, sm, nb, st);
    else launch_sk_force_u<2>(d, f_src, f_dst, s, g, vpart, sm, nb, st);
    prof_mark("sk_force", st);
}

}  // namespace mtd
