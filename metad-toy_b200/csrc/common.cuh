// common.cuh -- shared types, switching functions and small device helpers.
#pragma once

#include <cuda_runtime.h>
#include <cstdint>
#include <type_traits>

namespace mtd {

constexpr double kPi = 3.14159265358979323846;
constexpr int kBlock = 256;          // threads per block for per-atom kernels
constexpr int kMaxSymbols = 16;      // SYMBOL entries per context
constexpr int kMaxDim = 4;           // CV_dim handled by the device grid kernel
constexpr int kFlagBit = 30;         // pair.j bit: neighbour kept by the centre (STEINH Q cap)

enum SwType { SW_LINE = 0, SW_STEP = 1, SW_FERMI = 2, SW_TANH = 3, SW_RATIONAL = 4 };

// Switching-function parameters passed by value to kernels; the same fields as
// SwitchFunctionRequest (include/utils/zqc_switch_function.h:24-31).
struct SwParams {
    int type;
    double r0, d0, alpha;
    int n, m;
};

template <typename T> __host__ __device__ __forceinline__ T ipow_t(T x, int n) {
    T r = T(1);
    T b = x;
    int e = n < 0 ? -n : n;
    while (e) {
        if (e & 1) r *= b;
        b *= b;
        e >>= 1;
    }
    return n < 0 ? T(1) / r : r;
}

template <typename T> __host__ __device__ __forceinline__ T t_exp(T x);
template <> __host__ __device__ __forceinline__ double t_exp<double>(double x) { return exp(x); }
template <> __host__ __device__ __forceinline__ float t_exp<float>(float x) { return expf(x); }
template <typename T> __host__ __device__ __forceinline__ T t_tanh(T x);
template <> __host__ __device__ __forceinline__ double t_tanh<double>(double x) { return tanh(x); }
template <> __host__ __device__ __forceinline__ float t_tanh<float>(float x) { return tanhf(x); }
template <typename T> __host__ __device__ __forceinline__ T t_sqrt(T x);
template <> __host__ __device__ __forceinline__ double t_sqrt<double>(double x) { return sqrt(x); }
template <> __host__ __device__ __forceinline__ float t_sqrt<float>(float x) { return sqrtf(x); }

// f and df of the switching functions, following
// include/utils/zqc_switch_function.h:163-313 case by case (the RATIONAL n == 2m
// branch returns 1 + x^m exactly as the reference does).
template <typename T> __host__ __device__ __forceinline__ T sw_f(const SwParams &p, T x) {
    switch (p.type) {
    case SW_LINE: return T(1);
    case SW_STEP: return (x < T(p.r0)) ? T(1) : T(0);
    case SW_FERMI: return T(1) / (T(1) + t_exp<T>(-T(p.alpha) * (x - T(p.r0))));
    case SW_TANH: return T(0.5) * (T(1) + t_tanh<T>(T(p.alpha) * (x - T(p.r0))));
    case SW_RATIONAL: {
        const int n = p.n, m = p.m;
        T y = (x - T(p.d0)) / T(p.r0);
        if (n == 6 && m == 12) { T y2 = y * y; T y6 = y2 * y2 * y2; return T(1) / (T(1) + y6); }
        if (n == 4 && m == 8) { T y2 = y * y; T y4 = y2 * y2; return T(1) / (T(1) + y4); }
        if (2 * n == m) return T(1) / (T(1) + ipow_t(y, n));
        if (n == 2 * m) return T(1) + ipow_t(y, m);
        return (T(1) - ipow_t(y, n)) / (T(1) - ipow_t(y, m));
    }
    default: return T(1);
    }
}

template <typename T> __host__ __device__ __forceinline__ T sw_df(const SwParams &p, T x) {
    switch (p.type) {
    case SW_LINE: return T(0);
    case SW_STEP: return T(0);
    case SW_FERMI: {
        T e = t_exp<T>(-T(p.alpha) * (x - T(p.r0)));
        T den = T(1) + e;
        return (T(p.alpha) * e) / (den * den);
    }
    case SW_TANH: {
        T t = t_tanh<T>(T(p.alpha) * (x - T(p.r0)));
        return T(0.5) * T(p.alpha) * (T(1) - t * t);
    }
    case SW_RATIONAL: {
        const int n = p.n, m = p.m;
        T y = (x - T(p.d0)) / T(p.r0);
        if (n == 6 && m == 12) {
            T y2 = y * y, y5 = y2 * y2 * y, y6 = y2 * y2 * y2;
            return -T(n) * y5 / ((T(1) + y6) * (T(1) + y6)) / T(p.r0);
        }
        if (n == 4 && m == 8) {
            T y2 = y * y, y3 = y2 * y, y4 = y2 * y2;
            return -T(n) * y3 / ((T(1) + y4) * (T(1) + y4)) / T(p.r0);
        }
        if (2 * n == m) {
            T a = ipow_t(y, n - 1), b = ipow_t(y, n);
            return -T(n) * a / ((T(1) + b) * (T(1) + b)) / T(p.r0);
        }
        if (n == 2 * m) return T(m) * ipow_t(y, m - 1) / T(p.r0);
        T ymm1 = ipow_t(y, m - 1), ym = ymm1 * y;
        T one_m = T(1) - ym;
        if ((one_m < T(0) ? -one_m : one_m) < T(1e-12)) return T(-0.5) * T(n * (n - m)) / T(m) / T(p.r0);
        T ynm1 = ipow_t(y, n - 1);
        return (T(n - m) * ynm1 * ym + T(m) * ymm1 - T(n) * ynm1) / (one_m * one_m) / T(p.r0);
    }
    default: return T(0);
    }
}

// Pair record of the neighbour lists: displacement x_j - x_i (minimum image,
// computed in FP64 and rounded to T) and the sorted index of j (bit kFlagBit
// marks a neighbour kept by the centre's cap).
template <typename T> struct alignas(16) Pair;
template <> struct alignas(16) Pair<float> { float x, y, z; int j; };
template <> struct alignas(16) Pair<double> { double x, y, z; int j; int pad; };

// Device-side error word shared by the kernels of one context.
struct DevStatus {
    unsigned int overflow;        // max neighbour count seen when above capacity
    unsigned int nan_force;       // a force component was not finite
    unsigned int timeout;         // a bounded wait gave up
    unsigned int bad_pos;         // an atom position was not finite (NaN or Inf)
    unsigned int cand_overflow;   // max skin-list candidate count seen when above capacity
    unsigned int cap_overflow;    // the part of `overflow` that capped lists (STEINH Q) saw
    unsigned int pad[2];
};

// First statement of every step kernel: wait until the previous kernel of the
// stream has completed and its writes are visible, then let the next kernel's
// blocks be scheduled as this one's drain (no-ops without the PDL attribute).
__device__ __forceinline__ void pdl_entry() {
    asm volatile("griddepcontrol.wait;" ::: "memory");
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}

// The two halves, for a kernel that does work before its wait.  A block of a
// kernel K starts only after every block of the previous kernel P has let
// dependents launch; when P let them launch after its own wait, P's
// predecessor (and everything before it) has completed and is visible.  So
// before its wait K may read what the kernel two places back (or earlier)
// wrote, and must not read what P writes.  A kernel that lets dependents
// launch before its wait gives its successor no such window: that successor
// must open with its wait.
__device__ __forceinline__ void pdl_release() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

// Deterministic block sum of up to NV doubles per thread (fixed shuffle tree,
// then warp 0 over the warp partials).  Result valid in thread 0.
template <int NV>
__device__ __forceinline__ void block_sum(double (&v)[NV], double *smem /* NV * 32 */) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int nw = (blockDim.x + 31) >> 5;
#pragma unroll
    for (int t = 0; t < NV; ++t) {
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) v[t] += __shfl_down_sync(0xffffffffu, v[t], o);
    }
    if (lane == 0) {
#pragma unroll
        for (int t = 0; t < NV; ++t) smem[t * 32 + warp] = v[t];
    }
    __syncthreads();
    if (warp == 0) {
#pragma unroll
        for (int t = 0; t < NV; ++t) {
            double s = lane < nw ? smem[t * 32 + lane] : 0.0;
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) s += __shfl_down_sync(0xffffffffu, s, o);
            v[t] = s;
        }
    }
}

// Warp sums of NV = 2^P doubles per lane, spread over the lanes: lane l ends
// with the sum of value l >> (5 - P).  Lanes 16, 8, ... apart swap the halves
// of their values each step (NV - 1 shuffles), then the remaining steps add
// whole sums.  Every value is summed over the same tree of lanes as
// block_sum's shuffle-down steps (pairs 16, 8, 4, 2, 1 apart; each addition
// has the same two operands, possibly swapped), so the sums are equal bit
// for bit.
template <int NV> struct Log2NV { static constexpr int v = NV <= 1 ? 0 : 1 + Log2NV<NV / 2>::v; };
template <> struct Log2NV<1> { static constexpr int v = 0; };

template <int NV> __device__ __forceinline__ double warp_sum_spread(double (&v)[NV], int lane) {
    constexpr int P = Log2NV<NV>::v;
    static_assert((1 << P) == NV && P <= 5, "NV: a power of two up to 32");
#pragma unroll
    for (int st = 0; st < P; ++st) {
        const int o = 16 >> st, h = (NV >> st) / 2;
        const bool up = (lane & o) != 0;
#pragma unroll
        for (int j = 0; j < h; ++j) {
            const double send = up ? v[j] : v[j + h];
            const double keep = up ? v[j + h] : v[j];
            v[j] = keep + __shfl_xor_sync(0xffffffffu, send, o);
        }
    }
    double r = v[0];
#pragma unroll
    for (int st = P; st < 5; ++st) r += __shfl_xor_sync(0xffffffffu, r, 16 >> st);
    return r;
}

// block_sum with the totals spread over warp 0 (lane l of warp 0 returns the
// total of value l >> (5 - P); other warps return 0): the same totals bit
// for bit, with NV - 1 + 5 - P shuffles per warp instead of 5 NV.
template <int NV> __device__ __forceinline__ double block_sum_spread(double (&v)[NV], double *smem /* NV * 32 */) {
    constexpr int P = Log2NV<NV>::v;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int nw = (blockDim.x + 31) >> 5;
    const double r = warp_sum_spread<NV>(v, lane);
    if ((lane & ((32 >> P) - 1)) == 0) smem[(lane >> (5 - P)) * 32 + warp] = r;
    __syncthreads();
    double tot = 0.0;
    if (warp == 0) {
        double w[NV];
#pragma unroll
        for (int t = 0; t < NV; ++t) w[t] = lane < nw ? smem[t * 32 + lane] : 0.0;
        tot = warp_sum_spread<NV>(w, lane);
    }
    return tot;
}

}  // namespace mtd

namespace mtd {
template <typename T> __device__ __forceinline__ T t_rsqrt(T x);
template <> __device__ __forceinline__ float t_rsqrt<float>(float x) { return rsqrtf(x); }
template <> __device__ __forceinline__ double t_rsqrt<double>(double x) { return rsqrt(x); }

constexpr int pad4(int v) { return (v + 3) & ~3; }

// LAMMPS packed image flags (default 10-bit layout: IMGBITS 10, IMGMAX 512).
__device__ __forceinline__ void unpack_image(int img, int &ix, int &iy, int &iz) {
    ix = (img & 1023) - 512;
    iy = ((img >> 10) & 1023) - 512;
    iz = (img >> 20) - 512;
}
// sin and cos of pi * u for an FP64 phase u in half turns (the mixed-
// precision k-vector sums scale k by 1 / pi once, so u = (k / pi) . x):
// u is rounded to the nearest integer n in FP64 (adding 1.5 * 2^52 leaves n
// in the low mantissa bits, so no rounding or conversion instruction), the
// remainder f = u - n in [-1/2, 1/2] is exact in FP64 and goes to FP32,
// sin(pi f) = f P(f^2) and cos(pi f) = Q(f^2) come from polynomials of
// degree 4 and 5 in f^2, and (-1)^n flips both signs.  |u| < 2^51.
// P and Q are near-minimax on f in [0, 1/2]: least squares on Chebyshev
// nodes, reweighted toward equal error peaks (Lawson's algorithm), with
// maximum errors 6.7e-9 and 2.2e-10 in exact arithmetic, below the FP32
// rounding of the result (1.6e-7 with FP32 evaluation, the same as the
// degree-13 / degree-12 Taylor series they replace, two and one FMA fewer;
// fit_sincospi.py beside the library regenerates them).
constexpr float kSinP0 = (float)3.1415926402242746, kSinP1 = (float)-5.167710094404562,
                kSinP2 = (float)2.5500777409855013, kSinP3 = (float)-0.5982926899608115,
                kSinP4 = (float)0.07766048988359421;
constexpr float kCosQ0 = (float)0.9999999997811803, kCosQ1 = (float)-4.934802137317261,
                kCosQ2 = (float)4.058709167239208, kCosQ3 = (float)-1.3352120902337075,
                kCosQ4 = (float)0.23493771734282284, kCosQ5 = (float)-0.02439697684324065;
constexpr double kInvPi = 0.31830988618379067154;

// The sign flip of halfturn_sincos_f32 as a bit mask (bit 31 set for odd n),
// with sin(pi f) and cos(pi f) unsigned: callers that fold the sign into a
// later product take these three.
__device__ __forceinline__ unsigned halfturn_sincos_f32_parts(double u, float &s0, float &c0) {
    constexpr double kRound = 6755399441055744.0;   // 1.5 * 2^52
    const double t = u + kRound;
    const double f = u - (t - kRound);
    const float z = (float)f, z2 = z * z;
    float p = fmaf(z2, kSinP4, kSinP3);
    p = fmaf(p, z2, kSinP2);
    p = fmaf(p, z2, kSinP1);
    p = fmaf(p, z2, kSinP0);
    s0 = p * z;
    float q = fmaf(z2, kCosQ5, kCosQ4);
    q = fmaf(q, z2, kCosQ3);
    q = fmaf(q, z2, kCosQ2);
    q = fmaf(q, z2, kCosQ1);
    c0 = fmaf(q, z2, kCosQ0);
    return (unsigned)__double2loint(t) << 31;
}

__device__ __forceinline__ void halfturn_sincos_f32(double u, float &s, float &c) {
    float s0, c0;
    const unsigned sgn = halfturn_sincos_f32_parts(u, s0, c0);
    s = __uint_as_float(__float_as_uint(s0) ^ sgn);
    c = __uint_as_float(__float_as_uint(c0) ^ sgn);
}

// The k-vector passes' form of the same, for a pair of phases: the FP64 sum
// k.x runs on top of kTurnBase = 1.5 * 2^20, whose last bit is worth 2^-32, so
// each of its three FMAs rounds the phase to 2^-33 half turns (1.2e-10, where
// the FP32 remainder itself rounds to 1.5e-8) and the low word of the result
// is the remainder f = u - n in units of 2^-32, signed, with the parity of n
// in the bit above it and the low word's sign.  Three FP64 additions and the
// FP64-to-FP32 conversion (0.44 warp instructions per clock and SM, against
// 0.95 for the integer one) are gone.  Valid for |u| < 2^18 (kTurnMax).
// Rms errors against 80 bits of the passes that reduced each phase in FP64, and of
// these (1,372 to 256,000 atoms, 12 and 24 k): S(k) 3.6e-8 to 5.9e-8 and 3.6e-8 to
// 4.9e-8, forces 1.33e-7 to 1.66e-7 and 1.12e-7 to 1.54e-7.
constexpr double kTurnBase = 1572864.0;
constexpr double kTurnMax = 262144.0;

__device__ __forceinline__ float2 dup2(float v) { return make_float2(v, v); }
// (-1)^n of a phase as a sign mask.
__device__ __forceinline__ unsigned turn_sign(double t) {
    return ((unsigned)__double2hiint(t) << 31) ^ ((unsigned)__double2loint(t) & 0x80000000u);
}
// sin(pi f) (and cos(pi f)) of two based phases, unsigned, by the polynomials
// of halfturn_sincos_f32_parts on FP32 pairs (the same roundings per element;
// one instruction for two FMAs).
__device__ __forceinline__ float2 turn_sin2(double ta, double tb, float2 &s0) {
    const float2 zi = make_float2((float)__double2loint(ta), (float)__double2loint(tb));
    const float2 z = __fmul2_rn(zi, dup2(2.3283064365386963e-10f));   // 2^-32: exact
    const float2 z2 = __fmul2_rn(z, z);
    float2 p = __ffma2_rn(z2, dup2(kSinP4), dup2(kSinP3));
    p = __ffma2_rn(p, z2, dup2(kSinP2));
    p = __ffma2_rn(p, z2, dup2(kSinP1));
    p = __ffma2_rn(p, z2, dup2(kSinP0));
    s0 = __fmul2_rn(p, z);
    return z2;
}
__device__ __forceinline__ void turn_sincos2(double ta, double tb, float2 &s0, float2 &c0) {
    const float2 z2 = turn_sin2(ta, tb, s0);
    float2 q = __ffma2_rn(z2, dup2(kCosQ5), dup2(kCosQ4));
    q = __ffma2_rn(q, z2, dup2(kCosQ3));
    q = __ffma2_rn(q, z2, dup2(kCosQ2));
    q = __ffma2_rn(q, z2, dup2(kCosQ1));
    c0 = __ffma2_rn(q, z2, dup2(kCosQ0));
}

// FP64: a phase in radians less n half turns (or quarters), pi in two words
// (Cody and Waite, Software Manual for the Elementary Functions, 1980): both
// products are exact inside their FMA up to n = 2^51, so the remainder is off by
// its own rounding.  The phase itself is not scaled first: k / pi is rounded once
// more than k, and with k.x of some hundred radians the phase is most of an error
// (rms of the forces against 80 bits, 55,296 atoms x 12 k: 2.9e-14 scaled, 2.2e-14
// so, 2.6e-14 with sincos() of k.x).  |phase| < 2^50 (kPhaseMax).
constexpr double kPhaseMax = 1125899906842624.0;
__device__ __forceinline__ double phase_units(double ph, double per_unit, int &n) {
    constexpr double kRound = 6755399441055744.0;   // 1.5 * 2^52
    const double t = fma(ph, per_unit, kRound);
    n = __double2loint(t);
    return t - kRound;
}
__device__ __forceinline__ double flip(double v, int n) {   // (-1)^n v
    return __hiloint2double(__double2hiint(v) ^ (n << 31), __double2loint(v));
}

// sin(ph - shift) by its Taylor polynomial on |r| <= pi / 2 (remainder r^23 / 23!
// = 1e-18); the shift, |shift| <= pi, is taken off the small remainder.
__device__ __forceinline__ double phase_sin_f64(double ph, double shift) {
    constexpr double S[10] = {-0.16666666666666666, 0.008333333333333333, -0.0001984126984126984,
                              2.7557319223985893e-06, -2.505210838544172e-08, 1.6059043836821613e-10,
                              -7.647163731819816e-13, 2.8114572543455206e-15, -8.22063524662433e-18,
                              1.9572941063391263e-20};
    int n;
    const double q = phase_units(ph - shift, kInvPi, n);
    const double r = fma(-q, 1.2246467991473532e-16, fma(-q, 3.141592653589793, ph) - shift), z = r * r;
    double p = S[9];
#pragma unroll
    for (int k = 8; k >= 0; --k) p = fma(p, z, S[k]);
    return flip(fma(r * z, p, r), n);
}

// sin and cos by theirs on |r| <= pi / 4 (remainders r^19 / 19! = 8e-20 and
// r^18 / 18! = 2e-18), exchanged in odd quarters.
__device__ __forceinline__ void phase_sincos_f64(double ph, double &s, double &c) {
    constexpr double S[8] = {-0.16666666666666666, 0.008333333333333333, -0.0001984126984126984,
                             2.7557319223985893e-06, -2.505210838544172e-08, 1.6059043836821613e-10,
                             -7.647163731819816e-13, 2.8114572543455206e-15};
    constexpr double C[8] = {-0.5, 0.041666666666666664, -0.001388888888888889, 2.48015873015873e-05,
                             -2.755731922398589e-07, 2.08767569878681e-09, -1.1470745597729725e-11,
                             4.779477332387385e-14};
    int n;
    const double u = phase_units(ph, 2.0 * kInvPi, n);
    const double r = fma(-u, 6.123233995736766e-17, fma(-u, 1.5707963267948966, ph)), z = r * r;
    double p = S[7], q = C[7];
#pragma unroll
    for (int k = 6; k >= 0; --k) {
        p = fma(p, z, S[k]);
        q = fma(q, z, C[k]);
    }
    p = fma(r * z, p, r);
    q = fma(q, z, 1.0);
    s = flip(n & 1 ? q : p, n >> 1);
    c = flip(n & 1 ? p : q, (n + 1) >> 1);
}

// The same for a phase in radians (one FP64 multiply by 1 / pi first).
__device__ __forceinline__ void phase_sincos_f32(double ph, float &s, float &c) {
    halfturn_sincos_f32(ph * kInvPi, s, c);
}

}  // namespace mtd
