// mlp.cu -- learned bias V_theta(s) for CV_dim >= 3: an MLP D -> 128 -> 128 -> 1
// with SiLU activations, BF16 weights and FP32 accumulation, trained on the GPU
// on the FP64 hill sum the method deposits, which stays the measure of its error
// and the fallback.  No counterpart in the reference (its grids are the only
// bias representation: src/grids/GH_t0_uniformGrid.cu, GH_t1_sparseGrid.cu).
//
// Kernels
//   hillsum_batch     exact FP64 V and dV/ds for a batch of points (hillsum.cu)
//   k_hillsum_point   exact FP64 V and dV/ds at one point, hills spread over the grid
//   k_mlp_eval        V and dV/ds of 128-point tiles: layers 1 and 3 on CUDA cores, the
//                     128 x 128 layer and its backward contraction on tcgen05 (TMEM accumulators)
//   k_mlp_train       one 128-point tile's parameter gradients: three tcgen05 contractions
//   k_mlp_adam        sums the per-tile gradients in tile order, Adam step, BF16 copies
//   k_mlp_point       V_theta and dV_theta/ds at one point (CUDA cores, one block)
//
// Network on normalised inputs u = 2 (s - lo) / (hi - lo) - 1 and outputs
// V = vscale * y:  z1 = W1 u + b1, h1 = silu(z1), z2 = W2 h1 + b2,
// h2 = silu(z2), y = w3 . h2 + b3.  W1, W2, w3 are used as BF16 values
// (FP32 masters for Adam); h1 and dL/dz2 are rounded to BF16 as tensor-core
// operands, every sum accumulates in FP32.
#include <cuda_bf16.h>

#include <cmath>
#include <cstring>
#include <mutex>
#include <random>
#include <string>
#include <vector>

#include "../../include/metad_b200.h"
#include "common.cuh"
#include "hillsum.h"
#include "umma.cuh"

namespace mtd {

namespace {

constexpr int kH = 128;                 // hidden width
constexpr int kIn = 4;                  // input slots (D <= 4)
constexpr int oW1 = 0;                  // flat parameter layout
constexpr int ob1 = oW1 + kH * kIn;
constexpr int oW2 = ob1 + kH;
constexpr int ob2 = oW2 + kH * kH;
constexpr int ow3 = ob2 + kH;
constexpr int ob3 = ow3 + kH;
constexpr int kNP = ob3 + 1;            // 17,281 parameters
constexpr int kNPpad = (kNP + 3) / 4 * 4;
constexpr int kWaitTries = 1 << 20;     // bounded mbarrier waits (default limit)

struct MlpDev {
    int D;
    const float *W1, *b1, *b2, *w3, *b3;       // W1, w3: BF16-rounded values
    const __nv_bfloat16 *W2, *W2t;             // [n][k] and [k][n]
};

// 1 / (1 + exp(-z)): exp by the SFU, and the reciprocal by the SFU with one Newton
// step, which leaves it within half a unit of the last place and a little.  The
// outputs of 65,536 points are those of a correctly rounded reciprocal bit for bit,
// and the batch takes 27 us where that takes 44.  Where the exponential overflows
// (the cap keeps the step finite) the SFU's reciprocal is 0, and so are z * sigmoid
// and its derivative.
__device__ __forceinline__ float sigmoid(float z) {
    const float a = fminf(1.0f + __expf(-z), 3.402823466e38f);
    float r;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(a));
    return fmaf(r, fmaf(-a, r, 1.0f), r);
}
__device__ __forceinline__ float silu(float z, float &dsilu) {
    const float s = sigmoid(z);
    dsilu = s * (1.0f + z * (1.0f - s));
    return z * s;
}

// Barrier `id` of 128 threads; the second form also votes.
__device__ __forceinline__ void wg_sync(int id) {
    asm volatile("barrier.cta.sync %0, 128;" ::"r"(id) : "memory");
    __syncwarp();
}
__device__ __forceinline__ bool wg_all(int id, bool v) {
    uint32_t r;
    asm volatile(
        "{\n\t.reg .pred p, q;\n\t"
        "setp.ne.u32 p, %2, 0;\n\t"
        "barrier.cta.red.and.pred q, %1, 128, p;\n\t"
        "selp.u32 %0, 1, 0, q;\n\t}\n"
        : "=r"(r)
        : "r"(id), "r"((uint32_t)v)
        : "memory");
    __syncwarp();
    return r != 0;
}

// Where a batch's points come from and its results go: network units (x, y,
// ds: rows of kIn floats) or the caller's doubles (pts, V, dV: rows of D),
// normalised and scaled here.
struct MlpIo {
    const float *x;
    float *y, *ds;
    const double *pts;
    double *V, *dV;
    double lo[kIn], sc[kIn], vscale;
};

__device__ __forceinline__ void mlp_input(const MlpIo &io, int D, int row, bool valid, float (&u)[kIn]) {
#pragma unroll
    for (int i = 0; i < kIn; ++i) {
        u[i] = 0.f;
        if (valid && i < D)
            u[i] = io.pts ? (float)(io.sc[i] * (io.pts[(size_t)row * D + i] - io.lo[i]) - 1.0)
                          : io.x[(size_t)row * kIn + i];
    }
}

// Shared memory of both tile kernels: W2, W2^T (32 KB each, operand layout),
// the small weights (W1 as float4 rows, b1, b2, w3), then the kernel's own.
constexpr int kSmW = 2 * 32768, kSmSmall = (4 + 3) * kH * 4;

__device__ __forceinline__ void load_weights(const MlpDev &p, unsigned char *sm, bool back) {
    // 16-byte vectors, eight rows by four K chunks a warp: 64 contiguous bytes
    // of each row, and eight lanes fill one 128-byte core matrix (a row's chunks
    // side by side in a warp hit one bank group)
#pragma unroll 4
    for (int e = threadIdx.x; e < kH * kH / 8; e += blockDim.x) {
        const int r = (e >> 7) * 8 + (e & 7), c = (e >> 3) & 15;
        const uint4 v = reinterpret_cast<const uint4 *>(p.W2)[r * (kH / 8) + c];
        const uint4 vt = back ? reinterpret_cast<const uint4 *>(p.W2t)[r * (kH / 8) + c] : v;
        *reinterpret_cast<uint4 *>(sm + umma_off(r, 8 * c, kH)) = v;
        if (back) *reinterpret_cast<uint4 *>(sm + 32768 + umma_off(r, 8 * c, kH)) = vt;
    }
    float *w = reinterpret_cast<float *>(sm + kSmW);
    for (int e = threadIdx.x; e < kH * kIn; e += blockDim.x) w[e] = p.W1[e];
    for (int e = threadIdx.x; e < kH; e += blockDim.x) {
        w[4 * kH + e] = p.b1[e];
        w[5 * kH + e] = p.b2[e];
        w[6 * kH + e] = p.w3[e];
    }
}

__device__ __forceinline__ float layer1(const float4 *sW1, const float *sb1, int j, const float (&u)[kIn]) {
    const float4 w = sW1[j];
    return fmaf(w.w, u[3], fmaf(w.z, u[2], fmaf(w.y, u[1], fmaf(w.x, u[0], sb1[j]))));
}

// Columns [c0, c0 + n) of h1 = silu(z1) of this thread's row, in BF16, into the
// A operand.
__device__ __forceinline__ void write_h1(const float4 *sW1, const float *sb1, const float (&u)[kIn], int m, int c0,
                                         int n, unsigned char *sA) {
#pragma unroll 2
    for (int c = c0; c < c0 + n; c += 8) {
        __align__(16) __nv_bfloat16 hb[8];
#pragma unroll
        for (int e = 0; e < 8; ++e) {
            const float z = layer1(sW1, sb1, c + e, u);
            hb[e] = __float2bfloat16_rn(z * sigmoid(z));
        }
        *reinterpret_cast<uint4 *>(sA + umma_off(m, c, kH)) = *reinterpret_cast<const uint4 *>(hb);
    }
}

// D[128 x 128] = A B^T over K = 128, both K-major, issued by one thread.
__device__ __forceinline__ void mma_tile(uint32_t d, const unsigned char *sA, const unsigned char *sB) {
#pragma unroll
    for (int kk = 0; kk < kH / 16; ++kk)
        umma_bf16(d, umma_desc(smem_addr(sA) + kk * 2 * kH * 16, kH * 16, 128),
                  umma_desc(smem_addr(sB) + kk * 2 * kH * 16, kH * 16, 128), umma_idesc_bf16(kH, kH), kk > 0 ? 1u : 0u);
}

// Forward pass (GRAD: and input gradient) of 128 points per tile.  Each of the
// block's four warpgroups has its own A operand (32 KB) and 128 columns of
// tensor memory, so that one's SiLU work runs beside another's MMA; the block
// stays for all its tiles and loads the weights once.  CS = 1: a tile per
// warpgroup.  CS = 4: a tile per block, each warpgroup taking 32 of the 128
// columns of every layer (batches too small to give every warpgroup a tile).
// Bound by the SFU and FP32 work of three SiLU evaluations per hidden unit and
// point (the MMAs are under 5 % of it): 5.7 us per tile and SM, of which the
// SFU's two calls a SiLU take 3.1.  V and dV/ds at 65,536 points: 198 us before
// (one warpgroup and one tile a block, four SiLU evaluations, inputs and
// outputs converted by kernels of their own), 31 now; up to 148 tiles 14.
//
// A bounded wait that runs out (in any thread: the warpgroup votes) ends the
// warpgroup's work: it issues no further MMA, reads no TMEM and overwrites no
// operand the tensor core may still be reading; it waits once more (same
// limit) for the batch in flight, sets *err and meets the others at the end,
// where the block's TMEM is released.  stall != 0 is the check of that path:
// after its first batch has completed, every warpgroup waits on the barrier's
// next phase, which no commit will complete.
template <bool GRAD, int CS>
__global__ void __launch_bounds__(512, 1)
    k_mlp_eval(MlpDev p, int npts, MlpIo io, int *err, int tries, int stall) {
    extern __shared__ __align__(1024) unsigned char sm[];
    __shared__ uint64_t mbar[4];
    __shared__ uint32_t tbase;
    const float4 *sW1 = reinterpret_cast<const float4 *>(sm + kSmW);
    const float *sb1 = reinterpret_cast<const float *>(sm + kSmW) + 4 * kH, *sb2 = sb1 + kH, *sw3 = sb2 + kH;
    const int wg = threadIdx.x >> 7, m = threadIdx.x & 127, warp = threadIdx.x >> 5;
    constexpr int NC = kH / CS;                         // columns of a thread
    const int c0 = CS > 1 ? NC * wg : 0, who = CS > 1 ? 0 : wg;
    unsigned char *sA = sm + kSmW + kSmSmall + who * 32768;
    float *red = reinterpret_cast<float *>(sm + kSmW + kSmSmall + 32768);   // CS > 1: [4][1 + kIn][128]
    if (threadIdx.x < 4) mbar_init(&mbar[threadIdx.x], 1);
    if (warp == 0) tmem_alloc(&tbase, 512);
    load_weights(p, sm, GRAD);
    tc_fence_before();
    fence_async_smem();
    __syncthreads();
    tc_fence_after();
    const uint32_t taddr = tbase + who * kH, lane_addr = taddr + (static_cast<uint32_t>((warp & 3) * 32) << 16);
    const int ntiles = (npts + kH - 1) / kH;
    uint32_t phase = 0;
    bool alive = true;
    auto sync = [&] {
        if (CS > 1) __syncthreads();
        else wg_sync(1 + wg);
    };
    auto vote = [&](bool v) { return CS > 1 ? __syncthreads_and(v) != 0 : wg_all(1 + wg, v); };
    // operand written by this warpgroup -> one thread issues -> every thread waits
    auto run_mma = [&](const unsigned char *sB) {
        tc_fence_before();
        fence_async_smem();
        sync();
        tc_fence_after();
        if (CS > 1 ? threadIdx.x == 0 : m == 0) {
            mma_tile(taddr, sA, sB);
            umma_commit(&mbar[who]);
        }
        bool ok = mbar_wait(&mbar[who], phase, tries);
        if (stall) ok = mbar_wait(&mbar[who], phase ^ 1, tries) && ok;
        ok = vote(ok);
        if (!ok) mbar_wait(&mbar[who], phase, tries);
        tc_fence_after();
        phase ^= 1;
        return ok;
    };
    for (int tile = CS > 1 ? blockIdx.x : wg * gridDim.x + blockIdx.x; tile < ntiles;
         tile += CS > 1 ? gridDim.x : 4 * gridDim.x) {
        const int row = tile * kH + m;
        const bool valid = row < npts;
        float u[kIn];
        mlp_input(io, p.D, row, valid, u);
        write_h1(sW1, sb1, u, m, c0, NC, sA);
        if (!(alive = run_mma(sm))) break;
        // z2 = D + b2, y = w3 . silu(z2) + b3, dy/dz2 in BF16 over the consumed h1
        float y = CS > 1 && wg ? 0.f : p.b3[0];
#pragma unroll 1
        for (int c = c0; c < c0 + NC; c += 16) {
            float z[16];
            tmem_ld16(lane_addr + c, z);
            __align__(16) __nv_bfloat16 gb[16];
#pragma unroll
            for (int e = 0; e < 16; ++e) {
                float dsl;
                y = fmaf(sw3[c + e], silu(z[e] + sb2[c + e], dsl), y);
                if (GRAD) gb[e] = __float2bfloat16_rn(sw3[c + e] * dsl);
            }
            if (GRAD) {
                *reinterpret_cast<uint4 *>(sA + umma_off(m, c, kH)) = reinterpret_cast<const uint4 *>(gb)[0];
                *reinterpret_cast<uint4 *>(sA + umma_off(m, c + 8, kH)) = reinterpret_cast<const uint4 *>(gb)[1];
            }
        }
        float du[kIn] = {0.f, 0.f, 0.f, 0.f};
        if (GRAD) {
            if (!(alive = run_mma(sm + 32768))) break;   // dy/dh1 = dy/dz2 W2
#pragma unroll 1
            for (int c = c0; c < c0 + NC; c += 16) {
                float dh[16];
                tmem_ld16(lane_addr + c, dh);
#pragma unroll
                for (int e = 0; e < 16; ++e) {
                    const float4 w = sW1[c + e];
                    float dsl;
                    silu(layer1(sW1, sb1, c + e, u), dsl);
                    const float g = dh[e] * dsl;
                    du[0] = fmaf(g, w.x, du[0]);
                    du[1] = fmaf(g, w.y, du[1]);
                    du[2] = fmaf(g, w.z, du[2]);
                    du[3] = fmaf(g, w.w, du[3]);
                }
            }
        }
        if (CS > 1) {   // the column groups' sums, in their order
            red[(wg * (1 + kIn)) * kH + m] = y;
            for (int i = 0; i < kIn; ++i) red[(wg * (1 + kIn) + 1 + i) * kH + m] = du[i];
            __syncthreads();
            if (wg == 0)
                for (int q = 1; q < 4; ++q) {
                    y += red[q * (1 + kIn) * kH + m];
                    for (int i = 0; i < kIn; ++i) du[i] += red[(q * (1 + kIn) + 1 + i) * kH + m];
                }
        }
        if (valid && (CS == 1 || wg == 0)) {
            if (io.pts) {
                io.V[row] = io.vscale * (double)y;
                if (GRAD)
#pragma unroll
                    for (int i = 0; i < kIn; ++i)
                        if (i < p.D) io.dV[(size_t)row * p.D + i] = io.vscale * (double)du[i] * io.sc[i];
            } else {
                io.y[row] = y;
                if (GRAD) *reinterpret_cast<float4 *>(io.ds + (size_t)row * kIn) = make_float4(du[0], du[1], du[2], du[3]);
            }
        }
    }
    if (!alive && m == 0) atomicExch(err, 1);
    tc_fence_before();
    __syncthreads();
    if (warp == 0) tmem_dealloc(tbase, 512);
}

// Sums over the 32 lanes of N values a lane (N a power of two up to 32): lanes
// 16, 8, ... apart swap halves of their values, so lane l ends with the sum of
// value l * N / 32.
template <int N> __device__ __forceinline__ float lanes_sum(float (&v)[N], int lane) {
    constexpr int P = N == 32 ? 5 : N == 16 ? 4 : 3;
    static_assert(N == 1 << P, "N: 8, 16 or 32");
#pragma unroll
    for (int st = 0; st < P; ++st) {
        const int o = 16 >> st, h = (N >> st) / 2;
        const bool up = (lane & o) != 0;
#pragma unroll
        for (int j = 0; j < h; ++j) {
            const float send = up ? v[j] : v[j + h], keep = up ? v[j + h] : v[j];
            v[j] = keep + __shfl_xor_sync(0xffffffffu, send, o);
        }
    }
    float r = v[0];
#pragma unroll
    for (int st = P; st < 5; ++st) r += __shfl_xor_sync(0xffffffffu, r, 16 >> st);
    return r;
}

// One 128-point training tile per block: loss and the parameter gradients of
// sum (y - t)^2 scaled by grad_scale, as one row of `part`.  Four warpgroups
// take 32 columns each of every layer.  The three MMAs share two operands: h1
// and dL/dz2, rows of points; dL/dW2 = dL/dz2^T h1 reads both transposed
// (M-major descriptors), so no transposed copies are written (two-byte stores
// down a column cost a bank conflict each).  Sums over a tile's points go
// through warp butterflies (lanes_sum) and the four warps' rows in order.
// 8,192 points (64 tiles): 72 us before (128 threads a tile; row sums through a
// [128][97] scratch tile), 20 now; latency of one tile's serial phases.
// Timeouts as in k_mlp_eval, the whole block together.
constexpr int kEvalSmem = kSmW + kSmSmall + 4 * 32768;
constexpr int kTrainRed = 7 * 4 * kH;   // [value][row warp][column]: b2, w3, b1, W1 x 4
constexpr int kTrainSmem = kSmW + kSmSmall + 2 * 32768 + kTrainRed * 4;
// A training batch: network units (x rows of kIn, t), or the caller's doubles
// (pts rows of D, tgt), normalised here by the operations of nb_normalise.
struct MlpBatch {
    const float *x, *t;
    const double *pts, *tgt;
    double lo[kIn], span[kIn], vscale;
};
__global__ void __launch_bounds__(512, 1)
    k_mlp_train(MlpDev p, int npts, MlpBatch in, float *part, float *loss_part, float grad_scale, int *err, int tries,
                int stall) {
    extern __shared__ __align__(1024) unsigned char sm[];
    __shared__ uint64_t mbar;
    __shared__ uint32_t tbase;
    __shared__ float srow[2][4][kH], sdy[kH], sl[4], sb3[4];
    const float4 *sW1 = reinterpret_cast<const float4 *>(sm + kSmW);
    const float *sb1 = reinterpret_cast<const float *>(sm + kSmW) + 4 * kH, *sb2 = sb1 + kH, *sw3 = sb2 + kH;
    unsigned char *sH = sm + kSmW + kSmSmall, *sG = sH + 32768;
    float *red = reinterpret_cast<float *>(sG + 32768);
    const int wg = threadIdx.x >> 7, m = threadIdx.x & 127, warp = threadIdx.x >> 5, rw = warp & 3;
    const int lane = threadIdx.x & 31, c0 = 32 * wg, row = blockIdx.x * kH + m;
    const bool valid = row < npts;
    if (threadIdx.x == 0) mbar_init(&mbar, 1);
    if (warp == 0) tmem_alloc(&tbase, 512);
    load_weights(p, sm, true);
    float u[kIn] = {0.f, 0.f, 0.f, 0.f};
    if (valid && in.pts) {
#pragma unroll
        for (int i = 0; i < kIn; ++i)
            if (i < p.D)
                u[i] = (float)(2.0 * (in.pts[(size_t)row * p.D + i] - in.lo[i]) / in.span[i] - 1.0);
    } else if (valid) {
        const float4 v = *reinterpret_cast<const float4 *>(in.x + (size_t)row * kIn);
        u[0] = v.x;
        u[1] = v.y;
        u[2] = v.z;
        u[3] = v.w;
    }
    __syncthreads();
    write_h1(sW1, sb1, u, m, c0, 32, sH);
    uint32_t phase = 0;
    auto wait = [&] {
        bool ok = mbar_wait(&mbar, phase, tries);
        if (stall) ok = mbar_wait(&mbar, phase ^ 1, tries) && ok;
        ok = __syncthreads_and(ok) != 0;
        if (!ok) mbar_wait(&mbar, phase, tries);
        tc_fence_after();
        phase ^= 1;
        return ok;
    };
    tc_fence_before();
    fence_async_smem();
    __syncthreads();
    tc_fence_after();
    const uint32_t taddr = tbase, lane_addr = taddr + (static_cast<uint32_t>(rw * 32) << 16);
    if (threadIdx.x == 0) {
        mma_tile(taddr, sH, sm);
        umma_commit(&mbar);
    }
    bool ok = wait();
    if (ok) {
        // forward: this column group's part of y; w3 silu'(z2) and silu(z2) wait for dy
        float wd[32], h2[32];
        float y = wg ? 0.f : p.b3[0];
#pragma unroll
        for (int c = 0; c < 32; c += 16) {
            float z[16];
            tmem_ld16(lane_addr + c0 + c, z);
#pragma unroll
            for (int e = 0; e < 16; ++e) {
                const int n = c0 + c + e;
                float dsl;
                h2[c + e] = silu(z[e] + sb2[n], dsl);
                y = fmaf(sw3[n], h2[c + e], y);
                wd[c + e] = dsl;
            }
        }
        srow[0][wg][m] = y;
        __syncthreads();
        if (wg == 0) {
            y = srow[0][0][m] + srow[0][1][m] + srow[0][2][m] + srow[0][3][m];
            const float target = !valid ? y : in.pts ? (float)(in.tgt[row] / in.vscale) : in.t[row];
            const float d = y - target;
            sdy[m] = grad_scale * d;
            float l = d * d, g = grad_scale * d;
            for (int o = 16; o > 0; o >>= 1) {
                l += __shfl_xor_sync(0xffffffffu, l, o);
                g += __shfl_xor_sync(0xffffffffu, g, o);
            }
            if (lane == 0) {
                sl[rw] = l;
                sb3[rw] = g;
            }
        }
        __syncthreads();
        if (threadIdx.x == 0) {
            loss_part[blockIdx.x] = sl[0] + sl[1] + sl[2] + sl[3];
            part[(size_t)blockIdx.x * kNPpad + ob3] = sb3[0] + sb3[1] + sb3[2] + sb3[3];
        }
        const float dy = sdy[m];
        // dL/dz2 = dy w3 silu'(z2) in BF16; b2 and w3 gradients summed in FP32
#pragma unroll
        for (int e = 0; e < 32; ++e) {
            wd[e] = dy * sw3[c0 + e] * wd[e];
            h2[e] = dy * h2[e];
        }
#pragma unroll
        for (int c = 0; c < 32; c += 8) {
            __align__(16) __nv_bfloat16 gb[8];
#pragma unroll
            for (int e = 0; e < 8; ++e) gb[e] = __float2bfloat16_rn(wd[c + e]);
            *reinterpret_cast<uint4 *>(sG + umma_off(m, c0 + c, kH)) = *reinterpret_cast<const uint4 *>(gb);
        }
        red[(0 * 4 + rw) * kH + c0 + lane] = lanes_sum<32>(wd, lane);
        red[(1 * 4 + rw) * kH + c0 + lane] = lanes_sum<32>(h2, lane);
        tc_fence_before();
        fence_async_smem();
        __syncthreads();
        tc_fence_after();
        if (threadIdx.x == 0) {
            mma_tile(taddr + kH, sG, sm + 32768);   // dL/dh1 = dL/dz2 W2
#pragma unroll
            for (int kk = 0; kk < kH / 16; ++kk)    // dL/dW2 = dL/dz2^T h1, K = the tile's points
                umma_bf16(taddr + 2 * kH, umma_desc(smem_addr(sG) + kk * 256, 128, kH * 16),
                          umma_desc(smem_addr(sH) + kk * 256, 128, kH * 16),
                          umma_idesc_bf16(kH, kH) | kIdescTransA | kIdescTransB, kk > 0 ? 1u : 0u);
            umma_commit(&mbar);
        }
        ok = wait();
    }
    if (ok) {
        // layer 1: dL/dz1 = dL/dh1 silu'(z1), eight columns at a time
#pragma unroll 1
        for (int c = c0; c < c0 + 32; c += 8) {
            float dh[8], g[8], q[8];
            tmem_ld8(lane_addr + kH + c, dh);
#pragma unroll
            for (int e = 0; e < 8; ++e) {
                float dsl;
                silu(layer1(sW1, sb1, c + e, u), dsl);
                g[e] = dh[e] * dsl;
            }
#pragma unroll
            for (int v = 0; v < 1 + kIn; ++v) {
#pragma unroll
                for (int e = 0; e < 8; ++e) q[e] = v ? g[e] * u[v ? v - 1 : 0] : g[e];
                const float sum = lanes_sum<8>(q, lane);
                if ((lane & 3) == 0) red[((2 + v) * 4 + rw) * kH + c + (lane >> 2)] = sum;
            }
        }
        // rows of the W2 gradient: this thread's row n = m, 32 columns
        float *dst = part + (size_t)blockIdx.x * kNPpad + oW2 + (size_t)m * kH + c0;
#pragma unroll
        for (int c = 0; c < 32; c += 16) {
            float g[16];
            tmem_ld16(lane_addr + 2 * kH + c0 + c, g);
#pragma unroll
            for (int e = 0; e < 16; e += 4)
                *reinterpret_cast<float4 *>(dst + c + e) = make_float4(g[e], g[e + 1], g[e + 2], g[e + 3]);
        }
        __syncthreads();
        for (int e = threadIdx.x; e < 7 * kH; e += blockDim.x) {
            const int v = e / kH, n = e % kH;
            const float *r = red + (size_t)v * 4 * kH + n;
            const float s = r[0] + r[kH] + r[2 * kH] + r[3 * kH];
            const int at = v == 0 ? ob2 + n : v == 1 ? ow3 + n : v == 2 ? ob1 + n : oW1 + n * kIn + (v - 3);
            part[(size_t)blockIdx.x * kNPpad + at] = s;
        }
    } else if (threadIdx.x == 0) {
        atomicExch(err, 1);
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 0) tmem_dealloc(tbase, 512);
}

__device__ __forceinline__ float bf16_round(float v) { return __bfloat162float(__float2bfloat16_rn(v)); }

// Parameter q of a block of 256: 64 parameters by 4 groups of tiles (tiles g,
// g + 4, ...), whose sums are added in order; true on the thread that goes on.
constexpr int kSumQ = 64, kSumBlocks = (kNP + kSumQ - 1) / kSumQ;
__device__ __forceinline__ bool tile_sum(int ntiles, const float *__restrict__ part, int &q, float &g) {
    __shared__ float sums[4][kSumQ];
    const int grp = threadIdx.x / kSumQ, at = threadIdx.x % kSumQ;
    q = blockIdx.x * kSumQ + at;
    float s = 0.0f;
    if (q < kNP) {
#pragma unroll 4
        for (int t = grp; t < ntiles; t += 4) s += part[(size_t)t * kNPpad + q];
    }
    sums[grp][at] = s;
    __syncthreads();
    g = sums[0][at] + sums[1][at] + sums[2][at] + sums[3][at];
    return grp == 0 && q < kNP;
}

// Adam on the FP32 masters with the gradient summed over tiles in a fixed
// order; refreshes the forward copies (BF16 W1, W2, W2^T, w3; FP32 biases).
__global__ void k_mlp_adam(int ntiles, const float *__restrict__ part, float *master, float *mom, float *vel,
                           float lr, float b1c, float b2c, float *W1, float *b1, __nv_bfloat16 *W2,
                           __nv_bfloat16 *W2t, float *b2, float *w3, float *b3, int update) {
    int q;
    float g;
    if (!tile_sum(ntiles, part, q, g)) return;
    float w = master[q];
    if (update) {
        const float m1 = 0.9f * mom[q] + 0.1f * g;
        const float v1 = 0.999f * vel[q] + 0.001f * g * g;
        mom[q] = m1;
        vel[q] = v1;
        w -= lr * (m1 / b1c) / (sqrtf(v1 / b2c) + 1e-8f);
        master[q] = w;
    }
    if (q < ob1) W1[q] = bf16_round(w);
    else if (q < oW2) b1[q - ob1] = w;
    else if (q < ob2) {
        const int n = (q - oW2) / kH, k = (q - oW2) % kH;
        W2[n * kH + k] = __float2bfloat16_rn(w);
        W2t[k * kH + n] = __float2bfloat16_rn(w);
    } else if (q < ow3) b2[q - ob2] = w;
    else if (q < ob3) w3[q - ow3] = bf16_round(w);
    else b3[0] = w;
}

// Gradient summed over tiles without an update (for checks), followed by the
// timeout flag and the tiles' losses, so that one copy brings all of it.
__global__ void k_mlp_gradsum(int ntiles, const float *__restrict__ part, const float *__restrict__ loss,
                              const int *__restrict__ err, float *g) {
    for (int t = blockIdx.x * blockDim.x + threadIdx.x; t <= ntiles; t += gridDim.x * blockDim.x)
        g[kNPpad + t] = t ? loss[t - 1] : __int_as_float(*err);
    int q;
    float s;
    if (tile_sum(ntiles, part, q, s)) g[q] = s;
}

// Hills packed as in hillsum.h.  A hill farther than sqrt(80) sigma from the
// point contributes below h e^-40 (4e-18 h) and is skipped; its gradient term
// is smaller still.
constexpr double kExpCut = 40.0;

// One point, hills spread over blocks; block partials reduced in block order by the last block.
constexpr int kPointBlocks = 80;
__global__ void __launch_bounds__(256) k_hillsum_point(int D, const double *__restrict__ s_in, int h_begin, int nh,
                                                       const double *__restrict__ hills, double *part,
                                                       unsigned int *ticket, double *V, double *dV,
                                                       int accumulate) {
    __shared__ double smem[5 * 32];
    __shared__ bool last;
    double s[kIn] = {0, 0, 0, 0};
    for (int k = 0; k < D; ++k) s[k] = s_in[k];
    double acc[5] = {0, 0, 0, 0, 0};
    for (int h = h_begin + blockIdx.x * blockDim.x + threadIdx.x; h < nh; h += gridDim.x * blockDim.x) {
        const double *c = hills + (size_t)h * 8;
        double r2 = 0.0, d[kIn];
#pragma unroll
        for (int k = 0; k < kIn; ++k) {
            d[k] = k < D ? s[k] - c[k] : 0.0;
            r2 += d[k] * d[k];
        }
        const double a = r2 * c[5];
        if (a < kExpCut) {
            const double e = c[4] * exp(-a);
            acc[0] += e;
#pragma unroll
            for (int k = 0; k < kIn; ++k) acc[1 + k] -= e * d[k] * c[6];
        }
    }
    block_sum<5>(acc, smem);
    if (threadIdx.x == 0) {
        for (int q = 0; q < 5; ++q) part[blockIdx.x * 5 + q] = acc[q];
        __threadfence();
        last = atomicAdd(ticket, 1u) == gridDim.x - 1;
    }
    __syncthreads();
    if (last && threadIdx.x < 5) {
        __threadfence();
        double t = 0.0;
        for (int b = 0; b < (int)gridDim.x; ++b) t += *((volatile double *)part + b * 5 + threadIdx.x);
        if (threadIdx.x == 0) *V = accumulate ? *V + t : t;
        else if ((int)threadIdx.x - 1 < D) dV[threadIdx.x - 1] = accumulate ? dV[threadIdx.x - 1] + t : t;
        if (threadIdx.x == 0) *ticket = 0u;
    }
}

// V_theta and dV_theta/ds at one point (FP64 in/out), one block of 128 threads.
__global__ void __launch_bounds__(128) k_mlp_point(MlpDev p, const double *__restrict__ s_in, double lo0, double lo1,
                                                   double lo2, double lo3, double sc0, double sc1, double sc2,
                                                   double sc3, double vscale, double *V, double *dV) {
    __shared__ float h1[kH], dz2[kH], red[kIn + 1][4];
    const int j = threadIdx.x, warp = j >> 5;
    const double lo[kIn] = {lo0, lo1, lo2, lo3}, sc[kIn] = {sc0, sc1, sc2, sc3};   // sc = 2 / (hi - lo)
    float u[kIn] = {0.f, 0.f, 0.f, 0.f};
    for (int i = 0; i < p.D; ++i) u[i] = (float)((s_in[i] - lo[i]) * sc[i] - 1.0);
    float z1 = p.b1[j];
    for (int i = 0; i < kIn; ++i) z1 = fmaf(p.W1[j * kIn + i], u[i], z1);
    float ds1;
    h1[j] = __bfloat162float(__float2bfloat16_rn(silu(z1, ds1)));
    __syncthreads();
    float z2 = p.b2[j];
    const uint4 *w = reinterpret_cast<const uint4 *>(p.W2 + (size_t)j * kH);   // row j, 8 BF16 per load
    uint4 wv[kH / 8];
#pragma unroll
    for (int c = 0; c < kH / 8; ++c) wv[c] = __ldg(w + c);
#pragma unroll
    for (int c = 0; c < kH / 8; ++c) {
        const __nv_bfloat162 *pr = reinterpret_cast<const __nv_bfloat162 *>(&wv[c]);
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            const float2 f = __bfloat1622float2(pr[e]);
            z2 = fmaf(f.x, h1[8 * c + 2 * e], z2);
            z2 = fmaf(f.y, h1[8 * c + 2 * e + 1], z2);
        }
    }
    float ds2;
    const float h2 = silu(z2, ds2);
    float yv = p.w3[j] * h2;
    dz2[j] = __bfloat162float(__float2bfloat16_rn(p.w3[j] * ds2));
    __syncthreads();
    float dh = 0.0f;
    const uint4 *wt = reinterpret_cast<const uint4 *>(p.W2t + (size_t)j * kH);
#pragma unroll
    for (int c = 0; c < kH / 8; ++c) wv[c] = __ldg(wt + c);
#pragma unroll
    for (int c = 0; c < kH / 8; ++c) {
        const __nv_bfloat162 *pr = reinterpret_cast<const __nv_bfloat162 *>(&wv[c]);
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            const float2 f = __bfloat1622float2(pr[e]);
            dh = fmaf(f.x, dz2[8 * c + 2 * e], dh);
            dh = fmaf(f.y, dz2[8 * c + 2 * e + 1], dh);
        }
    }
    const float g = dh * ds1;
    float q[kIn + 1] = {yv, 0.f, 0.f, 0.f, 0.f};
    for (int i = 0; i < kIn; ++i) q[1 + i] = g * p.W1[j * kIn + i];
    for (int t = 0; t < kIn + 1; ++t)
        for (int o = 16; o > 0; o >>= 1) q[t] += __shfl_xor_sync(0xffffffffu, q[t], o);
    if ((j & 31) == 0)
        for (int t = 0; t < kIn + 1; ++t) red[t][warp] = q[t];
    __syncthreads();
    if (j < kIn + 1) {
        const float s = red[j][0] + red[j][1] + red[j][2] + red[j][3];
        if (j == 0) *V = vscale * (double)(s + p.b3[0]);
        else if (j - 1 < p.D) dV[j - 1] = vscale * (double)s * sc[j - 1];
    }
}

}  // namespace

}  // namespace mtd

// ------------------------------------------------------------------ host object
using namespace mtd;

struct mtd_nnbias {
    int D = 0, device = 0;
    double lo[kIn] = {0, 0, 0, 0}, hi[kIn] = {1, 1, 1, 1};
    double vscale = 1.0;
    cudaStream_t st = nullptr;
    // scratch of the batched hill sum (grown on demand), an event behind its
    // last use (a call on another stream waits for it), and a lock over the wait,
    // the launches and the event (calls of several threads)
    void *d_hs = nullptr;
    size_t cap_hs = 0;
    cudaEvent_t hs_ev = nullptr;
    std::mutex hs_mu;
    std::string err;
    std::vector<double> hills;   // packed, 8 doubles per hill
    double *d_hills = nullptr;
    int nh = 0, cap_h = 0;
    float *d_master = nullptr, *d_mom = nullptr, *d_vel = nullptr;
    float *d_W1 = nullptr, *d_b1 = nullptr, *d_b2 = nullptr, *d_w3 = nullptr, *d_b3 = nullptr;
    __nv_bfloat16 *d_W2 = nullptr, *d_W2t = nullptr;
    float *d_part = nullptr, *d_loss = nullptr;
    int cap_tiles = 0;
    int adam_t = 0;
    int *d_err = nullptr;
    double *d_pt = nullptr, *d_ppart = nullptr, *d_pout = nullptr;
    unsigned int *d_ticket = nullptr;
    float *h_stage = nullptr, *d_stage = nullptr;   // nb_ensure_stage
    size_t cap_hstage = 0, cap_stage = 0;
    static constexpr int kStages = 4;
    cudaEvent_t stage_ev[kStages] = {};   // behind the last copy of each piece of h_stage
    // training pool
    int ntrain = 0;
    float *d_xt = nullptr, *d_tt = nullptr;
    bool validated = false;
    double tol = 1e-3, last_max_err = -1.0;
    unsigned long long seed = 1;
    int wait_tries = kWaitTries;   // limit of the tile kernel's mbarrier waits
    int wait_stall = 0;            // 1: tiles take their timeout path (mtd_nnbias_set_wait)
};

namespace {

std::mutex g_attr_mutex;
bool g_attr_done[64] = {};

mtd_status nb_fail(mtd_nnbias *b, mtd_status s, const std::string &m) {
    if (b) b->err = m;
    return s;
}

#define NB_CU(call, what)                                                                          \
    do {                                                                                           \
        cudaError_t e_ = (call);                                                                   \
        if (e_ != cudaSuccess)                                                                     \
            return nb_fail(b, e_ == cudaErrorMemoryAllocation ? MTD_ERR_OOM : MTD_ERR_CUDA,        \
                           std::string(what) + ": " + cudaGetErrorString(e_));                     \
    } while (0)

MlpDev nb_dev(const mtd_nnbias *b) {
    MlpDev p;
    p.D = b->D;
    p.W1 = b->d_W1;
    p.b1 = b->d_b1;
    p.b2 = b->d_b2;
    p.w3 = b->d_w3;
    p.b3 = b->d_b3;
    p.W2 = b->d_W2;
    p.W2t = b->d_W2t;
    return p;
}

mtd_status nb_tile_attr(mtd_nnbias *b) {
    std::lock_guard<std::mutex> lock(g_attr_mutex);
    if (b->device >= 0 && b->device < 64 && g_attr_done[b->device]) return MTD_OK;
    const auto set = [](auto *k, int bytes) {
        return cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
    };
    NB_CU(set(k_mlp_eval<false, 1>, kEvalSmem), "smem attribute");
    NB_CU(set(k_mlp_eval<true, 1>, kEvalSmem), "smem attribute");
    NB_CU(set(k_mlp_eval<false, 4>, kEvalSmem), "smem attribute");
    NB_CU(set(k_mlp_eval<true, 4>, kEvalSmem), "smem attribute");
    NB_CU(set(k_mlp_train, kTrainSmem), "smem attribute");
    if (b->device >= 0 && b->device < 64) g_attr_done[b->device] = true;
    return MTD_OK;
}

// Staging of mtd_nnbias_loss_grad: device memory for `nin` floats in and `nout`
// out, and pinned memory of kStages pieces that the inputs cross in turn (at
// least `nout`: the results come back whole).  Pinned memory for a whole batch
// grew with the batch, and a first call took 2,000-3,800 us at 30,000 points
// where this takes about 1,000: new pinned memory costs more than the copies.
constexpr size_t kStage = 16384;   // floats, 64 KB
mtd_status nb_ensure_stage(mtd_nnbias *b, size_t nin, size_t nout) {
    const size_t nh = std::max(b->kStages * kStage, nout), nd = (nin + 3) / 4 * 4 + nout;
    if (nh > b->cap_hstage) {
        cudaFreeHost(b->h_stage);
        b->h_stage = nullptr;
        b->cap_hstage = 0;
        NB_CU(cudaMallocHost(&b->h_stage, sizeof(float) * nh), "staging");
        b->cap_hstage = nh;
    }
    if (nd > b->cap_stage) {
        cudaFree(b->d_stage);
        b->d_stage = nullptr;
        b->cap_stage = 0;
        NB_CU(cudaMalloc(&b->d_stage, sizeof(float) * nd), "staging");
        b->cap_stage = nd;
    }
    return MTD_OK;
}

// n doubles of the caller to the device through the pieces of h_stage; `used`
// counts those of this call so far.
mtd_status nb_stage_in(mtd_nnbias *b, float *dst, const double *src, size_t n, int &used) {
    constexpr size_t kPiece = kStage / 2;
    for (size_t at = 0; at < n; at += kPiece, ++used) {
        const size_t m = std::min(kPiece, n - at);
        const int q = used % b->kStages;
        if (used >= b->kStages) NB_CU(cudaEventSynchronize(b->stage_ev[q]), "staging");
        std::memcpy(b->h_stage + q * kStage, src + at, sizeof(double) * m);
        NB_CU(cudaMemcpyAsync(dst + 2 * at, b->h_stage + q * kStage, sizeof(double) * m, cudaMemcpyHostToDevice,
                              b->st), "points");
        NB_CU(cudaEventRecord(b->stage_ev[q], b->st), "staging");
    }
    return MTD_OK;
}

mtd_status nb_ensure_tiles(mtd_nnbias *b, int ntiles) {
    if (ntiles <= b->cap_tiles) return MTD_OK;
    if (b->d_part) cudaFree(b->d_part);
    if (b->d_loss) cudaFree(b->d_loss);
    b->d_part = nullptr;
    b->d_loss = nullptr;
    NB_CU(cudaMalloc(&b->d_part, sizeof(float) * (size_t)kNPpad * ntiles), "gradient partials");
    NB_CU(cudaMalloc(&b->d_loss, sizeof(float) * (size_t)ntiles), "loss partials");
    b->cap_tiles = ntiles;
    return MTD_OK;
}

void nb_normalise(const mtd_nnbias *b, const double *s, float *u) {
    for (int i = 0; i < kIn; ++i)
        u[i] = i < b->D ? (float)(2.0 * (s[i] - b->lo[i]) / (b->hi[i] - b->lo[i]) - 1.0) : 0.0f;
}

mtd_status nb_refresh_forward(mtd_nnbias *b) {
    k_mlp_adam<<<kSumBlocks, 256, 0, b->st>>>(0, b->d_part, b->d_master, b->d_mom, b->d_vel, 0.f, 1.f, 1.f,
                                                     b->d_W1, b->d_b1, b->d_W2, b->d_W2t, b->d_b2, b->d_w3,
                                                     b->d_b3, 0);
    NB_CU(cudaGetLastError(), "forward copies");
    return MTD_OK;
}

// The batched hill sum with the object's scratch.  During a stream capture it runs
// without any: the scratch may have grown, and so moved, by the time the graph
// runs, and memory nodes would keep the graph from being cloned, nested or
// instantiated twice.
cudaError_t nb_hillsum(mtd_nnbias *b, int npts, const double *pts, int ps, double *V, double *dV, int gs,
                       cudaStream_t st) {
    cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
    cudaError_t e = cudaStreamIsCapturing(st, &cap);
    if (e != cudaSuccess) return e;
    const size_t need = cap == cudaStreamCaptureStatusNone ? hillsum_scratch(npts, b->nh) : 0;
    if (need == 0) return hillsum_batch(b->D, b->lo, b->hi, npts, pts, ps, b->nh, b->d_hills, V, dV, gs, nullptr, st);
    std::lock_guard<std::mutex> lock(b->hs_mu);
    if (need > b->cap_hs) {
        // another thread's capture on another stream is no reason to refuse these
        cudaStreamCaptureMode mode = cudaStreamCaptureModeRelaxed;
        if ((e = cudaThreadExchangeStreamCaptureMode(&mode)) != cudaSuccess) return e;
        e = cudaEventSynchronize(b->hs_ev);
        if (e == cudaSuccess) {
            cudaFree(b->d_hs);
            b->d_hs = nullptr;
            b->cap_hs = 0;
            e = cudaMalloc(&b->d_hs, need + need / 4);
            if (e == cudaSuccess) b->cap_hs = need + need / 4;
        }
        cudaThreadExchangeStreamCaptureMode(&mode);
        if (e != cudaSuccess) return e;
    } else if ((e = cudaStreamWaitEvent(st, b->hs_ev, 0)) != cudaSuccess) {
        return e;
    }
    e = hillsum_batch(b->D, b->lo, b->hi, npts, pts, ps, b->nh, b->d_hills, V, dV, gs, b->d_hs, st);
    const cudaError_t er = cudaEventRecord(b->hs_ev, st);
    return e != cudaSuccess ? e : er;
}

// Exact FP64 V (and dV) at host points, computed on the device.
mtd_status nb_exact_host(mtd_nnbias *b, int npts, const double *pts, double *V, double *dV) {
    if (npts <= 0) return MTD_OK;
    std::vector<double> p4((size_t)npts * kIn, 0.0);
    for (int i = 0; i < npts; ++i)
        for (int k = 0; k < b->D; ++k) p4[(size_t)i * kIn + k] = pts[(size_t)i * b->D + k];
    double *d_p = nullptr, *d_V = nullptr, *d_dV = nullptr;
    NB_CU(cudaMalloc(&d_p, sizeof(double) * p4.size()), "points");
    NB_CU(cudaMalloc(&d_V, sizeof(double) * npts), "values");
    NB_CU(cudaMalloc(&d_dV, sizeof(double) * (size_t)npts * kIn), "gradients");
    cudaMemcpyAsync(d_p, p4.data(), sizeof(double) * p4.size(), cudaMemcpyHostToDevice, b->st);
    const cudaError_t el = nb_hillsum(b, npts, d_p, kIn, d_V, d_dV, kIn, b->st);
    std::vector<double> g((size_t)npts * kIn);
    cudaMemcpyAsync(V, d_V, sizeof(double) * npts, cudaMemcpyDeviceToHost, b->st);
    cudaMemcpyAsync(g.data(), d_dV, sizeof(double) * g.size(), cudaMemcpyDeviceToHost, b->st);
    const cudaError_t es = cudaStreamSynchronize(b->st), e = el != cudaSuccess ? el : es;
    cudaFree(d_p);
    cudaFree(d_V);
    cudaFree(d_dV);
    NB_CU(e, "exact hill sum");
    if (dV)
        for (int i = 0; i < npts; ++i)
            for (int k = 0; k < b->D; ++k) dV[(size_t)i * b->D + k] = g[(size_t)i * kIn + k];
    return MTD_OK;
}

// Points for training / validation: half near hill centres (N(0, 1.5 sigma)),
// half uniform in the CV box.
void nb_sample(const mtd_nnbias *b, int npts, unsigned long long seed, std::vector<double> &out) {
    std::mt19937_64 g(seed);
    std::uniform_real_distribution<double> U(0.0, 1.0);
    std::normal_distribution<double> N(0.0, 1.0);
    out.assign((size_t)npts * b->D, 0.0);
    for (int i = 0; i < npts; ++i) {
        const bool near = b->nh > 0 && (i & 1);
        const int h = near ? (int)(U(g) * b->nh) % b->nh : 0;
        for (int k = 0; k < b->D; ++k) {
            double v;
            if (near) {
                const double sig = std::sqrt(1.0 / b->hills[(size_t)h * 8 + 6]);
                v = b->hills[(size_t)h * 8 + k] + 1.5 * sig * N(g);
            } else {
                v = b->lo[k] + (b->hi[k] - b->lo[k]) * U(g);
            }
            out[(size_t)i * b->D + k] = std::min(b->hi[k], std::max(b->lo[k], v));
        }
    }
}

// A tile per block while every tile has an SM to itself (14.4 us, 16.5 with a
// tile per warpgroup), beyond that a tile per warpgroup (200 tiles: 20.7 us
// against 22.6 with two rounds of blocks; 1,184 tiles: 53 against 66).
void nb_launch_eval(const mtd_nnbias *b, int npts, const MlpIo &io, bool grad, cudaStream_t st) {
    const int ntiles = (npts + kH - 1) / kH;
    const bool whole = ntiles <= 148;
    const int grid = std::min(ntiles, 148);
    const auto k = whole ? (grad ? k_mlp_eval<true, 4> : k_mlp_eval<false, 4>)
                         : (grad ? k_mlp_eval<true, 1> : k_mlp_eval<false, 1>);
    k<<<grid, 512, kEvalSmem, st>>>(nb_dev(b), npts, io, b->d_err, b->wait_tries, b->wait_stall);
}

mtd_status nb_forward_batch(mtd_nnbias *b, int npts, const float *d_x, float *d_y, float *d_ds) {
    mtd_status s = nb_tile_attr(b);
    if (s != MTD_OK) return s;
    MlpIo io{};
    io.x = d_x;
    io.y = d_y;
    io.ds = d_ds;
    nb_launch_eval(b, npts, io, d_ds != nullptr, b->st);
    NB_CU(cudaGetLastError(), "MLP forward");
    return MTD_OK;
}

// Reads and clears the tile kernels' timeout flag.
mtd_status nb_check_err(mtd_nnbias *b) {
    int h = 0;
    NB_CU(cudaMemcpyAsync(&h, b->d_err, sizeof(int), cudaMemcpyDeviceToHost, b->st), "status");
    NB_CU(cudaStreamSynchronize(b->st), "sync");
    if (h) {
        NB_CU(cudaMemsetAsync(b->d_err, 0, sizeof(int), b->st), "status");
        return nb_fail(b, MTD_ERR_TIMEOUT, "tensor-core wait ran out of tries");
    }
    return MTD_OK;
}

}  // namespace

extern "C" {

mtd_status mtd_nnbias_create(int D, const double *lo, const double *hi, unsigned long long seed, mtd_nnbias **out) {
    if (!out) return MTD_ERR_INVALID_ARG;
    *out = nullptr;
    mtd_nnbias *b = new mtd_nnbias();
    *out = b;
    if (D < 1 || D > kIn || !lo || !hi) return nb_fail(b, MTD_ERR_INVALID_ARG, "D must be in [1, 4] with lo, hi");
    b->D = D;
    for (int k = 0; k < D; ++k) {
        if (!(hi[k] > lo[k])) return nb_fail(b, MTD_ERR_INVALID_ARG, "hi must exceed lo in every dimension");
        b->lo[k] = lo[k];
        b->hi[k] = hi[k];
    }
    b->seed = seed;
    NB_CU(cudaGetDevice(&b->device), "device");
    NB_CU(cudaStreamCreateWithFlags(&b->st, cudaStreamNonBlocking), "stream");
    NB_CU(cudaEventCreateWithFlags(&b->hs_ev, cudaEventDisableTiming), "event");
    for (cudaEvent_t &ev : b->stage_ev) NB_CU(cudaEventCreateWithFlags(&ev, cudaEventDisableTiming), "event");
    NB_CU(cudaMalloc(&b->d_master, sizeof(float) * kNPpad), "params");
    NB_CU(cudaMalloc(&b->d_mom, sizeof(float) * kNPpad), "params");
    NB_CU(cudaMalloc(&b->d_vel, sizeof(float) * kNPpad), "params");
    NB_CU(cudaMalloc(&b->d_W1, sizeof(float) * kH * kIn), "params");
    NB_CU(cudaMalloc(&b->d_b1, sizeof(float) * kH), "params");
    NB_CU(cudaMalloc(&b->d_b2, sizeof(float) * kH), "params");
    NB_CU(cudaMalloc(&b->d_w3, sizeof(float) * kH), "params");
    NB_CU(cudaMalloc(&b->d_b3, sizeof(float) * 4), "params");
    NB_CU(cudaMalloc(&b->d_W2, sizeof(__nv_bfloat16) * kH * kH), "params");
    NB_CU(cudaMalloc(&b->d_W2t, sizeof(__nv_bfloat16) * kH * kH), "params");
    NB_CU(cudaMalloc(&b->d_err, sizeof(int)), "status");
    NB_CU(cudaMalloc(&b->d_pt, sizeof(double) * 8), "point");
    NB_CU(cudaMalloc(&b->d_pout, sizeof(double) * 8), "point");
    NB_CU(cudaMalloc(&b->d_ppart, sizeof(double) * 5 * kPointBlocks), "point partials");
    NB_CU(cudaMalloc(&b->d_ticket, sizeof(unsigned int)), "ticket");
    cudaMemsetAsync(b->d_err, 0, sizeof(int), b->st);
    cudaMemsetAsync(b->d_ticket, 0, sizeof(unsigned int), b->st);
    // He-style initialisation of the masters, zero biases
    std::vector<float> w(kNPpad, 0.0f);
    std::mt19937_64 g(seed);
    std::normal_distribution<double> N(0.0, 1.0);
    for (int j = 0; j < kH; ++j)
        for (int i = 0; i < kIn; ++i) w[oW1 + j * kIn + i] = i < D ? (float)(N(g) * std::sqrt(2.0 / D)) : 0.0f;
    for (int q = 0; q < kH * kH; ++q) w[oW2 + q] = (float)(N(g) * std::sqrt(2.0 / kH));
    for (int q = 0; q < kH; ++q) w[ow3 + q] = (float)(N(g) * std::sqrt(1.0 / kH));
    NB_CU(cudaMemcpyAsync(b->d_master, w.data(), sizeof(float) * kNPpad, cudaMemcpyHostToDevice, b->st), "init");
    cudaMemsetAsync(b->d_mom, 0, sizeof(float) * kNPpad, b->st);
    cudaMemsetAsync(b->d_vel, 0, sizeof(float) * kNPpad, b->st);
    mtd_status s = nb_refresh_forward(b);
    if (s != MTD_OK) return s;
    NB_CU(cudaStreamSynchronize(b->st), "init");
    return MTD_OK;
}

void mtd_nnbias_destroy(mtd_nnbias *b) {
    if (!b) return;
    if (b->st) cudaStreamSynchronize(b->st);
    void *ptrs[] = {b->d_hills, b->d_master, b->d_mom, b->d_vel, b->d_W1, b->d_b1, b->d_b2, b->d_w3, b->d_b3,
                    b->d_W2, b->d_W2t, b->d_part, b->d_loss, b->d_err, b->d_pt, b->d_pout, b->d_ppart,
                    b->d_ticket, b->d_xt, b->d_tt, b->d_hs, b->d_stage};
    for (void *p : ptrs)
        if (p) cudaFree(p);
    if (b->h_stage) cudaFreeHost(b->h_stage);
    for (cudaEvent_t ev : b->stage_ev)
        if (ev) cudaEventDestroy(ev);
    if (b->hs_ev) cudaEventDestroy(b->hs_ev);
    if (b->st) cudaStreamDestroy(b->st);
    delete b;
}

const char *mtd_nnbias_last_error(const mtd_nnbias *b) { return b ? b->err.c_str() : "null object"; }

mtd_status mtd_nnbias_add_hills(mtd_nnbias *b, int n, const double *centers, const double *heights,
                                const double *sigmas) {
    if (!b || n < 0 || (n > 0 && (!centers || !heights || !sigmas))) return MTD_ERR_INVALID_ARG;
    for (int h = 0; h < n; ++h) {
        if (!(sigmas[h] > 0)) return nb_fail(b, MTD_ERR_INVALID_ARG, "hill widths must be positive");
        const double s2 = sigmas[h] * sigmas[h];
        double rec[8] = {0, 0, 0, 0, heights[h], 0.5 / s2, 1.0 / s2, 2.0 * kExpCut * s2};
        for (int k = 0; k < b->D; ++k) rec[k] = centers[(size_t)h * b->D + k];
        b->hills.insert(b->hills.end(), rec, rec + 8);
    }
    const int nh = (int)(b->hills.size() / 8);
    if (nh > b->cap_h) {
        if (b->d_hills) cudaFree(b->d_hills);
        b->d_hills = nullptr;
        const int cap = nh + nh / 2 + 64;
        NB_CU(cudaMalloc(&b->d_hills, sizeof(double) * 8 * (size_t)cap), "hills");
        b->cap_h = cap;
        NB_CU(cudaMemcpyAsync(b->d_hills, b->hills.data(), sizeof(double) * b->hills.size(), cudaMemcpyHostToDevice,
                              b->st),
              "hills");
    } else if (n > 0) {
        NB_CU(cudaMemcpyAsync(b->d_hills + (size_t)b->nh * 8, b->hills.data() + (size_t)b->nh * 8,
                              sizeof(double) * 8 * (size_t)n, cudaMemcpyHostToDevice, b->st),
              "hills");
    }
    b->nh = nh;
    b->validated = false;
    NB_CU(cudaStreamSynchronize(b->st), "hills");
    return MTD_OK;
}

int mtd_nnbias_num_hills(const mtd_nnbias *b) { return b ? b->nh : 0; }

mtd_status mtd_nnbias_exact(mtd_nnbias *b, int npts, const double *pts, double *V, double *dV) {
    if (!b || npts < 0 || (npts > 0 && (!pts || !V))) return MTD_ERR_INVALID_ARG;
    return nb_exact_host(b, npts, pts, V, dV);
}

mtd_status mtd_nnbias_eval(mtd_nnbias *b, int npts, const double *pts, double *V, double *dV) {
    if (!b || npts < 0 || (npts > 0 && (!pts || !V))) return MTD_ERR_INVALID_ARG;
    if (npts == 0) return MTD_OK;
    std::vector<float> x((size_t)npts * kIn);
    for (int i = 0; i < npts; ++i) nb_normalise(b, pts + (size_t)i * b->D, x.data() + (size_t)i * kIn);
    float *d_x = nullptr, *d_y = nullptr, *d_ds = nullptr;
    NB_CU(cudaMalloc(&d_x, sizeof(float) * x.size()), "points");
    NB_CU(cudaMalloc(&d_y, sizeof(float) * npts), "values");
    NB_CU(cudaMalloc(&d_ds, sizeof(float) * x.size()), "gradients");
    cudaMemcpyAsync(d_x, x.data(), sizeof(float) * x.size(), cudaMemcpyHostToDevice, b->st);
    mtd_status s = nb_forward_batch(b, npts, d_x, d_y, dV ? d_ds : nullptr);
    std::vector<float> y(npts), g(x.size());
    if (s == MTD_OK) {
        cudaMemcpyAsync(y.data(), d_y, sizeof(float) * npts, cudaMemcpyDeviceToHost, b->st);
        if (dV) cudaMemcpyAsync(g.data(), d_ds, sizeof(float) * g.size(), cudaMemcpyDeviceToHost, b->st);
        s = nb_check_err(b);
    }
    cudaFree(d_x);
    cudaFree(d_y);
    cudaFree(d_ds);
    if (s != MTD_OK) return s;
    for (int i = 0; i < npts; ++i) {
        V[i] = b->vscale * (double)y[i];
        if (dV)
            for (int k = 0; k < b->D; ++k)
                dV[(size_t)i * b->D + k] = b->vscale * (double)g[(size_t)i * kIn + k] * 2.0 / (b->hi[k] - b->lo[k]);
    }
    return MTD_OK;
}

// One gradient of the MSE loss on given points and targets (no update): for
// checks against an independent implementation.  grad in the flat layout
// W1[128][4], b1, W2[128][128], b2, w3, b3 (17,281 values).
mtd_status mtd_nnbias_loss_grad(mtd_nnbias *b, int npts, const double *pts, const double *targets, double vscale,
                                float *grad, double *loss) {
    if (!b || npts <= 0 || !pts || !targets || !grad || !(vscale > 0)) return MTD_ERR_INVALID_ARG;
    const int ntiles = (npts + kH - 1) / kH;
    mtd_status s = nb_ensure_tiles(b, ntiles);
    if (s != MTD_OK) return s;
    s = nb_tile_attr(b);
    if (s != MTD_OK) return s;
    // points and targets go over as they are, through pinned memory in pieces
    // (the divisions of their normalisation took the host 40 us at 8,192
    // points), and the results come back in one copy
    const size_t np = (size_t)npts * b->D, nin = 2 * (np + npts), nout = (size_t)kNPpad + 1 + ntiles;
    s = nb_ensure_stage(b, nin, nout);
    if (s != MTD_OK) return s;
    int used = 0;
    s = nb_stage_in(b, b->d_stage, pts, np, used);
    if (s == MTD_OK) s = nb_stage_in(b, b->d_stage + 2 * np, targets, npts, used);
    if (s != MTD_OK) return s;
    float *d_g = b->d_stage + (nin + 3) / 4 * 4;
    MlpBatch in{};
    in.pts = reinterpret_cast<const double *>(b->d_stage);
    in.tgt = in.pts + np;
    in.vscale = vscale;
    for (int k = 0; k < b->D; ++k) {
        in.lo[k] = b->lo[k];
        in.span[k] = b->hi[k] - b->lo[k];
    }
    k_mlp_train<<<ntiles, 512, kTrainSmem, b->st>>>(nb_dev(b), npts, in, b->d_part, b->d_loss, 2.0f / npts, b->d_err,
                                                    b->wait_tries, b->wait_stall);
    k_mlp_gradsum<<<kSumBlocks, 256, 0, b->st>>>(ntiles, b->d_part, b->d_loss, b->d_err, d_g);
    NB_CU(cudaGetLastError(), "gradient");
    NB_CU(cudaMemcpyAsync(b->h_stage, d_g, sizeof(float) * nout, cudaMemcpyDeviceToHost, b->st), "gradient");
    NB_CU(cudaStreamSynchronize(b->st), "gradient");
    int timeout;
    std::memcpy(&timeout, b->h_stage + kNPpad, sizeof timeout);
    if (timeout) return nb_check_err(b);   // clears the flag
    std::memcpy(grad, b->h_stage, sizeof(float) * kNP);
    if (loss) {
        double l = 0.0;
        for (int v = 0; v < ntiles; ++v) l += b->h_stage[kNPpad + 1 + v];
        *loss = l / npts;
    }
    return MTD_OK;
}

mtd_status mtd_nnbias_get_params(mtd_nnbias *b, float *out) {
    if (!b || !out) return MTD_ERR_INVALID_ARG;
    NB_CU(cudaMemcpyAsync(out, b->d_master, sizeof(float) * kNP, cudaMemcpyDeviceToHost, b->st), "params");
    NB_CU(cudaStreamSynchronize(b->st), "params");
    return MTD_OK;
}

mtd_status mtd_nnbias_set_params(mtd_nnbias *b, const float *in, double vscale) {
    if (!b || !in || !(vscale > 0)) return MTD_ERR_INVALID_ARG;
    NB_CU(cudaMemcpyAsync(b->d_master, in, sizeof(float) * kNP, cudaMemcpyHostToDevice, b->st), "params");
    b->vscale = vscale;
    mtd_status s = nb_refresh_forward(b);
    if (s != MTD_OK) return s;
    NB_CU(cudaStreamSynchronize(b->st), "params");
    return MTD_OK;
}

double mtd_nnbias_vscale(const mtd_nnbias *b) { return b ? b->vscale : 0.0; }

// Fits the network to the hill sum: a pool of ntrain sampled points with
// exact FP64 targets, `iters` Adam steps on minibatches of `batch` points.
mtd_status mtd_nnbias_fit(mtd_nnbias *b, int ntrain, int iters, int batch, double lr, unsigned long long seed,
                          double *final_loss) {
    if (!b || ntrain < kH || iters < 0 || batch < kH || batch > ntrain || !(lr > 0)) return MTD_ERR_INVALID_ARG;
    if (b->nh == 0) return nb_fail(b, MTD_ERR_INVALID_ARG, "no hills to fit");
    std::vector<double> pts;
    nb_sample(b, ntrain, seed, pts);
    std::vector<double> V(ntrain);
    mtd_status s = nb_exact_host(b, ntrain, pts.data(), V.data(), nullptr);
    if (s != MTD_OK) return s;
    double vmax = 0.0;
    for (double v : V) vmax = std::max(vmax, std::fabs(v));
    const bool rescale = b->adam_t == 0 || vmax > 1.25 * b->vscale || vmax < 0.5 * b->vscale;
    if (rescale && vmax > 0) {   // output scale: refresh the last layer's scale with the data
        const double old = b->vscale;
        b->vscale = vmax;
        if (b->adam_t > 0 && old > 0) {
            std::vector<float> w(kNP);
            s = mtd_nnbias_get_params(b, w.data());
            if (s != MTD_OK) return s;
            const float f = (float)(old / vmax);
            for (int q = ow3; q < kNP; ++q) w[q] *= f;
            s = mtd_nnbias_set_params(b, w.data(), vmax);
            if (s != MTD_OK) return s;
        }
    }
    std::vector<float> x((size_t)ntrain * kIn), t(ntrain);
    for (int i = 0; i < ntrain; ++i) {
        nb_normalise(b, pts.data() + (size_t)i * b->D, x.data() + (size_t)i * kIn);
        t[i] = (float)(V[i] / b->vscale);
    }
    if (b->d_xt) cudaFree(b->d_xt);
    if (b->d_tt) cudaFree(b->d_tt);
    b->d_xt = nullptr;
    b->d_tt = nullptr;
    NB_CU(cudaMalloc(&b->d_xt, sizeof(float) * x.size()), "training points");
    NB_CU(cudaMalloc(&b->d_tt, sizeof(float) * ntrain), "training targets");
    cudaMemcpyAsync(b->d_xt, x.data(), sizeof(float) * x.size(), cudaMemcpyHostToDevice, b->st);
    cudaMemcpyAsync(b->d_tt, t.data(), sizeof(float) * ntrain, cudaMemcpyHostToDevice, b->st);
    b->ntrain = ntrain;
    const int ntiles = (batch + kH - 1) / kH;
    s = nb_ensure_tiles(b, ntiles);
    if (s != MTD_OK) return s;
    s = nb_tile_attr(b);
    if (s != MTD_OK) return s;
    const int nbatches = ntrain / batch;
    for (int it = 0; it < iters; ++it) {
        const int bi = it % nbatches;
        const int nb = batch;
        ++b->adam_t;
        const float b1c = 1.0f - std::pow(0.9f, (float)b->adam_t), b2c = 1.0f - std::pow(0.999f, (float)b->adam_t);
        const float lr_t = (float)(lr * (it < iters / 2 ? 1.0 : 0.5 * (1.0 + std::cos(M_PI * (it - iters / 2) /
                                                                                   std::max(1, iters - iters / 2)))));
        MlpBatch in{};
        in.x = b->d_xt + (size_t)bi * batch * kIn;
        in.t = b->d_tt + (size_t)bi * batch;
        k_mlp_train<<<ntiles, 512, kTrainSmem, b->st>>>(nb_dev(b), nb, in, b->d_part, b->d_loss, 2.0f / nb, b->d_err,
                                                        b->wait_tries, b->wait_stall);
        k_mlp_adam<<<kSumBlocks, 256, 0, b->st>>>(ntiles, b->d_part, b->d_master, b->d_mom, b->d_vel,
                                                         std::max(lr_t, (float)(lr * 0.02)), b1c, b2c, b->d_W1,
                                                         b->d_b1, b->d_W2, b->d_W2t, b->d_b2, b->d_w3, b->d_b3, 1);
    }
    NB_CU(cudaGetLastError(), "training");
    std::vector<float> lp(ntiles);
    cudaMemcpyAsync(lp.data(), b->d_loss, sizeof(float) * ntiles, cudaMemcpyDeviceToHost, b->st);
    s = nb_check_err(b);
    if (s != MTD_OK) return s;
    if (final_loss) {
        double l = 0.0;
        for (float v : lp) l += v;
        *final_loss = l / batch * b->vscale * b->vscale;
    }
    b->validated = false;
    return MTD_OK;
}

// Max and RMS of |V_theta - V_exact| on npts sampled points (the measure of the
// network's error); marks the network usable when max <= tol.
mtd_status mtd_nnbias_validate(mtd_nnbias *b, int npts, unsigned long long seed, double tol, double *max_err,
                               double *rms_err) {
    if (!b || npts <= 0) return MTD_ERR_INVALID_ARG;
    std::vector<double> pts;
    nb_sample(b, npts, seed, pts);
    std::vector<double> Ve(npts), Vn(npts);
    mtd_status s = nb_exact_host(b, npts, pts.data(), Ve.data(), nullptr);
    if (s != MTD_OK) return s;
    s = mtd_nnbias_eval(b, npts, pts.data(), Vn.data(), nullptr);
    if (s != MTD_OK) return s;
    double mx = 0.0, ss = 0.0;
    for (int i = 0; i < npts; ++i) {
        const double d = std::fabs(Vn[i] - Ve[i]);
        mx = std::max(mx, d);
        ss += d * d;
    }
    if (max_err) *max_err = mx;
    if (rms_err) *rms_err = std::sqrt(ss / npts);
    b->tol = tol;
    b->last_max_err = mx;
    b->validated = mx <= tol;
    return MTD_OK;
}

int mtd_nnbias_usable(const mtd_nnbias *b) { return b && b->validated ? 1 : 0; }

// Bias at one device-resident point (D doubles) into d_V (1) and d_dV (D),
// enqueued on `stream`: use_nn = 1 the network, 0 the exact hill sum,
// -1 the network when the last validation passed, else the exact sum.
mtd_status mtd_nnbias_eval_device(mtd_nnbias *b, int npts, const double *d_pts, double *d_V, double *d_dV,
                                  int use_nn, void *stream) {
    if (!b || npts < 0 || (npts > 0 && (!d_pts || !d_V))) return MTD_ERR_INVALID_ARG;
    if (npts == 0) return MTD_OK;
    cudaStream_t st = stream ? static_cast<cudaStream_t>(stream) : b->st;
    const bool nn = use_nn > 0 || (use_nn < 0 && b->validated);
    if (!nn) {
        if (b->nh == 0) {
            NB_CU(cudaMemsetAsync(d_V, 0, sizeof(double) * npts, st), "bias");
            if (d_dV) NB_CU(cudaMemsetAsync(d_dV, 0, sizeof(double) * npts * b->D, st), "bias");
            return MTD_OK;
        }
        NB_CU(nb_hillsum(b, npts, d_pts, b->D, d_V, d_dV, b->D, st), "exact hill sum");
        return MTD_OK;
    }
    mtd_status s = nb_tile_attr(b);
    if (s != MTD_OK) return s;
    MlpIo io{};
    io.pts = d_pts;
    io.V = d_V;
    io.dV = d_dV;
    io.vscale = b->vscale;
    for (int k = 0; k < b->D; ++k) {
        io.lo[k] = b->lo[k];
        io.sc[k] = 2.0 / (b->hi[k] - b->lo[k]);
    }
    nb_launch_eval(b, npts, io, d_dV != nullptr, st);
    NB_CU(cudaGetLastError(), "network");
    return MTD_OK;
}

mtd_status mtd_nnbias_sync(mtd_nnbias *b) {
    if (!b) return MTD_ERR_INVALID_ARG;
    return nb_check_err(b);
}

mtd_status mtd_nnbias_set_wait(mtd_nnbias *b, int tries, int stall) {
    if (!b || tries < 0) return MTD_ERR_INVALID_ARG;
    b->wait_tries = tries > 0 ? tries : kWaitTries;
    b->wait_stall = stall ? 1 : 0;
    return MTD_OK;
}

mtd_status mtd_nnbias_point_device(mtd_nnbias *b, const double *d_s, double *d_V, double *d_dV, int use_nn,
                                   void *stream) {
    if (!b || !d_s || !d_V || !d_dV) return MTD_ERR_INVALID_ARG;
    cudaStream_t st = stream ? static_cast<cudaStream_t>(stream) : b->st;
    const bool nn = use_nn > 0 || (use_nn < 0 && b->validated);
    if (nn) {
        double sc[kIn];
        for (int k = 0; k < kIn; ++k) sc[k] = 2.0 / (b->hi[k] - b->lo[k]);
        k_mlp_point<<<1, 128, 0, st>>>(nb_dev(b), d_s, b->lo[0], b->lo[1], b->lo[2], b->lo[3], sc[0], sc[1], sc[2],
                                       sc[3], b->vscale, d_V, d_dV);
    } else {
        if (b->nh == 0) {
            NB_CU(cudaMemsetAsync(d_V, 0, sizeof(double), st), "bias");
            NB_CU(cudaMemsetAsync(d_dV, 0, sizeof(double) * b->D, st), "bias");
            return MTD_OK;
        }
        k_hillsum_point<<<kPointBlocks, 256, 0, st>>>(b->D, d_s, 0, b->nh, b->d_hills, b->d_ppart, b->d_ticket, d_V,
                                                      d_dV, 0);
    }
    NB_CU(cudaGetLastError(), "bias at a point");
    return MTD_OK;
}

}  // extern "C"

namespace mtd {

mtd_status nnbias_enqueue_vdv(mtd_nnbias *b, const double *d_s, double *d_vdv, bool nn, int h_from,
                              cudaStream_t st) {
    double *d_V = d_vdv, *d_dV = d_vdv + 1;
    int h0 = 0;
    if (nn) {
        double sc[kIn];
        for (int k = 0; k < kIn; ++k) sc[k] = 2.0 / (b->hi[k] - b->lo[k]);
        k_mlp_point<<<1, 128, 0, st>>>(nb_dev(b), d_s, b->lo[0], b->lo[1], b->lo[2], b->lo[3], sc[0], sc[1], sc[2],
                                       sc[3], b->vscale, d_V, d_dV);
        h0 = std::max(0, std::min(h_from, b->nh));
    } else if (b->nh == 0 || h_from >= b->nh) {
        NB_CU(cudaMemsetAsync(d_vdv, 0, sizeof(double) * (1 + b->D), st), "bias");
    }
    if (h0 < b->nh)
        k_hillsum_point<<<kPointBlocks, 256, 0, st>>>(b->D, d_s, h0, b->nh, b->d_hills, b->d_ppart, b->d_ticket, d_V,
                                                      d_dV, nn ? 1 : 0);
    NB_CU(cudaGetLastError(), "bias at the CV point");
    return MTD_OK;
}

}  // namespace mtd
