// Training and batch inference of the warm-start MLP (see mlp.cuh) with
// hand-written BF16 tensor-core kernels (mma.sync m16n8k16, FP32 accumulate).
//
//   k_mlp_forward   rows -> 3 outputs; each warp runs 16-row tiles.
//   k_mlp_train     up to TRAIN_STEPS Adam steps (or one gradient) in one
//                   cooperative launch.
//
// A step of a minibatch: a CTA (16 warps) takes tiles of 64 rows.  Warp
// (rg, ng) owns rows 16 rg .. + 15 and columns 16 ng .. + 15 of every layer, in
// the forward pass, the delta recursion and (as row and column of the weight)
// the weight gradients delta^T h, which stay in its registers over the CTA's
// tiles; activations and deltas pass through shared memory, read as ldmatrix
// fragments from rows of 144 bytes (no bank conflicts).  GELU' stays in the
// registers of the thread that uses it again.  Biases and W4's gradient are
// small and use SIMT sums.  The CTAs' partial gradients are summed in a fixed
// order, so the gradient is deterministic, and the sum of a parameter, its Adam
// update and its BF16 copy are one thread's; two grid barriers a step.
//
// A minibatch of 4,096 is 64 tiles, so a step is bound by latency: its layers'
// dependent chain, the partial sums' trips through L2 and the barriers.
// 12.5 us a step of 4,096 rows, against 52 us as three kernels and a copy of
// the loss (64-row tiles on 4 warps, weights converted from FP32 by every CTA,
// fragments read as 2-byte words); 32 steps with their two permutations 2,130
// -> 640 us.
// Loss: mean over rows of the squared error summed over the 3 outputs.
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstring>
#include <random>
#include <vector>

#include "../../include/phybs.h"
#include "exchange.cuh"
#include "mlp.cuh"

namespace pbs {
namespace mlp {

constexpr int TILE = 64;           // rows per CTA tile
constexpr int TRAIN_THREADS = 512;
constexpr int TRAIN_STEPS = 64;    // steps of a launch (their Adam constants are kernel parameters)
constexpr int NPART = NPARAM + 1;  // partial gradient + loss
constexpr int LDX = 40, LDH = 72;  // shared-memory row strides (BF16) of 32- and 64-wide rows

__global__ void __launch_bounds__(128) k_mlp_forward(const float *theta, const float *X, int rows, float *Y) {
    __shared__ SmemWeights s;
    stage_weights(theta, s);
    __syncthreads();
    const int lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
    const int warps = blockDim.x >> 5, wid = blockIdx.x * warps + (threadIdx.x >> 5);
    const int nwarps = gridDim.x * warps;
    for (int row0 = wid * 16; row0 < rows; row0 += nwarps * 16) {
        uint32_t x[2][4];
        input_frags(X, row0, rows, x);
        float out[4];
        forward_tile(s, x, out);
#pragma unroll
        for (int e = 0; e < 2; ++e) {
            const int col = 2 * t + e;
            if (col < OUT) {
                if (row0 + g < rows) Y[(size_t)(row0 + g) * OUT + col] = out[e];
                if (row0 + g + 8 < rows) Y[(size_t)(row0 + g + 8) * OUT + col] = out[2 + e];
            }
        }
    }
}

// The weights as a step stages them: BF16 rows at the shared-memory strides
// (the padding zero), FP32 biases.  Written by the Adam update beside the FP32
// masters, so that staging is a plain copy.
struct alignas(16) TrainImage {
    __nv_bfloat16 w1[HID * LDX];
    __nv_bfloat16 w2[HID * LDH], w3[HID * LDH];
    __nv_bfloat16 w4[NOUT * LDH];
    float b1[HID], b2[HID], b3[HID], b4[NOUT];
};
static_assert(sizeof(TrainImage) % 16 == 0, "copied in 16-byte words");

__device__ __forceinline__ void put_param(TrainImage *im, int i, float v) {
    const __nv_bfloat16 b = __float2bfloat16_rn(v);
    if (i < OFF_B1) im->w1[i / IN * LDX + i % IN] = b;
    else if (i < OFF_W2) im->b1[i - OFF_B1] = v;
    else if (i < OFF_B2) im->w2[(i - OFF_W2) / HID * LDH + (i - OFF_W2) % HID] = b;
    else if (i < OFF_W3) im->b2[i - OFF_B2] = v;
    else if (i < OFF_B3) im->w3[(i - OFF_W3) / HID * LDH + (i - OFF_W3) % HID] = b;
    else if (i < OFF_W4) im->b3[i - OFF_B3] = v;
    else if (i < OFF_B4) im->w4[(i - OFF_W4) / HID * LDH + (i - OFF_W4) % HID] = b;
    else im->b4[i - OFF_B4] = v;
}

struct TrainSmem {
    TrainImage w;
    __nv_bfloat16 xs[TILE * LDX];
    __nv_bfloat16 h1[TILE * LDH], h2[TILE * LDH], h3[TILE * LDH];
    __nv_bfloat16 d1[TILE * LDH], d2[TILE * LDH], d3[TILE * LDH];
    float d4[TILE * 4];
    float ys[TILE * OUT], ws[TILE];
    float loss[4];
};

struct TrainArgs {
    float *theta, *m, *v, *grad, *part;  // grad: the last step's gradient, loss last
    TrainImage *image;
    const float *X, *Y, *W;  // W: sample weights, or null
    const int *idx;          // rows of the minibatches, or null: rows 0, 1, ...
    float *losses;           // a step each
    unsigned *bar;           // grid barrier count, `base` at launch
    int *err;                // a wait gave up
    unsigned base;
    int batch, steps, update;
    float lr, b1, b2, eps;
    float2 c[TRAIN_STEPS];   // 1 - b1^t, 1 - b2^t
};

__device__ __forceinline__ void ldsm4(uint32_t (&r)[4], const __nv_bfloat16 *p) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
                 : "r"((unsigned)__cvta_generic_to_shared(p))
                 : "memory");
}
__device__ __forceinline__ void ldsm4t(uint32_t (&r)[4], const __nv_bfloat16 *p) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
                 : "r"((unsigned)__cvta_generic_to_shared(p))
                 : "memory");
}

// acc (two 8-column tiles from n0) += A (16 rows x 16 KB) * W^T, W [n][k].
template <int KB, int LDA, int LDW>
__device__ __forceinline__ void mm_forward(const __nv_bfloat16 *A, const __nv_bfloat16 *W, int n0, float (&acc)[2][4]) {
    const int lane = threadIdx.x & 31;
    const __nv_bfloat16 *pa = A + (lane & 15) * LDA + (lane >> 4) * 8;
    const __nv_bfloat16 *pb = W + (n0 + (lane >> 4) * 8 + (lane & 7)) * LDW + ((lane >> 3) & 1) * 8;
#pragma unroll
    for (int kb = 0; kb < KB; ++kb) {
        uint32_t a[4], b[4];
        ldsm4(a, pa + 16 * kb);
        ldsm4(b, pb + 16 * kb);
        mma16816(acc[0], a, b[0], b[1]);
        mma16816(acc[1], a, b[2], b[3]);
    }
}
// acc += A (16 rows x 64) * W, W [k][n]: a delta through a layer.
__device__ __forceinline__ void mm_backward(const __nv_bfloat16 *A, const __nv_bfloat16 *W, int n0, float (&acc)[2][4]) {
    const int lane = threadIdx.x & 31;
    const __nv_bfloat16 *pa = A + (lane & 15) * LDH + (lane >> 4) * 8;
    const __nv_bfloat16 *pb = W + (((lane >> 3) & 1) * 8 + (lane & 7)) * LDH + n0 + (lane >> 4) * 8;
#pragma unroll
    for (int kb = 0; kb < HID / 16; ++kb) {
        uint32_t a[4], b[4];
        ldsm4(a, pa + 16 * kb);
        ldsm4t(b, pb + 16 * kb * LDH);
        mma16816(acc[0], a, b[0], b[1]);
        mma16816(acc[1], a, b[2], b[3]);
    }
}
// dW[m0 + ..][n0 + ..] += sum over the tile's rows of delta[r][m] h[r][n], for
// NT column tiles from n0 (one: the second of the loaded pair is not used).
template <int NT, int LDN>
__device__ __forceinline__ void weight_grad(const __nv_bfloat16 *delta, const __nv_bfloat16 *h, int m0, int n0,
                                            float (&acc)[NT][4]) {
    const int lane = threadIdx.x & 31, mat = lane >> 3;
    const __nv_bfloat16 *pa = delta + ((mat >> 1) * 8 + (lane & 7)) * LDH + m0 + (mat & 1) * 8;
    const __nv_bfloat16 *pb = h + ((mat & 1) * 8 + (lane & 7)) * LDN + n0 + (NT == 2 ? (mat >> 1) * 8 : 0);
#pragma unroll
    for (int kb = 0; kb < TILE / 16; ++kb) {
        uint32_t a[4], b[4];
        ldsm4t(a, pa + 16 * kb * LDH);
        ldsm4t(b, pb + 16 * kb * LDN);
        mma16816(acc[0], a, b[0], b[1]);
        if (NT == 2) mma16816(acc[NT - 1], a, b[2], b[3]);
    }
}

// Activations (BF16) of the warp's 16 x 16 block; gd: GELU' of the thread's.
__device__ __forceinline__ void store_act(const float (&acc)[2][4], int r0, int n0, __nv_bfloat16 *h, float (&gd)[2][4]) {
    const int lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
#pragma unroll
    for (int j = 0; j < 2; ++j)
#pragma unroll
        for (int q = 0; q < 4; q += 2) {
            const int r = r0 + g + (q >= 2 ? 8 : 0), c = n0 + 8 * j + 2 * t;
            gd[j][q] = gelu_grad(acc[j][q]);
            gd[j][q + 1] = gelu_grad(acc[j][q + 1]);
            *reinterpret_cast<uint32_t *>(h + r * LDH + c) = pack_bf16(gelu(acc[j][q]), gelu(acc[j][q + 1]));
        }
}
// delta = acc (.) GELU'(z), BF16.
__device__ __forceinline__ void store_delta(const float (&acc)[2][4], int r0, int n0, const float (&gd)[2][4],
                                            __nv_bfloat16 *d) {
    const int lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
#pragma unroll
    for (int j = 0; j < 2; ++j)
#pragma unroll
        for (int q = 0; q < 4; q += 2) {
            const int r = r0 + g + (q >= 2 ? 8 : 0), c = n0 + 8 * j + 2 * t;
            *reinterpret_cast<uint32_t *>(d + r * LDH + c) =
                pack_bf16(acc[j][q] * gd[j][q], acc[j][q + 1] * gd[j][q + 1]);
        }
}
__device__ __forceinline__ void init_bias(float (&acc)[2][4], const float *bias, int n0) {
    const int t = threadIdx.x & 3;
#pragma unroll
    for (int j = 0; j < 2; ++j) {
        acc[j][0] = acc[j][2] = bias[n0 + 8 * j + 2 * t];
        acc[j][1] = acc[j][3] = bias[n0 + 8 * j + 2 * t + 1];
    }
}

// Arrives at the grid barrier and waits until every CTA has (count: this
// launch's arrivals with this one); false when the wait gave up.
__device__ __forceinline__ bool grid_barrier(const TrainArgs &a, unsigned count) {
    bool ok = true;
    __syncthreads();
    if (threadIdx.x == 0) {
        __threadfence();
        asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(a.bar) : "memory");
        Spin spin;
        for (;;) {
            unsigned v;
            asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(a.bar) : "memory");
            if ((int)(v - (a.base + count)) >= 0) break;
            if (spin.expired(a.err)) {
                ok = false;
                break;
            }
        }
        __threadfence();
    }
    return !__syncthreads_or(!ok);
}

__global__ void __launch_bounds__(TRAIN_THREADS, 1) k_mlp_train(const __grid_constant__ TrainArgs a) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    TrainSmem &s = *reinterpret_cast<TrainSmem *>(smem_raw);
    const int tid = threadIdx.x, lane = tid & 31, g = lane >> 2, t = lane & 3, w = tid >> 5;
    const int rg = w & 3, r0 = 16 * rg, n0 = 16 * (w >> 2);
    const int G = gridDim.x, b = blockIdx.x;
    const int per = (NPART + G - 1) / G, i0 = min(b * per, NPART), i1 = min(i0 + per, NPART);
    const float inv_b = 1.0f / (float)a.batch;
    // the tile's inputs, held in registers while the CTA is at a barrier
    constexpr int XV = TILE * IN / TRAIN_THREADS;
    static_assert(XV * TRAIN_THREADS == TILE * IN && TILE * OUT <= TRAIN_THREADS, "one tile a pass of the CTA");
    float xv[XV], yv = 0.f, wv = 1.f;
    auto load_inputs = [&](int step, int base) {
        const int *idx = a.idx ? a.idx + (size_t)step * a.batch : nullptr;
        auto row = [&](int r) { return idx ? idx[base + r] : base + r; };
#pragma unroll
        for (int q = 0; q < XV; ++q) {
            const int e = tid + q * TRAIN_THREADS, r = e / IN;
            xv[q] = base + r < a.batch ? a.X[(size_t)row(r) * IN + e % IN] : 0.f;
        }
        if (tid < TILE * OUT) yv = base + tid / OUT < a.batch ? a.Y[(size_t)row(tid / OUT) * OUT + tid % OUT] : 0.f;
        if (tid < TILE && a.W) wv = base + tid < a.batch ? a.W[row(tid)] : 0.f;
    };
    auto store_inputs = [&]() {
#pragma unroll
        for (int q = 0; q < XV; ++q) {
            const int e = tid + q * TRAIN_THREADS;
            s.xs[e / IN * LDX + e % IN] = __float2bfloat16_rn(xv[q]);
        }
        if (tid < TILE * OUT) s.ys[tid] = yv;
        if (tid < TILE) s.ws[tid] = wv;
    };
    for (int i = i0 + tid; i < min(i1, NPARAM); i += TRAIN_THREADS) put_param(a.image, i, a.theta[i]);
    for (int i = tid; i < TILE * (LDX - IN); i += TRAIN_THREADS)
        s.xs[i / (LDX - IN) * LDX + IN + i % (LDX - IN)] = __float2bfloat16_rn(0.f);
    load_inputs(0, b * TILE);
    unsigned arrivals = G;
    if (!grid_barrier(a, arrivals)) return;
    for (int step = 0; step < a.steps; ++step) {
        {
            const float4 *src = reinterpret_cast<const float4 *>(a.image);
            float4 *dst = reinterpret_cast<float4 *>(&s.w);
            for (int i = tid; i < (int)(sizeof(TrainImage) / 16); i += TRAIN_THREADS) cp_async16(dst + i, src + i);
            cp_async_commit();
        }
        float gw1[1][4] = {}, gw2[2][4] = {}, gw3[2][4] = {};
        float loss = 0.f, bsum = 0.f;
        for (int base = b * TILE; base < a.batch; base += G * TILE) {
            if (base != b * TILE) {
                load_inputs(step, base);
                __syncthreads();  // the last tile's readers are done
            }
            store_inputs();
            cp_async_wait_all();
            __syncthreads();
            // ---- forward
            float acc[2][4], gd1[2][4], gd2[2][4], gd3[2][4];
            init_bias(acc, s.w.b1, n0);
            mm_forward<KIN / 16, LDX, LDX>(s.xs + r0 * LDX, s.w.w1, n0, acc);
            store_act(acc, r0, n0, s.h1, gd1);
            __syncthreads();
            init_bias(acc, s.w.b2, n0);
            mm_forward<HID / 16, LDH, LDH>(s.h1 + r0 * LDH, s.w.w2, n0, acc);
            store_act(acc, r0, n0, s.h2, gd2);
            __syncthreads();
            init_bias(acc, s.w.b3, n0);
            mm_forward<HID / 16, LDH, LDH>(s.h2 + r0 * LDH, s.w.w3, n0, acc);
            store_act(acc, r0, n0, s.h3, gd3);
            __syncthreads();
            if (n0 == 0) {  // the output layer, by one warp of the row group
                float o[4] = {s.w.b4[2 * t], s.w.b4[2 * t + 1], s.w.b4[2 * t], s.w.b4[2 * t + 1]};
                const __nv_bfloat16 *pa = s.h3 + (r0 + (lane & 15)) * LDH + (lane >> 4) * 8;
                const __nv_bfloat16 *pb = s.w.w4 + (lane & 7) * LDH + (lane >> 3) * 8;
#pragma unroll
                for (int kb = 0; kb < HID / 16; kb += 2) {
                    uint32_t a0[4], a1[4], bb[4];
                    ldsm4(a0, pa + 16 * kb);
                    ldsm4(a1, pa + 16 * kb + 16);
                    ldsm4(bb, pb + 16 * kb);
                    mma16816(o, a0, bb[0], bb[1]);
                    mma16816(o, a1, bb[2], bb[3]);
                }
                // output deltas 2 w (y - t) / B (w = 1 without sample weights)
#pragma unroll
                for (int q = 0; q < 4; ++q) {
                    const int rl = r0 + g + (q >= 2 ? 8 : 0), c = 2 * t + (q & 1);
                    float dlt = 0.f;
                    if (c < OUT && base + rl < a.batch) {
                        const float diff = o[q] - s.ys[rl * OUT + c];
                        const float wd = a.W ? s.ws[rl] * diff : diff;
                        loss += wd * diff;
                        dlt = 2.0f * wd * inv_b;
                    }
                    if (c < 4) s.d4[rl * 4 + c] = dlt;
                }
            }
            __syncthreads();
            // ---- backward deltas
#pragma unroll
            for (int j = 0; j < 2; ++j)
#pragma unroll
                for (int q = 0; q < 4; ++q) {
                    const int rl = r0 + g + (q >= 2 ? 8 : 0), c = n0 + 8 * j + 2 * t + (q & 1);
                    acc[j][q] = s.d4[rl * 4] * __bfloat162float(s.w.w4[c]) +
                                s.d4[rl * 4 + 1] * __bfloat162float(s.w.w4[LDH + c]) +
                                s.d4[rl * 4 + 2] * __bfloat162float(s.w.w4[2 * LDH + c]);
                }
            store_delta(acc, r0, n0, gd3, s.d3);
            __syncthreads();
#pragma unroll
            for (int q = 0; q < 8; ++q) acc[q >> 2][q & 3] = 0.f;
            mm_backward(s.d3 + r0 * LDH, s.w.w3, n0, acc);
            store_delta(acc, r0, n0, gd2, s.d2);
            __syncthreads();
#pragma unroll
            for (int q = 0; q < 8; ++q) acc[q >> 2][q & 3] = 0.f;
            mm_backward(s.d2 + r0 * LDH, s.w.w2, n0, acc);
            store_delta(acc, r0, n0, gd1, s.d1);
            __syncthreads();
            // ---- weight gradients: rows r0 .. + 15 of each matrix, columns n0 ..
            // + 15 (w1: 8 (n0 / 16) .. + 7)
            weight_grad<1, LDX>(s.d1, s.xs, r0, n0 / 2, gw1);
            weight_grad<2, LDH>(s.d2, s.h1, r0, n0, gw2);
            weight_grad<2, LDH>(s.d3, s.h2, r0, n0, gw3);
            // biases and W4 (SIMT; each entry owned by one thread)
            static_assert(3 * HID + OUT + OUT * HID <= TRAIN_THREADS, "one entry a thread");
            float sum = 0.f;
            if (tid < 3 * HID) {
                const __nv_bfloat16 *d = (tid < HID ? s.d1 : tid < 2 * HID ? s.d2 : s.d3) + tid % HID;
#pragma unroll 16
                for (int r = 0; r < TILE; ++r) sum += __bfloat162float(d[r * LDH]);
            } else if (tid < 3 * HID + OUT) {
#pragma unroll 16
                for (int r = 0; r < TILE; ++r) sum += s.d4[r * 4 + tid - 3 * HID];
            } else if (tid < 3 * HID + OUT + OUT * HID) {
                const int k = tid - 3 * HID - OUT, oo = k / HID, c = k % HID;
#pragma unroll 16
                for (int r = 0; r < TILE; ++r) sum += s.d4[r * 4 + oo] * __bfloat162float(s.h3[r * LDH + c]);
            }
            bsum += sum;
        }
        // ---- partial gradient of this CTA
        float *P = a.part + (size_t)b * NPART;
        auto put2 = [&](int at, float x, float y) { *reinterpret_cast<float2 *>(P + at) = make_float2(x, y); };
#pragma unroll
        for (int q = 0; q < 4; q += 2) {
            const int oo = r0 + g + (q >= 2 ? 8 : 0), c1 = n0 / 2 + 2 * t;
            if (c1 < IN) put2(OFF_W1 + oo * IN + c1, gw1[0][q], gw1[0][q + 1]);
#pragma unroll
            for (int j = 0; j < 2; ++j) {
                const int c = n0 + 8 * j + 2 * t;
                put2(OFF_W2 + oo * HID + c, gw2[j][q], gw2[j][q + 1]);
                put2(OFF_W3 + oo * HID + c, gw3[j][q], gw3[j][q + 1]);
            }
        }
        if (tid < HID) P[OFF_B1 + tid] = bsum;
        else if (tid < 2 * HID) P[OFF_B2 + tid - HID] = bsum;
        else if (tid < 3 * HID) P[OFF_B3 + tid - 2 * HID] = bsum;
        else if (tid < 3 * HID + OUT) P[OFF_B4 + tid - 3 * HID] = bsum;
        else if (tid < 3 * HID + OUT + OUT * HID) P[OFF_W4 + tid - 3 * HID - OUT] = bsum;
        // loss: fixed-order warp then CTA sum
        if (n0 == 0) {
#pragma unroll
            for (int off = 16; off > 0; off >>= 1) loss += __shfl_down_sync(0xffffffffu, loss, off);
            if (lane == 0) s.loss[rg] = loss;
        }
        __syncthreads();
        if (tid == 0) P[NPARAM] = (((s.loss[0] + s.loss[1]) + s.loss[2]) + s.loss[3]) * inv_b;
        if (step + 1 < a.steps) load_inputs(step + 1, b * TILE);
        arrivals += G;
        if (!grid_barrier(a, arrivals)) return;
        // ---- the gradient, in CTA order, and Adam on the FP32 masters
        for (int i = i0 + tid; i < i1; i += TRAIN_THREADS) {
            constexpr int U = 32;  // partials in flight
            float gi = 0.f;
            for (int p0 = 0; p0 < G; p0 += U) {
                float q[U];
#pragma unroll
                for (int u = 0; u < U; ++u) q[u] = p0 + u < G ? __ldcg(a.part + (size_t)(p0 + u) * NPART + i) : 0.f;
#pragma unroll
                for (int u = 0; u < U; ++u)
                    if (p0 + u < G) gi += q[u];
            }
            if (step + 1 == a.steps) a.grad[i] = gi;
            if (i == NPARAM) {
                a.losses[step] = gi;
            } else if (a.update) {
                // (roundings spelled out: the same bits wherever this is compiled)
                const float mi = __fmaf_rn(1.f - a.b1, gi, __fmul_rn(a.b1, a.m[i]));
                const float vi = __fmaf_rn(__fmul_rn(1.f - a.b2, gi), gi, __fmul_rn(a.b2, a.v[i]));
                a.m[i] = mi;
                a.v[i] = vi;
                const float th = a.theta[i] - a.lr * (mi / a.c[step].x) / (sqrtf(vi / a.c[step].y) + a.eps);
                a.theta[i] = th;
                put_param(a.image, i, th);
            }
        }
        if (step + 1 == a.steps) break;
        arrivals += G;
        if (!grid_barrier(a, arrivals)) return;
    }
}

int grad_ctas(int batch, int sms) {
    int tiles = (batch + TILE - 1) / TILE;
    return tiles < sms ? (tiles > 0 ? tiles : 1) : sms;
}

}  // namespace mlp
}  // namespace pbs

using namespace pbs::mlp;

struct pbs_mlp {
    cudaStream_t stream = nullptr;
    int sms = 148;
    float *theta = nullptr, *m = nullptr, *v = nullptr, *grad = nullptr, *part = nullptr;
    float *X = nullptr, *Y = nullptr, *W = nullptr, *io = nullptr;
    TrainImage *image = nullptr;
    unsigned *sync = nullptr;  // [0] the grid barrier's count, [1] a wait gave up
    float *losses = nullptr;
    int *idx = nullptr;
    int n = 0, cap_part = 0, cap_io = 0, cap_losses = 0, step = 0;
    unsigned arrivals = 0;  // the barrier's count after the launches so far
    int launch_steps = TRAIN_STEPS;  // steps of a launch at most
    bool refuse_launch = false;      // (tests) the next launch fails
};

#define MCK(x)                                                                               \
    do {                                                                                     \
        cudaError_t e__ = (x);                                                               \
        if (e__ != cudaSuccess) return e__ == cudaErrorMemoryAllocation ? PBS_E_OUT_OF_MEMORY : PBS_E_CUDA; \
    } while (0)

static int ensure_io(pbs_mlp *t, int n) {
    if (n <= t->cap_io) return PBS_OK;
    if (t->io) cudaFree(t->io);
    t->io = nullptr;
    t->cap_io = 0;
    MCK(cudaMalloc(&t->io, sizeof(float) * (size_t)n * (IN + OUT)));
    t->cap_io = n;
    return PBS_OK;
}

static int ensure_part(pbs_mlp *t, int nparts) {
    if (nparts <= t->cap_part) return PBS_OK;
    if (t->part) cudaFree(t->part);
    t->part = nullptr;
    t->cap_part = 0;
    MCK(cudaMalloc(&t->part, sizeof(float) * (size_t)nparts * NPART));
    t->cap_part = nparts;
    return PBS_OK;
}

static int ensure_losses(pbs_mlp *t, int steps) {
    if (steps <= t->cap_losses) return PBS_OK;
    if (t->losses) cudaFree(t->losses);
    t->losses = nullptr;
    t->cap_losses = 0;
    MCK(cudaMalloc(&t->losses, sizeof(float) * (size_t)steps));
    t->cap_losses = steps;
    return PBS_OK;
}

// Enqueues `steps` (at most TRAIN_STEPS) minibatches of rows idx[0 .. batch),
// idx[batch .. 2 batch), ... (idx null: one, of rows 0 .. batch), with Adam
// updates or (lr = 0) the gradient only.
static int run_train(pbs_mlp *t, const float *X, const float *Y, const float *W, const int *idx, int batch, int steps,
                     float lr, float *losses) {
    TrainArgs a{};
    const int ctas = grad_ctas(batch, t->sms);
    int rc = ensure_part(t, ctas);
    if (rc != PBS_OK) return rc;
    a.theta = t->theta; a.m = t->m; a.v = t->v; a.grad = t->grad; a.part = t->part;
    a.image = t->image;
    a.X = X; a.Y = Y; a.W = W;
    a.idx = idx;
    a.losses = losses;
    a.bar = t->sync;
    a.err = (int *)(t->sync + 1);
    a.base = t->arrivals;
    a.batch = batch;
    a.steps = steps;
    a.update = lr > 0.f;
    a.lr = lr;
    a.b1 = 0.9f; a.b2 = 0.999f; a.eps = 1e-8f;
    for (int s = 0; s < steps && a.update; ++s) {
        const float n = (float)(t->step + 1 + s);
        a.c[s] = make_float2(1.f - std::pow(a.b1, n), 1.f - std::pow(a.b2, n));
    }
    MCK(cudaFuncSetAttribute(k_mlp_train, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(TrainSmem)));
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeCooperative;
    at[0].val.cooperative = 1;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(ctas);
    cfg.blockDim = dim3(TRAIN_THREADS);
    cfg.dynamicSmemBytes = sizeof(TrainSmem);
    cfg.stream = t->stream;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    if (t->refuse_launch) {
        t->refuse_launch = false;
        return PBS_E_CUDA;
    }
    MCK(cudaLaunchKernelEx(&cfg, k_mlp_train, a));
    if (a.update) t->step += steps;  // (a launch that failed took no step)
    t->arrivals += 2u * (unsigned)steps * (unsigned)ctas;
    return PBS_OK;
}

// Waits for the trainer's stream; PBS_E_DEVICE_TIMEOUT when a device wait gave
// up (the barrier then starts over).
static int finish(pbs_mlp *t) {
    unsigned flag = 0;
    MCK(cudaMemcpyAsync(&flag, t->sync + 1, sizeof(flag), cudaMemcpyDeviceToHost, t->stream));
    MCK(cudaStreamSynchronize(t->stream));
    if (!flag) return PBS_OK;
    MCK(cudaMemset(t->sync, 0, 2 * sizeof(unsigned)));
    t->arrivals = 0;
    return PBS_E_DEVICE_TIMEOUT;
}

extern "C" {

int pbs_mlp_param_count(void) { return NPARAM; }

int pbs_mlp_create(pbs_mlp **out, const float *theta, unsigned long long seed) {
    if (!out) return PBS_E_INVALID_ARG;
    *out = nullptr;
    int dev = 0, ndev = 0;
    if (cudaGetDeviceCount(&ndev) != cudaSuccess || ndev == 0) return PBS_E_NO_DEVICE;
    cudaGetDevice(&dev);
    cudaDeviceProp prop;
    if (cudaGetDeviceProperties(&prop, dev) != cudaSuccess || prop.major != 10 || prop.minor != 3) return PBS_E_NO_DEVICE;
    pbs_mlp *t = new pbs_mlp();
    t->sms = pbs::context_sms(prop);
    std::vector<float> th(NPARAM, 0.f);
    if (theta) {
        std::memcpy(th.data(), theta, sizeof(float) * NPARAM);
    } else {  // He initialisation, zero biases
        std::mt19937_64 rng(seed);
        const int sizes[4][3] = {{OFF_W1, HID, IN}, {OFF_W2, HID, HID}, {OFF_W3, HID, HID}, {OFF_W4, OUT, HID}};
        for (auto &L : sizes) {
            std::normal_distribution<float> nd(0.f, std::sqrt(2.f / L[2]));
            for (int i = 0; i < L[1] * L[2]; ++i) th[L[0] + i] = nd(rng);
        }
    }
    auto fail = [&](int rc) { pbs_mlp_destroy(t); return rc; };
    if (cudaStreamCreateWithFlags(&t->stream, cudaStreamNonBlocking) != cudaSuccess) return fail(PBS_E_CUDA);
    if (cudaMalloc(&t->theta, sizeof(float) * NPARAM) != cudaSuccess || cudaMalloc(&t->m, sizeof(float) * NPARAM) != cudaSuccess ||
        cudaMalloc(&t->v, sizeof(float) * NPARAM) != cudaSuccess || cudaMalloc(&t->grad, sizeof(float) * NPART) != cudaSuccess ||
        cudaMalloc(&t->image, sizeof(TrainImage)) != cudaSuccess || cudaMalloc(&t->sync, 2 * sizeof(unsigned)) != cudaSuccess)
        return fail(PBS_E_OUT_OF_MEMORY);
    if (cudaMemcpy(t->theta, th.data(), sizeof(float) * NPARAM, cudaMemcpyHostToDevice) != cudaSuccess ||
        cudaMemset(t->m, 0, sizeof(float) * NPARAM) != cudaSuccess || cudaMemset(t->v, 0, sizeof(float) * NPARAM) != cudaSuccess ||
        cudaMemset(t->image, 0, sizeof(TrainImage)) != cudaSuccess || cudaMemset(t->sync, 0, 2 * sizeof(unsigned)) != cudaSuccess)
        return fail(PBS_E_CUDA);
    *out = t;
    return PBS_OK;
}

void pbs_mlp_destroy(pbs_mlp *t) {
    if (!t) return;
    if (t->stream) cudaStreamSynchronize(t->stream);
    float *bufs[] = {t->theta, t->m, t->v, t->grad, t->part, t->X, t->Y, t->W, t->io, t->losses};
    for (float *b : bufs)
        if (b) cudaFree(b);
    if (t->image) cudaFree(t->image);
    if (t->sync) cudaFree(t->sync);
    if (t->idx) cudaFree(t->idx);
    if (t->stream) cudaStreamDestroy(t->stream);
    delete t;
}

int pbs_mlp_get_params(pbs_mlp *t, float *theta) {
    if (!t || !theta) return PBS_E_INVALID_ARG;
    MCK(cudaMemcpy(theta, t->theta, sizeof(float) * NPARAM, cudaMemcpyDeviceToHost));
    return PBS_OK;
}

int pbs_mlp_set_params(pbs_mlp *t, const float *theta) {
    if (!t || !theta) return PBS_E_INVALID_ARG;
    MCK(cudaMemcpy(t->theta, theta, sizeof(float) * NPARAM, cudaMemcpyHostToDevice));
    MCK(cudaMemset(t->m, 0, sizeof(float) * NPARAM));
    MCK(cudaMemset(t->v, 0, sizeof(float) * NPARAM));
    t->step = 0;
    return PBS_OK;
}

int pbs_mlp_forward(pbs_mlp *t, const float *X, int n, float *Y) {
    if (!t || !X || !Y || n <= 0) return PBS_E_INVALID_ARG;
    int rc = ensure_io(t, n);
    if (rc != PBS_OK) return rc;
    float *dX = t->io, *dY = t->io + (size_t)n * IN;
    MCK(cudaMemcpyAsync(dX, X, sizeof(float) * (size_t)n * IN, cudaMemcpyHostToDevice, t->stream));
    const int blocks = std::min((n + 63) / 64, 4 * t->sms);
    k_mlp_forward<<<blocks, 128, 0, t->stream>>>(t->theta, dX, n, dY);
    MCK(cudaGetLastError());
    MCK(cudaMemcpyAsync(Y, dY, sizeof(float) * (size_t)n * OUT, cudaMemcpyDeviceToHost, t->stream));
    MCK(cudaStreamSynchronize(t->stream));
    return PBS_OK;
}

int pbs_mlp_gradient(pbs_mlp *t, const float *X, const float *Y, int n, float *grad, float *loss) {
    if (!t || !X || !Y || n <= 0 || !grad) return PBS_E_INVALID_ARG;
    int rc = ensure_io(t, n);
    if (rc == PBS_OK) rc = ensure_losses(t, 1);
    if (rc != PBS_OK) return rc;
    float *dX = t->io, *dY = t->io + (size_t)n * IN;
    MCK(cudaMemcpyAsync(dX, X, sizeof(float) * (size_t)n * IN, cudaMemcpyHostToDevice, t->stream));
    MCK(cudaMemcpyAsync(dY, Y, sizeof(float) * (size_t)n * OUT, cudaMemcpyHostToDevice, t->stream));
    rc = run_train(t, dX, dY, nullptr, nullptr, n, 1, 0.f, t->losses);
    if (rc != PBS_OK) return rc;
    std::vector<float> g(NPART);
    MCK(cudaMemcpyAsync(g.data(), t->grad, sizeof(float) * NPART, cudaMemcpyDeviceToHost, t->stream));
    rc = finish(t);
    if (rc != PBS_OK) return rc;
    std::memcpy(grad, g.data(), sizeof(float) * NPARAM);
    if (loss) *loss = g[NPARAM];
    return PBS_OK;
}

int pbs_mlp_set_data(pbs_mlp *t, const float *X, const float *Y, const float *W, int n) {
    if (!t || !X || !Y || n <= 0) return PBS_E_INVALID_ARG;
    if (W)
        for (int i = 0; i < n; ++i)
            if (!(W[i] >= 0.f) || !std::isfinite(W[i])) return PBS_E_INVALID_ARG;
    if (t->X) cudaFree(t->X);
    if (t->Y) cudaFree(t->Y);
    if (t->W) cudaFree(t->W);
    if (t->idx) cudaFree(t->idx);
    t->X = t->Y = t->W = nullptr;
    t->idx = nullptr;
    t->n = 0;
    MCK(cudaMalloc(&t->X, sizeof(float) * (size_t)n * IN));
    MCK(cudaMalloc(&t->Y, sizeof(float) * (size_t)n * OUT));
    if (W) MCK(cudaMalloc(&t->W, sizeof(float) * (size_t)n));
    MCK(cudaMalloc(&t->idx, sizeof(int) * (size_t)n));
    MCK(cudaMemcpyAsync(t->X, X, sizeof(float) * (size_t)n * IN, cudaMemcpyHostToDevice, t->stream));
    MCK(cudaMemcpyAsync(t->Y, Y, sizeof(float) * (size_t)n * OUT, cudaMemcpyHostToDevice, t->stream));
    if (W) MCK(cudaMemcpyAsync(t->W, W, sizeof(float) * (size_t)n, cudaMemcpyHostToDevice, t->stream));
    MCK(cudaStreamSynchronize(t->stream));
    t->n = n;
    return PBS_OK;
}

// `steps` Adam steps on minibatches of `batch` rows drawn without replacement
// (a fresh permutation each epoch).  losses (optional, `steps` floats) gets
// each step's minibatch loss.  An epoch's permutation (192 us for 65,536 rows)
// is drawn while the device trains on the one before.
int pbs_mlp_train(pbs_mlp *t, int steps, int batch, float lr, unsigned long long seed, float *losses) {
    if (!t || steps < 0 || batch <= 0 || !(lr > 0.f) || t->n <= 0) return PBS_E_INVALID_ARG;
    if (batch > t->n) batch = t->n;
    int rc = ensure_losses(t, steps);
    if (rc != PBS_OK) return rc;
    std::mt19937_64 rng(seed);
    std::vector<int> perm[2];  // the other one may still be on its way to the device
    const int epoch = t->n / batch;
    for (int done = 0, e = 0; done < steps; ++e) {
        std::vector<int> &p = perm[e & 1];
        p.resize(t->n);
        for (int i = 0; i < t->n; ++i) p[i] = i;
        std::shuffle(p.begin(), p.end(), rng);
        if (e) MCK(cudaStreamSynchronize(t->stream));
        MCK(cudaMemcpyAsync(t->idx, p.data(), sizeof(int) * t->n, cudaMemcpyHostToDevice, t->stream));
        for (int k = 0; k < epoch && done < steps;) {
            const int now = std::min({epoch - k, steps - done, t->launch_steps});
            rc = run_train(t, t->X, t->Y, t->W, t->idx + (size_t)k * batch, batch, now, lr, t->losses + done);
            if (rc != PBS_OK) {
                cudaStreamSynchronize(t->stream);
                return rc;
            }
            k += now;
            done += now;
        }
    }
    if (losses && steps > 0)
        MCK(cudaMemcpyAsync(losses, t->losses, sizeof(float) * steps, cudaMemcpyDeviceToHost, t->stream));
    return finish(t);
}

// For the tests only (not in phybs.h): at most `steps` steps a launch.
int pbs_mlp_test_launch_steps(pbs_mlp *t, int steps) {
    if (!t || steps < 1 || steps > TRAIN_STEPS) return PBS_E_INVALID_ARG;
    t->launch_steps = steps;
    return PBS_OK;
}

// For the tests only: the next launch fails.
int pbs_mlp_test_refuse(pbs_mlp *t) {
    if (!t) return PBS_E_INVALID_ARG;
    t->refuse_launch = true;
    return PBS_OK;
}

}  // extern "C"
