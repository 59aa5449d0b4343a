// mlp.cu -- training and inference of the learned Drucker-Prager projection
// (mlp.cuh) on the tensor cores.
//
// Training: one CTA takes 128 samples (a row of every tile each, TMEM lane =
// row) through
//   forward   Z1 = X W1^T, H1 = gelu(Z1 + b1); Z2 = H1 W2^T, H2 = gelu(..);
//             Y = H2 W3^T + b3
//   backward  dZ3 = 2 (Y - T) / (3 B); dH2 = dZ3 W3; dZ2 = dH2 gelu'(..);
//             dH1 = dZ2 W2; dZ1 = dH1 gelu'(..)
//   weights   dW3^T = H2^T dZ3, dW2 = dZ2^T H1, dW1 = dZ1^T X
// with every product a tcgen05 BF16 MMA (M = 128 over samples, M = 64 over
// hidden units for the weight gradients) accumulating in TMEM; transposed
// operands are the same tiles read MN-major. The per-CTA gradients go to a
// slice of an FP32 buffer with plain stores, and an Adam step (FP32 master
// weights) adds the slices up and writes the next step's BF16 operand tiles.
// Every sum has a fixed order: training is deterministic.
//
// Bound by the latency of the six products and the epilogues between them
// (TMEM read, bias, GELU, BF16 tiles): 16 warps share the epilogues, a warp
// taking 16 columns of its quarter of the rows, and keep gelu' in registers
// for the backward pass. With four warps, transposed copies in 2-byte
// stores, warp sums of every bias column, atomics and a serial sum over the
// slices a step of 64 tiles took 78 us (49 this kernel, 9.5 Adam, 5 the
// operand tiles, a clear and the gaps); now 13.5 + 4.6 us, each launch
// starting before the one ahead of it ends. Two CTAs fit an SM: 296 tiles a
// step 18.7 us (one CTA 21.8, before 74).
#include <cuda_runtime.h>
#include <sys/mman.h>
#include <unistd.h>

#include <algorithm>
#include <cmath>
#include <cstring>
#include <string>
#include <system_error>
#include <thread>

#include "../../include/icempm.h"
#include "errors.h"
#include "mlp.cuh"
#include "tc05.cuh"

namespace icm {

namespace {

// BF16 operand tiles of the tensor-core form, K-major core-matrix layout
// (tc05.cuh): W1k [64 x 16], W2k [64 x 64], W3k [16 x 64] (rows >= 3 zero).
struct MlpTcNet {
    __nv_bfloat16 W1k[64 * 16], W2k[64 * 64], W3k[16 * 64];
};

constexpr int kRows = 128, kTileThreads = 4 * kRows;  // rows of a tile; threads (four per row)
// Floats of a gradient slice: the weights and biases, then the loss, padded
// so that every slice's rows of W2 start on 16 bytes.
constexpr int kGradBlocks = kOffXMu / 32 + 1, kSliceFloats = 32 * kGradBlocks;
static_assert(kOffW2 % 4 == 0);
// TMEM columns of the accumulators (32-aligned starts). Accumulators share
// columns where one is dead before the next is written: Z1 is read before
// dH1 is formed, Z3 before dH2, dH2 before dW2, dW3^T before dW1.
constexpr uint32_t kTmemCols = 256;
constexpr int cZ1 = 0, cDH1 = 0, cZ2 = 64, cZ3 = 128, cDH2 = 128, cDW2 = 128, cDW3T = 192, cDW1 = 192;
constexpr int kWaitPolls = 1 << 24;

// shared-memory layout of k_mlp_tile (bytes). dZ2 takes H2's tile (last read
// by the product for dW3^T, which completes before dZ2 is formed) and dZ1
// H1's.
constexpr int sW1 = 0, sW2 = sW1 + 2048, sW3 = sW2 + 8192, sX = sW3 + 2048, sH1 = sX + 4096, sH2 = sH1 + 16384,
              sDZ3 = sH2 + 16384, kTileSmem = sDZ3 + 4096;

// 16 consecutive columns (c0 a multiple of 16) of a row of a K-major tile
__device__ __forceinline__ void put_row16(unsigned char *tile, int row, int c0, int cols, const float v[16])
{
    uint4 a, b;
    a.x = pack_bf16(v[0], v[1]); a.y = pack_bf16(v[2], v[3]); a.z = pack_bf16(v[4], v[5]); a.w = pack_bf16(v[6], v[7]);
    b.x = pack_bf16(v[8], v[9]); b.y = pack_bf16(v[10], v[11]); b.z = pack_bf16(v[12], v[13]); b.w = pack_bf16(v[14], v[15]);
    *reinterpret_cast<uint4 *>(tile + tc05::kmajor_offset(row, c0, cols)) = a;
    *reinterpret_cast<uint4 *>(tile + tc05::kmajor_offset(row, c0 + 8, cols)) = b;
}

__device__ __forceinline__ uint32_t sample_index(uint32_t seed, int step, int row, int n)
{
    uint32_t h = seed ^ ((uint32_t)step * 0x9E3779B9u) ^ ((uint32_t)row * 0x85EBCA6Bu);
    h ^= h >> 16;
    h *= 0x7feb352du;
    h ^= h >> 15;
    h *= 0x846ca68bu;
    h ^= h >> 16;
    return h % (uint32_t)n;
}

// The sums over the warp's lanes of 16 values per lane: 16 shuffles, each
// halving the values a lane still holds. Lane l returns the sum of value
// (l >> 1) & 15.
__device__ __forceinline__ float warp_sum16(float v[16], int lane)
{
#pragma unroll
    for (int w = 8; w > 0; w >>= 1) {
        const bool up = (lane & (2 * w)) != 0;  // this lane keeps the upper half
#pragma unroll
        for (int j = 0; j < w; j++) {
            const float give = up ? v[j] : v[w + j], keep = up ? v[w + j] : v[j];
            v[j] = keep + __shfl_xor_sync(0xffffffffu, give, 2 * w);
        }
    }
    return v[0] + __shfl_xor_sync(0xffffffffu, v[0], 1);
}

__device__ __forceinline__ float warp_sum(float v)
{
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

struct TileArgs {
    const float *X, *Y;      // raw features [n][6], targets [n][3]
    int n;
    int sequential;          // rows blockIdx*128 + r (else hashed samples)
    uint32_t seed;
    int step;
    float inv_count;         // 1 / (3 * samples in the batch)
    const MlpTcNet *tc;      // BF16 operand tiles
    const float *net;        // FP32 parameters (biases, normalisation)
    float *grad;             // FP32 gradient slices (net's layout; at kOffXMu the CTA's share of the loss)
    int first_tile;          // tile of CTA 0 (sequential)
    float *Yout;             // inference: denormalised outputs [n][3]
    int *status;             // set to 1 when a wait gives up
};

// GELU and its derivative at one point (the tanh form of gelu and gelu_grad)
__device__ __forceinline__ float gelu_both(float z, float &grad)
{
    const float c = 0.7978845608028654f, a = 0.044715f;
    const float th = tanhf(c * (z + a * z * z * z));
    grad = 0.5f * (1.0f + th) + 0.5f * z * (1.0f - th * th) * c * (1.0f + 3.0f * a * z * z);
    return 0.5f * z * (1.0f + th);
}

template <bool TRAIN>
__global__ void __launch_bounds__(kTileThreads, 2) k_mlp_tile(const __grid_constant__ TileArgs a)
{
    extern __shared__ __align__(1024) unsigned char sm[];
    __shared__ __align__(8) uint64_t mbar;
    __shared__ uint32_t s_tmem;
    __shared__ float s_bias[2 * kMlpHid + 4];
    __shared__ float s_db[2][4][kMlpHid], s_db3[4][4];  // bias gradients and loss by quarter of the rows
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    // the warp's quarter of the rows (its TMEM lanes) and its 16 columns
    const int q = warp & 3, c0 = (warp >> 2) * 16, row = q * 32 + lane;
    const float *net = a.net;
    float *grad = a.grad + (size_t)blockIdx.x * kSliceFloats;

    // sample of this row
    int idx;
    bool valid;
    if (a.sequential) {
        idx = (a.first_tile + blockIdx.x) * kRows + row;
        valid = idx < a.n;
    } else {
        idx = (int)sample_index(a.seed, a.step, blockIdx.x * kRows + row, a.n);
        valid = true;
    }
    // normalised inputs and targets: of the network only its normalisation
    // is read here, which training leaves alone
    float t[kMlpOut] = {0.f, 0.f, 0.f};
    if (c0 == 0) {
        float x[16];
#pragma unroll
        for (int k = 0; k < kMlpInPad; k++) {
            x[k] = 0.f;
            if (k < kMlpIn && valid) x[k] = (a.X[(size_t)idx * kMlpIn + k] - net[kOffXMu + k]) / net[kOffXSd + k];
        }
        put_row16(sm + sX, row, 0, 16, x);
        if (TRAIN && valid)
#pragma unroll
            for (int o = 0; o < kMlpOut; o++) t[o] = (a.Y[(size_t)idx * kMlpOut + o] - net[kOffYMu + o]) / net[kOffYSd + o];
    }
    if (tid == 0) tc05::mbar_init(&mbar, 1);
    if (warp == 0) tc05::alloc(&s_tmem, kTmemCols);
    // in training a programmatic dependent of the Adam step before
    asm volatile("griddepcontrol.wait;" ::: "memory");
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    // operand tiles of the weights, biases
    {
        const uint4 *src = reinterpret_cast<const uint4 *>(a.tc);
        uint4 *dst = reinterpret_cast<uint4 *>(sm + sW1);
        const int nvec = (int)(sizeof(MlpTcNet) / 16);
        for (int i = tid; i < nvec; i += kTileThreads) dst[i] = src[i];
        if (tid < kMlpHid) s_bias[tid] = net[kOffB1 + tid];
        else if (tid < 2 * kMlpHid) s_bias[tid] = net[kOffB2 + tid - kMlpHid];
        else if (tid < 2 * kMlpHid + kMlpOut) s_bias[tid] = net[kOffB3 + tid - 2 * kMlpHid];
    }
    uint32_t phase = 0;
    bool ok = true;
    auto wait_mma = [&]() {
        ok = tc05::mbar_wait(&mbar, phase, kWaitPolls) && ok;
        phase ^= 1;
        tc05::fence_after_sync();
    };
    auto publish = [&]() {  // shared-memory operands written by all threads -> MMA
        tc05::fence_smem_for_mma();
        tc05::fence_before_sync();
        __syncthreads();
        tc05::fence_after_sync();
    };
    publish();
    const uint32_t tmem = s_tmem;
    constexpr uint32_t id128x64 = tc05::idesc_bf16(128, 64), id128x16 = tc05::idesc_bf16(128, 16);
    constexpr uint32_t id128x64t = tc05::idesc_bf16(128, 64, false, true);  // B read transposed
    constexpr uint32_t id64x16tt = tc05::idesc_bf16(64, 16, true, true), id64x64tt = tc05::idesc_bf16(64, 64, true, true);
    // bytes to the next K = 16 of a tile of 64 / 16 columns: along a row, down the rows
    constexpr int kAlong = 256, kDown64 = 2048, kDown16 = 512;
    float z[16], d1[16], d2[16];

    // ---- Z1 = X W1^T
    if (tid == 0) {
        tc05::mma(tmem + cZ1, tc05::desc_kmajor(sm + sX, 16), tc05::desc_kmajor(sm + sW1, 16), id128x64, false);
        tc05::commit(&mbar);
    }
    wait_mma();
    tc05::ld16(tc05::taddr(tmem, q, cZ1 + c0), z);
#pragma unroll
    for (int j = 0; j < 16; j++) z[j] = TRAIN ? gelu_both(z[j] + s_bias[c0 + j], d1[j]) : gelu(z[j] + s_bias[c0 + j]);
    put_row16(sm + sH1, row, c0, 64, z);
    publish();
    // ---- Z2 = H1 W2^T
    if (tid == 0) {
        for (int kk = 0; kk < 4; kk++)
            tc05::mma(tmem + cZ2, tc05::desc_kmajor(sm + sH1 + kAlong * kk, 64),
                      tc05::desc_kmajor(sm + sW2 + kAlong * kk, 64), id128x64, kk > 0);
        tc05::commit(&mbar);
    }
    wait_mma();
    tc05::ld16(tc05::taddr(tmem, q, cZ2 + c0), z);
#pragma unroll
    for (int j = 0; j < 16; j++)
        z[j] = TRAIN ? gelu_both(z[j] + s_bias[kMlpHid + c0 + j], d2[j]) : gelu(z[j] + s_bias[kMlpHid + c0 + j]);
    put_row16(sm + sH2, row, c0, 64, z);
    publish();
    // ---- Y = H2 W3^T + b3
    if (tid == 0) {
        for (int kk = 0; kk < 4; kk++)
            tc05::mma(tmem + cZ3, tc05::desc_kmajor(sm + sH2 + kAlong * kk, 64),
                      tc05::desc_kmajor(sm + sW3 + kAlong * kk, 64), id128x16, kk > 0);
        tc05::commit(&mbar);
    }
    wait_mma();
    if (c0 == 0) {
        tc05::ld16(tc05::taddr(tmem, q, cZ3), z);
        float y[kMlpOut];
#pragma unroll
        for (int o = 0; o < kMlpOut; o++) y[o] = z[o] + s_bias[2 * kMlpHid + o];
        if (!TRAIN) {
            if (valid)
                for (int o = 0; o < kMlpOut; o++)
                    a.Yout[(size_t)idx * kMlpOut + o] = y[o] * net[kOffYSd + o] + net[kOffYMu + o];
        } else {
            // ---- loss and dZ3
            float dy[16], se = 0.f;
#pragma unroll
            for (int o = 0; o < 16; o++) {
                dy[o] = 0.f;
                if (o < kMlpOut && valid) {
                    const float d = y[o] - t[o];
                    se += d * d;
                    dy[o] = 2.f * d * a.inv_count;
                }
            }
            put_row16(sm + sDZ3, row, 0, 16, dy);
            se = warp_sum(se);
#pragma unroll
            for (int o = 0; o < kMlpOut; o++) dy[o] = warp_sum(dy[o]);
            if (lane == 0) {
#pragma unroll
                for (int o = 0; o < kMlpOut; o++) s_db3[q][o] = dy[o];
                s_db3[q][3] = se * a.inv_count;
            }
        }
    }
    if (TRAIN) {
        publish();
        // ---- dH2 = dZ3 W3 ; dW3^T = H2^T dZ3
        if (tid == 0) {
            tc05::mma(tmem + cDH2, tc05::desc_kmajor(sm + sDZ3, 16), tc05::desc_mnmajor(sm + sW3, 64), id128x64t, false);
            for (int kk = 0; kk < 8; kk++)
                tc05::mma(tmem + cDW3T, tc05::desc_mnmajor(sm + sH2 + kDown64 * kk, 64),
                          tc05::desc_mnmajor(sm + sDZ3 + kDown16 * kk, 16), id64x16tt, kk > 0);
            tc05::commit(&mbar);
        }
        if (tid < kMlpOut + 1) {
            const float s = s_db3[0][tid] + s_db3[1][tid] + s_db3[2][tid] + s_db3[3][tid];
            grad[tid < kMlpOut ? kOffB3 + tid : kOffXMu] = s;
        }
        wait_mma();
        tc05::ld16(tc05::taddr(tmem, q, cDH2 + c0), z);
#pragma unroll
        for (int j = 0; j < 16; j++) z[j] *= d2[j];
        put_row16(sm + sH2, row, c0, 64, z);  // dZ2 over H2 (no longer read)
        {
            const float s = warp_sum16(z, lane);
            if ((lane & 1) == 0) s_db[1][q][c0 + (lane >> 1)] = s;
        }
        // dW3^T rows (hidden unit 16 q + lane for lanes < 16)
        if (c0 == 0) {
            tc05::ld16(tc05::taddr(tmem, q, cDW3T), z);
            if (lane < 16)
                for (int o = 0; o < kMlpOut; o++) grad[kOffW3 + o * kMlpHid + q * 16 + lane] = z[o];
        }
        publish();
        // ---- dH1 = dZ2 W2 ; dW2 = dZ2^T H1
        if (tid == 0) {
            for (int kk = 0; kk < 4; kk++)
                tc05::mma(tmem + cDH1, tc05::desc_kmajor(sm + sH2 + kAlong * kk, 64),
                          tc05::desc_mnmajor(sm + sW2 + kDown64 * kk, 64), id128x64t, kk > 0);
            for (int kk = 0; kk < 8; kk++)
                tc05::mma(tmem + cDW2, tc05::desc_mnmajor(sm + sH2 + kDown64 * kk, 64),
                          tc05::desc_mnmajor(sm + sH1 + kDown64 * kk, 64), id64x64tt, kk > 0);
            tc05::commit(&mbar);
        }
        wait_mma();
        tc05::ld16(tc05::taddr(tmem, q, cDH1 + c0), z);
#pragma unroll
        for (int j = 0; j < 16; j++) z[j] *= d1[j];
        put_row16(sm + sH1, row, c0, 64, z);  // dZ1 over H1 (no longer read)
        {
            const float s = warp_sum16(z, lane);
            if ((lane & 1) == 0) s_db[0][q][c0 + (lane >> 1)] = s;
        }
        publish();
        // ---- dW1 = dZ1^T X
        if (tid == 0) {
            for (int kk = 0; kk < 8; kk++)
                tc05::mma(tmem + cDW1, tc05::desc_mnmajor(sm + sH1 + kDown64 * kk, 64),
                          tc05::desc_mnmajor(sm + sX + kDown16 * kk, 16), id64x16tt, kk > 0);
            tc05::commit(&mbar);
        }
        // meanwhile dW2 (columns 128-191) and the bias gradients
        tc05::ld16(tc05::taddr(tmem, q, cDW2 + c0), z);
        if (lane < 16) {
            float4 *w = reinterpret_cast<float4 *>(grad + kOffW2 + (q * 16 + lane) * kMlpHid + c0);
#pragma unroll
            for (int j = 0; j < 4; j++) w[j] = make_float4(z[4 * j], z[4 * j + 1], z[4 * j + 2], z[4 * j + 3]);
        }
        if (tid < 2 * kMlpHid) {
            const int l = tid >> 6, u = tid & 63;
            grad[(l ? kOffB2 : kOffB1) + u] = s_db[l][0][u] + s_db[l][1][u] + s_db[l][2][u] + s_db[l][3][u];
        }
        wait_mma();
        if (c0 == 0) {
            tc05::ld16(tc05::taddr(tmem, q, cDW1), z);
            if (lane < 16)
                for (int i = 0; i < kMlpIn; i++) grad[kOffW1 + (q * 16 + lane) * kMlpIn + i] = z[i];
        }
    }
    if (!ok && a.status) atomicExch(a.status, 1);
    tc05::fence_before_sync();
    __syncthreads();
    tc05::fence_after_sync();
    if (warp == 0) tc05::dealloc(tmem, kTmemCols);
}

// FP32 parameters -> the BF16 operand tiles of both tensor-core forms
__global__ void k_mlp_prep(const float *net, MlpTcNet *tc, MlpWarpNet *wn)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    auto put = [](__nv_bfloat16 *tile, int row, int k, int K, float w) {
        *reinterpret_cast<__nv_bfloat16 *>(reinterpret_cast<unsigned char *>(tile) + tc05::kmajor_offset(row, k, K)) =
            __float2bfloat16(w);
    };
    if (i < 64 * 16) {  // W1 [64][16]
        const int o = i / 16, k = i % 16;
        const float w = k < kMlpIn ? net[kOffW1 + o * kMlpIn + k] : 0.f;
        put(tc->W1k, o, k, 16, w);
        if (wn) wn->W1[o * 16 + k] = __float2bfloat16(w);
    }
    if (i < 64 * 64) {  // W2 [64][64]
        const int o = i / 64, k = i % 64;
        const float w = net[kOffW2 + o * 64 + k];
        put(tc->W2k, o, k, 64, w);
        if (wn) wn->W2[o * 64 + k] = __float2bfloat16(w);
    }
    if (i < 16 * 64) {  // W3 [16][64] (3 real rows)
        const int o = i / 64, k = i % 64;
        const float w = o < kMlpOut ? net[kOffW3 + o * 64 + k] : 0.f;
        put(tc->W3k, o, k, 64, w);
        if (wn && o < 8) wn->W3[o * 64 + k] = __float2bfloat16(w);
    }
    if (wn && i < 64) {
        wn->b1[i] = net[kOffB1 + i];
        wn->b2[i] = net[kOffB2 + i];
        if (i < 8) {
            wn->b3[i] = i < kMlpOut ? net[kOffB3 + i] : 0.f;
            wn->x_mu[i] = i < kMlpIn ? net[kOffXMu + i] : 0.f;
            wn->x_isd[i] = i < kMlpIn ? 1.0f / net[kOffXSd + i] : 0.f;
        }
        if (i < 4) {
            wn->y_mu[i] = i < kMlpOut ? net[kOffYMu + i] : 0.f;
            wn->y_sd[i] = i < kMlpOut ? net[kOffYSd + i] : 0.f;
        }
    }
}

// The sum of nslices gradient slices for the 32 parameters of a block: eight
// warps share the slices (coalesced rows of 32), their sums are added in a
// fixed order and returned in warp 0. (One thread per parameter over all 64
// slices took 9.5 us, waiting for one load after another.)
constexpr int kSumWarps = 8;
__device__ __forceinline__ float slice_sum(const float *grad, int nslices, int i, bool on)
{
    __shared__ float s_part[kSumWarps][32];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    float g = 0.f;
    if (on) {
#pragma unroll 8
        for (int b = w; b < nslices; b += kSumWarps) g += grad[(size_t)b * kSliceFloats + i];
    }
    s_part[w][lane] = g;
    __syncthreads();
    g = 0.f;
    if (w == 0) {
#pragma unroll
        for (int k = 0; k < kSumWarps; k++) g += s_part[k][lane];
    }
    return g;
}

// Adam step on the weights and biases (not the normalisation) with the sum
// of the gradient slices; writes the BF16 operand tiles of the next step
// (their padding stays as k_mlp_prep left it) and the step's loss.
__global__ void __launch_bounds__(32 * kSumWarps) k_mlp_adam(float *net, float *m, float *v, const float *grad, int nslices,
                                                            MlpTcNet *tc, float *loss, float lr, float b1, float b2,
                                                            float eps, float c1, float c2)
{
    asm volatile("griddepcontrol.wait;" ::: "memory");
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    const int i = blockIdx.x * 32 + (threadIdx.x & 31);
    const float g = slice_sum(grad, nslices, i, i <= kOffXMu);
    if (threadIdx.x >= 32 || i > kOffXMu) return;
    if (i == kOffXMu) {
        *loss = g;
        return;
    }
    const float mi = b1 * m[i] + (1.f - b1) * g, vi = b2 * v[i] + (1.f - b2) * g * g;
    m[i] = mi;
    v[i] = vi;
    const float w = net[i] - lr * (mi * c1) / (sqrtf(vi * c2) + eps);
    net[i] = w;
    auto put = [&](__nv_bfloat16 *tile, int row, int k, int K) {
        *reinterpret_cast<__nv_bfloat16 *>(reinterpret_cast<unsigned char *>(tile) + tc05::kmajor_offset(row, k, K)) =
            __float2bfloat16(w);
    };
    if (i < kOffB1) put(tc->W1k, (i - kOffW1) / kMlpIn, (i - kOffW1) % kMlpIn, 16);
    else if (i >= kOffW2 && i < kOffB2) put(tc->W2k, (i - kOffW2) / 64, (i - kOffW2) % 64, 64);
    else if (i >= kOffW3 && i < kOffB3) put(tc->W3k, (i - kOffW3) / 64, (i - kOffW3) % 64, 64);
}

// Adds the sum of the gradient slices to sum (kOffXMu: the loss).
__global__ void __launch_bounds__(32 * kSumWarps) k_mlp_sum(float *sum, const float *grad, int nslices)
{
    const int i = blockIdx.x * 32 + (threadIdx.x & 31);
    const float g = slice_sum(grad, nslices, i, i <= kOffXMu);
    if (threadIdx.x < 32 && i <= kOffXMu) sum[i] += g;
}

// the warp form over a batch (tests and measurements of the in-kernel form)
__global__ void __launch_bounds__(128) k_mlp_warp_infer(const MlpWarpNet *N, const float *X, int n, float *Yout)
{
    __shared__ __align__(16) unsigned char rows[4][32 * 16];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int r = (blockIdx.x * 4 + warp) * 32 + lane;
    __nv_bfloat16 *xrow = reinterpret_cast<__nv_bfloat16 *>(rows[warp]);
#pragma unroll
    for (int k = 0; k < 8; k++) {
        float v = 0.f;
        if (k < kMlpIn && r < n) v = (X[(size_t)r * kMlpIn + k] - N->x_mu[k]) * N->x_isd[k];
        xrow[lane * 8 + k] = __float2bfloat16(v);
    }
    warp_mlp(N, rows[warp]);
    const float *yrow = reinterpret_cast<const float *>(rows[warp]);
    if (r < n)
        for (int o = 0; o < kMlpOut; o++) Yout[(size_t)r * kMlpOut + o] = yrow[lane * 4 + o] * N->y_sd[o] + N->y_mu[o];
}

// harvested trial states (H00, H01, H10, H11, Jp_inv, meta word) ->
// features and exact targets
__global__ void k_mlp_label(const icy_SimParams P, const float *harvest, int n, float *X, float *Y)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const float *h = harvest + (size_t)i * 6;
    const M2d F = {1.0 + (double)h[0], (double)h[1], (double)h[2], 1.0 + (double)h[3]};
    const double jp = h[4];
    const Svd64 d = svd2x2_64(F);
    float x[kMlpIn], y[kMlpOut];
    mlp_features(P, d.s0, d.s1, jp, x);
    const DpResult r = dp_project64(P, d.s0, d.s1, jp);
    mlp_targets(d.s0, d.s1, jp, r.s0, r.s1, r.jp, y);
    for (int k = 0; k < kMlpIn; k++) X[(size_t)i * kMlpIn + k] = x[k];
    for (int k = 0; k < kMlpOut; k++) Y[(size_t)i * kMlpOut + k] = y[k];
}

// ------------------------------------------------------------ host side

// One device allocation for all buffers of a call. An allocation and its
// release take 0.3-0.6 ms each, whatever the size: with one per buffer they
// were half of a 300-step training (9 buffers) and of an evaluation (6).
class Arena {
public:
    ~Arena()
    {
        if (base) cudaFree(base);
    }
    template <class T> void want(T *&p, size_t count)
    {
        parts[n++] = {reinterpret_cast<void **>(&p), bytes};
        bytes += (sizeof(T) * std::max<size_t>(count, 1) + 255) & ~(size_t)255;
    }
    int alloc()
    {
        if (cudaMalloc((void **)&base, bytes) != cudaSuccess) {
            base = nullptr;
            return icm::fail(ICM_ERR_NOMEM, "mlp: device allocation failed");
        }
        for (int i = 0; i < n; i++) *parts[i].p = base + parts[i].offset;
        return ICM_OK;
    }

private:
    struct Part { void **p; size_t offset; } parts[10];
    int n = 0;
    size_t bytes = 0;
    unsigned char *base = nullptr;
};

// Maps the pages of a result buffer while the GPU works. A copy from the
// device takes 1.6 us for each page that its program has not written yet
// (6 MB: 2.65 ms against 0.35 ms), mapping them ahead 0.75 us. Only a hint:
// contents stay, and where the kernel or a thread refuses it the copy maps
// them as before. Below 256 KB a thread costs more than it saves.
class Prefault {
public:
    Prefault(void *p, size_t bytes)
    {
#ifdef MADV_POPULATE_WRITE
        if (bytes < ((size_t)256 << 10)) return;
        const uintptr_t page = (uintptr_t)sysconf(_SC_PAGESIZE);
        const uintptr_t a = ((uintptr_t)p + page - 1) / page * page, b = ((uintptr_t)p + bytes) / page * page;
        try {
            t = std::thread([a, b] { (void)madvise((void *)a, b - a, MADV_POPULATE_WRITE); });
        } catch (const std::system_error &) {
        }
#endif
    }
    ~Prefault() { wait(); }
    void wait()
    {
        if (t.joinable()) t.join();
    }

private:
    std::thread t;
};

struct Stream {
    cudaStream_t s = nullptr;
    ~Stream()
    {
        if (s) cudaStreamDestroy(s);
    }
    int create()
    {
        return cudaStreamCreateWithFlags(&s, cudaStreamNonBlocking) == cudaSuccess
                   ? ICM_OK
                   : icm::fail(ICM_ERR_CUDA, "mlp: stream");
    }
};

// a launch that may start before the kernel ahead of it on the stream ends
// (dependent; the kernels wait for it themselves)
template <class... KArgs, class... Args>
cudaError_t launch_next(cudaStream_t s, bool dependent, void (*kernel)(KArgs...), int blocks, int threads, size_t smem,
                        Args... args)
{
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(blocks);
    cfg.blockDim = dim3(threads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = at;
    cfg.numAttrs = dependent ? 1 : 0;
    return cudaLaunchKernelEx(&cfg, kernel, static_cast<KArgs>(args)...);
}

// the opt-in is per device (cudaFuncSetAttribute acts on the current one)
int set_tile_smem()
{
    constexpr int kMaxDevices = 64;
    static bool done[kMaxDevices] = {};
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess) return icm::fail(ICM_ERR_CUDA, "mlp: cudaGetDevice");
    if (dev >= 0 && dev < kMaxDevices && done[dev]) return ICM_OK;
    if (cudaFuncSetAttribute(k_mlp_tile<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, kTileSmem) != cudaSuccess ||
        cudaFuncSetAttribute(k_mlp_tile<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, kTileSmem) != cudaSuccess)
        return icm::fail(ICM_ERR_CUDA, "mlp: shared-memory opt-in failed");
    if (dev >= 0 && dev < kMaxDevices) done[dev] = true;
    return ICM_OK;
}

int finish_device(const char *what, const int *d_status)
{
    if (cudaDeviceSynchronize() != cudaSuccess)
        return icm::fail(ICM_ERR_CUDA, std::string(what) + ": " + cudaGetErrorString(cudaGetLastError()));
    int s = 0;
    if (d_status && cudaMemcpy(&s, d_status, sizeof(int), cudaMemcpyDeviceToHost) != cudaSuccess)
        return icm::fail(ICM_ERR_CUDA, std::string(what) + ": status copy");
    if (s) return icm::fail(ICM_ERR_CUDA, std::string(what) + ": a tensor-core wait gave up");
    return ICM_OK;
}

int select_device(int device)
{
    int count = 0;
    if (cudaGetDeviceCount(&count) != cudaSuccess || count == 0)
        return icm::fail(ICM_ERR_NODEVICE, "No avaialble CUDA devices");
    if (device < 0 || device >= count) return icm::fail(ICM_ERR_ARG, "mlp: device index out of range");
    if (cudaSetDevice(device) != cudaSuccess) return icm::fail(ICM_ERR_CUDA, "mlp: cudaSetDevice");
    return ICM_OK;
}

void launch_prep(const float *net, MlpTcNet *tc, MlpWarpNet *wn, cudaStream_t s = 0)
{
    k_mlp_prep<<<(64 * 64 + 255) / 256, 256, 0, s>>>(net, tc, wn);
}

}  // namespace

// used by the surrogate form of the substep (device_layer.cu)
int mlp_prepare_warp_net(const float *host_net, MlpWarpNet **out)
{
    float *net;
    MlpTcNet *tc;
    Arena mem;
    mem.want(net, kMlpFloats);
    mem.want(tc, 1);
    int rc = mem.alloc();
    if (rc) return rc;
    MlpWarpNet *wn = nullptr;
    if (cudaMalloc((void **)&wn, sizeof(MlpWarpNet)) != cudaSuccess) return icm::fail(ICM_ERR_NOMEM, "mlp: allocation");
    cudaMemcpy(net, host_net, sizeof(float) * kMlpFloats, cudaMemcpyHostToDevice);
    launch_prep(net, tc, wn);
    if ((rc = finish_device("mlp prep", nullptr))) {
        cudaFree(wn);
        return rc;
    }
    *out = wn;
    return ICM_OK;
}

int mlp_label(const icy_SimParams &P, const float *d_harvest, int n, float *d_x, float *d_y, cudaStream_t s)
{
    if (n <= 0) return ICM_OK;
    k_mlp_label<<<(n + 127) / 128, 128, 0, s>>>(P, d_harvest, n, d_x, d_y);
    const cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return icm::fail(ICM_ERR_CUDA, std::string("k_mlp_label: ") + cudaGetErrorString(e));
    return ICM_OK;
}

}  // namespace icm

using namespace icm;

extern "C" int icm_mlp_floats(void) { return kMlpFloats; }

extern "C" int icm_mlp_normalise(float *net, const float *x, const float *y, int n)
{
    if (!net || !x || !y || n < 2) return icm::fail(ICM_ERR_ARG, "icm_mlp_normalise: bad arguments");
    auto stats = [&](const float *a, int dim, int k, float &mu, float &sd) {
        double s = 0, q = 0;
        for (int i = 0; i < n; i++) s += a[(size_t)i * dim + k];
        const double m = s / n;
        for (int i = 0; i < n; i++) {
            const double d = a[(size_t)i * dim + k] - m;
            q += d * d;
        }
        const double v = std::sqrt(q / (n - 1));
        mu = (float)m;
        sd = (float)(v > 1e-6 * std::max(1.0, std::fabs(m)) ? v : 1.0);
    };
    for (int k = 0; k < kMlpIn; k++) stats(x, kMlpIn, k, net[kOffXMu + k], net[kOffXSd + k]);
    for (int k = 0; k < kMlpOut; k++) stats(y, kMlpOut, k, net[kOffYMu + k], net[kOffYSd + k]);
    return ICM_OK;
}

extern "C" int icm_mlp_train(int device, const float *x, const float *y, int n, const icm_mlp_train_cfg *cfg,
                             float *net_io, float *loss_hist)
{
    if (!x || !y || !cfg || !net_io || n < 1 || cfg->steps < 0 || cfg->batch_tiles < 1)
        return icm::fail(ICM_ERR_ARG, "icm_mlp_train: bad arguments");
    int rc = select_device(device);
    if (rc || (rc = set_tile_smem())) return rc;
    float *X, *Y, *net, *m, *v, *grad, *loss;
    MlpTcNet *tc;
    int *status;
    Arena mem;
    Stream stream;
    const int steps = cfg->steps;
    mem.want(X, (size_t)n * kMlpIn);
    mem.want(Y, (size_t)n * kMlpOut);
    mem.want(net, kMlpFloats);
    mem.want(m, kMlpFloats);
    mem.want(v, kMlpFloats);
    mem.want(grad, (size_t)cfg->batch_tiles * kSliceFloats);
    mem.want(loss, std::max(steps, 1));
    mem.want(tc, 1);
    mem.want(status, 1);
    if ((rc = mem.alloc()) || (rc = stream.create())) return rc;
    cudaMemcpy(X, x, sizeof(float) * n * kMlpIn, cudaMemcpyHostToDevice);
    cudaMemcpy(Y, y, sizeof(float) * n * kMlpOut, cudaMemcpyHostToDevice);
    cudaMemcpy(net, net_io, sizeof(float) * kMlpFloats, cudaMemcpyHostToDevice);
    cudaMemset(m, 0, sizeof(float) * kMlpFloats);
    cudaMemset(v, 0, sizeof(float) * kMlpFloats);
    cudaMemset(loss, 0, sizeof(float) * std::max(steps, 1));
    cudaMemset(status, 0, sizeof(int));
    const float b1 = 0.9f, b2 = 0.999f, eps = 1e-8f;
    TileArgs a{};
    a.X = X;
    a.Y = Y;
    a.n = n;
    a.sequential = 0;
    a.seed = cfg->seed;
    a.inv_count = 1.0f / (3.0f * kRows * cfg->batch_tiles);
    a.tc = tc;
    a.net = net;
    a.grad = grad;
    a.status = status;
    // the default stream's copies and clears first: the steps run on a stream
    // of their own, each launch a programmatic dependent of the one before
    if (cudaStreamSynchronize(0) != cudaSuccess) return icm::fail(ICM_ERR_CUDA, "icm_mlp_train: set-up");
    launch_prep(net, tc, nullptr, stream.s);
    for (int s = 0; s < steps; s++) {
        a.step = s;
        const cudaError_t e1 = launch_next(stream.s, s > 0, k_mlp_tile<true>, cfg->batch_tiles, kTileThreads, kTileSmem, a);
        if (e1 != cudaSuccess) return icm::fail(ICM_ERR_CUDA, std::string("icm_mlp_train: ") + cudaGetErrorString(e1));
        // cosine decay from lr to lr/20
        const float frac = steps > 1 ? (float)s / (float)(steps - 1) : 0.f;
        const float lr = cfg->lr * (0.05f + 0.95f * 0.5f * (1.0f + std::cos(3.14159265f * frac)));
        const float c1 = 1.0f / (1.0f - std::pow(b1, (float)(s + 1))), c2 = 1.0f / (1.0f - std::pow(b2, (float)(s + 1)));
        const cudaError_t e2 = launch_next(stream.s, true, k_mlp_adam, kGradBlocks, 32 * kSumWarps, 0, net, m, v,
                                           (const float *)grad, cfg->batch_tiles, tc, loss + s, lr, b1, b2, eps, c1, c2);
        if (e2 != cudaSuccess) return icm::fail(ICM_ERR_CUDA, std::string("icm_mlp_train: ") + cudaGetErrorString(e2));
    }
    if ((rc = finish_device("icm_mlp_train", status))) return rc;
    cudaMemcpy(net_io, net, sizeof(float) * kMlpFloats, cudaMemcpyDeviceToHost);
    if (loss_hist && steps > 0) cudaMemcpy(loss_hist, loss, sizeof(float) * steps, cudaMemcpyDeviceToHost);
    return ICM_OK;
}

extern "C" int icm_mlp_gradient(int device, const float *net_in, const float *x, const float *y, int n,
                                float *grad_out, float *loss_out)
{
    if (!net_in || !x || !y || !grad_out || n < 1) return icm::fail(ICM_ERR_ARG, "icm_mlp_gradient: bad arguments");
    int rc = select_device(device);
    if (rc || (rc = set_tile_smem())) return rc;
    float *X, *Y, *net, *grad, *sum;
    MlpTcNet *tc;
    int *status;
    Arena mem;
    const int tiles = (n + kRows - 1) / kRows, kSlices = 1024;  // tiles per launch
    mem.want(X, (size_t)n * kMlpIn);
    mem.want(Y, (size_t)n * kMlpOut);
    mem.want(net, kMlpFloats);
    mem.want(grad, (size_t)std::min(tiles, kSlices) * kSliceFloats);
    mem.want(sum, kMlpFloats);
    mem.want(tc, 1);
    mem.want(status, 1);
    if ((rc = mem.alloc())) return rc;
    cudaMemcpy(X, x, sizeof(float) * n * kMlpIn, cudaMemcpyHostToDevice);
    cudaMemcpy(Y, y, sizeof(float) * n * kMlpOut, cudaMemcpyHostToDevice);
    cudaMemcpy(net, net_in, sizeof(float) * kMlpFloats, cudaMemcpyHostToDevice);
    cudaMemset(sum, 0, sizeof(float) * kMlpFloats);
    cudaMemset(status, 0, sizeof(int));
    launch_prep(net, tc, nullptr);
    TileArgs a{};
    a.X = X;
    a.Y = Y;
    a.n = n;
    a.sequential = 1;
    a.inv_count = 1.0f / (3.0f * n);
    a.tc = tc;
    a.net = net;
    a.grad = grad;
    a.status = status;
    for (a.first_tile = 0; a.first_tile < tiles; a.first_tile += kSlices) {
        const int k = std::min(tiles - a.first_tile, kSlices);
        k_mlp_tile<true><<<k, kTileThreads, kTileSmem>>>(a);
        k_mlp_sum<<<kGradBlocks, 32 * kSumWarps>>>(sum, grad, k);
    }
    if ((rc = finish_device("icm_mlp_gradient", status))) return rc;
    float loss = 0.f;
    cudaMemcpy(grad_out, sum, sizeof(float) * kMlpFloats, cudaMemcpyDeviceToHost);
    std::swap(loss, grad_out[kOffXMu]);  // the normalisation has no gradient
    if (loss_out) *loss_out = loss;
    return ICM_OK;
}

extern "C" int icm_mlp_infer(int device, const float *net_in, const float *x, int n, float *y_out, int warp_form)
{
    if (!net_in || !x || !y_out || n < 1) return icm::fail(ICM_ERR_ARG, "icm_mlp_infer: bad arguments");
    int rc = select_device(device);
    if (rc || (rc = set_tile_smem())) return rc;
    float *X, *Yo, *net;
    MlpTcNet *tc;
    MlpWarpNet *wn;
    int *status;
    Prefault result(y_out, sizeof(float) * n * kMlpOut);
    Arena mem;
    mem.want(X, (size_t)n * kMlpIn);
    mem.want(Yo, (size_t)n * kMlpOut);
    mem.want(net, kMlpFloats);
    mem.want(tc, 1);
    mem.want(wn, 1);
    mem.want(status, 1);
    if ((rc = mem.alloc())) return rc;
    cudaMemcpy(X, x, sizeof(float) * n * kMlpIn, cudaMemcpyHostToDevice);
    cudaMemcpy(net, net_in, sizeof(float) * kMlpFloats, cudaMemcpyHostToDevice);
    cudaMemset(status, 0, sizeof(int));
    launch_prep(net, tc, wn);
    if (warp_form) {
        k_mlp_warp_infer<<<(n + 127) / 128, 128>>>(wn, X, n, Yo);
    } else {
        TileArgs a{};
        a.X = X;
        a.n = n;
        a.sequential = 1;
        a.tc = tc;
        a.net = net;
        a.Yout = Yo;
        a.status = status;
        k_mlp_tile<false><<<(n + kRows - 1) / kRows, kTileThreads, kTileSmem>>>(a);
    }
    if ((rc = finish_device("icm_mlp_infer", status))) return rc;
    result.wait();
    cudaMemcpy(y_out, Yo, sizeof(float) * n * kMlpOut, cudaMemcpyDeviceToHost);
    return ICM_OK;
}
