// aep_mlp.cu -- training and batched inference of the learned return map
// (see aep_mlp.cuh).  Everything runs on the device with hand-written kernels:
//   k_mlp_train_tile : forward + backward of 64 training rows per block on the tensor
//                      cores (mma.sync bf16, f32 accumulation); each block writes its
//                      weight and bias gradients to its own row of a partial array
//   k_mlp_reduce     : sums the partial rows in block order (training is
//                      deterministic: the same records give the same parameters); Adam
//                      on the f32 master parameters, refreshes the bf16 copies
//   k_mlp_infer      : batched forward pass (32 rows per warp), as used inside G2P
// Training records (harvested from the exact return mapping where it changed the
// state, 8 floats each):
//   [ln s0, ln s1, ln s2 (trial, sorted descending), q, material, d0, d1, d2]
// with d = ln s_projected - ln s_trial in the same order.  The loss is the mean
// squared error of the network output against d in the scaling of mlp_features.
#include <algorithm>
#include <cmath>
#include <cstring>
#include <random>
#include <string>
#include <vector>

#include "../../include/aep.h"
#include "aep_mlp.cuh"

using namespace aep;

namespace {

// packed f32 parameter vector: W^T blocks then biases
constexpr int kOffW1 = 0;
constexpr int kOffW2 = kOffW1 + 64 * 16;
constexpr int kOffW3 = kOffW2 + 64 * 64;
constexpr int kOffW4 = kOffW3 + 64 * 64;
constexpr int kOffB1 = kOffW4 + 8 * 64;
constexpr int kOffB2 = kOffB1 + 64;
constexpr int kOffB3 = kOffB2 + 64;
constexpr int kOffB4 = kOffB3 + 64;
constexpr int kNumParams = kOffB4 + 8;  // 9928
constexpr int kNumWeights = kOffB1;     // 9728 bf16 copies
static_assert(kNumParams == AEP_MLP_NUM_PARAMS, "parameter count");

constexpr int kTrainRows = 64;
constexpr int kPartBlocks = 256;  // blocks of one gradient pass (16,384 rows)
constexpr int kTrainThreads = 256;
constexpr int kTrainWarps = kTrainThreads / 32;

using bf16 = __nv_bfloat16;

// as ldmatrix_x4, each 8x8 matrix transposed: register j of lane l holds rows 2(l%4),
// 2(l%4)+1 of column l/4
__device__ __forceinline__ void ldmatrix_x4_t(const bf16* p, uint32_t& r0, uint32_t& r1, uint32_t& r2, uint32_t& r3) {
    const unsigned a = (unsigned)__cvta_generic_to_shared(p);
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];\n"
                 : "=r"(r0), "=r"(r1), "=r"(r2), "=r"(r3)
                 : "r"(a));
}

// A 16x32 strip of four 16x8 tiles: c[j] += sum_{k < K} A(m0+i, k) B(k, n0+8j+i'), the k
// tiles in order.  kAT false: A row-major at A[i * as + k], true: A[k * as + i];
// kBT false: B column-major at B[j * bs + k], true: B[k * bs + j].
template <bool kAT, bool kBT, int K>
__device__ __forceinline__ void strip_mma(float (&c)[4][4], const bf16* A, int as, int m0, const bf16* B, int bs,
                                          int n0, int lane) {
    const int i = lane & 7, lo = (lane >> 3) & 1, hi = lane >> 4;
#pragma unroll
    for (int k0 = 0; k0 < K; k0 += 16) {
        uint32_t a[4], b[8];
        if (kAT) ldmatrix_x4_t(A + (k0 + i + 8 * hi) * as + m0 + 8 * lo, a[0], a[1], a[2], a[3]);
        else ldmatrix_x4(A + (m0 + i + 8 * lo) * as + k0 + 8 * hi, a[0], a[1], a[2], a[3]);
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            if (kBT) ldmatrix_x4_t(B + (k0 + i + 8 * lo) * bs + n0 + 16 * h + 8 * hi, b[4 * h], b[4 * h + 1], b[4 * h + 2], b[4 * h + 3]);
            else ldmatrix_x4(B + (n0 + 16 * h + i + 8 * hi) * bs + k0 + 8 * lo, b[4 * h], b[4 * h + 1], b[4 * h + 2], b[4 * h + 3]);
        }
#pragma unroll
        for (int j = 0; j < 4; ++j) mma_bf16(c[j], a[0], a[1], a[2], a[3], b[2 * j], b[2 * j + 1]);
    }
}

// Rows of 24 and 72 halves: the eight rows of an ldmatrix lie on distinct banks.
struct __align__(16) TrainSmem {
    bf16 W1[64 * kStrideIn], W2[64 * kStrideH], W3[64 * kStrideH], W4[8 * kStrideH];  // W^T
    bf16 X[kTrainRows * kStrideIn];
    bf16 H[3][kTrainRows * kStrideH];   // post-activations
    bf16 dZ[3][kTrainRows * kStrideH];  // of the layers 1..3
    bf16 dY[kTrainRows * 8];
    float b[200];
    float T[kTrainRows * 4];
    float g1[64 * 17];  // W1's gradient, before its hi and lo columns are added
    float wloss[kTrainWarps];
};
static_assert(sizeof(TrainSmem) == 88256, "two blocks on an SM of 227 KB");

__device__ __forceinline__ float dsilu(float z) {
    const float s = __frcp_rn(1.0f + __expf(-z));
    return s * (1.0f + z * (1.0f - s));
}

// Forward and backward of one block of rows.  The block's gradient (f32, packed)
// goes to its own row of `part` and its loss to part_loss[block]; k_mlp_reduce
// sums the rows in block order, so training repeats bit for bit.
// A pass of 16,384 rows is one wave of 256 blocks: its time is one block's latency.  Warp w
// owns rows 16 (w >> 1).. and columns 32 (w & 1).. of every 64 x 64 product, so a layer's
// SiLU derivatives stay in the registers of the lanes that need them in the backward pass;
// the fragments, transposed ones too, come by ldmatrix from padded rows; the bias
// gradients, serial sums over 64 rows, are left for the end, each layer on its own warps.
// Measured (16,384 rows, one Adam step with its reduction): 95 -> 20 us against single
// 2-byte fragment loads from unpadded rows.
__global__ void __launch_bounds__(kTrainThreads, 2) k_mlp_train_tile(const float* params, const bf16* wb,
                                                                     const float* __restrict__ rec, int n, int row0,
                                                                     int row_end, int rows_total, float* part,
                                                                     float* part_loss) {
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    extern __shared__ __align__(16) unsigned char smem_raw[];
    TrainSmem& S = *reinterpret_cast<TrainSmem*>(smem_raw);
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int base = row0 + blockIdx.x * kTrainRows;
    float* const grad = part + (long)blockIdx.x * kNumParams;
    // the records do not depend on the previous kernel (the first pass has none)
    for (int r = tid; r < kTrainRows; r += kTrainThreads) {
        const long gi = (long)(base + r) % n;  // wrap around the record set
        const float* q = rec + 8 * gi;
        const bool live = base + r < row_end;
        float ln[3] = {q[0], q[1], q[2]};
        const float sc = mlp_features(ln, q[3], (int)q[4], S.X + r * kStrideIn);
        for (int k = 0; k < 3; ++k) S.T[r * 4 + k] = live ? q[5 + k] * sc : 0.0f;
        S.T[r * 4 + 3] = live ? 1.0f : 0.0f;  // row weight
    }
    asm volatile("griddepcontrol.wait;" ::: "memory");
    // the bf16 copy of the weights, refreshed by every Adam step, 16 bytes at a time; the
    // rows of W1^T repeat their 7 weights in columns 7..13, against the lo halves of the
    // features (mlp_features)
    static_assert(kNumWeights % 8 == 0 && kOffW2 == 128 * 8, "weight copy in 16-byte pieces");
    const uint4* const w16 = reinterpret_cast<const uint4*>(wb);
    for (int r = tid; r < 64; r += kTrainThreads) {
        const uint4 a = w16[2 * r], b = w16[2 * r + 1];
        const uint32_t u[8] = {a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w};
        const bf16* w = reinterpret_cast<const bf16*>(u);
        __align__(16) bf16 d[16];
#pragma unroll
        for (int k = 0; k < kMlpFeat; ++k) d[k] = d[kMlpFeat + k] = w[k];
        d[14] = d[15] = __float2bfloat16(0.0f);
        reinterpret_cast<uint4*>(S.W1 + kStrideIn * r)[0] = reinterpret_cast<const uint4*>(d)[0];
        reinterpret_cast<uint4*>(S.W1 + kStrideIn * r)[1] = reinterpret_cast<const uint4*>(d)[1];
    }
    for (int i = tid; i < (64 + 64 + 8) * 8; i += kTrainThreads)  // W2, W3, W4: rows of 8 pieces, in sequence
        *reinterpret_cast<uint4*>(S.W2 + (i >> 3) * kStrideH + (i & 7) * 8) = w16[128 + i];
    for (int i = tid; i < 200; i += kTrainThreads) S.b[i] = params[kOffB1 + i];
    __syncthreads();
    const int g = lane >> 2, t = lane & 3;
    const int m0 = 16 * (warp >> 1), n0 = 32 * (warp & 1);
    // the lane's entries of tile j: rows m0 + g and m0 + g + 8, columns n0 + 8 j + 2 t, + 1
    float ds[3][4][4];  // silu' at the pre-activations of the lane's entries
    // ---- forward
#pragma unroll
    for (int l = 0; l < 3; ++l) {
        float c[4][4] = {};
        if (l == 0) strip_mma<false, false, 16>(c, S.X, kStrideIn, m0, S.W1, kStrideIn, n0, lane);
        else strip_mma<false, false, 64>(c, S.H[l - 1], kStrideH, m0, l == 1 ? S.W2 : S.W3, kStrideH, n0, lane);
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const int col = n0 + 8 * j + 2 * t;
            const float b0 = S.b[64 * l + col], b1 = S.b[64 * l + col + 1];
            const float z[4] = {c[j][0] + b0, c[j][1] + b1, c[j][2] + b0, c[j][3] + b1};
#pragma unroll
            for (int e = 0; e < 4; ++e) ds[l][j][e] = dsilu(z[e]);
            *reinterpret_cast<uint32_t*>(&S.H[l][(m0 + g) * kStrideH + col]) = pack_bf16x2(silu(z[0]), silu(z[1]));
            *reinterpret_cast<uint32_t*>(&S.H[l][(m0 + g + 8) * kStrideH + col]) = pack_bf16x2(silu(z[2]), silu(z[3]));
        }
        __syncthreads();
    }
    if (warp >= 4) {
        if (lane == 0) S.wloss[warp] = 0.0f;
    } else {  // output layer: 4 m-tiles x 1 n-tile, one per warp
        const int r0 = 16 * warp;
        float c[4] = {0, 0, 0, 0};
#pragma unroll
        for (int k0 = 0; k0 < 64; k0 += 32) {
            uint32_t a[4], b[4];
            ldmatrix_x4(S.W4 + (lane & 7) * kStrideH + k0 + 8 * (lane >> 3), b[0], b[1], b[2], b[3]);
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                ldmatrix_x4(S.H[2] + (r0 + (lane & 15)) * kStrideH + k0 + 16 * h + 8 * (lane >> 4), a[0], a[1], a[2], a[3]);
                mma_bf16(c, a[0], a[1], a[2], a[3], b[2 * h], b[2 * h + 1]);
            }
        }
        float lsum = 0.0f;
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            const int r = r0 + g + (e >> 1) * 8, col = 2 * t + (e & 1);
            const float y = c[e] + S.b[192 + col];
            float d = 0.0f;
            if (col < 3) {
                const float diff = y - S.T[r * 4 + col];
                d = S.T[r * 4 + 3] * diff;
                lsum += d * diff;
            }
            // d loss / d y for loss = sum w (y - t)^2 / (3 rows_total)
            S.dY[r * 8 + col] = __float2bfloat16(2.0f * d / (3.0f * rows_total));
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) lsum += __shfl_xor_sync(0xffffffffu, lsum, o);
        if (lane == 0) S.wloss[warp] = lsum;
    }
    __syncthreads();
    // ---- backward
    // dZ3 = (dY W4^T) * silu'(Z3):  dH3[r][k] = sum_j dY[r][j] W4t[j][k] (8 of 16 k used)
    {
        float c[4][4] = {};
        uint32_t b[4];
        ldmatrix_x4_t(S.W4 + (lane & 7) * kStrideH + n0 + 8 * (lane >> 3), b[0], b[1], b[2], b[3]);
        const uint32_t a0 = ld_pair(S.dY + (m0 + g) * 8 + 2 * t), a1 = ld_pair(S.dY + (m0 + g + 8) * 8 + 2 * t);
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            mma_bf16(c[j], a0, a1, 0u, 0u, b[j], 0u);
            const int col = n0 + 8 * j + 2 * t;
            *reinterpret_cast<uint32_t*>(&S.dZ[2][(m0 + g) * kStrideH + col]) =
                pack_bf16x2(c[j][0] * ds[2][j][0], c[j][1] * ds[2][j][1]);
            *reinterpret_cast<uint32_t*>(&S.dZ[2][(m0 + g + 8) * kStrideH + col]) =
                pack_bf16x2(c[j][2] * ds[2][j][2], c[j][3] * ds[2][j][3]);
        }
    }
    {  // dW4t[j][k] = sum_r dY[r][j] H3[r][k], columns 8 * warp.. (rows j >= 8 of the tile are zero)
        float c[4] = {0, 0, 0, 0};
#pragma unroll
        for (int k0 = 0; k0 < kTrainRows; k0 += 32) {
            uint32_t a[4], b[4];
            ldmatrix_x4_t(S.dY + (k0 + lane) * 8, a[0], a[1], a[2], a[3]);
            ldmatrix_x4_t(S.H[2] + (k0 + lane) * kStrideH + 8 * warp, b[0], b[1], b[2], b[3]);
            mma_bf16(c, a[0], 0u, a[1], 0u, b[0], b[1]);
            mma_bf16(c, a[2], 0u, a[3], 0u, b[2], b[3]);
        }
        *reinterpret_cast<float2*>(grad + kOffW4 + g * 64 + 8 * warp + 2 * t) = make_float2(c[0], c[1]);
    }
    __syncthreads();
    // layers 3, 2: dZ_{l-1} = (dZ_l W_l^T) * silu', then dW_l^T[n][k] = sum_r dZ_l[r][n] H_{l-1}[r][k]
#pragma unroll
    for (int l = 2; l > 0; --l) {
        float c[4][4] = {};
        strip_mma<false, true, 64>(c, S.dZ[l], kStrideH, m0, l == 1 ? S.W2 : S.W3, kStrideH, n0, lane);
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const int col = n0 + 8 * j + 2 * t;
            *reinterpret_cast<uint32_t*>(&S.dZ[l - 1][(m0 + g) * kStrideH + col]) =
                pack_bf16x2(c[j][0] * ds[l - 1][j][0], c[j][1] * ds[l - 1][j][1]);
            *reinterpret_cast<uint32_t*>(&S.dZ[l - 1][(m0 + g + 8) * kStrideH + col]) =
                pack_bf16x2(c[j][2] * ds[l - 1][j][2], c[j][3] * ds[l - 1][j][3]);
#pragma unroll
            for (int e = 0; e < 4; ++e) c[j][e] = 0.0f;
        }
        strip_mma<true, true, kTrainRows>(c, S.dZ[l], kStrideH, m0, S.H[l - 1], kStrideH, n0, lane);
        float* const gw = grad + (l == 1 ? kOffW2 : kOffW3);
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const int k = n0 + 8 * j + 2 * t;
            *reinterpret_cast<float2*>(gw + (m0 + g) * 64 + k) = make_float2(c[j][0], c[j][1]);
            *reinterpret_cast<float2*>(gw + (m0 + g + 8) * 64 + k) = make_float2(c[j][2], c[j][3]);
        }
        __syncthreads();
    }
    {  // layer 1: one 16x8 tile per warp
        const int k1 = 8 * (warp & 1);
        float c[4] = {0, 0, 0, 0};
#pragma unroll
        for (int k0 = 0; k0 < kTrainRows; k0 += 32) {
            uint32_t b[4];
            ldmatrix_x4_t(S.X + (k0 + lane) * kStrideIn + k1, b[0], b[1], b[2], b[3]);
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                uint32_t a[4];
                ldmatrix_x4_t(S.dZ[0] + (k0 + 16 * h + (lane & 7) + 8 * (lane >> 4)) * kStrideH + m0 + 8 * ((lane >> 3) & 1),
                              a[0], a[1], a[2], a[3]);
                mma_bf16(c, a[0], a[1], a[2], a[3], b[2 * h], b[2 * h + 1]);
            }
        }
#pragma unroll
        for (int e = 0; e < 4; ++e) S.g1[(m0 + g + (e >> 1) * 8) * 17 + k1 + 2 * t + (e & 1)] = c[e];
    }
    // bias gradients: the sums over the rows in order
    if (tid < 200) {
        const int l = tid >> 6, j = tid & 63, stride = l < 3 ? kStrideH : 8;
        const bf16* z = (l < 3 ? S.dZ[l] : S.dY) + j;
        float s = 0.0f;
#pragma unroll 16
        for (int r = 0; r < kTrainRows; ++r) s += __bfloat162float(z[r * stride]);
        grad[kOffB1 + tid] = s;
    }
    __syncthreads();
    // W1's gradient: the hi and lo columns of a feature share its weight
    for (int i = tid; i < 64 * 16; i += kTrainThreads) {
        const float* r = S.g1 + (i >> 4) * 17;
        const int k = i & 15;
        grad[kOffW1 + i] = k < kMlpFeat ? r[k] + r[kMlpFeat + k] : k < 2 * kMlpFeat ? 0.0f : r[k];
    }
    if (tid == 0) {
        float l = 0.0f;
        for (int w = 0; w < kTrainWarps; ++w) l += S.wloss[w];
        part_loss[blockIdx.x] = l / (3.0f * rows_total);
    }
}

// Adam (Kingma & Ba 2015) on the f32 master parameters
struct AdamArgs {
    float *p, *m, *v;
    bf16* wb;
    float lr, b1, b2, eps, c1, c2;
};

// grad[i] (+)= sum over the blocks of part[b][i]; loss likewise.  A block of 256
// threads takes 32 parameters: thread (q, i) sums the blocks q*c .. q*c + c - 1 of
// parameter i in order (c = ceil(blocks / 8)), and the eight partial sums are added
// in q order, so the result is the same on every run.  kAdam (a step's last pass): the
// parameter, its moments and its bf16 copy are updated here and the gradient is left zero;
// a launch of its own for that took 3 us of every step.
constexpr int kReduceParams = 32;
constexpr int kReduceSplit = 8;
template <bool kAdam>
__global__ void __launch_bounds__(kReduceParams * kReduceSplit) k_mlp_reduce(const float* part,
                                                                            const float* part_loss, int blocks,
                                                                            float* grad, float* loss, int accumulate,
                                                                            AdamArgs A) {
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    __shared__ float ps[kReduceSplit][kReduceParams + 1];
    __shared__ float pl[kPartBlocks];
    const int ii = threadIdx.x % kReduceParams, q = threadIdx.x / kReduceParams;
    const int i = blockIdx.x * kReduceParams + ii;
    const int c = (blocks + kReduceSplit - 1) / kReduceSplit;
    const int b0 = q * c, b1 = min(blocks, b0 + c);
    asm volatile("griddepcontrol.wait;" ::: "memory");
    if (blockIdx.x == 0)  // the losses, summed in order below
        for (int b = threadIdx.x; b < blocks; b += kReduceParams * kReduceSplit) pl[b] = part_loss[b];
    float s = 0.0f;
    if (i < kNumParams) {
#pragma unroll 16
        for (int b = b0; b < b1; ++b) s += part[(long)b * kNumParams + i];
    }
    ps[q][ii] = s;
    __syncthreads();
    if (q == 0 && i < kNumParams) {
        float t = accumulate ? grad[i] : 0.0f;
#pragma unroll
        for (int k = 0; k < kReduceSplit; ++k) t += ps[k][ii];
        if (kAdam) {
            const float mi = A.b1 * A.m[i] + (1.0f - A.b1) * t;
            const float vi = A.b2 * A.v[i] + (1.0f - A.b2) * t * t;
            A.m[i] = mi;
            A.v[i] = vi;
            const float pi = A.p[i] - A.lr * (mi / A.c1) / (sqrtf(vi / A.c2) + A.eps);
            A.p[i] = pi;
            if (i < kNumWeights) A.wb[i] = __float2bfloat16(pi);
        }
        grad[i] = kAdam ? 0.0f : t;
    }
    if (blockIdx.x == 0 && threadIdx.x == kReduceParams) {
        float l = accumulate ? *loss : 0.0f;
        for (int b = 0; b < blocks; ++b) l += pl[b];
        *loss = l;
    }
}

__global__ void k_mlp_refresh_bf16(const float* __restrict__ p, bf16* __restrict__ wb) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < kNumWeights) wb[i] = __float2bfloat16(p[i]);
}

// batched inference, 32 rows per warp; kStep: with the SiLU of the step's kernels
template <bool kStep>
__global__ void __launch_bounds__(128) k_mlp_infer(MlpParams P, const float* __restrict__ rec, int n,
                                                   float* __restrict__ out) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const MlpSmem W = mlp_smem_carve(smem_raw);
    mlp_load_smem(P, W, threadIdx.x, blockDim.x);
    __syncthreads();
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    unsigned char* wbase = smem_raw + kMlpSmemBytes + warp * kMlpWarpBytes;
    bf16* X = reinterpret_cast<bf16*>(wbase);
    float* Y = reinterpret_cast<float*>(X + kMlpWarpX);
    const long r = ((long)blockIdx.x * 4 + warp) * 32 + lane;
    float sc = 1.0f;
    if (r < n) {
        const float* q = rec + 8 * r;
        float ln[3] = {q[0], q[1], q[2]};
        sc = mlp_features(ln, q[3], (int)q[4], X + lane * kStrideIn);
    } else {
        float ln[3] = {0, 0, 0};
        mlp_features(ln, 0.0f, 0, X + lane * kStrideIn);
    }
    mlp_forward_warp<kStep>(W, X, Y, lane);
    if (r < n)
        for (int k = 0; k < 3; ++k) out[3 * r + k] = Y[lane * kMlpOut + k] / sc;
}

}  // namespace

struct aep_mlp {
    float* p = nullptr;   // f32 master parameters
    float* g = nullptr;   // gradient
    float* m = nullptr;   // Adam moments
    float* v = nullptr;
    bf16* wb = nullptr;   // bf16 weights (W^T blocks)
    float* loss = nullptr;
    float* part = nullptr;       // per-block gradients of one pass [kPartBlocks][kNumParams]
    float* part_loss = nullptr;  // per-block losses
    int64_t t = 0;        // Adam step
    std::string err;
};

namespace aep {
// device view for the learned G2P path (defined here, used by aep_capi.cu)
MlpParams mlp_device_params(const aep_mlp* m) {
    MlpParams P;
    P.w1t = m->wb + kOffW1;
    P.w2t = m->wb + kOffW2;
    P.w3t = m->wb + kOffW3;
    P.w4t = m->wb + kOffW4;
    P.b1 = m->p + kOffB1;
    P.b2 = m->p + kOffB2;
    P.b3 = m->p + kOffB3;
    P.b4 = m->p + kOffB4;
    return P;
}
}  // namespace aep

#define MCK(call)                                                               \
    do {                                                                        \
        cudaError_t e_ = (call);                                                \
        if (e_ != cudaSuccess) {                                                \
            if (mlp) mlp->err = std::string(#call) + ": " + cudaGetErrorString(e_); \
            return e_ == cudaErrorMemoryAllocation ? AEP_OUT_OF_MEMORY : AEP_CUDA_ERROR; \
        }                                                                       \
    } while (0)

// a launch whose kernel waits for the previous one itself (griddepcontrol.wait), so that
// its start overlaps that one's end
template <typename... KArgs, typename... Args>
static cudaError_t launch_after(void (*kernel)(KArgs...), int grid, int block, size_t smem, bool early, cudaStream_t s,
                                Args... args) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)grid);
    cfg.blockDim = dim3((unsigned)block);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = early ? 1 : 0;
    return cudaLaunchKernelEx(&cfg, kernel, static_cast<KArgs>(args)...);
}

extern "C" {

aep_status aep_mlp_create(uint64_t seed, aep_mlp** out) {
    if (!out) return AEP_INVALID_ARG;
    aep_mlp* mlp = new aep_mlp();
    *out = nullptr;
    MCK(cudaMalloc(&mlp->p, sizeof(float) * kNumParams));
    MCK(cudaMalloc(&mlp->g, sizeof(float) * kNumParams));
    MCK(cudaMalloc(&mlp->m, sizeof(float) * kNumParams));
    MCK(cudaMalloc(&mlp->v, sizeof(float) * kNumParams));
    MCK(cudaMalloc(&mlp->wb, sizeof(bf16) * kNumWeights));
    MCK(cudaMalloc(&mlp->loss, sizeof(float)));
    MCK(cudaMalloc(&mlp->part, sizeof(float) * kNumParams * kPartBlocks));
    MCK(cudaMalloc(&mlp->part_loss, sizeof(float) * kPartBlocks));
    // He-normal weights (SiLU), zero biases, seeded
    std::vector<float> h(kNumParams, 0.0f);
    std::mt19937_64 rng(seed);
    auto fill = [&](int off, int nout, int kin_used, int kin) {
        std::normal_distribution<float> nd(0.0f, std::sqrt(2.0f / kin_used));
        for (int o = 0; o < nout; ++o)
            for (int k = 0; k < kin; ++k) h[off + o * kin + k] = k < kin_used ? nd(rng) : 0.0f;
    };
    fill(kOffW1, 64, 6, 16);
    fill(kOffW2, 64, 64, 64);
    fill(kOffW3, 64, 64, 64);
    fill(kOffW4, 8, 64, 64);
    for (int o = 3; o < 8; ++o)
        for (int k = 0; k < 64; ++k) h[kOffW4 + o * 64 + k] = 0.0f;
    for (int k = 0; k < 3 * 64; ++k) h[kOffW4 + k] *= 0.1f;  // small initial output
    MCK(cudaMemcpy(mlp->p, h.data(), sizeof(float) * kNumParams, cudaMemcpyHostToDevice));
    MCK(cudaMemset(mlp->g, 0, sizeof(float) * kNumParams));
    MCK(cudaMemset(mlp->m, 0, sizeof(float) * kNumParams));
    MCK(cudaMemset(mlp->v, 0, sizeof(float) * kNumParams));
    k_mlp_refresh_bf16<<<(kNumWeights + 255) / 256, 256>>>(mlp->p, mlp->wb);
    MCK(cudaGetLastError());
    MCK(cudaDeviceSynchronize());
    *out = mlp;
    return AEP_OK;
}

aep_status aep_mlp_destroy(aep_mlp* mlp) {
    if (!mlp) return AEP_INVALID_ARG;
    cudaFree(mlp->p);
    cudaFree(mlp->g);
    cudaFree(mlp->m);
    cudaFree(mlp->v);
    cudaFree(mlp->wb);
    cudaFree(mlp->loss);
    cudaFree(mlp->part);
    cudaFree(mlp->part_loss);
    delete mlp;
    return AEP_OK;
}

aep_status aep_mlp_get_params(aep_mlp* mlp, float* host, int64_t count) {
    if (!mlp || !host || count != kNumParams) return AEP_INVALID_ARG;
    MCK(cudaMemcpy(host, mlp->p, sizeof(float) * kNumParams, cudaMemcpyDeviceToHost));
    return AEP_OK;
}

aep_status aep_mlp_set_params(aep_mlp* mlp, const float* host, int64_t count) {
    if (!mlp || !host || count != kNumParams) return AEP_INVALID_ARG;
    MCK(cudaMemcpy(mlp->p, host, sizeof(float) * kNumParams, cudaMemcpyHostToDevice));
    k_mlp_refresh_bf16<<<(kNumWeights + 255) / 256, 256>>>(mlp->p, mlp->wb);
    MCK(cudaGetLastError());
    MCK(cudaDeviceSynchronize());
    return AEP_OK;
}

// gradient and loss of `rows` records from row0 (cyclic) into mlp->g / mlp->loss:
// passes of at most kPartBlocks blocks, each reduced in block order; adam: the last
// reduction updates the parameters.  follows: the previous kernel in the stream is a
// reduction of this network (the records are read before that one has completed)
static aep_status grad_pass(aep_mlp* mlp, const float* rec, int64_t n, int64_t row0, int rows, cudaStream_t s,
                            const AdamArgs* adam = nullptr, bool follows = false) {
    static bool attr = false;
    if (!attr) {
        MCK(cudaFuncSetAttribute(k_mlp_train_tile, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(TrainSmem)));
        attr = true;
    }
    const int blocks = (rows + kTrainRows - 1) / kTrainRows;
    for (int b0 = 0; b0 < blocks; b0 += kPartBlocks) {
        const int nb = std::min(kPartBlocks, blocks - b0);
        MCK(launch_after(k_mlp_train_tile, nb, kTrainThreads, sizeof(TrainSmem), follows || b0 > 0, s, mlp->p, mlp->wb,
                         rec, (int)n, (int)(row0 + (int64_t)b0 * kTrainRows), (int)(row0 + rows), rows, mlp->part,
                         mlp->part_loss));
        const bool last = adam && b0 + kPartBlocks >= blocks;
        MCK(launch_after(last ? k_mlp_reduce<true> : k_mlp_reduce<false>, (kNumParams + kReduceParams - 1) / kReduceParams,
                         kReduceParams * kReduceSplit, 0, true, s, mlp->part, mlp->part_loss, nb, mlp->g, mlp->loss,
                         b0 > 0 ? 1 : 0, last ? *adam : AdamArgs{}));
    }
    return AEP_OK;
}

aep_status aep_mlp_gradient(aep_mlp* mlp, const float* d_records, int64_t n, float* host_grad, double* loss) {
    if (!mlp || !d_records || n <= 0 || n > (1 << 24) || !host_grad) return AEP_INVALID_ARG;
    aep_status st = grad_pass(mlp, d_records, n, 0, (int)n, nullptr);
    if (st) return st;
    MCK(cudaDeviceSynchronize());
    MCK(cudaMemcpy(host_grad, mlp->g, sizeof(float) * kNumParams, cudaMemcpyDeviceToHost));
    float l = 0.f;
    MCK(cudaMemcpy(&l, mlp->loss, sizeof(float), cudaMemcpyDeviceToHost));
    if (loss) *loss = l;
    MCK(cudaMemset(mlp->g, 0, sizeof(float) * kNumParams));
    return AEP_OK;
}

aep_status aep_mlp_train(aep_mlp* mlp, const float* d_records, int64_t n, int64_t steps, int32_t batch, double lr,
                         double lr_final, double* final_loss, void* cuda_stream) {
    if (!mlp || !d_records || n <= 0 || steps <= 0 || batch <= 0 || batch > (1 << 20) || !(lr > 0))
        return AEP_INVALID_ARG;
    cudaStream_t s = static_cast<cudaStream_t>(cuda_stream);
    const float b1 = 0.9f, b2 = 0.999f, eps = 1e-8f;
    int64_t row0 = 0;
    double last = 0.0;
    for (int64_t it = 0; it < steps; ++it) {
        // cosine decay from lr to lr_final
        const double frac = steps > 1 ? (double)it / (double)(steps - 1) : 1.0;
        const double lri = lr_final + 0.5 * (lr - lr_final) * (1.0 + std::cos(3.14159265358979323846 * frac));
        const bool report = it == steps - 1;
        const double t = (double)(mlp->t + 1);
        const float c1 = 1.0f - (float)std::pow(b1, t), c2 = 1.0f - (float)std::pow(b2, t);
        const AdamArgs adam{mlp->p, mlp->m, mlp->v, mlp->wb, (float)lri, b1, b2, eps, c1, c2};
        aep_status st = grad_pass(mlp, d_records, n, row0 % n, batch, s, &adam, it > 0);
        if (st) return st;
        ++mlp->t;
        row0 += batch;
        if (report) {
            float l = 0.f;
            MCK(cudaMemcpyAsync(&l, mlp->loss, sizeof(float), cudaMemcpyDeviceToHost, s));
            MCK(cudaStreamSynchronize(s));
            last = l;
        }
    }
    if (final_loss) *final_loss = last;
    return AEP_OK;
}

static aep_status mlp_forward(aep_mlp* mlp, const float* d_records, int64_t n, float* d_out, void* cuda_stream,
                              bool step_form) {
    if (!mlp || !d_records || !d_out || n <= 0 || n > (int64_t)INT32_MAX / 2) return AEP_INVALID_ARG;
    cudaStream_t s = static_cast<cudaStream_t>(cuda_stream);
    const int smem = kMlpSmemBytes + 4 * kMlpWarpBytes;
    const auto kernel = step_form ? k_mlp_infer<true> : k_mlp_infer<false>;
    MCK(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
    kernel<<<(int)((n + 127) / 128), 128, smem, s>>>(mlp_device_params(mlp), d_records, (int)n, d_out);
    MCK(cudaGetLastError());
    return AEP_OK;
}

aep_status aep_mlp_forward(aep_mlp* mlp, const float* d_records, int64_t n, float* d_out, void* cuda_stream) {
    return mlp_forward(mlp, d_records, n, d_out, cuda_stream, false);
}

aep_status aep_mlp_forward_step_form(aep_mlp* mlp, const float* d_records, int64_t n, float* d_out,
                                     void* cuda_stream) {
    return mlp_forward(mlp, d_records, n, d_out, cuda_stream, true);
}

const char* aep_mlp_last_error(aep_mlp* mlp) { return mlp ? mlp->err.c_str() : "null mlp"; }

}  // extern "C"
