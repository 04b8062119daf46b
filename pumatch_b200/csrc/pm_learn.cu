// pm_learn.cu -- the learned scheduler's device code: per-root features and
// a 16 -> 64 -> 64 -> 2 MLP (ReLU) with BF16 weights and FP32 accumulation,
// trained with hand-written forward, backward and Adam kernels.
//
// The network predicts, per root edge, log(1 + DFS cost) and log(1 + adjacency
// reads) of the root's subtree.  Predictions only reorder work (heavy roots
// first) and choose which pages to keep resident; they never prune, so every
// count stays exact.  Nothing here exists in the reference.
//
// The layers are far too small for tensor cores to matter (5,378 parameters;
// a 64-wide layer is one 64x64 product per sample), so they run on the FMA
// pipes, in FP32 throughout (activations are not rounded): a block takes tiles
// of samples through shared memory and each thread a register tile of every
// layer's product, so that two 16-byte shared-memory reads feed 16 or 32
// multiply-adds.
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <cmath>
#include <cstring>
#include <memory>
#include <vector>

#include "pm_device.cuh"

using namespace pm;
namespace pm {
const Plan* plan_of(const pm_plan* h);
}

#define CKL(call)                                                                             \
  do {                                                                                        \
    cudaError_t e_ = (call);                                                                  \
    if (e_ != cudaSuccess)                                                                    \
      return fail(PM_ERR_CUDA, "%s: %s (%s:%d)", #call, cudaGetErrorString(e_), __FILE__, __LINE__); \
  } while (0)

namespace {

constexpr int NIN = PM_MLP_IN, NH = PM_MLP_HIDDEN, NOUT = PM_MLP_OUT;
// parameter layout (row-major, input-major): W1[NIN][NH] b1[NH] W2[NH][NH] b2[NH] W3[NH][NOUT] b3[NOUT]
constexpr int OFF_W1 = 0;
constexpr int OFF_B1 = OFF_W1 + NIN * NH;
constexpr int OFF_W2 = OFF_B1 + NH;
constexpr int OFF_B2 = OFF_W2 + NH * NH;
constexpr int OFF_W3 = OFF_B2 + NH;
constexpr int OFF_B3 = OFF_W3 + NH * NOUT;
constexpr int NPARAM = OFF_B3 + NOUT;
static_assert(NPARAM == PM_MLP_PARAMS, "parameter count");

__device__ __forceinline__ float bf(const __nv_bfloat16 v) { return __bfloat162float(v); }

// Two FP32 multiply-adds in one instruction (each rounded as fmaf rounds).
__device__ __forceinline__ unsigned long long fma2(unsigned long long a, unsigned long long b, unsigned long long c) {
  unsigned long long d;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
  return d;
}
__device__ __forceinline__ unsigned long long pack2(float lo, float hi) {
  unsigned long long d;
  asm("mov.b64 %0, {%1, %2};" : "=l"(d) : "f"(lo), "f"(hi));
  return d;
}
__device__ __forceinline__ float2 unpack2(unsigned long long v) {
  float2 r;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(v));
  return r;
}

// ---------------------------------------------------------------- forward
// 128 samples per tile, 256 threads: thread (tx, ty) computes samples
// [8 ty, 8 ty + 8) x units [4 tx, 4 tx + 4) of each 64-unit layer, sample
// pairs packed.  Activations are kept unit-major, so a thread's eight samples
// of a unit are two 16-byte reads; the last layer's two outputs are summed
// over the 16 threads of a sample group by shuffles.  Bound: multiply-adds
// (5,248 per sample).  Measured (B200), 262,144 samples: 325 us with one
// thread per sample and a weight read per multiply-add, 79 us so.
constexpr int FT = 128, FTP = FT + 4;

struct ForwardSmem {  // (16-byte vectors are read from every array)
  alignas(16) float w[NPARAM];
  alignas(16) float xt[NIN][FTP];
  alignas(16) float ht[NH][FTP];
};
static_assert(OFF_W2 % 4 == 0 && FTP % 4 == 0, "16-byte rows");

template <int K>
__device__ __forceinline__ void layer8x4(const float* __restrict__ in, const float* __restrict__ w, int tx, int ty,
                                         unsigned long long (&acc)[4][4]) {
#pragma unroll 8
  for (int k = 0; k < K; k++) {
    const ulonglong2 a0 = *reinterpret_cast<const ulonglong2*>(in + k * FTP + 8 * ty);
    const ulonglong2 a1 = *reinterpret_cast<const ulonglong2*>(in + k * FTP + 8 * ty + 4);
    const float4 b = *reinterpret_cast<const float4*>(w + k * NH + 4 * tx);
    const unsigned long long b2[4] = {pack2(b.x, b.x), pack2(b.y, b.y), pack2(b.z, b.z), pack2(b.w, b.w)};
#pragma unroll
    for (int j = 0; j < 4; j++) {
      acc[0][j] = fma2(a0.x, b2[j], acc[0][j]);
      acc[1][j] = fma2(a0.y, b2[j], acc[1][j]);
      acc[2][j] = fma2(a1.x, b2[j], acc[2][j]);
      acc[3][j] = fma2(a1.y, b2[j], acc[3][j]);
    }
  }
}

__global__ void __launch_bounds__(256) mlp_forward_kernel(const __nv_bfloat16* __restrict__ wq,
                                                          const float* __restrict__ x, int64_t n,
                                                          float* __restrict__ y) {
  extern __shared__ float4 smem_raw[];
  ForwardSmem& S = *reinterpret_cast<ForwardSmem*>(smem_raw);
  const int tid = threadIdx.x, tx = tid & 15, ty = tid >> 4;
  for (int i = tid; i < NPARAM; i += 256) S.w[i] = bf(wq[i]);
  const int64_t tiles = (n + FT - 1) / FT;
  for (int64_t tile = blockIdx.x; tile < tiles; tile += gridDim.x) {
    const int64_t base = tile * FT;
    __syncthreads();  // the last tile's reads (and the weights' writes)
    for (int i = tid; i < FT * NIN; i += 256) {
      const int r = i / NIN, k = i % NIN;
      S.xt[k][r] = base + r < n ? x[(base + r) * NIN + k] : 0.f;
    }
    __syncthreads();
    unsigned long long acc[4][4];
#pragma unroll
    for (int j = 0; j < 4; j++) {
      const float b = S.w[OFF_B1 + 4 * tx + j];
#pragma unroll
      for (int r = 0; r < 4; r++) acc[r][j] = pack2(b, b);
    }
    layer8x4<NIN>(&S.xt[0][0], S.w + OFF_W1, tx, ty, acc);
#pragma unroll
    for (int j = 0; j < 4; j++) {
      const float2 v0 = unpack2(acc[0][j]), v1 = unpack2(acc[1][j]), v2 = unpack2(acc[2][j]), v3 = unpack2(acc[3][j]);
      float4* o = reinterpret_cast<float4*>(&S.ht[4 * tx + j][8 * ty]);
      o[0] = make_float4(fmaxf(v0.x, 0.f), fmaxf(v0.y, 0.f), fmaxf(v1.x, 0.f), fmaxf(v1.y, 0.f));
      o[1] = make_float4(fmaxf(v2.x, 0.f), fmaxf(v2.y, 0.f), fmaxf(v3.x, 0.f), fmaxf(v3.y, 0.f));
    }
    __syncthreads();
#pragma unroll
    for (int j = 0; j < 4; j++) {
      const float b = S.w[OFF_B2 + 4 * tx + j];
#pragma unroll
      for (int r = 0; r < 4; r++) acc[r][j] = pack2(b, b);
    }
    layer8x4<NH>(&S.ht[0][0], S.w + OFF_W2, tx, ty, acc);
    float o0[8], o1[8];
#pragma unroll
    for (int r = 0; r < 8; r++) o0[r] = o1[r] = 0.f;
#pragma unroll
    for (int j = 0; j < 4; j++) {
      const float w0 = S.w[OFF_W3 + (4 * tx + j) * NOUT], w1 = S.w[OFF_W3 + (4 * tx + j) * NOUT + 1];
#pragma unroll
      for (int r = 0; r < 4; r++) {
        const float2 v = unpack2(acc[r][j]);
        const float a0 = fmaxf(v.x, 0.f), a1 = fmaxf(v.y, 0.f);
        o0[2 * r] = fmaf(a0, w0, o0[2 * r]);
        o1[2 * r] = fmaf(a0, w1, o1[2 * r]);
        o0[2 * r + 1] = fmaf(a1, w0, o0[2 * r + 1]);
        o1[2 * r + 1] = fmaf(a1, w1, o1[2 * r + 1]);
      }
    }
#pragma unroll
    for (int r = 0; r < 8; r++) {
#pragma unroll
      for (int d = 8; d; d >>= 1) {
        o0[r] += __shfl_xor_sync(0xffffffffu, o0[r], d);
        o1[r] += __shfl_xor_sync(0xffffffffu, o1[r], d);
      }
      const int64_t s = base + 8 * ty + r;
      if (tx == r && s < n) {
        y[s * NOUT] = o0[r] + S.w[OFF_B3];
        y[s * NOUT + 1] = o1[r] + S.w[OFF_B3 + 1];
      }
    }
  }
}

// ---------------------------------------------------------------- backward
// Mean-squared-error gradients over the batch, accumulated in FP32.  64
// samples per tile, 256 threads: thread (tx, ty) holds samples [4 ty, 4 ty + 4)
// x units [4 tx, 4 tx + 4) of every layer in registers.  What the next product
// contracts over decides the layout it reads: activations and their gradients
// go to shared memory unit-major for the layers' products and sample-major
// for the weights' outer products.  Weight gradients stay in registers over
// all of a block's tiles and are added to the result once.  Bound: multiply-
// adds (14,720 per sample), 16 per two 16-byte reads.  Measured (B200), 8,192
// samples: 86 us with a quarter of the threads taking one sample
// each (serial chains, 32-way bank conflicts), 18 us so.
constexpr int TILE = 64, TP = TILE + 4;
static_assert(TP % 4 == 0 && NH % 4 == 0, "16-byte rows");

struct BackwardSmem {
  alignas(16) float w[NPARAM];
  alignas(16) float w2t[NH][NH];   // W2 transposed: [k][j]
  alignas(16) float xt[NIN][TP];
  alignas(16) float h1[TILE][NH];    // relu(z1)
  alignas(16) float h1t[NH][TP];
  alignas(16) float dz2[TILE][NH];   // dL/dz2
  alignas(16) float dz2t[NH][TP];
  alignas(16) float dz1[TILE][NH];   // dL/dz1
  float x[TILE][NIN];
  float t[TILE][NOUT];
  float red[16][4 * NH + 4];          // per sample group: b1, b2, W3 (two outputs) sums; b3, loss
};

// acc[r][j] += sum over k of in[k][4 ty + r] * w[k][4 tx + j] (rows of `in`
// TP apart, of `w` NH apart).
template <int K>
__device__ __forceinline__ void tile4x4(const float* __restrict__ in, const float* __restrict__ w, int tx, int ty,
                                        float (&acc)[4][4]) {
#pragma unroll 8
  for (int k = 0; k < K; k++) {
    const float4 a = *reinterpret_cast<const float4*>(in + k * TP + 4 * ty);
    const float4 b = *reinterpret_cast<const float4*>(w + k * NH + 4 * tx);
    const float av[4] = {a.x, a.y, a.z, a.w}, bv[4] = {b.x, b.y, b.z, b.w};
#pragma unroll
    for (int r = 0; r < 4; r++)
#pragma unroll
      for (int j = 0; j < 4; j++) acc[r][j] = fmaf(av[r], bv[j], acc[r][j]);
  }
}

// A thread's 4 x 4 values to the sample-major and (unless null) unit-major arrays.
__device__ __forceinline__ void put4x4(const float (&v)[4][4], float (*rows)[NH], float (*units)[TP], int tx, int ty) {
#pragma unroll
  for (int r = 0; r < 4; r++)
    *reinterpret_cast<float4*>(&rows[4 * ty + r][4 * tx]) = make_float4(v[r][0], v[r][1], v[r][2], v[r][3]);
  if (units) {
#pragma unroll
    for (int j = 0; j < 4; j++)
      *reinterpret_cast<float4*>(&units[4 * tx + j][4 * ty]) = make_float4(v[0][j], v[1][j], v[2][j], v[3][j]);
  }
}

__device__ __forceinline__ void add4(float* p, float a, float b, float c, float d) {
  asm volatile("red.global.add.v4.f32 [%0], {%1, %2, %3, %4};" ::"l"(p), "f"(a), "f"(b), "f"(c), "f"(d) : "memory");
}

// out: NPARAM gradients, then the loss (zeroed before).
__global__ void __launch_bounds__(256) mlp_backward_kernel(const __nv_bfloat16* __restrict__ wq,
                                                           const float* __restrict__ x, const float* __restrict__ t,
                                                           int64_t n, float* __restrict__ out) {
  extern __shared__ float4 smem_raw[];
  BackwardSmem& S = *reinterpret_cast<BackwardSmem*>(smem_raw);
  const int tid = threadIdx.x, tx = tid & 15, ty = tid >> 4;
  for (int i = tid; i < NPARAM; i += 256) {
    const float v = bf(wq[i]);
    S.w[i] = v;
    if (i >= OFF_W2 && i < OFF_B2) S.w2t[(i - OFF_W2) % NH][(i - OFF_W2) / NH] = v;
  }
  const float inv_n = 1.f / (float)(n * NOUT);
  float gw2[4][4] = {}, gw1[4] = {};                    // W2 rows 4 ty.., columns 4 tx..; W1 row ty, columns 4 tx..
  float gb1[4] = {}, gb2[4] = {}, gw3[4][NOUT] = {}, gb3[NOUT] = {}, lsum = 0.f;  // over this thread's samples
  for (int64_t base = (int64_t)blockIdx.x * TILE; base < n; base += (int64_t)gridDim.x * TILE) {
    __syncthreads();  // the last tile's reads (and the weights' writes)
    for (int i = tid; i < TILE * NIN; i += 256) {
      const int r = i / NIN, k = i % NIN;
      const float v = base + r < n ? x[(base + r) * NIN + k] : 0.f;
      S.x[r][k] = v;
      S.xt[k][r] = v;
    }
    if (tid < TILE * NOUT) S.t[tid / NOUT][tid % NOUT] = base + tid / NOUT < n ? t[base * NOUT + tid] : 0.f;
    __syncthreads();
    float h1[4][4], v[4][4];
#pragma unroll
    for (int r = 0; r < 4; r++)
#pragma unroll
      for (int j = 0; j < 4; j++) h1[r][j] = S.w[OFF_B1 + 4 * tx + j];
    tile4x4<NIN>(&S.xt[0][0], S.w + OFF_W1, tx, ty, h1);
#pragma unroll
    for (int r = 0; r < 4; r++)
#pragma unroll
      for (int j = 0; j < 4; j++) h1[r][j] = fmaxf(h1[r][j], 0.f);
    put4x4(h1, S.h1, S.h1t, tx, ty);
    __syncthreads();
#pragma unroll
    for (int r = 0; r < 4; r++)
#pragma unroll
      for (int j = 0; j < 4; j++) v[r][j] = S.w[OFF_B2 + 4 * tx + j];
    tile4x4<NH>(&S.h1t[0][0], S.w + OFF_W2, tx, ty, v);
    // outputs, summed over the 16 threads of the sample group
    float o0[4] = {}, o1[4] = {}, w30[4], w31[4];
#pragma unroll
    for (int j = 0; j < 4; j++) {
      w30[j] = S.w[OFF_W3 + (4 * tx + j) * NOUT];
      w31[j] = S.w[OFF_W3 + (4 * tx + j) * NOUT + 1];
#pragma unroll
      for (int r = 0; r < 4; r++) {
        const float a = fmaxf(v[r][j], 0.f);
        o0[r] = fmaf(a, w30[j], o0[r]);
        o1[r] = fmaf(a, w31[j], o1[r]);
      }
    }
#pragma unroll
    for (int r = 0; r < 4; r++) {
#pragma unroll
      for (int d = 8; d; d >>= 1) {
        o0[r] += __shfl_xor_sync(0xffffffffu, o0[r], d);
        o1[r] += __shfl_xor_sync(0xffffffffu, o1[r], d);
      }
      const int row = 4 * ty + r;
      const bool valid = base + row < n;
      const float e0 = valid ? o0[r] + S.w[OFF_B3] - S.t[row][0] : 0.f;
      const float e1 = valid ? o1[r] + S.w[OFF_B3 + 1] - S.t[row][1] : 0.f;
      const float d0 = 2.f * e0 * inv_n, d1 = 2.f * e1 * inv_n;
      if (tx == 0) {
        lsum += e0 * e0 + e1 * e1;
        gb3[0] += d0;
        gb3[1] += d1;
      }
#pragma unroll
      for (int j = 0; j < 4; j++) {
        const float z = v[r][j], a = fmaxf(z, 0.f);
        gw3[j][0] = fmaf(a, d0, gw3[j][0]);
        gw3[j][1] = fmaf(a, d1, gw3[j][1]);
        const float dz = z > 0.f ? fmaf(w30[j], d0, w31[j] * d1) : 0.f;
        v[r][j] = dz;
        gb2[j] += dz;
      }
    }
    put4x4(v, S.dz2, S.dz2t, tx, ty);
    __syncthreads();
#pragma unroll
    for (int r = 0; r < 4; r++)
#pragma unroll
      for (int j = 0; j < 4; j++) v[r][j] = 0.f;
    tile4x4<NH>(&S.dz2t[0][0], &S.w2t[0][0], tx, ty, v);
#pragma unroll
    for (int r = 0; r < 4; r++)
#pragma unroll
      for (int j = 0; j < 4; j++) {
        v[r][j] = h1[r][j] > 0.f ? v[r][j] : 0.f;
        gb1[j] += v[r][j];
      }
    put4x4(v, S.dz1, nullptr, tx, ty);
    __syncthreads();
    // outer products over the tile's samples
#pragma unroll 4
    for (int r = 0; r < TILE; r++) {
      const float4 a = *reinterpret_cast<const float4*>(&S.h1[r][4 * ty]);
      const float4 b = *reinterpret_cast<const float4*>(&S.dz2[r][4 * tx]);
      const float4 c = *reinterpret_cast<const float4*>(&S.dz1[r][4 * tx]);
      const float xi = S.x[r][ty];
      const float av[4] = {a.x, a.y, a.z, a.w}, bv[4] = {b.x, b.y, b.z, b.w}, cv[4] = {c.x, c.y, c.z, c.w};
#pragma unroll
      for (int i = 0; i < 4; i++) {
#pragma unroll
        for (int j = 0; j < 4; j++) gw2[i][j] = fmaf(av[i], bv[j], gw2[i][j]);
        gw1[i] = fmaf(xi, cv[i], gw1[i]);
      }
    }
  }
  static_assert(NIN == 16 && NH == 64 && NOUT == 2, "thread layout");
  add4(out + OFF_W1 + ty * NH + 4 * tx, gw1[0], gw1[1], gw1[2], gw1[3]);
#pragma unroll
  for (int i = 0; i < 4; i++)
    add4(out + OFF_W2 + (4 * ty + i) * NH + 4 * tx, gw2[i][0], gw2[i][1], gw2[i][2], gw2[i][3]);
  // the sums over samples: per group, then over the groups
#pragma unroll
  for (int j = 0; j < 4; j++) {
    const int u = 4 * tx + j;
    S.red[ty][u] = gb1[j];
    S.red[ty][NH + u] = gb2[j];
    S.red[ty][2 * NH + NOUT * u] = gw3[j][0];
    S.red[ty][2 * NH + NOUT * u + 1] = gw3[j][1];
  }
  if (tx == 0) {
    S.red[ty][4 * NH] = gb3[0];
    S.red[ty][4 * NH + 1] = gb3[1];
    S.red[ty][4 * NH + 2] = lsum;
  }
  __syncthreads();
  for (int i = tid; i < 4 * NH + 3; i += 256) {
    float sum = 0.f;
#pragma unroll
    for (int g = 0; g < 16; g++) sum += S.red[g][i];
    if (i < NH) atomicAdd(out + OFF_B1 + i, sum);
    else if (i < 2 * NH) atomicAdd(out + OFF_B2 + i - NH, sum);
    else if (i < 4 * NH) atomicAdd(out + OFF_W3 + i - 2 * NH, sum);
    else if (i < 4 * NH + 2) atomicAdd(out + OFF_B3 + i - 4 * NH, sum);
    else atomicAdd(out + NPARAM, sum * inv_n);
  }
}

// ---------------------------------------------------------------- Adam
__global__ void adam_kernel(float* __restrict__ w, __nv_bfloat16* __restrict__ wq, const float* __restrict__ g,
                            float* __restrict__ m, float* __restrict__ v, float lr, float b1, float b2, float eps,
                            float c1, float c2) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= NPARAM) return;
  const float gi = g[i];
  const float mi = b1 * m[i] + (1.f - b1) * gi;
  const float vi = b2 * v[i] + (1.f - b2) * gi * gi;
  m[i] = mi;
  v[i] = vi;
  const float wi = w[i] - lr * (mi / c1) / (sqrtf(vi / c2) + eps);
  w[i] = wi;
  wq[i] = __float2bfloat16_rn(wi);
}

__global__ void quantize_kernel(const float* __restrict__ w, __nv_bfloat16* __restrict__ wq) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < NPARAM) wq[i] = __float2bfloat16_rn(w[i]);
}

// ---------------------------------------------------------------- features
// 16 features of a root edge (v0, v1); f[15] depends on the plan (how many
// neighbours of v1 carry pattern vertex 2's label, as a fraction of deg v1).
// What the first two levels of a root's DFS will see, for the cost features:
// v2's candidates are v1's neighbours with v2's label (labeled) or below v0
// (unlabeled, when the plan bounds v2 by v0); each contributes its neighbours
// with v3's label (the label-group offsets give them directly) or its degree.
struct FeatPlan {
  int lab2, lab3;      // pattern labels of v2 and v3 (labeled; -1 when absent)
  int bound_v0;        // unlabeled: v2 < v0
  int nl1;             // label-group stride of lab_off, 0 without groups
  const int32_t* lab_off;
};

// A degree's bucket: quarters of a power of two.
__device__ __forceinline__ int deg_bucket(float deg) { return min((int)floorf(log2f(1.f + deg) * 4.f), 255); }

__global__ void features_kernel(const uint64_t* __restrict__ rowptr, const int32_t* __restrict__ colidx,
                                const uint8_t* __restrict__ labels, const int32_t* __restrict__ maxnbrdeg,
                                const unsigned* __restrict__ cdf, int64_t n, FeatPlan fp, const int2* roots,
                                int64_t nroots, float* __restrict__ out) {
  const int lab2 = fp.lab2;
  const int lane = threadIdx.x & 31;
  const int64_t warps = (int64_t)gridDim.x * (blockDim.x >> 5);
  for (int64_t r = (int64_t)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5); r < nroots; r += warps) {
    const int2 e = roots[r];
    const uint64_t b1 = rowptr[e.y], e1 = rowptr[e.y + 1];
    float two_hop = 0.f, pairs = 0.f;
    int hist[8] = {0, 0, 0, 0, 0, 0, 0, 0};
    int match2 = 0, cand2 = 0;
    for (uint64_t i = b1 + lane; i < e1; i += 32) {
      const int u = colidx[i];
      const float du = (float)(rowptr[u + 1] - rowptr[u]);
      two_hop += du;
      bool is_cand;
      if (labels) {
        const int l = labels[u];
        hist[l & 7]++;
        match2 += (l == lab2);
        is_cand = (l == lab2);
      } else {
        is_cand = !fp.bound_v0 || u < e.x;
      }
      if (is_cand) {
        cand2++;
        if (labels && fp.lab_off && fp.lab3 >= 0 && fp.lab3 < fp.nl1 - 1) {
          const int32_t* o = fp.lab_off + (int64_t)u * fp.nl1;
          pairs += (float)(o[fp.lab3 + 1] - o[fp.lab3]);
        } else {
          pairs += du;
        }
      }
    }
    for (int o = 16; o; o >>= 1) {
      two_hop += __shfl_xor_sync(0xffffffffu, two_hop, o);
      pairs += __shfl_xor_sync(0xffffffffu, pairs, o);
      match2 += __shfl_xor_sync(0xffffffffu, match2, o);
      cand2 += __shfl_xor_sync(0xffffffffu, cand2, o);
#pragma unroll
      for (int k = 0; k < 8; k++) hist[k] += __shfl_xor_sync(0xffffffffu, hist[k], o);
    }
    if (lane == 0) {
      const float d0 = (float)(rowptr[e.x + 1] - rowptr[e.x]);
      const float d1 = (float)(e1 - b1);
      float* f = out + r * NIN;
      f[0] = log2f(1.f + d0);
      f[1] = log2f(1.f + d1);
      f[2] = log2f(1.f + (float)cand2);  // level 1's candidates (v2)
      f[3] = log2f(1.f + pairs);         // (v2, v3) candidate pairs below them
      f[4] = log2f(1.f + two_hop);
      f[5] = log2f(1.f + (float)maxnbrdeg[e.y]);
      f[6] = (float)cdf[deg_bucket(d1)] / (float)n;
      for (int k = 0; k < 8; k++) f[7 + k] = d1 > 0.f ? (float)hist[k] / d1 : 0.f;
      f[15] = d1 > 0.f ? (float)match2 / d1 : 0.f;
    }
  }
}

// Vertices per degree bucket, then (by one block) how many are in each bucket
// or below it.
__global__ void deg_hist_kernel(const uint64_t* rowptr, int64_t n, unsigned int* hist) {
  __shared__ unsigned int h[256];
  for (int i = threadIdx.x; i < 256; i += blockDim.x) h[i] = 0;
  __syncthreads();
  for (int64_t v = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; v < n; v += (int64_t)gridDim.x * blockDim.x)
    atomicAdd(&h[deg_bucket((float)(rowptr[v + 1] - rowptr[v]))], 1u);
  __syncthreads();
  for (int i = threadIdx.x; i < 256; i += blockDim.x)
    if (h[i]) atomicAdd(&hist[i], h[i]);
}

__global__ void deg_cdf_kernel(unsigned int* hist) {  // 256 threads
  __shared__ unsigned int h[256];
  const int i = threadIdx.x;
  h[i] = hist[i];
  __syncthreads();
  for (int o = 1; o < 256; o <<= 1) {
    const unsigned int t = i >= o ? h[i - o] : 0u;
    __syncthreads();
    h[i] += t;
    __syncthreads();
  }
  hist[i] = h[i];
}

// Labeled graphs: all features but the first are v1's alone, and a vertex is
// v1 of as many root edges as it has neighbours of the first label.  So each
// vertex that can be v1 is read once, into rows[v], and the roots copy its
// row; sums are of whole numbers.  Reading N(v1) for every root cost the
// square of the hubs' degrees: measured (B200), R-MAT 524,288 vertices, 8
// labels, 131,000 root edges, a call 4.7 -> 1.0 ms.
__global__ void __launch_bounds__(512) vertex_features_kernel(
    const uint64_t* __restrict__ rowptr, const int32_t* __restrict__ colidx, const uint8_t* __restrict__ labels,
    const int32_t* __restrict__ maxnbrdeg, const unsigned* __restrict__ cdf, int64_t n, FeatPlan fp, int lab1, int d1,
    int d2, float* __restrict__ rows) {
  __shared__ unsigned long long acc[11];  // two_hop, pairs, match2, hist[8]
  const int lane = threadIdx.x & 31;
  struct Sums {
    unsigned long long two_hop = 0, pairs = 0;
    int match2 = 0, hist[8] = {0, 0, 0, 0, 0, 0, 0, 0};
  };
  auto is_v1 = [&](long long v, uint64_t b, uint64_t e) {
    return labels[v] == lab1 && (long long)(e - b) >= d1 && maxnbrdeg[v] >= d2;
  };
  auto walk = [&](uint64_t b, uint64_t e, Sums& r) {
    unsigned long long packed = 0;  // eight 8-bit counts of this lane
    int steps = 0;
    auto unpack = [&]() {
#pragma unroll
      for (int k = 0; k < 8; k++) r.hist[k] += (int)((packed >> (8 * k)) & 255u);
      packed = 0;
      steps = 0;
    };
    for (uint64_t i0 = b; i0 < e; i0 += 128) {
      int u[4], l[4];
      unsigned long long deg[4];
#pragma unroll
      for (int q = 0; q < 4; q++) u[q] = i0 + 32 * q + lane < e ? colidx[i0 + 32 * q + lane] : -1;
#pragma unroll
      for (int q = 0; q < 4; q++) {
        l[q] = u[q] >= 0 ? (int)labels[u[q]] : -1;
        deg[q] = u[q] >= 0 ? rowptr[u[q] + 1] - rowptr[u[q]] : 0ull;
      }
#pragma unroll
      for (int q = 0; q < 4; q++) {
        if (u[q] < 0) continue;
        r.two_hop += deg[q];
        packed += 1ull << (8 * (l[q] & 7));
        if (l[q] == fp.lab2) {
          r.match2++;
          if (fp.lab_off && fp.lab3 >= 0 && fp.lab3 < fp.nl1 - 1) {
            const int32_t* o = fp.lab_off + (int64_t)u[q] * fp.nl1;
            r.pairs += (unsigned long long)(o[fp.lab3 + 1] - o[fp.lab3]);
          } else {
            r.pairs += deg[q];
          }
        }
      }
      if ((steps += 4) > 248) unpack();
    }
    unpack();
    for (int o = 16; o; o >>= 1) {
      r.two_hop += __shfl_xor_sync(0xffffffffu, r.two_hop, o);
      r.pairs += __shfl_xor_sync(0xffffffffu, r.pairs, o);
    }
    r.match2 = __reduce_add_sync(0xffffffffu, r.match2);
#pragma unroll
    for (int k = 0; k < 8; k++) r.hist[k] = __reduce_add_sync(0xffffffffu, r.hist[k]);
  };
  auto write = [&](long long v, uint64_t b, uint64_t e, const Sums& r) {
    const float deg = (float)(e - b);
    float* f = rows + v * NIN;
    f[1] = log2f(1.f + deg);
    f[2] = log2f(1.f + (float)r.match2);  // level 1's candidates (v2)
    f[3] = log2f(1.f + (float)r.pairs);   // (v2, v3) candidate pairs below them
    f[4] = log2f(1.f + (float)r.two_hop);
    f[5] = log2f(1.f + (float)maxnbrdeg[v]);
    f[6] = (float)cdf[deg_bucket(deg)] / (float)n;
#pragma unroll
    for (int k = 0; k < 8; k++) f[7 + k] = deg > 0.f ? (float)r.hist[k] / deg : 0.f;
    f[15] = deg > 0.f ? (float)r.match2 / deg : 0.f;
  };
  for_lists(rowptr, 0, n,
            [&](long long v, uint64_t b, uint64_t e) {
              if (!is_v1(v, b, e)) return;
              Sums r;
              walk(b, e, r);
              if (lane == 0) write(v, b, e, r);
            },
            [&](long long v, uint64_t b, uint64_t e, uint64_t b0, uint64_t e0, int) {
              if (!is_v1(v, b, e)) return;  // the same for all of the block
              if (threadIdx.x < 11) acc[threadIdx.x] = 0;
              __syncthreads();
              Sums r;
              walk(b0, e0, r);
              if (lane == 0) {
                atomicAdd(&acc[0], r.two_hop);
                atomicAdd(&acc[1], r.pairs);
                atomicAdd(&acc[2], (unsigned long long)r.match2);
#pragma unroll
                for (int k = 0; k < 8; k++) atomicAdd(&acc[3 + k], (unsigned long long)r.hist[k]);
              }
              __syncthreads();
              if (threadIdx.x == 0) {
                r.two_hop = acc[0];
                r.pairs = acc[1];
                r.match2 = (int)acc[2];
#pragma unroll
                for (int k = 0; k < 8; k++) r.hist[k] = (int)acc[3 + k];
                write(v, b, e, r);
              }
              __syncthreads();
            });
}

// Four threads per root: v0's degree and v1's row.
__global__ void copy_features_kernel(const uint64_t* __restrict__ rowptr, const int2* __restrict__ roots,
                                     int64_t nroots, const float* __restrict__ rows, float* __restrict__ out) {
  const int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  const int64_t r = t >> 2;
  if (r >= nroots) return;
  const int k = 4 * (int)(t & 3);
  const int2 e = roots[r];
  float4 f = *reinterpret_cast<const float4*>(rows + (int64_t)e.y * NIN + k);
  if (k == 0) f.x = log2f(1.f + (float)(rowptr[e.x + 1] - rowptr[e.x]));
  float* o = out + r * NIN + k;
  if ((reinterpret_cast<uintptr_t>(out) & 15) == 0) {
    *reinterpret_cast<float4*>(o) = f;
  } else {
    o[0] = f.x; o[1] = f.y; o[2] = f.z; o[3] = f.w;
  }
}

}  // namespace

// =====================================================================
// C-ABI
// =====================================================================

struct pm_mlp {
  int device = 0;
  float* w = nullptr;            // FP32 master weights
  __nv_bfloat16* wq = nullptr;   // BF16 copy used by forward/backward
  float* g = nullptr;            // gradients, then the loss
  float* m = nullptr;
  float* v = nullptr;
  float h_out[NPARAM + 1];       // gradients and loss on their way to the caller
  int64_t step = 0;
  int nsm = 148;
};

extern "C" void pm_mlp_free(pm_mlp* m) {
  if (!m) return;
  cudaSetDevice(m->device);
  cudaFree(m->w);
  delete m;
}

extern "C" pm_status pm_mlp_create(int device, uint64_t seed, pm_mlp** out) {
  if (!out) return fail(PM_ERR_INVALID, "pm_mlp_create: null argument");
  int count = 0;
  if (cudaGetDeviceCount(&count) != cudaSuccess || count == 0)
    return fail(PM_ERR_NO_DEVICE, "no CUDA device available; libpumatch_b200 has no CPU path");
  CKL(cudaSetDevice(device));
  std::unique_ptr<pm_mlp, void (*)(pm_mlp*)> m(new pm_mlp, pm_mlp_free);
  m->device = device;
  CKL(cudaDeviceGetAttribute(&m->nsm, cudaDevAttrMultiProcessorCount, device));
  constexpr size_t kPart = (sizeof(float) * (NPARAM + 1) + 255) & ~(size_t)255;
  CKL(cudaMalloc(&m->w, 5 * kPart));  // one allocation, five 256-byte aligned parts
  m->g = reinterpret_cast<float*>(reinterpret_cast<char*>(m->w) + kPart);
  m->m = reinterpret_cast<float*>(reinterpret_cast<char*>(m->w) + 2 * kPart);
  m->v = reinterpret_cast<float*>(reinterpret_cast<char*>(m->w) + 3 * kPart);
  m->wq = reinterpret_cast<__nv_bfloat16*>(reinterpret_cast<char*>(m->w) + 4 * kPart);
  // He-uniform init from the seed (host side, deterministic)
  std::vector<float> h(NPARAM, 0.f);
  Rng r(seed, 77);
  auto fill = [&](int off, int fan_in, int count) {
    const float lim = std::sqrt(6.f / (float)fan_in);
    for (int i = 0; i < count; i++) h[off + i] = (float)((r.uniform() * 2.0 - 1.0) * lim);
  };
  fill(OFF_W1, NIN, NIN * NH);
  fill(OFF_W2, NH, NH * NH);
  fill(OFF_W3, NH, NH * NOUT);
  CKL(cudaMemcpy(m->w, h.data(), sizeof(float) * NPARAM, cudaMemcpyHostToDevice));
  CKL(cudaMemset(m->m, 0, 2 * kPart));  // and v after it
  PM_CK_PENDING("pm_mlp_create");
  quantize_kernel<<<(NPARAM + 255) / 256, 256>>>(m->w, m->wq);
  CKL(cudaGetLastError());
  CKL(cudaDeviceSynchronize());
  *out = m.release();
  return PM_OK;
}

extern "C" pm_status pm_mlp_get_weights(pm_mlp* m, float* host_out) {
  if (!m || !host_out) return fail(PM_ERR_INVALID, "pm_mlp_get_weights: null argument");
  CKL(cudaSetDevice(m->device));
  CKL(cudaMemcpy(host_out, m->w, sizeof(float) * NPARAM, cudaMemcpyDeviceToHost));
  return PM_OK;
}

extern "C" pm_status pm_mlp_set_weights(pm_mlp* m, const float* host_in) {
  if (!m || !host_in) return fail(PM_ERR_INVALID, "pm_mlp_set_weights: null argument");
  CKL(cudaSetDevice(m->device));
  CKL(cudaMemcpy(m->w, host_in, sizeof(float) * NPARAM, cudaMemcpyHostToDevice));
  PM_CK_PENDING("pm_mlp_set_weights");
  quantize_kernel<<<(NPARAM + 255) / 256, 256>>>(m->w, m->wq);
  CKL(cudaGetLastError());
  CKL(cudaDeviceSynchronize());
  m->step = 0;
  CKL(cudaMemset(m->m, 0, sizeof(float) * NPARAM));
  CKL(cudaMemset(m->v, 0, sizeof(float) * NPARAM));
  return PM_OK;
}

extern "C" pm_status pm_mlp_forward(pm_mlp* m, const float* d_x, int64_t n, float* d_y) {
  if (!m || (n > 0 && (!d_x || !d_y))) return fail(PM_ERR_INVALID, "pm_mlp_forward: bad arguments");
  CKL(cudaSetDevice(m->device));
  if (n == 0) return PM_OK;
  const int blocks = (int)std::min<int64_t>((n + FT - 1) / FT, 3 * m->nsm);  // three fit an SM
  PM_CK_PENDING("MLP kernels");
  CKL(cudaFuncSetAttribute(mlp_forward_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(ForwardSmem)));
  mlp_forward_kernel<<<blocks, 256, sizeof(ForwardSmem)>>>(m->wq, d_x, n, d_y);
  CKL(cudaGetLastError());
  CKL(cudaDeviceSynchronize());
  return PM_OK;
}

extern "C" pm_status pm_mlp_gradient(pm_mlp* m, const float* d_x, const float* d_t, int64_t n, float* host_grad,
                                     float* loss_out) {
  if (!m || n <= 0 || !d_x || !d_t) return fail(PM_ERR_INVALID, "pm_mlp_gradient: bad arguments");
  CKL(cudaSetDevice(m->device));
  CKL(cudaMemsetAsync(m->g, 0, sizeof(float) * (NPARAM + 1)));
  const int blocks = (int)std::min<int64_t>((n + TILE - 1) / TILE, m->nsm);
  PM_CK_PENDING("MLP kernels");
  CKL(cudaFuncSetAttribute(mlp_backward_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                           (int)sizeof(BackwardSmem)));
  mlp_backward_kernel<<<blocks, 256, sizeof(BackwardSmem)>>>(m->wq, d_x, d_t, n, m->g);
  CKL(cudaGetLastError());
  // one copy (which waits for the kernel): the gradients when asked for, and the loss
  const int first = host_grad ? 0 : NPARAM;
  CKL(cudaMemcpy(m->h_out + first, m->g + first, sizeof(float) * (NPARAM + 1 - first), cudaMemcpyDeviceToHost));
  if (host_grad) memcpy(host_grad, m->h_out, sizeof(float) * NPARAM);
  if (loss_out) *loss_out = m->h_out[NPARAM];
  return PM_OK;
}

extern "C" pm_status pm_mlp_train_step(pm_mlp* m, const float* d_x, const float* d_t, int64_t n, float lr,
                                       float* loss_out) {
  pm_status st = pm_mlp_gradient(m, d_x, d_t, n, nullptr, loss_out);
  if (st != PM_OK) return st;
  m->step++;
  const float b1 = 0.9f, b2 = 0.999f;
  const float c1 = 1.f - std::pow(b1, (float)m->step), c2 = 1.f - std::pow(b2, (float)m->step);
  PM_CK_PENDING("MLP kernels");
  adam_kernel<<<(NPARAM + 255) / 256, 256>>>(m->w, m->wq, m->g, m->m, m->v, lr, b1, b2, 1e-8f, c1, c2);
  CKL(cudaGetLastError());
  CKL(cudaDeviceSynchronize());
  return PM_OK;
}

namespace pm {
pm_status root_list_for(pm_ctx* c, const pm_graph* g, const pm_plan* p, const int2** roots, int64_t* n);
}

extern "C" pm_status pm_root_features(pm_ctx* c, const pm_graph* g, const pm_plan* p, float* d_features,
                                      int64_t cap, int64_t* n_roots) {
  if (!c || !g || !p || !n_roots) return fail(PM_ERR_INVALID, "pm_root_features: null argument");
  if (!d_features) return pm_count_roots(c, g, p, n_roots);
  const int2* roots = nullptr;
  int64_t n = 0;
  pm_status st = root_list_for(c, g, p, &roots, &n);
  if (st != PM_OK) return st;
  *n_roots = n;
  if (n == 0) return PM_OK;
  if (cap < n) return fail(PM_ERR_INVALID, "pm_root_features: feature buffer holds %lld roots, need %lld",
                           (long long)cap, (long long)n);
  const Plan* pl = plan_of(p);
  // a row per vertex, unless the graph is so large that they would not pay or
  // there is no room for them: then the features of each root by itself
  const size_t rows_bytes = pl->labeled ? (size_t)g->n * NIN * sizeof(float) : 0;
  bool by_vertex = rows_bytes > 0 && rows_bytes <= (1ull << 30);
  auto grow = [&](size_t want) {
    if (c->feat_bytes >= want) return cudaSuccess;
    cudaFree(c->d_feat);
    c->d_feat = nullptr;
    c->feat_bytes = 0;
    const cudaError_t e = cudaMalloc(&c->d_feat, want);
    if (e == cudaSuccess) c->feat_bytes = want;
    return e;
  };
  if (by_vertex && grow(1024 + rows_bytes) == cudaErrorMemoryAllocation) {
    (void)cudaGetLastError();
    by_vertex = false;
  }
  CKL(grow(1024));
  unsigned int* cdf = (unsigned int*)c->d_feat;
  float* rows = (float*)((char*)c->d_feat + 1024);
  const int32_t* colidx = g->residency == PM_RESIDENT_HBM ? g->d_colidx : g->h_colidx_dev;
  FeatPlan fp;
  fp.lab2 = pl->nnodes > 2 ? pl->vertex_label[2] : -1;
  fp.lab3 = pl->nnodes > 3 ? pl->vertex_label[3] : -1;
  fp.bound_v0 = !pl->labeled && (pl->partial[pl->level_begin[1]] & 1u);
  fp.nl1 = g->d_lab_off ? g->nl1 : 0;
  fp.lab_off = g->d_lab_off;
  // (on the default stream: the caller's buffer may have been filled there)
  PM_CK_PENDING("pm_root_features");
  CKL(cudaMemsetAsync(cdf, 0, 1024));
  deg_hist_kernel<<<(int)std::min<int64_t>((g->n + 1023) / 1024, 4 * c->nsm), 256>>>(g->d_rowptr, g->n, cdf);
  deg_cdf_kernel<<<1, 256>>>(cdf);
  if (by_vertex) {
    vertex_features_kernel<<<list_blocks(g->n), 512>>>(g->d_rowptr, colidx, g->d_labels, g->d_maxnbrdeg, cdf, g->n, fp,
                                                       pl->vertex_label[1], pl->degree[1], pl->degree[2], rows);
    copy_features_kernel<<<(unsigned)((4 * n + 255) / 256), 256>>>(g->d_rowptr, roots, n, rows, d_features);
  } else {
    features_kernel<<<4 * c->nsm, 256>>>(g->d_rowptr, colidx, g->d_labels, g->d_maxnbrdeg, cdf, g->n, fp, roots, n,
                                         d_features);
  }
  CKL(cudaGetLastError());
  CKL(cudaDeviceSynchronize());
  return PM_OK;
}
