// fcdem_sdf.cu -- neural signed-distance field of an obstacle, used to cull
// the distance-map boundary test (boundaries.cuh:38-63) for particles far
// from the obstacle.  No counterpart in the reference: the map query stays
// the fallback inside the skin band and the judge of the network's error.
//
// Network: inputs (x, y, z) normalised to the obstacle box, optionally with a
// one-hot shape code; `layers` hidden SiLU layers of width `hidden`; one
// linear output, the distance divided by outScale.  Parameters, FP32, in one
// vector: W0 [H][D], b0 [H], then per further hidden layer W [H][H], b [H],
// then wOut [H], bOut.  Weight matrices are row-major [out][in].
//
//  * training (FP32): kSdfTrain runs forward and backward for tiles of 16
//    samples per CTA with the weights and every activation in shared memory
//    and the weight gradients in registers; kSdfReduce adds the CTAs' sums and
//    applies Adam;
//  * inference (BF16 weights and activations, FP32 accumulate): kSdfInfer
//    and the culled integrate give each CTA 128 points.  The first layer
//    (3 or 11 inputs) and the output layer run on the CUDA cores; each H x H
//    hidden layer is one tcgen05.mma chain (M = 128 points, N = H, K = H in
//    steps of 16) from shared-memory operands into a TMEM accumulator, read
//    back with tcgen05.ld for the bias + SiLU epilogue, which writes the next
//    layer's operand tile.
#include <cuda_bf16.h>

#include <atomic>
#include <cmath>
#include <cstring>
#include <vector>

#include "fcdem_map.cuh"

namespace fcdem {
namespace {

constexpr int kSdfMaxInputs = 16;  // 3 coordinates + up to 13 shape codes
constexpr unsigned kSdfWaitLimit = 1u << 22;

struct SdfLayout {
  int D, H, L;              // inputs, width, hidden layers (1..3)
  unsigned w0, b0;          // first layer
  unsigned wh[2], bh[2];    // further hidden layers 1 .. L-1
  unsigned wo, bo;          // output layer
  unsigned total;
};

SdfLayout makeLayout(int D, int H, int L) {
  SdfLayout s{};
  s.D = D;
  s.H = H;
  s.L = L;
  unsigned o = 0;
  s.w0 = o;
  o += (unsigned)(H * D);
  s.b0 = o;
  o += (unsigned)H;
  for (int l = 1; l < L; ++l) {
    s.wh[l - 1] = o;
    o += (unsigned)(H * H);
    s.bh[l - 1] = o;
    o += (unsigned)H;
  }
  s.wo = o;
  o += (unsigned)H;
  s.bo = o;
  o += 1;
  s.total = o;
  return s;
}

// What the kernels read of a network.
struct SdfView {
  SdfLayout lay;
  const float *p;                // parameters
  const __nv_bfloat16 *__restrict__ w16;  // hidden layers 1..L-1, tensor-core tiles
  float shift[3], scale[3], outScale;
};

__device__ __forceinline__ float sigm(float z) { return 1.0f / (1.0f + expf(-z)); }
__device__ __forceinline__ float silu(float z) { return z * sigm(z); }
// Inference SiLU: silu(z) = h + h tanh(h) with h = z / 2, the hardware
// tanh approximation (one special-function op; relative error about 2^-11,
// near the bf16 rounding of the activations it feeds).  The culling
// threshold is calibrated on this arithmetic (the prediction the kernels
// make), so its error is part of what the exact map judges.  The kernels hold
// every weight and bias of a SiLU layer halved -- an exact scaling, all sums
// round as before -- so their layers give h itself.
__device__ __forceinline__ float tanhApprox(float x) {
  float y;
  asm("tanh.approx.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
// silu of two halved arguments
__device__ __forceinline__ f32x2 siluHalf2(f32x2 h) {
  float a, b;
  unpack2(h, a, b);
  return fma2(h, pack2(tanhApprox(a), tanhApprox(b)), h);
}
__device__ __forceinline__ float dsilu(float z) {
  const float s = sigm(z);
  return s * (1.0f + z * (1.0f - s));
}

// splitmix64 stream: value number k of stream `seed`
__device__ __forceinline__ unsigned long long mix64(unsigned long long z) {
  z = (z ^ (z >> 30)) * 0xbf58476d1ce4e5b9ull;
  z = (z ^ (z >> 27)) * 0x94d049bb133111ebull;
  return z ^ (z >> 31);
}
__device__ __forceinline__ float uniform01(unsigned long long seed, unsigned long long k) {
  return (float)(mix64(seed + 0x9e3779b97f4a7c15ull * (k + 1)) >> 40) * (1.0f / 16777216.0f);
}

// ---------------------------------------------------------------------------
// Training samples: (x, y, z, d) with d the map's trilinear distance
// (queryMap, the value the boundary test uses).  Sample t < nNear is drawn
// until |d| < band (at most 64 draws; the last draw is kept otherwise), the
// others uniformly in the map box.
__global__ void __launch_bounds__(256)
kSdfSamples(MapView M, float4 *__restrict__ out, int *__restrict__ shapeOut, int shape,
            unsigned n, unsigned nNear, float band, unsigned long long seed) {
  const unsigned t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= n) return;
  const int tries = t < nNear ? 64 : 1;
  float3 q = make_float3(0.0f, 0.0f, 0.0f);
  float d = 0.0f;
  for (int a = 0; a < tries; ++a) {
    const unsigned long long k = ((unsigned long long)t * 64u + (unsigned)a) * 3u;
    q = make_float3(M.vmin.x + (M.vmax.x - M.vmin.x) * uniform01(seed, k),
                    M.vmin.y + (M.vmax.y - M.vmin.y) * uniform01(seed, k + 1),
                    M.vmin.z + (M.vmax.z - M.vmin.z) * uniform01(seed, k + 2));
    float3 cp;
    d = queryMap(M, q, cp);
    if (fabsf(d) < band) break;
  }
  out[t] = make_float4(q.x, q.y, q.z, d);
  if (shapeOut) shapeOut[t] = shape;
}

// ---------------------------------------------------------------------------
// Training: forward (+ backward) of kTrainS samples per CTA at a time.
//
// A mini-batch of the obstacle networks is a few thousand samples, 0.1 GFLOP:
// what bounds it is how many SMs it reaches and the latency of its chain of
// layers, so a tile is small (16 samples; a batch of 2,048 is 128 CTAs) and 4 H
// threads share it, four outputs of one sample each.  The hidden layers'
// weights sit in shared memory row-major [out][in], rows padded by four floats:
// the forward product reads rows j, j + H/4, ... (lanes on consecutive rows)
// and the backward one the columns of a row (lanes on consecutive 16-byte
// words), both without bank conflicts.  Each thread keeps its 4 x 4 blocks of
// the weight gradients in registers over the CTA's tiles; the CTA's sums go to
// its row of `partial`, and kSdfReduce adds the rows in order (no atomics: the
// same bits every time; the loss alone is summed sample by sample).  3 -> 64 ->
// 64 -> 64 -> 1, batches of 2,048 samples: 17 us a batch against 67 us with
// tiles of 64 samples (32 CTAs), weights read from L2 and a gradient added with
// 277,000 atomics.  In large batches the eight warps of a width-64 CTA leave the
// SM idle in every layer's latency, and two CTAs share it (kCtas, 128 registers a
// thread): one batch of 262,144 samples, two layers, 460 against 598 us, three layers
// 783 against 981.  That is from 16 tiles per SM on; smaller batches keep the order of
// their sums.  (With a tile each the registers' spills cost more: two layers, 32
// batches of 2,048 samples 457 against 353 us.)
constexpr int kTrainS = 16;

// Floats of one row of gradient sums: the parameters, rounded up to 16 bytes
// (every hidden layer's weights start on 16 bytes in it).
__host__ __device__ constexpr unsigned partialRow(unsigned total) { return (total + 3u) & ~3u; }

template <int H, int L>
struct TrainSmem {
  static constexpr int kRow = H + 4;
  float w[L - 1][H][kRow];                 // hidden layers, [out][in]
  float z[L][kTrainS][kRow];               // pre-activations
  float a[L][kTrainS][kRow];               // activations
  float d[2][kTrainS][kRow];               // deltas
  float x[kTrainS][kSdfMaxInputs];
  float w0[kSdfMaxInputs][H];              // first layer, [in][out]
  float b[L][H], wo[H];
  float dy[kTrainS];
};

// Sample s of a tile is samples[base + s]: input (x - shift) * scale and the
// one-hot shape code, target d / outScale, weight 1 + 9 [|d| < band].
// kBackward: the CTA's sums of invB * the gradient of sum_s w (y - t)^2 go to
// partial[blockIdx.x] and the loss terms are added to *lossSum; otherwise
// writes the distance prediction to yOut.
template <int H, int L, bool kBackward, int kCtas>
__global__ void __launch_bounds__(4 * H, kCtas)
kSdfTrain(SdfView net, const float4 *samples, const int *shapes,
          unsigned n, float band, float invB, float *partial,
          float *lossSum, float *yOut) {
  extern __shared__ __align__(1024) unsigned char smraw[];
  TrainSmem<H, L> &sm = *reinterpret_cast<TrainSmem<H, L> *>(smraw);
  constexpr int T = 4 * H, S = kTrainS, Q = H / 4;
  constexpr int kBlocks = Q * Q / T;  // 4 x 4 weight-gradient blocks per thread and layer
  const SdfLayout &ly = net.lay;
  const int D = ly.D;
  const int t = threadIdx.x;
  const int row = t / Q, col = t % Q;  // this thread's sample and column group
  chainTrigger();
  const unsigned tiles = (n + S - 1) / S;
  // thread t < 256 stages input t % 16 of sample t / 16, read one tile ahead
  auto input = [&](unsigned tile) {
    const int s = t / kSdfMaxInputs, d = t % kSdfMaxInputs;
    const unsigned idx = tile * S + s;
    float v = 0.0f;
    if (tile < tiles && t < S * kSdfMaxInputs && idx < n && d < D) {
      const float4 q = __ldg(samples + idx);
      if (d < 3)
        v = ((d == 0 ? q.x : (d == 1 ? q.y : q.z)) - net.shift[d]) * net.scale[d];
      else
        v = (shapes && __ldg(shapes + idx) == d - 3) ? 1.0f : 0.0f;
    }
    return v;
  };
  float x0 = input(blockIdx.x);
  chainWait();  // the weights
#pragma unroll 1
  for (int l = 1; l < L; ++l) {  // (the layers' weights start on 16 bytes: widths of 64 or 128)
    const float4 *src = reinterpret_cast<const float4 *>(net.p + ly.wh[l - 1]);
#pragma unroll 4
    for (int e = t; e < H * Q; e += T)
      *reinterpret_cast<float4 *>(&sm.w[l - 1][e / Q][4 * (e % Q)]) = src[e];
  }
  for (int e = t; e < H * D; e += T) sm.w0[e / H][e % H] = net.p[ly.w0 + (e % H) * D + e / H];
  if (t < H) {
    sm.b[0][t] = net.p[ly.b0 + t];
    for (int l = 1; l < L; ++l) sm.b[l][t] = net.p[ly.bh[l - 1] + t];
    sm.wo[t] = net.p[ly.wo + t];
  }
  const float bo = net.p[ly.bo];
  // gradient sums over the CTA's tiles
  float gW[L - 1][kBlocks][4][4] = {}, gW0[4] = {}, gB[L] = {}, gWo = 0.0f, gBo = 0.0f;
  for (unsigned tile = blockIdx.x; tile < tiles; tile += gridDim.x) {
    const unsigned base = tile * S;
    __syncthreads();  // the weights are in place; the last tile's readers are done
    if (t < S * kSdfMaxInputs) sm.x[t / kSdfMaxInputs][t % kSdfMaxInputs] = x0;
    __syncthreads();
    x0 = input(tile + gridDim.x);
    float act[4];  // this thread's activations of the layer
    {  // first layer
      float acc[4];
#pragma unroll
      for (int u = 0; u < 4; ++u) acc[u] = sm.b[0][col + Q * u];
      for (int k = 0; k < D; ++k) {
        const float x = sm.x[row][k];
#pragma unroll
        for (int u = 0; u < 4; ++u) acc[u] = fmaf(x, sm.w0[k][col + Q * u], acc[u]);
      }
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        sm.z[0][row][col + Q * u] = acc[u];
        act[u] = silu(acc[u]);
        sm.a[0][row][col + Q * u] = act[u];
      }
    }
#pragma unroll
    for (int l = 1; l < L; ++l) {
      __syncthreads();
      float acc[4];
#pragma unroll
      for (int u = 0; u < 4; ++u) acc[u] = sm.b[l][col + Q * u];
#pragma unroll 4
      for (int k = 0; k < H; k += 4) {
        const float4 x = *reinterpret_cast<const float4 *>(&sm.a[l - 1][row][k]);
#pragma unroll
        for (int u = 0; u < 4; ++u) {
          const float4 w = *reinterpret_cast<const float4 *>(&sm.w[l - 1][col + Q * u][k]);
          acc[u] = fmaf(x.w, w.w, fmaf(x.z, w.z, fmaf(x.y, w.y, fmaf(x.x, w.x, acc[u]))));
        }
      }
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        sm.z[l][row][col + Q * u] = acc[u];
        act[u] = silu(acc[u]);
        sm.a[l][row][col + Q * u] = act[u];
      }
    }
    // output layer, loss and its derivative: the Q lanes of a sample share it
    float dy = 0.0f;
    {
      float y = 0.0f;
#pragma unroll
      for (int u = 0; u < 4; ++u) y = fmaf(act[u], sm.wo[col + Q * u], y);
#pragma unroll
      for (int o = Q / 2; o > 0; o >>= 1) y += __shfl_xor_sync(0xffffffffu, y, o);
      y += bo;
      const unsigned idx = base + row;
      if (!kBackward) {
        if (col == 0 && idx < n) yOut[idx] = y * net.outScale;
        continue;
      }
      if (idx < n) {
        const float d = __ldg(&samples[idx].w);
        const float w = fabsf(d) < band ? 10.0f : 1.0f;
        const float r = y - d / net.outScale;
        dy = 2.0f * w * r * invB;
        if (col == 0) atomicAdd(lossSum, w * r * r * invB);
      }
      if (col == 0) sm.dy[row] = dy;
    }
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const int k = col + Q * u;
      sm.d[(L - 1) & 1][row][k] = dy * sm.wo[k] * dsilu(sm.z[L - 1][row][k]);
    }
    __syncthreads();
    if (t < H) {
#pragma unroll 4
      for (int s = 0; s < S; ++s) gWo = fmaf(sm.dy[s], sm.a[L - 1][s][t], gWo);
    }
    if (t == T - 1) {
#pragma unroll 4
      for (int s = 0; s < S; ++s) gBo += sm.dy[s];
    }
#pragma unroll
    for (int l = L - 1; l >= 1; --l) {
      if (l < L - 1) __syncthreads();
      const float(*cur)[TrainSmem<H, L>::kRow] = sm.d[l & 1];
      float(*nxt)[TrainSmem<H, L>::kRow] = sm.d[(l - 1) & 1];
      // weight gradient: block e of the layer is rows 4 (e / Q), columns 4 (e % Q)
#pragma unroll
      for (int e = 0; e < kBlocks; ++e) {
        const int j0 = 4 * ((t + e * T) / Q), k0 = 4 * ((t + e * T) % Q);
#pragma unroll 4
        for (int s = 0; s < S; ++s) {
          const float4 dj = *reinterpret_cast<const float4 *>(&cur[s][j0]);
          const float4 ak = *reinterpret_cast<const float4 *>(&sm.a[l - 1][s][k0]);
          const float dv[4] = {dj.x, dj.y, dj.z, dj.w}, av[4] = {ak.x, ak.y, ak.z, ak.w};
#pragma unroll
          for (int u = 0; u < 4; ++u)
#pragma unroll
            for (int v = 0; v < 4; ++v) gW[l - 1][e][u][v] = fmaf(dv[u], av[v], gW[l - 1][e][u][v]);
        }
      }
      if (t < H) {
        float acc = 0.0f;
#pragma unroll 4
        for (int s = 0; s < S; ++s) acc += cur[s][t];
        gB[l] += acc;
      }
      // nxt[row][k] = dsilu * sum_j cur[row][j] W[j][k], four columns from 4 col
      float acc[4] = {};
#pragma unroll 4
      for (int j = 0; j < H; j += 4) {
        const float4 c = *reinterpret_cast<const float4 *>(&cur[row][j]);
        const float cv[4] = {c.x, c.y, c.z, c.w};
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          const float4 w = *reinterpret_cast<const float4 *>(&sm.w[l - 1][j + q][4 * col]);
          acc[0] = fmaf(cv[q], w.x, acc[0]);
          acc[1] = fmaf(cv[q], w.y, acc[1]);
          acc[2] = fmaf(cv[q], w.z, acc[2]);
          acc[3] = fmaf(cv[q], w.w, acc[3]);
        }
      }
#pragma unroll
      for (int u = 0; u < 4; ++u)
        nxt[row][4 * col + u] = acc[u] * dsilu(sm.z[l - 1][row][4 * col + u]);
    }
    __syncthreads();
    // first layer: thread t has output t % H, inputs t / H, t / H + 4, ...
    const float(*d0)[TrainSmem<H, L>::kRow] = sm.d[0];
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const int k = t / H + 4 * u;
      if (k < D)
#pragma unroll 4
        for (int s = 0; s < S; ++s) gW0[u] = fmaf(d0[s][t % H], sm.x[s][k], gW0[u]);
    }
    if (t < H) {
      float acc = 0.0f;
#pragma unroll 4
      for (int s = 0; s < S; ++s) acc += d0[s][t];
      gB[0] += acc;
    }
  }
  if (!kBackward) return;
  float *g = partial + (size_t)blockIdx.x * partialRow(ly.total);
#pragma unroll
  for (int l = 1; l < L; ++l)
#pragma unroll
    for (int e = 0; e < kBlocks; ++e)
#pragma unroll
      for (int u = 0; u < 4; ++u)
        *reinterpret_cast<float4 *>(g + ly.wh[l - 1] + (4 * ((t + e * T) / Q) + u) * H +
                                    4 * ((t + e * T) % Q)) =
            make_float4(gW[l - 1][e][u][0], gW[l - 1][e][u][1], gW[l - 1][e][u][2],
                        gW[l - 1][e][u][3]);
#pragma unroll
  for (int u = 0; u < 4; ++u)
    if (t / H + 4 * u < D) g[ly.w0 + (t % H) * D + t / H + 4 * u] = gW0[u];
  if (t < H) {
    g[ly.b0 + t] = gB[0];
#pragma unroll
    for (int l = 1; l < L; ++l) g[ly.bh[l - 1] + t] = gB[l];
    g[ly.wo + t] = gWo;
  }
  if (t == T - 1) g[ly.bo] = gBo;
}

// Adds the `parts` rows of partial (32 parameters per CTA, the rows shared out
// over its warps, added in a fixed order).  kAdam: one Adam step on the
// parameters; otherwise the sums go to grad.
constexpr int kReduceWarps = 8;
template <bool kAdam>
__global__ void __launch_bounds__(32 * kReduceWarps)
kSdfReduce(const float *partial, unsigned parts, unsigned total, float *p,
           float *grad, float *m, float *v,
           float lr, float b1, float b2, float eps, float c1, float c2) {
  __shared__ float sSum[kReduceWarps][32];
  const unsigned lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
  const unsigned i = blockIdx.x * 32u + lane;
  chainTrigger();
  chainWait();
  float acc = 0.0f, p0 = 0.0f, m0 = 0.0f, v0 = 0.0f;
  if (kAdam && warp == 0 && i < total) {
    p0 = p[i];
    m0 = m[i];
    v0 = v[i];
  }
  if (i < total) {
#pragma unroll 8
    for (unsigned r = warp; r < parts; r += kReduceWarps)
      acc += partial[(size_t)r * partialRow(total) + i];
  }
  sSum[warp][lane] = acc;
  __syncthreads();
  if (warp != 0 || i >= total) return;
#pragma unroll
  for (int w = 1; w < kReduceWarps; ++w) acc += sSum[w][lane];
  if (!kAdam) {
    grad[i] = acc;
  } else {
    const float mi = b1 * m0 + (1.0f - b1) * acc;
    const float vi = b2 * v0 + (1.0f - b2) * acc * acc;
    m[i] = mi;
    v[i] = vi;
    p[i] = p0 - lr * (mi * c1) / (sqrtf(vi * c2) + eps);
  }
}

// ---------------------------------------------------------------------------
// Tensor-core inference.
//
// Operand tiles in shared memory, K-major, no swizzle: 8-row x 16-byte core
// matrices; element (row r, k) of a tile with R rows at byte
//   (k / 8) * (R * 16) + r * 16 + (k % 8) * 2,
// so the core matrices adjacent in K are R * 16 bytes apart (the descriptor's
// leading byte offset) and those adjacent in rows 128 bytes apart (its stride
// byte offset).  A: R = 128 points; B: R = H outputs of a hidden layer.
// The accumulator D[m][n] (FP32) sits in TMEM lane m, column n.

__host__ __device__ constexpr unsigned tileOffset(int r, int k, int R) {
  return (unsigned)((k / 8) * (R * 8) + r * 8 + (k % 8));  // in bf16 elements
}

__device__ __forceinline__ unsigned smemU32(const void *p) {
  return (unsigned)__cvta_generic_to_shared(p);
}

// Shared-memory matrix descriptor: start address, leading / stride byte
// offsets (16-byte units), descriptor version 1, no swizzle.
__device__ __forceinline__ unsigned long long umDesc(unsigned addr, unsigned lbo,
                                                     unsigned sbo) {
  return (unsigned long long)((addr & 0x3FFFFu) >> 4) |
         ((unsigned long long)((lbo >> 4) & 0x3FFFu) << 16) |
         ((unsigned long long)((sbo >> 4) & 0x3FFFu) << 32) | (1ull << 46);
}

// Instruction descriptor of kind::f16: FP32 accumulator, BF16 A and B, both
// K-major, shape M x N.
__host__ __device__ constexpr unsigned umIdesc(int M, int N) {
  return (1u << 4) | (1u << 7) | (1u << 10) | ((unsigned)(N >> 3) << 17) |
         ((unsigned)(M >> 4) << 24);
}

__device__ __forceinline__ void tmemAlloc(unsigned dstSmem, unsigned cols) {
  asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(dstSmem),
               "r"(cols)
               : "memory");
}
__device__ __forceinline__ void tmemRelinquish() {
  asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmemDealloc(unsigned taddr, unsigned cols) {
  asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(cols)
               : "memory");
}
__device__ __forceinline__ void tcFenceBefore() {
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
}
__device__ __forceinline__ void tcFenceAfter() {
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
}
__device__ __forceinline__ void proxyFence() {
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
}
__device__ __forceinline__ void umma(unsigned dTmem, unsigned long long a, unsigned long long b,
                                     unsigned idesc, unsigned accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}" ::"r"(dTmem),
      "l"(a), "l"(b), "r"(idesc), "r"(accumulate)
      : "memory");
}
__device__ __forceinline__ void ummaCommit(unsigned mbar) {
  asm volatile(
      "tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(mbar)
      : "memory");
}
__device__ __forceinline__ void mbarInit1(unsigned mbar) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(mbar) : "memory");
}
__device__ __forceinline__ bool mbarWaitParity(unsigned mbar, unsigned parity) {
  for (unsigned k = 0; k < kSdfWaitLimit; ++k) {
    unsigned done;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(done)
        : "r"(mbar), "r"(parity)
        : "memory");
    if (done) return true;
  }
  return false;
}
// 16 consecutive FP32 columns of this thread's TMEM lane
__device__ __forceinline__ void tmemLoad16(unsigned taddr, float (&r)[16]) {
  unsigned u[16];
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 "
      "{%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
      : "=r"(u[0]), "=r"(u[1]), "=r"(u[2]), "=r"(u[3]), "=r"(u[4]), "=r"(u[5]), "=r"(u[6]),
        "=r"(u[7]), "=r"(u[8]), "=r"(u[9]), "=r"(u[10]), "=r"(u[11]), "=r"(u[12]),
        "=r"(u[13]), "=r"(u[14]), "=r"(u[15])
      : "r"(taddr)
      : "memory");
#pragma unroll
  for (int c = 0; c < 16; ++c) r[c] = __uint_as_float(u[c]);
}
__device__ __forceinline__ void tmemWaitLoad() {
  asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
}

__device__ __forceinline__ unsigned packBf16(float a, float b) {
  const __nv_bfloat16 x = __float2bfloat16_rn(a), y = __float2bfloat16_rn(b);
  return (unsigned)__bfloat16_as_ushort(x) | ((unsigned)__bfloat16_as_ushort(y) << 16);
}

template <int H, int L, int T = 1>
struct SdfTileSmem {
  static_assert(H == 64 || H == 128, "width");
  static_assert(L >= 2 && L <= 3, "hidden layers");
  static_assert(T == 1 || T == 2, "tiles per CTA");
  __nv_bfloat16 a[T * 128 * H];        // activation tiles (A operands), 128 points each
  __nv_bfloat16 w[(L - 1) * H * H];    // hidden-layer weights (B operands), halved
  float w0[kSdfMaxInputs][H];          // first layer, [D][H], halved
  float b[L * H];                      // biases of the hidden layers, halved
  float wo[H];
  float bo;
  unsigned tmem;
  unsigned long long bar[T];           // one per tile
};

// Per-CTA set-up of the tile forward: TMEM columns (H per tile), the
// barrier, the weights.  All threads of the CTA.
template <int H, int L, int T = 1>
__device__ __forceinline__ void sdfTileSetup(SdfTileSmem<H, L, T> &sm, const SdfView &net) {
  const int t = threadIdx.x;
  if (t < 32) {
    tmemAlloc(smemU32(&sm.tmem), H * T);
    tmemRelinquish();
  }
  if (t == 0) {
    for (int k = 0; k < T; ++k) mbarInit1(smemU32(&sm.bar[k]));
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  const uint4 *src = reinterpret_cast<const uint4 *>(net.w16);
  uint4 *dst = reinterpret_cast<uint4 *>(sm.w);
  for (int e = t; e < (L - 1) * H * H / 8; e += blockDim.x) dst[e] = __ldg(src + e);
  const SdfLayout &ly = net.lay;
  for (int e = t; e < H * ly.D; e += blockDim.x)
    sm.w0[e / H][e % H] = 0.5f * __ldg(net.p + ly.w0 + (e % H) * ly.D + e / H);
  for (int e = t; e < H; e += blockDim.x) {
    sm.b[e] = 0.5f * __ldg(net.p + ly.b0 + e);
    for (int l = 1; l < L; ++l) sm.b[l * H + e] = 0.5f * __ldg(net.p + ly.bh[l - 1] + e);
    sm.wo[e] = __ldg(net.p + ly.wo + e);
  }
  if (t == 0) sm.bo = __ldg(net.p + ly.bo);
  proxyFence();
  tcFenceBefore();
  __syncthreads();
  tcFenceAfter();
}

template <int H, int L, int T = 1>
__device__ __forceinline__ void sdfTileTeardown(SdfTileSmem<H, L, T> &sm) {
  tcFenceBefore();
  __syncthreads();
  if (threadIdx.x < 32) {
    tcFenceAfter();
    tmemDealloc(sm.tmem, H * T);
  }
}

// Barrier of one tile's 128 threads, and the same with an OR over them.  (The
// barrier's number is an immediate: a register would reserve all 16.)
template <int T>
__device__ __forceinline__ void tileSync(int tile) {
  if (T == 1)
    __syncthreads();
  else if (tile == 0)
    asm volatile("barrier.cta.sync 1, 128;" ::: "memory");
  else
    asm volatile("barrier.cta.sync 2, 128;" ::: "memory");
}
template <int kId>
__device__ __forceinline__ bool barrierOr(bool v) {
  unsigned r;
  asm volatile(
      "{\n\t.reg .pred p, q;\n\t"
      "setp.ne.u32 p, %1, 0;\n\t"
      "barrier.cta.red.or.pred q, %2, 128, p;\n\t"
      "selp.u32 %0, 1, 0, q;\n\t}"
      : "=r"(r)
      : "r"((unsigned)v), "n"(kId)
      : "memory");
  return r != 0u;
}
template <int T>
__device__ __forceinline__ bool tileSyncOr(int tile, bool v) {
  if (T == 1) return __syncthreads_or(v);
  return tile == 0 ? barrierOr<1>(v) : barrierOr<2>(v);
}

// The distance prediction for this thread's point (x normalised, shape code
// `shape` or -1); 128 * T threads, one point each, all threads of a tile.
// Thread t works on tile t / 128, row t % 128: the tile's A operand is its
// own 128-row block of sm.a and its accumulator TMEM columns tile * H ..,
// read by the warp's lane quarter (warp % 4).  The tiles of a CTA share the
// weights only; each has its barrier, MMA chain and commit, so that one's
// products overlap with another's activations.  `phase` is the tile's mbarrier
// parity, flipped per layer.  Returns false (for every thread of the tile)
// when an MMA chain did not complete in time.
//
// Bound by the special-function unit: a tanh.approx keeps it for 15 cycles per
// warp (measured: 192 of them per point of 3-64-64-64-1, 77% active over the
// kernel's 91 us per 1M points, so 70 us at best).  Everything else is kept out
// of its way: biases, the SiLU's multiply-add and the output product work on
// packed pairs, weights are halved once instead of every argument, the first
// layer's weights lie [input][output] for 16-byte loads: 112 us per call
// against 120 (43% issue active).
template <int H, int L, int kLdBatch = 1, int T = 1>
__device__ __forceinline__ bool sdfTileForward(SdfTileSmem<H, L, T> &sm, const SdfView &net,
                                               float x0, float x1, float x2, int shape,
                                               unsigned &phase, float &dOut) {
  const int t = threadIdx.x, warp = t >> 5;
  const int tile = t >> 7, row = t & 127, quarter = warp & 3;
  __nv_bfloat16 *aTile = sm.a + tile * 128 * H;
  const unsigned bar = smemU32(&sm.bar[tile]);
  const bool coded = shape >= 0 && 3 + shape < net.lay.D;
  // four consecutive floats of shared memory as two pairs
  auto four = [](const float *p) { return *reinterpret_cast<const ulonglong2 *>(p); };
  auto packed = [](f32x2 v) {
    float a, b;
    unpack2(v, a, b);
    return packBf16(a, b);
  };
  // first layer on the CUDA cores, 8 outputs per 16-byte chunk of the A row
  const f32x2 xx0 = pack2(x0, x0), xx1 = pack2(x1, x1), xx2 = pack2(x2, x2);
#pragma unroll 1
  for (int c = 0; c < H / 8; ++c) {
    unsigned v[4];
#pragma unroll
    for (int u = 0; u < 2; ++u) {
      const int j = c * 8 + u * 4;
      ulonglong2 z = four(sm.b + j);
      const ulonglong2 w0 = four(&sm.w0[0][j]), w1 = four(&sm.w0[1][j]), w2 = four(&sm.w0[2][j]);
      z.x = fma2(w2.x, xx2, fma2(w1.x, xx1, fma2(w0.x, xx0, z.x)));
      z.y = fma2(w2.y, xx2, fma2(w1.y, xx1, fma2(w0.y, xx0, z.y)));
      if (coded) {
        const ulonglong2 ws = four(&sm.w0[3 + shape][j]);
        z.x = add2(z.x, ws.x);
        z.y = add2(z.y, ws.y);
      }
      v[2 * u] = packed(siluHalf2(z.x));
      v[2 * u + 1] = packed(siluHalf2(z.y));
    }
    *reinterpret_cast<uint4 *>(aTile + tileOffset(row, c * 8, 128)) =
        make_uint4(v[0], v[1], v[2], v[3]);
  }
  proxyFence();
  tcFenceBefore();
  tileSync<T>(tile);
  const unsigned idesc = umIdesc(128, H);
  f32x2 y = pack2(sm.bo, 0.0f);
  bool ok = true;
#pragma unroll 1
  for (int l = 1; l < L; ++l) {
    if (row == 0) {
      tcFenceAfter();
      const unsigned aBase = smemU32(aTile), bBase = smemU32(sm.w + (l - 1) * H * H);
#pragma unroll
      for (int s = 0; s < H / 16; ++s)
        umma(sm.tmem + (unsigned)(tile * H), umDesc(aBase + s * 2 * 128 * 16, 128 * 16, 128),
             umDesc(bBase + s * 2 * H * 16, H * 16, 128), idesc, s > 0 ? 1u : 0u);
      ummaCommit(bar);
    }
    const bool done = mbarWaitParity(bar, phase);
    phase ^= 1u;
    if (tileSyncOr<T>(tile, !done)) {
      // let the chain finish (bounded) before the tile buffers are reused
      mbarWaitParity(bar, phase ^ 1u);
      ok = false;
      break;
    }
    tcFenceAfter();
    const bool last = (l == L - 1);
    // kLdBatch column chunks of 16 are read from TMEM before one wait (more
    // loads in flight, more registers: the standalone inference kernel uses
    // 4, the fused culling kernels, which hold a particle's state, 1)
    static_assert((H / 16) % kLdBatch == 0, "column chunks per batch");
#pragma unroll 1
    for (int c0 = 0; c0 < H / 16; c0 += kLdBatch) {
      float r[kLdBatch][16];
#pragma unroll
      for (int q = 0; q < kLdBatch; ++q)
        tmemLoad16(sm.tmem + ((unsigned)(32 * quarter) << 16) +
                       (unsigned)(tile * H + (c0 + q) * 16),
                   r[q]);
      tmemWaitLoad();
#pragma unroll
      for (int q = 0; q < kLdBatch; ++q) {
        const int c = (c0 + q) * 16;
#pragma unroll
        for (int h = 0; h < 2; ++h) {  // eight columns at a time
          unsigned v[4];
#pragma unroll
          for (int u = 0; u < 2; ++u) {
            const int k = 8 * h + 4 * u;
            const ulonglong2 b = four(sm.b + l * H + c + k);
            const f32x2 s0 = siluHalf2(add2(pack2(r[q][k], r[q][k + 1]), b.x));
            const f32x2 s1 = siluHalf2(add2(pack2(r[q][k + 2], r[q][k + 3]), b.y));
            if (last) {
              const ulonglong2 w = four(sm.wo + c + k);
              y = fma2(s1, w.y, fma2(s0, w.x, y));
            } else {
              v[2 * u] = packed(s0);
              v[2 * u + 1] = packed(s1);
            }
          }
          if (!last)
            *reinterpret_cast<uint4 *>(aTile + tileOffset(row, c + 8 * h, 128)) =
                make_uint4(v[0], v[1], v[2], v[3]);
        }
      }
    }
    tcFenceBefore();
    if (!last) proxyFence();
    tileSync<T>(tile);
  }
  float ya, yb;
  unpack2(y, ya, yb);
  dOut = (ya + yb) * net.outScale;
  return ok;
}

// d[i] for point i (float4, w ignored) with shape code shapes[i] (or none).
// kInferTiles 128-point tiles per CTA share the weights; inferLd<H>() TMEM
// column loads are in flight per wait.
constexpr int kInferTiles = 2;
template <int H> constexpr int inferLd() { return H == 64 ? 2 : 4; }
template <int H, int L>
__global__ void __launch_bounds__(128 * kInferTiles)
kSdfInfer(SdfView net, const float4 *__restrict__ pts, const int *__restrict__ shapes,
          unsigned n, float *__restrict__ dOut, DeviceStatus *status) {
  extern __shared__ __align__(1024) unsigned char smraw[];
  SdfTileSmem<H, L, kInferTiles> &sm =
      *reinterpret_cast<SdfTileSmem<H, L, kInferTiles> *>(smraw);
  sdfTileSetup<H, L, kInferTiles>(sm, net);
  unsigned phase = 0;
  const unsigned groups = (n + 128u * kInferTiles - 1) / (128u * kInferTiles);
  for (unsigned g = blockIdx.x; g < groups; g += gridDim.x) {
    const unsigned i = g * 128u * kInferTiles + threadIdx.x;
    const bool valid = i < n;
    const float4 q = valid ? __ldg(pts + i) : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    const int shape = (valid && shapes) ? __ldg(shapes + i) : -1;
    float d = 0.0f;
    if (!sdfTileForward<H, L, inferLd<H>(), kInferTiles>(
            sm, net, (q.x - net.shift[0]) * net.scale[0], (q.y - net.shift[1]) * net.scale[1],
            (q.z - net.shift[2]) * net.scale[2], shape, phase, d)) {
      if ((threadIdx.x & 127u) == 0) report(status, kStatusTimeout);
      break;
    }
    if (valid) dOut[i] = d;
  }
  sdfTileTeardown<H, L, kInferTiles>(sm);
}

// Per-tile hints of the culling kernels (performance only: results never
// depend on them).  h[tile] = 1 when, the last time the network ran on the
// tile, more than half of its in-box particles still needed the exact query;
// such a tile then queries the map directly, without the network, until a
// refresh step (every kHintRefresh steps) runs the network on every tile
// again.  h == nullptr: the network runs on every tile with a particle in
// the map box.
constexpr unsigned kHintRefresh = 8;
struct TileHints {
  unsigned char *h;
  int refresh;
};

// Culling per tile (fcdemSdfSetTileCulling).  The network runs once per
// tile of kCullTile consecutive slots, at the centre c of the box that
// bounds the tile's particles in the map box (after this step's velocity
// and position update), and the tile's exact queries are skipped when
// pred(c) - lip * rho > skin, rho being the distance from c to the box's
// corners.  With lip a Lipschitz bound of the network's prediction, every
// particle p of such a tile has pred(p) >= pred(c) - lip * |p - c| > skin:
// the per-particle rule would have skipped it as well.  Where the rule
// does not cull, every particle of the tile in the map box is queried.  A
// tile whose particles in the map box belong to scenes of different
// obstacles is not culled.
constexpr unsigned kCullTile = 32;
struct TileCull {
  const float4 *centre;  // per tile: c (x, y, z) and rho (w)
  const int *shape;      // per tile: the obstacle's shape code; -1 none in the box, -2 mixed
  const float *pred;     // per tile: the network's distance at c
  float lip, skin;
  __device__ __forceinline__ bool cull(unsigned tile) const {
    return __ldg(shape + tile) >= 0 &&
           __ldg(pred + tile) - lip * __ldg(&centre[tile].w) > skin;
  }
};

// One warp per tile: the bounding box of the tile's advanced positions in
// the map box (umAdvance: the arithmetic of the integrate that follows).
// kBatch: slot i belongs to scene sceneOf[i] with its own parameters and
// obstacle; otherwise every particle has kp and the map M.
template <bool kBatch>
__global__ void __launch_bounds__(256)
kTileCentres(const BatchScene *__restrict__ scenes, const unsigned *__restrict__ sceneOf,
             const MapView *__restrict__ maps, KParams kp, MapView M,
             const float4 *__restrict__ pos, const float4 *__restrict__ vel, float dt,
             unsigned n, float4 *__restrict__ centre, int *__restrict__ shapeOut) {
  const unsigned lane = threadIdx.x & 31u;
  const unsigned tile = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const unsigned tiles = (n + kCullTile - 1) / kCullTile;
  if (tile >= tiles) return;  // whole warps leave together
  const unsigned i = tile * kCullTile + lane;
  bool in = false;
  int shape = -1;
  float3 p = make_float3(0.0f, 0.0f, 0.0f);
  if (i < n) {
    const float4 p4 = __ldg(pos + i), v4 = __ldg(vel + i);
    p = make_float3(p4.x, p4.y, p4.z);
    float3 v = make_float3(v4.x, v4.y, v4.z);
    if (kBatch) {
      const BatchScene &S = scenes[__ldg(sceneOf + i)];
      umAdvance(p, v, dt, S.p);
      shape = S.shape;
      in = shape >= 0 && inMapBox(maps[shape], p);
    } else {
      umAdvance(p, v, dt, kp.p);
      shape = 0;
      in = inMapBox(M, p);
    }
  }
  const float inf = __int_as_float(0x7f800000);
  float lx = in ? p.x : inf, ly = in ? p.y : inf, lz = in ? p.z : inf;
  float hx = in ? p.x : -inf, hy = in ? p.y : -inf, hz = in ? p.z : -inf;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    lx = fminf(lx, __shfl_xor_sync(0xffffffffu, lx, o));
    ly = fminf(ly, __shfl_xor_sync(0xffffffffu, ly, o));
    lz = fminf(lz, __shfl_xor_sync(0xffffffffu, lz, o));
    hx = fmaxf(hx, __shfl_xor_sync(0xffffffffu, hx, o));
    hy = fmaxf(hy, __shfl_xor_sync(0xffffffffu, hy, o));
    hz = fmaxf(hz, __shfl_xor_sync(0xffffffffu, hz, o));
  }
  const int smin = __reduce_min_sync(0xffffffffu, in ? shape : 0x7fffffff);
  const int smax = __reduce_max_sync(0xffffffffu, in ? shape : -1);
  if (lane == 0) {
    if (smax < 0) {
      centre[tile] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
      shapeOut[tile] = -1;
    } else {
      const float ex = hx - lx, ey = hy - ly, ez = hz - lz;
      // rho with a margin for the roundings of the centre and of the root
      const float rho = 0.5f * sqrtf(ex * ex + ey * ey + ez * ez) * 1.0001f + 1e-6f;
      centre[tile] = make_float4(0.5f * (lx + hx), 0.5f * (ly + hy), 0.5f * (lz + hz), rho);
      shapeOut[tile] = smin == smax ? smin : -2;
    }
  }
}

// kIntegrateDistMap's step with the map query of culled tiles skipped.
template <bool kCount>
__global__ void __launch_bounds__(256)
kIntegrateTileCull(float4 *__restrict__ pos, float4 *__restrict__ vel, float dt, unsigned n,
                   KParams kp, MapView M, TileCull tc, unsigned *exact,
                   unsigned *__restrict__ hashOut, unsigned *__restrict__ rankOut,
                   unsigned *__restrict__ cnt, unsigned *__restrict__ tileCnt) {
  const unsigned i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const SimParams &P = kp.p;
  const float4 p4 = pos[i], v4 = vel[i];
  float3 p = make_float3(p4.x, p4.y, p4.z), v = make_float3(v4.x, v4.y, v4.z);
  const float r = kp.radiusFromW ? p4.w : P.particleRadius;
  umAdvance(p, v, dt, P);
  const bool test = inMapBox(M, p) && !tc.cull(i / kCullTile);
  if (test && exact) atomicAdd(exact, 1u);
  umBoundary(M, test, r, P.boundaryDamping, p, v);
  if (kCount) {  // the next step's calcHash and cell count
    const int3 gp = gridPos(p.x, p.y, p.z, P);
    const unsigned h = gridHash(gp.x, gp.y, gp.z, P);
    hashOut[i] = h;
    rankOut[i] = atomicAdd(cnt + h, 1u);
    countTile(tileCnt, h >> 12);
  }
  pos[i] = make_float4(p.x, p.y, p.z, p4.w);
  vel[i] = make_float4(v.x, v.y, v.z, p4.w);
}

// d_integrateSystem + d_checkBoundaryDistMap (kIntegrateDistMap's
// arithmetic) with the map query skipped where the network predicts a
// distance above `skin`: a point outside the map box reads 5.0 from the map
// and is never tested; inside, the exact query runs only when the prediction
// is at most `skin`.  `exact` (optional) counts the exact queries.  kCount:
// also the next step's calcHash and cell count (counting-sort pipeline).
template <int H, int L, bool kCount>
__global__ void __launch_bounds__(128)
kIntegrateSdf(float4 *__restrict__ pos, float4 *__restrict__ vel, float dt, unsigned n,
              KParams kp, MapView M, SdfView net, float skin, unsigned *exact,
              unsigned *__restrict__ hashOut, unsigned *__restrict__ rankOut,
              unsigned *__restrict__ cnt, unsigned *__restrict__ tileCnt, TileHints hints,
              DeviceStatus *status) {
  extern __shared__ __align__(1024) unsigned char smraw[];
  SdfTileSmem<H, L> &sm = *reinterpret_cast<SdfTileSmem<H, L> *>(smraw);
  sdfTileSetup<H, L>(sm, net);
  const SimParams &P = kp.p;
  unsigned phase = 0;
  const unsigned tiles = (n + 127) / 128;
  for (unsigned tile = blockIdx.x; tile < tiles; tile += gridDim.x) {
    const unsigned i = tile * 128 + threadIdx.x;
    const bool valid = i < n;
    float4 p4 = make_float4(0.0f, 0.0f, 0.0f, 0.0f), v4 = p4;
    if (valid) {
      p4 = pos[i];
      v4 = vel[i];
    }
    float3 p = make_float3(p4.x, p4.y, p4.z), v = make_float3(v4.x, v4.y, v4.z);
    const float r = kp.radiusFromW ? p4.w : P.particleRadius;
    umAdvance(p, v, dt, P);
    const bool inBox = valid && inMapBox(M, p);
    float dPred = 0.0f;
    // a tile with no particle in the map box needs no prediction (the map
    // reads 5.0 outside its box); the decisions are the same for every thread
    const bool anyIn = __syncthreads_or(inBox);
    const bool useNet = anyIn && (!hints.h || hints.refresh || hints.h[tile] == 0);
    if (useNet &&
        !sdfTileForward<H, L>(sm, net, (p.x - net.shift[0]) * net.scale[0],
                              (p.y - net.shift[1]) * net.scale[1],
                              (p.z - net.shift[2]) * net.scale[2], 0, phase, dPred)) {
      if (threadIdx.x == 0) report(status, kStatusTimeout);
      break;
    }
    const bool test = inBox && (!useNet || !(dPred > skin));
    if (useNet && hints.h) {
      const int nIn = __syncthreads_count(inBox), nTest = __syncthreads_count(test);
      if (threadIdx.x == 0) hints.h[tile] = 2 * nTest > nIn ? 1 : 0;
    }
    if (!valid) continue;
    if (test && exact) atomicAdd(exact, 1u);
    umBoundary(M, test, r, P.boundaryDamping, p, v);
    if (kCount) {  // the next step's calcHash and cell count
      const int3 gp = gridPos(p.x, p.y, p.z, P);
      const unsigned h = gridHash(gp.x, gp.y, gp.z, P);
      hashOut[i] = h;
      rankOut[i] = atomicAdd(cnt + h, 1u);
      countTile(tileCnt, h >> 12);
    }
    pos[i] = make_float4(p.x, p.y, p.z, p4.w);
    vel[i] = make_float4(v.x, v.y, v.z, p4.w);
  }
  sdfTileTeardown<H, L>(sm);
}

// integrateOneBox's clamp to the scene box, same faces in the same order,
// the roundings spelled out.
__device__ __forceinline__ void boxClamp(float3 &p, float3 &v, float r, float bd,
                                         const float *lo, const float *hi) {
  if (p.x > hi[0] - r) { p.x = hi[0] - r; v.x = __fmul_rn(v.x, bd); }
  if (p.x < lo[0] + r) { p.x = lo[0] + r; v.x = __fmul_rn(v.x, bd); }
  if (p.y > hi[1] - r) { p.y = hi[1] - r; v.y = __fmul_rn(v.y, bd); }
  if (p.z > hi[2] - r) { p.z = hi[2] - r; v.z = __fmul_rn(v.z, bd); }
  if (p.z < lo[2] + r) { p.z = lo[2] + r; v.z = __fmul_rn(v.z, bd); }
  if (p.y < lo[1] + r) { p.y = lo[1] + r; v.y = __fmul_rn(v.y, bd); }
}

// Batch integrate with obstacles: particle / slot i belongs to scene
// sceneOf[i]; the velocity and position update, the contact of the scene's
// obstacle map (checkDistMap), the clamp to the scene's box, and with
// doCount the next global cell id and count.  kNet: a tile of 128 with a
// particle in its obstacle's map box runs the network (the scene's shape as
// the one-hot code) and only particles predicted within `skin` query the map.
// Without kNet, tc (when set) holds the decisions of the culling per tile.
template <int H, int L, bool kNet, bool kW>
__global__ void __launch_bounds__(128)
kBatchObstacle(const BatchScene *__restrict__ scenes, const unsigned *__restrict__ sceneOf,
               const MapView *__restrict__ maps, SdfView net, float skin,
               const float4 *__restrict__ inPos, float4 *__restrict__ pos,
               float4 *__restrict__ vel, float dt, unsigned n, UmCount count, int doCount,
               unsigned *exact, TileHints hints, TileCull tc, DeviceStatus *status) {
  extern __shared__ __align__(1024) unsigned char smraw[];
  SdfTileSmem<H, L> &sm = *reinterpret_cast<SdfTileSmem<H, L> *>(smraw);
  if (kNet) sdfTileSetup<H, L>(sm, net);
  unsigned phase = 0;
  const unsigned tiles = (n + 127) / 128;
  for (unsigned tile = blockIdx.x; tile < tiles; tile += gridDim.x) {
    const unsigned i = tile * 128 + threadIdx.x;
    const bool valid = i < n;
    const BatchScene *S = valid ? scenes + __ldg(sceneOf + i) : scenes;
    const SimParams &P = S->p;
    float4 p4 = make_float4(0.0f, 0.0f, 0.0f, 0.0f), v4 = p4;
    if (valid) {
      p4 = inPos[i];
      v4 = vel[i];
    }
    float3 p = make_float3(p4.x, p4.y, p4.z), v = make_float3(v4.x, v4.y, v4.z);
    const float r = kW ? p4.w : P.particleRadius;
    umAdvance(p, v, dt, P);
    const int shape = valid ? S->shape : -1;
    MapView M{};
    if (shape >= 0) M = maps[shape];
    const bool inBox = shape >= 0 && inMapBox(M, p);
    float dPred = 0.0f;
    bool useNet = false;
    if (kNet) {
      const bool anyIn = __syncthreads_or(inBox);
      useNet = anyIn && (!hints.h || hints.refresh || hints.h[tile] == 0);
      if (useNet &&
          !sdfTileForward<H, L>(sm, net, (p.x - net.shift[0]) * net.scale[0],
                                (p.y - net.shift[1]) * net.scale[1],
                                (p.z - net.shift[2]) * net.scale[2], shape, phase, dPred)) {
        if (threadIdx.x == 0) report(status, kStatusTimeout);
        break;
      }
    }
    // without the network in the kernel: the tiles' decisions (TileCull), if any
    const bool test = inBox && (!useNet || !(dPred > skin)) &&
                      (kNet || !tc.shape || !tc.cull(i / kCullTile));
    if (kNet && useNet && hints.h) {
      const int nIn = __syncthreads_count(inBox), nTest = __syncthreads_count(test);
      if (threadIdx.x == 0) hints.h[tile] = 2 * nTest > nIn ? 1 : 0;
    }
    if (!valid) continue;
    if (test) {
      if (exact) atomicAdd(exact, 1u);
      checkDistMap(M, r, P.boundaryDamping, p, v);
    }
    boxClamp(p, v, r, P.boundaryDamping, S->lo, S->hi);
    pos[i] = make_float4(p.x, p.y, p.z, p4.w);
    vel[i] = make_float4(v.x, v.y, v.z, v4.w);
    if (doCount) {
      const int3 gp = gridPos(p.x, p.y, p.z, P);
      const unsigned h = S->cellBase + gridHash(gp.x, gp.y, gp.z, P);
      count.hash[i] = h;
      count.rank[i] = atomicAdd(count.cnt + h, 1u);
      countTile(count.tileCnt, h >> 12);
    }
  }
  if (kNet) sdfTileTeardown<H, L>(sm);
}

// Hidden-layer weights, FP32 [out][in], halved (siluHalf2), to the BF16
// B-operand tiles.
__global__ void __launch_bounds__(256)
kSdfPackBf16(const float *__restrict__ p, SdfLayout ly, __nv_bfloat16 *__restrict__ w16) {
  const int H = ly.H;
  const unsigned per = (unsigned)(H * H);
  const unsigned total = per * (unsigned)(ly.L - 1);
  for (unsigned e = blockIdx.x * blockDim.x + threadIdx.x; e < total;
       e += gridDim.x * blockDim.x) {
    const unsigned l = e / per, r = e % per;
    const int o = (int)(r / H), k = (int)(r % H);
    w16[l * per + tileOffset(o, k, H)] = __float2bfloat16_rn(0.5f * p[ly.wh[l] + r]);
  }
}

}  // namespace
}  // namespace fcdem

using namespace fcdem;

struct fcdemSdfNet {
  int device = -1;
  SdfLayout lay{};
  float shift[3] = {0.0f, 0.0f, 0.0f}, scale[3] = {1.0f, 1.0f, 1.0f}, outScale = 1.0f;
  float *params = nullptr, *grad = nullptr, *m = nullptr, *v = nullptr;
  float *loss = nullptr;  // one device float
  float *partial = nullptr;  // kSdfTrain: rows of gradient sums (first training call)
  __nv_bfloat16 *w16 = nullptr;
  bool w16Fresh = false;
  unsigned adamStep = 0;
  unsigned version = 0;  // bumped whenever the weights or the normalisation change
  unsigned char *hints = nullptr;  // per-tile culling hints (TileHints)
  unsigned hintTiles = 0;
  float tileLip = 0.0f;          // > 0: cull per tile of kCullTile slots (TileCull)
  void *tileBuf = nullptr;       // TileCull's centres, shapes and predictions
  unsigned tileCap = 0;          // tiles tileBuf holds
};

namespace fcdem {
namespace {

bool shapeOk(int D, int H, int L) {
  return D >= 3 && D <= kSdfMaxInputs && (H == 64 || H == 128) && L >= 2 && L <= 3;
}

SdfView sdfView(const fcdemSdfNet *net) {
  SdfView v;
  v.lay = net->lay;
  v.p = net->params;
  v.w16 = net->w16;
  for (int k = 0; k < 3; ++k) {
    v.shift[k] = net->shift[k];
    v.scale[k] = net->scale[k];
  }
  v.outScale = net->outScale;
  return v;
}

void freeNet(fcdemSdfNet *net) {
  if (!net) return;
  cudaFree(net->params);
  cudaFree(net->grad);
  cudaFree(net->m);
  cudaFree(net->v);
  cudaFree(net->loss);
  cudaFree(net->partial);
  cudaFree(net->w16);
  cudaFree(net->hints);
  cudaFree(net->tileBuf);
  delete net;
}

bool uploadParams(fcdemSdfNet *net, const std::vector<float> &p) {
  const size_t bytes = sizeof(float) * p.size();
  net->w16Fresh = false;
  net->version++;
  return uploadNow(net->params, p.data(), bytes);
}

template <int H, int L>
size_t tileSmemBytes() {
  return sizeof(SdfTileSmem<H, L>) + 1024;  // + alignment slack
}

// Opts a kernel into its dynamic shared memory, once per device (a bit each).
template <class Kernel>
bool smemReady(Kernel *kernel, int bytes, std::atomic<unsigned long long> &ready) {
  int dev = 0;
  if (!cudaOk(cudaGetDevice(&dev))) return false;
  const unsigned long long bit = 1ull << (dev & 63);
  if (ready.load(std::memory_order_relaxed) & bit) return true;
  if (!cudaOk(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes)))
    return false;
  ready.fetch_or(bit, std::memory_order_relaxed);
  return true;
}

bool packWeights(fcdemSdfNet *net) {
  if (net->w16Fresh) return true;
  kSdfPackBf16<<<64, 256, 0, curStream()>>>(net->params, net->lay, net->w16);
  if (!launchOk()) return false;
  net->w16Fresh = true;
  return true;
}

// Runs the forward (+ backward) tile kernel over n samples; parts receives
// the rows of net->partial that the backward pass wrote.  chained: the kernel
// before it on the stream is this call's own.
bool runTrainKernel(fcdemSdfNet *net, bool backward, const float4 *samples, const int *shapes,
                    unsigned n, float band, float invB, float *yOut, unsigned *parts = nullptr,
                    bool chained = false) {
  const unsigned sms = numSms();
  const int H = net->lay.H, L = net->lay.L;
  const unsigned rows = H == 64 ? 2u * sms : sms;  // CTAs of a backward pass at most
  if (backward && !net->partial &&
      cudaMalloc(&net->partial, sizeof(float) * (size_t)rows * partialRow(net->lay.total)) !=
          cudaSuccess) {
    cudaGetLastError();
    net->partial = nullptr;
    setError(FCDEM_ERR_ALLOC);
    return false;
  }
  const SdfView v = sdfView(net);
  const unsigned tiles = (n + kTrainS - 1) / kTrainS;
  // one CTA per SM, two of the narrow ones forward and in large batches (kTrainS)
  const bool two = H == 64 && tiles > 16u * sms;
  const unsigned most = H == 64 && (!backward || two) ? 2u * sms : sms;
  const unsigned blocks = tiles < most ? tiles : most;
  if (parts) *parts = blocks;
#define FCDEM_SDF_TRAIN(HH, LL)                                                               \
  if (H == HH && L == LL) {                                                                   \
    constexpr int smem = (int)sizeof(TrainSmem<HH, LL>);                                      \
    static_assert(smem <= 227 * 1024, "shared memory of a CTA");                              \
    if (backward && two) {                                                                    \
      static std::atomic<unsigned long long> ready{0};                                        \
      constexpr int kCtas = HH == 64 ? 2 : 1;                                                 \
      if (!smemReady(kSdfTrain<HH, LL, true, kCtas>, smem, ready)) return false;              \
      launchChained(chained, kSdfTrain<HH, LL, true, kCtas>, blocks, 4 * HH, smem, v,         \
                    samples, shapes, n, band, invB, net->partial, net->loss, nullptr);        \
    } else if (backward) {                                                                    \
      static std::atomic<unsigned long long> ready{0};                                        \
      if (!smemReady(kSdfTrain<HH, LL, true, 1>, smem, ready)) return false;                  \
      launchChained(chained, kSdfTrain<HH, LL, true, 1>, blocks, 4 * HH, smem, v, samples,    \
                    shapes, n, band, invB, net->partial, net->loss, nullptr);                 \
    } else {                                                                                  \
      static std::atomic<unsigned long long> ready{0};                                        \
      if (!smemReady(kSdfTrain<HH, LL, false, 1>, smem, ready)) return false;                 \
      launchChained(false, kSdfTrain<HH, LL, false, 1>, blocks, 4 * HH, smem, v, samples,     \
                    shapes, n, band, invB, nullptr, nullptr, yOut);                           \
    }                                                                                         \
    return launchOk();                                                                        \
  }
  FCDEM_SDF_TRAIN(64, 3)
  FCDEM_SDF_TRAIN(64, 2)
  FCDEM_SDF_TRAIN(128, 2)
  FCDEM_SDF_TRAIN(128, 3)
#undef FCDEM_SDF_TRAIN
  setError(FCDEM_ERR_INVALID_VALUE);
  return false;
}

// The batch gradient (lr < 0) or one Adam step from the rows of net->partial.
bool reducePartials(fcdemSdfNet *net, unsigned parts, float lr) {
  const unsigned total = net->lay.total, blocks = (total + 31u) / 32u;
  const float b1 = 0.9f, b2 = 0.999f, eps = 1e-8f;
  if (lr < 0.0f) {
    launchChained(
        true, kSdfReduce<false>, blocks, 32 * kReduceWarps, 0, net->partial, parts, total, net->params, net->grad, net->m, net->v, 0.0f, b1,
        b2, eps, 0.0f, 0.0f);
    return launchOk();
  }
  net->adamStep++;
  net->version++;
  const double t = (double)net->adamStep;
  const float c1 = (float)(1.0 / (1.0 - std::pow((double)b1, t)));
  const float c2 = (float)(1.0 / (1.0 - std::pow((double)b2, t)));
  launchChained(
      true, kSdfReduce<true>, blocks, 32 * kReduceWarps, 0, net->partial, parts, total, net->params, net->grad, net->m, net->v, lr, b1, b2,
      eps, c1, c2);
  net->w16Fresh = false;
  return launchOk();
}

// CTAs per SM that fit both the shared memory (227 KB) and the 512 TMEM
// columns (H per CTA); the persistent grid is the SM count times that.
template <int H, int L>
constexpr unsigned sdfCtasPerSm() {
  constexpr unsigned bySmem = (unsigned)((227u * 1024u) / (sizeof(SdfTileSmem<H, L>) + 1024u));
  constexpr unsigned byTmem = 512u / (unsigned)H;
  return bySmem < byTmem ? bySmem : byTmem;
}

template <int H, int L>
bool launchInfer(fcdemSdfNet *net, const float4 *pts, const int *shapes, unsigned n,
                 float *d) {
  const size_t smem = sizeof(SdfTileSmem<H, L, kInferTiles>) + 1024;  // + alignment slack
  const int threads = 128 * kInferTiles;
  // persistent grid: the CTAs that are resident at once (registers, shared
  // memory), capped by the 512 TMEM columns of an SM (H per tile): a CTA
  // beyond that would wait in tcgen05.alloc for columns no CTA frees.
  // Worked out once per device (the attribute calls cost more host time
  // than a launch).
  static int residentOf[64] = {};
  int dev = 0;
  if (!cudaOk(cudaGetDevice(&dev))) return false;
  if (dev < 0 || dev >= 64) dev = 0;
  int resident = residentOf[dev];
  if (resident == 0) {
    // the whole carveout as shared memory
    if (!cudaOk(cudaFuncSetAttribute(kSdfInfer<H, L>,
                                     cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem)) ||
        !cudaOk(cudaFuncSetAttribute(kSdfInfer<H, L>,
                                     cudaFuncAttributePreferredSharedMemoryCarveout,
                                     (int)cudaSharedmemCarveoutMaxShared)))
      return false;
    cudaFuncAttributes fa;
    if (!cudaOk(cudaFuncGetAttributes(&fa, kSdfInfer<H, L>))) return false;
    // registers are allocated per warp in units of 256
    const int regsPerWarp = ((fa.numRegs * 32 + 255) / 256) * 256;
    const int byRegs = regsPerWarp > 0 ? (65536 / regsPerWarp) / (threads / 32) : 1;
    const int bySmem = (int)((227u * 1024u) / (smem + 1024u));  // + the per-CTA reserve
    const int byTmem = 512 / (H * kInferTiles);
    resident = byRegs < bySmem ? byRegs : bySmem;
    if (resident > byTmem) resident = byTmem;
    if (resident < 1) resident = 1;
    residentOf[dev] = resident;
  }
  unsigned grid = (n + 128u * kInferTiles - 1) / (128u * kInferTiles);
  if (grid > numSms() * (unsigned)resident) grid = numSms() * (unsigned)resident;
  kSdfInfer<H, L><<<grid, threads, smem, curStream()>>>(sdfView(net), pts, shapes, n, d,
                                                        ctx().dStatus);
  return launchOk();
}

template <int H, int L>
bool launchIntegrateSdf(fcdemSdfNet *net, float4 *pos, float4 *vel, float dt, unsigned n,
                        const KParams &kp, const MapView &M, float skin, unsigned *exact,
                        const UmCount *count, TileHints hints) {
  const size_t smem = tileSmemBytes<H, L>();
  unsigned grid = (n + 127) / 128;
  if (grid > numSms() * sdfCtasPerSm<H, L>()) grid = numSms() * sdfCtasPerSm<H, L>();
  if (count) {
    cudaFuncSetAttribute(kIntegrateSdf<H, L, true>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                         (int)smem);
    kIntegrateSdf<H, L, true><<<grid, 128, smem, curStream()>>>(
        pos, vel, dt, n, kp, M, sdfView(net), skin, exact, count->hash, count->rank, count->cnt,
        count->tileCnt, hints, ctx().dStatus);
  } else {
    cudaFuncSetAttribute(kIntegrateSdf<H, L, false>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                         (int)smem);
    kIntegrateSdf<H, L, false><<<grid, 128, smem, curStream()>>>(
        pos, vel, dt, n, kp, M, sdfView(net), skin, exact, nullptr, nullptr, nullptr, nullptr,
        hints, ctx().dStatus);
  }
  return launchOk();
}

template <int H, int L, bool kNet, bool kW>
bool launchBatchObstacle(fcdemSdfNet *net, const BatchScene *scenes, const unsigned *sceneOf,
                         const MapView *maps, float skin, const float4 *inPos, float4 *pos,
                         float4 *vel, float dt, unsigned n, const UmCount *count,
                         unsigned *exact, TileHints hints, TileCull tc = TileCull{}) {
  unsigned grid = (n + 127) / 128;
  size_t smem = 0;
  SdfView v{};
  if (kNet) {
    smem = tileSmemBytes<H, L>();
    cudaFuncSetAttribute(kBatchObstacle<H, L, kNet, kW>,
                         cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (grid > numSms() * sdfCtasPerSm<H, L>()) grid = numSms() * sdfCtasPerSm<H, L>();
    v = sdfView(net);
  }
  kBatchObstacle<H, L, kNet, kW><<<grid, 128, smem, curStream()>>>(
      scenes, sceneOf, maps, v, skin, inPos, pos, vel, dt, n, count ? *count : UmCount{},
      count ? 1 : 0, exact, hints, tc, ctx().dStatus);
  return launchOk();
}

}  // namespace
}  // namespace fcdem

namespace fcdem {

unsigned sdfVersion(const fcdemSdfNet *net) { return net ? net->version : 0u; }

// The net's hint array for `tiles` tiles (grown on demand, cleared when
// grown); nullptr (no hints) when it cannot be had.
unsigned char *sdfHints(fcdemSdfNet *net, unsigned tiles) {
  if (net->hints && net->hintTiles >= tiles) return net->hints;
  if (!cudaOk(cudaDeviceSynchronize())) return nullptr;
  cudaFree(net->hints);
  net->hints = nullptr;
  net->hintTiles = 0;
  if (cudaMalloc(&net->hints, tiles) != cudaSuccess) {
    cudaGetLastError();
    net->hints = nullptr;
    return nullptr;
  }
  if (!clearNow(net->hints, 0, tiles)) return nullptr;
  net->hintTiles = tiles;
  return net->hints;
}

// The net's per-tile arrays of the culling per tile, for n slots (grown on
// demand); nullptr when they cannot be had.
bool sdfTileBuffers(fcdemSdfNet *net, unsigned n, TileCull &tc) {
  const unsigned tiles = (n + kCullTile - 1) / kCullTile;
  if (!net->tileBuf || net->tileCap < tiles) {
    if (!cudaOk(cudaDeviceSynchronize())) return false;
    cudaFree(net->tileBuf);
    net->tileBuf = nullptr;
    net->tileCap = 0;
    if (cudaMalloc(&net->tileBuf, (size_t)tiles * 24) != cudaSuccess) {
      cudaGetLastError();
      setError(FCDEM_ERR_ALLOC);
      return false;
    }
    net->tileCap = tiles;
  }
  float4 *centre = (float4 *)net->tileBuf;
  int *shape = (int *)(centre + net->tileCap);
  float *pred = (float *)(shape + net->tileCap);
  tc = TileCull{centre, shape, pred, net->tileLip, 0.0f};
  return true;
}

bool sdfPrepareTiles(fcdemSdfNet *net, unsigned n) {
  TileCull tc{};
  return !net || !(net->tileLip > 0.0f) || n == 0 || sdfTileBuffers(net, n, tc);
}

// The tiles' centres and the network's predictions there (culling per tile).
template <bool kBatch>
bool tileDecisions(fcdemSdfNet *net, const BatchScene *scenes, const unsigned *sceneOf,
                   const MapView *maps, const KParams &kp, const MapView &M,
                   const float4 *inPos, const float4 *vel, float dt, unsigned n, float skin,
                   TileCull &tc) {
  if (!sdfTileBuffers(net, n, tc)) return false;
  tc.skin = skin;
  const unsigned tiles = (n + kCullTile - 1) / kCullTile;
  kTileCentres<kBatch><<<(tiles * 32 + 255) / 256, 256, 0, curStream()>>>(
      scenes, sceneOf, maps, kp, M, inPos, vel, dt, n, const_cast<float4 *>(tc.centre),
      const_cast<int *>(tc.shape));
  if (!launchOk()) return false;
  // the shape codes go to the network too (a negative code: no one-hot input)
  const int *shapes = kBatch ? tc.shape : nullptr;
  const int H = net->lay.H, L = net->lay.L;
  float *pred = const_cast<float *>(tc.pred);
  if (H == 64 && L == 3) return launchInfer<64, 3>(net, tc.centre, shapes, tiles, pred);
  if (H == 64 && L == 2) return launchInfer<64, 2>(net, tc.centre, shapes, tiles, pred);
  if (H == 128 && L == 2) return launchInfer<128, 2>(net, tc.centre, shapes, tiles, pred);
  if (H == 128 && L == 3) return launchInfer<128, 3>(net, tc.centre, shapes, tiles, pred);
  setError(FCDEM_ERR_INVALID_VALUE);
  return false;
}

bool batchObstacleIntegrate(const BatchScene *scenes, const unsigned *sceneOf, bool radiusFromW,
                            const MapView *maps, fcdemSdfNet *net, float skin,
                            const float4 *inPos, float4 *pos, float4 *vel, float dt,
                            unsigned n, const UmCount *count, unsigned *exact, unsigned step) {
  if (n == 0) return true;
  if (net && net->tileLip > 0.0f) {
    if (!packWeights(net)) return false;
    TileCull tc{};
    if (!tileDecisions<true>(net, scenes, sceneOf, maps, KParams{}, MapView{}, inPos, vel, dt,
                             n, skin, tc))
      return false;
    const TileHints none{nullptr, 1};
    return radiusFromW
               ? launchBatchObstacle<64, 3, false, true>(net, scenes, sceneOf, maps, skin, inPos,
                                                         pos, vel, dt, n, count, exact, none, tc)
               : launchBatchObstacle<64, 3, false, false>(net, scenes, sceneOf, maps, skin,
                                                          inPos, pos, vel, dt, n, count, exact,
                                                          none, tc);
  }
  if (!net) {
    const TileHints none{nullptr, 1};
    return radiusFromW
               ? launchBatchObstacle<64, 3, false, true>(net, scenes, sceneOf, maps, skin, inPos,
                                                         pos, vel, dt, n, count, exact, none)
               : launchBatchObstacle<64, 3, false, false>(net, scenes, sceneOf, maps, skin,
                                                          inPos, pos, vel, dt, n, count, exact,
                                                          none);
  }
  if (!packWeights(net)) return false;
  const TileHints hints{sdfHints(net, (n + 127) / 128), step % kHintRefresh == 0 ? 1 : 0};
  const int H = net->lay.H, L = net->lay.L;
#define FCDEM_BATCH_OBST(HH, LL)                                                             \
  if (H == HH && L == LL)                                                                    \
    return radiusFromW ? launchBatchObstacle<HH, LL, true, true>(net, scenes, sceneOf, maps, \
                                                                 skin, inPos, pos, vel, dt,  \
                                                                 n, count, exact, hints)     \
                       : launchBatchObstacle<HH, LL, true, false>(                           \
                             net, scenes, sceneOf, maps, skin, inPos, pos, vel, dt, n,       \
                             count, exact, hints);
  FCDEM_BATCH_OBST(64, 3)
  FCDEM_BATCH_OBST(64, 2)
  FCDEM_BATCH_OBST(128, 2)
  FCDEM_BATCH_OBST(128, 3)
#undef FCDEM_BATCH_OBST
  setError(FCDEM_ERR_INVALID_VALUE);
  return false;
}

bool sdfIntegrate(fcdemSdfNet *net, float4 *pos, float4 *vel, float dt, unsigned n,
                  const KParams &kp, const fcdemDistanceMap *map, float skin, unsigned *exact,
                  const UmCount *count, int step) {
  if (!packWeights(net)) return false;
  const int H = net->lay.H, L = net->lay.L;
  const MapView M = view(map);
  if (net->tileLip > 0.0f) {
    if (n == 0) return true;
    TileCull tc{};
    if (!tileDecisions<false>(net, nullptr, nullptr, nullptr, kp, M, pos, vel, dt, n, skin, tc))
      return false;
    const unsigned blocks = (n + 255) / 256;
    if (count)
      kIntegrateTileCull<true><<<blocks, 256, 0, curStream()>>>(
          pos, vel, dt, n, kp, M, tc, exact, count->hash, count->rank, count->cnt,
          count->tileCnt);
    else
      kIntegrateTileCull<false><<<blocks, 256, 0, curStream()>>>(
          pos, vel, dt, n, kp, M, tc, exact, nullptr, nullptr, nullptr, nullptr);
    return launchOk();
  }
  // step < 0: a lone call, no hints
  const TileHints hints{step < 0 ? nullptr : sdfHints(net, (n + 127) / 128),
                        (step < 0 || step % (int)kHintRefresh == 0) ? 1 : 0};
  if (H == 64 && L == 3) return launchIntegrateSdf<64, 3>(net, pos, vel, dt, n, kp, M, skin, exact, count, hints);
  if (H == 64 && L == 2) return launchIntegrateSdf<64, 2>(net, pos, vel, dt, n, kp, M, skin, exact, count, hints);
  if (H == 128 && L == 2) return launchIntegrateSdf<128, 2>(net, pos, vel, dt, n, kp, M, skin, exact, count, hints);
  if (H == 128 && L == 3) return launchIntegrateSdf<128, 3>(net, pos, vel, dt, n, kp, M, skin, exact, count, hints);
  setError(FCDEM_ERR_INVALID_VALUE);
  return false;
}

}  // namespace fcdem

extern "C" {

fcdemSdfNet *fcdemSdfCreate(int inputs, int hidden, int hiddenLayers, unsigned long long seed) {
  if (!shapeOk(inputs, hidden, hiddenLayers)) {
    setError(FCDEM_ERR_INVALID_VALUE);
    return nullptr;
  }
  ctx();
  fcdemSdfNet *net = new fcdemSdfNet();
  cudaGetDevice(&net->device);
  net->lay = makeLayout(inputs, hidden, hiddenLayers);
  const size_t bytes = sizeof(float) * net->lay.total;
  const size_t w16 = sizeof(__nv_bfloat16) * (size_t)(hiddenLayers - 1) * hidden * hidden;
  bool ok = cudaMalloc(&net->params, bytes) == cudaSuccess &&
            cudaMalloc(&net->grad, bytes) == cudaSuccess &&
            cudaMalloc(&net->m, bytes) == cudaSuccess && cudaMalloc(&net->v, bytes) == cudaSuccess &&
            cudaMalloc(&net->loss, sizeof(float)) == cudaSuccess &&
            cudaMalloc(&net->w16, w16) == cudaSuccess;
  if (!ok) {
    cudaGetLastError();
    setError(FCDEM_ERR_ALLOC);
    freeNet(net);
    return nullptr;
  }
  // uniform initialisation, bound sqrt(6 / fan_in) (weights), zero biases
  std::vector<float> p(net->lay.total, 0.0f);
  unsigned long long z = seed;
  auto next = [&z]() {
    z += 0x9e3779b97f4a7c15ull;
    unsigned long long x = z;
    x = (x ^ (x >> 30)) * 0xbf58476d1ce4e5b9ull;
    x = (x ^ (x >> 27)) * 0x94d049bb133111ebull;
    x ^= x >> 31;
    return (double)(x >> 11) * (1.0 / 9007199254740992.0);
  };
  const SdfLayout &ly = net->lay;
  auto fill = [&](unsigned off, unsigned count, int fanIn) {
    const double bound = std::sqrt(6.0 / (double)fanIn);
    for (unsigned k = 0; k < count; ++k) p[off + k] = (float)((2.0 * next() - 1.0) * bound);
  };
  fill(ly.w0, (unsigned)(ly.H * ly.D), 3);
  for (int l = 1; l < ly.L; ++l) fill(ly.wh[l - 1], (unsigned)(ly.H * ly.H), ly.H);
  fill(ly.wo, (unsigned)ly.H, ly.H);
  if (!uploadParams(net, p) || !clearNow(net->m, 0, bytes) || !clearNow(net->v, 0, bytes)) {
    freeNet(net);
    return nullptr;
  }
  return net;
}

void fcdemSdfDestroy(fcdemSdfNet *net) { freeNet(net); }

uint fcdemSdfNumParams(const fcdemSdfNet *net) { return net ? net->lay.total : 0u; }

void fcdemSdfGetParams(const fcdemSdfNet *net, float *host) {
  if (!net || !host) { setError(FCDEM_ERR_INVALID_VALUE); return; }
  downloadNow(host, net->params, sizeof(float) * net->lay.total);
}

void fcdemSdfSetParams(fcdemSdfNet *net, const float *host) {
  if (!net || !host) { setError(FCDEM_ERR_INVALID_VALUE); return; }
  std::vector<float> p(host, host + net->lay.total);
  uploadParams(net, p);
}

void fcdemSdfSetNormalization(fcdemSdfNet *net, const float shift[3], const float scale[3],
                              float outScale) {
  if (!net || !shift || !scale || !(outScale > 0.0f)) {
    setError(FCDEM_ERR_INVALID_VALUE);
    return;
  }
  for (int k = 0; k < 3; ++k) {
    net->shift[k] = shift[k];
    net->scale[k] = scale[k];
  }
  net->outScale = outScale;
  net->version++;
}

void fcdemSdfSetTileCulling(fcdemSdfNet *net, float lipschitz) {
  if (!net || !(lipschitz >= 0.0f)) {
    setError(FCDEM_ERR_INVALID_VALUE);
    return;
  }
  net->tileLip = lipschitz;
  net->version++;  // a recorded batch graph holds the launches of the other mode
}

void fcdemSdfGetNormalization(const fcdemSdfNet *net, float shift[3], float scale[3],
                              float *outScale) {
  if (!net) { setError(FCDEM_ERR_INVALID_VALUE); return; }
  for (int k = 0; k < 3; ++k) {
    if (shift) shift[k] = net->shift[k];
    if (scale) scale[k] = net->scale[k];
  }
  if (outScale) *outScale = net->outScale;
}

void fcdemSdfSamples(const fcdemDistanceMap *map, int shape, uint n, float nearFraction,
                     float band, unsigned long long seed, float *samples4, int *shapes) {
  if (!map || (n && !samples4) || !(nearFraction >= 0.0f && nearFraction <= 1.0f)) {
    setError(FCDEM_ERR_INVALID_VALUE);
    return;
  }
  if (n == 0) return;
  const unsigned nNear = (unsigned)((double)n * nearFraction);
  kSdfSamples<<<(n + 255) / 256, 256, 0, curStream()>>>(view(map), (float4 *)samples4, shapes,
                                                        shape, n, nNear, band, seed);
  launchOk();
}

float fcdemSdfGradient(fcdemSdfNet *net, const float *samples4, const int *shapes, uint n,
                       float band, float *gradHost) {
  if (!net || !samples4 || n == 0) { setError(FCDEM_ERR_INVALID_VALUE); return 0.0f; }
  const size_t bytes = sizeof(float) * net->lay.total;
  if (!cudaOk(cudaMemsetAsync(net->loss, 0, sizeof(float), curStream()))) return 0.0f;
  unsigned parts = 0;
  if (!runTrainKernel(net, true, (const float4 *)samples4, shapes, n, band, 1.0f / (float)n,
                      nullptr, &parts) ||
      !reducePartials(net, parts, -1.0f))
    return 0.0f;
  float loss = 0.0f;
  downloadNow(&loss, net->loss, sizeof(float));
  if (gradHost) downloadNow(gradHost, net->grad, bytes);
  return loss;
}

float fcdemSdfTrainSamples(fcdemSdfNet *net, const float *samples4, const int *shapes, uint n,
                           uint epochs, uint batch, float lr, float band) {
  if (!net || !samples4 || n == 0 || batch == 0 || epochs == 0) {
    setError(FCDEM_ERR_INVALID_VALUE);
    return 0.0f;
  }
  const unsigned batches = (n + batch - 1) / batch;
  const unsigned total = batches * epochs;
  float last = 0.0f;
  for (unsigned e = 0; e < epochs; ++e) {
    if (!cudaOk(cudaMemsetAsync(net->loss, 0, sizeof(float), curStream()))) return 0.0f;
    for (unsigned b = 0; b < batches; ++b) {
      const unsigned off = b * batch;
      const unsigned cnt = (n - off) < batch ? (n - off) : batch;
      // cosine decay to lr / 20 over the whole run
      const double prog = (double)(e * batches + b) / (double)total;
      const float lrNow =
          (float)(lr * (0.05 + 0.95 * 0.5 * (1.0 + std::cos(3.14159265358979 * prog))));
      unsigned parts = 0;
      if (!runTrainKernel(net, true, (const float4 *)samples4 + off, shapes ? shapes + off : nullptr,
                          cnt, band, 1.0f / (float)cnt, nullptr, &parts, e + b > 0) ||
          !reducePartials(net, parts, lrNow))
        return 0.0f;
    }
    if (e + 1 == epochs) {
      downloadNow(&last, net->loss, sizeof(float));
      last /= (float)batches;
    }
  }
  return last;
}

void fcdemSdfEvalF32(fcdemSdfNet *net, const float *points4, const int *shapes, uint n,
                     float *d) {
  if (!net || (n && (!points4 || !d))) { setError(FCDEM_ERR_INVALID_VALUE); return; }
  if (n == 0) return;
  runTrainKernel(net, false, (const float4 *)points4, shapes, n, 0.0f, 0.0f, d);
}

void fcdemSdfInfer(fcdemSdfNet *net, const float *points4, const int *shapes, uint n,
                   float *d) {
  if (!net || (n && (!points4 || !d))) { setError(FCDEM_ERR_INVALID_VALUE); return; }
  if (n == 0) return;
  if (!packWeights(net)) return;
  const int H = net->lay.H, L = net->lay.L;
  if (H == 64 && L == 3) launchInfer<64, 3>(net, (const float4 *)points4, shapes, n, d);
  else if (H == 64 && L == 2) launchInfer<64, 2>(net, (const float4 *)points4, shapes, n, d);
  else if (H == 128 && L == 2) launchInfer<128, 2>(net, (const float4 *)points4, shapes, n, d);
  else if (H == 128 && L == 3) launchInfer<128, 3>(net, (const float4 *)points4, shapes, n, d);
  else setError(FCDEM_ERR_INVALID_VALUE);
}

void fcdemUM_integrateSystemSdf(float *pos, float *vel, float deltaTime, uint numParticles,
                                const fcdemDistanceMap *map, fcdemSdfNet *net, float skin,
                                uint *exactQueries) {
  Context &c = ctx();
  if (!c.haveParams) { setError(FCDEM_ERR_NO_PARAMS); return; }
  if (numParticles == 0) return;
  if (!pos || !vel || !map || !net || !(skin >= 0.0f)) {
    setError(FCDEM_ERR_INVALID_VALUE);
    return;
  }
  sdfIntegrate(net, (float4 *)pos, (float4 *)vel, deltaTime, numParticles, kparams(c), map, skin,
               exactQueries, nullptr, -1);
}

}  // extern "C"
