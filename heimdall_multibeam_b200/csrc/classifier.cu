// classifier.cu -- the learned candidate classifier: a two-branch CNN over a
// candidate's DM-time patch (64 x 64) and frequency-time patch (64 x 256),
// trained and evaluated by BF16 tensor-core GEMMs with FP32 accumulation.
//
// Network (175 666 parameters):
//   branch A (DM-time, 1 x 64 x 64) and branch B (freq-time, 1 x 64 x 256),
//   each: conv3x3(1->8) ReLU maxpool2, conv3x3(8->16) ReLU maxpool2,
//         conv3x3(16->32) ReLU maxpool2   -> A: 32x8x8, B: 32x8x32
//   concat (10240) -> FC 16 ReLU -> FC 2 -> softmax (class 1 = pulse)
// Training runs the convolutions as GEMMs over an im2col matrix on the tensor
// cores (umma.cu): forward (W x col) and the weight gradients (dOut x col^T,
// split over the pixels); the data gradient is a kernel of its own that sums
// the nine taps' products (k_dgrad3, mma.sync m16n8k16).  Inference is one
// fused kernel (k_clf_infer).  All products take BF16 operands (weights rounded
// from FP32 master copies, activations stored in BF16) and accumulate in FP32.
// Adam updates the FP32 master weights.  Activation layout:
// [channel][batch][row][col].
#include <cuda_bf16.h>

#include <algorithm>
#include <cmath>
#include <cstdio>
#include <cstring>
#include <new>
#include <random>
#include <vector>

#include "heimdall_b200.h"
#include "internal.h"

namespace hdb {
namespace clf {

using bf16 = __nv_bfloat16;

// ===========================================================================
// BF16 GEMM, FP32 accumulation: C(m, n) (+)= sum_k A(m, k) B(k, n) with
// element strides A(m, k) = A[m*sam + k*sak], B(k, n) = B[k*sbk + n*sbn],
// C(m, n) = C[m*scm + n*scn].  Block tile 32 x 64 x 32, 4 warps of 16 x 32.
// blockIdx.z splits K into chunks of kchunk; with more than one split the
// partial sums are added atomically (C must hold the initial value).
// ===========================================================================
constexpr int GBM = 32, GBN = 64, GBK = 32, GPAD = 8;

struct GemmArgs {
  int M, N, K;
  const bf16* A;
  long long sam, sak;
  const bf16* B;
  long long sbk, sbn;
  float* C;
  long long scm, scn;
  int accumulate;  // add to C (single split) instead of overwriting
  int kchunk;      // K per blockIdx.z
};

__device__ __forceinline__ void mma_bf16(float* c, const uint32_t* a, const uint32_t* b) {
  asm volatile(
      "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 "
      "{%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};\n"
      : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b[0]), "r"(b[1]));
}

__global__ void __launch_bounds__(128) k_gemm_bf16(GemmArgs g) {
  __shared__ __align__(16) bf16 As[GBM][GBK + GPAD];  // [m][k]
  __shared__ __align__(16) bf16 Bs[GBN][GBK + GPAD];  // [n][k]
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int m0 = blockIdx.y * GBM, n0 = blockIdx.x * GBN;
  const int kb = blockIdx.z * g.kchunk;
  const int ke = min(g.K, kb + g.kchunk);
  const int wm = (warp & 1) * 16, wn = (warp >> 1) * 32;
  const int gr = lane >> 2, tq = lane & 3;
  float acc[4][4];
#pragma unroll
  for (int j = 0; j < 4; j++) acc[j][0] = acc[j][1] = acc[j][2] = acc[j][3] = 0.f;
  const bf16 zero = __float2bfloat16(0.f);
  for (int k0 = kb; k0 < ke; k0 += GBK) {
    // tiles, zero outside the matrix; the faster index follows the unit stride
    for (int e = tid; e < GBM * GBK; e += 128) {
      int m, k;
      if (g.sak == 1) { m = e / GBK; k = e % GBK; } else { k = e / GBM; m = e % GBM; }
      const int gm = m0 + m, gk = k0 + k;
      As[m][k] = (gm < g.M && gk < ke) ? g.A[gm * g.sam + gk * g.sak] : zero;
    }
    for (int e = tid; e < GBN * GBK; e += 128) {
      int n, k;
      if (g.sbn == 1) { k = e / GBN; n = e % GBN; } else { n = e / GBK; k = e % GBK; }
      const int gn = n0 + n, gk = k0 + k;
      Bs[n][k] = (gn < g.N && gk < ke) ? g.B[gk * g.sbk + gn * g.sbn] : zero;
    }
    __syncthreads();
#pragma unroll
    for (int kk = 0; kk < GBK; kk += 16) {
      uint32_t a[4];
      a[0] = *reinterpret_cast<const uint32_t*>(&As[wm + gr][kk + 2 * tq]);
      a[1] = *reinterpret_cast<const uint32_t*>(&As[wm + gr + 8][kk + 2 * tq]);
      a[2] = *reinterpret_cast<const uint32_t*>(&As[wm + gr][kk + 2 * tq + 8]);
      a[3] = *reinterpret_cast<const uint32_t*>(&As[wm + gr + 8][kk + 2 * tq + 8]);
#pragma unroll
      for (int j = 0; j < 4; j++) {
        uint32_t b[2];
        b[0] = *reinterpret_cast<const uint32_t*>(&Bs[wn + 8 * j + gr][kk + 2 * tq]);
        b[1] = *reinterpret_cast<const uint32_t*>(&Bs[wn + 8 * j + gr][kk + 2 * tq + 8]);
        mma_bf16(acc[j], a, b);
      }
    }
    __syncthreads();
  }
  const bool split = gridDim.z > 1;
#pragma unroll
  for (int j = 0; j < 4; j++) {
#pragma unroll
    for (int h = 0; h < 4; h++) {
      const int m = m0 + wm + gr + (h >> 1) * 8;
      const int n = n0 + wn + 8 * j + 2 * tq + (h & 1);
      if (m < g.M && n < g.N) {
        float* c = g.C + m * g.scm + n * g.scn;
        if (split) atomicAdd(c, acc[j][h]);
        else *c = g.accumulate ? *c + acc[j][h] : acc[j][h];
      }
    }
  }
}

cudaError_t gemm(const GemmArgs& a0, int splits, cudaStream_t s) {
  GemmArgs a = a0;
  if (a.M <= 0 || a.N <= 0 || a.K <= 0) return cudaSuccess;
  splits = std::max(1, std::min(splits, (a.K + GBK - 1) / GBK));
  a.kchunk = ((a.K + splits - 1) / splits + GBK - 1) / GBK * GBK;
  splits = (a.K + a.kchunk - 1) / a.kchunk;
  dim3 grid((unsigned)((a.N + GBN - 1) / GBN), (unsigned)((a.M + GBM - 1) / GBM), (unsigned)splits);
  if (grid.y > 65535 || grid.z > 65535) return cudaErrorInvalidValue;
  k_gemm_bf16<<<grid, 128, 0, s>>>(a); note_launch();
  return cudaGetLastError();
}

// ===========================================================================
// Elementwise and layout kernels
// ===========================================================================
__global__ void k_to_bf16(const float* __restrict__ in, bf16* __restrict__ out, size_t n) {
  for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < n;
       i += (size_t)gridDim.x * blockDim.x)
    out[i] = __float2bfloat16(in[i]);
}

// network input: patch values (in units of the row's robust deviation)
// limited to +-kInputClip, so that very bright rows do not saturate training
constexpr float kInputClip = 16.f;
__global__ void k_input_bf16(const float* __restrict__ in, bf16* __restrict__ out, size_t n) {
  for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < n;
       i += (size_t)gridDim.x * blockDim.x)
    out[i] = __float2bfloat16(fminf(fmaxf(in[i], -kInputClip), kInputClip));
}

// weights [co][k] (k < kw) -> BF16 [co][kp], zero columns kw..kp-1
__global__ void k_weights_bf16(const float* __restrict__ w, int co, int kw, int kp,
                               bf16* __restrict__ out) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= co * kp) return;
  const int o = i / kp, k = i % kp;
  out[i] = __float2bfloat16(k < kw ? w[o * kw + k] : 0.f);
}

// im2col of a 3x3, pad-1 convolution: in [ci][b][h][w] -> col [ci*9][b*h*w],
// row c*9 + ky*3 + kx (the weight gradient's operand).  Bound by its writes (9
// values out per value in).  A thread makes the nine taps of eight pixels of
// one image row from three 16-byte loads and their two neighbours, with
// 16-byte stores (w is a multiple of 8): 45 us for 8 x 128 x 32 x 128 values
// against 253 us with one value per thread.
__global__ void __launch_bounds__(256) k_im2col3(const bf16* __restrict__ in, int h, int w,
                                                 size_t P, bf16* __restrict__ col) {
  const size_t p = 8 * ((size_t)blockIdx.x * blockDim.x + threadIdx.x);
  if (p >= P) return;
  const int c = blockIdx.y;
  const int x = (int)(p % w), y = (int)((p / w) % h);
  const uint16_t* src = reinterpret_cast<const uint16_t*>(in) + (size_t)c * P + p;
#pragma unroll
  for (int ky = 0; ky < 3; ky++) {
    const int yy = y + ky - 1;
    uint4 m = make_uint4(0u, 0u, 0u, 0u);
    uint32_t left = 0, right = 0;  // pixel x - 1 in the upper half, x + 8 in the lower
    if (yy >= 0 && yy < h) {
      const uint16_t* r = src + (ptrdiff_t)(ky - 1) * w;
      m = *reinterpret_cast<const uint4*>(r);
      if (x > 0) left = (uint32_t)r[-1] << 16;
      if (x + 8 < w) right = r[8];
    }
    const uint32_t a = __byte_perm(left, m.x, 0x5432), b = __byte_perm(m.x, m.y, 0x5432),
                   d = __byte_perm(m.y, m.z, 0x5432), e = __byte_perm(m.z, m.w, 0x5432),
                   f = __byte_perm(m.w, right, 0x5432);
    bf16* o = col + (size_t)(c * 9 + ky * 3) * P + p;
    *reinterpret_cast<uint4*>(o) = make_uint4(a, b, d, e);
    *reinterpret_cast<uint4*>(o + P) = m;
    *reinterpret_cast<uint4*>(o + 2 * P) = make_uint4(b, d, e, f);
  }
}

// im2col in K-major order for the tensor-core GEMM: colT [b*h*w][KP], the KP
// taps of one output pixel contiguous (tap k = c*9 + ky*3 + kx; zeros from
// ci*9 on).  Bound by its writes.  A thread gathers all taps of one pixel: a
// warp's loads are 32 neighbouring pixels of one tap (with the taps across a
// warp's lanes each load touched about 20 sectors), and every index but the
// pixel's is a constant.  The rows go out through shared memory, pitched by an
// odd number of 16-byte units, so that stores are whole lines: 8 x 128 x 32 x
// 128 values in took 85 us with the taps across lanes, 57 us with each thread
// storing its own row, 26 us so.
template <int CI>
__global__ void __launch_bounds__(128) k_im2col3_t(const bf16* __restrict__ in, int h, int w,
                                                   size_t P, bf16* __restrict__ colT) {
  constexpr int KP = (CI * 9 + 15) / 16 * 16, Q = KP / 8, PITCH = Q | 1;
  __shared__ uint4 rows[128 * PITCH];
  const size_t p0 = (size_t)blockIdx.x * 128, p = p0 + threadIdx.x;
  if (p < P) {
    const int x = (int)(p % w), y = (int)((p / w) % h);
    const uint16_t* src = reinterpret_cast<const uint16_t*>(in) + p;
    bool ok[9];
#pragma unroll
    for (int t = 0; t < 9; t++) {
      const int yy = y + t / 3 - 1, xx = x + t % 3 - 1;
      ok[t] = yy >= 0 && yy < h && xx >= 0 && xx < w;
    }
#pragma unroll
    for (int q = 0; q < Q; q++) {
      uint32_t v[8];
#pragma unroll
      for (int j = 0; j < 8; j++) {
        const int k = 8 * q + j, c = k / 9, t = k % 9;
        v[j] = (k < CI * 9 && ok[t])
                   ? src[(ptrdiff_t)c * (ptrdiff_t)P + (t / 3 - 1) * w + (t % 3 - 1)] : 0u;
      }
      rows[threadIdx.x * PITCH + q] = make_uint4(v[0] | v[1] << 16, v[2] | v[3] << 16,
                                                 v[4] | v[5] << 16, v[6] | v[7] << 16);
    }
  }
  __syncthreads();
  const int n = (int)(P - p0 < 128 ? P - p0 : 128) * Q;
  uint4* out = reinterpret_cast<uint4*>(colT) + p0 * Q;
  for (int e = threadIdx.x; e < n; e += 128) out[e] = rows[e / Q * PITCH + e % Q];
}

// Data gradient of a convolution, straight from the layer's pre-activation
// gradient dz [CO][b][H][W] (BF16) to its input's gradient din [CI][b][H][W]:
// for each tap the product over the output channels (mma.sync m16n8k16, FP32),
// the nine taps added in order, as a GEMM to dcol [CI*9][b*H*W] and a col2im
// did through 168 MB of dcol.  A block takes R rows of one sample and stages
// their dz and a ring of zeros pixel-major in shared memory; a warp's 16 MMA
// rows are 16 neighbouring pixels, read shifted by each tap, and the weights'
// fragments stay in registers.  Bound by dz and din in memory, not by the
// product (K = 16 or 32).  The four layers of a 128-sample step: 354 us for the
// GEMMs and the col2ims, 63 us here (8 -> 16 channels of 32 x 128: 25 us).
template <int CI, int CO, int H, int W, int R>
__global__ void __launch_bounds__(256) k_dgrad3(const bf16* __restrict__ dz,
                                                const bf16* __restrict__ wb, size_t P,
                                                float* __restrict__ din) {
  constexpr int KP = (CI * 9 + 15) / 16 * 16;
  constexpr int NT = CI / 8, KS = CO / 16, PS = CO + 8, Wp = W + 2;
  extern __shared__ __align__(16) uint32_t dg_smem[];  // [R + 2][Wp][PS] BF16
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int g = lane >> 2, t = lane & 3;
  const int n = blockIdx.x / (H / R), y0 = blockIdx.x % (H / R) * R;
  // zero columns left and right; rows outside the image are zeroed below
  for (int e = threadIdx.x; e < (R + 2) * 2 * (PS / 2); e += 256) {
    const int r = e / (PS), o = e % PS;
    dg_smem[(r * Wp + (o < PS / 2 ? 0 : W + 1)) * (PS / 2) + o % (PS / 2)] = 0u;
  }
  // lane: channel pair cp, pixel group (8 pixels) gr
  constexpr int CPN = CO / 2, GR = 32 / CPN;  // pairs, groups per warp step
  const int cp = lane % CPN, gr = lane / CPN;
  for (int it = warp; it < (R + 2) * (W / 8 / GR); it += 8) {
    const int r = it / (W / 8 / GR), x8 = (it % (W / 8 / GR)) * GR + gr;
    const int y = y0 + r - 1;
    uint4 a = make_uint4(0u, 0u, 0u, 0u), b = a;
    if (y >= 0 && y < H) {
      const bf16* src = dz + (size_t)(2 * cp) * P + ((size_t)n * H + y) * W + 8 * x8;
      a = *reinterpret_cast<const uint4*>(src);
      b = *reinterpret_cast<const uint4*>(src + P);
    }
    uint32_t v[8];
    const uint32_t aw[4] = {a.x, a.y, a.z, a.w}, bw[4] = {b.x, b.y, b.z, b.w};
#pragma unroll
    for (int j = 0; j < 4; j++) {
      v[2 * j] = __byte_perm(aw[j], bw[j], 0x5410);
      v[2 * j + 1] = __byte_perm(aw[j], bw[j], 0x7632);
    }
    uint32_t* d = dg_smem + (size_t)(r * Wp + 1 + 8 * x8) * (PS / 2) + cp;
#pragma unroll
    for (int j = 0; j < 8; j++) d[j * (PS / 2)] = v[j];
  }
  // weights: fragment (k = output channel, n = input channel) of every tap
  uint2 frag[9][KS][NT];
#pragma unroll
  for (int tap = 0; tap < 9; tap++)
#pragma unroll
    for (int s = 0; s < KS; s++)
#pragma unroll
      for (int j = 0; j < NT; j++) {
        const uint16_t* wp = reinterpret_cast<const uint16_t*>(wb) + (8 * j + g) * 9 + tap;
        const int k = 16 * s + 2 * t;
        frag[tap][s][j].x = wp[k * KP] | (uint32_t)wp[(k + 1) * KP] << 16;
        frag[tap][s][j].y = wp[(k + 8) * KP] | (uint32_t)wp[(k + 9) * KP] << 16;
      }
  __syncthreads();
  for (int tile = warp; tile < R * W / 16; tile += 8) {
    const int r = tile / (W / 16), x0 = (tile % (W / 16)) * 16;
    float sum[NT][4];
#pragma unroll
    for (int j = 0; j < NT; j++) sum[j][0] = sum[j][1] = sum[j][2] = sum[j][3] = 0.f;
#pragma unroll
    for (int tap = 0; tap < 9; tap++) {
      // input pixel (y, x) was read through tap (ky, kx) by output pixel
      // (y - ky + 1, x - kx + 1); +1 each for the ring
      const int rr = r + 2 - tap / 3, xx = x0 + 2 - tap % 3;
      const uint32_t* p = dg_smem + (size_t)(rr * Wp + xx + g) * (PS / 2) + t;
      float acc[NT][4];
#pragma unroll
      for (int j = 0; j < NT; j++) acc[j][0] = acc[j][1] = acc[j][2] = acc[j][3] = 0.f;
#pragma unroll
      for (int s = 0; s < KS; s++) {
        const uint32_t a[4] = {p[8 * s], p[8 * (PS / 2) + 8 * s], p[8 * s + 4],
                               p[8 * (PS / 2) + 8 * s + 4]};
#pragma unroll
        for (int j = 0; j < NT; j++) {
          const uint32_t b[2] = {frag[tap][s][j].x, frag[tap][s][j].y};
          mma_bf16(acc[j], a, b);
        }
      }
#pragma unroll
      for (int j = 0; j < NT; j++)
#pragma unroll
        for (int q = 0; q < 4; q++) sum[j][q] = __fadd_rn(sum[j][q], acc[j][q]);
    }
    float* o = din + ((size_t)n * H + y0 + r) * W + x0 + g;
#pragma unroll
    for (int j = 0; j < NT; j++) {
      const size_t c = 8 * j + 2 * t;
      o[c * P] = sum[j][0];
      o[(c + 1) * P] = sum[j][1];
      o[c * P + 8] = sum[j][2];
      o[(c + 1) * P + 8] = sum[j][3];
    }
  }
}

template <int CI, int CO, int H, int W, int R>
cudaError_t launch_dgrad3(const bf16* dz, const bf16* wb, int nb, float* din, cudaStream_t s) {
  constexpr size_t smem = (size_t)(R + 2) * (W + 2) * (CO + 8) * sizeof(bf16);
  auto kern = k_dgrad3<CI, CO, H, W, R>;
  cudaError_t e = raise_smem_limit(kern, smem);
  if (e != cudaSuccess) return e;
  kern<<<(unsigned)nb * (H / R), 256, smem, s>>>(dz, wb, (size_t)nb * H * W, din); note_launch();
  return cudaGetLastError();
}

// FC1 weight gradient: g [16][10240] += sum over the batch of dz1 [16][b] x
// x [b][10240].  A thread takes two features of a quarter of the samples, 64
// at a time with the 16 gradients in shared memory; the quarters are added in
// order.  For 128 samples 33 us as a GEMM of 32 x 64 tiles, 28 us with one
// thread for all samples (two warps a block: bound by its loads' latency),
// 11 us so.
__global__ void __launch_bounds__(256) k_fc1_wgrad(const bf16* __restrict__ dz1,
                                                   const bf16* __restrict__ x, int nb,
                                                   float* __restrict__ g) {
  constexpr int FC_PART = 64;
  __shared__ float d[FC_PART][16];
  __shared__ float2 part[3][16][64];
  const int l = threadIdx.x % 64, q = threadIdx.x / 64;
  const int f = 2 * (blockIdx.x * 64 + l);
  float acc[16][2];
#pragma unroll
  for (int o = 0; o < 16; o++) acc[o][0] = acc[o][1] = 0.f;
  for (int n0 = 0; n0 < nb; n0 += FC_PART) {
    const int m = min(FC_PART, nb - n0);
    __syncthreads();
    for (int e = threadIdx.x; e < 16 * m; e += 256) {
      const int o = e / m, n = e % m;
      d[n][o] = __bfloat162float(dz1[(size_t)o * nb + n0 + n]);
    }
    __syncthreads();
    const int end = min(m, (q + 1) * (FC_PART / 4));
#pragma unroll 8
    for (int n = q * (FC_PART / 4); n < end; n++) {
      const float2 v = __bfloat1622float2(
          *reinterpret_cast<const __nv_bfloat162*>(x + (size_t)(n0 + n) * 10240 + f));
#pragma unroll
      for (int o = 0; o < 16; o++) {
        acc[o][0] = __fmaf_rn(d[n][o], v.x, acc[o][0]);
        acc[o][1] = __fmaf_rn(d[n][o], v.y, acc[o][1]);
      }
    }
  }
  if (q > 0)
#pragma unroll
    for (int o = 0; o < 16; o++) part[q - 1][o][l] = make_float2(acc[o][0], acc[o][1]);
  __syncthreads();
  if (q > 0) return;
#pragma unroll
  for (int o = 0; o < 16; o++) {
#pragma unroll
    for (int k = 0; k < 3; k++) {
      acc[o][0] = __fadd_rn(acc[o][0], part[k][o][l].x);
      acc[o][1] = __fadd_rn(acc[o][1], part[k][o][l].y);
    }
    float2* p = reinterpret_cast<float2*>(g + (size_t)o * 10240 + f);
    const float2 old = *p;
    *p = make_float2(__fadd_rn(old.x, acc[o][0]), __fadd_rn(old.y, acc[o][1]));
  }
}

// conv output [co][b][h][w] (FP32) + bias -> ReLU -> 2x2 max pool ->
// act [co][b][h/2][w/2] (BF16), arg = position of the maximum (0..3).  Bound by
// its reads; a thread takes two pooled elements of a row (16-byte loads).
__global__ void __launch_bounds__(256) k_bias_relu_pool(const float* __restrict__ z,
                                                        const float* __restrict__ bias, int nb,
                                                        int h, int w, bf16* __restrict__ act,
                                                        unsigned char* __restrict__ arg) {
  const int c = blockIdx.y, q2 = w / 4;              // pairs of a pooled row
  const unsigned i = blockIdx.x * 256 + threadIdx.x;  // pair of this channel
  if (i >= (unsigned)(nb * (h / 2) * q2)) return;
  const unsigned x4 = i % q2, row = i / q2;           // row = n * h/2 + y2
  const float* zp = z + ((size_t)c * nb * h + 2 * (size_t)row) * w + 4 * x4;
  const float4 a = *reinterpret_cast<const float4*>(zp), b = *reinterpret_cast<const float4*>(zp + w);
  const float v[2][4] = {{a.x, a.y, b.x, b.y}, {a.z, a.w, b.z, b.w}};
  const float bc = bias[c];
  uint32_t o = 0, g = 0;
#pragma unroll
  for (int k = 0; k < 2; k++) {
    float best = -INFINITY;
    int bi = 0;
#pragma unroll
    for (int q = 0; q < 4; q++) {
      const float x = fmaxf(v[k][q] + bc, 0.f);
      if (x > best) { best = x; bi = q; }
    }
    o |= (uint32_t)__bfloat16_as_ushort(__float2bfloat16(best)) << (16 * k);
    g |= (uint32_t)bi << (8 * k);
  }
  const size_t j = (size_t)c * nb * (h / 2) * (w / 2) + 2 * (size_t)i;
  *reinterpret_cast<uint32_t*>(act + j) = o;
  *reinterpret_cast<uint16_t*>(arg + j) = (uint16_t)g;
}

// backward of bias/ReLU/pool: dact [co][b][h/2][w/2] (FP32) -> dz [co][b][h][w]
// (BF16, the next GEMM's operand), and the bias gradient's partial sums.  Each
// pooled element passes its gradient to the one position that held its
// maximum, so the bias gradient is the sum of dact over the positive pooled
// activations: the kernel that reads them adds them up, a quarter of the
// pre-pool elements.  A thread takes four pooled elements of a row (two 16-byte
// stores; w is a multiple of 8); block (x, c) leaves its sum in part[c][x].
// The former bias kernel walked all pre-pool elements with one block per
// channel and was 80 % of a training step (8.5 ms of the largest layer; 12 us
// now, the pre-activation gradient included).
constexpr int kBiasParts = 64;
__global__ void __launch_bounds__(256) k_pool_relu_back(const float* __restrict__ dact,
                                                        const bf16* __restrict__ act,
                                                        const unsigned char* __restrict__ arg,
                                                        int nb, int h, int w,
                                                        bf16* __restrict__ dz,
                                                        float* __restrict__ part) {
  const int c = blockIdx.y;
  const int h2 = h / 2, q2 = w / 8;  // quads of a pooled row
  const int nq = nb * h2 * q2;       // quads of this channel
  float sum = 0.f;
  for (int i = blockIdx.x * 256 + threadIdx.x; i < nq; i += gridDim.x * 256) {
    const size_t j = ((size_t)c * nq + i) * 4;
    const float4 d = *reinterpret_cast<const float4*>(dact + j);
    const uint2 a = *reinterpret_cast<const uint2*>(act + j);
    const uint32_t g = *reinterpret_cast<const uint32_t*>(arg + j);
    const float dv[4] = {d.x, d.y, d.z, d.w};
    const uint32_t ab[4] = {a.x & 0xFFFFu, a.x >> 16, a.y & 0xFFFFu, a.y >> 16};
    uint32_t lo[4], hi[4];  // the two rows of the 2 x 2 windows
#pragma unroll
    for (int k = 0; k < 4; k++) {
      // a positive activation: the sign bit clear, the value not zero, not NaN
      const bool on = ab[k] - 1u < 0x7F80u;
      const int q = (int)((g >> (8 * k)) & 0xFFu);
      const float v = on ? dv[k] : 0.f;
      const uint32_t b = __bfloat16_as_ushort(__float2bfloat16(v));
      if (on) sum += dv[k];
      lo[k] = q < 2 ? b << (16 * q) : 0u;
      hi[k] = q >= 2 ? b << (16 * (q - 2)) : 0u;
    }
    const int x8 = i % q2, row = i / q2;  // row = n * h2 + y2
    bf16* o = dz + ((size_t)c * nb * h + 2 * (size_t)row) * w + 8 * x8;
    *reinterpret_cast<uint4*>(o) = make_uint4(lo[0], lo[1], lo[2], lo[3]);
    *reinterpret_cast<uint4*>(o + w) = make_uint4(hi[0], hi[1], hi[2], hi[3]);
  }
  __shared__ float warp_sum[8];
#pragma unroll
  for (int o = 16; o; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
  if ((threadIdx.x & 31) == 0) warp_sum[threadIdx.x >> 5] = sum;
  __syncthreads();
  if (threadIdx.x == 0) {
    float v = 0.f;
    for (int k = 0; k < 8; k++) v += warp_sum[k];
    part[c * kBiasParts + blockIdx.x] = v;
  }
}

// the six layers' bias gradients, each channel's partial sums in a fixed order
// (two per lane, then a fixed tree), so every run gives the same bits
struct BiasSum {
  int first[7];    // first channel of each layer among all channels
  int parts[6];    // partial sums per channel
  float* out[6];   // += the layer's bias gradient
};
__global__ void k_bias_sum(const float* __restrict__ part, BiasSum b) {
  const int lane = threadIdx.x, c = blockIdx.x;
  int l = 0;
  while (c >= b.first[l + 1]) l++;
  float v = lane < b.parts[l] ? part[c * kBiasParts + lane] : 0.f;
  if (lane + 32 < b.parts[l]) v += part[c * kBiasParts + lane + 32];
#pragma unroll
  for (int o = 16; o; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  if (lane == 0) b.out[l][c - b.first[l]] += v;
}

// pooled activations of both branches -> x [b][10240] (A: 2048, B: 8192)
__global__ void k_flatten(const bf16* __restrict__ a, const bf16* __restrict__ bb, int nb,
                          bf16* __restrict__ x) {
  const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= (size_t)nb * 10240) return;
  const int n = (int)(i / 10240), f = (int)(i % 10240);
  if (f < 2048) {
    const int c = f / 64, s = f % 64;  // A: 32 x (8 x 8)
    x[i] = a[((size_t)c * nb + n) * 64 + s];
  } else {
    const int g = f - 2048, c = g / 256, s = g % 256;  // B: 32 x (8 x 32)
    x[i] = bb[((size_t)c * nb + n) * 256 + s];
  }
}

__global__ void k_unflatten(const float* __restrict__ dx, int nb, float* __restrict__ da,
                            float* __restrict__ db) {
  const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= (size_t)nb * 10240) return;
  const int n = (int)(i / 10240), f = (int)(i % 10240);
  if (f < 2048) {
    const int c = f / 64, s = f % 64;
    da[((size_t)c * nb + n) * 64 + s] = dx[i];
  } else {
    const int g = f - 2048, c = g / 256, s = g % 256;
    db[((size_t)c * nb + n) * 256 + s] = dx[i];
  }
}

// FC1 bias + ReLU: z1 [16][b] -> h [b][16] (FP32)
__global__ void k_fc1_act(const float* __restrict__ z1, const float* __restrict__ b1, int nb,
                          float* __restrict__ h) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= nb * 16) return;
  const int n = i / 16, o = i % 16;
  h[i] = fmaxf(z1[o * nb + n] + b1[o], 0.f);
}

// FC2, softmax, cross-entropy and their backward, FC2 weight/bias gradients,
// the FC1 pre-activation gradient dz1 [16][b] (BF16) and its bias gradient.
// One thread per sample; w2 [2][16], b2 [2].
// The per-sample terms of the loss and of the FC2/FC1-bias gradients go to
// hs [b][18] (loss / nb, dL/dl1, the 16 dz) and k_head_reduce sums them over
// the batch in sample order.
constexpr int kHeadTerms = 18;
__global__ void k_head(const float* __restrict__ h, const float* __restrict__ w2,
                       const float* __restrict__ b2, const int* __restrict__ labels, int nb,
                       int backward, float* __restrict__ prob, bf16* __restrict__ dz1,
                       float* __restrict__ hs) {
  const int n = blockIdx.x * blockDim.x + threadIdx.x;
  if (n >= nb) return;
  const float* hn = h + n * 16;
  float l0 = b2[0], l1 = b2[1];
  for (int o = 0; o < 16; o++) {
    l0 += w2[o] * hn[o];
    l1 += w2[16 + o] * hn[o];
  }
  const float mx = fmaxf(l0, l1);
  const float e0 = expf(l0 - mx), e1 = expf(l1 - mx);
  const float p1 = e1 / (e0 + e1);
  prob[n] = p1;
  if (!backward) return;
  const int y = labels[n];
  const float lse = mx + logf(e0 + e1);
  float* t = hs + (size_t)n * kHeadTerms;
  t[0] = (lse - (y ? l1 : l0)) / nb;
  const float d1 = (p1 - (y ? 1.f : 0.f)) / nb;  // dL/dl1; dL/dl0 = -d1
  const float d0 = -d1;
  t[1] = d1;
  for (int o = 0; o < 16; o++) {
    const float dh = d0 * w2[o] + d1 * w2[16 + o];
    const float dz = hn[o] > 0.f ? dh : 0.f;
    dz1[o * nb + n] = __float2bfloat16(dz);
    t[2 + o] = dz;
  }
}

// loss (+= the per-sample terms), gb2, gw2 [2][16] and gb1 [16] from hs and
// h, each a sum over the samples in order (thread per output).  The chain of
// adds is short; what took time (70 us at 128 samples) was a global load per
// sample and output on it, so the block stages 128 samples at a time.
constexpr int kHeadChunk = 128;
__global__ void __launch_bounds__(256) k_head_reduce(const float* __restrict__ h,
                                                     const float* __restrict__ hs, int nb,
                                                     float* __restrict__ loss,
                                                     float* __restrict__ gw2,
                                                     float* __restrict__ gb2,
                                                     float* __restrict__ gb1) {
  __shared__ float sh[kHeadChunk * 16], st[kHeadChunk * kHeadTerms];
  const int k = threadIdx.x;  // 0: loss, 1-2: gb2, 3-34: gw2, 35-50: gb1
  // every output's term is +-(one of the sample's terms) times 1 or one of its
  // hidden units, so that no thread branches in the loop (dL/dl0 = -dL/dl1)
  const int term = k == 0 ? 0 : k < 35 ? 1 : k - 33;
  const float sign = k == 1 || (k >= 3 && k < 19) ? -1.f : 1.f;
  const bool hidden = k >= 3 && k < 35;
  const int unit = hidden ? (k - 3) % 16 : 0;
  float acc = 0.f;
  for (int n0 = 0; n0 < nb; n0 += kHeadChunk) {
    const int m = min(kHeadChunk, nb - n0);
    __syncthreads();
    for (int i = k; i < m * 16; i += 256) sh[i] = h[(size_t)n0 * 16 + i];
    for (int i = k; i < m * kHeadTerms; i += 256) st[i] = hs[(size_t)n0 * kHeadTerms + i];
    __syncthreads();
    if (k > 50) continue;
#pragma unroll 8
    for (int n = 0; n < m; n++) {
      const float hv = hidden ? sh[n * 16 + unit] : 1.f;
      acc = __fadd_rn(acc, __fmul_rn(sign * st[n * kHeadTerms + term], hv));
    }
  }
  if (k == 0) loss[0] = __fadd_rn(loss[0], acc);
  else if (k < 3) gb2[k - 1] = __fadd_rn(gb2[k - 1], acc);
  else if (k < 35) gw2[k - 3] = __fadd_rn(gw2[k - 3], acc);
  else if (k < 51) gb1[k - 35] = __fadd_rn(gb1[k - 35], acc);
}

// per-sample batch gather: dataset [n][len] (BF16) rows idx -> [b][len]
__global__ void k_gather(const bf16* __restrict__ src, const int* __restrict__ idx, int nb,
                         int len, bf16* __restrict__ dst) {
  const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= (size_t)nb * len) return;
  const int n = (int)(i / len), k = (int)(i % len);
  dst[i] = src[(size_t)idx[n] * len + k];
}

// Adam (Kingma & Ba 2015) on the FP32 master weights
__global__ void k_adam(float* __restrict__ w, const float* __restrict__ g, float* __restrict__ m,
                       float* __restrict__ v, size_t n, float lr, float b1, float b2, float eps,
                       float c1, float c2) {
  for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < n;
       i += (size_t)gridDim.x * blockDim.x) {
    const float gi = g[i];
    const float mi = b1 * m[i] + (1.f - b1) * gi;
    const float vi = b2 * v[i] + (1.f - b2) * gi * gi;
    m[i] = mi;
    v[i] = vi;
    w[i] -= lr * (mi / c1) / (sqrtf(vi / c2) + eps);
  }
}

inline unsigned nblk(size_t n, int t = 256) { return (unsigned)((n + t - 1) / t); }

}  // namespace clf

// ===========================================================================
// Fused inference: the whole network for one candidate per CTA iteration.
//
// A persistent CTA of 16 warps takes candidates in turn.  Activations live in
// shared memory as [row + 1][col + 1][channel] BF16 with a zero ring (the
// convolutions' padding).  Each 3x3 convolution is an implicit GEMM on the
// tensor cores (mma.sync m16n8k16, FP32 accumulation) with the 16 rows of an
// MMA tile = 2 image rows x 8 columns and its columns = output channels; the
// K dimension runs over taps and input channels: one tap x 16 channels
// (c_in = 16), two taps x 8 channels (c_in = 8) or the 9 taps of the single
// input channel.  Bias, ReLU and the 2x2 max-pool are applied to the
// accumulators in registers (the vertical pair sits in one thread, the
// horizontal pair in lanes 4 apart) and the pooled value is rounded to BF16
// once, as in the training path.  The last layer of each branch writes the
// flattened feature vector (10240 BF16) to shared memory; each warp then
// computes one FC1 unit (fixed lane order and shuffle tree), and thread 0 the
// FC2 logits and the softmax.  Every candidate is summed in the same order
// whatever the grid, so all scoring entry points agree bit for bit.
// ===========================================================================
namespace inf {
using namespace clf;
constexpr int kWarps = 16, kThreads = kWarps * 32;
// shared-memory regions (bytes)
// Pixels of 16 channels are stored 24 elements (48 bytes) apart, so that the
// 8 pixels of an MMA fragment load fall on distinct banks; 1 and 8 channels
// are dense.
template <int C>
__host__ __device__ constexpr int pix_stride() { return C == 16 ? 24 : C; }
// Pixels from one row of a layer's input to the next, and the padded row's
// first: 1-channel rows are W + 16 apart (8 banks apart modulo 32, so the four
// taps that a fragment load takes from three rows miss one another) and start
// 7 in, which puts the image on 16-byte boundaries.
__host__ __device__ constexpr int row_pitch(int c, int w) { return c == 1 ? w + 16 : w + 2; }
__host__ __device__ constexpr int row_start(int c) { return c == 1 ? 7 : 0; }
constexpr int kR0 = 18 * 66 * 24 * 2;   // B input [66][272]; B pool-2 [18][66][24]; A pool-1 [34][34][8]
constexpr int kR1 = 34 * 130 * 8 * 2;   // B pool-1 [34][130][8]; A input [66][80]; A pool-2 [18][18][24]
static_assert(66 * 272 * 2 <= kR0 && 66 * 80 * 2 <= kR1, "input regions");
constexpr int kF = 10240 * 2;           // flattened features
// weight fragments per layer: ksteps x (c_out / 8) x 32 lanes of uint2
constexpr int kFragL1 = 1 * 1 * 32, kFragL2 = 5 * 2 * 32, kFragL3 = 9 * 4 * 32;
constexpr int kFragBranch = kFragL1 + kFragL2 + kFragL3;
constexpr int kWF = 2 * kFragBranch * 8;
constexpr size_t kSmem = (size_t)kR0 + kR1 + kF + kWF + 256 * sizeof(float);

struct Args {
  const float* dm;   // [n][64][64] FP32 patches
  const float* ft;   // [n][64][256]
  int n;
  const float* w;    // FP32 parameters
  int off_w[2][3], off_b[2][3], off_b1, off_w2, off_b2;
  const bf16* wb1;   // FC1 weights [16][10240] BF16
  float* prob;       // [n]
};

__device__ __forceinline__ uint32_t pack2(bf16 lo, bf16 hi) {
  return (uint32_t)__bfloat16_as_ushort(lo) | ((uint32_t)__bfloat16_as_ushort(hi) << 16);
}

// weight fragment b0/b1 of k-step s, n-tile j for this lane; K order as the
// A fragments below
template <int CI>
__device__ uint2 weight_frag(const float* W, int s, int j, int lane) {
  const int g = lane >> 2, t = lane & 3;
  const int co = 8 * j + g;
  auto wk = [&](int k) -> bf16 {
    int tap, ci;
    if (CI == 16) { tap = s; ci = k; }
    else if (CI == 8) { tap = 2 * s + (k >> 3); ci = k & 7; }
    else { tap = k; ci = 0; }
    if (tap >= 9) return __float2bfloat16(0.f);
    return __float2bfloat16(W[co * (CI * 9) + ci * 9 + tap]);
  };
  uint2 r;
  r.x = pack2(wk(2 * t), wk(2 * t + 1));
  r.y = pack2(wk(2 * t + 8), wk(2 * t + 9));
  return r;
}

template <int CI, int CO>
__device__ void build_frags(const float* W, uint2* wf) {
  constexpr int KS = CI == 16 ? 9 : (CI == 8 ? 5 : 1);
  constexpr int NT = CO / 8;
  for (int e = threadIdx.x; e < KS * NT * 32; e += blockDim.x) {
    const int lane = e & 31, j = (e >> 5) % NT, s = (e >> 5) / NT;
    wf[e] = weight_frag<CI>(W, s, j, lane);
  }
}

// zero ring of a [H2 + 2][W2 + 2][C] buffer (C a multiple of 8)
template <int H2, int W2, int C>
__device__ void zero_ring(bf16* buf) {
  constexpr int Wp = W2 + 2, Hp = H2 + 2, Q = C / 8;  // 16-byte pieces of a pixel
  constexpr int ring = 2 * Wp + 2 * H2;               // pixels
  for (int e = threadIdx.x; e < ring * Q; e += kThreads) {
    const int px = e / Q;
    int y, x;
    if (px < Wp) { y = 0; x = px; }
    else if (px < 2 * Wp) { y = Hp - 1; x = px - Wp; }
    else { const int q = px - 2 * Wp; y = 1 + (q >> 1); x = (q & 1) ? Wp - 1 : 0; }
    reinterpret_cast<uint4*>(buf + ((size_t)y * Wp + x) * C)[e % Q] = make_uint4(0u, 0u, 0u, 0u);
  }
}

// patch rows (FP32, global) -> BF16 [66][W + 16] with a zero ring around the
// image (row_start), limited to +-kInputClip as the training input
template <int W>
__device__ void load_input(const float* __restrict__ src, bf16* dst) {
  constexpr int P = row_pitch(1, W);
  const bf16 z = __float2bfloat16(0.f);
  for (int e = threadIdx.x; e < P; e += kThreads) {
    dst[e] = z;
    dst[65 * P + e] = z;
  }
  for (int y = threadIdx.x; y < 64; y += kThreads) {
    dst[(y + 1) * P + 7] = z;
    dst[(y + 1) * P + 8 + W] = z;
  }
  constexpr int n4 = 64 * W / 4, N = n4 / kThreads;  // all loads in flight at once
  float4 v[N];
#pragma unroll
  for (int k = 0; k < N; k++)
    v[k] = __ldg(reinterpret_cast<const float4*>(src) + threadIdx.x + k * kThreads);
  auto clip = [](float x) { return __float2bfloat16(fminf(fmaxf(x, -kInputClip), kInputClip)); };
#pragma unroll
  for (int k = 0; k < N; k++) {
    const int e = threadIdx.x + k * kThreads, y = (4 * e) / W, x = (4 * e) % W;
    *reinterpret_cast<uint2*>(dst + (y + 1) * P + 8 + x) =
        make_uint2(pack2(clip(v[k].x), clip(v[k].y)), pack2(clip(v[k].z), clip(v[k].w)));
  }
}

// conv 3x3 (pad 1) + bias + ReLU + 2x2 max-pool of an H x W x CI image
// (pixels pix_stride<CI>() elements apart).
// out: [H/2 + 2][W/2 + 2][pix_stride<CO>()] interior, or (feat) the flattened features at
// feat[c * (H/2 * W/2) + y * W/2 + x].
// A warp's weight fragments stay in registers over its tiles (two wavefronts
// of shared memory per fragment and tile otherwise, twice the pixels' share in
// the last layer).
template <int CI, int CO, int H, int W>
__device__ void conv_layer(const bf16* __restrict__ in_, const uint2* __restrict__ wf,
                           const float* __restrict__ bias, bf16* __restrict__ out,
                           bf16* __restrict__ feat) {
  constexpr int KS = CI == 16 ? 9 : (CI == 8 ? 5 : 1);
  constexpr int NT = CO / 8;
  constexpr int PSI = pix_stride<CI>(), PSO = pix_stride<CO>();
  constexpr int Wp = row_pitch(CI, W), W2 = W / 2, H2 = H / 2;
  constexpr int ntx = W / 8, ntiles = H2 * ntx;
  const bf16* in = in_ + row_start(CI) * PSI;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int g = lane >> 2, t = lane & 3;
  float bia[NT][2];
#pragma unroll
  for (int j = 0; j < NT; j++) {
    bia[j][0] = bias[8 * j + 2 * t];
    bia[j][1] = bias[8 * j + 2 * t + 1];
  }
  uint2 frag[KS][NT];
#pragma unroll
  for (int s = 0; s < KS; s++)
#pragma unroll
    for (int j = 0; j < NT; j++) frag[s][j] = wf[(s * NT + j) * 32 + lane];
  for (int tile = warp; tile < ntiles; tile += kWarps) {
    const int ty = tile / ntx, tx = tile % ntx;
    // pixel rows of the MMA tile: row g -> (2ty, 8tx + g), row g + 8 -> (2ty + 1, 8tx + g);
    // padded index of pixel (y, x) at tap (ky, kx) = (y + ky) * Wp + x + kx
    const int p0 = (2 * ty) * Wp + 8 * tx + g;
    const int p1 = p0 + Wp;
    float acc[NT][4];
#pragma unroll
    for (int j = 0; j < NT; j++) acc[j][0] = acc[j][1] = acc[j][2] = acc[j][3] = 0.f;
#pragma unroll
    for (int s = 0; s < KS; s++) {
      uint32_t a[4];
      if (CI == 16) {
        const int o = (s / 3) * Wp + (s % 3);
        a[0] = *reinterpret_cast<const uint32_t*>(in + (size_t)(p0 + o) * PSI + 2 * t);
        a[1] = *reinterpret_cast<const uint32_t*>(in + (size_t)(p1 + o) * PSI + 2 * t);
        a[2] = *reinterpret_cast<const uint32_t*>(in + (size_t)(p0 + o) * PSI + 2 * t + 8);
        a[3] = *reinterpret_cast<const uint32_t*>(in + (size_t)(p1 + o) * PSI + 2 * t + 8);
      } else if (CI == 8) {
        const int j0 = 2 * s, j1 = 2 * s + 1;
        const int o0 = (j0 / 3) * Wp + (j0 % 3);
        a[0] = *reinterpret_cast<const uint32_t*>(in + (size_t)(p0 + o0) * PSI + 2 * t);
        a[1] = *reinterpret_cast<const uint32_t*>(in + (size_t)(p1 + o0) * PSI + 2 * t);
        if (j1 < 9) {
          const int o1 = (j1 / 3) * Wp + (j1 % 3);
          a[2] = *reinterpret_cast<const uint32_t*>(in + (size_t)(p0 + o1) * PSI + 2 * t);
          a[3] = *reinterpret_cast<const uint32_t*>(in + (size_t)(p1 + o1) * PSI + 2 * t);
        } else {
          a[2] = a[3] = 0u;
        }
      } else {
        // K = tap; taps 2t, 2t + 1 and (t = 0 only) tap 8
        const int ta = 2 * t, tb = 2 * t + 1;
        const int oa = (ta / 3) * Wp + (ta % 3), ob = (tb / 3) * Wp + (tb % 3);
        a[0] = pack2(in[p0 + oa], in[p0 + ob]);
        a[1] = pack2(in[p1 + oa], in[p1 + ob]);
        const bf16 z = __float2bfloat16(0.f);
        const int o8 = 2 * Wp + 2;
        a[2] = t == 0 ? pack2(in[p0 + o8], z) : 0u;
        a[3] = t == 0 ? pack2(in[p1 + o8], z) : 0u;
      }
#pragma unroll
      for (int j = 0; j < NT; j++) {
        const uint32_t bb[2] = {frag[s][j].x, frag[s][j].y};
        mma_bf16(acc[j], a, bb);
      }
    }
    // epilogue: c0 (row g, co 2t), c1 (row g, co 2t+1), c2/c3 the same for row g + 8
    const int py = ty, px = 4 * tx + (g >> 1);
#pragma unroll
    for (int j = 0; j < NT; j++) {
      float m0 = fmaxf(fmaxf(acc[j][0] + bia[j][0], 0.f), fmaxf(acc[j][2] + bia[j][0], 0.f));
      float m1 = fmaxf(fmaxf(acc[j][1] + bia[j][1], 0.f), fmaxf(acc[j][3] + bia[j][1], 0.f));
      m0 = fmaxf(m0, __shfl_xor_sync(0xffffffffu, m0, 4));
      m1 = fmaxf(m1, __shfl_xor_sync(0xffffffffu, m1, 4));
      if ((g & 1) == 0) {
        const int co = 8 * j + 2 * t;
        if (feat) {
          feat[(size_t)co * (H2 * W2) + py * W2 + px] = __float2bfloat16(m0);
          feat[(size_t)(co + 1) * (H2 * W2) + py * W2 + px] = __float2bfloat16(m1);
        } else {
          *reinterpret_cast<uint32_t*>(out + ((size_t)(py + 1) * (W2 + 2) + px + 1) * PSO + co) =
              pack2(__float2bfloat16(m0), __float2bfloat16(m1));
        }
      }
    }
  }
}

__global__ void __launch_bounds__(kThreads, 1) k_clf_infer(Args a) {
  extern __shared__ __align__(128) uint8_t smem[];
  bf16* r0 = reinterpret_cast<bf16*>(smem);
  bf16* r1 = reinterpret_cast<bf16*>(smem + kR0);
  bf16* feat = reinterpret_cast<bf16*>(smem + kR0 + kR1);
  uint2* wf = reinterpret_cast<uint2*>(smem + kR0 + kR1 + kF);
  float* hid = reinterpret_cast<float*>(smem + kR0 + kR1 + kF + kWF);
  // weight fragments of both branches, once per CTA
  for (int br = 0; br < 2; br++) {
    uint2* f = wf + br * kFragBranch;
    build_frags<1, 8>(a.w + a.off_w[br][0], f);
    build_frags<8, 16>(a.w + a.off_w[br][1], f + kFragL1);
    build_frags<16, 32>(a.w + a.off_w[br][2], f + kFragL1 + kFragL2);
  }
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  for (int cand = blockIdx.x; cand < a.n; cand += gridDim.x) {
    __syncthreads();  // fragments ready / previous candidate's FC done
    // the next candidate's patches into L2 while this one is computed
    if (cand + (int)gridDim.x < a.n) {
      const size_t nx = (size_t)cand + gridDim.x;
      const char* p = reinterpret_cast<const char*>(a.ft + nx * 16384) + threadIdx.x * 128;
      asm volatile("prefetch.global.L2 [%0];" :: "l"(p));  // 512 lines of 128 bytes
      if (threadIdx.x < 128) {
        p = reinterpret_cast<const char*>(a.dm + nx * 4096) + threadIdx.x * 128;
        asm volatile("prefetch.global.L2 [%0];" :: "l"(p));
      }
    }
    // ---- branch B (freq-time, 64 x 256): features 2048.. ----
    const uint2* fB = wf + kFragBranch;
    load_input<256>(a.ft + (size_t)cand * 16384, r0);
    zero_ring<32, 128, 8>(r1);
    __syncthreads();
    conv_layer<1, 8, 64, 256>(r0, fB, a.w + a.off_b[1][0], r1, nullptr);
    __syncthreads();
    zero_ring<16, 64, pix_stride<16>()>(r0);
    conv_layer<8, 16, 32, 128>(r1, fB + kFragL1, a.w + a.off_b[1][1], r0, nullptr);
    __syncthreads();
    conv_layer<16, 32, 16, 64>(r0, fB + kFragL1 + kFragL2, a.w + a.off_b[1][2], nullptr,
                               feat + 2048);
    // ---- branch A (DM-time, 64 x 64): features 0..2047 ----
    const uint2* fA = wf;
    load_input<64>(a.dm + (size_t)cand * 4096, r1);
    __syncthreads();
    zero_ring<32, 32, 8>(r0);
    conv_layer<1, 8, 64, 64>(r1, fA, a.w + a.off_b[0][0], r0, nullptr);
    __syncthreads();
    zero_ring<16, 16, pix_stride<16>()>(r1);
    conv_layer<8, 16, 32, 32>(r0, fA + kFragL1, a.w + a.off_b[0][1], r1, nullptr);
    __syncthreads();
    conv_layer<16, 32, 16, 16>(r1, fA + kFragL1 + kFragL2, a.w + a.off_b[0][2], nullptr, feat);
    __syncthreads();
    // ---- FC1: warp o computes hidden unit o ----
    {
      const int o = warp;
      const uint4* wrow = reinterpret_cast<const uint4*>(a.wb1 + (size_t)o * 10240);
      const uint4* x = reinterpret_cast<const uint4*>(feat);
      float sum = 0.f;
#pragma unroll 8
      for (int i = lane; i < 10240 / 8; i += 32) {
        const uint4 wv = __ldg(wrow + i), xv = x[i];
        const uint32_t wa[4] = {wv.x, wv.y, wv.z, wv.w}, xa[4] = {xv.x, xv.y, xv.z, xv.w};
#pragma unroll
        for (int q = 0; q < 4; q++) {
          const float2 wf2 = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&wa[q]));
          const float2 xf2 = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&xa[q]));
          sum = __fadd_rn(sum, __fmul_rn(wf2.x, xf2.x));
          sum = __fadd_rn(sum, __fmul_rn(wf2.y, xf2.y));
        }
      }
#pragma unroll
      for (int off = 16; off; off >>= 1) sum = __fadd_rn(sum, __shfl_xor_sync(0xffffffffu, sum, off));
      if (lane == 0) hid[o] = fmaxf(sum + a.w[a.off_b1 + o], 0.f);
    }
    __syncthreads();
    if (threadIdx.x == 0) {
      const float* w2 = a.w + a.off_w2;
      const float* b2 = a.w + a.off_b2;
      float l0 = b2[0], l1 = b2[1];
      for (int o = 0; o < 16; o++) {
        l0 += w2[o] * hid[o];
        l1 += w2[16 + o] * hid[o];
      }
      const float mx = fmaxf(l0, l1);
      const float e0 = expf(l0 - mx), e1 = expf(l1 - mx);
      a.prob[cand] = e1 / (e0 + e1);
    }
  }
}
}  // namespace inf

// ===========================================================================
// Candidate patches (Applications/candidate_profiler.C)
// ===========================================================================
// DM-time: row r = DM trial dm - 32 + r (zero outside 0..D-1), column t = the
// width-w boxcar sum starting at first + t, first = ind - 32 - w/2 (0 if
// ind <= 32 + w/2), from the series' prefix sums S: S[first+t+w] - S[first+t]
// (zero when it would read past S[len]); gen_dm_time_plot:232-415 with
// do_filter (its boxcar spans scanned[t + w/2 + (w-1)/2 + 1] - scanned[t]).
__global__ void k_patch_dm(const float* __restrict__ scan, size_t scan_pitch, size_t len,
                           const PatchJob* __restrict__ jobs, float* __restrict__ out) {
  const PatchJob jb = jobs[blockIdx.x];
  const unsigned w = 1u << jb.filter;
  const long long first = (jb.ind > 32u + w / 2) ? (long long)jb.ind - 32 - w / 2 : 0;
  float* o = out + (size_t)blockIdx.x * 4096;
  for (int e = threadIdx.x; e < 4096; e += blockDim.x) {
    const int r = e / 64, t = e % 64;
    const int d = jb.dm - 32 + r;
    float v = 0.f;
    const long long a = first + t, b = a + w;
    if (d >= 0 && d < jb.ndm && b <= (long long)len) {
      const float* S = scan + (size_t)(jb.series0 + d) * scan_pitch;
      v = __fsub_rn(S[b], S[a]);
    }
    o[e] = v;
  }
}

// Freq-time: gen_freq_time_plot:136-230 on the undispersed filterbank (TF
// bytes): 64 sub-bands of fs = nchans/64 channels x 256 bins of ts samples
// from first; each pixel the float sum, time outer and channel inner, of
// x / 255 * 255 divided by ts * fs; samples outside the gulp read as 0.
// x / 255 * 255 comes from a 256-entry table of the same rounded operations;
// rows outside the gulp are skipped (they add +0 to a sum that is >= +0, which
// leaves it unchanged).  Grid: x = candidate, y = 64 groups of 4 time bins;
// block = 4 bins x 64 sub-bands, so a warp reads 32 adjacent sub-bands of one
// row.
__global__ void __launch_bounds__(256) k_patch_ft(const uint8_t* __restrict__ tf, size_t nsamps,
                                                  int nchans, const PatchJob* __restrict__ jobs,
                                                  float* __restrict__ out) {
  __shared__ float lut[256];
  lut[threadIdx.x] = __fmul_rn(__fdiv_rn((float)threadIdx.x, 255.f), 255.f);
  __syncthreads();
  const PatchJob jb = jobs[blockIdx.x];
  const int fs = nchans / 64;
  const int cs = threadIdx.x & 63;
  const int ti = blockIdx.y * 4 + (threadIdx.x >> 6);
  const uint8_t* fb = tf + (size_t)jb.unit * nsamps * nchans + (size_t)cs * fs;
  const long long t0 = jb.ft_first + (long long)ti * jb.ft_ts;
  const long long lo = t0 > 0 ? t0 : 0;
  const long long end = t0 + (long long)jb.ft_ts;
  const long long hi = end < (long long)nsamps ? end : (long long)nsamps;
  float sum = 0.f;
  for (long long t = lo; t < hi; t++) {
    const uint8_t* row = fb + (size_t)t * nchans;
    for (int f = 0; f < fs; f++) sum = __fadd_rn(sum, lut[row[f]]);
  }
  const float npix = (float)((size_t)jb.ft_ts * (size_t)fs);
  out[(size_t)blockIdx.x * 16384 + cs * 256 + ti] = __fdiv_rn(sum, npix);
}

// k-th smallest (0-based) of v[lo..hi) in shared memory, by ranks
__device__ float warp_kth(const float* v, int lo, int hi, int k) {
  const int lane = threadIdx.x & 31;
  float found = 0.f;
  bool have = false;
  for (int i = lo + lane; i < hi; i += 32) {
    const float x = v[i];
    int lt = 0, le = 0;
    for (int j = lo; j < hi; j++) {
      lt += v[j] < x;
      le += v[j] <= x;
    }
    if (lt <= k && k < le) { found = x; have = true; }
  }
  const unsigned m = __ballot_sync(0xffffffffu, have);
  return __shfl_sync(0xffffffffu, found, m ? __ffs(m) - 1 : 0);
}

// normalise_series_array (candidate_profiler.C:88-134) on rows of n values,
// one warp per row.  A row whose deviation is zero becomes zero for the
// classifier's patches (zero_flat); the profiler keeps the reference's
// arithmetic there (a division by zero: NaN or +-inf).
template <bool ZERO_FLAT>
__global__ void k_normalise_rows_t(float* __restrict__ data, int n, size_t nrows, size_t pitch,
                                   int rows_per_group, size_t group_pitch,
                                   const size_t* __restrict__ at, size_t nlist,
                                   size_t rest) {
  extern __shared__ float nr_smem[];
  const int wib = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const size_t row = (size_t)blockIdx.x * (blockDim.x >> 5) + wib;
  float* v = nr_smem + (size_t)wib * 2 * n;  // [n] values, [n] scratch
  float* a = v + n;
  if (row >= nrows) return;  // whole warp
  // nlist rows at listed offsets, then, from `rest` on, rows in groups (e.g.
  // the trials of one candidate's plot)
  const size_t g = row < nlist ? 0 : row - nlist;
  float* x = data + (row < nlist ? at[row] : rest + (g / rows_per_group) * group_pitch +
                                                 (g % rows_per_group) * pitch);
  for (int j = lane; j < n; j += 32) v[j] = x[j];
  __syncwarp();
  const float m1 = warp_kth(v, 0, n / 2, n / 4);
  const float m2 = warp_kth(v, n / 2, n, n / 4);
  const double gradient = (double)__fdiv_rn(__fsub_rn(m2, m1), (float)(n / 2));
  const float median0 = (float)((double)m1 - gradient * (double)(n / 4));
  for (int j = lane; j < n; j += 32) {
    const float base = (float)((double)median0 + (double)j * gradient);
    const float y = __fsub_rn(v[j], base);
    v[j] = y;
    a[j] = fabsf(y);
  }
  __syncwarp();
  const float mad = warp_kth(a, 0, n, n / 2);
  const float stddev = (float)((double)mad * 1.4826);
  const float val = (float)(1.0 / (double)stddev);
  for (int j = lane; j < n; j += 32)
    x[j] = (!ZERO_FLAT || stddev > 0.f) ? __fmul_rn(v[j], val) : 0.f;
}

static cudaError_t launch_normalise(float* data, int n, size_t nrows, size_t pitch,
                                    int rows_per_group, size_t group_pitch, bool zero_flat,
                                    const size_t* at, size_t nlist, size_t rest, cudaStream_t s) {
  if (n < 2 || nrows == 0) return cudaSuccess;
  const size_t smem = 2 * (size_t)n * sizeof(float);
  // rows of up to 1024 values: four warps per block; longer: one
  const int wpb = n <= 1024 ? 4 : 1;
  if (smem * wpb > 200 * 1024) return cudaErrorInvalidValue;
  auto kern = zero_flat ? k_normalise_rows_t<true> : k_normalise_rows_t<false>;
  cudaError_t e = raise_smem_limit(kern, smem * wpb);
  if (e != cudaSuccess) return e;
  kern<<<(unsigned)((nrows + wpb - 1) / wpb), 32 * wpb, smem * wpb, s>>>(
      data, n, nrows, pitch, rows_per_group, group_pitch, at, nlist, rest);
  note_launch();
  return cudaGetLastError();
}

cudaError_t normalise_rows(float* data, int n, size_t nrows, size_t pitch, int rows_per_group,
                           size_t group_pitch, bool zero_flat, cudaStream_t s) {
  return launch_normalise(data, n, nrows, pitch, rows_per_group, group_pitch, zero_flat, nullptr,
                          0, 0, s);
}

cudaError_t normalise_row_list(float* data, int n, const size_t* at, size_t nlist, size_t rest,
                               size_t nrest, cudaStream_t s) {
  return launch_normalise(data, n, nlist + nrest, 0, 1, (size_t)n, false, at, nlist, rest, s);
}

cudaError_t extract_patches(const float* scan, size_t scan_pitch, size_t len, const uint8_t* tf,
                            size_t nsamps, int nchans, const PatchJob* jobs, int njobs,
                            float* dm_out, float* ft_out, cudaStream_t s) {
  if (njobs <= 0) return cudaSuccess;
  k_patch_dm<<<njobs, 256, 0, s>>>(scan, scan_pitch, len, jobs, dm_out); note_launch();
  k_patch_ft<<<dim3((unsigned)njobs, 64), 256, 0, s>>>(tf, nsamps, nchans, jobs, ft_out); note_launch();
  const size_t r1 = (size_t)njobs * 64;
  cudaError_t e = normalise_rows(dm_out, 64, r1, 64, 1, 64, true, s);
  if (e == cudaSuccess) e = normalise_rows(ft_out, 256, r1, 256, 1, 256, true, s);
  return e == cudaSuccess ? cudaGetLastError() : e;
}
}  // namespace hdb

// ===========================================================================
// The model
// ===========================================================================
using hdb::clf::bf16;

namespace {

struct ConvSpec {
  int ci, co, h, w;  // input channels, output channels, input rows, cols
  int kw() const { return ci * 9; }
  int kp() const { return (ci * 9 + 15) / 16 * 16; }
};
// branch A: 64 x 64 input; branch B: 64 x 256 input
const ConvSpec kConv[2][3] = {{{1, 8, 64, 64}, {8, 16, 32, 32}, {16, 32, 16, 16}},
                              {{1, 8, 64, 256}, {8, 16, 32, 128}, {16, 32, 16, 64}}};
constexpr int kFeat = 10240, kHid = 16;

struct DBuf {
  void* p = nullptr;
  size_t cap = 0;
  ~DBuf() { if (p) cudaFree(p); }
  template <class T> T* as() { return reinterpret_cast<T*>(p); }
  cudaError_t ensure(size_t bytes) {
    if (bytes <= cap) return cudaSuccess;
    if (p) cudaFree(p);
    p = nullptr;
    cap = 0;
    cudaError_t e = hdb::dev_malloc(&p, std::max<size_t>(bytes, 256));
    if (e == cudaSuccess) cap = std::max<size_t>(bytes, 256);
    return e;
  }
};

}  // namespace

struct hd_classifier_t {
  int device = 0;
  cudaStream_t stream = nullptr;
  // flat FP32 parameters: per conv layer W [co][ci*9] then b [co], branch A
  // then B, then W1 [16][10240], b1 [16], W2 [2][16], b2 [2]
  size_t off_w[2][3], off_b[2][3], off_w1, off_b1, off_w2, off_b2, nparam;
  DBuf w, g, m, v;          // parameters, gradients, Adam moments
  DBuf wb_conv[2][3], wb1;  // BF16 weight copies
  bool bf16_stale = true;   // the FP32 weights changed since the BF16 copies
  long long step = 0;
  // per-batch work buffers
  int cap_batch = 0;
  DBuf in[2], col, z, act[2][3], arg[2][3], dz, in_f32, dact_a[2], dact_b[2], x, z1, h, dz1,
      dx, prob, loss, labels, idx, hs, bias_part;
  DBuf tc_ws, tc_err;               // tensor-core GEMM: split-K workspace, error word
  DBuf data_dm, data_ft, data_lab;  // resident training set
  DBuf stage_dm, stage_ft, sprob;    // scoring: host patches staged in FP32, scores
  int nsm = 0;
  size_t data_n = 0;
  cudaEvent_t ev[2] = {};  // around the last scoring call, on `stream`
  float score_ms = 0.f;

  ~hd_classifier_t() {
    for (auto& e : ev)
      if (e) cudaEventDestroy(e);
    if (stream) cudaStreamDestroy(stream);
  }
};

namespace {

using namespace hdb::clf;

#define CK(x)                                               \
  do {                                                      \
    cudaError_t e_ = (x);                                   \
    if (e_ != cudaSuccess) return e_;                       \
  } while (0)

cudaError_t alloc_batch(hd_classifier c, int nb) {
  if (nb <= c->cap_batch) return cudaSuccess;
  size_t maxcol = 0, maxz = 0;
  for (int br = 0; br < 2; br++)
    for (int l = 0; l < 3; l++) {
      const ConvSpec& s = kConv[br][l];
      const size_t P = (size_t)nb * s.h * s.w;
      maxcol = std::max(maxcol, (size_t)s.kp() * P);
      maxz = std::max(maxz, (size_t)s.co * P);
      CK(c->act[br][l].ensure((size_t)s.co * P / 4 * sizeof(bf16)));
      CK(c->arg[br][l].ensure((size_t)s.co * P / 4));
    }
  CK(c->in[0].ensure((size_t)nb * 64 * 64 * sizeof(bf16)));
  CK(c->in[1].ensure((size_t)nb * 64 * 256 * sizeof(bf16)));
  CK(c->col.ensure(maxcol * sizeof(bf16)));
  CK(c->z.ensure(maxz * sizeof(float)));
  CK(c->dz.ensure(maxz * sizeof(bf16)));
  for (int br = 0; br < 2; br++) {
    CK(c->dact_a[br].ensure(maxz / 4 * sizeof(float)));
    CK(c->dact_b[br].ensure(maxz / 4 * sizeof(float)));
  }
  CK(c->x.ensure((size_t)nb * kFeat * sizeof(bf16)));
  CK(c->dx.ensure((size_t)nb * kFeat * sizeof(float)));
  CK(c->z1.ensure((size_t)nb * kHid * sizeof(float)));
  CK(c->h.ensure((size_t)nb * kHid * sizeof(float)));
  CK(c->dz1.ensure((size_t)nb * kHid * sizeof(bf16)));
  CK(c->prob.ensure((size_t)nb * sizeof(float)));
  CK(c->hs.ensure((size_t)nb * kHeadTerms * sizeof(float)));
  CK(c->bias_part.ensure((size_t)2 * (8 + 16 + 32) * kBiasParts * sizeof(float)));
  CK(c->loss.ensure(sizeof(float)));
  CK(c->labels.ensure((size_t)nb * sizeof(int)));
  CK(c->idx.ensure((size_t)nb * sizeof(int)));
  c->cap_batch = nb;
  return cudaSuccess;
}

cudaError_t refresh_bf16(hd_classifier c) {
  if (!c->bf16_stale) return cudaSuccess;
  c->bf16_stale = false;
  cudaStream_t s = c->stream;
  float* w = c->w.as<float>();
  for (int br = 0; br < 2; br++)
    for (int l = 0; l < 3; l++) {
      const ConvSpec& sp = kConv[br][l];
      CK(c->wb_conv[br][l].ensure((size_t)sp.co * sp.kp() * sizeof(bf16)));
      k_weights_bf16<<<nblk((size_t)sp.co * sp.kp()), 256, 0, s>>>(
          w + c->off_w[br][l], sp.co, sp.kw(), sp.kp(), c->wb_conv[br][l].as<bf16>()); hdb::note_launch();
    }
  CK(c->wb1.ensure((size_t)kHid * kFeat * sizeof(bf16)));
  k_to_bf16<<<nblk((size_t)kHid * kFeat), 256, 0, s>>>(w + c->off_w1, c->wb1.as<bf16>(),
                                                       (size_t)kHid * kFeat); hdb::note_launch();
  return cudaGetLastError();
}

// C(m, n) (+)= sum_k A[m*lda + k] B[n*ldb + k] on the tcgen05 tensor cores
// (umma_gemm): both operands K-major; split K over `splits` CTAs per tile
// column, the splits added in order through c->tc_ws.
cudaError_t tc_gemm(hd_classifier c, int M, int N, int K, const bf16* A, long long lda,
                    const bf16* B, long long ldb, float* C, long long scm, long long scn,
                    int accumulate, int splits) {
  const size_t ws = hdb::umma_workspace_floats(M, N, K, splits);
  CK(c->tc_ws.ensure(std::max<size_t>(ws, 1) * sizeof(float)));
  CK(c->tc_err.ensure(sizeof(unsigned)));
  return hdb::umma_gemm(M, N, K, A, lda, B, ldb, C, scm, scn, accumulate, splits,
                        c->tc_ws.as<float>(), c->tc_err.as<unsigned>(), c->stream);
}

// Forward over the batch already in c->in[]; with backward, accumulates the
// gradients of the mean cross-entropy into c->g (which the caller zeroes).
cudaError_t run_batch(hd_classifier c, int nb, bool backward) {
  cudaStream_t s = c->stream;
  float* w = c->w.as<float>();
  float* g = c->g.as<float>();
  CK(refresh_bf16(c));
  // ---- forward ----
  for (int br = 0; br < 2; br++) {
    const bf16* cur = c->in[br].as<bf16>();
    for (int l = 0; l < 3; l++) {
      const ConvSpec& sp = kConv[br][l];
      const size_t P = (size_t)nb * sp.h * sp.w;
      // z [co][P] = W [co][kp] x col: on the tensor cores as z^T [P][co] =
      // colT [P][kp] x W^T, M = P pixels, N = co, K = kp
      const auto im2col = sp.ci == 1 ? k_im2col3_t<1> : sp.ci == 8 ? k_im2col3_t<8>
                                                                   : k_im2col3_t<16>;
      im2col<<<nblk(P, 128), 128, 0, s>>>(cur, sp.h, sp.w, P, c->col.as<bf16>()); hdb::note_launch();
      CK(tc_gemm(c, (int)P, sp.co, sp.kp(), c->col.as<bf16>(), sp.kp(),
                 c->wb_conv[br][l].as<bf16>(), sp.kp(), c->z.as<float>(), 1, (long long)P, 0,
                 1));
      k_bias_relu_pool<<<dim3(nblk(P / 8), sp.co), 256, 0, s>>>(
          c->z.as<float>(), w + c->off_b[br][l], nb, sp.h, sp.w,
          c->act[br][l].as<bf16>(), c->arg[br][l].as<unsigned char>()); hdb::note_launch();
      cur = c->act[br][l].as<bf16>();
    }
  }
  k_flatten<<<nblk((size_t)nb * kFeat), 256, 0, s>>>(c->act[0][2].as<bf16>(),
                                                     c->act[1][2].as<bf16>(), nb,
                                                     c->x.as<bf16>()); hdb::note_launch();
  // z1 [16][b] = W1 x x: z1^T [b][16] = x [b][10240] x W1^T, K split over 64
  CK(tc_gemm(c, nb, kHid, kFeat, c->x.as<bf16>(), kFeat, c->wb1.as<bf16>(), kFeat,
             c->z1.as<float>(), 1, nb, 0, 64));
  k_fc1_act<<<nblk((size_t)nb * kHid), 256, 0, s>>>(c->z1.as<float>(), w + c->off_b1, nb,
                                                    c->h.as<float>()); hdb::note_launch();
  if (backward) CK(cudaMemsetAsync(c->loss.p, 0, sizeof(float), s));
  k_head<<<nblk(nb, 128), 128, 0, s>>>(c->h.as<float>(), w + c->off_w2, w + c->off_b2,
                                       c->labels.as<int>(), nb, backward ? 1 : 0,
                                       c->prob.as<float>(), c->dz1.as<bf16>(),
                                       c->hs.as<float>()); hdb::note_launch();
  if (!backward) return cudaGetLastError();
  k_head_reduce<<<1, 256, 0, s>>>(c->h.as<float>(), c->hs.as<float>(), nb, c->loss.as<float>(),
                                 g + c->off_w2, g + c->off_b2, g + c->off_b1); hdb::note_launch();
  // ---- backward ----
  {
    k_fc1_wgrad<<<kFeat / 128, 256, 0, s>>>(c->dz1.as<bf16>(), c->x.as<bf16>(), nb,
                                           g + c->off_w1); hdb::note_launch();
    // dx [b][10240] = dz1^T x W1
    GemmArgs gd{kFeat, nb, kHid, c->wb1.as<bf16>(), 1, kFeat, c->dz1.as<bf16>(), nb, 1,
                c->dx.as<float>(), 1, kFeat, 0, 0};
    CK(gemm(gd, 1, s));
  }
  k_unflatten<<<nblk((size_t)nb * kFeat), 256, 0, s>>>(c->dx.as<float>(), nb,
                                                       c->dact_a[0].as<float>(),
                                                       c->dact_a[1].as<float>()); hdb::note_launch();
  BiasSum bias{};
  int chan = 0, layer = 0;
  for (int br = 0; br < 2; br++) {
    float* dcur = c->dact_a[br].as<float>();   // gradient of this layer's pooled output
    float* dnext = c->dact_b[br].as<float>();  // gradient of its input
    for (int l = 2; l >= 0; l--) {
      const ConvSpec& sp = kConv[br][l];
      const size_t P = (size_t)nb * sp.h * sp.w;
      const int parts = (int)std::min<size_t>(kBiasParts, nblk(P / 16));
      k_pool_relu_back<<<dim3(parts, sp.co), 256, 0, s>>>(
          dcur, c->act[br][l].as<bf16>(), c->arg[br][l].as<unsigned char>(), nb, sp.h, sp.w,
          c->dz.as<bf16>(), c->bias_part.as<float>() + chan * kBiasParts); hdb::note_launch();
      bias.first[layer] = chan;
      bias.parts[layer] = parts;
      bias.out[layer] = g + c->off_b[br][l];
      chan += sp.co;
      layer++;
      // the layer's input again, as im2col (recomputed rather than stored)
      const bf16* lin = l == 0 ? c->in[br].as<bf16>() : c->act[br][l - 1].as<bf16>();
      k_im2col3<<<dim3(nblk(P / 8), sp.ci), 256, 0, s>>>(lin, sp.h, sp.w, P,
                                                         c->col.as<bf16>()); hdb::note_launch();
      // dW [co][kw] += dz [co][P] x col^T, without the padded taps kw..kp:
      // on the tensor cores as dW^T [kw][co] += col [kw][P] x dz^T: M = kw
      // taps, N = co, K = P pixels split over the SMs; the splits are added
      // in order (the same gradient every run)
      const int splits = (int)std::min<size_t>(296, (P + 1023) / 1024);
      CK(tc_gemm(c, sp.kw(), sp.co, (int)P, c->col.as<bf16>(), (long long)P, c->dz.as<bf16>(),
                 (long long)P, g + c->off_w[br][l], 1, sp.kw(), 1, splits));
      if (l > 0) {
        // the gradient of the previous layer's output
        const bf16* dz = c->dz.as<bf16>();
        const bf16* wb = c->wb_conv[br][l].as<bf16>();
        CK(br == 0 ? (l == 1 ? launch_dgrad3<8, 16, 32, 32, 8>(dz, wb, nb, dnext, s)
                             : launch_dgrad3<16, 32, 16, 16, 16>(dz, wb, nb, dnext, s))
                   : (l == 1 ? launch_dgrad3<8, 16, 32, 128, 4>(dz, wb, nb, dnext, s)
                             : launch_dgrad3<16, 32, 16, 64, 4>(dz, wb, nb, dnext, s)));
        std::swap(dcur, dnext);
      }
    }
  }
  bias.first[layer] = chan;
  k_bias_sum<<<chan, 32, 0, s>>>(c->bias_part.as<float>(), bias); hdb::note_launch();
  return cudaGetLastError();
}

cudaError_t upload_patches(hd_classifier c, const float* dm, const float* ft, int nb) {
  cudaStream_t s = c->stream;
  // host floats -> device BF16 through a temporary FP32 copy
  CK(c->in_f32.ensure((size_t)nb * 16384 * sizeof(float)));
  CK(cudaMemcpyAsync(c->in_f32.p, dm, (size_t)nb * 4096 * sizeof(float), cudaMemcpyHostToDevice, s));
  k_input_bf16<<<nblk((size_t)nb * 4096), 256, 0, s>>>(c->in_f32.as<float>(), c->in[0].as<bf16>(),
                                                       (size_t)nb * 4096); hdb::note_launch();
  CK(cudaMemcpyAsync(c->in_f32.p, ft, (size_t)nb * 16384 * sizeof(float), cudaMemcpyHostToDevice, s));
  k_input_bf16<<<nblk((size_t)nb * 16384), 256, 0, s>>>(c->in_f32.as<float>(), c->in[1].as<bf16>(),
                                                        (size_t)nb * 16384); hdb::note_launch();
  return cudaGetLastError();
}

// The fused inference kernel over n device FP32 patch pairs -> d_prob.
cudaError_t infer(hd_classifier c, const float* d_dm, const float* d_ft, size_t n, float* d_prob) {
  cudaStream_t s = c->stream;
  if (n > 0x7FFFFFFFull) return cudaErrorInvalidValue;
  CK(refresh_bf16(c));
  if (c->nsm == 0) {
    CK(cudaDeviceGetAttribute(&c->nsm, cudaDevAttrMultiProcessorCount, c->device));
    CK(cudaFuncSetAttribute(hdb::inf::k_clf_infer, cudaFuncAttributeMaxDynamicSharedMemorySize,
                            (int)hdb::inf::kSmem));
  }
  hdb::inf::Args a{};
  a.dm = d_dm;
  a.ft = d_ft;
  a.n = (int)n;
  a.w = c->w.as<float>();
  for (int br = 0; br < 2; br++)
    for (int l = 0; l < 3; l++) {
      a.off_w[br][l] = (int)c->off_w[br][l];
      a.off_b[br][l] = (int)c->off_b[br][l];
    }
  a.off_b1 = (int)c->off_b1;
  a.off_w2 = (int)c->off_w2;
  a.off_b2 = (int)c->off_b2;
  a.wb1 = c->wb1.as<bf16>();
  a.prob = d_prob;
  const unsigned grid = (unsigned)std::min<size_t>(n, (size_t)c->nsm);
  hdb::inf::k_clf_infer<<<grid, hdb::inf::kThreads, hdb::inf::kSmem, s>>>(a); hdb::note_launch();
  return cudaGetLastError();
}

// Scores of n patch pairs (device FP32, or host FP32 staged in chunks); after
// `after` (an event on another stream, or null) when the patches come from
// that stream.  Device time between the events ev[0] and ev[1].
constexpr size_t kStageChunk = 2048;
cudaError_t score_batches(hd_classifier c, const float* dm, const float* ft, size_t n,
                          bool on_device, cudaEvent_t after, float* scores) {
  cudaStream_t s = c->stream;
  if (after) CK(cudaStreamWaitEvent(s, after, 0));
  CK(cudaEventRecord(c->ev[0], s));
  if (on_device) {
    CK(c->sprob.ensure(n * sizeof(float)));
    CK(infer(c, dm, ft, n, c->sprob.as<float>()));
    CK(cudaMemcpyAsync(scores, c->sprob.p, n * sizeof(float), cudaMemcpyDeviceToHost, s));
  } else {
    const size_t ch = std::min(n, kStageChunk);
    CK(c->stage_dm.ensure(ch * 4096 * sizeof(float)));
    CK(c->stage_ft.ensure(ch * 16384 * sizeof(float)));
    CK(c->sprob.ensure(ch * sizeof(float)));
    for (size_t i0 = 0; i0 < n; i0 += ch) {
      // the staging buffers are reused by the next chunk, whose copies are
      // ordered after this chunk's kernel on the same stream
      const size_t k = std::min(ch, n - i0);
      CK(cudaMemcpyAsync(c->stage_dm.p, dm + i0 * 4096, k * 4096 * sizeof(float),
                         cudaMemcpyHostToDevice, s));
      CK(cudaMemcpyAsync(c->stage_ft.p, ft + i0 * 16384, k * 16384 * sizeof(float),
                         cudaMemcpyHostToDevice, s));
      CK(infer(c, c->stage_dm.as<float>(), c->stage_ft.as<float>(), k, c->sprob.as<float>()));
      CK(cudaMemcpyAsync(scores + i0, c->sprob.p, k * sizeof(float), cudaMemcpyDeviceToHost, s));
    }
  }
  CK(cudaEventRecord(c->ev[1], s));
  CK(cudaStreamSynchronize(s));
  return cudaEventElapsedTime(&c->score_ms, c->ev[0], c->ev[1]);
}

// the tensor-core GEMM's error word: zeroed before a run, read after it
cudaError_t tc_reset(hd_classifier c) {
  CK(c->tc_err.ensure(sizeof(unsigned)));
  return cudaMemsetAsync(c->tc_err.p, 0, sizeof(unsigned), c->stream);
}
cudaError_t tc_check(hd_classifier c) {
  unsigned v = 0;
  CK(cudaMemcpy(&v, c->tc_err.p, sizeof(unsigned), cudaMemcpyDeviceToHost));
  return v ? cudaErrorLaunchTimeout : cudaSuccess;
}

hd_error to_hd(cudaError_t e) {
  if (e == cudaSuccess) return HD_NO_ERROR;
  if (e == cudaErrorMemoryAllocation) return HD_MEM_ALLOC_FAILED;
  return HD_INTERNAL_GPU_ERROR;
}

}  // namespace

extern "C" {

hd_size hd_classifier_param_count(void) {
  size_t n = 0;
  for (int br = 0; br < 2; br++)
    for (int l = 0; l < 3; l++) n += (size_t)kConv[br][l].co * kConv[br][l].kw() + kConv[br][l].co;
  return n + (size_t)kHid * kFeat + kHid + 2 * kHid + 2;
}

hd_error hd_classifier_create(hd_classifier* out, int gpu_id, unsigned long long seed) {
  if (!out) return HD_INVALID_POINTER;
  *out = nullptr;
  if (cudaSetDevice(gpu_id) != cudaSuccess) return HD_INVALID_DEVICE_INDEX;
  hd_classifier c = new (std::nothrow) hd_classifier_t();
  if (!c) return HD_MEM_ALLOC_FAILED;
  c->device = gpu_id;
  if (cudaStreamCreateWithFlags(&c->stream, cudaStreamNonBlocking) != cudaSuccess ||
      cudaEventCreate(&c->ev[0]) != cudaSuccess || cudaEventCreate(&c->ev[1]) != cudaSuccess) {
    delete c;
    return HD_PRIOR_GPU_ERROR;
  }
  size_t o = 0;
  for (int br = 0; br < 2; br++)
    for (int l = 0; l < 3; l++) {
      c->off_w[br][l] = o; o += (size_t)kConv[br][l].co * kConv[br][l].kw();
      c->off_b[br][l] = o; o += kConv[br][l].co;
    }
  c->off_w1 = o; o += (size_t)kHid * kFeat;
  c->off_b1 = o; o += kHid;
  c->off_w2 = o; o += 2 * kHid;
  c->off_b2 = o; o += 2;
  c->nparam = o;
  // He-normal initial weights (std sqrt(2 / fan_in)), zero conv biases
  std::vector<float> h(o, 0.f);
  std::mt19937_64 rng(seed);
  std::normal_distribution<float> nd(0.f, 1.f);
  auto fill = [&](size_t off, size_t n, int fan_in) {
    const float sd = std::sqrt(2.f / (float)fan_in);
    for (size_t i = 0; i < n; i++) h[off + i] = nd(rng) * sd;
  };
  for (int br = 0; br < 2; br++)
    for (int l = 0; l < 3; l++)
      fill(c->off_w[br][l], (size_t)kConv[br][l].co * kConv[br][l].kw(), kConv[br][l].kw());
  fill(c->off_w1, (size_t)kHid * kFeat, kFeat);
  fill(c->off_w2, 2 * kHid, kHid);
  // small positive FC1 biases keep the 16 hidden units active at the start
  for (int o = 0; o < kHid; o++) h[c->off_b1 + o] = 0.1f;
  cudaError_t e = c->w.ensure(o * sizeof(float));
  if (e == cudaSuccess) e = c->g.ensure(o * sizeof(float));
  if (e == cudaSuccess) e = c->m.ensure(o * sizeof(float));
  if (e == cudaSuccess) e = c->v.ensure(o * sizeof(float));
  if (e == cudaSuccess) e = cudaMemcpy(c->w.p, h.data(), o * sizeof(float), cudaMemcpyHostToDevice);
  if (e == cudaSuccess) e = cudaMemset(c->m.p, 0, o * sizeof(float));
  if (e == cudaSuccess) e = cudaMemset(c->v.p, 0, o * sizeof(float));
  if (e != cudaSuccess) {
    delete c;
    return to_hd(e);
  }
  *out = c;
  return HD_NO_ERROR;
}

void hd_classifier_destroy(hd_classifier c) {
  if (!c) return;
  cudaSetDevice(c->device);
  delete c;
}

hd_error hd_classifier_get_params(hd_classifier c, float* params, hd_size count) {
  if (!c) return HD_INVALID_PIPELINE;
  if (!params || count != c->nparam) return HD_INVALID_POINTER;
  cudaSetDevice(c->device);
  return to_hd(cudaMemcpy(params, c->w.p, c->nparam * sizeof(float), cudaMemcpyDeviceToHost));
}

hd_error hd_classifier_set_params(hd_classifier c, const float* params, hd_size count) {
  if (!c) return HD_INVALID_PIPELINE;
  if (!params || count != c->nparam) return HD_INVALID_POINTER;
  cudaSetDevice(c->device);
  c->bf16_stale = true;
  c->step = 0;
  cudaError_t e = cudaMemcpy(c->w.p, params, c->nparam * sizeof(float), cudaMemcpyHostToDevice);
  if (e == cudaSuccess) e = cudaMemset(c->m.p, 0, c->nparam * sizeof(float));
  if (e == cudaSuccess) e = cudaMemset(c->v.p, 0, c->nparam * sizeof(float));
  return to_hd(e);
}

hd_error hd_classifier_gradients(hd_classifier c, const float* dm_time, const float* freq_time,
                                 const int* labels, hd_size n, float* grads, float* loss) {
  if (!c) return HD_INVALID_PIPELINE;
  if (!dm_time || !freq_time || !labels || n == 0 || n > 4096) return HD_INVALID_POINTER;
  cudaSetDevice(c->device);
  cudaStream_t s = c->stream;
  cudaError_t e = alloc_batch(c, (int)n);
  if (e == cudaSuccess) e = tc_reset(c);
  if (e == cudaSuccess) e = upload_patches(c, dm_time, freq_time, (int)n);
  if (e == cudaSuccess) e = cudaMemcpyAsync(c->labels.p, labels, n * sizeof(int), cudaMemcpyHostToDevice, s);
  if (e == cudaSuccess) e = cudaMemsetAsync(c->g.p, 0, c->nparam * sizeof(float), s);
  if (e == cudaSuccess) e = run_batch(c, (int)n, true);
  if (e == cudaSuccess && grads)
    e = cudaMemcpyAsync(grads, c->g.p, c->nparam * sizeof(float), cudaMemcpyDeviceToHost, s);
  if (e == cudaSuccess && loss) e = cudaMemcpyAsync(loss, c->loss.p, sizeof(float), cudaMemcpyDeviceToHost, s);
  if (e == cudaSuccess) e = cudaStreamSynchronize(s);
  if (e == cudaSuccess) e = tc_check(c);
  return to_hd(e);
}

hd_error hd_classifier_train(hd_classifier c, const float* dm_time, const float* freq_time,
                             const int* labels, hd_size n, int epochs, int batch, float lr,
                             unsigned long long seed, float* epoch_loss) {
  if (!c) return HD_INVALID_PIPELINE;
  if (!dm_time || !freq_time || !labels || n == 0 || epochs <= 0 || batch <= 0 || batch > 4096)
    return HD_INVALID_POINTER;
  cudaSetDevice(c->device);
  cudaStream_t s = c->stream;
  const int nb = (int)std::min<size_t>(batch, n);
  cudaError_t e = alloc_batch(c, nb);
  if (e == cudaSuccess) e = tc_reset(c);
  // the training set stays on the device in BF16
  if (e == cudaSuccess) e = c->data_dm.ensure(n * 4096 * sizeof(bf16));
  if (e == cudaSuccess) e = c->data_ft.ensure(n * 16384 * sizeof(bf16));
  if (e == cudaSuccess) e = c->data_lab.ensure(n * sizeof(int));
  if (e != cudaSuccess) return to_hd(e);
  for (size_t i0 = 0; i0 < n && e == cudaSuccess; i0 += (size_t)nb) {
    const int k = (int)std::min<size_t>(nb, n - i0);
    e = upload_patches(c, dm_time + i0 * 4096, freq_time + i0 * 16384, k);
    if (e == cudaSuccess)
      e = cudaMemcpyAsync(c->data_dm.as<bf16>() + i0 * 4096, c->in[0].p, (size_t)k * 4096 * sizeof(bf16),
                          cudaMemcpyDeviceToDevice, s);
    if (e == cudaSuccess)
      e = cudaMemcpyAsync(c->data_ft.as<bf16>() + i0 * 16384, c->in[1].p, (size_t)k * 16384 * sizeof(bf16),
                          cudaMemcpyDeviceToDevice, s);
  }
  if (e == cudaSuccess)
    e = cudaMemcpyAsync(c->data_lab.p, labels, n * sizeof(int), cudaMemcpyHostToDevice, s);
  std::vector<int> order(n);
  for (size_t i = 0; i < n; i++) order[i] = (int)i;
  std::mt19937_64 rng(seed);
  std::vector<int> bidx(nb);
  for (int ep = 0; ep < epochs && e == cudaSuccess; ep++) {
    std::shuffle(order.begin(), order.end(), rng);
    double lsum = 0.0;
    int nbatches = 0;
    for (size_t i0 = 0; i0 + (size_t)nb <= n && e == cudaSuccess; i0 += (size_t)nb) {
      for (int j = 0; j < nb; j++) bidx[j] = order[i0 + j];
      e = cudaMemcpyAsync(c->idx.p, bidx.data(), nb * sizeof(int), cudaMemcpyHostToDevice, s);
      if (e != cudaSuccess) break;
      k_gather<<<nblk((size_t)nb * 4096), 256, 0, s>>>(c->data_dm.as<bf16>(), c->idx.as<int>(), nb, 4096,
                                                       c->in[0].as<bf16>()); hdb::note_launch();
      k_gather<<<nblk((size_t)nb * 16384), 256, 0, s>>>(c->data_ft.as<bf16>(), c->idx.as<int>(), nb, 16384,
                                                        c->in[1].as<bf16>()); hdb::note_launch();
      // labels of the batch (gather of one int per sample)
      {
        std::vector<int> hl(nb);
        for (int j = 0; j < nb; j++) hl[j] = labels[bidx[j]];
        e = cudaMemcpyAsync(c->labels.p, hl.data(), nb * sizeof(int), cudaMemcpyHostToDevice, s);
        if (e == cudaSuccess) e = cudaStreamSynchronize(s);  // hl and bidx are reused
      }
      if (e == cudaSuccess) e = cudaMemsetAsync(c->g.p, 0, c->nparam * sizeof(float), s);
      if (e == cudaSuccess) e = run_batch(c, nb, true);
      if (e != cudaSuccess) break;
      c->step++;
      const float b1 = 0.9f, b2 = 0.999f;
      const float c1 = 1.f - (float)std::pow(b1, (double)c->step);
      const float c2 = 1.f - (float)std::pow(b2, (double)c->step);
      c->bf16_stale = true;
      k_adam<<<nblk(c->nparam), 256, 0, s>>>(c->w.as<float>(), c->g.as<float>(), c->m.as<float>(),
                                             c->v.as<float>(), c->nparam, lr, b1, b2, 1e-8f, c1, c2); hdb::note_launch();
      float l = 0.f;
      e = cudaMemcpyAsync(&l, c->loss.p, sizeof(float), cudaMemcpyDeviceToHost, s);
      if (e == cudaSuccess) e = cudaStreamSynchronize(s);
      lsum += l;
      nbatches++;
    }
    if (epoch_loss) epoch_loss[ep] = nbatches ? (float)(lsum / nbatches) : 0.f;
  }
  if (e == cudaSuccess) e = cudaStreamSynchronize(s);
  if (e == cudaSuccess) e = tc_check(c);
  return to_hd(e);
}

hd_error hd_classifier_score(hd_classifier c, const float* dm_time, const float* freq_time,
                             hd_size n, float* scores) {
  if (!c) return HD_INVALID_PIPELINE;
  if (!dm_time || !freq_time || !scores) return HD_INVALID_POINTER;
  if (n == 0) return HD_NO_ERROR;
  cudaSetDevice(c->device);
  return to_hd(score_batches(c, dm_time, freq_time, n, false, nullptr, scores));
}

hd_error hd_classifier_score_device(hd_classifier c, const float* d_dm_time,
                                    const float* d_freq_time, hd_size n, float* scores) {
  if (!c) return HD_INVALID_PIPELINE;
  if (!d_dm_time || !d_freq_time || !scores) return HD_INVALID_POINTER;
  if (n == 0) return HD_NO_ERROR;
  cudaSetDevice(c->device);
  return to_hd(score_batches(c, d_dm_time, d_freq_time, n, true, nullptr, scores));
}

hd_error hd_classifier_get_timing(hd_classifier c, float* ms) {
  if (!c) return HD_INVALID_PIPELINE;
  if (!ms) return HD_INVALID_POINTER;
  *ms = c->score_ms;
  return HD_NO_ERROR;
}

hd_error hd_bf16_gemm_tc(int m, int n, int k, const void* d_a, long long sam, long long sak,
                         const void* d_b, long long sbk, long long sbn, float* d_c,
                         long long scm, long long scn, int accumulate, int splits) {
  if (!d_a || !d_b || !d_c) return HD_INVALID_POINTER;
  if (sak != 1 || sbk != 1) return HD_INVALID_STRIDE;
  float* ws = nullptr;
  unsigned* err = nullptr;
  const size_t nws = hdb::umma_workspace_floats(m, n, k, splits);
  cudaError_t e = hdb::dev_malloc(&err, sizeof(unsigned));
  if (e == cudaSuccess && nws) e = hdb::dev_malloc(&ws, nws * sizeof(float));
  if (e == cudaSuccess) e = cudaMemset(err, 0, sizeof(unsigned));
  if (e == cudaSuccess)
    e = hdb::umma_gemm(m, n, k, d_a, sam, d_b, sbn, d_c, scm, scn, accumulate, splits, ws, err, 0);
  hd_error he = HD_NO_ERROR;
  if (e == cudaErrorNotSupported) he = HD_INVALID_STRIDE;
  else if (e == cudaSuccess) e = cudaDeviceSynchronize();
  unsigned v = 0;
  if (he == HD_NO_ERROR && e == cudaSuccess) {
    e = cudaMemcpy(&v, err, sizeof(unsigned), cudaMemcpyDeviceToHost);
    if (e == cudaSuccess && v) he = HD_INTERNAL_GPU_ERROR;
  }
  if (he == HD_NO_ERROR) he = to_hd(e);
  if (ws) cudaFree(ws);
  if (err) cudaFree(err);
  return he;
}

hd_error hd_bf16_gemm(int m, int n, int k, const void* d_a, long long sam, long long sak,
                      const void* d_b, long long sbk, long long sbn, float* d_c, long long scm,
                      long long scn, int accumulate, int splits) {
  if (!d_a || !d_b || !d_c) return HD_INVALID_POINTER;
  GemmArgs a{m, n, k, static_cast<const bf16*>(d_a), sam, sak, static_cast<const bf16*>(d_b),
             sbk, sbn, d_c, scm, scn, accumulate, 0};
  cudaError_t e = gemm(a, splits, 0);
  if (e == cudaSuccess) e = cudaDeviceSynchronize();
  return to_hd(e);
}

}  // extern "C"

namespace hdb {
cudaError_t classifier_score_device(hd_classifier c, const float* d_dm, const float* d_ft,
                                    size_t n, cudaEvent_t after, float* scores) {
  if (n == 0) return cudaSuccess;
  return score_batches(c, d_dm, d_ft, n, true, after, scores);
}
int classifier_device(hd_classifier c) { return c->device; }
}  // namespace hdb
