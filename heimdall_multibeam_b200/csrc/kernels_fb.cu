// kernels_fb.cu -- filterbank-side kernels: layout change, zero-DM series,
// RFI zapping and brute-force dedispersion.
//
// Filterbank layouts:
//   TF  (input, as the reference receives it): spectrum t at in + t*nchans,
//       one byte per channel (8-bit data).
//   FT  (device working copy): channel c at ft + c*pitch, one byte per sample,
//       pitch a multiple of 64 bytes, so that rows are read and written in
//       16-byte pieces (what lies past nsamps reaches no result).
//   Four-sample words (what dedispersion reads): k_split_words.
#include <algorithm>
#include <map>
#include <mutex>
#include <vector>

#include "common.cuh"
#include "internal.h"

namespace hdb {

static unsigned long long g_launches = 0;
void note_launch() { __atomic_add_fetch(&g_launches, 1ull, __ATOMIC_RELAXED); }
unsigned long long launch_count() { return __atomic_load_n(&g_launches, __ATOMIC_RELAXED); }
void add_launches(long long n) {
  __atomic_add_fetch(&g_launches, (unsigned long long)n, __ATOMIC_RELAXED);
}

cudaError_t raise_smem_limit(const void* func, size_t bytes) {
  static std::mutex m;
  static std::map<std::pair<int, const void*>, size_t> limit;
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  std::lock_guard<std::mutex> g(m);
  size_t& cur = limit[{dev, func}];
  if (bytes <= cur) return cudaSuccess;
  e = cudaFuncSetAttribute(func, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
  if (e == cudaSuccess) cur = bytes;
  return e;
}

// ---------------------------------------------------------------------------
// TF -> FT byte transpose, 128 samples x 128 channels per block through
// shared memory.  The tile holds 128 sample rows of 32 channel words; word w
// of row t sits at column w ^ (((t >> 2) ^ (t & 3)) & 31), so the row-wise
// stores of the load phase (a warp stores four consecutive rows at once in
// the 16-byte form) and the sample-wise loads of the store phase (lane l
// reads rows 4l..4l+3 of one column) all hit 32 distinct banks.  A thread turns four
// samples x four channels into four output words with byte permutes.  Rows
// of whole 16-byte words are loaded 16 bytes at a time.
// ---------------------------------------------------------------------------
__device__ __forceinline__ int tp_col(int t, int w) { return w ^ (((t >> 2) ^ (t & 3)) & 31); }

// The staged tile's channel rows from sample t0 on.  Warp: channel words warp,
// warp + 8, ...; lane: samples 4l .. 4l+3.
__device__ __forceinline__ void transpose_store(const uint32_t* tile, size_t t0, size_t nsamps,
                                                int c0, int nchans, uint8_t* __restrict__ out,
                                                size_t pitch) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const size_t t = t0 + 4 * lane;
  for (int ws = warp; ws < 32; ws += 8) {
    if (4 * ws + c0 >= nchans) break;
    uint32_t a[4];
#pragma unroll
    for (int j = 0; j < 4; j++) {
      const int r = 4 * lane + j;
      a[j] = tile[r * 32 + tp_col(r, ws)];
    }
    // 4 x 4 byte transpose: o[b] = byte b of a[0..3]
    const uint32_t lo01 = __byte_perm(a[0], a[1], 0x5140), lo23 = __byte_perm(a[2], a[3], 0x5140);
    const uint32_t hi01 = __byte_perm(a[0], a[1], 0x7362), hi23 = __byte_perm(a[2], a[3], 0x7362);
    const uint32_t o[4] = {__byte_perm(lo01, lo23, 0x5410), __byte_perm(lo01, lo23, 0x7632),
                           __byte_perm(hi01, hi23, 0x5410), __byte_perm(hi01, hi23, 0x7632)};
    if (t < nsamps) {
#pragma unroll
      for (int b = 0; b < 4; b++) {
        const int c = c0 + 4 * ws + b;
        if (c < nchans) reinterpret_cast<uint32_t*>(out + (size_t)c * pitch + t)[0] = o[b];
      }
    }
  }
}

__global__ void __launch_bounds__(256) k_transpose_tf_ft(const uint8_t* __restrict__ in,
                                                         size_t nsamps, int nchans,
                                                         uint8_t* __restrict__ out,
                                                         size_t pitch, size_t out_unit) {
  __shared__ uint32_t tile[128 * 32];
  // blockIdx.z: unit (independent filterbank) of a batch
  in += (size_t)blockIdx.z * nsamps * (size_t)nchans;
  out += (size_t)blockIdx.z * out_unit;
  const size_t t0 = (size_t)blockIdx.x * 128;
  const int c0 = blockIdx.y * 128;
  const int nwords = nchans >> 2;
  const int w0 = c0 >> 2;
  if ((nchans & 15) == 0 && (reinterpret_cast<uintptr_t>(in) & 15) == 0) {
    // thread: 16-byte chunk q of rows r, r + 32, r + 64, r + 96
    const int q = threadIdx.x & 7, r0 = threadIdx.x >> 3;
    uint4 v[4];
#pragma unroll
    for (int k = 0; k < 4; k++) {
      const int r = r0 + 32 * k;
      const size_t t = t0 + r;
      v[k] = make_uint4(0u, 0u, 0u, 0u);
      if (t < nsamps && w0 + 4 * q < nwords)
        v[k] = *reinterpret_cast<const uint4*>(in + t * nchans + (size_t)(w0 + 4 * q) * 4);
    }
#pragma unroll
    for (int k = 0; k < 4; k++) {
      const int r = r0 + 32 * k;
      tile[r * 32 + tp_col(r, 4 * q)] = v[k].x;
      tile[r * 32 + tp_col(r, 4 * q + 1)] = v[k].y;
      tile[r * 32 + tp_col(r, 4 * q + 2)] = v[k].z;
      tile[r * 32 + tp_col(r, 4 * q + 3)] = v[k].w;
    }
  } else {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    uint32_t v[16];
#pragma unroll
    for (int k = 0; k < 16; k++) {
      const size_t t = t0 + warp + 8 * k;
      v[k] = 0u;
      if (t < nsamps && w0 + lane < nwords)
        v[k] = reinterpret_cast<const uint32_t*>(in + t * nchans)[w0 + lane];
    }
#pragma unroll
    for (int k = 0; k < 16; k++) {
      const int r = warp + 8 * k;
      tile[r * 32 + tp_col(r, lane)] = v[k];
    }
  }
  __syncthreads();
  transpose_store(tile, t0, nsamps, c0, nchans, out, pitch);
}

// ---------------------------------------------------------------------------
// Packed TF -> byte FT rows for NB = 1, 2, 4 and 16 bits per sample.  A
// spectrum is C * NB / 32 little-endian 32-bit words; channel c is the NB-bit
// field at bit (c mod (32 / NB)) * NB of word c / (32 / NB) (the order of the
// reference's writer and cleaning functor: Formats/giant_maker.C:385-392,
// Pipeline/clean_filterbank_rfi.cu:86-90).  NB < 8 unpacks into one byte
// plane; NB = 16 splits each sample into its low byte (plane `out`) and high
// byte (plane `out + hi_off`), dedispersed separately and combined as
// lo + 256 hi (exact integer sums).  128 x 128 tiles through shared memory.
// ---------------------------------------------------------------------------
template <int NB>
__global__ void __launch_bounds__(256) k_unpack_tf_ft(const uint32_t* __restrict__ in,
                                                      size_t nsamps, int nchans,
                                                      uint8_t* __restrict__ out, size_t pitch,
                                                      size_t out_unit, size_t hi_off) {
  constexpr int CPW = 32 / NB;                 // channels per word
  constexpr int WPR = 128 / CPW;               // words per tile row
  constexpr uint32_t MASK = (NB == 32) ? 0xFFFFFFFFu : ((1u << NB) - 1u);
  __shared__ uint16_t vals[128][130];          // [t][channel]
  const size_t row_words = (size_t)nchans * NB / 32;
  in += (size_t)blockIdx.z * nsamps * row_words;
  out += (size_t)blockIdx.z * out_unit;
  const size_t t0 = (size_t)blockIdx.x * 128;
  const int c0 = blockIdx.y * 128;
  const size_t w0 = (size_t)c0 / CPW;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  for (int r = warp; r < 128; r += 8) {
    const size_t t = t0 + r;
    for (int w = lane; w < WPR; w += 32) {
      uint32_t v = 0;
      if (t < nsamps && w0 + w < row_words) v = in[t * row_words + w0 + w];
#pragma unroll
      for (int k = 0; k < CPW; k++) vals[r][w * CPW + k] = (uint16_t)((v >> (k * NB)) & MASK);
    }
  }
  __syncthreads();
  for (int cr = warp; cr < 128; cr += 8) {
    const int c = c0 + cr;
    if (c >= nchans) break;
    const size_t t = t0 + 4 * lane;
    if (t >= nsamps) continue;
    uint32_t lo = 0, hi = 0;
#pragma unroll
    for (int j = 0; j < 4; j++) {
      const uint32_t v = vals[4 * lane + j][cr];
      lo |= (v & 0xFFu) << (8 * j);
      hi |= (v >> 8) << (8 * j);
    }
    reinterpret_cast<uint32_t*>(out + (size_t)c * pitch + t)[0] = lo;
    if (NB == 16) reinterpret_cast<uint32_t*>(out + hi_off + (size_t)c * pitch + t)[0] = hi;
  }
}

// rows x n floats (pitch apart): lo = RN(lo + 256 hi), both exact integer sums
__global__ void k_combine_planes(float* __restrict__ lo, const float* __restrict__ hi,
                                 size_t pitch, size_t n, size_t rows) {
  const size_t total = rows * n;
  for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < total;
       i += (size_t)gridDim.x * blockDim.x) {
    const size_t r = i / n, k = i - r * n;
    const size_t at = r * pitch + k;
    lo[at] = __uint2float_rn(__float2uint_rn(lo[at]) + 256u * __float2uint_rn(hi[at]));
  }
}

// ---------------------------------------------------------------------------
// Zero-DM series: s[t] = (float) sum_c in[t][c]  (dedisp at DM 0, all channels;
// Pipeline/clean_filterbank_rfi.cu:361-397).  One warp per spectrum.
// ---------------------------------------------------------------------------
__global__ void __launch_bounds__(256) k_dm0_sum(const uint8_t* __restrict__ in, size_t nsamps,
                                                 int nchans, float* __restrict__ s) {
  size_t t = (size_t)blockIdx.x * 8 + (threadIdx.x >> 5);
  int lane = threadIdx.x & 31;
  if (t >= nsamps) return;
  const uint32_t* row = reinterpret_cast<const uint32_t*>(in + t * nchans);
  unsigned acc = 0;
  for (int w = lane; w < (nchans >> 2); w += 32) acc = __dp4a(row[w], 0x01010101u, acc);
#pragma unroll
  for (int o = 16; o; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
  if (lane == 0) s[t] = (float)(int)acc;
}

// ---------------------------------------------------------------------------
// Broadband zapping (Pipeline/clean_filterbank_rfi.cu:33-113,197-234).
// ---------------------------------------------------------------------------
// Robert Jenkins' 32-bit integer mix.
__device__ __forceinline__ uint32_t mix32(uint32_t a) {
  a = (a + 0x7ed55d16u) + (a << 12);
  a = (a ^ 0xc761c23cu) ^ (a >> 19);
  a = (a + 0x165667b1u) + (a << 5);
  a = (a + 0xd3a2646cu) ^ (a << 9);
  a = (a + 0xfd7046c5u) + (a << 3);
  a = (a ^ 0xb55a4f09u) ^ (a >> 16);
  return a;
}

// Park-Miller minimal standard (a = 48271, m = 2^31 - 1) and Thrust's integer
// distribution: a double in [lo, hi + 1) from (x - 1) / (2^31 - 2), truncated.
__device__ __forceinline__ uint32_t minstd_next(uint32_t& s) {
  s = (uint32_t)((48271ull * (unsigned long long)s) % 2147483647ull);
  return s;
}
__device__ __forceinline__ uint32_t uniform_uint(uint32_t& s, uint32_t lo, uint32_t hi) {
  double a = (double)lo;
  double b = __dadd_rn((double)hi, 1.0);
  double u = (double)(minstd_next(s) - 1u);
  u = __ddiv_rn(u, 2147483646.0);
  double r = __dadd_rn(__dmul_rn(u, __dsub_rn(b, a)), a);
  return __double2uint_rz(r);
}

__device__ uint32_t zap_word(const uint32_t* __restrict__ win, const int* __restrict__ mask,
                             unsigned i, unsigned t, unsigned c, unsigned stride, unsigned ns,
                             unsigned r) {
  uint32_t s = mix32(i) % 2147483647u;
  if (s == 0) s = 1;
  uint32_t result = 0;
#pragma unroll 1
  for (unsigned k = 0; k < 32; k += 8) {
    unsigned min_t = t > r ? t - r : 0;
    unsigned max_t = t < ns - 1 - r ? t + r : ns - 1;
    unsigned nt = uniform_uint(s, min_t, max_t);
    int attempts = 0;
    while (mask[nt] && ++attempts < 11) nt = uniform_uint(s, min_t, max_t);
    uint32_t v = (win[nt * stride + c] >> k) & 0xFFu;
    result |= v << k;
  }
  return result;
}

// Zap masked spectra and write the result channel-major (FT), and optionally
// time-major (TF) for callers that want the cleaned filterbank back.  Bound by
// its reads and writes: the transpose's tile and word order, rows of whole
// 16-byte words loaded 16 bytes at a time, and the masked rows filled in by a
// warp each, a word per lane (their draws are long and few).  1024 channels x
// 262144 samples: 330 us with a word per lane in every row and bytes gathered
// one by one, 165 us so.
__global__ void __launch_bounds__(256) k_zap_to_ft(const uint8_t* __restrict__ in, size_t nsamps,
                                                   int nchans, const int* __restrict__ mask,
                                                   unsigned max_resample_dist,
                                                   uint8_t* __restrict__ out_ft, size_t pitch,
                                                   uint8_t* __restrict__ out_tf) {
  __shared__ uint32_t tile[128 * 32];
  const size_t t0 = (size_t)blockIdx.x * 128;
  const int c0 = blockIdx.y * 128;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const unsigned stride = (unsigned)(nchans >> 2);
  const unsigned w0 = (unsigned)(c0 >> 2);
  const uint32_t* win = reinterpret_cast<const uint32_t*>(in);
  // ---- the rows that stay as they are ----
  if ((nchans & 15) == 0 &&
      ((reinterpret_cast<uintptr_t>(in) | reinterpret_cast<uintptr_t>(out_tf)) & 15) == 0) {
    // thread: 16-byte chunk q of rows r0, r0 + 32, r0 + 64, r0 + 96
    const int q = threadIdx.x & 7, r0 = threadIdx.x >> 3;
    const unsigned w = w0 + 4 * q;
    uint4 v[4];
    bool masked[4];
#pragma unroll
    for (int k = 0; k < 4; k++) {
      const size_t t = t0 + r0 + 32 * k;
      const bool in_data = t < nsamps && w < stride;
      v[k] = make_uint4(0u, 0u, 0u, 0u);
      masked[k] = t < nsamps && mask[t] != 0;
      if (in_data) v[k] = *reinterpret_cast<const uint4*>(win + t * stride + w);
    }
#pragma unroll
    for (int k = 0; k < 4; k++) {
      if (masked[k]) continue;
      const int r = r0 + 32 * k;
      tile[r * 32 + tp_col(r, 4 * q)] = v[k].x;
      tile[r * 32 + tp_col(r, 4 * q + 1)] = v[k].y;
      tile[r * 32 + tp_col(r, 4 * q + 2)] = v[k].z;
      tile[r * 32 + tp_col(r, 4 * q + 3)] = v[k].w;
      if (out_tf && t0 + r < nsamps && w < stride)
        *reinterpret_cast<uint4*>(reinterpret_cast<uint32_t*>(out_tf) + (t0 + r) * stride + w) =
            v[k];
    }
  } else {
    for (int r = warp; r < 128; r += 8) {
      const size_t t = t0 + r;
      if (t < nsamps && mask[t]) continue;
      const bool in_data = t < nsamps && w0 + lane < stride;
      const uint32_t v = in_data ? win[t * stride + w0 + lane] : 0u;
      tile[r * 32 + tp_col(r, lane)] = v;
      if (out_tf && in_data) reinterpret_cast<uint32_t*>(out_tf)[t * stride + w0 + lane] = v;
    }
  }
  // ---- the masked rows: warp w those of rows w, w + 8, ... ----
  const size_t tl = t0 + warp + 8 * lane;
  unsigned todo = __ballot_sync(0xffffffffu, lane < 16 && tl < nsamps && mask[tl] != 0);
  for (; todo; todo &= todo - 1) {
    const int r = warp + 8 * (__ffs(todo) - 1);
    const unsigned t = (unsigned)(t0 + r), w = w0 + lane;
    uint32_t v = 0u;
    if (w < stride) {
      v = zap_word(win, mask, t * stride + w, t, w, stride, (unsigned)nsamps, max_resample_dist);
      if (out_tf) reinterpret_cast<uint32_t*>(out_tf)[(size_t)t * stride + w] = v;
    }
    tile[r * 32 + tp_col(r, lane)] = v;
  }
  if (!out_ft) return;
  __syncthreads();
  transpose_store(tile, t0, nsamps, c0, nchans, out_ft, pitch);
}

// ---------------------------------------------------------------------------
// Narrow-band RFI: the branch of Pipeline/clean_filterbank_rfi.cu:303-351 that
// the reference disables (measure_bandpass.cu:45-275 and
// zap_narrow_rfi_functor, clean_filterbank_rfi.cu:114-193).  The data are cut
// into stretches of baseline_length / dt spectra per filterbank (unit); each
// stretch gets its own bandpass and band deviation from 3125 spectra drawn
// with thrust::default_random_engine(123456), and its bytes are zapped
// against them.
// ---------------------------------------------------------------------------
constexpr int NB_SPECTRA = 3125;

// spectrum draws of each stretch, in order (measure_bandpass.cu:95-108)
__global__ void k_nb_indices(const unsigned* __restrict__ len, int nstretch,
                             unsigned* __restrict__ idx) {
  const int g = blockIdx.x * blockDim.x + threadIdx.x;
  if (g >= nstretch) return;
  uint32_t st = 123456u;
  for (int i = 0; i < NB_SPECTRA; i++)
    idx[(size_t)g * NB_SPECTRA + i] = uniform_uint(st, 0u, len[g] - 1u);
}

// spectra[g][i][c] = (float) fb[(start[g] + idx[g][i]) * C + c]
__global__ void k_nb_gather(const uint8_t* __restrict__ fb, int C,
                            const unsigned long long* __restrict__ start,
                            const unsigned* __restrict__ idx, size_t total,
                            float* __restrict__ out) {
  for (size_t e = (size_t)blockIdx.x * blockDim.x + threadIdx.x; e < total;
       e += (size_t)gridDim.x * blockDim.x) {
    const size_t gi = e / C;
    const int c = (int)(e % C);
    const size_t g = gi / NB_SPECTRA;
    out[e] = (float)fb[(size_t)(start[g] + idx[gi]) * C + c];
  }
}

// one level of the recursive median: out[g][a][c] = median of in[g][5a..5a+4][c]
__global__ void k_nb_scrunch5(const float* __restrict__ in, int C, int count_in, int nstretch,
                              float* __restrict__ out) {
  const int count_out = count_in / 5;
  const size_t total = (size_t)nstretch * count_out * C;
  for (size_t e = (size_t)blockIdx.x * blockDim.x + threadIdx.x; e < total;
       e += (size_t)gridDim.x * blockDim.x) {
    const int c = (int)(e % C);
    const size_t r = e / C;
    const size_t a = r % count_out, g = r / count_out;
    const float* b = in + ((size_t)g * count_in + 5 * a) * C + c;
    out[e] = med5(b[0], b[C], b[2 * (size_t)C], b[3 * (size_t)C], b[4 * (size_t)C]);
  }
}

// median_filter5_kernel (median_filter.cu:99-124): window shrunk at the ends
__device__ __forceinline__ float nb_filter5(const float* in, unsigned count, unsigned i) {
  if (i > 1 && i < count - 2) return med5(in[i - 2], in[i - 1], in[i], in[i + 1], in[i + 2]);
  if (i == 0) return med3(in[i], in[i + 1], in[i + 2]);
  if (i == 1) return med4(in[i - 1], in[i], in[i + 1], in[i + 2]);
  if (i == count - 1) return med3(in[i], in[i - 1], in[i - 2]);
  return med4(in[i + 1], in[i], in[i - 1], in[i - 2]);
}

// measure_bandpass.cu:141-163 / 220-245 on v[g] (C values, scaled first by
// `scale` unless it is 1): scrunch by 5, 5-wide median, mean of neighbours
// (thrust::adjacent_difference), stretch to C/5*5 and extrapolate the rest.
// One block per stretch; tmp[g] holds C/5 values.
__global__ void k_nb_smooth(float* __restrict__ v, float* __restrict__ tmp, int C, float scale) {
  float* x = v + (size_t)blockIdx.x * C;
  const unsigned n5 = (unsigned)C / 5;
  float* t = tmp + (size_t)blockIdx.x * (n5 + 1);
  if (scale != 1.f) {
    for (int i = threadIdx.x; i < C; i += blockDim.x) x[i] = __fmul_rn(x[i], scale);
    __syncthreads();
  }
  for (unsigned j = threadIdx.x; j < n5; j += blockDim.x)
    t[j] = med5(x[5 * j], x[5 * j + 1], x[5 * j + 2], x[5 * j + 3], x[5 * j + 4]);
  __syncthreads();
  for (unsigned j = threadIdx.x; j < n5; j += blockDim.x) x[j] = nb_filter5(t, n5, j);
  __syncthreads();
  for (unsigned j = threadIdx.x; j < n5; j += blockDim.x)
    t[j] = j == 0 ? x[0] : __fmul_rn(0.5f, __fadd_rn(x[j], x[j - 1]));
  // for some channel counts (1140, 2220, ...) the last stretched sample lands
  // just past the last input with a fraction above 1e-5 and reads t[n5] (the
  // reference reads past its vector there): defined as 0
  if (threadIdx.x == 0) t[n5] = 0.f;
  __syncthreads();
  const float step = __fdiv_rn((float)(n5 - 1), (float)(n5 * 5 - 1));
  for (unsigned j = threadIdx.x; j < n5 * 5; j += blockDim.x) x[j] = stretch_at(t, j, step);
  __syncthreads();
  if (threadIdx.x == 0)
    for (unsigned i = n5 * 5; i < (unsigned)C; i++)
      x[i] = __fsub_rn(__fmul_rn(2.f, x[i - 1]), x[i - 2]);
}

// spectra[g][i][c] = |spectra[g][i][c] - bandpass[g][c]|
__global__ void k_nb_absdev(float* __restrict__ sp, const float* __restrict__ bp, int C,
                            size_t total) {
  for (size_t e = (size_t)blockIdx.x * blockDim.x + threadIdx.x; e < total;
       e += (size_t)gridDim.x * blockDim.x) {
    const size_t g = e / ((size_t)NB_SPECTRA * C);
    sp[e] = fabsf(__fsub_rn(sp[e], bp[g * C + e % C]));
  }
}

// rms[g] = the (C/2)-th smallest of mad[g] (std::nth_element), by ranks
__global__ void k_nb_rms(const float* __restrict__ mad, int C, float* __restrict__ rms) {
  const float* m = mad + (size_t)blockIdx.x * C;
  const int k = C / 2;
  for (int i = threadIdx.x; i < C; i += blockDim.x) {
    const float x = m[i];
    int lt = 0, le = 0;
    for (int j = 0; j < C; j++) {
      lt += m[j] < x;
      le += m[j] <= x;
    }
    if (lt <= k && k < le) rms[blockIdx.x] = x;  // equal values only
  }
}

// zap_narrow_rfi_functor over each spectrum's words in order (one thread per
// spectrum; draws read the spectrum as earlier words left it, the sequential
// semantics of the functor's in-place reads).  Bandpass entry and draw range
// use channel w + k as the reference does; the hash takes the word's index
// within its filterbank.
__global__ void k_nb_zap(uint32_t* __restrict__ data, size_t nsamps, int units, int C,
                         size_t nsmooth, int nsub, const float* __restrict__ bp,
                         const float* __restrict__ rms, float rfi_tol, unsigned max_dist) {
  const size_t tg = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (tg >= nsamps * (size_t)units) return;
  const size_t u = tg / nsamps, tl = tg % nsamps;
  const size_t g = u * nsub + tl / nsmooth;
  const float* b = bp + g * C;
  const float thresh = __fmul_rn(rfi_tol, rms[g]);
  const unsigned stride = (unsigned)C / 4, nch = (unsigned)C;
  uint32_t* row = data + tg * stride;
  for (unsigned w = 0; w < stride; w++) {
    const unsigned i = (unsigned)(tl * stride + w);
    uint32_t word = row[w];
    uint32_t st = mix32(i) % 2147483647u;
    if (st == 0) st = 1;
    bool any = false;
    for (unsigned k = 0; k < 4; k++) {
      const unsigned c = w + k;
      const uint32_t val = (word >> (k * 8)) & 0xFFu;
      if (fabsf(__fsub_rn(__uint2float_rn(val), b[c])) > thresh) {
        any = true;
        const unsigned min_c = c > max_dist ? c - max_dist : 0;
        const unsigned max_c = c < nch - 1 - max_dist ? c + max_dist : nch - 1;
        unsigned nc = uniform_uint(st, min_c, max_c);
        uint32_t nv = (row[nc / 4] >> ((nc % 4) * 8)) & 0xFFu;
        int attempts = 0;
        while (fabsf(__fsub_rn(__uint2float_rn(nv), b[nc])) > thresh && ++attempts < 11) {
          nc = uniform_uint(st, min_c, max_c);
          nv = (row[nc / 4] >> ((nc % 4) * 8)) & 0xFFu;
        }
        word &= ~(0xFFu << (k * 8));
        word |= nv << (k * 8);
      }
    }
    if (any) row[w] = word;
  }
}

// ---------------------------------------------------------------------------
// Brute-force dedispersion.
//
//   out[d][t] = (float) sum_{c active} in[c][t + delay[d][c]],  t < nout
//
// Input: four-sample words.  With S = split (a quarter of nout, rounded up to
// 16), word t of channel c holds the bytes of samples t, t + S, t + 2S and
// t + 3S (k_split_words).  A delay then moves whole words: word t + delay has
// the four samples that outputs t + q S need, so a (DM, channel) term is one
// shared-memory load at any delay, without realignment, and the 32 lanes'
// loads (consecutive words) are one conflict-free wavefront.
//
// CTA = DB = DPW*NWD DMs x TBW = 32*W*NWT words (4 TBW samples), NWD*NWT
// consumer warps + 1 producer warp.  The producer walks the active channels in
// stages: as many channel row segments [t0 + min_d delay - align, t0 + max_d
// delay + TBW) as fit a stage buffer, each at the length its own DM block and
// channel need, come by one 1-D bulk async copy (TMA, cp.async.bulk) each,
// with the shared-memory byte offset of every (DM, channel) window in a table.
// It loads the next stage's tables before it waits for a free buffer.  A
// `full` mbarrier announces a stage, consumer warps release it through an
// `empty` mbarrier (one arrival per warp).  There is no block-wide barrier in
// the main loop.  Every mbarrier wait is bounded; a wait that gives up sets
// bit 0 of a.err and the warp leaves its loop.
//
// A consumer lane owns words lane + 32 w of DPW DMs and keeps two 32-bit
// accumulators per word for its four sums (dd_dot).  After each run of at most
// 256 channels the sums of a word go to the output row: a single run is
// converted and stored; with more channels the row holds 32-bit integer
// partial sums (stored, then added to in L2) until the last run adds its own
// and stores the float.  The sums are exact integers in any order.  The runs may
// be those of several launches over a part of the channels each (sums_before,
// sums_after).
//
// What bounds it: one shared load per word, DM and channel (128 sample terms a
// wavefront), so the shared-memory pipe (84 % busy in ncu) and instruction
// issue (76 %).  Measured sample-channel adds per second, the tile from the
// autotuner, against the byte-row kernel before it (8 x 1280 samples, funnel
// shifts to realign): 4096 channels, DM 0-500: 28.2 T/s (19.2); 1024 channels,
// DM 0-2000: 26.7 (16.8); 256 channels, DM 0-1000: 20.4 (15.0); 36 x 320
// channels at 655 us: 24 (19.6).
// ---------------------------------------------------------------------------
// Two forms of a word's four sums, each two accumulators (raw, odd):
//   permute: the words modulo 2^32, and the odd bytes in 16-bit lanes;
//   dot:     S0 + 65535 S1 and S2 + 65535 S3 by 2-way dot products (every sum
//            <= 256 * 255 < 65535, so a remainder and a quotient give both
//            back).
// The permutes and 3-input adds issue to the ALU pipe and the dot products to
// the FMA pipe, so two words of three take the dot form.
constexpr uint32_t kDot = 0xFFFF0001u;
__host__ __device__ constexpr bool dd_dot(int w) { return w % 3 != 0; }

constexpr int DD_NST = 2;      // stages of the row ring
constexpr int DD_ROWS = kDedispRows;
constexpr int DD_RUN = 256;    // channels between two flushes at most

// CTAs per SM the register budget allows: two registers per owned word and DM
// plus about 48 others, and a quarter of the SM's registers per scheduler.
constexpr int dd_min_blocks(int warps, int words) {
  const int per_sched = 16384 / (32 * ((2 * words + 48 + 7) / 8 * 8));
  const int n = 4 * per_sched / (warps + 1);
  return n < 1 ? 1 : n > 5 ? 5 : n;
}

// PART: launches over a part of the channels each (sums_before, sums_after), in
// instances of their own: with the choice made at run time the survey gulp takes
// 17.7 ms instead of 17.6.
template <int NWD, int NWT, int DPW, int W, int UC, bool PART>
__global__ void __launch_bounds__((NWD * NWT + 1) * 32, dd_min_blocks(NWD * NWT, DPW * W))
    k_dedisp(DedispArgs a) {
  extern __shared__ __align__(128) uint8_t smem[];
  constexpr int NW = NWD * NWT;
  constexpr int DB = DPW * NWD;
  constexpr int TBW = 32 * W * NWT;
  uint64_t* full = reinterpret_cast<uint64_t*>(smem);
  uint64_t* empty = full + DD_NST;
  int* nrows = reinterpret_cast<int*>(empty + DD_NST);  // channels of each stage buffer
  // [TBW] zero words (the window of a channel past the last one), then
  // [NST][DB][CH] byte offsets from smem of the (DM, channel) windows, then
  // [NST] stage buffers of a.cap bytes
  constexpr int CH = DD_ROWS;
  constexpr int ZERO = 128;
  constexpr int OFFS = ZERO + TBW * 4;
  constexpr int ROWS0 = OFFS + DD_NST * DB * CH * 4;
  const int dblk = blockIdx.x;
  const int t0 = blockIdx.y * TBW;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int d_lo = dblk * DB;

  for (int i = threadIdx.x; i < TBW; i += (NW + 1) * 32)
    reinterpret_cast<uint32_t*>(smem + ZERO)[i] = 0u;
  if (threadIdx.x == 0) {
    for (int b = 0; b < DD_NST; b++) {
      mbar_init(&full[b], 1);
      mbar_init(&empty[b], NW);
    }
    fence_mbar_init();
  }
  __syncthreads();

  if (warp == NW) {
    // ---------------- producer ----------------
    // blockIdx.z selects the unit (an independent filterbank of the batch)
    const uint32_t* __restrict__ in = a.in + (size_t)blockIdx.z * a.in_unit;
    const int2* __restrict__ brange = a.blk_range + (size_t)dblk * a.nchans;
    // lane k < CH of a stage: its k-th channel and that channel's delay range
    int c = 0;
    int2 r = make_int2(0, 0);
    auto channel = [&](int k0) {
      const bool have = lane < CH && k0 + lane < a.nact;
      c = have ? a.chans[k0 + lane] : 0;
      if constexpr (DB == 1) {
        const int dl = have ? a.delays[(size_t)d_lo * a.nchans + c] : 0;
        r = make_int2(dl, dl);
      } else {
        r = have ? brange[c] : make_int2(0, 0);
      }
    };
    channel(0);
    int st = 0;
    for (int k0 = 0; k0 < a.nact; st++) {
      const int buf = st % DD_NST;
      const bool have = lane < CH && k0 + lane < a.nact;
      const int lo = (t0 + r.x) & ~3;
      const int bytes = have ? (4 * (t0 + r.y - lo + TBW) + 15) & ~15 : 0;
      int end = bytes;  // inclusive scan: the rows lie back to back
#pragma unroll
      for (int o = 1; o < CH; o *= 2) {
        const int v = __shfl_up_sync(0xffffffffu, end, o);
        if (lane >= o) end += v;
      }
      // as many rows as fit the buffer, whole groups of UC where there are any
      int nk = __popc(__ballot_sync(0xffffffffu, have && end <= a.cap));
      if (nk > UC && k0 + nk < a.nact) nk -= nk % UC;
      const int total = __shfl_sync(0xffffffffu, end, nk - 1);
      const int at = ROWS0 + buf * a.cap + end - bytes;  // byte offset of the row
      // the stage's delays (channel lane % CH, DR DMs a round), all loads in
      // flight at once, and the next stage's channels, before the buffer is
      // waited for
      constexpr int DR = 32 / CH;  // DMs per round
      constexpr int NR = (DB + DR - 1) / DR;
      const int kl = lane % CH;
      const int ck = __shfl_sync(0xffffffffu, c, kl);
      const int row0 = __shfl_sync(0xffffffffu, at + 4 * (t0 - lo), kl);
      int dl[NR];
#pragma unroll
      for (int i = 0; i < NR; i++) {
        const int d = min(d_lo + DR * i + lane / CH, a.dm_count - 1);
        dl[i] = a.delays[(size_t)d * a.nchans + ck];
      }
      const int c_now = c;
      channel(k0 + nk);
      if (st >= DD_NST) {
        if (!mbar_wait(&empty[buf], (uint32_t)(((st / DD_NST) - 1) & 1), a.wait_limit)) {
          if (lane == 0) atomicOr(a.err, 1u);
          break;
        }
      }
      // error-path test: the last stage is never copied (nor announced), so
      // its `full` phase never completes and the consumers' wait gives up
      if (a.withhold_last && k0 + nk == a.nact) break;
      int* off = reinterpret_cast<int*>(smem + OFFS) + buf * DB * CH;
#pragma unroll
      for (int i = 0; i < NR; i++)
        if (DR * i + lane / CH < DB)
          off[32 * i + lane] = kl < nk ? row0 + 4 * dl[i] : ZERO;
      if (lane == 0) nrows[buf] = nk;
      __syncwarp();
      if (lane == 0) mbar_expect_tx(&full[buf], (uint32_t)total);
      __syncwarp();
      if (lane < nk)
        bulk_g2s(smem + at, in + (size_t)(PART ? c_now - a.chan0 : c_now) * a.in_pitch + lo,
                 (uint32_t)bytes, &full[buf]);
      k0 += nk;
    }
    const int issued = st;
    // let every copy this CTA issued land before the warp exits
    for (int j = (issued > DD_NST ? issued - DD_NST : 0); j < issued; j++)
      mbar_wait(&full[j % DD_NST], (uint32_t)((j / DD_NST) & 1), a.wait_limit);
    return;
  }

  // ---------------- consumers ----------------
  const int wd = warp % NWD, wt = warp / NWD;
  const int word0 = wt * 32 * W + lane;  // this lane's first word of the tile
  const uint8_t* lane_base = smem + 4 * word0;
  uint32_t raw[DPW][W], odd[DPW][W];
#pragma unroll
  for (int d = 0; d < DPW; d++)
#pragma unroll
    for (int w = 0; w < W; w++) raw[d][w] = odd[d][w] = 0;

  float* __restrict__ out = a.out + (size_t)blockIdx.z * a.out_unit;
  // the run's sums to the output rows; first / last: of this tile's runs
  auto flush = [&](bool first, bool last) {
#pragma unroll
    for (int d = 0; d < DPW; d++) {
      const int dd = d_lo + DPW * wd + d;
      if (dd < a.dm_count) {
        float* o = out + (size_t)dd * a.out_pitch;
#pragma unroll
        for (int w = 0; w < W; w++) {
          const int t = t0 + word0 + 32 * w;
          uint32_t v[4];
          if (dd_dot(w)) {
            v[0] = raw[d][w] % 65535u;
            v[1] = raw[d][w] / 65535u;
            v[2] = odd[d][w] % 65535u;
            v[3] = odd[d][w] / 65535u;
          } else {
            const uint32_t even = raw[d][w] - (odd[d][w] << 8);
            v[0] = even & 0xFFFFu;
            v[1] = odd[d][w] & 0xFFFFu;
            v[2] = even >> 16;
            v[3] = odd[d][w] >> 16;
          }
          if (t < a.split) {
#pragma unroll
            for (int q = 0; q < 4; q++) {
              const int at = t + q * a.split;
              if (at < a.nout) {
                if (last) {
                  uint32_t sum = v[q];
                  if (!first) sum += __ldcg(reinterpret_cast<const unsigned*>(o) + at);
                  o[at] = __uint2float_rn(sum);
                } else if (first) {
                  __stcg(reinterpret_cast<unsigned*>(o) + at, v[q]);
                } else {
                  atomicAdd(reinterpret_cast<unsigned*>(o) + at, v[q]);
                }
              }
            }
          }
        }
      }
#pragma unroll
      for (int w = 0; w < W; w++) raw[d][w] = odd[d][w] = 0;
    }
  };

  int nsum = 0;
  bool first = !(PART && a.sums_before);
  for (int st = 0, k0 = 0; k0 < a.nact; st++) {
    const int buf = st % DD_NST;
    if (!mbar_wait(&full[buf], (uint32_t)((st / DD_NST) & 1), a.wait_limit)) {
      if (lane == 0) atomicOr(a.err, 1u);
      return;
    }
    const int nk = nrows[buf];
    k0 += nk;
    if (nsum + nk > DD_RUN) {
      flush(first, false);
      first = false;
      nsum = 0;
    }
    const int* off = reinterpret_cast<const int*>(smem + OFFS) + (buf * DB + DPW * wd) * CH;
    for (int k = 0; k < nk; k += UC) {
#pragma unroll
      for (int d = 0; d < DPW; d++) {
        int o[UC];
        if constexpr (UC == 4) {
          const int4 v = *reinterpret_cast<const int4*>(off + d * CH + k);
          o[0] = v.x; o[1] = v.y; o[2] = v.z; o[3] = v.w;
        } else {
          const int2 v = *reinterpret_cast<const int2*>(off + d * CH + k);
          o[0] = v.x; o[1] = v.y;
        }
        const uint32_t* p[UC];
#pragma unroll
        for (int u = 0; u < UC; u++) p[u] = reinterpret_cast<const uint32_t*>(lane_base + o[u]);
#pragma unroll
        for (int w = 0; w < W; w++) {
          uint32_t x[UC];
#pragma unroll
          for (int u = 0; u < UC; u++) x[u] = p[u][32 * w];
#pragma unroll
          for (int u = 0; u < UC; u += 2) {
            if (dd_dot(w)) {
              raw[d][w] = __dp2a_lo(kDot, x[u + 1], __dp2a_lo(kDot, x[u], raw[d][w]));
              odd[d][w] = __dp2a_hi(kDot, x[u + 1], __dp2a_hi(kDot, x[u], odd[d][w]));
            } else {
              raw[d][w] += x[u] + x[u + 1];
              odd[d][w] += __byte_perm(x[u], 0u, 0x4341) + __byte_perm(x[u + 1], 0u, 0x4341);
            }
          }
        }
      }
    }
    nsum += nk;
    __syncwarp();
    if (lane == 0) mbar_arrive(&empty[buf]);
  }
  flush(first, !(PART && a.sums_after));
}

// Least and largest delay of each block of `db` trials, per channel, and over all
// of them the largest span and the sum of the spans (span[0], span[1], from 0).
// Thread: one channel of blocks blockIdx.y, + gridDim.y, ...
__global__ void __launch_bounds__(256) k_block_ranges(const int* __restrict__ delays, int ntrials,
                                                      int nchans, int db, int2* __restrict__ range,
                                                      unsigned long long* __restrict__ span) {
  const int c = blockIdx.x * 256 + threadIdx.x;
  unsigned most = 0;
  unsigned long long sum = 0;
  for (int b = blockIdx.y; (long long)b * db < ntrials && c < nchans; b += gridDim.y) {
    int lo = 0x7FFFFFFF, hi = 0;  // (delays are not negative)
    for (int d = b * db; d < min(ntrials, (b + 1) * db); d++) {
      const int v = delays[(size_t)d * nchans + c];
      lo = min(lo, v);
      hi = max(hi, v);
    }
    range[(size_t)b * nchans + c] = make_int2(lo, hi);
    most = max(most, (unsigned)(hi - lo));
    sum += (unsigned)(hi - lo);
  }
  most = __reduce_max_sync(0xffffffffu, most);
#pragma unroll
  for (int o = 16; o; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
  if ((threadIdx.x & 31) == 0) {
    atomicMax(span, (unsigned long long)most);
    atomicAdd(span + 1, sum);
  }
}

// Channel-major byte rows -> four-sample words: word t of channel c holds
// samples t, t + S, t + 2S, t + 3S of the row, for t < nwords (bytes past the
// row's pitch read as 0; they reach no output).  Thread: 16 words, four
// 16-byte loads and four 16-byte stores (S, the pitches and the bases are
// multiples of 16).
__global__ void __launch_bounds__(256) k_split_words(const uint8_t* __restrict__ in,
                                                     size_t in_pitch, size_t in_unit, int split,
                                                     int nwords, uint32_t* __restrict__ out,
                                                     size_t out_pitch, size_t out_unit) {
  const int t = 16 * (blockIdx.x * blockDim.x + threadIdx.x);
  if (t >= nwords) return;
  const uint8_t* row = in + (size_t)blockIdx.z * in_unit + (size_t)blockIdx.y * in_pitch;
  uint4 v[4];
#pragma unroll
  for (int q = 0; q < 4; q++) {
    const size_t at = (size_t)t + (size_t)q * split;
    v[q] = at + 16 <= in_pitch ? __ldg(reinterpret_cast<const uint4*>(row + at))
                               : make_uint4(0u, 0u, 0u, 0u);
  }
  uint4* o = reinterpret_cast<uint4*>(out + (size_t)blockIdx.z * out_unit +
                                      (size_t)blockIdx.y * out_pitch + t);
  const uint32_t* x = reinterpret_cast<const uint32_t*>(v);
#pragma unroll
  for (int j = 0; j < 4; j++) {
    const uint32_t a0 = x[j], a1 = x[4 + j], a2 = x[8 + j], a3 = x[12 + j];
    const uint32_t lo01 = __byte_perm(a0, a1, 0x5140), lo23 = __byte_perm(a2, a3, 0x5140);
    const uint32_t hi01 = __byte_perm(a0, a1, 0x7362), hi23 = __byte_perm(a2, a3, 0x7362);
    o[j] = make_uint4(__byte_perm(lo01, lo23, 0x5410), __byte_perm(lo01, lo23, 0x7632),
                      __byte_perm(hi01, hi23, 0x5410), __byte_perm(hi01, hi23, 0x7632));
  }
}

// ---------------------------------------------------------------------------
// Host launchers
// ---------------------------------------------------------------------------
cudaError_t launch_transpose_tf_ft(const uint8_t* in, size_t nsamps, int nchans, uint8_t* out,
                                   size_t pitch, cudaStream_t s, size_t units, size_t out_unit) {
  if (units < 1 || units > 65535) return cudaErrorInvalidValue;
  dim3 grid((unsigned)((nsamps + 127) / 128), (unsigned)((nchans + 127) / 128), (unsigned)units);
  k_transpose_tf_ft<<<grid, 256, 0, s>>>(in, nsamps, nchans, out, pitch, out_unit); note_launch();
  return cudaGetLastError();
}

cudaError_t launch_unpack_tf_ft(const uint8_t* in, size_t nsamps, int nchans, int nbits,
                                uint8_t* out, size_t pitch, cudaStream_t s, size_t units,
                                size_t out_unit, size_t hi_off) {
  if (units < 1 || units > 65535 || nchans < 1 || ((size_t)nchans * nbits) % 32 ||
      (reinterpret_cast<uintptr_t>(in) & 3) || pitch % 4)
    return cudaErrorInvalidValue;
  dim3 grid((unsigned)((nsamps + 127) / 128), (unsigned)((nchans + 127) / 128), (unsigned)units);
  const uint32_t* w = reinterpret_cast<const uint32_t*>(in);
  switch (nbits) {
    case 1: k_unpack_tf_ft<1><<<grid, 256, 0, s>>>(w, nsamps, nchans, out, pitch, out_unit, 0); break;
    case 2: k_unpack_tf_ft<2><<<grid, 256, 0, s>>>(w, nsamps, nchans, out, pitch, out_unit, 0); break;
    case 4: k_unpack_tf_ft<4><<<grid, 256, 0, s>>>(w, nsamps, nchans, out, pitch, out_unit, 0); break;
    case 16:
      k_unpack_tf_ft<16><<<grid, 256, 0, s>>>(w, nsamps, nchans, out, pitch, out_unit, hi_off);
      break;
    default: return cudaErrorInvalidValue;
  }
  note_launch();
  return cudaGetLastError();
}

cudaError_t launch_combine_planes(float* lo, const float* hi, size_t pitch, size_t n, size_t rows,
                                  cudaStream_t s) {
  if (rows == 0 || n == 0) return cudaSuccess;
  const size_t total = rows * n;
  const unsigned blocks = (unsigned)std::min<size_t>((total + 255) / 256, 148 * 16);
  k_combine_planes<<<blocks, 256, 0, s>>>(lo, hi, pitch, n, rows);
  note_launch();
  return cudaGetLastError();
}

// Scrunched input of adaptive dt: the byte mean of s consecutive samples (s a
// power of two; rounded half up) of each channel row, zero past nsamps / s.
// Bound by its reads.  A thread makes four outputs (one word) from 4 s bytes,
// read as whole words whose bytes are added four at a time (256 channels x
// 2^18 samples, s = 2..64: 24 us on average, 39 at s = 2 and 16 to 25 above; a
// byte and a thread at a time 78 us).
__global__ void __launch_bounds__(256) k_scrunch_ft(const uint8_t* __restrict__ in,
                                                    size_t in_pitch, unsigned ns, int log2s,
                                                    uint8_t* __restrict__ out, unsigned out_pitch,
                                                    size_t in_unit, size_t out_unit) {
  const unsigned u = 4 * (blockIdx.x * blockDim.x + threadIdx.x);
  if (u >= out_pitch) return;
  const unsigned s = 1u << log2s, half = s >> 1;
  const uint8_t* row = in + (size_t)blockIdx.z * in_unit + (size_t)blockIdx.y * in_pitch +
                       ((size_t)u << log2s);
  uint32_t v = 0;
  if (log2s == 1) {
    const uint32_t* w = reinterpret_cast<const uint32_t*>(row);  // two outputs a word
    const uint32_t a = u < ns ? w[0] : 0u, b = u + 2 < ns ? w[1] : 0u;
    const uint32_t M = 0x00FF00FFu, R = 0x00010001u;
    const uint32_t pa = (((a & M) + ((a >> 8) & M) + R) >> 1) & M;
    const uint32_t pb = (((b & M) + ((b >> 8) & M) + R) >> 1) & M;
    v = __byte_perm(pa, pb, 0x6420);
    if (u + 4 > ns) v &= u + 3 == ns ? 0x00FFFFFFu : u + 2 == ns ? 0x0000FFFFu
                         : u + 1 == ns ? 0x000000FFu : 0u;
  } else {
#pragma unroll
    for (unsigned j = 0; j < 4; j++) {
      if (u + j >= ns) break;
      const uint32_t* w = reinterpret_cast<const uint32_t*>(row + (j << log2s));
      unsigned sum = half;
      if (log2s == 2) {
        sum = __dp4a(w[0], 0x01010101u, sum);
      } else if (log2s == 3) {
        const uint2 x = *reinterpret_cast<const uint2*>(w);
        sum = __dp4a(x.x, 0x01010101u, __dp4a(x.y, 0x01010101u, sum));
      } else {
        for (unsigned k = 0; k < s / 16; k++) {
          const uint4 x = reinterpret_cast<const uint4*>(w)[k];
          sum = __dp4a(x.x, 0x01010101u, __dp4a(x.y, 0x01010101u, sum));
          sum = __dp4a(x.z, 0x01010101u, __dp4a(x.w, 0x01010101u, sum));
        }
      }
      v |= (sum >> log2s) << (8 * j);
    }
  }
  *reinterpret_cast<uint32_t*>(out + (size_t)blockIdx.z * out_unit +
                               (size_t)blockIdx.y * out_pitch + u) = v;
}

cudaError_t launch_scrunch_ft(const uint8_t* in, size_t in_pitch, size_t nsamps, int nchans,
                              int s, uint8_t* out, size_t out_pitch, size_t units,
                              size_t in_unit, size_t out_unit, cudaStream_t st) {
  // rows 16-byte aligned, so that every group of samples starts on its words
  if (s < 2 || (s & (s - 1)) || units < 1 || units > 65535 || nchans < 1 || nchans > 65535 ||
      in_pitch % 16 || in_unit % 16 || out_pitch % 4 || out_unit % 4 ||
      out_pitch > 0x7FFFFFFFull || (reinterpret_cast<uintptr_t>(in) & 15))
    return cudaErrorInvalidValue;
  int log2s = 0;
  while ((1 << log2s) < s) log2s++;
  const unsigned words = (unsigned)(out_pitch / 4);
  dim3 grid((words + 255) / 256, (unsigned)nchans, (unsigned)units);
  k_scrunch_ft<<<grid, 256, 0, st>>>(in, in_pitch, (unsigned)(nsamps / (size_t)s), log2s, out,
                                      (unsigned)out_pitch, in_unit, out_unit);
  note_launch();
  return cudaGetLastError();
}

cudaError_t launch_dm0_sum(const uint8_t* in, size_t nsamps, int nchans, float* out,
                           cudaStream_t s) {
  k_dm0_sum<<<(unsigned)((nsamps + 7) / 8), 256, 0, s>>>(in, nsamps, nchans, out); note_launch();
  return cudaGetLastError();
}

cudaError_t launch_zap(const uint8_t* in, size_t nsamps, int nchans, const int* mask,
                       unsigned max_resample_dist, uint8_t* out_ft, size_t pitch,
                       uint8_t* out_tf, cudaStream_t s) {
  dim3 grid((unsigned)((nsamps + 127) / 128), (unsigned)((nchans + 127) / 128));
  k_zap_to_ft<<<grid, 256, 0, s>>>(in, nsamps, nchans, mask, max_resample_dist, out_ft, pitch,
                                   out_tf); note_launch();
  return cudaGetLastError();
}

// Scratch layout of the narrow-band stage (bytes, 256-aligned pieces).
struct NbLayout {
  size_t idx, start, len, s1, s2, s3, s4, s5, bp, mad, tmp, rms, total;
};
static NbLayout nb_layout(size_t nstretch, int C) {
  NbLayout L{};
  size_t o = 0;
  auto take = [&](size_t bytes) {
    size_t at = o;
    o += (bytes + 255) / 256 * 256;
    return at;
  };
  const size_t n = nstretch;
  L.idx = take(n * NB_SPECTRA * sizeof(unsigned));
  L.start = take(n * sizeof(unsigned long long));
  L.len = take(n * sizeof(unsigned));
  L.s1 = take(n * NB_SPECTRA * C * sizeof(float));
  L.s2 = take(n * (NB_SPECTRA / 5) * C * sizeof(float));
  L.s3 = take(n * (NB_SPECTRA / 25) * C * sizeof(float));
  L.s4 = take(n * (NB_SPECTRA / 125) * C * sizeof(float));
  L.s5 = take(n * (NB_SPECTRA / 625) * C * sizeof(float));
  L.bp = take(n * C * sizeof(float));
  L.mad = take(n * C * sizeof(float));
  L.tmp = take(n * (C / 5 + 1) * sizeof(float));
  L.rms = take(n * sizeof(float));
  L.total = o;
  return L;
}

size_t narrow_band_stretches(size_t nsamps, float dt, float baseline_length) {
  const size_t nsmooth = (size_t)(baseline_length / (1 * dt));
  return nsmooth ? (nsamps + nsmooth - 1) / nsmooth : 0;
}

size_t narrow_band_scratch_bytes(size_t units, size_t nsamps, int nchans, float dt,
                                 float baseline_length) {
  return nb_layout(units * narrow_band_stretches(nsamps, dt, baseline_length), nchans).total;
}

cudaError_t narrow_band(uint8_t* tf, size_t units, size_t nsamps, int nchans, float dt,
                        float baseline_length, float rfi_tol, void* scratch, cudaStream_t s) {
  const size_t nsmooth = (size_t)(baseline_length / (1 * dt));
  const int C = nchans;
  if (nsmooth == 0 || C % 4 != 0 || C < 20 || units == 0) return cudaErrorInvalidValue;
  if (nsamps * (size_t)(C / 4) >= 0xFFFFFFFFull) return cudaErrorInvalidValue;
  const size_t nsub = (nsamps + nsmooth - 1) / nsmooth;
  const size_t ns = units * nsub;
  const NbLayout L = nb_layout(ns, C);
  uint8_t* base = static_cast<uint8_t*>(scratch);
  auto F = [&](size_t off) { return reinterpret_cast<float*>(base + off); };
  unsigned* idx = reinterpret_cast<unsigned*>(base + L.idx);
  unsigned long long* start = reinterpret_cast<unsigned long long*>(base + L.start);
  unsigned* len = reinterpret_cast<unsigned*>(base + L.len);
  std::vector<unsigned long long> h_start(ns);
  std::vector<unsigned> h_len(ns);
  for (size_t u = 0; u < units; u++)
    for (size_t g = 0; g < nsub; g++) {
      h_start[u * nsub + g] = u * nsamps + g * nsmooth;
      h_len[u * nsub + g] = (unsigned)std::min(nsmooth, nsamps - g * nsmooth);
    }
  cudaError_t e = cudaMemcpyAsync(start, h_start.data(), ns * sizeof(unsigned long long),
                                  cudaMemcpyHostToDevice, s);
  if (e == cudaSuccess)
    e = cudaMemcpyAsync(len, h_len.data(), ns * sizeof(unsigned), cudaMemcpyHostToDevice, s);
  // both copies read host vectors that go out of scope: finish them here
  if (e == cudaSuccess) e = cudaStreamSynchronize(s);
  if (e != cudaSuccess) return e;
  auto blocks = [](size_t n) { return (unsigned)std::min<size_t>((n + 255) / 256, 148 * 16); };
  k_nb_indices<<<(unsigned)((ns + 63) / 64), 64, 0, s>>>(len, (int)ns, idx); note_launch();
  const size_t tot1 = ns * NB_SPECTRA * (size_t)C;
  k_nb_gather<<<blocks(tot1), 256, 0, s>>>(tf, C, start, idx, tot1, F(L.s1)); note_launch();
  // bandpass: recursive median, smoothing
  const size_t lev[6] = {L.s1, L.s2, L.s3, L.s4, L.s5, L.bp};
  int count = NB_SPECTRA;
  for (int l = 0; l < 5; l++, count /= 5) {
    k_nb_scrunch5<<<blocks(ns * (count / 5) * (size_t)C), 256, 0, s>>>(F(lev[l]), C, count,
                                                                      (int)ns, F(lev[l + 1]));
    note_launch();
  }
  k_nb_smooth<<<(unsigned)ns, 256, 0, s>>>(F(L.bp), F(L.tmp), C, 1.f); note_launch();
  // band deviation: |spectra - bandpass|, recursive median, x 1.4826, smoothing
  k_nb_absdev<<<blocks(tot1), 256, 0, s>>>(F(L.s1), F(L.bp), C, tot1); note_launch();
  const size_t lev2[6] = {L.s1, L.s2, L.s3, L.s4, L.s5, L.mad};
  count = NB_SPECTRA;
  for (int l = 0; l < 5; l++, count /= 5) {
    k_nb_scrunch5<<<blocks(ns * (count / 5) * (size_t)C), 256, 0, s>>>(F(lev2[l]), C, count,
                                                                       (int)ns, F(lev2[l + 1]));
    note_launch();
  }
  k_nb_smooth<<<(unsigned)ns, 256, 0, s>>>(F(L.mad), F(L.tmp), C, 1.4826f); note_launch();
  k_nb_rms<<<(unsigned)ns, 256, 0, s>>>(F(L.mad), C, F(L.rms)); note_launch();
  const size_t nspec = units * nsamps;
  k_nb_zap<<<(unsigned)((nspec + 127) / 128), 128, 0, s>>>(
      reinterpret_cast<uint32_t*>(tf), nsamps, (int)units, C, nsmooth, (int)nsub, F(L.bp),
      F(L.rms), rfi_tol, (unsigned)(C / 60));
  note_launch();
  return cudaGetLastError();
}

// Shared memory of a tile with stage buffers of cap bytes.
size_t dedisp_smem_bytes(int dm_block, int time_block, int cap) {
  return 128 + (size_t)time_block + (size_t)DD_NST * dm_block * DD_ROWS * 4 +
         (size_t)DD_NST * cap;
}

// Bytes of a stage buffer: kDedispRows rows of the mean length, or what four
// CTAs on an SM leave for one (54 KB each, two buffers) if that is less, but
// the longest row at least, with fewer CTAs where that takes more (0: it fits
// nowhere).  Two long stages beat three short ones: each stage costs every
// warp a wait and a hand-over (survey gulp, 1024 channels x 2^18, 8 x 1280:
// 12.2 ms with two stages of 15 rows on average, 13.3 with three of 10, 14.5
// with four of 7).  The sums are exact integers, so the choice does not change
// the result.
int dedisp_stage_bytes(int dm_block, int time_block, int mean_row, int longest_row) {
  const size_t fixed = dedisp_smem_bytes(dm_block, time_block, 0);
  for (size_t room : {(size_t)54 * 1024, (size_t)72 * 1024, (size_t)110 * 1024,
                      (size_t)200 * 1024}) {
    const size_t cap = (room - fixed) / DD_NST & ~(size_t)15;
    if (cap >= (size_t)longest_row)
      return (int)std::min(cap, std::max<size_t>((size_t)kDedispRows * mean_row + 1024, longest_row) &
                                    ~(size_t)15);
  }
  return 0;
}

namespace {
template <int NWD, int NWT, int DPW, int W, int UC>
cudaError_t launch_dd(const DedispArgs& a, int units, size_t smem, cudaStream_t s) {
  const bool part = a.chan0 != 0 || a.sums_before || a.sums_after;
  auto kern = part ? k_dedisp<NWD, NWT, DPW, W, UC, true> : k_dedisp<NWD, NWT, DPW, W, UC, false>;
  cudaError_t e = raise_smem_limit(kern, smem);
  if (e != cudaSuccess) return e;
  const int DB = DPW * NWD, TBW = 32 * W * NWT;
  dim3 grid((unsigned)((a.dm_count + DB - 1) / DB), (unsigned)((a.split + TBW - 1) / TBW),
            (unsigned)units);
  kern<<<grid, (NWD * NWT + 1) * 32, smem, s>>>(a); note_launch();
  return cudaGetLastError();
}
}  // namespace

cudaError_t launch_dedisp(const DedispArgs& a0, int units, const DedispTile& t, cudaStream_t s) {
  if (units < 1 || units > 65535) return cudaErrorInvalidValue;
  DedispArgs a = a0;
  a.cap = t.stage;
  const size_t smem = dedisp_smem_bytes(t.dm_block, t.time_block, t.stage);
  // {dm_block, time_block} -> consumer warps over the DMs (NWD, DPW trials
  // each) and over the words (NWT), W words per lane: time_block = 128 W NWT
#define HDB_DD_TILE(DBk, NWDk, NWTk, DPWk, Wk)                                       \
  if (t.dm_block == DBk && t.time_block == 128 * Wk * NWTk)                          \
    return launch_dd<NWDk, NWTk, DPWk, Wk, 4>(a, units, smem, s);
  HDB_DD_TILE(8, 4, 1, 2, 8)
  HDB_DD_TILE(8, 4, 1, 2, 5)
  HDB_DD_TILE(8, 4, 1, 2, 6)
  HDB_DD_TILE(8, 4, 1, 2, 9)
  HDB_DD_TILE(8, 4, 1, 2, 10)
  HDB_DD_TILE(16, 8, 1, 2, 4)
  HDB_DD_TILE(16, 8, 1, 2, 3)
  HDB_DD_TILE(16, 8, 1, 2, 5)
  HDB_DD_TILE(16, 8, 1, 2, 6)
  HDB_DD_TILE(32, 16, 1, 2, 2)
  HDB_DD_TILE(32, 16, 1, 2, 3)
  HDB_DD_TILE(2, 1, 4, 2, 10)
  HDB_DD_TILE(1, 1, 4, 1, 16)
#undef HDB_DD_TILE
  return cudaErrorInvalidValue;
}

cudaError_t launch_block_ranges(const int* delays, size_t ntrials, size_t nchans, int db,
                                int2* range, unsigned long long* span, cudaStream_t s) {
  if (ntrials < 1 || ntrials > 0x3FFFFFFFull || nchans < 1 || nchans > 0x3FFFFFFFull)
    return cudaErrorInvalidValue;
  const size_t nblk = (ntrials + db - 1) / db;
  dim3 grid((unsigned)((nchans + 255) / 256), (unsigned)std::min<size_t>(nblk, 65535));
  k_block_ranges<<<grid, 256, 0, s>>>(delays, (int)ntrials, (int)nchans, db, range, span);
  note_launch();
  return cudaGetLastError();
}

cudaError_t launch_split_words(const uint8_t* in, size_t in_pitch, size_t in_unit, int nchans,
                               size_t units, int split, size_t nwords, uint32_t* out,
                               size_t out_pitch, size_t out_unit, cudaStream_t s) {
  if (units < 1 || units > 65535 || nchans < 1 || in_pitch % 16 ||
      in_unit % 16 || split % 16 || out_pitch % 16 || out_unit % 4 || nwords > out_pitch ||
      nwords > 0x7FFFFFF0ull)
    return cudaErrorInvalidValue;
  const unsigned nthr = (unsigned)((nwords + 15) / 16);
  // a channel per grid row, 65535 at most (a loop over channels in the kernel costs
  // registers: 133 us instead of 129 for 36 x 320 channels)
  for (int c = 0; c < nchans; c += 65535) {
    dim3 grid((nthr + 255) / 256, (unsigned)std::min(nchans - c, 65535), (unsigned)units);
    k_split_words<<<grid, 256, 0, s>>>(in + (size_t)c * in_pitch, in_pitch, in_unit, split,
                                       (int)nwords, out + (size_t)c * out_pitch, out_pitch,
                                       out_unit);
    note_launch();
    const cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return e;
  }
  return cudaSuccess;
}

}  // namespace hdb
