// profile.cu -- the candidate profiler (Applications/candidate_profiler.C) on
// the GPU for a batch of candidates of one filterbank.
//
// Per candidate, as the reference's application computes them:
//   * the DM-time plot (gen_dm_time_plot, candidate_profiler.C:232-415): the
//     trials [dm_begin, dm_end) around the candidate's trial re-dedispersed
//     over a window of the filterbank with adaptive dt on those trials (pulse
//     width 40 us, tolerance 1.15), then either summed over the boxcar at each
//     trial's resolution or (do_filter) unscrunched and boxcar-filtered
//     through a float prefix sum; each row normalised
//     (normalise_series_array, :88-134, with its division by zero kept);
//   * the DM-0 series: the same with the list's first trial alone;
//   * the freq-time plot (gen_freq_time_plot, :136-230) at filter - 2;
//   * from these, on the host: the plot's first maximum, SNR vs DM at its time
//     and SNR vs time along its row (:560-640).
// Windows are read from the filterbank as the application reads its file:
// samples past the end read as 0; a freq-time window that would start before
// the first sample reads 0 there.
//
// Kernels: k_prof_window copies each candidate's window channel-major;
// k_prof_dedisp computes from it each window trial's dedispersed samples
// (exact integer sums over channels of the byte-mean scrunched input, as
// include/dedisp.h defines them) into a scratch row; k_prof_boxcar and
// k_prof_filter form the plot rows in the reference's float order;
// k_prof_ft sums the freq-time pixels; normalise_row_list normalises every row.
#include <algorithm>
#include <cmath>
#include <cstring>
#include <mutex>
#include <vector>

#include "heimdall_b200.h"
#include "internal.h"
#include "plan.h"

namespace hdb {
namespace {

// One dedispersed row of a candidate's window (a trial of its DM-time plot
// or its DM-0 series).
struct ProfRow {
  float dm;            // trial DM
  int s;               // scrunch factor
  unsigned nd;         // samples of the row before scrunching (valid: nd / s)
  int cand;            // its candidate (whose window it starts with)
  size_t off;          // float offset of the row in the scratch (nd + 1 floats)
  size_t out;          // float offset of the plot row in the output
  int width;           // boxcar width of the plot (1 << filter)
};

// A candidate's part of the filterbank, channel-major: sample first + t of
// channel c at off + c * pitch + t, for t < n (to the filterbank's end at most;
// past it every sample is 0).
struct ProfWindow {
  long long first;     // first filterbank sample
  unsigned n, pitch;   // samples; bytes between channels (a multiple of 4)
  size_t off;          // byte offset of the window in the windows' buffer
};

// Channel-major copies of the windows.  Tiles of 128 samples x 32 channels
// through shared memory: byte loads along the channels, word stores along
// time.  The windows are read once here instead of once per trial, and the
// trials then read consecutive samples in consecutive lanes (a time-major row
// puts them nchans bytes apart, 32 lines per load).
__global__ void __launch_bounds__(256) k_prof_window(const uint8_t* __restrict__ tf,
                                                     size_t nsamps, int nchans,
                                                     const ProfWindow* __restrict__ windows,
                                                     uint8_t* __restrict__ out) {
  __shared__ uint8_t tile[32][132];
  const ProfWindow wn = windows[blockIdx.z];
  const unsigned t0 = blockIdx.x * 128;
  if (t0 >= wn.n) return;
  const int c0 = blockIdx.y * 32, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  for (int r = warp; r < 128; r += 8) {
    const long long t = wn.first + t0 + r;
    uint8_t v = 0;
    if (t < (long long)nsamps && c0 + lane < nchans) v = tf[(size_t)t * nchans + c0 + lane];
    tile[lane][r] = v;
  }
  __syncthreads();
  if (t0 + 4 * lane >= wn.pitch) return;
  for (int c = warp; c < 32 && c0 + c < nchans; c += 8)
    *reinterpret_cast<uint32_t*>(out + wn.off + (size_t)(c0 + c) * wn.pitch + t0 + 4 * lane) =
        *reinterpret_cast<const uint32_t*>(&tile[c][4 * lane]);
}

// dedispersed[u] = sum_c in_s[c][u + delay(dm, c) / s] for u < nd / s, with
// in_s the byte mean of s samples (rounded half up; s a power of two) from the
// window's start.  A thread reads whole words: four outputs of s = 1 or two of
// s = 2 from one word (realigned from two), one output of s >= 4 from the s / 4
// words of its samples (aligned, as s divides its offset and its delay).  The
// channels' delays are found once per block.  Bound by the loads (L2-resident
// windows) and their index arithmetic.  12 candidates of up to 8192 samples x
// 33 trials x 256 channels: 1290 us from the time-major filterbank a byte at a
// time, 324 us a byte at a time from the windows, 153 us so.
constexpr int kProfChans = 256;   // at most 257: 16-bit lanes hold a pass's sums
__global__ void __launch_bounds__(128) k_prof_dedisp(const uint8_t* __restrict__ in,
                                                     const ProfWindow* __restrict__ windows,
                                                     int window0, int nchans,
                                                     const float* __restrict__ table,
                                                     const ProfRow* __restrict__ rows,
                                                     float* __restrict__ scratch) {
  __shared__ unsigned shift[kProfChans];  // s * (delay / s)
  const ProfRow r = rows[blockIdx.y];
  const unsigned s = (unsigned)r.s, n = r.nd / s;
  const unsigned per = s < 4 ? 4 / s : 1;  // outputs per thread
  // the samples of a last, incomplete scrunched one count as 0
  if (blockIdx.x == 0 && threadIdx.x == 0) scratch[r.off + n] = 0.f;
  if ((size_t)blockIdx.x * 128 * per >= n) return;
  const unsigned u = (blockIdx.x * 128 + threadIdx.x) * per;
  const ProfWindow wn = windows[r.cand - window0];
  const uint32_t* src = reinterpret_cast<const uint32_t*>(in + wn.off);
  const unsigned words = (wn.n + 3) / 4, pitch = wn.pitch / 4;  // past `words` samples are 0
  const unsigned x0 = s * min(u, n - 1);
  const uint32_t M = 0x00FF00FFu;
  unsigned acc[4] = {0u, 0u, 0u, 0u};
  for (int c0 = 0; c0 < nchans; c0 += kProfChans) {
    const int m = min(kProfChans, nchans - c0);
    __syncthreads();
    for (int c = threadIdx.x; c < m; c += 128) {
      const float v = __fadd_rn(__fmul_rn(r.dm, table[c0 + c]), 0.5f);
      const unsigned dl = v > 0.f ? (unsigned)v : 0u;
      shift[c] = s * (dl / s);
    }
    __syncthreads();
    if (s < 4) {
      uint32_t even = 0, odd = 0;  // outputs 0, 2 and 1, 3 (s = 2: outputs 0, 1 in `even`)
#pragma unroll 8
      for (int c = 0; c < m; c++) {
        const unsigned x = x0 + shift[c], w = x >> 2;
        const uint32_t* p = src + (size_t)c * pitch;
        const uint32_t v = __funnelshift_r(w < words ? p[w] : 0u, w + 1 < words ? p[w + 1] : 0u,
                                           8 * (x & 3));
        const uint32_t lo = v & M, hi = (v >> 8) & M;
        if (s == 1) {
          even += lo;
          odd += hi;
        } else {
          even += ((lo + hi + 0x00010001u) >> 1) & M;
        }
      }
      acc[0] += even & 0xFFFFu;
      acc[s == 1 ? 2 : 1] += even >> 16;
      if (s == 1) {
        acc[1] += odd & 0xFFFFu;
        acc[3] += odd >> 16;
      }
    } else {
      const unsigned log2s = (unsigned)__ffs((int)s) - 1;
#pragma unroll 4
      for (int c = 0; c < m; c++) {
        const unsigned w = (x0 + shift[c]) >> 2, end = min(w + s / 4, words);
        const uint32_t* p = src + (size_t)c * pitch;
        unsigned sum = s / 2;
        if (w < words) sum = __dp4a(p[w], 0x01010101u, sum);
        for (unsigned k = w + 1; k < end; k++) sum = __dp4a(p[k], 0x01010101u, sum);
        acc[0] += sum >> log2s;
      }
    }
    src += (size_t)kProfChans * pitch;
  }
#pragma unroll
  for (unsigned k = 0; k < 4; k++)
    if (k < per && u + k < n) scratch[r.off + u + k] = (float)(int)acc[k];
}

// do_filter = 0: out[t] = sum over the boxcar at the trial's resolution,
// sum_{j < width / s} d[t * (width / s) + j] in float, left to right
__global__ void k_prof_boxcar(const ProfRow* __restrict__ rows, const float* __restrict__ scratch,
                              int out_nsamps, float* __restrict__ out) {
  const ProfRow r = rows[blockIdx.y];
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= out_nsamps) return;
  const unsigned k = (unsigned)r.width / (unsigned)r.s;
  const float* d = scratch + r.off + (size_t)t * k;
  float v = 0.f;
  for (unsigned j = 0; j < k; j++) v = __fadd_rn(v, d[j]);
  out[r.out + t] = v;
}

// do_filter = 1: the row unscrunched (sample t takes d[t / s]), its exclusive
// float prefix sum, and out[t] = S[t + width/2 + (width-1)/2 + 1] - S[t]; one
// thread per row walks the sum in order
__global__ void k_prof_filter(const ProfRow* __restrict__ rows, int nrows,
                              float* __restrict__ scratch, float* __restrict__ prefix,
                              int out_nsamps, float* __restrict__ out) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= nrows) return;
  const ProfRow r = rows[i];
  const float* d = scratch + r.off;
  float* S = prefix + r.off;
  float acc = 0.f;
  S[0] = 0.f;
  for (unsigned t = 0; t < r.nd; t++) {
    acc = __fadd_rn(acc, d[t / (unsigned)r.s]);
    S[t + 1] = acc;
  }
  const unsigned a = (unsigned)(r.width / 2 + (r.width - 1) / 2 + 1);
  for (int t = 0; t < out_nsamps; t++) out[r.out + t] = __fsub_rn(S[a + t], S[t]);
}

struct FtJob {
  long long first;   // first sample of the window (may be < 0)
  unsigned ts;       // samples per bin
  size_t out;        // float offset of the candidate's plot
};

// pixel (channel group cs, bin ti): the float sum, time outer and channel
// inner, of x / 255 * 255 over ts samples x fs channels, divided by ts * fs.
// Samples outside the filterbank are 0 and add +0 (a no-op on a sum >= +0).
//
// x / 255 * 255 rounds to x for every byte, so while the sum stays within 2^24
// every partial sum is exact in any order: k_prof_ft_exact adds whole words of
// four channels in integers (kFtExact: ts * fs up to 65793, i.e. every window
// but the longest).  A warp takes one bin and up to 128 channels, a lane four
// of them, eight rows in flight.  12 candidates of 64 x 16 pixels of up to
// 128 x 16 samples: 298 us with a lane per pixel reading its own bytes, 46
// us so.
constexpr unsigned kFtExact = (1u << 24) / 255u;
constexpr int FX_BINS = 4;  // warps per block
__global__ void __launch_bounds__(32 * FX_BINS) k_prof_ft_exact(const uint8_t* __restrict__ tf,
                                                                size_t nsamps, int nchans, int fs,
                                                                int ncs, int out_nsamps,
                                                                const FtJob* __restrict__ jobs,
                                                                float* __restrict__ out) {
  __shared__ unsigned sums[FX_BINS][32];
  const FtJob jb = jobs[blockIdx.z];
  if ((size_t)jb.ts * fs > kFtExact) return;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int cs0 = blockIdx.y * ncs, here = min(ncs, nchans / fs - cs0);
  const int ti = blockIdx.x * FX_BINS + warp;
  if (ti >= out_nsamps) return;
  sums[warp][lane] = 0u;
  __syncwarp();
  const long long t0 = jb.first + (long long)ti * jb.ts;
  const long long lo = t0 > 0 ? t0 : 0;
  const long long hi = min(t0 + (long long)jb.ts, (long long)nsamps);
  for (int x = 4 * lane; x < here * fs; x += 128) {
    const uint8_t* src = tf + (size_t)cs0 * fs + x;
    unsigned acc = 0;
#pragma unroll 8
    for (long long t = lo; t < hi; t++)
      acc = __dp4a(*reinterpret_cast<const uint32_t*>(src + (size_t)t * nchans), 0x01010101u, acc);
    atomicAdd(&sums[warp][x / fs], acc);
  }
  __syncwarp();
  if (lane < here)
    out[jb.out + (size_t)(cs0 + lane) * out_nsamps + ti] = __fdiv_rn(
        __uint2float_rn(sums[warp][lane]), (float)((size_t)jb.ts * (size_t)fs));
}

// The same for longer windows (and channel groups that are no whole words):
// the adds of a pixel are a chain in that order, so only the loads can be
// hidden.  A warp takes one bin and up to 32 channel groups (a lane each) and
// stages `nrow` samples of their channels at a time, whole runs of bytes.
constexpr int FT_BINS = 8;        // warps per block
constexpr int FT_STAGE = 4096;    // staged bytes per warp
__global__ void __launch_bounds__(32 * FT_BINS) k_prof_ft(const uint8_t* __restrict__ tf,
                                                          size_t nsamps, int nchans, int fs,
                                                          int ncs, int nf, int nrow,
                                                          int exact_done, int out_nsamps,
                                                          const FtJob* __restrict__ jobs,
                                                          float* __restrict__ out) {
  __shared__ float lut[256];
  __shared__ __align__(16) uint8_t stage[FT_BINS][FT_STAGE];
  const FtJob jb = jobs[blockIdx.z];
  if (exact_done && (size_t)jb.ts * fs <= kFtExact) return;
  for (int i = threadIdx.x; i < 256; i += blockDim.x) lut[i] = prof_scale((unsigned)i);
  __syncthreads();
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int cs0 = blockIdx.y * ncs, here = min(ncs, nchans / fs - cs0);
  const int ti = blockIdx.x * FT_BINS + warp;
  if (ti >= out_nsamps) return;
  uint8_t* st = stage[warp];
  // whole words where every run of channels starts on one
  const bool words = ((nchans | fs | nf) & 3) == 0 && (reinterpret_cast<uintptr_t>(tf) & 3) == 0;
  const long long t0 = jb.first + (long long)ti * jb.ts;
  float sum = 0.f;
  for (unsigned s0 = 0; s0 < jb.ts; s0 += nrow) {
    const int rows = (int)min((unsigned)nrow, jb.ts - s0);
    for (int f0 = 0; f0 < fs; f0 += nf) {  // nf < fs only with one group and one sample
      const int m = min(nf, fs - f0), len = here * m;
      __syncwarp();
      const uint8_t* src = tf + (size_t)cs0 * fs + f0;  // + t * nchans
      if (words) {
        // eight words in flight per lane
        const int wl = len / 4, all = rows * wl;
        for (int e0 = lane; e0 < all; e0 += 256) {
          uint32_t v[8];
#pragma unroll
          for (int j = 0; j < 8; j++) {
            const int e = e0 + 32 * j, r = e / wl;
            const long long t = t0 + s0 + r;
            v[j] = 0u;
            if (e < all && t >= 0 && t < (long long)nsamps)
              v[j] = reinterpret_cast<const uint32_t*>(src + (size_t)t * nchans)[e - r * wl];
          }
#pragma unroll
          for (int j = 0; j < 8; j++)
            if (e0 + 32 * j < all) reinterpret_cast<uint32_t*>(st)[e0 + 32 * j] = v[j];
        }
      } else {
        for (int r = 0; r < rows; r++) {
          const long long t = t0 + s0 + r;
          const bool in = t >= 0 && t < (long long)nsamps;
          for (int x = lane; x < len; x += 32)
            st[r * len + x] = in ? src[(size_t)t * nchans + x] : (uint8_t)0;
        }
      }
      __syncwarp();
      if (lane < here)
        for (int r = 0; r < rows; r++) {
          const uint8_t* p = st + r * len + lane * m;
#pragma unroll 8
          for (int f = 0; f < m; f++) sum = __fadd_rn(sum, lut[p[f]]);
        }
    }
  }
  if (lane < here)
    out[jb.out + (size_t)(cs0 + lane) * out_nsamps + ti] =
        __fdiv_rn(sum, (float)((size_t)jb.ts * (size_t)fs));
}

// A call's stream and device buffer.  Creating and freeing them took 0.85 ms
// of a 1.2 ms call, so a finished call leaves them for the next one: each call
// takes one for itself (threads never share one), at most two per device stay,
// of 256 MiB at most, and trim_pools() gives them back (dev_malloc calls it
// when the device is out of memory, a program hd_release_workspaces()).
struct Workspace {
  int dev = 0;
  cudaStream_t stream = nullptr;
  void* p = nullptr;
  size_t cap = 0;
  void release() {
    int now = 0;
    cudaGetDevice(&now);
    if (now != dev) cudaSetDevice(dev);
    if (p) cudaFree(p);
    if (stream) cudaStreamDestroy(stream);
    if (now != dev) cudaSetDevice(now);
    p = nullptr;
    stream = nullptr;
    cap = 0;
  }
};
struct WorkspacePool {
  std::mutex m;
  std::vector<Workspace> idle;
};
WorkspacePool& pool() {
  static WorkspacePool* p = new WorkspacePool;  // outlives the CUDA context's teardown
  return *p;
}
constexpr size_t kKeepBytes = (size_t)256 << 20, kKeepPerDevice = 2;

// One call's workspace; on every way out the call's work on the stream has
// ended before the next call may take it.
struct Held {
  Workspace w;
  cudaError_t take() {
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    {
      WorkspacePool& q = pool();
      std::lock_guard<std::mutex> g(q.m);
      for (size_t i = 0; i < q.idle.size(); i++)
        if (q.idle[i].dev == dev) {
          w = q.idle[i];
          q.idle.erase(q.idle.begin() + i);
          return cudaSuccess;
        }
    }
    w.dev = dev;
    return cudaStreamCreateWithFlags(&w.stream, cudaStreamNonBlocking);
  }
  cudaError_t ensure(size_t bytes) {
    if (bytes <= w.cap) return cudaSuccess;
    if (w.p) cudaFree(w.p);
    w.p = nullptr;
    w.cap = 0;
    const cudaError_t e = dev_malloc(&w.p, bytes);
    if (e == cudaSuccess) w.cap = bytes;
    return e;
  }
  ~Held() {
    if (!w.stream) return;
    const bool sound = cudaStreamSynchronize(w.stream) == cudaSuccess;
    if (sound && w.cap <= kKeepBytes) {
      WorkspacePool& q = pool();
      std::lock_guard<std::mutex> g(q.m);
      size_t n = 0;
      for (const Workspace& k : q.idle) n += k.dev == w.dev;
      if (n < kKeepPerDevice) {
        q.idle.push_back(w);
        return;
      }
    }
    w.release();
  }
};

}  // namespace

void trim_pools() {
  std::vector<Workspace> idle;
  {
    std::lock_guard<std::mutex> g(pool().m);
    idle.swap(pool().idle);
  }
  for (Workspace& w : idle) w.release();
}

}  // namespace hdb

extern "C" void hd_release_workspaces(void) { hdb::trim_pools(); }

extern "C" hd_error hd_profile_candidates(
    const hd_byte* filterbank, hd_size nsamps, hd_size nchans, int on_device, double tsamp,
    double fch1, double foff, const hd_float* dm_list, hd_size dm_count,
    const hd_profile_request* cands, hd_size ncands, hd_size out_nsamps, hd_size out_dm_count,
    hd_size fscrunch, int do_filter, hd_profile* out) {
  using namespace hdb;
  if (!filterbank || !dm_list || !cands || !out) return HD_INVALID_POINTER;
  if (ncands == 0) return HD_NO_ERROR;
  if (nchans == 0 || fscrunch == 0 || nchans % fscrunch != 0 || out_nsamps < 2 ||
      out_nsamps > 4096 || out_dm_count == 0 || dm_count == 0 || nsamps == 0)
    return HD_INVALID_STRIDE;
  for (size_t i = 0; i < ncands; i++)
    if (cands[i].dm_idx >= dm_count || cands[i].filter > 24) return HD_INVALID_STRIDE;
  const size_t C = nchans, out_nchans = nchans / fscrunch;
  // the dedisp plans take the header's values as float
  const float dt = (float)tsamp, f0 = (float)fch1, df = (float)foff;
  std::vector<float> table(C);
  delay_table(C, dt, f0, df, table.data());
  auto max_delay_of = [&](const float* dms, size_t n) {
    size_t m = 0;
    for (size_t d = 0; d < n; d++)
      for (size_t c = 0; c < C; c++) m = std::max(m, delay_of(dms[d], table[c]));
    return m;
  };
  const std::vector<float> dml(dm_list, dm_list + dm_count);

  // ---- host plan of every window ------------------------------------------
  std::vector<ProfRow> rows;
  std::vector<ProfWindow> windows(ncands);
  std::vector<FtJob> ftj(ncands);
  std::vector<size_t> n_dm(ncands), dm_begin(ncands), first_row(ncands + 1);
  const size_t plot = out_dm_count * out_nsamps;  // floats of one DM-time plot
  // the plots lie one after another: DM-time, DM-0, freq-time
  const size_t dm0_at = ncands * plot, ft_at = dm0_at + ncands * out_nsamps;
  const size_t plot_floats = ft_at + ncands * out_nchans * out_nsamps;
  size_t scratch = 0;
  for (size_t i = 0; i < ncands; i++) {
    const size_t samp = cands[i].samp, filter = cands[i].filter, dm_idx = cands[i].dm_idx;
    const size_t width = (size_t)1 << filter;
    size_t nd, first;
    if (!do_filter) {
      nd = out_nsamps * width;
      first = samp >= out_nsamps / 2 * width ? samp - out_nsamps / 2 * width : 0;
    } else {
      nd = out_nsamps + width - 1;
      first = samp > out_nsamps / 2 + width / 2 ? samp - out_nsamps / 2 - width / 2 : 0;
    }
    if (nd >= 0x7FFFFFFFu) return HD_INVALID_STRIDE;
    first_row[i] = rows.size();
    float dm_lo = dml[0], dm_hi = dml[0];
    // DM-time plot (candidate_profiler.C:265-344) and the DM-0 series
    for (int pass = 0; pass < 2; pass++) {
      const size_t di = pass == 0 ? dm_idx : 0;
      const size_t odc = pass == 0 ? out_dm_count : 1;
      const size_t b = di >= odc / 2 ? di - odc / 2 : 0;
      const size_t e = di < dm_count - ((odc - 1) / 2 + 1) ? di + (odc - 1) / 2 + 1 : dm_count;
      const size_t nd_trials = e - b;
      const std::vector<float> sub(dml.begin() + b, dml.begin() + e);
      const std::vector<dedisp_size> scr = scrunch_factors(sub, dt, 40.0, f0, df, C, 1.15);
      for (size_t d = 0; d < nd_trials; d++) {
        ProfRow r{};
        r.dm = sub[d];
        r.s = (int)scr[d];
        r.nd = (unsigned)nd;
        r.cand = (int)i;
        r.off = scratch;
        scratch += nd + 1;
        r.out = pass == 0 ? i * plot + d * out_nsamps : dm0_at + i * out_nsamps;
        r.width = (int)width;
        rows.push_back(r);
        dm_lo = std::min(dm_lo, r.dm);
        dm_hi = std::max(dm_hi, r.dm);
      }
      if (pass == 0) {
        n_dm[i] = nd_trials;
        dm_begin[i] = b;
      }
    }
    // the samples its trials reach (a channel's delay is monotone in the DM),
    // to the filterbank's end
    const size_t reach = nd + std::max(max_delay_of(&dm_lo, 1), max_delay_of(&dm_hi, 1));
    ProfWindow& wn = windows[i];
    wn.first = (long long)first;
    wn.n = (unsigned)std::min<size_t>(std::min(reach, first < nsamps ? nsamps - first : 0),
                                      0xFFFFFF00u);
    wn.pitch = std::max(4u, (wn.n + 3) & ~3u);
    // freq-time plot (candidate_profiler.C:136-184) at filter - 2
    const size_t ftf = filter > 2 ? filter - 2 : 0;
    const float dmv = dml[dm_idx];
    const size_t md = max_delay_of(&dmv, 1);
    size_t delay = 2, ts = (size_t)1 << ftf, in_n = out_nsamps * ts;
    if (in_n < md) {
      while (delay < md) delay *= 2;
      in_n = delay;
      ts = in_n / out_nsamps;
    }
    if (ts >= 0x7FFFFFFFu) return HD_INVALID_STRIDE;
    ftj[i].first = (long long)(samp + md / 2) - (long long)(in_n / 2);
    ftj[i].ts = (unsigned)ts;
    ftj[i].out = ft_at + i * out_nchans * out_nsamps;
  }
  first_row[ncands] = rows.size();
  if (rows.size() > 65535) return HD_INVALID_STRIDE;  // grid y

  // candidates whose windows are on the device at a time: up to 256 MiB of
  // them, one at least (a window is no larger than the filterbank)
  constexpr size_t kWindowBytes = (size_t)256 << 20;
  std::vector<size_t> batch{0};
  size_t window_bytes = 0;
  for (size_t i = 0, at = 0; i < ncands; i++) {
    const size_t bytes = ((size_t)windows[i].pitch * C + 255) & ~(size_t)255;
    if (i > batch.back() && at + bytes > kWindowBytes) {
      batch.push_back(i);
      at = 0;
    }
    windows[i].off = at;
    at += bytes;
    window_bytes = std::max(window_bytes, at);
  }
  batch.push_back(ncands);

  // ---- device work ------------------------------------------------------------
  Held ws;
  if (ws.take() != cudaSuccess) return HD_PRIOR_GPU_ERROR;
  cudaStream_t s = ws.w.stream;
  // one buffer: what the host planned (copied at once), then the buffers
  size_t total = 0;
  auto take = [&](size_t bytes) {
    const size_t at = total;
    total += (bytes + 255) & ~(size_t)255;
    return at;
  };
  const size_t o_table = take(C * sizeof(float)), o_rows = take(rows.size() * sizeof(ProfRow)),
               o_win = take(ncands * sizeof(ProfWindow)), o_ftj = take(ncands * sizeof(FtJob)),
               o_at = take(rows.size() * sizeof(size_t));
  std::vector<uint8_t> plan(total);
  std::memcpy(plan.data() + o_table, table.data(), C * sizeof(float));
  std::memcpy(plan.data() + o_rows, rows.data(), rows.size() * sizeof(ProfRow));
  std::memcpy(plan.data() + o_win, windows.data(), ncands * sizeof(ProfWindow));
  std::memcpy(plan.data() + o_ftj, ftj.data(), ncands * sizeof(FtJob));
  for (size_t k = 0; k < rows.size(); k++)
    reinterpret_cast<size_t*>(plan.data() + o_at)[k] = rows[k].out;
  const size_t o_plots = take(plot_floats * sizeof(float)),
               o_scr = take(scratch * sizeof(float)),
               o_pre = take(do_filter ? scratch * sizeof(float) : 0),
               o_windows = take(window_bytes), o_fb = take(on_device ? 0 : nsamps * C);
  if (ws.ensure(total) != cudaSuccess) return HD_MEM_ALLOC_FAILED;
  uint8_t* base = static_cast<uint8_t*>(ws.w.p);
  const uint8_t* tf = filterbank;
  if (!on_device) {
    if (cudaMemcpyAsync(base + o_fb, filterbank, nsamps * C, cudaMemcpyHostToDevice, s) !=
        cudaSuccess)
      return HD_MEM_COPY_FAILED;
    tf = base + o_fb;
  }
  const float* d_table = reinterpret_cast<const float*>(base + o_table);
  const ProfRow* d_rows = reinterpret_cast<const ProfRow*>(base + o_rows);
  const ProfWindow* d_win = reinterpret_cast<const ProfWindow*>(base + o_win);
  float* d_plots = reinterpret_cast<float*>(base + o_plots);
  float* d_scr = reinterpret_cast<float*>(base + o_scr);
  if (cudaMemcpyAsync(base, plan.data(), plan.size(), cudaMemcpyHostToDevice, s) ||
      cudaMemsetAsync(d_plots, 0, dm0_at * sizeof(float), s))
    return HD_MEM_COPY_FAILED;
  const unsigned nrows = (unsigned)rows.size();
  for (size_t k = 0; k + 1 < batch.size(); k++) {
    const size_t i0 = batch[k], i1 = batch[k + 1];
    const size_t r0 = first_row[i0], r1 = first_row[i1];
    unsigned max_n = 0, max_w = 0;
    for (size_t i = i0; i < i1; i++) max_w = std::max(max_w, windows[i].n);
    for (size_t r = r0; r < r1; r++) {
      const unsigned sr = (unsigned)rows[r].s;  // blocks of 128 threads of max(1, 4 / s) outputs
      max_n = std::max(max_n, rows[r].nd / sr / (sr < 4 ? 4 / sr : 1));
    }
    if (max_w) {
      for (size_t i = i0; i < i1; i += 65535) {
        k_prof_window<<<dim3((max_w + 127) / 128, (unsigned)((C + 31) / 32),
                             (unsigned)std::min<size_t>(i1 - i, 65535)),
                        256, 0, s>>>(tf, nsamps, (int)C, d_win + i, base + o_windows);
        note_launch();
      }
    }
    k_prof_dedisp<<<dim3(max_n / 128 + 1, (unsigned)(r1 - r0)), 128, 0, s>>>(
        base + o_windows, d_win + i0, (int)i0, (int)C, d_table, d_rows + r0, d_scr);
    note_launch();
  }
  // plot rows: the DM-time rows and the DM-0 rows share the row list
  const int on = (int)out_nsamps;
  if (!do_filter)
    k_prof_boxcar<<<dim3((on + 127) / 128, nrows), 128, 0, s>>>(d_rows, d_scr, on, d_plots);
  else
    k_prof_filter<<<(nrows + 63) / 64, 64, 0, s>>>(
        d_rows, (int)nrows, d_scr, reinterpret_cast<float*>(base + o_pre), on, d_plots);
  note_launch();
  // channel groups per warp and samples per stage (k_prof_ft)
  const int fs = (int)fscrunch;
  const int ncs = (int)std::min<size_t>(out_nchans, (size_t)std::max(1, std::min(32, 2048 / fs)));
  const int nf = std::min(fs, FT_STAGE);
  const int nrow = nf < fs ? 1 : std::max(1, std::min(64, FT_STAGE / (ncs * fs)));
  const bool whole_words = C % 4 == 0 && fs % 4 == 0 && (reinterpret_cast<uintptr_t>(tf) & 3) == 0;
  bool any_exact = false, any_long = !whole_words;
  for (const FtJob& j : ftj) {
    const bool exact = whole_words && (size_t)j.ts * fs <= kFtExact;
    any_exact = any_exact || exact;
    any_long = any_long || !exact;
  }
  for (size_t i = 0; i < ncands; i += 65535) {
    const unsigned nz = (unsigned)std::min<size_t>(ncands - i, 65535);
    const FtJob* d_ftj = reinterpret_cast<const FtJob*>(base + o_ftj) + i;
    if (any_exact) {
      const int groups = std::max(1, 128 / fs);  // 32 at most: fs >= 4
      k_prof_ft_exact<<<dim3((on + FX_BINS - 1) / FX_BINS,
                             (unsigned)((out_nchans + groups - 1) / groups), nz),
                        32 * FX_BINS, 0, s>>>(tf, nsamps, (int)C, fs, groups, on, d_ftj, d_plots);
      note_launch();
    }
    if (any_long) {
      k_prof_ft<<<dim3((on + FT_BINS - 1) / FT_BINS, (unsigned)((out_nchans + ncs - 1) / ncs),
                       nz),
                  32 * FT_BINS, 0, s>>>(tf, nsamps, (int)C, fs, ncs, nf, nrow, whole_words, on,
                                        d_ftj, d_plots);
      note_launch();
    }
  }
  if (cudaGetLastError() != cudaSuccess) return HD_INTERNAL_GPU_ERROR;
  // normalise every DM-time and DM-0 row and the freq-time rows, in one launch
  const cudaError_t e = normalise_row_list(
      d_plots, on, reinterpret_cast<const size_t*>(base + o_at), nrows, ft_at,
      ncands * out_nchans, s);
  if (e != cudaSuccess) return e == cudaErrorMemoryAllocation ? HD_MEM_ALLOC_FAILED
                                                              : HD_INTERNAL_GPU_ERROR;

  // ---- results to the host and the extractions (candidate_profiler.C:560-640)
  std::vector<float> h_plots(plot_floats);
  if (cudaMemcpyAsync(h_plots.data(), d_plots, plot_floats * sizeof(float),
                      cudaMemcpyDeviceToHost, s))
    return HD_MEM_COPY_FAILED;
  if (cudaStreamSynchronize(s) != cudaSuccess) return HD_INTERNAL_GPU_ERROR;
  for (size_t i = 0; i < ncands; i++) {
    hd_profile& o = out[i];
    const float* dmt = h_plots.data() + i * plot;
    const float* dm0 = h_plots.data() + dm0_at + i * out_nsamps;
    if (o.freq_time)
      std::memcpy(o.freq_time, h_plots.data() + ft_at + i * out_nchans * out_nsamps,
                  out_nchans * out_nsamps * sizeof(float));
    if (o.dm_time) std::memcpy(o.dm_time, dmt, plot * sizeof(float));
    if (o.dm0_time) std::memcpy(o.dm0_time, dm0, out_nsamps * sizeof(float));
    // first maximum (std::max_element: a NaN never replaces a number)
    size_t mx = 0;
    for (size_t k = 1; k < plot; k++)
      if (dmt[mx] < dmt[k]) mx = k;
    o.max_idx = mx;
    o.n_dm = n_dm[i];
    o.dm_begin = dm_begin[i];
    const size_t dm_idx = cands[i].dm_idx;
    o.snr_dm_first = dm_idx > out_dm_count / 2 ? dm_idx - out_dm_count / 2 : 0;
    const size_t tmax = mx % out_nsamps, dmax = mx / out_nsamps;
    if (o.snr_dm)
      for (size_t d = 0; d < out_dm_count; d++)
        o.snr_dm[d] = d < n_dm[i] ? dmt[d * out_nsamps + tmax] : 0.f;
    if (o.snr_time) {
      const float width = (float)((size_t)1 << cands[i].filter);
      for (size_t t = 0; t < out_nsamps; t++) {
        float* r = o.snr_time + t * 5;
        r[0] = (float)((double)((float)cands[i].samp +
                                ((float)t - (float)(out_nsamps / 2)) * width) *
                       tsamp);
        r[1] = dmt[dmax * out_nsamps + t];
        r[2] = dmax > 0 ? dmt[(dmax - 1) * out_nsamps + t] : 0.f;
        r[3] = dmax + 1 < out_dm_count ? dmt[(dmax + 1) * out_nsamps + t] : 0.f;
        r[4] = dm0[t];
      }
    }
  }
  return HD_NO_ERROR;
}
