// Post-processing of receiver traces (python/FDTDfilter.py:13-19,
// matlab/functions/FDTDpostFilter.m:1-31, matlab/testBench.m:203-204): a
// causal FIR low-pass, an optional DC blocker y[n] = x[n] - x[n-1] + a y[n-1],
// and a polyphase rational resampler, over many channels.  Arithmetic in
// double; float or double input and output.
#include "common.cuh"

#include <algorithm>

namespace pfdtd {
namespace {

// y[c][n] = sum_{k <= min(n, nb-1)} b[k] x[c][n-k]; one thread per output.
template <typename T>
__global__ void k_fir(const T* __restrict__ x, int64_t n_ch, int64_t n, const double* __restrict__ b,
                      int nb, T* __restrict__ y) {
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n_ch * n;
       i += (int64_t)gridDim.x * blockDim.x) {
    const int64_t c = i / n, t = i - c * n;
    const T* xc = x + c * n;
    double acc = 0.0;
    const int kmax = t < (int64_t)(nb - 1) ? (int)t : nb - 1;
    for (int k = 0; k <= kmax; ++k) acc += b[k] * (double)xc[t - k];
    y[i] = (T)acc;
  }
}

// DC blocker in place, one thread per channel: the recursion as written, for
// short or many traces (dc_scan_pays) and for coefficients outside [-1, 1], whose
// powers k_dc_block could not hold.
template <typename T>
__global__ void k_dc_block_serial(T* __restrict__ y, int64_t n_ch, int64_t n, double a) {
  const int64_t c = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (c >= n_ch) return;
  T* yc = y + c * n;
  double xp = 0.0, yp = 0.0;
  for (int64_t t = 0; t < n; ++t) {
    const double xv = (double)yc[t];
    const double v = xv - xp + a * yp;
    xp = xv;
    yp = v;
    yc[t] = (T)v;
  }
}

// Unevaluated sums of two doubles (Knuth's two-sum, Dekker's product): the
// states that the DC blocker's threads hand on carry no rounding of their own.
struct Dd { double h, l; };

__host__ __device__ inline Dd dd_norm(double h, double l) {
  const double s = h + l;
  // an overflowed trace stays at its infinity
  return fabs(h) <= 1.7976931348623157e308 ? Dd{s, l - (s - h)} : Dd{h, 0.0};
}
__host__ __device__ inline Dd dd_add(Dd x, Dd y) {
  const double s = x.h + y.h, b = s - x.h;
  return dd_norm(s, (x.h - (s - b)) + (y.h - b) + (x.l + y.l));
}
__host__ __device__ inline Dd dd_mul(Dd x, Dd y) {
  const double p = x.h * y.h;
  return dd_norm(p, fma(x.h, y.h, -p) + (x.h * y.l + x.l * y.h));
}
__device__ __forceinline__ Dd dd_shfl_up(Dd v, int by) {
  return Dd{__shfl_up_sync(0xffffffffu, v.h, by), __shfl_up_sync(0xffffffffu, v.l, by)};
}

// DC blocker in place, one block per channel, |a| <= 1.  The recursion is a
// serial chain over the trace: one thread per channel spent 1137 us on 16
// traces of 8000 samples, a global load and two dependent FP64 operations a
// sample.  Here a thread takes kDcPer neighbouring samples of a tile, finds
// their final state from a zero state, a scan combines those (state = b +
// a^kDcPer * state before) into the state that each thread starts from, and
// each thread runs the recursion from there.  States are sums of two doubles:
// a scan in plain doubles was 1.4 times as far from the exact trace as the
// serial chain, this one rounds the exact trace (1e-17 of it off against 1e-15).  FP64 operations bound it
// (an SM issues about two a cycle), so the scan is spread over 16 samples a
// thread: 103 us on the same traces.
constexpr int kDcThreads = 512, kDcPer = 16;
struct DcPowers { Dd p[9]; };  // a^(kDcPer 2^k)

template <typename T>
__global__ void __launch_bounds__(kDcThreads) k_dc_block(T* __restrict__ y, int64_t n, double a,
                                                         const DcPowers pw) {
  constexpr int kWarps = kDcThreads / 32;
  __shared__ Dd warp_state[kWarps];
  __shared__ Dd carry_state;
  __shared__ double carry_x;
  T* yc = y + blockIdx.x * n;
  const int t = threadIdx.x, lane = t & 31, w = t >> 5;
  if (t == 0) {
    carry_state = Dd{0.0, 0.0};
    carry_x = 0.0;
  }
  // A state times a power of a; one that is not finite stays as it is, also where
  // the power has underflowed to 0 (as in the recursion, unless a itself is 0;
  // the powers are even, so positive).
  const bool lasting = a != 0.0;
  auto damped = [&](Dd power, Dd state) {
    return lasting && not_finite(state.h) ? Dd{state.h, 0.0} : dd_mul(power, state);
  };
  Dd damp{1.0, 0.0};  // a^(kDcPer lane)
#pragma unroll
  for (int k = 0; k < 5; ++k)
    if (lane & (1 << k)) damp = dd_mul(damp, pw.p[k]);
  for (int64_t base = 0; base < n; base += kDcThreads * kDcPer) {
    const int64_t i0 = base + t * kDcPer;
    __syncthreads();  // the tile before is written, its carry in place
    const double x0 = t == 0 ? carry_x : (i0 - 1 < n ? (double)yc[i0 - 1] : 0.0);
    double x[kDcPer];
#pragma unroll
    for (int k = 0; k < kDcPer; ++k) x[k] = i0 + k < n ? (double)yc[i0 + k] : 0.0;
    // one step of the recursion on v + low: what the difference, the product
    // and the sum round away is carried in low
    double v = 0.0, low = 0.0, xp = x0;
    auto step = [&](double xv) {
      const double d = xv - xp, c = d - xv, p = a * v, s = p + d, b = s - p;
      low = fma(a, low, fma(a, v, -p)) + ((p - (s - b)) + (d - b)) + ((xv - (d - c)) - (xp + c));
      v = s;
      xp = xv;
    };
    // the thread's final state from a zero state, then the scan over the warp
#pragma unroll
    for (int k = 0; k < kDcPer; ++k) step(x[k]);
    Dd inc = dd_norm(v, low);
#pragma unroll
    for (int k = 0; k < 5; ++k) {
      const Dd u = dd_shfl_up(inc, 1 << k);
      if (lane >= (1 << k)) inc = dd_add(inc, damped(pw.p[k], u));
    }
    Dd in = dd_shfl_up(inc, 1);  // state after the thread before, from the warp's start
    if (lane == 0) in = Dd{0.0, 0.0};
    if (lane == 31) warp_state[w] = inc;
    __syncthreads();
    if (w == 0) {  // the states after each warp, from the tile's start
      Dd s = lane < kWarps ? warp_state[lane] : Dd{0.0, 0.0};
      if (lane == 0) s = dd_add(s, damped(pw.p[5], carry_state));
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        const Dd u = dd_shfl_up(s, 1 << k);
        if (lane >= (1 << k)) s = dd_add(s, damped(pw.p[5 + k], u));
      }
      if (lane < kWarps) warp_state[lane] = s;
    }
    __syncthreads();
    const Dd before = w == 0 ? carry_state : warp_state[w - 1];
    in = dd_add(in, damped(damp, before));
    __syncthreads();  // every thread has read its samples and the carried values
    // a tile that is not the trace's last is whole
    if (t == kDcThreads - 1) {
      carry_state = warp_state[kWarps - 1];
      carry_x = x[kDcPer - 1];
    }
    v = in.h;
    low = in.l;
    xp = x0;
#pragma unroll
    for (int k = 0; k < kDcPer; ++k) {
      step(x[k]);
      if (i0 + k < n) yc[i0 + k] = (T)(fabs(v) <= 1.7976931348623157e308 ? v + low : v);
    }
  }
}

// Polyphase resampler: y[c][j] = sum_i h[(j + offset) * down - i * up] x[c][i]
// over the i with the tap index in [0, nh) (zero-stuffing by `up`, FIR `h`,
// keeping every `down`-th sample from `offset` on); one thread per output.
template <typename T>
__global__ void k_resample(const T* __restrict__ x, int64_t n_ch, int64_t n_in,
                           const double* __restrict__ h, int nh, int up, int down, int64_t offset,
                           int64_t n_out, T* __restrict__ y) {
  for (int64_t k = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; k < n_ch * n_out;
       k += (int64_t)gridDim.x * blockDim.x) {
    const int64_t c = k / n_out, j = k - c * n_out;
    const int64_t t = (j + offset) * down;  // position on the up-sampled axis
    int64_t i_hi = t / up;                  // largest i with t - i*up >= 0
    const int64_t lo_num = t - (nh - 1);    // smallest i with t - i*up <= nh - 1
    int64_t i_lo = lo_num <= 0 ? 0 : (lo_num + up - 1) / up;
    if (i_hi > n_in - 1) i_hi = n_in - 1;
    const T* xc = x + c * n_in;
    double acc = 0.0;
    for (int64_t i = i_lo; i <= i_hi; ++i) acc += h[t - i * up] * (double)xc[i];
    y[k] = (T)acc;
  }
}

template <typename T>
int resample_t(const T* x, int64_t n_ch, int64_t n_in, const double* h, int nh, int up, int down,
               int64_t offset, int64_t n_out, T* out, int device) {
  int prev = -1;
  cudaGetDevice(&prev);
  if (prev != device) cudaSetDevice(device);
  struct Restore {
    int p;
    ~Restore() { if (p >= 0) cudaSetDevice(p); }
  } restore{prev};
  cudaStream_t s = nullptr;
  PFDTD_CK(cudaStreamCreateWithFlags(&s, cudaStreamNonBlocking));
  const size_t in_bytes = (size_t)n_ch * (size_t)n_in * sizeof(T);
  const size_t out_bytes = (size_t)n_ch * (size_t)n_out * sizeof(T);
  T *dx = nullptr, *dy = nullptr;
  double* dh = nullptr;
  cudaError_t e = cudaMallocAsync((void**)&dx, in_bytes, s);
  if (e == cudaSuccess) e = cudaMallocAsync((void**)&dy, out_bytes, s);
  if (e == cudaSuccess) e = cudaMallocAsync((void**)&dh, sizeof(double) * nh, s);
  if (e == cudaSuccess) e = cudaMemcpyAsync(dx, x, in_bytes, cudaMemcpyHostToDevice, s);
  if (e == cudaSuccess) e = cudaMemcpyAsync(dh, h, sizeof(double) * nh, cudaMemcpyHostToDevice, s);
  if (e == cudaSuccess) {
    const int64_t tot = n_ch * n_out;
    const int grid = (int)std::max<int64_t>(1, std::min<int64_t>((tot + 255) / 256, kGridSMs * 32));
    k_resample<T><<<grid, 256, 0, s>>>(dx, n_ch, n_in, dh, nh, up, down, offset, n_out, dy);
    count_launch();
    e = cudaGetLastError();
  }
  if (e == cudaSuccess) e = cudaMemcpyAsync(out, dy, out_bytes, cudaMemcpyDeviceToHost, s);
  for (void* p : {(void*)dx, (void*)dy, (void*)dh})
    if (p) cudaFreeAsync(p, s);
  const cudaError_t e2 = cudaStreamSynchronize(s);
  cudaStreamDestroy(s);
  if (e == cudaSuccess) e = e2;
  if (e != cudaSuccess) return cuda_fail(e, "resample", __FILE__, __LINE__);
  return PFDTD_OK;
}

// Whether the DC blocker's block scan is faster than one thread per channel.  A
// serial thread takes 0.14 us a sample (0.18 where the samples are floats), the
// channels side by side; the scan takes an SM's FP64 units for 105 us a tile and
// channel, also where the trace is shorter than the tile.  Measured, us, serial /
// scan, FP64: 16 x 500 71 / 126, 16 x 1000 127 / 96, 16 x 8000 1039 / 101, 304 x 8000
// 1803 / 209, 1000 x 8000 1294 / 735, 1000 x 500 162 / 719, 4000 x 500 277 / 2735,
// 20000 x 100 117 / 13340.
bool dc_scan_pays(int64_t n_ch, int64_t n) {
  constexpr int64_t tile = kDcThreads * kDcPer;
  const int64_t tiles = (n + tile - 1) / tile, waves = (n_ch + kGridSMs - 1) / kGridSMs;
  return 105.0 * (double)tiles * (double)waves < 0.15 * (double)n;
}

template <typename T>
int post_filter_t(const T* x, int64_t n_ch, int64_t n, const double* b, int nb, int dc, double a,
                  T* out, int device) {
  int prev = -1;
  cudaGetDevice(&prev);
  if (prev != device) cudaSetDevice(device);
  struct Restore {
    int p;
    ~Restore() { if (p >= 0) cudaSetDevice(p); }
  } restore{prev};
  cudaStream_t s = nullptr;
  PFDTD_CK(cudaStreamCreateWithFlags(&s, cudaStreamNonBlocking));
  const size_t bytes = (size_t)n_ch * (size_t)n * sizeof(T);
  T *dx = nullptr, *dy = nullptr;
  double* db = nullptr;
  cudaError_t e = cudaMallocAsync((void**)&dx, bytes, s);
  if (e == cudaSuccess) e = cudaMallocAsync((void**)&dy, bytes, s);
  if (e == cudaSuccess) e = cudaMallocAsync((void**)&db, sizeof(double) * nb, s);
  if (e == cudaSuccess) e = cudaMemcpyAsync(dx, x, bytes, cudaMemcpyHostToDevice, s);
  if (e == cudaSuccess) e = cudaMemcpyAsync(db, b, sizeof(double) * nb, cudaMemcpyHostToDevice, s);
  if (e == cudaSuccess) {
    const int64_t tot = n_ch * n;
    const int grid = (int)std::max<int64_t>(1, std::min<int64_t>((tot + 255) / 256, kGridSMs * 32));
    k_fir<T><<<grid, 256, 0, s>>>(dx, n_ch, n, db, nb, dy);
    count_launch();
    if (dc) {
      if (std::fabs(a) <= 1.0 && dc_scan_pays(n_ch, n)) {
        DcPowers pw;
        pw.p[0] = Dd{a, 0.0};
        for (int k = 1; k < kDcPer; k *= 2) pw.p[0] = dd_mul(pw.p[0], pw.p[0]);
        for (int k = 1; k < 9; ++k) pw.p[k] = dd_mul(pw.p[k - 1], pw.p[k - 1]);
        k_dc_block<T><<<(unsigned)n_ch, kDcThreads, 0, s>>>(dy, n, a, pw);
      } else {
        k_dc_block_serial<T><<<(int)((n_ch + 127) / 128), 128, 0, s>>>(dy, n_ch, n, a);
      }
      count_launch();
    }
    e = cudaGetLastError();
  }
  if (e == cudaSuccess) e = cudaMemcpyAsync(out, dy, bytes, cudaMemcpyDeviceToHost, s);
  for (void* p : {(void*)dx, (void*)dy, (void*)db})
    if (p) cudaFreeAsync(p, s);
  const cudaError_t e2 = cudaStreamSynchronize(s);
  cudaStreamDestroy(s);
  if (e == cudaSuccess) e = e2;
  if (e != cudaSuccess) return cuda_fail(e, "post filter", __FILE__, __LINE__);
  return PFDTD_OK;
}

}  // namespace
}  // namespace pfdtd

using namespace pfdtd;

extern "C" int pfdtd_resample(const void* x, int64_t n_channels, int64_t n_in, int is_double,
                              const double* taps, int n_taps, int up, int down, int64_t offset,
                              int64_t n_out, void* out, int device) {
  if (n_channels < 0 || n_in < 1 || n_out < 0 || n_taps < 1 || !taps || up < 1 || down < 1 ||
      offset < 0 || (n_channels * n_out > 0 && (!x || !out)))
    return fail(PFDTD_ERR_ARG, "invalid resampling arguments");
  if (n_channels * n_out == 0) return PFDTD_OK;
  return is_double ? resample_t<double>((const double*)x, n_channels, n_in, taps, n_taps, up, down,
                                        offset, n_out, (double*)out, device)
                   : resample_t<float>((const float*)x, n_channels, n_in, taps, n_taps, up, down,
                                       offset, n_out, (float*)out, device);
}

extern "C" int pfdtd_post_filter(const void* x, int64_t n_channels, int64_t n_samples,
                                 int is_double, const double* taps, int n_taps, int dc_block,
                                 double dc_coef, void* out, int device) {
  if (n_channels < 0 || n_samples < 0 || n_taps < 1 || !taps ||
      (n_channels * n_samples > 0 && (!x || !out)))
    return fail(PFDTD_ERR_ARG, "invalid filter arguments");
  if (n_channels * n_samples == 0) return PFDTD_OK;
  return is_double ? post_filter_t<double>((const double*)x, n_channels, n_samples, taps, n_taps,
                                           dc_block, dc_coef, (double*)out, device)
                   : post_filter_t<float>((const float*)x, n_channels, n_samples, taps, n_taps,
                                          dc_block, dc_coef, (float*)out, device);
}
