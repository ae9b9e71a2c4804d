// HHG spectrum of a current on the device: the recipe of the reference's scripts/pol_scan.py:34-40,
//   S = fftshift(fft(ifftshift(gradient(J, h))))      (numpy semantics, h = sample spacing)
// and the harmonic intensities of its order axis (scripts/pol_scan.py:50-57):
//   order_i = linspace(-wmax, wmax, n)_i / w0,  wmax = n pi / tmax,  w0 = 2 pi 300 / lambda_nm,
//   I_h = sum over order_i in (h - 1/2, h + 1/2) of |S_i|^2   for odd h.
//
// The FFT is a batched mixed-radix Stockham transform (autosorting, so no bit reversal): n is
// factored into radices 4, 2, 3, 5 and any remaining prime, and each pass reads the previous pass's
// buffer and writes the other.  For a pass of radix R after a product Ns of earlier radices, butterfly
// j (of n/R) takes the R inputs j + r n/R, multiplies input r by e^{-2 pi i r (j mod Ns) / (Ns R)},
// forms their length-R DFT and writes output q to (j div Ns) Ns R + (j mod Ns) + q Ns.  The first pass
// reads the gradient of the current through the ifftshift, the last one writes through the fftshift.
// A block runs all passes of one signal in shared memory (up to 7040 samples; longer ones go pass by pass
// through global memory).  Radices up to 8 take a thread per butterfly, larger ones a thread per output, and all
// factors come from one table of the n-th roots: a radix-4093 pass was one thread with a sincospi per term.
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdio>
#include <vector>

#include "sbe_device.h"
#include "smem_limit.h"

namespace hhg {
namespace {

// The order axis of n samples: linspace(-wmax, wmax, n) / w0, its divisions made once on the host.
struct OrderAxis {
  int n;
  double w0, wmax, step, per_step;
};
OrderAxis order_axis(int n, double tmax, double lambda_nm) {
  OrderAxis x;
  x.n = n;
  x.w0 = 2.0 * M_PI * 300.0 / lambda_nm;
  x.wmax = n * (2.0 * M_PI / tmax) / 2.0;
  x.step = n > 1 ? 2.0 * x.wmax / (double)(n - 1) : 1.0;
  x.per_step = 1.0 / x.step;
  return x;
}

// Samples [lo, hi) that can hold orders between a and b: two more on either side than the axis says.
__host__ __device__ inline void harmonic_window(const OrderAxis& ax, double a, double b, int* lo, int* hi) {
  const double n = (double)ax.n;
  const double x = floor((a * ax.w0 + ax.wmax) * ax.per_step) - 2.0, y = ceil((b * ax.w0 + ax.wmax) * ax.per_step) + 3.0;
  *lo = x < 0.0 ? 0 : (x > n ? ax.n : (int)x);
  *hi = y < 0.0 ? 0 : (y > n ? ax.n : (int)y);
}

__device__ __forceinline__ double2 sp_mul(double2 a, double2 b) {
  return make_double2(fma(a.x, b.x, -a.y * b.y), fma(a.x, b.y, a.y * b.x));
}

// e^{-2 pi i num / den} for 0 <= num < den.
__device__ __forceinline__ double2 sp_twiddle(long long num, long long den) {
  double s, c;
  sincospi(-2.0 * (double)num / (double)den, &s, &c);
  return make_double2(c, s);
}

// numpy.gradient (second-order central differences inside, first-order at the ends, the same
// divisions as numpy) of a signal at index i, read through ifftshift: element i of ifftshift(g) is
// g[(i + n/2) mod n].
__device__ __forceinline__ double2 sp_grad_shifted(const double2* J, int n, int i, double h) {
  const int g = (i + n / 2) % n;
  if (g == 0) return make_double2((J[1].x - J[0].x) / h, (J[1].y - J[0].y) / h);
  if (g == n - 1) return make_double2((J[n - 1].x - J[n - 2].x) / h, (J[n - 1].y - J[n - 2].y) / h);
  const double h2 = 2.0 * h;
  return make_double2((J[g + 1].x - J[g - 1].x) / h2, (J[g + 1].y - J[g - 1].y) / h2);
}

__device__ __forceinline__ double2 sp_fma(double2 a, double2 w, double2 acc) {
  return make_double2(fma(a.x, w.x, fma(-a.y, w.y, acc.x)), fma(a.x, w.y, fma(a.y, w.x, acc.y)));
}

// w[k] = e^{-2 pi i k / n}.
__global__ void roots_kernel(double2* w, int n) {
  const int k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k < n) w[k] = sp_twiddle(k, n);
}

// Work item `it` of a pass: a butterfly (radix up to 8: n / R items) or one output of one (n items).
// in(i): input i of the pass; out(o, value).  All factors are powers of the n-th root w.
template <typename In, typename Out>
__device__ __forceinline__ void stockham_item(int it, int n, int R, int Ns, const double2* w, In&& in, Out&& out) {
  constexpr int kMaxReg = 8;
  const int stride = n / R;
  const int j = R <= kMaxReg ? it : it % stride, k = j % Ns, base = (j / Ns) * Ns * R + k;
  const int tk = k * (n / (Ns * R));  // input r's factor: root r tk (r k < Ns R, so r tk < n)
  const int fq = stride;              // the DFT's root: e^{-2 pi i / R} = w^(n / R)
  if (R <= kMaxReg) {
    double2 v[kMaxReg];
#pragma unroll
    for (int r = 0; r < kMaxReg; ++r)
      if (r < R) {
        v[r] = in(j + r * stride);
        if (r > 0) v[r] = sp_mul(v[r], w[r * tk]);
      }
#pragma unroll
    for (int q = 0; q < kMaxReg; ++q)
      if (q < R) {
        double2 acc = v[0];
#pragma unroll
        for (int r = 1; r < kMaxReg; ++r)
          if (r < R) acc = sp_fma(v[r], w[r * q % R * fq], acc);
        out(base + q * Ns, acc);
      }
  } else {
    const int q = it / stride;
    double2 acc = make_double2(0.0, 0.0);
    int rq = 0, rt = 0;  // r q mod R, r tk mod n
    for (int r = 0; r < R; ++r) {
      const double2 x = in(j + r * stride);
      acc = sp_fma(r == 0 ? x : sp_mul(x, w[rt]), w[rq * fq], acc);
      rq += q;
      if (rq >= R) rq -= R;
      rt += tk;
    }
    out(base + q * Ns, acc);
  }
}

// Radices of a length (a length below 2^31 has at most 30 factors).
struct Radices {
  int count, r[30];
};
constexpr int kBlockSamples = 7040;  // two buffers of a signal in 220 KB of shared memory
constexpr int kBlockThreads = 512;  // at most: a thread per sample of shorter signals

// A block per signal, all passes in shared memory.
__global__ void __launch_bounds__(kBlockThreads) stockham_block_kernel(const double2* J, double2* S, const double2* w,
                                                                       int n, Radices rad, double h) {
  extern __shared__ __align__(16) double2 sp_buf[];
  const double2* Jb = J + (size_t)blockIdx.x * n;
  double2* Sb = S + (size_t)blockIdx.x * n;
  int Ns = 1;
  for (int p = 0; p < rad.count; ++p) {
    const int R = rad.r[p], items = R <= 8 ? n / R : n;
    const bool first = p == 0, last = p == rad.count - 1;
    const double2* src = sp_buf + (size_t)(p & 1) * n;
    double2* dst = sp_buf + (size_t)(~p & 1) * n;
    // (a large first radix reads each input for every output: the gradient is formed once)
    if (first && R > 8) {
      for (int i = threadIdx.x; i < n; i += blockDim.x) sp_buf[i] = sp_grad_shifted(Jb, n, i, h);
      __syncthreads();
    }
    for (int it = threadIdx.x; it < items; it += blockDim.x)
      stockham_item(
          it, n, R, Ns, w, [&](int i) { return first && R <= 8 ? sp_grad_shifted(Jb, n, i, h) : src[i]; },
          [&](int o, double2 v) {
            if (last)
              Sb[o + n / 2 < n ? o + n / 2 : o + n / 2 - n] = v;  // fftshift: element i of the result is X[(i - n/2) mod n]
            else
              dst[o] = v;
          });
    Ns *= R;
    __syncthreads();
  }
}

// One pass over `count` signals through global memory.  first: read gradients of J through the ifftshift; last:
// write through the fftshift.
__global__ void stockham_pass_kernel(const double2* in, double2* out, const double2* J, const double2* w, int n, int count,
                                     int R, int Ns, int first, int last, double h) {
  const int items = R <= 8 ? n / R : n;
  const long long gid = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (gid >= (long long)count * items) return;
  const int b = (int)(gid / items), it = (int)(gid % items);
  const double2* src = first ? nullptr : in + (size_t)b * n;
  const double2* Jb = J + (size_t)b * n;
  double2* dst = out + (size_t)b * n;
  stockham_item(
      it, n, R, Ns, w, [&](int i) { return first ? sp_grad_shifted(Jb, n, i, h) : src[i]; },
      [&](int o, double2 v) { dst[last ? (o + n / 2) % n : o] = v; });
}

// I[b][h'] for odd harmonics h = 2 h' + 1: sum of |S|^2 over order in (h - 1/2, h + 1/2).  `lanes` lanes per value, as
// many as its window has samples, up to a warp; the samples of the window are found from the order axis (with a margin
// for its rounding) and each is tested as written above.  S holds the samples i0 .. i0 + ni - 1 of each signal.
// (A thread per value that tested all n samples took 1 ms for any number of signals; a warp per value whatever its
// window 20.6 ms a call, copies included, for 300 000 signals of 3 samples and 25 values, against 18.2.)
__global__ void harmonics_kernel(const double2* S, OrderAxis ax, int i0, int ni, long long values, int nh, int lanes,
                                 double* I) {
  // (in 64 bits: 2^27 values of a warp each are 2^32 threads)
  const long long gid = ((long long)blockIdx.x * blockDim.x + threadIdx.x) / lanes;
  const int lane = threadIdx.x & (lanes - 1);
  double acc = 0.0;
  if (gid < values) {
    const long long b = gid / nh;
    const double h = 2.0 * (double)(gid - b * nh) + 1.0;
    int lo, hi;
    harmonic_window(ax, h - 0.5, h + 0.5, &lo, &hi);
    lo = max(lo, i0);
    hi = min(hi, i0 + ni);
    for (int i = lo + lane; i < hi; i += lanes) {
      const double order = (-ax.wmax + ax.step * i) / ax.w0;
      if (order > h - 0.5 && order < h + 0.5) {
        const double2 s = S[(size_t)b * ni + (i - i0)];
        acc += s.x * s.x + s.y * s.y;
      }
    }
  }
  for (int o = lanes / 2; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
  if (gid < values && lane == 0) I[gid] = acc;
}

std::vector<int> factor_radices(int n) {
  std::vector<int> f;
  while (n % 4 == 0) {
    f.push_back(4);
    n /= 4;
  }
  for (int p : {2, 3, 5}) {
    while (n % p == 0) {
      f.push_back(p);
      n /= p;
    }
  }
  for (int p = 7; (long long)p * p <= n; p += 2)
    while (n % p == 0) {
      f.push_back(p);
      n /= p;
    }
  if (n > 1) f.push_back(n);
  return f;
}

}  // namespace

// scratch: count n values and, after them, n for the table of roots.
int spectrum_device(const double2* J, int n, int count, double h, double2* S, double2* scratch, cudaStream_t stream) {
  if (n < 2 || count < 1 || h <= 0.0) return -1;
  const std::vector<int> rad = factor_radices(n);
  const int passes = (int)rad.size();
  double2* w = scratch + (size_t)count * n;
  roots_kernel<<<(n + 255) / 256, 256, 0, stream>>>(w, n);
  const size_t smem = 2 * (size_t)n * sizeof(double2);
  if (n <= kBlockSamples && allow_shared_memory(stockham_block_kernel, smem)) {
    Radices r{};
    r.count = passes;
    for (int p = 0; p < passes; ++p) r.r[p] = rad[p];
    stockham_block_kernel<<<count, std::min(kBlockThreads, (n + 31) / 32 * 32), smem, stream>>>(J, S, w, n, r, h);
    return cudaGetLastError() == cudaSuccess ? passes : -1;
  }
  // Ping-pong between S and scratch so that the last pass lands in S.
  double2* bufs[2] = {S, scratch};
  int cur = passes % 2 == 1 ? 0 : 1;  // buffer written by the first pass
  int Ns = 1;
  const double2* prev = nullptr;
  for (int p = 0; p < passes; ++p) {
    const int R = rad[p];
    const long long threads = (long long)count * (R <= 8 ? n / R : n);
    const int block = 128;
    const int grid = (int)((threads + block - 1) / block);
    stockham_pass_kernel<<<grid, block, 0, stream>>>(prev, bufs[cur], J, w, n, count, R, Ns, p == 0, p == passes - 1, h);
    prev = bufs[cur];
    cur ^= 1;
    Ns *= R;
  }
  return cudaGetLastError() == cudaSuccess ? passes : -1;
}

void harmonics_range(int n, double tmax, double lambda_nm, int nh, int* i0, int* ni) {
  int lo, hi;
  harmonic_window(order_axis(n, tmax, lambda_nm), 0.5, 2.0 * nh - 0.5, &lo, &hi);
  *i0 = lo;
  *ni = hi > lo ? hi - lo : 0;
}

int harmonics_device(const double2* S, int n, int i0, int ni, int count, double tmax, double lambda_nm, int nh, double* I,
                     cudaStream_t stream) {
  if (n < 2 || count < 1 || nh < 1 || tmax <= 0.0 || lambda_nm <= 0.0) return -1;
  const OrderAxis ax = order_axis(n, tmax, lambda_nm);
  const double window = ax.w0 * ax.per_step + 6.0;  // samples tested per value, at most
  int lanes = 1;
  while (lanes < 32 && lanes < window) lanes *= 2;
  const long long values = (long long)count * nh;
  harmonics_kernel<<<(unsigned)((values * lanes + 127) / 128), 128, 0, stream>>>(S, ax, i0, ni, values, nh, lanes, I);
  return cudaGetLastError() == cudaSuccess ? 0 : -1;
}

}  // namespace hhg
