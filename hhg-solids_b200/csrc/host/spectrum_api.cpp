// HHG spectra on the device (the post-processing of the reference's scripts/pol_scan.py:34-40),
// for a solve's recorded current or for caller-supplied currents.
#include <cuda_runtime.h>

#include <algorithm>
#include <stdexcept>
#include <string>
#include <vector>

#include "swe_sim.hpp"

using hhg::check_cuda;

namespace {

// Device workspace of one call, from the device's stream-ordered pool (as a solve's buffers), which is asked to
// keep kKeepBytes between calls if it keeps less: a cudaMalloc and cudaFree per buffer and call took 1 to 30 ms a
// call, both wait for the whole device, and the transform of a solve's current takes 0.05.  Allocated and freed in
// the order of the call's stream, so calls of several threads and streams do not share memory that is in use.
constexpr uint64_t kKeepBytes = uint64_t(256) << 20;

void keep_pool_memory() {
  int dev = 0;
  check_cuda(cudaGetDevice(&dev), "cudaGetDevice");
  cudaMemPool_t pool = nullptr;
  check_cuda(cudaDeviceGetDefaultMemPool(&pool, dev), "cudaDeviceGetDefaultMemPool");
  uint64_t keep = 0;
  check_cuda(cudaMemPoolGetAttribute(pool, cudaMemPoolAttrReleaseThreshold, &keep), "cudaMemPoolGetAttribute");
  if (keep >= kKeepBytes) return;
  keep = kKeepBytes;
  check_cuda(cudaMemPoolSetAttribute(pool, cudaMemPoolAttrReleaseThreshold, &keep), "cudaMemPoolSetAttribute");
}

struct Workspace {
  char* p = nullptr;
  cudaStream_t stream;
  Workspace(size_t bytes, cudaStream_t s) : stream(s) {
    keep_pool_memory();
    check_cuda(cudaMallocAsync(reinterpret_cast<void**>(&p), bytes, s), "cudaMallocAsync");
  }
  ~Workspace() { cudaFreeAsync(p, stream); }
  Workspace(const Workspace&) = delete;
  Workspace& operator=(const Workspace&) = delete;
};

// S = fftshift(fft(ifftshift(gradient(J, h)))) for `count` host signals of length n.
void spectrum_host(const double2* J, int n, int count, double h, double2* S, cudaStream_t stream) {
  if (n < 2) throw std::runtime_error("spectrum: a signal needs at least 2 samples");
  if (count < 1) throw std::runtime_error("spectrum: no signals");
  if (!(h > 0.0)) throw std::runtime_error("spectrum: the sample spacing must be positive");
  const size_t total = (size_t)n * count;
  Workspace ws(sizeof(double2) * (3 * total + n), stream);  // J, S, scratch and the table of roots
  double2* dJ = reinterpret_cast<double2*>(ws.p);
  double2 *dS = dJ + total, *dT = dS + total;
  check_cuda(cudaMemcpyAsync(dJ, J, sizeof(double2) * total, cudaMemcpyHostToDevice, stream), "H2D");
  if (hhg::spectrum_device(dJ, n, count, h, dS, dT, stream) < 0)
    throw std::runtime_error("spectrum: launch failed: " + std::string(cudaGetErrorString(cudaGetLastError())));
  check_cuda(cudaMemcpyAsync(S, dS, sizeof(double2) * total, cudaMemcpyDeviceToHost, stream), "D2H");
  check_cuda(cudaStreamSynchronize(stream), "spectrum");
}

int no_device_check(const char* name) {
  int ndev = 0;
  if (cudaGetDeviceCount(&ndev) != cudaSuccess || ndev == 0)
    throw std::runtime_error(std::string(name) + ": no CUDA device (this library has no CPU path)");
  return ndev;
}

}  // namespace

extern "C" {

int HHG_spectrum(const hhg_cdouble* J, int n, int count, double spacing, hhg_cdouble* S) {
  try {
    no_device_check("HHG_spectrum");
    if (!J || !S) throw std::runtime_error("HHG_spectrum: null buffer");
    spectrum_host(reinterpret_cast<const double2*>(J), n, count, spacing, reinterpret_cast<double2*>(S), nullptr);
    return 0;
  } catch (const std::exception& e) {
    hhg::set_thread_error(e.what());
    return -1;
  }
}

int HHG_harmonic_intensities(const hhg_cdouble* S, int n, int count, double tmax_fs, double lambda_nm, int nh,
                             double* I) {
  try {
    no_device_check("HHG_harmonic_intensities");
    if (!S || !I) throw std::runtime_error("HHG_harmonic_intensities: null buffer");
    if (n < 2 || count < 1 || nh < 1) throw std::runtime_error("HHG_harmonic_intensities: empty input");
    if (!(tmax_fs > 0.0) || !(lambda_nm > 0.0))
      throw std::runtime_error("HHG_harmonic_intensities: tmax and lambda must be positive");
    // Only the samples the windows can hold go to the device (a tenth of a 90 fs pulse's for 25 harmonics), gathered on
    // the host where they are at most half of all: 100 000 signals of 8 samples, 6 of them held, took longer to gather.
    int i0 = 0, ni = 0;
    hhg::harmonics_range(n, tmax_fs, lambda_nm, nh, &i0, &ni);
    if (ni == 0) {
      std::fill(I, I + (size_t)count * nh, 0.0);
      return 0;
    }
    const double2* src = reinterpret_cast<const double2*>(S);
    std::vector<double2> part;
    if (ni <= n / 2) {
      part.resize((size_t)count * ni);
      for (int b = 0; b < count; ++b) std::copy_n(src + (size_t)b * n + i0, ni, part.data() + (size_t)b * ni);
      src = part.data();
    } else {
      i0 = 0;
      ni = n;
    }
    const size_t total = (size_t)count * ni;
    cudaStream_t stream = nullptr;
    Workspace ws(sizeof(double2) * total + sizeof(double) * (size_t)count * nh, stream);
    double2* dS = reinterpret_cast<double2*>(ws.p);
    double* dI = reinterpret_cast<double*>(dS + total);
    check_cuda(cudaMemcpyAsync(dS, src, sizeof(double2) * total, cudaMemcpyHostToDevice, stream), "H2D");
    if (hhg::harmonics_device(dS, n, i0, ni, count, tmax_fs, lambda_nm, nh, dI, stream) != 0)
      throw std::runtime_error("HHG_harmonic_intensities: launch failed");
    check_cuda(cudaMemcpyAsync(I, dI, sizeof(double) * (size_t)count * nh, cudaMemcpyDeviceToHost, stream), "D2H");
    check_cuda(cudaStreamSynchronize(stream), "HHG_harmonic_intensities");
    return 0;
  } catch (const std::exception& e) {
    hhg::set_thread_error(e.what());
    return -1;
  }
}

void SWESim_get_spectrum(SWESim* swe, double spacing, hhg_cdouble* sx, hhg_cdouble* sy, hhg_cdouble* sz) {
  try {
    if (!swe) throw std::runtime_error("SWESim_get_spectrum: null SWESim");
    swe->has_err = false;
    if (!swe->ready && !swe->served) throw std::runtime_error("SWESim_get_spectrum: SWESim_init has not succeeded");
    if ((int)swe->Jhist[0].size() < swe->nt)
      throw std::runtime_error("SWESim_get_spectrum: run_simulation has not been called");
    const int n = swe->nt;
    const double h = spacing > 0.0 ? spacing : swe->settings->dt;  // scripts/pol_scan.py:34 uses param["dt"]
    std::vector<double2> J((size_t)3 * n), S((size_t)3 * n);
    for (int a = 0; a < 3; ++a)
      for (int i = 0; i < n; ++i) J[(size_t)a * n + i] = make_double2(swe->Jhist[a][i].real(), swe->Jhist[a][i].imag());
    if (swe->device >= 0) check_cuda(cudaSetDevice(swe->device), "cudaSetDevice");
    spectrum_host(J.data(), n, 3, h, S.data(), swe->ready ? swe->stream : nullptr);
    hhg_cdouble* out[3] = {sx, sy, sz};
    for (int a = 0; a < 3; ++a)
      if (out[a])
        for (int i = 0; i < n; ++i) out[a][i] = hhg_cdouble{S[(size_t)a * n + i].x, S[(size_t)a * n + i].y};
  } catch (const std::exception& e) {
    hhg::set_thread_error(e.what());
    if (swe) {
      swe->err = e.what();
      swe->has_err = true;
    }
  }
}

}  // extern "C"
