// Launch helpers of the spectral passes (occupancy and register caches,
// FFT lane counts, supported lengths) and the per-device shared-memory
// attributes of their kernels.  The kernels are instantiated and launched
// in spectral_xfwd.cu, spectral_xinv.cu and spectral_ypass.cu.
#include "spectral_launch.cuh"
#include <atomic>
#include <mutex>

#include "launch.cuh"
#include "launch_cache.hpp"

namespace les {

thread_local LaunchHook* g_hook = nullptr;

// SMs of the current device
int sm_count() {
  static std::atomic<int> count[256] = {};
  int dev = 0;
  LES_CUDA(cudaGetDevice(&dev));
  if (dev < 0 || dev >= 256) throw CudaError(1, "device ordinal out of range");
  int n = count[dev].load(std::memory_order_relaxed);
  if (n == 0) {
    LES_CUDA(cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev));
    n = std::max(1, n);
    count[dev].store(n, std::memory_order_relaxed);
  }
  return n;
}

// CTAs of `kern` resident on the current device at once
int resident_ctas(const void* kern, int threads, size_t smem) {
  static std::mutex mu;
  static LaunchCache<int, RESIDENT_CACHE> cache;
  int dev = 0;
  LES_CUDA(cudaGetDevice(&dev));
  std::lock_guard<std::mutex> lock(mu);
  if (const int* n = cache.find(dev, kern, threads, smem)) return *n;
  int per_sm = 0;
  LES_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, threads, smem));
  const int n = std::max(1, per_sm) * sm_count();
  cache.put(dev, kern, threads, smem, n);
  return n;
}

// registers per thread and the largest CTA of `kern` on the current device
KernelLimits kernel_limits(const void* kern) {
  static std::mutex mu;
  static LaunchCache<KernelLimits, LIMITS_CACHE> cache;
  int dev = 0;
  LES_CUDA(cudaGetDevice(&dev));
  std::lock_guard<std::mutex> lock(mu);
  if (const KernelLimits* l = cache.find(dev, kern, 0, 0)) return *l;
  cudaFuncAttributes fa;
  LES_CUDA(cudaFuncGetAttributes(&fa, kern));
  const KernelLimits lim{fa.numRegs, fa.maxThreadsPerBlock};
  cache.put(dev, kern, 0, 0, lim);
  return lim;
}

// lanes per sequence of the register FFT of length n (fft2.cuh plans)
int lanes(int n) {
  switch (n) {
    case 8: return Geo<8>::T;
    case 12: return Geo<12>::T;
    case 16: return Geo<16>::T;
    case 24: return Geo<24>::T;
    case 32: return Geo<32>::T;
    case 48: return Geo<48>::T;
    case 64: return Geo<64>::T;
    case 96: return Geo<96>::T;
    case 128: return Geo<128>::T;
    case 192: return Geo<192>::T;
    case 256: return Geo<256>::T;
    case 384: return Geo<384>::T;
    case 512: return Geo<512>::T;
    case 768: return Geo<768>::T;
    default: throw CudaError(1, "no FFT plan for length " + std::to_string(n));
  }
}
int pad_seqs(int nseq, int M) {
  const int spw = 32 / lanes(M);
  return ((nseq + spw - 1) / spw) * spw;
}

bool supported_length(int n) {
  switch (n) {
    case 16: case 24: case 32: case 48: case 64: case 96: case 128:
    case 192: case 256: case 384: case 512: case 768:
      return true;
    default:
      return false;
  }
}

namespace {
int length_index(int n) {  // of a supported length
  int i = 0;
#define LI(N) if (n == N) return i; ++i;
  LES_LENGTHS(LI)
#undef LI
  throw CudaError(1, "no FFT plan for length " + std::to_string(n));
}
// done already: type, device, use, direction, length (not inside the template,
// whose statics two copies of the library in one process would share)
std::mutex g_init_mutex;
bool g_init_done[2][256][3][2][12];
}  // namespace

// cudaFuncSetAttribute applies to the current device only, and loads the
// kernel: done for the kernels of a grid, once per device ordinal (fixed table
// and a mutex, no heap allocation), so states on several devices of one
// process, and threads creating them at once, all launch with the
// shared-memory limit raised.  (Loading all 264 kernels of every length, type
// and class took a process's first state 74 ms; its own twenty or thirty 43 to
// 58 ms, 23 to 30 ms with uncompressed device code, see build.py.)
template <typename T>
void init_spectral_attributes(SpectralUse use, int nx, int ny) {
  int dev = 0;
  LES_CUDA(cudaGetDevice(&dev));
  if (dev < 0 || dev >= 256) throw CudaError(1, "device ordinal out of range");
  auto& done = g_init_done[std::is_same<T, double>::value][dev][use];
  bool& dx = done[0][length_index(nx)];
  bool& dy = done[1][length_index(ny)];
  std::lock_guard<std::mutex> lock(g_init_mutex);
  if (!dx) {
    set_attrs_xfwd<T>(use, nx);
    if (use != SU_PRESSURE) set_attrs_xinv<T>(use, nx);
    if (use == SU_STATE) {  // the padded products' length
      set_attrs_xfwd<T>(use, 3 * nx / 2);
      set_attrs_xinv<T>(use, 3 * nx / 2);
    }
    dx = true;
  }
  if (!dy) {
    set_attrs_ypass<T>(use, ny);
    dy = true;
  }
}
template void init_spectral_attributes<float>(SpectralUse, int, int);
template void init_spectral_attributes<double>(SpectralUse, int, int);

}  // namespace les
