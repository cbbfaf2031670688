// les_grad_xy_noalloc: horizontal spectral derivatives of a device field
// with every intermediate in one fixed, file-scope device buffer.
//
// The arithmetic of les_grad_velocity_filt (x r2c FFT with the 1/(nx*ny)
// scaling, y pass with the ik multiplications and the Nyquist kill, inverse x
// transforms of the filtered field and both derivatives): in one launch, a CTA
// per level, where a plane fits into shared memory, else in three passes,
// launched on caller-owned device pointers.  It exists for callers that must
// not change the device memory footprint and so cannot allocate: an in-situ
// analysis hook called from a coupled model whose device memory is fully
// committed to its own fields, or code running in a process where a caching
// allocator holds the free memory, so that a cudaMalloc can fail or force the
// cache to be released.  Nothing here allocates: no cudaMalloc/cudaFree, no
// CUDA events, no host containers, no library that allocates.
//
// Scratch: g_noalloc_scratch (LES_NOALLOC_SCRATCH_BYTES) has room for, 256-byte
// aligned, the wavenumber tables kkx, kky [ny][nx/2+1], the twiddle tables of
// nx and ny, and three spectra [nlev][ny][nx/2+1] (complex FP64): what a call
// may need, and what decides whether its size is accepted; the three-pass form
// uses two of the spectra, the plane form at most one and no tables.  Every
// call writes what it reads there first, so nothing has to start at zero.  All
// calls in the process share the buffer of their device: two calls in flight
// at the same time on one device (different streams or host threads) race on
// it.
#include <atomic>
#include <cmath>
#include <cstdint>
#include <cstdio>
#include <cstring>

#include "../../include/lesgpu.h"
#include "launch.cuh"

namespace les {
namespace {

constexpr size_t kScratchBytes = LES_NOALLOC_SCRATCH_BYTES;
__device__ __align__(256) unsigned char g_noalloc_scratch[kScratchBytes];
__device__ unsigned g_noalloc_status;  // sticky status bits (les_noalloc_status)

constexpr int kMaxDevices = 64;
// per device, set by the first call on it (the scratch last)
std::atomic<unsigned char*> g_scratch_addr[kMaxDevices] = {};
std::atomic<unsigned*> g_status_addr[kMaxDevices] = {};

constexpr size_t align256(size_t b) { return (b + 255) / 256 * 256; }

struct ScratchLayout {
  size_t kkx, kky, twx, twy, spec[3], total;
};
ScratchLayout scratch_layout(int nx, int ny, int nlev) {
  const size_t lhx = size_t(nx / 2 + 1);
  const size_t tab = align256(sizeof(double) * size_t(ny) * lhx);
  const size_t spec = align256(sizeof(cplx<double>) * size_t(nlev) * size_t(ny) * lhx);
  ScratchLayout L;
  size_t o = 0;
  L.kkx = o;
  o += tab;
  L.kky = o;
  o += tab;
  L.twx = o;
  o += align256(sizeof(cplx<double>) * size_t(nx));
  L.twy = o;
  o += align256(sizeof(cplx<double>) * size_t(ny));
  for (int i = 0; i < 3; ++i) {
    L.spec[i] = o;
    o += spec;
  }
  L.total = o;
  return L;
}

// wavenumber tables (fft_engine.f90:127-143, Nyquist row and column zeroed)
// and the exp(-2 pi i m / n) twiddle tables, computed on the device
__global__ void k_noalloc_tables(double* kkx, double* kky, cplx<double>* twx, cplx<double>* twy, int nx, int ny,
                                 double lx, double ly) {
  dep_wait();
  const int lhx = nx / 2 + 1, lhy = ny / 2 + 1;
  const double pi = 3.14159265358979323846;
  const long n = (long)ny * lhx;
  for (long q = blockIdx.x * (long)blockDim.x + threadIdx.x; q < n; q += (long)gridDim.x * blockDim.x) {
    const int i = int(q % lhx), j = int(q / lhx);
    double kx = double(i);
    double ky = double(((j + ny / 2) % ny) - ny / 2);
    if (i == lhx - 1 || j == lhy - 1) {
      kx = 0.0;
      ky = 0.0;
    }
    kkx[q] = 2.0 * pi / lx * kx;
    kky[q] = 2.0 * pi / ly * ky;
  }
  for (long m = blockIdx.x * (long)blockDim.x + threadIdx.x; m < nx + ny; m += (long)gridDim.x * blockDim.x) {
    const bool isx = m < nx;
    const int len = isx ? nx : ny;
    const int mm = int(isx ? m : m - nx);
    double s, c;
    sincospi(-2.0 * double(mm) / double(len), &s, &c);
    (isx ? twx : twy)[mm] = cplx<double>{c, s};
  }
}

// ---- whole planes in shared memory ----
// A level whose spectrum fits into shared memory is differentiated by one CTA
// in one launch: rows in by bulk copies, x transforms in place, the columns'
// y transforms there and (F and i ky F) back without leaving registers, the x
// inverses out; i kx F is formed as the rows are read.  The spectrum of d/dy
// waits in a second array (two) or, where that does not fit, in the scratch
// buffer, which L2 holds.  The twiddles and wavenumbers are computed by the
// CTA, so the call needs no table launch.  Small planes are bound by launches
// and latency, which the four launches of the three-pass form pay four times,
// larger ones by shared memory, ~25 accesses per value.  us, three passes / this:
// 16 x 16 x 100 26.6 / 6.2, 64 x 64 x 148 41 / 12.3, 96 x 64 x 100 41 / 16.4, 128
// x 64 x 159 (two waves) 61 / 34, 128 x 128 x 79 54 / 37; with dependent launches
// 16.4 / 4.0, 39 / 10.3, 33 / 13.8, 51 / 31.8 and 45 / 34.4.
template <int NX, int NY>
struct PlaneGrad {
  static constexpr int M = NX / 2;
  static constexpr int SLX = slot_stride(M, 16);
  static constexpr int need = SLX > M + 1 ? SLX : M + 1;
  // row stride in complex values: the row's slot and the M + 1 modes, 4 modulo
  // 8, so that four columns of two neighbouring rows, and four values of two
  // neighbouring rows, fall on eight different 16-byte banks
  static constexpr int RS = (need + 3) / 8 * 8 + 4;
  static constexpr int lanes_x = NY * Geo<M>::T, lanes_y = M * Geo<NY>::T;
  static constexpr int want = ((lanes_x > lanes_y ? lanes_x : lanes_y) + 31) / 32 * 32;
  // a thread holds two transforms of up to 24 values: all 255 registers
  static constexpr int threads = want < 64 ? 64 : (want > 256 ? 256 : want);
  static constexpr size_t array = sizeof(cplx<double>) * (size_t)NY * RS;
  static constexpr size_t tables = sizeof(cplx<double>) * (NX + NY + twm_len(M, false) + twm_len(M, true) +
                                                           twm_len(NY, false) + twm_len(NY, true)) + 16;
  static constexpr size_t cap = 227 * 1024;
  static constexpr bool two = 2 * array + tables <= cap;
  static constexpr size_t smem = (two ? 2 : 1) * array + tables;
  static_assert(smem <= cap, "plane beyond shared memory");
  // Levels from which the plane form is the faster one.  One wave of CTAs takes
  // the same time at any number of levels, three passes of few levels a launch's
  // time each: planes of up to 8192 points and 192 x 64 win at any number (us,
  // plane / three passes: 128 x 64 x 1 16.0 / 20.5, 64 x 128 x 1 17.4 / 18.5, 192
  // x 64 x 2 25.7 / 25.7), the larger ones where three passes grow past them: 128
  // x 128 x 42 34.3 / 30.8, x 44 34.3 / 34.8; 256 x 64 x 29 29.0 / 26.7, x 30 29.0
  // / 30.2; 96 x 128 x 28 25.4 / 24.6, x 30 25.4 / 25.5.
  static constexpr int from = NX * NY <= 8192 || NX == 192 ? 1 : NX == 128 ? 44 : 30;
};

template <int NX, int NY>
__global__ void __launch_bounds__(PlaneGrad<NX, NY>::threads)
    k_grad_plane(double* f, double* dfdx, double* dfdy, cplx<double>* scratch, unsigned* status, double lx, double ly) {
  using G = PlaneGrad<NX, NY>;
  constexpr bool TWO = G::two;
  using C = cplx<double>;
  constexpr int M = G::M, RS = G::RS, TH = G::threads;
  constexpr int TX = Geo<M>::T, EX = Geo<M>::E, TY = Geo<NY>::T, EY = Geo<NY>::E;
  constexpr int XI_ = Layout<M, false>::in, XO = Layout<M, false>::out;
  constexpr int VI = Layout<M, true>::in, VO = Layout<M, true>::out;
  constexpr int YI = Layout<NY, false>::in, YO = Layout<NY, false>::out;
  constexpr int ZI = Layout<NY, true>::in, ZO = Layout<NY, true>::out;
  static_assert(ZI == YO, "the inverse y transform takes the forward one's registers");
  // exchanges of a column: lanes of a quarter warp lie on two rows only where
  // a column has eight lanes (NY = 128: radices 16, 8 and 8, 16)
  using SlotF = ColSlot<double, TY == 8 ? 4 : -1>;
  using SlotI = ColSlot<double, TY == 8 ? 3 : -1>;
  static_assert(TY <= 4 || NY == 128, "exchange swizzle of a column");
  extern __shared__ __align__(16) unsigned char smem_raw[];
  C* A = reinterpret_cast<C*>(smem_raw);
  C* B = A + (TWO ? (long)NY * RS : 0);
  C* twx = B + (long)NY * RS;  // exp(-2 pi i m / NX)
  C* twy = twx + NX;
  C* mxf = twy + NY;  // twiddle matrices: x forward, x inverse, y forward, y inverse
  C* mxi = mxf + Twm<M, false>::len;
  C* myf = mxi + Twm<M, true>::len;
  C* myi = myf + Twm<NY, false>::len;
  uint64_t* bar = reinterpret_cast<uint64_t*>(myi + Twm<NY, true>::len);
  const int tid = threadIdx.x;
  const long plane = (long)blockIdx.x * NY * NX;
  if (tid < 32) {
    if (tid == 0) {
      tc::mbar_init(bar, 1);
      tc::fence_mbar_init();
      mbar_expect_tx(bar, unsigned(NY * NX * sizeof(double)));
    }
    dep_wait();
    __syncwarp();
    for (int r = tid; r < NY; r += 32) bulk_g2s(A + r * RS, f + plane + (long)r * NX, unsigned(NX * sizeof(double)), bar);
  }
  for (int m = tid; m < NX + NY; m += TH) {
    const bool isx = m < NX;
    double s, c;
    if (isx) sincospi(-2.0 * double(m) / double(NX), &s, &c);
    else sincospi(-2.0 * double(m - NX) / double(NY), &s, &c);
    twx[m] = C{c, s};  // twy follows twx
  }
  __syncthreads();
  twm_build<double, M, false, 2>(twx, mxf, tid, TH);
  twm_build<double, M, true, 2>(twx, mxi, tid, TH);
  twm_build<double, NY, false>(twy, myf, tid, TH);
  twm_build<double, NY, true>(twy, myi, tid, TH);
  dep_wait();
  const bool late = !tc::mbar_wait(bar, 0);
  if (__syncthreads_or(late)) {  // as in the spectral passes: record it, a last bounded wait, leave
    if (tid == 0) atomicOr(status, unsigned(ST_COPY_WAIT));
    tc::mbar_wait(bar, 0);
    return;
  }
  const double pi = 3.14159265358979323846;
  const double kx1 = 2.0 * pi / lx, ky1 = 2.0 * pi / ly;
  // rows: body(row, lane of it, whether it is one).  (A warp reaches past the
  // last row only where a row is one lane, whose transform exchanges nothing.)
  static_assert(TX == 1 || NY % (32 / TX) == 0, "lanes past the last row must not exchange");
  auto rows = [&](auto body) {
    for (int r0 = 0; r0 < NY; r0 += TH / TX) {
      const int r = r0 + tid / TX;
      if (r0 + (tid & ~31) / TX >= NY) break;  // whole warp beyond the rows
      body(r < NY ? r : 0, tid % TX, r < NY);
    }
  };
  // x: r2c in place; mode M, the Nyquist bin, is killed
  rows([&](int r, int t, bool live) {
    const double c0 = 1.0 / (double(NX) * double(NY));
    C* row = A + r * RS;
    C v[EX];
#pragma unroll
    for (int g = 0; g < EX / XI_; ++g)
#pragma unroll
      for (int q = 0; q < XI_; ++q) v[g * XI_ + q] = c_scl(row[t + TX * g + q * (M / XI_)], c0);
    reg_fft<double, M, false>(v, row, t, mxf);
    __syncwarp();
    if (live) {
#pragma unroll
      for (int g = 0; g < EX / XO; ++g)
#pragma unroll
        for (int q = 0; q < XO; ++q) row[t + TX * g + q * (M / XO)] = v[g * XO + q];
    }
    __syncwarp();
    if (live)
      for (int k = t; k <= M / 2; k += TX) {  // modes k and M - k need the same two values
        const int k2 = k == 0 ? 0 : M - k;
        const C zk = row[k], zm = row[k2];
        row[k] = r2c_split(zk, zm, c_scl(twx[k], 0.5));
        if (k2 > k) row[k2] = r2c_split(zm, zk, c_scl(twx[k2], 0.5));
      }
    __syncwarp();  // before the next row's exchange of this warp
  });
  __syncthreads();
  // y: the columns of a warp vary fastest, so that the lanes of a
  // shared-memory wavefront walk along a row.  The Nyquist row is killed; F
  // comes back in place, i ky F in B or the scratch buffer.
  constexpr int CW = 32 / TY;  // columns per warp
  C* const ys = TWO ? nullptr : scratch + (long)blockIdx.x * NY * M;
  for (int c0 = 0; c0 < M; c0 += TH / TY) {
    const int cw = c0 + (tid >> 5) * CW;
    if (cw >= M) break;  // whole warp
    const int t = (tid & 31) / CW, cc = cw + (tid & 31) % CW;
    const bool live = cc < M;
    // lanes past the last column read it and exchange in column M, which
    // nothing else uses
    const int c = live ? cc : M - 1, cx = live ? cc : M;
    C v[EY], w[EY];
#pragma unroll
    for (int g = 0; g < EY / YI; ++g)
#pragma unroll
      for (int q = 0; q < YI; ++q) v[g * YI + q] = A[(t + TY * g + q * (NY / YI)) * RS + c];
    reg_fft<double, NY, false>(v, SlotF{A + cx, RS}, t, myf);
#pragma unroll
    for (int g = 0; g < EY / YO; ++g)
#pragma unroll
      for (int q = 0; q < YO; ++q) {
        const int ky = t + TY * g + q * (NY / YO);
        C& F = v[g * YO + q];
        if (ky == NY / 2) F = C{0.0, 0.0};
        w[g * YO + q] = ik_mul(ky1 * double(ky < NY / 2 ? ky : ky - NY), F);
      }
    reg_fft<double, NY, true>(w, SlotI{B + cx, RS}, t, myi);
    if constexpr (!TWO) {
      if (live) {
#pragma unroll
        for (int g = 0; g < EY / ZO; ++g)
#pragma unroll
          for (int q = 0; q < ZO; ++q) ys[(t + TY * g + q * (NY / ZO)) * M + c] = w[g * ZO + q];
      }
    } else {
      __syncwarp();
      if (live) {
#pragma unroll
        for (int g = 0; g < EY / ZO; ++g)
#pragma unroll
          for (int q = 0; q < ZO; ++q) B[(t + TY * g + q * (NY / ZO)) * RS + c] = w[g * ZO + q];
      }
    }
    reg_fft<double, NY, true>(v, SlotI{A + cx, RS}, t, myi);
    __syncwarp();
    if (live) {
#pragma unroll
      for (int g = 0; g < EY / ZO; ++g)
#pragma unroll
        for (int q = 0; q < ZO; ++q) A[(t + TY * g + q * (NY / ZO)) * RS + c] = v[g * ZO + q];
    }
  }
  __syncthreads();
  // x: c2r of a row out of A (f, df/dx) and of i ky F (df/dy)
  auto store = [&](const C* v, double* o, int r, int t) {
#pragma unroll
    for (int g = 0; g < EX / VO; ++g)
#pragma unroll
      for (int q = 0; q < VO; ++q)
        *reinterpret_cast<C*>(o + plane + (long)r * NX + 2 * (t + TX * g + q * (M / VO))) = v[g * VO + q];
  };
  rows([&](int r, int t, bool live) {
    C* row = A + r * RS;
    C v[EX], w[EX];
#pragma unroll
    for (int g = 0; g < EX / VI; ++g)
#pragma unroll
      for (int q = 0; q < VI; ++q) {
        const int m = t + TX * g + q * (M / VI);
        C xk = row[m], xm = m == 0 ? C{0.0, 0.0} : row[M - m];
        w[g * VI + q] = c2r_split(ik_mul(kx1 * double(m), xk), ik_mul(kx1 * double(M - m), xm), twx[m]);
        if (m == 0) xk.y = 0.0;
        v[g * VI + q] = c2r_split(xk, xm, twx[m]);
      }
    reg_fft<double, M, true>(v, row, t, mxi);
    if (live) store(v, f, r, t);
    reg_fft<double, M, true>(w, row, t, mxi);
    if (live) store(w, dfdx, r, t);
    const C* yr = TWO ? B + r * RS : ys + (long)r * M;
#pragma unroll
    for (int g = 0; g < EX / VI; ++g)
#pragma unroll
      for (int q = 0; q < VI; ++q) {
        const int m = t + TX * g + q * (M / VI);
        C xk = yr[m], xm = m == 0 ? C{0.0, 0.0} : yr[M - m];
        if (m == 0) xk.y = 0.0;
        v[g * VI + q] = c2r_split(xk, xm, twx[m]);
      }
    reg_fft<double, M, true>(v, row, t, mxi);
    if (live) store(v, dfdy, r, t);
    __syncwarp();
  });
}

// the plane kernel of a grid (nullptr: none)
struct PlaneKernel {
  void (*run)(double*, double*, double*, cplx<double>*, unsigned*, double, double) = nullptr;
  int threads = 0;
  size_t smem = 0;
  int from = 0;
};
template <int NX, int NY>
PlaneKernel plane_kernel_of() {
  using G = PlaneGrad<NX, NY>;
  return {k_grad_plane<NX, NY>, G::threads, G::smem, G::from};
}
template <int NX>
PlaneKernel plane_kernel_ny(int ny) {
  switch (ny) {
    case 16: return plane_kernel_of<NX, 16>();
    case 32: return plane_kernel_of<NX, 32>();
    case 64: return plane_kernel_of<NX, 64>();
    case 128:
      if constexpr (NX < 192) return plane_kernel_of<NX, 128>();  // beyond: more than one array
      else return {};
    default: return {};
  }
}
PlaneKernel plane_kernel(int nx, int ny) {
  switch (nx) {
    case 16: return plane_kernel_ny<16>(ny);
    case 24: return plane_kernel_ny<24>(ny);
    case 32: return plane_kernel_ny<32>(ny);
    case 48: return plane_kernel_ny<48>(ny);
    case 64: return plane_kernel_ny<64>(ny);
    case 96: return plane_kernel_ny<96>(ny);
    case 128: return plane_kernel_ny<128>(ny);
    case 192: return plane_kernel_ny<192>(ny);
    case 256: return plane_kernel_ny<256>(ny);
    default: return {};
  }
}

// whether a call of nlev levels takes the plane form
bool plane_form(const PlaneKernel& k, int nlev) { return k.run && nlev >= k.from; }

// address of this device's scratch buffer; the first call on a device does
// the setup (symbol address, kernel shared-memory attributes)
int scratch_for_device(unsigned char** out) {
  int dev = -1;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) throw CudaError(LES_ERR_INVALID, std::string("cudaGetDevice: ") + cudaGetErrorString(e));
  if (dev < 0 || dev >= kMaxDevices) throw CudaError(LES_ERR_INVALID, "device ordinal out of range");
  unsigned char* addr = g_scratch_addr[dev].load();
  if (!addr) {
    void* p = nullptr;
    e = cudaGetSymbolAddress(&p, g_noalloc_scratch);
    if (e != cudaSuccess)
      throw CudaError(LES_ERR_INVALID, std::string("cudaGetSymbolAddress: ") + cudaGetErrorString(e));
    for (int nx : {16, 24, 32, 48, 64, 96, 128, 192, 256, 384, 512, 768})
      for (int ny : {16, 32, 64, 128, 256, 512}) init_spectral_attributes<double>(SU_GRAD, nx, ny);
    for (int nx : {16, 24, 32, 48, 64, 96, 128, 192, 256})
      for (int ny : {16, 32, 64, 128}) {
        if (const PlaneKernel k = plane_kernel(nx, ny); k.run)
          LES_CUDA(cudaFuncSetAttribute((const void*)k.run, cudaFuncAttributeMaxDynamicSharedMemorySize, int(k.smem)));
      }
    addr = static_cast<unsigned char*>(p);
    e = cudaGetSymbolAddress(&p, g_noalloc_status);
    if (e != cudaSuccess)
      throw CudaError(LES_ERR_INVALID, std::string("cudaGetSymbolAddress: ") + cudaGetErrorString(e));
    g_status_addr[dev].store(static_cast<unsigned*>(p));
    g_scratch_addr[dev].store(addr);
  }
  *out = addr;
  return dev;
}

}  // namespace
}  // namespace les

namespace {
thread_local char g_noalloc_error[256];
}

extern "C" const char* les_noalloc_last_error(void) { return g_noalloc_error; }

extern "C" int les_noalloc_status(unsigned* bits, void* stream) {
  using namespace les;
  g_noalloc_error[0] = '\0';
  auto fail = [](const char* msg) {
    std::snprintf(g_noalloc_error, sizeof(g_noalloc_error), "%s", msg);
    return LES_ERR_INVALID;
  };
  if (!bits) return fail("les_noalloc_status: null argument");
  *bits = 0;
  int dev = -1;
  cudaError_t e = cudaGetDevice(&dev);
  if (e == cudaSuccess && (dev < 0 || dev >= kMaxDevices)) return fail("device ordinal out of range");
  if (e == cudaSuccess) {
    unsigned* const word = g_status_addr[dev].load();
    if (!word) return LES_OK;  // no call on this device yet
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    e = cudaMemcpyAsync(bits, word, sizeof(unsigned), cudaMemcpyDeviceToHost, st);
    if (e == cudaSuccess) e = cudaMemsetAsync(word, 0, sizeof(unsigned), st);
    if (e == cudaSuccess) e = cudaStreamSynchronize(st);
  }
  if (e != cudaSuccess) {
    std::snprintf(g_noalloc_error, sizeof(g_noalloc_error), "%s", cuda_error_text("les_noalloc_status", e).c_str());
    return cuda_status_code(e);
  }
  return LES_OK;
}

extern "C" int les_grad_xy_noalloc(double* f, double* dfdx, double* dfdy, int nx, int ny, int nlev, double lx,
                                   double ly, void* stream) {
  using namespace les;
  g_noalloc_error[0] = '\0';
  auto fail = [](int code, const char* msg) {
    std::snprintf(g_noalloc_error, sizeof(g_noalloc_error), "%s", msg);
    return code;
  };
  if (!f || !dfdx || !dfdy) return fail(LES_ERR_INVALID, "les_grad_xy_noalloc: null field pointer");
  if ((reinterpret_cast<uintptr_t>(f) | reinterpret_cast<uintptr_t>(dfdx) | reinterpret_cast<uintptr_t>(dfdy)) & 15u)
    return fail(LES_ERR_INVALID, "les_grad_xy_noalloc: field pointers must be 16-byte aligned");
  if (nx <= 0 || ny <= 0 || nlev <= 0 || !(lx > 0) || !(ly > 0))
    return fail(LES_ERR_INVALID, "les_grad_xy_noalloc: invalid grid or domain size");
  // x: every length with a register FFT plan; y: the lengths with an
  // equal-length y pass (powers of two), checked before anything is queued
  const bool ny_ok = ny == 16 || ny == 32 || ny == 64 || ny == 128 || ny == 256 || ny == 512;
  if (!supported_length(nx) || !ny_ok)
    return fail(LES_ERR_INVALID,
                "les_grad_xy_noalloc: nx must be one of 16 24 32 48 64 96 128 192 256 384 512 768 and ny one of "
                "16 32 64 128 256 512");
  const ScratchLayout L = scratch_layout(nx, ny, nlev);
  if (L.total > kScratchBytes) {
    std::snprintf(g_noalloc_error, sizeof(g_noalloc_error),
                  "les_grad_xy_noalloc: %dx%dx%d needs %zu bytes of scratch, the static buffer holds %zu "
                  "(LES_NOALLOC_SCRATCH_BYTES)",
                  nx, ny, nlev, L.total, kScratchBytes);
    return LES_ERR_INVALID;
  }
  // launches here are not observed by a solver's profiling hook; the hook is
  // per host thread, so only states profiled on the calling thread are
  // affected, and only for the duration of this call
  LaunchHook* saved = g_hook;
  g_hook = nullptr;
  int rc = LES_OK;
  try {
    unsigned char* base = nullptr;
    unsigned* const status = g_status_addr[scratch_for_device(&base)].load();
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    if (const PlaneKernel pk = plane_kernel(nx, ny); plane_form(pk, nlev)) {
      auto* ys = reinterpret_cast<cplx<double>*>(base + L.spec[0]);
      launch_dep(pk.run, nlev, pk.threads, pk.smem, st, f, dfdx, dfdy, ys, status, lx, ly);
      LES_CHECK_LAUNCH();
      g_hook = saved;
      return rc;
    }
    double* kkx = reinterpret_cast<double*>(base + L.kkx);
    double* kky = reinterpret_cast<double*>(base + L.kky);
    auto* twx = reinterpret_cast<cplx<double>*>(base + L.twx);
    auto* twy = reinterpret_cast<cplx<double>*>(base + L.twy);
    cplx<double>* sp[2];
    for (int i = 0; i < 2; ++i) sp[i] = reinterpret_cast<cplx<double>*>(base + L.spec[i]);
    const int lhx = nx / 2 + 1;
    launch_dep(k_noalloc_tables, 64, 256, 0, st, kkx, kky, twx, twy, nx, ny, lx, ly);
    LES_CHECK_LAUNCH();

    XFArgs<double> a;
    std::memset(&a, 0, sizeof(a));
    a.op = XF_SCALE;
    a.status = status;
    a.nf = 1;
    a.rows_pp = ny;
    a.nrows = (long)nlev * ny;
    a.nk = lhx;
    a.nz = nlev - 2;
    a.in_pstride = (long)ny * nx;
    a.out_pstride = (long)ny * lhx;
    a.tw = twx;
    a.c0 = 1.0 / double(nx * ny);
    a.in[0] = f;
    a.out[0] = sp[0];
    launch_xfwd<double>(nx, a, st);

    YPArgs<double> b;
    std::memset(&b, 0, sizeof(b));
    b.dep = 1;  // (the x pass above has waited for the tables)
    b.op = YP_GRADY;  // F and i ky F; the x inverse forms i kx F from the staged F row
    b.nin = 1;
    b.nout = 2;
    b.ncols = lhx;
    b.nk_in = lhx;
    b.nk_out = lhx;
    b.in_pstride = (long)ny * lhx;
    b.out_pstride = (long)ny * lhx;
    b.nxh = nx / 2;
    b.lhx = lhx;
    b.kkx = kkx;
    b.kky = kky;
    b.tw_in = twy;
    b.tw_out = twy;
    b.in[0] = sp[0];
    b.out[0] = sp[0];
    b.out[1] = sp[1];
    launch_ypass<double>(ny, ny, b, nlev, 1, st);

    XIArgs<double> c;
    std::memset(&c, 0, sizeof(c));
    c.dep = 1;
    c.op = XI_STORE;
    c.status = status;
    c.nin = 3;
    c.rows_pp = ny;
    c.nrows = (long)nlev * ny;
    c.nk = lhx;
    c.nz = nlev - 2;
    c.in_pstride = (long)ny * lhx;
    c.out_pstride = (long)ny * nx;
    c.tw = twx;
    c.nstage = 2;
    c.kxr = kkx;
    c.in[0] = sp[0];
    c.in[1] = sp[1];
    double* const outs[3] = {f, dfdx, dfdy};
    for (int q = 0; q < 3; ++q) {
      c.src[q] = q == 2 ? 1 : 0;
      c.dx[q] = q == 1;
      c.out[q] = outs[q];
      c.lo[q] = 0;
      c.hi[q] = nlev - 1;
    }
    launch_xinv<double>(nx, c, st);
  } catch (const CudaError& e) {
    std::snprintf(g_noalloc_error, sizeof(g_noalloc_error), "%s", e.what());
    rc = e.code ? e.code : LES_ERR_INVALID;
  } catch (const std::exception& e) {
    std::snprintf(g_noalloc_error, sizeof(g_noalloc_error), "%s", e.what());
    rc = LES_ERR_INVALID;
  }
  g_hook = saved;
  return rc;
}
