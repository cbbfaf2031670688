// Instantiation and launch of the y passes (k_ypass) for every supported
// length pair.
#include "spectral_launch.cuh"

#include "launch.cuh"

namespace les {

// the y-pass kernel of a length pair and class (nullptr: none)
template <typename T, int A, int B>
static void (*ypass_kernel(int cls))(YPArgs<T>) {
  if constexpr (A == B) {
    switch (cls) {
      case YC_FWD: return k_ypass<T, A, A, YC_FWD>;
      case YC_GRADY: return k_ypass<T, A, A, YC_GRADY>;
      case YC_PGRAD: return k_ypass<T, A, A, YC_PGRAD>;
      case YC_FILTER: return k_ypass<T, A, A, YC_FILTER>;
      case YC_DIV2: return k_ypass<T, A, A, YC_DIV2>;
      default: break;
    }
  } else if (cls != YC_OTHER) {
    return nullptr;
  }
  return k_ypass<T, A, B, YC_OTHER>;
}

template <typename T>
void launch_ypass(int NY, int NYO, YPArgs<T> a, int nplanes, int ngroups, cudaStream_t st) {
  if (a.ipitch == 0) a.ipitch = a.nk_in;
  if (a.opitch == 0) a.opitch = a.nk_out;
  if (a.opitch1 == 0) a.opitch1 = a.nk_out1;
  const int TL = lanes(NY);
  if (lanes(NYO) != TL) throw CudaError(1, "ypass: length pair with different lane counts");
  // column stride of the shared stages: the load and store loops run c
  // (column) fastest and 32/C rows per warp, so a stride congruent to 32/C
  // modulo the complex values per 128-byte wavefront spreads a warp evenly
  // over the banks; room for the padded exchange layout of the longer of the
  // two transforms (the inverse runs in the first input row of each column)
  const int W = 128 / int(sizeof(cplx<T>));
  const int NL = std::max(NY, NYO);
  auto stride = [&](int C) {
    const int target = (32 / C) % W;
    const int base = NL + NL / 16;
    return base + ((target - base % W) % W + W) % W;
  };
  auto smem_for = [&](int C, int ns) {  // twiddle matrices, the ky row, ns stages of nin rows per column
    return sizeof(cplx<T>) * (twm_len(NY, false) + twm_len(NYO, true) + (size_t)C * ns * a.nin * stride(C)) +
           sizeof(T) * ((NY + 3) & ~3);
  };
  const int key = NY * 10000 + NYO;
  const int cls = yp_class(a.op);
  void (*kern)(YPArgs<T>) = nullptr;
  switch (key) {
#define YP_CASE(A, B) \
  case A * 10000 + B: kern = ypass_kernel<T, A, B>(cls); break;
    YP_CASE(16, 16) YP_CASE(32, 32) YP_CASE(64, 64) YP_CASE(128, 128) YP_CASE(256, 256) YP_CASE(512, 512)
    YP_CASE(16, 24) YP_CASE(32, 48) YP_CASE(64, 96) YP_CASE(128, 192) YP_CASE(256, 384) YP_CASE(512, 768)
    YP_CASE(24, 16) YP_CASE(48, 32) YP_CASE(96, 64) YP_CASE(192, 128) YP_CASE(384, 256) YP_CASE(768, 512)
#undef YP_CASE
    default:
      throw CudaError(1, "ypass: unsupported length pair " + std::to_string(NY) + "->" + std::to_string(NYO));
  }
  if (!kern) throw CudaError(1, "ypass: this op keeps the length");
  // columns per CTA (C * TL threads, at least a warp) and input stages: the
  // most busy warps per SM -- resident CTAs (shared memory, registers,
  // threads) times the warps whose columns exist; on a tie two stages (the
  // loads of the next item overlap this one), then the CTA size nearest 128
  // threads (measured at 256^3: 128-thread CTAs beat 64 and 256 at equal
  // occupancy).  One stage wins where shared memory, not registers, limits
  // the resident CTAs (the two-input stress divergence on 512-point columns).
  {
    const KernelLimits lim = kernel_limits((const void*)kern);
    const int regs = lim.regs;
    double best = -1.0;
    int best_lc = 0, best_ns = 2;
    while ((1 << best_lc) * TL < 32) ++best_lc;  // at least one full warp
    auto off128 = [&](int lc) { return std::abs(std::log2(double((1 << lc) * TL) / 128.0)); };
    for (int ns = 2; ns >= 1; --ns)
      for (int lc = 0; (1 << lc) * TL <= std::min(256, lim.max_threads); ++lc) {
        const int C = 1 << lc, threads = C * TL;
        // whole sectors per row piece (FP32 256-point columns two at a time for a
        // seventeenth warp took 364 us where eight at a time take 195)
        if (threads < 32 || C * sizeof(cplx<T>) < 32) continue;
        const size_t sm = smem_for(C, ns);
        if (sm > SMEM_CAP) break;
        const int warp_regs = ((regs * 32 + 255) / 256) * 256;
        const int by_regs = 65536 / (warp_regs * (threads / 32));
        const int ctas = std::min({int(SM_SMEM / (sm + 1024)), by_regs, 2048 / threads, 32});
        if (ctas < 1) break;
        const double busy = ctas * double(threads / 32) * std::min(1.0, double(a.ncols) / C);
        if (busy > best + 1e-9 || (busy > best - 1e-9 && ns == best_ns && off128(lc) < off128(best_lc))) {
          best = busy;
          best_lc = lc;
          best_ns = ns;
        }
      }
    // a launch of few columns (a plane of the wall law, a small grid): narrower
    // items while they do not fill the chip, down to 32-byte row pieces (whole
    // sectors) -- the time of an item hardly depends on its columns
    const auto items = [&](int lc) { return (long)ceil_div(a.ncols, 1 << lc) * nplanes * ngroups; };
    while (best_lc > 0 && items(best_lc) < sm_count() && (TL << (best_lc - 1)) >= 32 &&
           (sizeof(cplx<T>) << (best_lc - 1)) >= 32)
      --best_lc;
    a.lc = best_lc;
    a.nstage = best_ns;
  }
  a.C = 1 << a.lc;
  a.SI = stride(a.C);
  const size_t smem = smem_for(a.C, a.nstage);
  if (smem > SMEM_CAP) throw CudaError(1, "ypass: shared memory request too large");
  const int threads = a.C * TL;
  a.nplanes = nplanes;
  a.ngroups = ngroups;
  a.d_ncb = fast_div(ceil_div(a.ncols, a.C));
  a.d_np = fast_div(nplanes);
  const long nitems = (long)ceil_div(a.ncols, a.C) * nplanes * ngroups;
  if (nitems == 0) return;
  // persistent grid: the CTAs that fit on the device at once
  const int grid = int(std::min<long>(nitems, (long)resident_ctas((const void*)kern, threads, smem)));
  // columns written: an output may be left out, the narrower filter has fewer,
  // the wall law's is one plane, the boundary layers add one
  double ocols = 0.0;
  for (int q = 0; q < ngroups * a.nout; ++q)
    if (a.out[q]) ocols += double(nplanes) * (a.op == YP_FILTER2 && q % a.nout == 1 ? a.ncols1 : a.ncols);
  if (a.op == YP_GRADY)
    for (int q = 0; q < std::min(ngroups, 2); ++q) ocols += a.wall[q] ? a.ncols1 : 0;
  if (a.op == YP_PRESS) ocols += a.ncols;
  hook_before("ypass", sizeof(cplx<T>) * (double(nplanes) * ngroups * a.ncols * (a.op == YP_PGRAD ? 1 : a.nin) * NY +
                                          ocols * NYO));
  if (a.dep) launch_dep(kern, grid, threads, smem, st, a);
  else kern<<<grid, threads, smem, st>>>(a);
  LES_CHECK_LAUNCH();
  hook_after();
}


template <typename T>
void launch_yrhs(int NF, int N, YRArgs<T> a, cudaStream_t st) {
  const int TL = lanes(N);
  if (lanes(NF) != TL) throw CudaError(1, "yrhs: length pair with different lane counts");
  const int W = 128 / int(sizeof(cplx<T>));
  const int NL = std::max(NF, N);
  auto stride = [&](int C) {  // as in launch_ypass
    const int target = (32 / C) % W;
    const int base = NL + NL / 16;
    return base + ((target - base % W) % W + W) % W;
  };
  auto smem_for = [&](int C, int ns) {
    return sizeof(cplx<T>) * ((NF == N ? 0 : twm_len(NF, false)) + twm_len(N, false) + twm_len(N, true) +
                              (size_t)ns * C * stride(C)) +
           sizeof(T) * ((N + 3) & ~3);
  };
  void (*kern)(YRArgs<T>) = nullptr;
  switch (N) {
#define YR_CASE(B) \
  case B: kern = NF == B ? k_yrhs<T, B, B> : (NF == 3 * B / 2 ? k_yrhs<T, 3 * B / 2, B> : nullptr); break;
    YR_CASE(16) YR_CASE(32) YR_CASE(64) YR_CASE(128) YR_CASE(256) YR_CASE(512)
#undef YR_CASE
    default: break;
  }
  if (!kern) throw CudaError(1, "yrhs: unsupported length pair " + std::to_string(NF) + "->" + std::to_string(N));
  // columns per CTA and slots: the most busy warps per SM, on a tie two slots,
  // then the CTA size nearest 128 threads; narrower where the items do not
  // fill the chip (the rules of launch_ypass)
  const KernelLimits lim = kernel_limits((const void*)kern);
  const int warp_regs = ((lim.regs * 32 + 255) / 256) * 256;
  double best = -1.0;
  int lc = 0, nslot = 2;
  auto off128 = [&](int q) { return std::abs(std::log2(double((1 << q) * TL) / 128.0)); };
  for (int ns = 2; ns >= 1; --ns)
    for (int q = 0; (1 << q) * TL <= std::min(256, lim.max_threads); ++q) {
      const int threads = (1 << q) * TL;
      const size_t sm = smem_for(1 << q, ns);
      if (threads < 32 || (sizeof(cplx<T>) << q) < 32) continue;  // whole sectors per row piece
      if (sm > SMEM_CAP) break;
      const int ctas = std::min({int(SM_SMEM / (sm + 1024)), 65536 / (warp_regs * (threads / 32)), 2048 / threads, 32});
      if (ctas < 1) break;
      const double busy = ctas * double(threads / 32) * std::min(1.0, double(a.ncols) / (1 << q));
      if (busy > best + 1e-9 || (busy > best - 1e-9 && ns == nslot && off128(q) < off128(lc))) {
        best = busy;
        lc = q;
        nslot = ns;
      }
    }
  const auto items = [&](int q) { return (long)ceil_div(a.ncols, 1 << q) * a.nplanes * a.ngroups; };
  while (lc > 0 && items(lc) < sm_count() && (TL << (lc - 1)) >= 32 && (sizeof(cplx<T>) << (lc - 1)) >= 32) --lc;
  a.lc = lc;
  a.C = 1 << lc;
  a.nslot = nslot;
  a.SI = stride(a.C);
  const size_t smem = smem_for(a.C, nslot);
  if (smem > SMEM_CAP) throw CudaError(1, "yrhs: shared memory request too large");
  if (items(lc) == 0) return;
  const int threads = a.C * TL;
  const int grid = int(std::min<long>(items(lc), (long)resident_ctas((const void*)kern, threads, smem)));
  a.d_ncb = fast_div(ceil_div(a.ncols, a.C));
  a.d_np = fast_div(a.nplanes);
  hook_before("yrhs", double(a.nplanes) * a.ngroups * sizeof(cplx<T>) *
                          (double(a.nkp) * NF + 2.0 * a.ncols * N + double(a.ncols) * N));
  if (a.dep) launch_dep(kern, grid, threads, smem, st, a);
  else kern<<<grid, threads, smem, st>>>(a);
  LES_CHECK_LAUNCH();
  hook_after();
}

template <typename T>
void set_attrs_ypass(SpectralUse use, int NY) {
  switch (NY) {
#define YA(N)                                                             \
  case N:                                                                 \
    if (use == SU_STATE) {                                                \
      for (int c : {YC_FWD, YC_GRADY, YC_PGRAD, YC_FILTER, YC_DIV2, YC_OTHER}) raise_smem(ypass_kernel<T, N, N>(c)); \
      raise_smem(ypass_kernel<T, N, 3 * N / 2>(YC_OTHER));                \
      raise_smem(ypass_kernel<T, 3 * N / 2, N>(YC_OTHER));                \
      raise_smem(k_yrhs<T, N, N>);                                        \
      raise_smem(k_yrhs<T, 3 * N / 2, N>);                                \
    } else {                                                              \
      raise_smem(ypass_kernel<T, N, N>(use == SU_PRESSURE ? YC_FWD : YC_GRADY)); \
    }                                                                     \
    break;
    YA(16) YA(32) YA(64) YA(128) YA(256) YA(512)
#undef YA
    default: break;
  }
}

// one translation unit per type (they compile side by side)
#ifdef LES_YPASS_DOUBLE
template void launch_ypass<double>(int, int, YPArgs<double>, int, int, cudaStream_t);
template void launch_yrhs<double>(int, int, YRArgs<double>, cudaStream_t);
template void set_attrs_ypass<double>(SpectralUse, int);
#else
template void launch_ypass<float>(int, int, YPArgs<float>, int, int, cudaStream_t);
template void launch_yrhs<float>(int, int, YRArgs<float>, cudaStream_t);
template void set_attrs_ypass<float>(SpectralUse, int);
#endif

}  // namespace les
