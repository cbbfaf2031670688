// Instantiation and launch of the x forward passes (k_xfwd, k_xfwd_row) for
// every supported transform length.
#include "spectral_launch.cuh"

#include "launch.cuh"

namespace les {

// the x forward pass of whole rows
template <typename T, typename S>
static void launch_xfwd_row(int NX, XFArgs<T>& a, cudaStream_t st) {
  const int M = NX / 2;
  const int SL = slot_stride(M, int(sizeof(cplx<T>)));
  a.nsrc = a.op == XF_PRESS ? 4 : a.nf;
  a.d_ns = fast_div(a.nsrc);
  auto stage_rows = [&](int R) { return R * (a.nsrc - a.nf) + pad_seqs(R * a.nf, M); };
  auto smem_nb = [&](int R, int nb) {
    return sizeof(cplx<T>) * (NX + twm_len(M, false) + (size_t)nb * stage_rows(R) * SL) + 2 * sizeof(uint64_t) +
           sizeof(T) * ((R * a.nf + 1) & ~1) + 2 * sizeof(int) * R + 16;
  };
  void (*kern)(XFArgs<T>) = nullptr;
  switch (NX) {
#define XR_CASE(N) \
  case N: kern = k_xfwd_row<T, N, S>; break;
    LES_LENGTHS(XR_CASE)
#undef XR_CASE
    default:
      throw CudaError(1, "xfwd: unsupported transform length " + std::to_string(NX));
  }
  // two stages unless one keeps strictly more sequence slots busy (as
  // launch_xinv)
  double s2 = -1.0, s1 = -1.0;
  const int r2 = best_rows((const void*)kern, a.nf, lanes(M), [&](int R) { return smem_nb(R, 2); }, a.nrows, &s2);
  const int r1 = best_rows((const void*)kern, a.nf, lanes(M), [&](int R) { return smem_nb(R, 1); }, a.nrows, &s1);
  a.nbuf = (s1 > s2 + 1e-9) ? 1 : 2;
  a.R = (a.nbuf == 1) ? r1 : r2;
  a.stage_rows = stage_rows(a.R);
  const size_t smem = smem_nb(a.R, a.nbuf);
  if (smem > SMEM_CAP || a.R * a.nf > 256) throw CudaError(1, "xfwd: shared memory request too large");
  const long nitems = ceil_div(a.nrows, a.R);
  if (nitems == 0) return;
  const int grid = int(std::min<long>(nitems, (long)resident_ctas((const void*)kern, 256, smem)));
  if (a.dep) launch_dep(kern, grid, 256, smem, st, a);
  else kern<<<grid, 256, smem, st>>>(a);
  LES_CHECK_LAUNCH();
}

template <typename T>
void launch_xfwd(int NX, XFArgs<T> a, cudaStream_t st) {
  const int M = NX / 2;
  if (a.opitch == 0) a.opitch = a.nk;
  a.d_rows = fast_div(a.rows_pp);
  a.d_nf = fast_div(a.nf);
  a.in_rstride = NX;
  const bool press = a.op == XF_PRESS;
  static const int nin_of_op[] = {0, 9, 6, 10, 3, 6, 14, 9};
  const int nin = a.op == XF_SCALE ? a.nf : nin_of_op[a.op];
  const size_t isz = (a.in_f32 ? sizeof(float) : sizeof(T));
  hook_before("xfwd", double(a.nrows) * NX * nin * isz + double(a.nrows) * (press ? 2 : a.nf) * a.nk * sizeof(cplx<T>));
  // scalings and the pressure take whole rows, which go by bulk copies: every
  // caller's rows are 16-byte aligned
  if (press || a.op == XF_SCALE) {
    bool aligned = (isz * a.in_pstride) % 16 == 0 && (isz * NX) % 16 == 0;
    for (int f = 0; f < (press ? 5 : a.nf); ++f)
      aligned = aligned && reinterpret_cast<uintptr_t>(a.in_f32 ? (const void*)a.inf[f] : (const void*)a.in[f]) % 16 == 0;
    if (!aligned) throw CudaError(1, "xfwd: input rows not 16-byte aligned");
    if (a.in_f32) {
      if constexpr (std::is_same<T, double>::value) launch_xfwd_row<T, float>(NX, a, st);
      else throw CudaError(1, "xfwd: FP32 inputs are for FP64 transforms");
    } else {
      launch_xfwd_row<T, T>(NX, a, st);
    }
    hook_after();
    return;
  }
  const int SL = slot_stride(M, int(sizeof(cplx<T>)));
  auto smem_for = [&](int R) {
    return sizeof(cplx<T>) * (NX + twm_len(M, false) + (size_t)pad_seqs(R * a.nf, M) * SL) + sizeof(T) * R * a.nf +
           2 * sizeof(int) * R + 16;
  };
  void (*kern)(XFArgs<T>) = nullptr;
  switch (NX) {
#define XF_CASE(N) \
  case N: kern = k_xfwd<T, N>; break;
    LES_LENGTHS(XF_CASE)
#undef XF_CASE
    default:
      throw CudaError(1, "xfwd: unsupported transform length " + std::to_string(NX));
  }
  // the convective input and product passes load many inputs per point
  // straight from global memory: 128-thread CTAs (twice the CTAs per SM at
  // the same register budget) overlap one CTA's loads with the transforms of
  // others at a finer grain (measured at 256^3: 0.667 -> 0.633 ms per step);
  // the other ops keep 256 threads (the stress divergence measured slower
  // with 128: 0.236 -> 0.256 ms)
  const int XF_THREADS = (a.op == XF_CONV_IN || a.op == XF_PROD || a.op == XF_PROD_SC) ? 128 : 256;
  a.R = best_rows((const void*)kern, a.nf, lanes(M), smem_for, a.nrows, nullptr, XF_THREADS);
  const size_t smem = smem_for(a.R);
  if (smem > SMEM_CAP) throw CudaError(1, "xfwd: shared memory request too large");
  // ops that read a level and its neighbours: the CTA's rows are one row of R
  // consecutive levels, whose neighbours' values the same SM has just read
  // (the convective products at 256^3, mixed 165 -> 160 us, FP64 310 -> 303;
  // at 128^3 FP64 28.7 -> 27.7), unless the last group of levels would leave
  // more than an eighth of the rows' slots empty
  const int nlev = a.nrows / a.rows_pp, ngrp = ceil_div(nlev, a.R);
  a.lfast = (a.op == XF_PROD || a.op == XF_PROD_SC || a.op == XF_LASD || a.op == XF_SCDYN) &&
            8L * ngrp * a.R <= 9L * nlev;
  const int grid = a.lfast ? a.rows_pp * ngrp : ceil_div(a.nrows, a.R);
  if (grid == 0) return;
  if (a.dep) launch_dep(kern, grid, XF_THREADS, smem, st, a);
  else kern<<<grid, XF_THREADS, smem, st>>>(a);
  LES_CHECK_LAUNCH();
  hook_after();
}


template <typename T>
void set_attrs_xfwd(SpectralUse use, int NX) {
  switch (NX) {
#define XA(N)                                                                                             \
  case N:                                                                                                 \
    if (use == SU_STATE) raise_smem(k_xfwd<T, N>);                                                         \
    if (use != SU_PRESSURE) raise_smem(k_xfwd_row<T, N, T>);                                               \
    if constexpr (std::is_same<T, double>::value) if (use == SU_PRESSURE) raise_smem(k_xfwd_row<T, N, float>); \
    break;
    LES_LENGTHS(XA)
#undef XA
    default: break;
  }
}

template void launch_xfwd<float>(int, XFArgs<float>, cudaStream_t);
template void launch_xfwd<double>(int, XFArgs<double>, cudaStream_t);
template void set_attrs_xfwd<float>(SpectralUse, int);
template void set_attrs_xfwd<double>(SpectralUse, int);

}  // namespace les
