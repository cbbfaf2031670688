// Instantiation and launch of the x inverse pass (k_xinv) for every
// supported transform length.
#include "spectral_launch.cuh"

#include "launch.cuh"

namespace les {

// the kernel of a length and class (nullptr: none): the products' lengths for
// plain stores and the convective inputs, the grids' own for the rest
template <typename T>
static auto xinv_kernel(int NX, int cls) -> void (*)(XIArgs<T>) {
  switch (NX) {
#define XI_CASE(N) \
  case N: if (cls == XC_STORE) return k_xinv<T, N, XC_STORE>; if (cls == XC_CONV) return k_xinv<T, N, XC_CONV>; break;
    LES_LENGTHS(XI_CASE)
#undef XI_CASE
    default: return nullptr;
  }
  switch (NX) {
#define XI_CASE(N)                                           \
  case N:                                                    \
    if (cls == XC_DIV) return k_xinv<T, N, XC_DIV>;          \
    if (cls == XC_DYN) return k_xinv<T, N, XC_DYN>;          \
    if (cls == XC_WALL) return k_xinv<T, N, XC_WALL>;        \
    break;
    XI_CASE(16) XI_CASE(32) XI_CASE(64) XI_CASE(128) XI_CASE(256) XI_CASE(512)
#undef XI_CASE
    default: break;
  }
  return nullptr;
}

template <typename T>
void launch_xinv(int NX, XIArgs<T> a, cudaStream_t st) {
  const int M = NX / 2;
  if (a.ipitch == 0) a.ipitch = a.nk;
  a.pair_store = (a.out_pstride % 2 == 0);
  for (int f = 0; f < a.nin && f < 16; ++f)
    if (a.out[f] && reinterpret_cast<uintptr_t>(a.out[f]) % (2 * sizeof(T)) != 0) a.pair_store = 0;
  // sequence slots and one or two input stages per CTA; rows per work item
  // and stages from best_rows below
  const int SL = slot_stride(M, int(sizeof(cplx<T>)));
  const int ns = a.nstage ? a.nstage : a.nin;  // staged rows per grid row
  a.d_rows = fast_div(a.rows_pp);
  a.d_ns = fast_div(ns);
  a.d_nin = fast_div(a.nin);
  a.d_nk = fast_div(a.nk);
  {
    // staged row stride: the split reads a row's modes at consecutive
    // lanes, the TL lanes of 32 / TL sequences per warp in different rows;
    // a stride of TL (mod the values per wavefront) puts those rows on
    // disjoint banks, as slot_stride does for the sequence slots
    // (an odd FP32 row is copied with one value more, whole 16 bytes: its
    // last value alone went by a load in front of every batch, and where the
    // stride then was odd the rows went without bulk copies)
    const int W = 128 / int(sizeof(cplx<T>)), TL = lanes(M);
    a.nkc = (a.nk * sizeof(cplx<T>)) % 16 != 0 && a.ipitch > a.nk ? a.nk + 1 : a.nk;
    a.nks = TL < W ? a.nk : a.nkc;
    if (TL < W) a.nks += ((TL % W - a.nk % W) % W + W) % W;
  }
  // a plain store with one staged row per sequence transforms each sequence
  // in its own staged row (the exchange slot is the row), which leaves room
  // for more rows per work item
  // (XI_CONV: six of its seven staged rows become sequences)
  a.merged = ((a.op == XI_STORE && a.nstage == 0) || a.op == XI_CONV || a.op == XI_CONVS) ? 1 : 0;
  if (a.merged) a.nks = std::max(a.nks, SL);
  auto stage_rows = [&](int R) {
    return a.merged ? R * (ns - a.nin) + pad_seqs(R * a.nin, M) : R * ns;
  };
  // bulk staging: one cp.async.bulk per staged row needs 16-byte aligned
  // rows in global memory (base, pitch and plane stride) and in the stages
  // (stage base and row stride)
  {
    const size_t cs = sizeof(cplx<T>);
    a.bulk = ((cs * a.ipitch) % 16 == 0 && (cs * a.in_pstride) % 16 == 0 && (cs * a.nks) % 16 == 0 &&
              (cs * (NX + twm_len(M, true))) % 16 == 0 && a.nk * cs >= 16)
                 ? 1
                 : 0;
    for (int f = 0; f < ns; ++f)
      if (reinterpret_cast<uintptr_t>(a.in[f]) % 16 != 0) a.bulk = 0;
  }
  auto smem_nb = [&](int R, int nb) {
    return sizeof(cplx<T>) * (NX + twm_len(M, true) + nb * (((size_t)stage_rows(R) * a.nks + 1) & ~size_t(1)) +
                              (a.merged ? 0 : (size_t)pad_seqs(R * a.nin, M) * SL)) +
           2 * sizeof(int) * R + (a.nstage ? sizeof(T) * (a.nk + 2) : 0) + (a.bulk ? 2 * sizeof(uint64_t) + 8 : 0);
  };
  void (*const kern)(XIArgs<T>) = xinv_kernel<T>(NX, xi_class(a.op));
  if (!kern) throw CudaError(1, "xinv: unsupported transform length " + std::to_string(NX));
  // two stages unless one stage keeps strictly more sequence slots busy
  // (more resident CTAs where shared memory limits them)
  {
    double s2 = -1.0, s1 = -1.0;
    const int r2 = best_rows((const void*)kern, a.nin, lanes(M), [&](int R) { return smem_nb(R, 2); }, a.nrows, &s2);
    const int r1 = best_rows((const void*)kern, a.nin, lanes(M), [&](int R) { return smem_nb(R, 1); }, a.nrows, &s1);
    a.nbuf = (s1 > s2 + 1e-9) ? 1 : 2;
    a.R = (a.nbuf == 1) ? r1 : r2;
  }
  a.stage_rows = stage_rows(a.R);
  const size_t smem = smem_nb(a.R, a.nbuf);
  if (smem > SMEM_CAP) throw CudaError(1, "xinv: shared memory request too large");
  {
    // the combining ops read the sequence slots four reals at a time
    const size_t stage_len = ((size_t)a.stage_rows * a.nks + 1) & ~size_t(1);
    const size_t slots = sizeof(cplx<T>) * (NX + twm_len(M, true) + a.nbuf * stage_len);
    if (!a.merged && slots % 16 != 0) throw CudaError(1, "xinv: sequence slots not 16-byte aligned");
  }
  const long nitems = ceil_div(a.nrows, a.R);
  if (nitems == 0) return;
  const int grid = int(std::min<long>(nitems, (long)resident_ctas((const void*)kern, 256, smem)));
  {
    int rows = 0, vals = a.nin;  // spectral rows read (a spectrum staged at two levels once), values read and written
    for (int f = 0; f < ns; ++f) rows += std::find(a.in, a.in + f, a.in[f]) == a.in + f;
    if (a.op == XI_DIV)  // tz and rhs, the old rhs unless fresh; with the advance the variable twice and the last rhs
      for (int q = 0; q < a.nin; ++q) vals += 1 + (a.fresh ? 0 : 1) + (a.adv_v[q] ? 3 : 0);
    else if (a.op == XI_LASD || a.op == XI_SCDYN) vals = 2;
    else if (a.op == XI_WALL) vals = 7;
    hook_before("xinv", double(a.nrows) * rows * a.nk * sizeof(cplx<T>) + double(a.nrows) * NX * vals * sizeof(T));
  }
  if (a.dep) launch_dep(kern, grid, 256, smem, st, a);
  else kern<<<grid, 256, smem, st>>>(a);
  LES_CHECK_LAUNCH();
  hook_after();
}


template <typename T>
void set_attrs_xinv(SpectralUse use, int NX) {
  for (int c : {XC_STORE, XC_CONV, XC_DIV, XC_DYN, XC_WALL})
    if (c == XC_STORE || use == SU_STATE) raise_smem(xinv_kernel<T>(NX, c));
}

// one translation unit per type (they compile side by side)
#ifdef LES_XINV_DOUBLE
template void launch_xinv<double>(int, XIArgs<double>, cudaStream_t);
template void set_attrs_xinv<double>(SpectralUse, int);
#else
template void launch_xinv<float>(int, XIArgs<float>, cudaStream_t);
template void set_attrs_xinv<float>(SpectralUse, int);
#endif

}  // namespace les
