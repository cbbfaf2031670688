// Launch helpers shared by the translation units of the spectral passes
// (spectral_xfwd.cu, spectral_xinv.cu, spectral_ypass.cu): occupancy and
// register queries with per-device caches, the rows-per-item choice of the
// x passes, the FFT lane counts and the supported lengths.
#pragma once
#include <algorithm>
#include <cmath>
#include <cstdint>
#include <string>

#include "launch.cuh"
#include "spectral.cuh"

namespace les {

#define LES_LENGTHS(X) X(16) X(24) X(32) X(48) X(64) X(96) X(128) X(192) X(256) X(384) X(512) X(768)

struct KernelLimits {
  int regs, max_threads;
};
int resident_ctas(const void* kern, int threads, size_t smem);
KernelLimits kernel_limits(const void* kern);
inline int kernel_regs(const void* kern) { return kernel_limits(kern).regs; }
int lanes(int n);
int pad_seqs(int nseq, int M);

inline constexpr int SMEM_CAP = 200 * 1024;
inline constexpr size_t SM_SMEM = 228 * 1024;  // shared memory per SM (1 KB of it reserved per CTA)

int sm_count();  // of the current device (cached)

// Rows per work item of an x pass (TL lanes per sequence, seq_per_row
// sequences per grid row, nrows rows in the launch): the count that keeps the
// most sequence slots of an SM busy -- resident CTAs (shared memory,
// registers) times the fraction of the slots of each pass that hold a
// sequence; on a tie the larger count (fewer items).
// A launch whose items at that count fill less than two rounds of resident
// CTAs (a plane of the wall law, a small grid) is bound by the time of one
// item, not by throughput: it takes the count with the fewest rounds of
// passes, on a tie the fewest rows, so that its items spread over the chip
// (the wall law's x inverse of a 256 x 256 plane in FP32: 32 CTAs became 256,
// 35.5 -> 14.5 us; of 64 x 64: 20.8 -> 11.3 us).
template <typename SmemFn>
inline int best_rows(const void* kern, int seq_per_row, int TL, SmemFn smem_for, long nrows, double* best_score = nullptr,
              int threads = 256) {
  const int rmax = 32;
  const int regs = kernel_regs(kern);
  const int warp_regs = ((regs * 32 + 255) / 256) * 256;
  const int by_regs = std::max(1, 65536 / (warp_regs * (threads / 32)));
  const int S = threads / TL;
  const long sms = sm_count();
  double best = -1.0;
  int best_r = 1, best_ctas = 1;
  long few = -1;  // rounds of passes of the launch at few_r
  int few_r = 1;
  for (int R = 1; R <= rmax; ++R) {
    const size_t sm = smem_for(R);
    if (sm > SMEM_CAP) break;
    const int ctas = std::min({int(SM_SMEM / (sm + 1024)), by_regs, 2048 / threads, 32});
    if (ctas < 1) break;
    const int nseq = R * seq_per_row;
    const int passes = (nseq + S - 1) / S;
    const double score = ctas * double(nseq) / double(passes * S);
    if (score >= best - 1e-9) {
      best = score;
      best_r = R;
      best_ctas = ctas;
    }
    const long items = (nrows + R - 1) / R;
    const long rounds = ((items + sms * ctas - 1) / (sms * ctas)) * passes;
    if (few < 0 || rounds < few) {
      few = rounds;
      few_r = R;
    }
  }
  if (best_score) *best_score = best;
  return (nrows + best_r - 1) / best_r < 2 * sms * best_ctas ? few_r : best_r;
}


// shared-memory limit of a kernel on the current device
template <typename... P>
inline void raise_smem(void (*kern)(P...)) {
  if (kern) LES_CUDA(cudaFuncSetAttribute((const void*)kern, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM_CAP));
}
// of each family's kernels of a length (y: of a grid) for a use
template <typename T> void set_attrs_xfwd(SpectralUse use, int NX);
template <typename T> void set_attrs_xinv(SpectralUse use, int NX);
template <typename T> void set_attrs_ypass(SpectralUse use, int NY);

}  // namespace les
