// What the runtime says about a kernel (registers, CTAs per SM), kept per
// kernel and launch shape: the launchers ask several times per launch.
#pragma once
#include <cstddef>
#include <cstdint>

namespace les {

// Spectral kernels of the library (every length, type and class of op) and the
// launch shapes a process may use them at; the tables below take a few times
// as many before they start over.
inline constexpr int SPECTRAL_KERNELS = 264;

// Open-addressing hash table in fixed storage (no heap: the allocation-free
// entry point launches these kernels too).  A table that is three quarters full
// is emptied, so that it never stops taking entries.  The caller locks.
template <typename Val, int N>
class LaunchCache {
  static_assert((N & (N - 1)) == 0, "a power of two");

 public:
  const Val* find(int dev, const void* kern, int threads, size_t smem) const {
    for (unsigned i = slot(dev, kern, threads, smem);; i = (i + 1) & (N - 1)) {
      const Entry& e = table[i];
      if (!e.kern) return nullptr;
      if (e.kern == kern && e.smem == smem && e.dev == dev && e.threads == threads) return &e.val;
    }
  }
  // (not there yet)
  void put(int dev, const void* kern, int threads, size_t smem, const Val& v) {
    if (4 * used >= 3 * N) {
      for (Entry& e : table) e.kern = nullptr;
      used = 0;
    }
    unsigned i = slot(dev, kern, threads, smem);
    while (table[i].kern) i = (i + 1) & (N - 1);
    table[i] = Entry{kern, smem, dev, threads, v};
    ++used;
  }

 private:
  struct Entry {
    const void* kern;
    size_t smem;
    int dev, threads;
    Val val;
  };
  static unsigned slot(int dev, const void* kern, int threads, size_t smem) {
    uint64_t h = uint64_t(reinterpret_cast<uintptr_t>(kern));
    h = (h ^ (uint64_t(smem) << 20) ^ (uint64_t(threads) << 44) ^ (uint64_t(dev) << 56)) * 0x9e3779b97f4a7c15ull;
    return unsigned(h >> 32) & (N - 1);
  }
  Entry table[N] = {};
  int used = 0;
};

inline constexpr int LIMITS_CACHE = 2048, RESIDENT_CACHE = 8192;

}  // namespace les
