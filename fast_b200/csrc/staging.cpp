// staging.cpp - host copies between a caller's arrays and the pinned staging
// buffer.
//
// A single thread moves 3 MB in about 0.35 ms, twice that into a result array
// whose pages are touched for the first time, while the DMA of the pinned
// buffer takes 0.06.  Up to eight threads (as many as OpenMP is allowed) each
// take a slice of a large copy.  Threads that have slept through a long solve
// take 0.2 ms to wake: copies of 2.3 MB behind solves of 18 ms cost 0.4 ms more
// in parallel, 1.1 to 3.3 MB in calls that follow each other 0.1 to 0.5 ms
// less, 12 to 40 MB 4 to 11 ms less.  So copies from 3 MB on are shared.
// (Threads started for each copy: 0.2 ms for each of them.)  A team of another
// size than the last one's costs the next parallel region its missing threads:
// the pattern of an upload behind such a copy takes 0.38 instead of 0.22 ms on
// 16 cores, once.
#include <omp.h>

#include <algorithm>
#include <cstring>

#include "internal.h"

namespace fastgpu {

static int copy_threads(size_t bytes) {
  if (bytes < ((size_t)3 << 20)) return 1;
  return std::max(1, std::min(std::min(8, omp_get_max_threads()), (int)std::min<size_t>(8, bytes >> 18)));
}

void copy_host(void *dst, const void *src, size_t bytes) {
  const int nt = copy_threads(bytes);
  if (nt == 1) {
    std::memcpy(dst, src, bytes);
    return;
  }
  const size_t slice = (bytes / nt + 4095) / 4096 * 4096;
#pragma omp parallel for num_threads(nt) schedule(static, 1)
  for (int t = 0; t < nt; t++) {
    const size_t a = std::min(bytes, t * slice), b = t + 1 == nt ? bytes : std::min(bytes, a + slice);
    std::memcpy((char *)dst + a, (const char *)src + a, b - a);
  }
}

void gather_host(double *dst, const double *src, const int32_t *at, int64_t n) {
  const int nt = copy_threads(sizeof(double) * (size_t)n);
#pragma omp parallel for num_threads(nt) schedule(static) if (nt > 1)
  for (int64_t i = 0; i < n; i++) dst[i] = src[at[i]];
}

}  // namespace fastgpu
