// Host check of cluster_blocks (solver.cuh) with the three runtime calls it makes
// replaced by fakes: a refused attribute or query falls back to a smaller
// cluster or to none and leaves no CUDA error behind for the next call's check.
#include <cuda_runtime.h>

#include <cstdio>

static cudaError_t g_last = cudaSuccess;  // what cudaGetLastError returns and clears
static bool g_refuse_attr = false, g_refuse_query = false;
static int g_fit = 1;

template <typename T>
static cudaError_t fake_set(T, cudaFuncAttribute, int) {
  return g_refuse_attr ? (g_last = cudaErrorInvalidValue) : cudaSuccess;
}
template <typename T>
static cudaError_t fake_query(int* fit, T, const cudaLaunchConfig_t*) {
  *fit = g_fit;
  return g_refuse_query ? (g_last = cudaErrorInvalidConfiguration) : cudaSuccess;
}
static cudaError_t fake_last() {
  const cudaError_t e = g_last;
  g_last = cudaSuccess;
  return e;
}
#define cudaFuncSetAttribute fake_set
#define cudaOccupancyMaxActiveClusters fake_query
#define cudaGetLastError fake_last
#include "../../axia-fem_gb300/csrc/solver.cuh"

static int check(const char* what, int64_t work, int want) {
  const int got = cluster_blocks(nullptr, work);
  const bool clean = g_last == cudaSuccess;
  g_last = cudaSuccess;
  if (got == want && clean) return 0;
  std::printf("%s, %lld threads: %d blocks (%d expected)%s\n", what, (long long)work, got, want,
              clean ? "" : ", a CUDA error is left behind");
  return 1;
}

int main() {
  int bad = 0;
  const int64_t t = PCG_THREADS;
  bad += check("plain", 1, 1) + check("plain", t, 1) + check("plain", t + 1, 2) + check("plain", 3 * t, 4);
  bad += check("plain", 9 * t, 16) + check("plain", 1000 * t, 16);
  g_refuse_attr = true;
  bad += check("no large clusters", 4 * t, 4) + check("no large clusters", 9 * t, 8);
  g_refuse_attr = false;
  g_refuse_query = true;
  bad += check("query refused", 4 * t, 0);
  g_refuse_query = false;
  g_fit = 0;
  bad += check("does not fit", 4 * t, 0);
  return bad;
}
