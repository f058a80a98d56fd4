// Host-side rules of the tensor-core launches, run without a GPU: the three runtime calls they make are
// defined here, ahead of the runtime library's.  Prints one line per check that fails.
#include "tc_common.cuh"

#include <cstdio>

namespace {
int device = 0, clusters_of[2] = {10, 5}, queries = 0;
bool failing = false;
int failures = 0;
void check(bool ok, const char* what) { if (!ok) { printf("failed: %s\n", what); ++failures; } }
}  // namespace

#ifndef __CUDA_ARCH__      // the device pass has its own
extern "C" {
cudaError_t CUDARTAPI cudaGetDevice(int* d) { *d = device; return cudaSuccess; }
cudaError_t CUDARTAPI cudaFuncSetAttribute(const void*, cudaFuncAttribute, int) { return cudaSuccess; }
cudaError_t CUDARTAPI cudaOccupancyMaxActiveClusters(int* n, const void*, const cudaLaunchConfig_t*) {
  ++queries;
  if (failing) return cudaErrorUnknown;
  *n = clusters_of[device];
  return cudaSuccess;
}
cudaError_t CUDARTAPI cudaGetLastError(void) { return cudaSuccess; }
}
#endif

using namespace attn;
using namespace attn::tc;

static void some_kernel() {}

static void cluster_queries() {
  TileKernelState state;
  auto slots = [&] { return cluster_slots(&some_kernel, 4, 352, 200000, state); };
  failing = true;
  check(slots() <= 0, "a failed query gives no slots");
  failing = false;
  check(slots() == 40, "a failed query is made again");
  device = 1;
  check(slots() == 20, "the second device has its own number");
  device = 0;
  const int before = queries;
  check(slots() == 40 && queries == before, "a known number is not asked for again");
}

int main() {
  cluster_queries();
  return failures;
}
