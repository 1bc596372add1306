// The LU analysis against a CUDA runtime of this file's own (no GPU): memory
// is host memory, launches do nothing, and the call that the arguments name
// fails with the error a device gives for it.  The multifrontal path is tried
// by the analysis itself; whatever refuses it must leave the row-wise paths,
// with no error pending.
//   lu_trial_check matrix [what [k]]
//     cluster c   clusters of more than c blocks are not granted
//     launch c    the same, found by the launch alone
//     copies k    copies to the host fail from the k-th on
//     memory k    the k-th allocation fails
//     pivot       the trial refactor reports a bad pivot
// Prints "rc <rc> path <front|rows> pending <error> status <bits> allocations <n>".
#include <cuda_runtime.h>

#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <string>
#include <vector>

#include "lu_front.h"
#include "xg.h"
#include "xg_internal.h"

static std::string what;
static int arg = 0, n_alloc = 0, n_copy = 0, n_launch = 0;
static cudaError_t pending = cudaSuccess;
static cudaError_t say(cudaError_t e) {
  if (e != cudaSuccess) pending = e;
  return e;
}

extern "C" {
void **__cudaRegisterFatBinary(void *) {
  static void *h;
  return &h;
}
void __cudaRegisterFatBinaryEnd(void **) {}
void __cudaUnregisterFatBinary(void **) {}
void __cudaRegisterFunction() {}
void __cudaRegisterVar() {}
int __cudaPushCallConfiguration() { return 0; }
int __cudaPopCallConfiguration() { return 0; }
int __cudaGetKernel() { return 0; }
int __cudaLaunchKernel() { return 0; }
}
cudaError_t cudaLaunchKernelExC(const cudaLaunchConfig_t *c, const void *, void **args) {
  if (what == "pivot" && ++n_launch == 1) {  // front_open(a, a_copy, nnz, status)
    unsigned *status = *static_cast<unsigned **>(args[3]);
    status[0] = 1;
    status[1] = 5;
  }
  for (unsigned k = 0; k < c->numAttrs; ++k)
    if (c->attrs[k].id == cudaLaunchAttributeClusterDimension && (what == "launch" || what == "cluster") &&
        int(c->attrs[k].val.clusterDim.x) > arg)
      return say(cudaErrorInvalidClusterSize);
  return cudaSuccess;
}
cudaError_t cudaOccupancyMaxActiveClusters(int *n, const void *, const cudaLaunchConfig_t *c) {
  *n = what == "cluster" && int(c->attrs[0].val.clusterDim.x) > arg ? 0 : 8;
  return cudaSuccess;
}
cudaError_t cudaMalloc(void **p, size_t bytes) {
  *p = nullptr;
  if (++n_alloc == arg && what == "memory") return say(cudaErrorMemoryAllocation);
  *p = std::calloc(bytes ? bytes : 1, 1);
  return cudaSuccess;
}
cudaError_t cudaFree(void *p) {
  std::free(p);
  return cudaSuccess;
}
cudaError_t cudaMemcpy(void *d, const void *s, size_t n, cudaMemcpyKind) {
  std::memcpy(d, s, n);
  return cudaSuccess;
}
cudaError_t cudaMemcpyAsync(void *d, const void *s, size_t n, cudaMemcpyKind k, cudaStream_t) {
  if (what == "copies" && k == cudaMemcpyDeviceToHost && ++n_copy >= arg) return say(cudaErrorInvalidValue);
  std::memcpy(d, s, n);
  return cudaSuccess;
}
cudaError_t cudaMemset(void *p, int v, size_t n) {
  std::memset(p, v, n);
  return cudaSuccess;
}
cudaError_t cudaMemsetAsync(void *p, int v, size_t n, cudaStream_t) { return cudaMemset(p, v, n); }
cudaError_t cudaDeviceGetAttribute(int *v, cudaDeviceAttr a, int) {
  *v = a == cudaDevAttrMultiProcessorCount ? 152 : a == cudaDevAttrMaxSharedMemoryPerBlockOptin ? 232448 : 0;
  return cudaSuccess;
}
cudaError_t cudaFuncSetAttribute(const void *, cudaFuncAttribute, int) { return cudaSuccess; }
cudaError_t cudaOccupancyMaxActiveBlocksPerMultiprocessorWithFlags(int *n, const void *, int, size_t, unsigned) {
  *n = 2;
  return cudaSuccess;
}
cudaError_t cudaOccupancyMaxActiveBlocksPerMultiprocessor(int *n, const void *, int, size_t) {
  *n = 2;
  return cudaSuccess;
}
cudaError_t cudaGetDevice(int *d) {
  *d = 0;
  return cudaSuccess;
}
cudaError_t cudaSetDevice(int) { return cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaGetLastError() {
  const cudaError_t e = pending;
  pending = cudaSuccess;
  return e;
}
const char *cudaGetErrorString(cudaError_t) { return "as asked for"; }

// what the analysis takes from the rest of the library
namespace xg {
void set_error(const std::string &s) { std::fprintf(stderr, "%s\n", s.c_str()); }
void count_launches(int) {}
int ctx_info(xg_ctx *, int *device, void **stream) {
  *device = 0;
  *stream = nullptr;
  return XG_OK;
}
}  // namespace xg

int main(int argc, char **argv) {
  FILE *f = std::fopen(argv[1], "rb");
  int64_t head[2];
  if (!f || std::fread(head, 8, 2, f) != 2) return 2;
  std::vector<int> rp(head[0] + 1), ci(head[1]);
  std::vector<double> a(head[1]);
  if (std::fread(rp.data(), 4, rp.size(), f) != rp.size() || std::fread(ci.data(), 4, ci.size(), f) != ci.size() ||
      std::fread(a.data(), 8, a.size(), f) != a.size())
    return 2;
  std::fclose(f);
  if (argc > 2) what = argv[2];
  if (argc > 3) arg = std::atoi(argv[3]);
  xg_lu *lu = nullptr;
  const int rc = xg_lu_analyze(reinterpret_cast<xg_ctx *>(&lu), int(head[0]), rp.data(), ci.data(), a.data(),
                               XG_LU_FP64, &lu);
  const int left = int(pending), allocs = n_alloc;
  what.clear();
  int status = -1, row = -1, front = -1;
  if (!rc) {
    xg_lu_status(lu, &status, &row);
    front = xg_lu_get_path(lu) == XG_LU_PATH_FRONT;
    xg_lu_destroy(lu);
  }
  std::printf("rc %d path %s pending %d status %d allocations %d\n", rc, front == 1 ? "front" : front ? "none" : "rows", left,
              status, allocs);
  return 0;
}
