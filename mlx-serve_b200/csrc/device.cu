// Per-device facts the launch planners need, looked up once per device under a lock.
#include <mutex>
#include <set>

#include "kernels.h"

namespace qb {

std::mutex& setup_mutex() {
  static std::mutex mu;
  return mu;
}

namespace {
std::mutex g_reader_mu;
std::set<const void*>& readers() {
  static std::set<const void*>* s = new std::set<const void*>;
  return *s;
}
}  // namespace

void note_reader(const void* kernel) {
  std::lock_guard<std::mutex> lk(g_reader_mu);
  readers().insert(kernel);
}

bool weights_settled(cudaStream_t st) {
  cudaStreamCaptureStatus status = cudaStreamCaptureStatusNone;
  if (cudaStreamIsCapturing(st, &status) != cudaSuccess) { (void)cudaGetLastError(); return false; }
  if (status != cudaStreamCaptureStatusActive) return false;
  const cudaGraphNode_t* before = nullptr;
  const cudaGraphEdgeData* edges = nullptr;
  size_t n = 0;
  unsigned long long id;
  cudaGraph_t graph;
  if (cudaStreamGetCaptureInfo_v3(st, &status, &id, &graph, &before, &edges, &n) != cudaSuccess || status != cudaStreamCaptureStatusActive) {
    (void)cudaGetLastError();
    return false;
  }
  for (size_t i = 0; i < n; ++i) {   // (none: the graph starts here, and a graph starts when all work before it is complete)
    cudaGraphNodeType type;
    cudaKernelNodeParams kp;
    if (cudaGraphNodeGetType(before[i], &type) != cudaSuccess || type != cudaGraphNodeTypeKernel ||
        cudaGraphKernelNodeGetParams(before[i], &kp) != cudaSuccess) {   // (another library's kernel may have no name here)
      (void)cudaGetLastError();
      return false;
    }
    std::lock_guard<std::mutex> lk(g_reader_mu);
    if (!readers().count(kp.func)) return false;
  }
  return true;
}

int& wait_polls() {
  static thread_local int polls = 0;
  return polls;
}

bool& refuse_clusters() {
  static thread_local bool refuse = false;
  return refuse;
}

// Streaming multiprocessors of the current device (148 on B200).  A failed query (no device, as in a
// host-only check of the library) answers 148 so that size queries stay deterministic.
int sm_count() {
  static std::mutex mu;
  static int cached[64] = {};
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess) { (void)cudaGetLastError(); return 148; }
  if (dev < 0 || dev >= 64) dev = 0;
  std::lock_guard<std::mutex> lk(mu);
  if (cached[dev] == 0) {
    int n = 0;
    if (cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || n <= 0) {
      (void)cudaGetLastError();
      return 148;
    }
    cached[dev] = n;
  }
  return cached[dev];
}

}  // namespace qb
