// A CUDA runtime over host memory and the launchers whose results the host
// code reads, for the tests of hb_index.cu on the CPU (tests/host/__init__.py).
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdlib>
#include <cstring>
#include <map>
#include <set>
#include <string>
#include <vector>

#include "hb_internal.hpp"

namespace {
std::map<uintptr_t, size_t> live;  // device allocations
size_t used = 0, largest = 0, limit = ~size_t(0);
long long failures = 0, stale = 0, captures = 0, graph_launches = 0;
int overflow_queries = 0, device_err = 0, failing_copies = 0;
bool capturing = false;
std::vector<std::string> launches;
// Buffers the launches of a captured graph were given.
std::set<const void*> captured;
std::map<cudaGraphExec_t, std::set<const void*>> graphs;

bool is_live(const void* p) {
  auto it = live.upper_bound(reinterpret_cast<uintptr_t>(p));
  if (it == live.begin()) return false;
  --it;
  return reinterpret_cast<uintptr_t>(p) < it->first + it->second;
}
// A launch's name and its buffers, which have to be live.
void note(const char* name, std::initializer_list<const void*> bufs) {
  launches.push_back(name);
  for (const void* b : bufs) {
    if (b && !is_live(b)) ++stale;
    if (b && capturing) captured.insert(b);
  }
}
}  // namespace

extern "C" {
// ---- what the tests ask and set -------------------------------------------
void fake_reset() {
  limit = ~size_t(0);
  failures = stale = captures = graph_launches = 0;
  overflow_queries = device_err = failing_copies = 0;
  launches.clear();
  largest = 0;
}
void fake_limit(size_t bytes) { limit = bytes; }
size_t fake_used() { return used; }
// The largest block asked for since the last reset, which this makes.
size_t fake_largest() {
  const size_t n = largest;
  largest = 0;
  return n;
}
long long fake_failures() { return failures; }
long long fake_stale() { return stale; }
long long fake_captures() { return captures; }
long long fake_graph_launches() { return graph_launches; }
void fake_overflow(int queries) { overflow_queries = queries; }
void fake_err(int code) { device_err = code; }
void fake_fail_copies(int n) { failing_copies = n; }
int fake_launched(const char* name) {
  return static_cast<int>(std::count(launches.begin(), launches.end(), std::string(name)));
}

// ---- runtime ----------------------------------------------------------------
cudaError_t cudaMalloc(void** p, size_t n) {
  if (used + n > limit) {
    ++failures;
    *p = nullptr;
    return cudaErrorMemoryAllocation;
  }
  *p = std::calloc(1, n ? n : 1);  // (large blocks cost nothing until they are written)
  if (!*p) return cudaErrorMemoryAllocation;
  live[reinterpret_cast<uintptr_t>(*p)] = n;
  used += n;
  largest = std::max(largest, n);
  return cudaSuccess;
}
cudaError_t cudaFree(void* p) {
  auto it = live.find(reinterpret_cast<uintptr_t>(p));
  if (it == live.end()) {
    ++stale;
    return cudaErrorInvalidValue;
  }
  used -= it->second;
  live.erase(it);
  std::free(p);
  return cudaSuccess;
}
cudaError_t cudaHostAlloc(void** p, size_t n, unsigned) { return (*p = std::calloc(1, n)) ? cudaSuccess : cudaErrorMemoryAllocation; }
cudaError_t cudaMallocHost(void** p, size_t n) { return cudaHostAlloc(p, n, 0); }
cudaError_t cudaFreeHost(void* p) { return std::free(p), cudaSuccess; }
cudaError_t cudaPointerGetAttributes(cudaPointerAttributes* a, const void* p) {
  std::memset(a, 0, sizeof(*a));
  a->type = is_live(p) ? cudaMemoryTypeDevice : cudaMemoryTypeUnregistered;
  return cudaSuccess;
}
cudaError_t cudaMemcpyAsync(void* d, const void* s, size_t n, cudaMemcpyKind, cudaStream_t) {
  if (failing_copies > 0) return --failing_copies, cudaErrorMemoryAllocation;
  if (!capturing) std::memmove(d, s, n);
  return cudaSuccess;
}
cudaError_t cudaMemcpy(void* d, const void* s, size_t n, cudaMemcpyKind) { return std::memmove(d, s, n), cudaSuccess; }
cudaError_t cudaMemcpy2DAsync(void* d, size_t dp, const void* s, size_t sp, size_t w, size_t h, cudaMemcpyKind,
                              cudaStream_t) {
  for (size_t i = 0; i < h; ++i) std::memmove(static_cast<char*>(d) + i * dp, static_cast<const char*>(s) + i * sp, w);
  return cudaSuccess;
}
cudaError_t cudaMemsetAsync(void* d, int v, size_t n, cudaStream_t) {
  if (!capturing) std::memset(d, v, n);
  return cudaSuccess;
}
cudaError_t cudaGetDeviceCount(int* n) { return *n = 1, cudaSuccess; }
cudaError_t cudaSetDevice(int) { return cudaSuccess; }
cudaError_t cudaGetDevice(int* d) { return *d = 0, cudaSuccess; }
cudaError_t cudaDeviceGetAttribute(int* v, cudaDeviceAttr, int) { return *v = 148, cudaSuccess; }
cudaError_t cudaGetLastError() { return cudaSuccess; }
const char* cudaGetErrorString(cudaError_t e) { return e == cudaErrorMemoryAllocation ? "out of memory" : "error"; }
cudaError_t cudaStreamCreateWithFlags(cudaStream_t* s, unsigned) { return *s = reinterpret_cast<cudaStream_t>(8), cudaSuccess; }
cudaError_t cudaStreamDestroy(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaEventCreate(cudaEvent_t* e) { return *e = reinterpret_cast<cudaEvent_t>(8), cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaEventSynchronize(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventElapsedTime(float* t, cudaEvent_t, cudaEvent_t) { return *t = 0.f, cudaSuccess; }
cudaError_t cudaStreamBeginCapture(cudaStream_t, cudaStreamCaptureMode) {
  ++captures;
  capturing = true;
  captured.clear();
  return cudaSuccess;
}
cudaError_t cudaStreamEndCapture(cudaStream_t, cudaGraph_t* g) {
  capturing = false;
  *g = reinterpret_cast<cudaGraph_t>(captures);
  return cudaSuccess;
}
cudaError_t cudaGraphInstantiate(cudaGraphExec_t* e, cudaGraph_t g, unsigned long long) {
  *e = reinterpret_cast<cudaGraphExec_t>(g);
  graphs[*e] = captured;
  return cudaSuccess;
}
cudaError_t cudaGraphLaunch(cudaGraphExec_t e, cudaStream_t) {
  ++graph_launches;
  for (const void* b : graphs[e])
    if (!is_live(b)) ++stale;
  return cudaSuccess;
}
cudaError_t cudaGraphDestroy(cudaGraph_t) { return cudaSuccess; }
cudaError_t cudaGraphExecDestroy(cudaGraphExec_t e) { return graphs.erase(e), cudaSuccess; }
}  // extern "C"

// ---- launchers ----------------------------------------------------------------
namespace hb {

size_t scan_exact_smem_bytes(int, int, int, int, int* tv, int* qt, int* qgroup) {
  *tv = 128;
  *qt = 8;
  *qgroup = 32;
  return 1024;
}
int scan_bf16_stages(int) { return 4; }
size_t build_work_tmp_bytes(int nq, int P, int nlist) { return 16 * (static_cast<size_t>(nq) * P + nlist) + 1024; }
size_t cand_segments_tmp_bytes(int nq, int P) { return 16 * static_cast<size_t>(nq) * P + 1024; }
size_t list_offsets_tmp_bytes(int nlist) { return 16 * static_cast<size_t>(nlist) + 1024; }
int assign_kpad(int dpad) { return (dpad + 63) / 64 * 64; }

// Point i goes to list i % nlist.
void launch_l2_argmin(const float*, int nq, const float*, int nrows, int, int32_t* arg, float* dist, cudaStream_t) {
  for (int i = 0; i < nq; ++i) {
    arg[i] = i % nrows;
    if (dist) dist[i] = 0.0f;
  }
}
int launch_assign_tc(const AssignArgs& a, int, cudaStream_t) {
  launch_l2_argmin(a.x, a.n, a.cent, a.nlist, a.dpad, a.arg, a.dist, nullptr);
  return 1;
}
void sort_pairs_u64(uint64_t* keys_in, uint64_t*, uint32_t*, uint32_t*, size_t, int, void*, size_t* bytes, cudaStream_t) {
  if (!keys_in) *bytes = 1024;
}
void launch_list_offsets(const int32_t* assign, size_t n, int nlist, int64_t* off, void*, size_t, cudaStream_t) {
  std::fill(off, off + nlist + 1, 0);
  for (size_t i = 0; i < n; ++i) ++off[assign[i] + 1];
  for (int l = 0; l < nlist; ++l) off[l + 1] += off[l];
}

void launch_scan_exact(const ScanArgs& a, int, cudaStream_t) {
  note("scan_exact", {a.q, a.codes, a.list_q, a.slot_base, a.part});
}
void launch_merge(const uint64_t* part, const int64_t* slot_base, int, int, int, const int64_t* ids, float*, int64_t*,
                  cudaStream_t) {
  note("merge", {part, slot_base, ids});
}
int launch_build_work(const int32_t* probes, int, int, const int64_t*, int, int, int, int32_t* list_cnt, int64_t*,
                      int32_t* list_q, int64_t* item_off, int64_t* slot_base, void* tmp, size_t, cudaStream_t) {
  note("build_work", {probes, list_cnt, list_q, item_off, slot_base, tmp});
  return 1;
}
int launch_seed_bound(const float* q, int, const float*, int, int, const void*, const int64_t*, int, const int64_t*,
                      const int32_t*, const float*, const float*, int, int, uint32_t* thr, int* cnt, cudaStream_t,
                      const int32_t*, int) {
  note("seed", {q, thr, cnt});
  return 1;
}
void launch_scan_bf16(const void*, const TcArgs& a, int, cudaStream_t) {
  note("scan_bf16", {a.q, a.thr, a.cand, a.cand_ub, a.cand_cnt, a.list_q});
  if (!capturing) *a.err = device_err;
}
void launch_rerank_bf16(uint64_t* cand, const uint32_t* cand_ub, const int* cnt, int, int, int, const float* codes,
                        const float* q, int, const int64_t* ids, float*, int64_t*, int* over_list, int* over_n, int* m_out,
                        cudaStream_t) {
  note("rerank", {cand, cand_ub, cnt, codes, q, ids, over_list, over_n, m_out});
  if (!capturing) *over_n = overflow_queries;
}
void launch_cand_scan(const void*, const void*, const CandArgs& a, int, cudaStream_t) {
  note("cand_scan", {a.cand, a.seg, a.qcd, a.list_q});
  if (!capturing) *a.err = device_err;
}
void launch_cand_select(const float* cand, const int64_t* seg, const int32_t*, int, int, int, int, const int64_t*,
                        const float* pcd, const float*, const float*, const float*, int, int, int64_t* rows, float*,
                        int* m_out, int*, int* over_list, int* over_n, cudaStream_t) {
  note("cand_select", {cand, seg, pcd, rows, m_out, over_list});
  if (!capturing && over_list) *over_n = overflow_queries;
}
void launch_cand_exact(const int64_t* rows, const float*, const int* m, const int*, int, int, int, const float* codes,
                       const float* q, int, const int64_t* ids, float*, int64_t*, cudaStream_t) {
  note("cand_exact", {rows, m, codes, q, ids});
}

#include "stubs.inc"

}  // namespace hb
