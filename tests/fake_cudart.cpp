// A CUDA runtime without a device, for tests of the engine's host side on the CPU. The engine's own
// objects are linked against it. Allocations are host memory that is never touched unless the host
// does, copies are copies, launches run nothing; a graph is the list of its launches. Everything is
// written to a log, allocations and graph instantiations can be made to fail, and what the kernels
// would have left for the host (the rates of k_lane_rate, a run's counters) is given by the test.
// A run's kernels are checked: none of the buffers that their parameters name may be null or freed.
#include <cuda_runtime_api.h>
#include <vector_types.h>

#include <cmath>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <deque>
#include <map>
#include <mutex>
#include <string>
#include <vector>

#define __forceinline__ inline
static struct { unsigned x; } blockIdx, threadIdx;
static inline unsigned long long __umul64hi(unsigned long long a, unsigned long long b) {
  return (unsigned long long)(((unsigned __int128)a * b) >> 64);
}
static inline int __ffsll(long long x) { return x ? __builtin_ctzll((unsigned long long)x) + 1 : 0; }
static inline int __clzll(long long x) { return x ? __builtin_clzll((unsigned long long)x) : 64; }
static inline unsigned atomicOr(unsigned *p, unsigned v) { const unsigned o = *p; *p |= v; return o; }
#include "../erdos-strauss_gb300/csrc/es_kernels.cuh"
using namespace es;

namespace {
struct Launch {
  std::string name;
  std::vector<unsigned char> arg;                    // its parameter block, of the run's kernels
  int stream;
};
struct Graph {
  std::vector<Launch> launches;
};
struct Counts {
  unsigned long long surv, chunks;
};

std::recursive_mutex mu;
std::string text;
std::map<void *, size_t> live;
std::map<const void *, std::string> names;
std::map<const void *, int> streams, events;
std::map<int, Graph *> capturing;
std::deque<Counts> counts;                           // of the runs to come
double rate_all = 0, rate_dense = 0;
long fail_alloc = 0, fail_instantiate = 0;
size_t bytes_now = 0;
int bad = 0;
cudaError_t last = cudaSuccess;                     // of the calls so far, until it is asked for

void note(const std::string &s) { text += s + "\n"; }
// The n-th from now fails (a countdown; 0: none).
bool fails(long &n) { return n > 0 && --n == 0; }

cudaError_t take(void **p, size_t n, const char *what) {
  std::lock_guard<std::recursive_mutex> lk(mu);
  *p = nullptr;
  if (fails(fail_alloc)) return last = cudaErrorMemoryAllocation;
  note(std::string(what) + " " + std::to_string(n));
  *p = calloc(n ? n : 1, 1);
  live[*p] = n;
  bytes_now += n;
  return cudaSuccess;
}
cudaError_t give(void *p) {
  std::lock_guard<std::recursive_mutex> lk(mu);
  if (!p) return cudaSuccess;
  const auto it = live.find(p);
  if (it == live.end()) { note("BAD free"); ++bad; return cudaErrorInvalidValue; }
  bytes_now -= it->second;
  live.erase(it);
  free(p);
  return cudaSuccess;
}
// A buffer of at least n bytes that is still there.
void want(const std::string &kernel, const char *field, const void *p, size_t n) {
  auto it = live.upper_bound(const_cast<void *>(p));
  if (p && it != live.begin()) {
    --it;
    if ((const char *)p + n <= (const char *)it->first + it->second) return;
  }
  note("BAD " + kernel + " " + field);
  ++bad;
}
#define WANT(f, n) want(L.name, #f, f, n)
void run(const Launch &L) {
  if (L.name == "k_rows" || L.name == "k_mark_short" || L.name == "k_sift") {
    const RowParams &P = *reinterpret_cast<const RowParams *>(L.arg.data());
    WANT(P.h_hdr, sizeof(BatchHdr)); WANT(P.hdr, sizeof(BatchHdr)); WANT(P.status, 4); WANT(P.ctr, 8 * CTR_OUT);
    if (P.h_hdr && live.count(const_cast<BatchHdr *>(P.h_hdr))) {
      const BatchHdr &H = *P.h_hdr;
      WANT(P.h_win, H.nwin * sizeof(WinDev)); WANT(P.win, H.nwin * sizeof(WinDev)); WANT(P.cnt, H.nwin * sizeof(WinCount));
      WANT(P.h_roww, H.nshort * sizeof(RowWin)); WANT(P.piece, H.npieces * sizeof(Piece));
      WANT(P.pidx, (size_t)H.npieces * P.n1p * sizeof(u16)); WANT(P.rowinfo, H.nrows * sizeof(u32));
    }
    WANT(P.cand, (size_t)P.chunk_cap * 32 * sizeof(uint2)); WANT(P.chunk, (size_t)P.chunk_cap * sizeof(u32));
    WANT(P.surv, P.surv_cap * sizeof(Surv));
  } else if (L.name == "k_mr" || L.name == "k_rung" || L.name == "k_search" || L.name == "k_direct") {
    const TailParams &T = *reinterpret_cast<const TailParams *>(L.arg.data());
    WANT(T.surv, T.cap * sizeof(Surv)); WANT(T.primes, T.cap * sizeof(u32)); WANT(T.direct, T.cap * sizeof(u32));
    WANT(T.recs, T.cap * sizeof(RecDev)); WANT(T.out.recs, T.cap * sizeof(RecDev)); WANT(T.out.ctr, 8 * CTR_OUT);
    WANT(T.out.status, 4); WANT(T.out.cnt, sizeof(WinCount)); WANT(T.cnt, sizeof(WinCount));
    if (L.name == "k_direct" && !bad) {              // the run's results
      const Counts c = counts.empty() ? Counts{0, 0} : counts.front();
      if (!counts.empty()) counts.pop_front();
      memset(T.out.ctr, 0, 8 * CTR_OUT);
      T.out.ctr[1] = c.surv;
      T.out.ctr[10] = c.chunks;
      *T.out.status = 0;
    }
  }
}
}  // namespace

extern "C" {
// ---- the test's side
size_t fake_log(char *buf, size_t cap) {             // the log since the last call
  std::lock_guard<std::recursive_mutex> lk(mu);
  const size_t n = text.size() < cap ? text.size() : cap;
  memcpy(buf, text.data(), n);
  text.erase(0, n);
  return n;
}
void fake_fail(long alloc, long instantiate) {
  std::lock_guard<std::recursive_mutex> lk(mu);
  fail_alloc = alloc;
  fail_instantiate = instantiate;
  counts.clear();
}
void fake_rates(double all, double dense) { rate_all = all; rate_dense = dense; }
void fake_counts(unsigned long long surv, unsigned long long chunks) {
  std::lock_guard<std::recursive_mutex> lk(mu);
  counts.push_back(Counts{surv, chunks});
}
size_t fake_bytes() { std::lock_guard<std::recursive_mutex> lk(mu); return bytes_now; }
int fake_bad() { std::lock_guard<std::recursive_mutex> lk(mu); return bad; }

// ---- the runtime's side
cudaError_t cudaMalloc(void **p, size_t n) { return take(p, n, "device"); }
cudaError_t cudaHostAlloc(void **p, size_t n, unsigned) { return take(p, n, "pinned"); }
cudaError_t cudaMallocHost(void **p, size_t n) { return take(p, n, "pinned"); }
cudaError_t cudaFree(void *p) { return give(p); }
cudaError_t cudaFreeHost(void *p) { return give(p); }
cudaError_t cudaMemcpyAsync(void *d, const void *s, size_t n, cudaMemcpyKind, cudaStream_t) {
  memcpy(d, s, n);
  return cudaSuccess;
}
cudaError_t cudaMemsetAsync(void *, int, size_t, cudaStream_t) { return cudaSuccess; }   // allocations are zero
cudaError_t cudaGetDevice(int *d) { *d = 0; return cudaSuccess; }
cudaError_t cudaSetDevice(int) { return cudaSuccess; }
cudaError_t cudaGetDeviceCount(int *n) { *n = 1; return cudaSuccess; }
cudaError_t cudaDeviceGetAttribute(int *v, cudaDeviceAttr a, int) {
  *v = a == cudaDevAttrMultiProcessorCount ? 152 : 228 * 1024;
  return cudaSuccess;
}
cudaError_t cudaMemGetInfo(size_t *f, size_t *t) { *f = *t = (size_t)280 << 30; return cudaSuccess; }
cudaError_t cudaFuncSetAttribute(const void *, cudaFuncAttribute, int) { return cudaSuccess; }
cudaError_t cudaOccupancyMaxActiveBlocksPerMultiprocessorWithFlags(int *n, const void *, int, size_t, unsigned) {
  *n = 1;
  return cudaSuccess;
}
const char *cudaGetErrorString(cudaError_t) { return "a failure the test asked for"; }
cudaError_t cudaGetLastError() {
  std::lock_guard<std::recursive_mutex> lk(mu);
  const cudaError_t e = last;
  last = cudaSuccess;
  return e;
}
cudaError_t cudaGetSymbolAddress(void **, const void *) { return cudaErrorInvalidValue; }
cudaError_t cudaGetDriverEntryPointByVersion(const char *, void **, unsigned, unsigned long long, cudaDriverEntryPointQueryResult *) {
  return cudaErrorInvalidValue;
}

cudaError_t cudaStreamCreateWithFlags(cudaStream_t *s, unsigned) {
  *s = (cudaStream_t)malloc(8);
  const int n = (int)streams.size();
  streams[*s] = n;
  return cudaSuccess;
}
cudaError_t cudaStreamDestroy(cudaStream_t s) { streams.erase(s); free(s); return cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaEventCreate(cudaEvent_t *e) {
  *e = (cudaEvent_t)malloc(8);
  const int n = (int)events.size();
  events[*e] = n;
  return cudaSuccess;
}
cudaError_t cudaEventDestroy(cudaEvent_t e) { events.erase(e); free(e); return cudaSuccess; }
cudaError_t cudaEventElapsedTime(float *ms, cudaEvent_t, cudaEvent_t) { *ms = 1; return cudaSuccess; }
cudaError_t cudaEventRecordWithFlags(cudaEvent_t e, cudaStream_t s, unsigned flags) {
  std::lock_guard<std::recursive_mutex> lk(mu);
  note("record " + std::to_string(events[e]) + (capturing.count(streams[s]) ? flags == cudaEventRecordExternal ? " node" : " inside" : ""));
  return cudaSuccess;
}
cudaError_t cudaEventRecord(cudaEvent_t e, cudaStream_t s) { return cudaEventRecordWithFlags(e, s, 0); }
cudaError_t cudaStreamWaitEvent(cudaStream_t s, cudaEvent_t e, unsigned) {
  std::lock_guard<std::recursive_mutex> lk(mu);
  note("stream " + std::to_string(streams[s]) + " waits " + std::to_string(events[e]));
  return cudaSuccess;
}
cudaError_t cudaStreamBeginCapture(cudaStream_t s, cudaStreamCaptureMode) {
  std::lock_guard<std::recursive_mutex> lk(mu);
  capturing[streams[s]] = new Graph();
  note("capture " + std::to_string(streams[s]));
  return cudaSuccess;
}
cudaError_t cudaStreamEndCapture(cudaStream_t s, cudaGraph_t *g) {
  std::lock_guard<std::recursive_mutex> lk(mu);
  *g = (cudaGraph_t)capturing[streams[s]];
  capturing.erase(streams[s]);
  return cudaSuccess;
}
cudaError_t cudaStreamGetCaptureInfo(cudaStream_t s, cudaStreamCaptureStatus *status, unsigned long long *id, cudaGraph_t *g,
                                     const cudaGraphNode_t **deps, const cudaGraphEdgeData **edges, size_t *n) {
  std::lock_guard<std::recursive_mutex> lk(mu);
  static const cudaGraphNode_t last_node = nullptr;  // what the stream's next node would follow
  const auto c = capturing.find(streams[s]);
  *status = c == capturing.end() ? cudaStreamCaptureStatusNone : cudaStreamCaptureStatusActive;
  *id = 0;
  *g = c == capturing.end() ? nullptr : (cudaGraph_t)c->second;
  *deps = &last_node;
  *edges = nullptr;
  *n = 1;
  return cudaSuccess;
}
cudaError_t cudaGraphAddEventRecordNode(cudaGraphNode_t *, cudaGraph_t, const cudaGraphNode_t *, size_t n, cudaEvent_t e) {
  std::lock_guard<std::recursive_mutex> lk(mu);
  note("record " + std::to_string(events[e]) + (n == 1 ? " node" : ""));
  return cudaSuccess;
}
cudaError_t cudaGraphInstantiate(cudaGraphExec_t *x, cudaGraph_t g, unsigned long long) {
  std::lock_guard<std::recursive_mutex> lk(mu);
  if (fails(fail_instantiate)) return last = cudaErrorMemoryAllocation;
  note("instantiate");
  *x = (cudaGraphExec_t) new Graph(*(Graph *)g);
  return cudaSuccess;
}
cudaError_t cudaGraphDestroy(cudaGraph_t g) { delete (Graph *)g; return cudaSuccess; }
cudaError_t cudaGraphExecDestroy(cudaGraphExec_t x) { delete (Graph *)x; return cudaSuccess; }
cudaError_t cudaGraphLaunch(cudaGraphExec_t x, cudaStream_t s) {
  std::lock_guard<std::recursive_mutex> lk(mu);
  note("graph on " + std::to_string(streams[s]));
  for (const Launch &l : ((Graph *)x)->launches) run(l);
  return cudaSuccess;
}

void **__cudaRegisterFatBinary(void *) { static void *h; return &h; }
void __cudaRegisterFatBinaryEnd(void **) {}
void __cudaUnregisterFatBinary(void **) {}
void __cudaRegisterVar(void **, char *, char *, const char *, int, size_t, int, int) {}
void __cudaRegisterFunction(void **, const char *host, char *, const char *device, int, uint3 *, uint3 *, dim3 *, dim3 *, int *) {
  std::string n(device);                             // _ZN2es<length><name>...
  if (n.rfind("_ZN2es", 0) == 0) {
    char *end = nullptr;
    const long len = strtol(n.c_str() + 6, &end, 10);
    n = std::string(end, (size_t)len);
  }
  names[host] = n;
}
cudaError_t __cudaGetKernel(cudaKernel_t *k, const void *host) { *k = (cudaKernel_t)host; return cudaSuccess; }
static thread_local struct { dim3 grid, block; size_t smem; cudaStream_t stream; } config;
unsigned __cudaPushCallConfiguration(dim3 grid, dim3 block, size_t smem, cudaStream_t s) {
  config.grid = grid; config.block = block; config.smem = smem; config.stream = s;
  return 0;
}
cudaError_t __cudaPopCallConfiguration(dim3 *grid, dim3 *block, size_t *smem, void *s) {
  *grid = config.grid; *block = config.block; *smem = config.smem; *(cudaStream_t *)s = config.stream;
  return cudaSuccess;
}
cudaError_t __cudaLaunchKernel(cudaKernel_t k, dim3 grid, dim3 block, void **args, size_t, cudaStream_t s) {
  std::lock_guard<std::recursive_mutex> lk(mu);
  Launch l{names[(const void *)k], {}, streams[s]};
  note("launch " + l.name + " " + std::to_string(grid.x) + " " + std::to_string(block.x));
  const bool rows = l.name == "k_rows" || l.name == "k_mark_short" || l.name == "k_sift";
  const bool tail = l.name == "k_mr" || l.name == "k_rung" || l.name == "k_search" || l.name == "k_direct";
  if (rows || tail) {
    const unsigned char *a = (const unsigned char *)args[0];
    l.arg.assign(a, a + (rows ? sizeof(RowParams) : sizeof(TailParams)));
  }
  if (l.name == "k_lane_rate") {                     // sums over the lanes
    const double L = (double)*(const u32 *)args[8];
    double *sum = *(double **)args[9];
    sum[0] = rate_all * L;
    sum[1] = rate_dense * L;
  }
  const auto c = capturing.find(l.stream);
  if (c != capturing.end()) c->second->launches.push_back(l);
  else run(l);
  return cudaSuccess;
}
}  // extern "C"
