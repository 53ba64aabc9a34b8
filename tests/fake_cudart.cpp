// A CUDA runtime without a GPU, preloaded ahead of libcudart by
// test_host_paths.py: device memory is host memory, kernels do not run.  Calls
// can be made to fail, and every launch of a Fock quartet kernel has its
// pointers checked against the live allocations and the quartets it covers
// counted, so that the host's routing, error paths and buffer lifetimes can be
// tested where no kernel could fault.
#include <cuda_runtime_api.h>

#include <algorithm>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <map>
#include <set>
#include <string>
#include <unordered_map>
#include <vector>

#include "dgf_internal.h"
#include "dgf_work.h"

namespace {

std::map<const char *, size_t> g_alloc;  // live device allocations
std::map<const void *, std::string> g_kernel;
std::unordered_map<unsigned long long, int> g_cover;  // quartet -> times covered
std::vector<std::string> g_bad;
std::string g_names;  // kernel families launched since the last reset
long g_launches = 0, g_replays = 0, g_streams = 0, g_malloc_calls = 0;
long g_fail_malloc = -1, g_fail_malloc_n = 0;  // the calls [first, first + n) from now on fail
int g_fail_instantiate = 0;
cudaStream_t g_capturing = nullptr;  // the captured origin stream
bool g_user_capture = false;
struct Copy {
  const char *dst;
  cudaStream_t st;
};
std::vector<Copy> g_pending;                               // copies to the device that may not have landed
std::map<cudaEvent_t, cudaStream_t> g_recorded;            // where an event was recorded last
std::map<cudaStream_t, std::set<cudaStream_t>> g_waits;    // stream -> those whose work it waited for
struct Range {
  const char *begin, *end;
};
std::vector<Range> g_busy;  // what launches that may still run read
cudaError_t g_last = cudaSuccess;
// A captured launch of a quartet kernel, checked and counted at each replay.
struct Launch {
  std::string name;
  dgf::JKArgs args;
  int nchunk;
};
using Graph = std::vector<Launch>;
Graph g_recording;
struct Config {
  dim3 grid, block;
  size_t smem;
  cudaStream_t st;
} g_cfg;

cudaError_t ret(cudaError_t e) {
  if (e != cudaSuccess) g_last = e;
  return e;
}

bool live(const void *p, size_t n) {
  auto it = g_alloc.upper_bound((const char *)p);
  if (!p || it == g_alloc.begin()) return false;
  --it;
  return (const char *)p + n <= it->first + it->second;
}

const char *block(const void *p) {  // the allocation p lies in
  auto it = g_alloc.upper_bound((const char *)p);
  return it == g_alloc.begin() ? nullptr : std::prev(it)->first;
}

void bad(const std::string &name, const char *what) { g_bad.push_back(name + ": " + what); }

// Quartets of a launch of one of the Fock kernels.
void jk_launch(const std::string &name, const dgf::JKArgs &a, int nchunk) {
  using dgf::PairRec;
  int l[4] = {0, 0, 0, 0};
  const size_t at = name.find("ILi");
  if (at == std::string::npos || sscanf(name.c_str() + at, "ILi%dELi%dELi%dELi%dE", l, l + 1, l + 2, l + 3) != 4) return;
  if (a.diag_out) {  // Schwarz factors: made up, from 1 to 1e-6
    if (!live(a.diag_out, a.nbra * 8)) return bad(name, "diag_out");
    for (int i = 0; i < a.nbra; ++i) a.diag_out[i] = std::pow(10.0, -(double)(i % 7));
    return;
  }
  for (const char *k : {"jk_row_stored", "jk_row", "jk_pack", "jk_warp", "jk_thread", "jk_team"})
    if (name.find(k) != std::string::npos) {
      if (g_names.find(k) == std::string::npos) g_names += std::string(k) + " ";
      break;
    }
  if (!live(a.bra, a.nbra * sizeof(PairRec))) return bad(name, "bra pairs");
  auto reads = [](const void *q, size_t n) { g_busy.push_back({(const char *)q, (const char *)q + n}); };
  const bool same = a.same_class;
  const unsigned long long cls = ((l[0] * 4 + l[1]) * 4 + l[2]) * 4 + l[3];
  auto cover = [&](int ib, int ic) {
    if (same && ic + a.ket_off > ib) return;
    if (a.bra[ib].Q * a.ket[ic].Q < a.schwarz_thr) return;
    ++g_cover[((cls << 28 | (unsigned)ib) << 28) | (unsigned)(ic + a.ket_off)];
  };
  if (name.find("jk_row") != std::string::npos || name.find("jk_pack") != std::string::npos) {
    if (!live(a.row_tasks + a.row_task0, (a.row_task1 - a.row_task0) * sizeof(int4))) return bad(name, "row tasks");
    if (!live(a.row_work, nchunk * sizeof(unsigned))) return bad(name, "task counters");
    reads(a.row_tasks + a.row_task0, (a.row_task1 - a.row_task0) * sizeof(int4));
    for (int t = a.row_task0; t < a.row_task1; ++t) {
      const int4 tk = a.row_tasks[t];
      const int nb = tk.y & 0xffff, kend = std::min(tk.w, tk.z + 32 * (tk.y >> 16));
      if (tk.x < 0 || nb < 1 || tk.x + nb > a.nbra || tk.z < 0) return bad(name, "a task's range");
      if (!live(a.row_bra + tk.x, nb * sizeof(int))) return bad(name, "row order");
      if (!live(a.ket + tk.z, (kend - tk.z) * sizeof(PairRec))) return bad(name, "a task's kets");
      for (int r = 0; r < nb; ++r)
        for (int ic = tk.z; ic < kend; ++ic) cover(a.row_bra[tk.x + r], ic);
    }
    return;
  }
  if (!live(a.qoff, (a.nbra + 1) * sizeof(int64_t))) return bad(name, "prefix sums");
  if (a.qoff[a.nbra] < a.nquartet) return bad(name, "prefix sums of another plan");
  reads(a.qoff, (a.nbra + 1) * sizeof(int64_t));
  for (int ib = 0; ib < a.nbra; ++ib)
    for (int64_t q = std::max(a.qoff[ib], a.q_begin); q < std::min(a.qoff[ib + 1], a.nquartet); ++q) {
      const int ic = (int)(q - a.qoff[ib]);
      if (!live(a.ket + ic, sizeof(PairRec))) return bad(name, "a ket");
      cover(ib, ic);
    }
}

}  // namespace

extern "C" {

// ------------------------------------------------------------ test controls
void fake_reset() {
  g_cover.clear();
  g_bad.clear();
  g_names.clear();
  g_launches = 0;
}
long fake_quartets() { return (long)g_cover.size(); }
long fake_not_once() {
  long n = 0;
  for (const auto &e : g_cover) n += e.second != 1;
  return n;
}
long fake_launches() { return g_launches; }
long fake_replays() { return g_replays; }
long fake_streams() { return g_streams; }
long fake_live() { return (long)g_alloc.size(); }
const char *fake_kernels() { return g_names.c_str(); }
const char *fake_bad() { return g_bad.empty() ? "" : g_bad[0].c_str(); }
void fake_fail_malloc(long first, long n) {
  g_fail_malloc = g_malloc_calls + first;
  g_fail_malloc_n = n;
}
long fake_malloc_calls() { return g_malloc_calls; }
void fake_fail_instantiate(int n) { g_fail_instantiate = n; }
void fake_user_capture(int on) { g_user_capture = on != 0; }

// ------------------------------------------------------------------ runtime
cudaError_t cudaGetDeviceCount(int *n) { return *n = 1, cudaSuccess; }
cudaError_t cudaGetDevice(int *d) { return *d = 0, cudaSuccess; }
cudaError_t cudaSetDevice(int) { return cudaSuccess; }
cudaError_t cudaDeviceGetAttribute(int *v, cudaDeviceAttr, int) { return *v = 148, cudaSuccess; }
cudaError_t cudaGetDeviceProperties_v2(cudaDeviceProp *p, int) {
  memset(p, 0, sizeof(*p));
  p->multiProcessorCount = 148;
  return cudaSuccess;
}
const char *cudaGetErrorString(cudaError_t) { return "fake error"; }
cudaError_t cudaGetLastError() {
  const cudaError_t e = g_last;
  g_last = cudaSuccess;
  return e;
}
cudaError_t cudaMalloc(void **p, size_t n) {
  const long call = g_malloc_calls++;
  *p = nullptr;
  if (g_user_capture) return ret(cudaErrorStreamCaptureUnsupported);
  if (g_fail_malloc >= 0 && call >= g_fail_malloc && call < g_fail_malloc + g_fail_malloc_n)
    return ret(cudaErrorMemoryAllocation);
  char *q = (char *)aligned_alloc(256, (n + 255) / 256 * 256);
  memset(q, 0, n);
  g_alloc[q] = n;
  *p = q;
  return cudaSuccess;
}
cudaError_t cudaFree(void *p) {
  if (!p) return cudaSuccess;
  if (!g_alloc.erase((const char *)p)) {
    g_bad.push_back("cudaFree of a pointer that is not live");
    return ret(cudaErrorInvalidValue);
  }
  g_busy.clear();  // waits for the device
  g_pending.clear();
  free(p);
  return cudaSuccess;
}
// From pageable memory cudaMemcpy returns once the data is staged, and between
// device buffers at once: kernels on streams that do not wait for the legacy
// stream may find the old contents.
static void copied(void *d, size_t n, cudaMemcpyKind kind, cudaStream_t st) {
  if (kind == cudaMemcpyDeviceToHost || !n) return;
  for (const Range &r : g_busy)
    if ((const char *)d < r.end && (const char *)d + n > r.begin) {
      g_bad.push_back("a copy over what a running build reads");
      break;
    }
  g_pending.push_back({(const char *)d, st});
}
cudaError_t cudaMemcpy(void *d, const void *s, size_t n, cudaMemcpyKind kind) {
  if (g_user_capture) return ret(cudaErrorStreamCaptureUnsupported);
  if (n) memcpy(d, s, n);
  copied(d, n, kind, nullptr);
  return cudaSuccess;
}
cudaError_t cudaMemcpyAsync(void *d, const void *s, size_t n, cudaMemcpyKind kind, cudaStream_t st) {
  if (n) memcpy(d, s, n);
  copied(d, n, kind, st);
  return cudaSuccess;
}
cudaError_t cudaDeviceSynchronize() {
  g_busy.clear();
  g_pending.clear();
  return cudaSuccess;
}
cudaError_t cudaMemsetAsync(void *d, int v, size_t n, cudaStream_t) {
  if (n && !live(d, n))
    g_bad.push_back("memset outside the live allocations");
  else if (n && !g_capturing)
    memset(d, v, n);
  return cudaSuccess;
}
cudaError_t cudaStreamCreateWithFlags(cudaStream_t *s, unsigned) {
  ++g_streams;
  return *s = (cudaStream_t)malloc(8), cudaSuccess;
}
cudaError_t cudaStreamDestroy(cudaStream_t s) {
  --g_streams;
  free(s);
  return cudaSuccess;
}
cudaError_t cudaStreamSynchronize(cudaStream_t s) {
  g_pending.erase(std::remove_if(g_pending.begin(), g_pending.end(), [s](const Copy &c) { return c.st == s; }),
                  g_pending.end());
  return cudaSuccess;
}
cudaError_t cudaStreamWaitEvent(cudaStream_t s, cudaEvent_t e, unsigned) {
  g_waits[s].insert(g_recorded[e]);
  return cudaSuccess;
}
cudaError_t cudaEventCreate(cudaEvent_t *e) { return *e = (cudaEvent_t)malloc(8), cudaSuccess; }
cudaError_t cudaEventCreateWithFlags(cudaEvent_t *e, unsigned) { return *e = (cudaEvent_t)malloc(8), cudaSuccess; }
cudaError_t cudaEventDestroy(cudaEvent_t e) { return free(e), cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t e, cudaStream_t s) { return g_recorded[e] = s, cudaSuccess; }
cudaError_t cudaEventSynchronize(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventElapsedTime(float *ms, cudaEvent_t, cudaEvent_t) { return *ms = 1.f, cudaSuccess; }
cudaError_t cudaStreamIsCapturing(cudaStream_t s, cudaStreamCaptureStatus *c) {
  *c = (g_user_capture || (g_capturing && s == g_capturing)) ? cudaStreamCaptureStatusActive : cudaStreamCaptureStatusNone;
  return cudaSuccess;
}
cudaError_t cudaStreamBeginCapture(cudaStream_t s, cudaStreamCaptureMode) {
  g_recording.clear();
  return g_capturing = s, cudaSuccess;
}
cudaError_t cudaStreamEndCapture(cudaStream_t, cudaGraph_t *g) {
  g_capturing = nullptr;
  return *g = (cudaGraph_t) new Graph(g_recording), cudaSuccess;
}
cudaError_t cudaGraphInstantiate(cudaGraphExec_t *x, cudaGraph_t g, unsigned long long) {
  *x = nullptr;
  if (g_fail_instantiate > 0) {
    --g_fail_instantiate;
    return ret(cudaErrorMemoryAllocation);
  }
  return *x = (cudaGraphExec_t) new Graph(*(Graph *)g), cudaSuccess;
}
cudaError_t cudaGraphLaunch(cudaGraphExec_t x, cudaStream_t) {
  ++g_replays;
  for (const Launch &l : *(Graph *)x) jk_launch(l.name, l.args, l.nchunk);
  return cudaSuccess;
}
cudaError_t cudaGraphDestroy(cudaGraph_t g) { return delete (Graph *)g, cudaSuccess; }
cudaError_t cudaGraphExecDestroy(cudaGraphExec_t x) { return delete (Graph *)x, cudaSuccess; }
cudaError_t cudaGetSymbolAddress(void **p, const void *s) { return *p = (void *)s, cudaSuccess; }
cudaError_t cudaFuncSetAttribute(const void *, cudaFuncAttribute, int) { return cudaSuccess; }

cudaError_t cudaLaunchKernel(const void *f, dim3 grid, dim3, void **args, size_t, cudaStream_t st) {
  ++g_launches;
  const auto it = g_kernel.find(f);
  if (it == g_kernel.end()) return ret(cudaErrorInvalidDeviceFunction);
  if (it->second.find("work_combine_kernel") != std::string::npos) {
    const dgf::WorkMaps &m = *(const dgf::WorkMaps *)args[0];
    for (int k = 1; k <= 2; ++k)
      if (!live(*(const double **)args[k], m.w_elem[m.nmol] * sizeof(double))) bad(it->second, "half Fock matrices");
  }
  if (it->second.find("jk_") != std::string::npos && it->second.find("JKArgs") != std::string::npos) {
    const dgf::JKArgs &a = *(const dgf::JKArgs *)args[0];
    const void *reads[] = {a.bra,  a.ket,  a.pp,   a.boys,  a.sph,       a.qoff,    a.blk_gab,
                           a.ks_i, a.ks_q, a.ks_pp, a.row_bra, a.row_tasks, a.boys_fine};
    for (const Copy &c : g_pending)
      for (const void *r : reads)
        if (c.st != st && !g_waits[st].count(c.st) && r && block(r) == block(c.dst))
          g_bad.push_back(it->second + ": on a stream that does not wait for an upload");
    if (g_capturing)
      g_recording.push_back(Launch{it->second, a, (int)grid.y});
    else
      jk_launch(it->second, a, (int)grid.y);
  }
  return cudaSuccess;
}

// ------------------------------------------------- the compiler's entry points
void **__cudaRegisterFatBinary(void *) { return (void **)malloc(8); }
void __cudaRegisterFatBinaryEnd(void **) {}
void __cudaUnregisterFatBinary(void **) {}
void __cudaRegisterFunction(void **, const char *host, char *, const char *name, int, uint3 *, uint3 *, dim3 *, dim3 *,
                            int *) {
  g_kernel[host] = name;
}
void __cudaRegisterVar(void **, char *, char *, const char *, int, size_t, int, int) {}
unsigned __cudaPushCallConfiguration(dim3 grid, dim3 block, size_t smem, struct CUstream_st *st) {
  g_cfg = Config{grid, block, smem, st};
  return 0;
}
cudaError_t __cudaPopCallConfiguration(dim3 *grid, dim3 *block, size_t *smem, void *st) {
  *grid = g_cfg.grid;
  *block = g_cfg.block;
  *smem = g_cfg.smem;
  *(cudaStream_t *)st = g_cfg.st;
  return cudaSuccess;
}

}  // extern "C"
