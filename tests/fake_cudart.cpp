// A CUDA runtime for host-side tests: device memory is host memory, kernels do
// nothing, and an allocation of choice fails.  k_export, from which the solver
// reads the size of the next level, answers with the numbers the test gives.
#include <cuda_runtime_api.h>
#include <stdlib.h>
#include <string.h>
#include <map>
#include <string>
#include <vector>

static std::map<const void *, std::string> g_names;
static cudaError_t g_last = cudaSuccess;
static long g_allocs, g_fail_at = -1;
static int g_idle;           // idle buffer sets of the dense drivers
struct Launch { std::string name; std::vector<void *> args; };
static std::vector<Launch> g_launches;
static std::map<std::string, std::vector<int>> g_ptr_args;   // positions of pointer parameters
static std::vector<int> g_levels;                           // per export: n_cl, arena need, n_sng
static size_t g_at;
static struct { dim3 g, b; size_t s; cudaStream_t st; } g_cfg;

static cudaError_t err(cudaError_t e) { if (e != cudaSuccess) g_last = e; return e; }
static cudaError_t alloc(void **p, size_t n) {
  if (g_allocs++ == g_fail_at) { *p = nullptr; return err(cudaErrorMemoryAllocation); }
  *p = calloc(n ? n : 1, 1);
  return cudaSuccess;
}
extern "C" {
// test controls
void fake_idle(int n) { g_idle = n; }
int mr3_dense_release() { const int n = g_idle; g_idle = 0; return n; }
void fake_fail(long k) { g_allocs = 0; g_fail_at = k; }
long fake_allocs() { return g_allocs; }
void fake_levels(const int *v, int n) { g_levels.assign(v, v + n); g_at = 0; }
void fake_ptr_args(const char *name, const int *at, int n) { g_ptr_args[name].assign(at, at + n); }
void fake_clear() { g_launches.clear(); }
// launches since the last clear as text: the kernel and which pointers were null
const char *fake_launches() {
  static std::string s;
  s.clear();
  for (auto &l : g_launches) {
    s += l.name + ":";
    for (void *q : l.args) s += q ? 'p' : '0';
    s += "\n";
  }
  return s.c_str();
}
// the runtime
void **__cudaRegisterFatBinary(void *) { static void *h; return &h; }
void __cudaRegisterFatBinaryEnd(void **) {}
void __cudaUnregisterFatBinary(void **) {}
void __cudaRegisterFunction(void **, const char *host, char *, const char *name, int, void *, void *,
                            void *, void *, int *) { g_names[host] = name; }
unsigned __cudaPushCallConfiguration(dim3 g, dim3 b, size_t s, cudaStream_t st) {
  g_cfg = {g, b, s, st};
  return 0;
}
cudaError_t __cudaPopCallConfiguration(dim3 *g, dim3 *b, size_t *s, void *st) {
  *g = g_cfg.g; *b = g_cfg.b; *s = g_cfg.s; *(cudaStream_t *)st = g_cfg.st;
  return cudaSuccess;
}
cudaError_t cudaLaunchKernel(const void *f, dim3, dim3, void **args, size_t, cudaStream_t) {
  const std::string &mangled = g_names[f];
  Launch l;
  for (auto &k : g_ptr_args) {
    const std::string tag = std::to_string(k.first.size()) + k.first;
    const size_t at = mangled.find(tag);
    if (at == std::string::npos || (mangled[at + tag.size()] >= 'a' && mangled[at + tag.size()] <= 'z' &&
                                    mangled[at + tag.size()] == '_')) continue;
    l.name = mangled;
    for (int i : k.second) l.args.push_back(*(void **)args[i]);
  }
  g_launches.push_back(l);
  if (mangled.find("8k_export") != std::string::npos && *(void **)args[2]) {
    int *lc = *(int **)args[2], *sc = *(int **)args[4];
    const size_t o = g_at < g_levels.size() ? g_at : 0;
    const bool more = g_at < g_levels.size();
    lc[0] = more ? g_levels[o] : 0; lc[1] = 0;
    *(unsigned long long *)(lc + 2) = more ? g_levels[o + 1] : 0;
    sc[0] = more ? g_levels[o + 2] : 0;
    g_at += 3;
  }
  return cudaSuccess;
}
cudaError_t cudaMalloc(void **p, size_t n) { return alloc(p, n); }
cudaError_t cudaMallocHost(void **p, size_t n) { return alloc(p, n); }
cudaError_t cudaFree(void *p) { free(p); return cudaSuccess; }
cudaError_t cudaFreeHost(void *p) { free(p); return cudaSuccess; }
cudaError_t cudaMemcpy(void *d, const void *s, size_t n, cudaMemcpyKind) { memcpy(d, s, n); return cudaSuccess; }
cudaError_t cudaMemcpyAsync(void *d, const void *s, size_t n, cudaMemcpyKind, cudaStream_t) {
  memcpy(d, s, n);
  return cudaSuccess;
}
cudaError_t cudaMemcpy2DAsync(void *, size_t, const void *, size_t, size_t, size_t, cudaMemcpyKind,
                              cudaStream_t) { return cudaSuccess; }
cudaError_t cudaMemset(void *p, int v, size_t n) { memset(p, v, n); return cudaSuccess; }
cudaError_t cudaMemsetAsync(void *p, int v, size_t n, cudaStream_t) { memset(p, v, n); return cudaSuccess; }
cudaError_t cudaGetLastError() { const cudaError_t e = g_last; g_last = cudaSuccess; return e; }
const char *cudaGetErrorString(cudaError_t) { return "fake error"; }
cudaError_t cudaHostGetDevicePointer(void **d, void *h, unsigned) { *d = h; return cudaSuccess; }
cudaError_t cudaGetDeviceProperties_v2(cudaDeviceProp *p, int) {
  memset(p, 0, sizeof(*p));
  p->multiProcessorCount = 148;
  return cudaSuccess;
}
cudaError_t cudaDeviceGetStreamPriorityRange(int *a, int *b) { *a = *b = 0; return cudaSuccess; }
cudaError_t cudaDeviceSynchronize() { return cudaSuccess; }
cudaError_t cudaSetDevice(int) { return cudaSuccess; }
cudaError_t cudaFuncSetAttribute(const void *, cudaFuncAttribute, int) { return cudaSuccess; }
cudaError_t cudaOccupancyMaxActiveBlocksPerMultiprocessorWithFlags(int *n, const void *, int, size_t,
                                                                  unsigned) { *n = 2; return cudaSuccess; }
static cudaError_t handle(void **p) { *p = (void *)8; return cudaSuccess; }
cudaError_t cudaEventCreate(cudaEvent_t *e) { return handle((void **)e); }
cudaError_t cudaEventCreateWithFlags(cudaEvent_t *e, unsigned) { return handle((void **)e); }
cudaError_t cudaEventDestroy(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventElapsedTime(float *t, cudaEvent_t, cudaEvent_t) { *t = 0; return cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaEventSynchronize(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaStreamCreateWithPriority(cudaStream_t *s, unsigned, int) { return handle((void **)s); }
cudaError_t cudaStreamDestroy(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamWaitEvent(cudaStream_t, cudaEvent_t, unsigned) { return cudaSuccess; }
}
