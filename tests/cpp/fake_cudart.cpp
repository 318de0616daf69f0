// A CUDA runtime without a GPU, for tests of the library's host code on the
// CPU: device memory is host memory, kernels do nothing, and every launch is
// recorded by its kernel's name. Linked with the library's own objects in place
// of the runtime (tests/fake_gpu.py).
//
// It keeps the rules that the host code has to respect: more than 48 KB of
// dynamic shared memory needs the opt-in of that kernel on the current device,
// a refused launch leaves its error behind and no node in a graph under
// capture, and a copy may not run past its allocation.
#include <cuda.h>
#include <cuda_runtime.h>

#include <cstdlib>
#include <cstring>
#include <map>
#include <set>
#include <string>
#include <utility>
#include <vector>

namespace {
struct Block {
  size_t bytes;
  int device;
};
std::map<const char *, Block> g_mem;  // by first byte
std::map<const void *, std::string> g_name;
std::map<std::pair<int, const void *>, int> g_smem;  // the opt-ins
std::map<std::string, double> g_cost;                // ms per launch, by a part of the name
std::set<std::string> g_refused;
std::string g_log;
std::vector<std::string> *g_capture = nullptr;
cudaError_t g_last = cudaSuccess;
int g_device = 0, g_sms = 152, g_raster_bad = 0;
long long g_load = -1;
double g_clock = 0;

cudaError_t fail(cudaError_t e) {
  if (e != cudaSuccess) g_last = e;
  return e;
}
const std::string &name_of(const void *f) {
  static const std::string none = "?";
  auto it = g_name.find(f);
  return it == g_name.end() ? none : it->second;
}
const Block *block_of(const void *p, size_t *left) {
  auto it = g_mem.upper_bound(static_cast<const char *>(p));
  if (it == g_mem.begin()) return nullptr;
  --it;
  const size_t at = static_cast<const char *>(p) - it->first;
  if (at >= it->second.bytes) return nullptr;
  *left = it->second.bytes - at;
  return &it->second;
}
void run(const std::string &name) {
  g_log += name + "\n";
  double ms = 1e-3;
  for (auto &c : g_cost)
    if (name.find(c.first) != std::string::npos) ms = c.second;
  g_clock += ms;
}
// the heads of two kernels' parameters: dcg::ClusterSolve and dcg::SolveBatch
struct ClusterArgs {
  int n, csize, sweeps, prolong;
  long long limit;
  int hi[16], lo[16];
};
struct SolveArgs {
  int n, prolong;
  void *planes[6];
  unsigned long long arena[16];
  int lev[16];
  long long cl_max[16], res_max;
};
// which levels a solver takes, behind its name: ":highest-lowest" of every
// member, or ":level>blocks that it leaves", and the launch's "<blocks that it leaves"
std::string levels_of(const std::string &name, void **args) {
  std::string t;
  if (name.find("k_cluster_solve") != std::string::npos) {
    const ClusterArgs &a = *static_cast<const ClusterArgs *>(args[0]);
    for (int i = 0; i < a.n; i++) t += ":" + std::to_string(a.hi[i]) + "-" + std::to_string(a.lo[i]);
  }
  if (name.find("k_resident_solve") != std::string::npos || name.find("k_level_solve_batch") != std::string::npos) {
    const SolveArgs &a = *static_cast<const SolveArgs *>(args[0]);
    for (int i = 0; i < a.n; i++) t += ":" + std::to_string(a.lev[i]) + ">" + std::to_string(a.cl_max[i]);
    t += "<" + std::to_string(a.res_max);
  }
  return t;
}
cudaError_t launch(const void *f, size_t smem, void **args) {
  const std::string name = name_of(f) + levels_of(name_of(f), args);
  for (auto &r : g_refused)
    if (name.find(r) != std::string::npos) return fail(cudaErrorLaunchOutOfResources);
  if (smem > 48 * 1024) {
    auto it = g_smem.find({g_device, f});
    if (it == g_smem.end() || (size_t)it->second < smem) return fail(cudaErrorInvalidValue);
  }
  if (name.find("k_check_raster") != std::string::npos)  // (Dev, level, bad)
    **static_cast<unsigned **>(args[2]) = (unsigned)g_raster_bad;
  if (g_capture) g_capture->push_back(name);
  else run(name);
  return cudaSuccess;
}
cudaError_t copy(void *dst, const void *src, size_t n) {
  size_t left = 0;
  if ((block_of(dst, &left) && left < n) || (block_of(src, &left) && left < n)) return fail(cudaErrorInvalidValue);
  std::memcpy(dst, src, n);
  if (g_load >= 0 && n == sizeof g_load && block_of(src, &left)) std::memcpy(dst, &g_load, n);
  return cudaSuccess;
}
cudaError_t fill(void *dst, int v, size_t n) {
  size_t left = 0;
  if (block_of(dst, &left) && left < n) return fail(cudaErrorInvalidValue);
  std::memset(dst, v, n);
  return cudaSuccess;
}
}  // namespace

extern "C" {
// ---------------------------------------------------------------- the tests' side
const char *fake_log(void) { return g_log.c_str(); }  // launches since the last fake_clear, a name per line
void fake_clear(void) { g_log.clear(); }
void fake_refuse(const char *part) {  // launches of kernels with this in their name too; "": none
  if (*part) g_refused.insert(part);
  else g_refused.clear();
}
void fake_cost(const char *part, double ms) { g_cost[part] = ms; }
long long fake_held(void) {  // bytes allocated
  long long n = 0;
  for (auto &b : g_mem) n += (long long)b.second.bytes;
  return n;
}
void fake_sms(int n) { g_sms = n; }
void fake_raster_bad(int bad) { g_raster_bad = bad; }
void fake_load(long long blocks) { g_load = blocks; }  // what a read of one level's load gives; -1: what is there

// ---------------------------------------------------------------- the runtime
cudaError_t cudaPeekAtLastError(void) { return g_last; }
cudaError_t cudaGetLastError(void) {
  const cudaError_t e = g_last;
  g_last = cudaSuccess;
  return e;
}
const char *cudaGetErrorString(cudaError_t e) { return e == cudaSuccess ? "no error" : "refused"; }
cudaError_t cudaGetDevice(int *d) {
  *d = g_device;
  return cudaSuccess;
}
cudaError_t cudaSetDevice(int d) {
  g_device = d;
  return cudaSuccess;
}
cudaError_t cudaDeviceGetAttribute(int *v, enum cudaDeviceAttr a, int) {
  *v = a == cudaDevAttrMultiProcessorCount ? g_sms : 0;
  return cudaSuccess;
}
cudaError_t cudaMalloc(void **p, size_t n) {
  *p = std::aligned_alloc(256, (n + 511) / 256 * 256);
  std::memset(*p, 0, n);
  g_mem[static_cast<char *>(*p)] = {n, g_device};
  return cudaSuccess;
}
cudaError_t cudaFree(void *p) {
  g_mem.erase(static_cast<char *>(p));
  std::free(p);
  return cudaSuccess;
}
cudaError_t cudaHostAlloc(void **p, size_t n, unsigned) {
  *p = std::calloc(n, 1);
  return cudaSuccess;
}
cudaError_t cudaFreeHost(void *p) {
  std::free(p);
  return cudaSuccess;
}
cudaError_t cudaMemcpy(void *d, const void *s, size_t n, enum cudaMemcpyKind) { return copy(d, s, n); }
cudaError_t cudaMemcpyAsync(void *d, const void *s, size_t n, enum cudaMemcpyKind, cudaStream_t) { return copy(d, s, n); }
cudaError_t cudaMemset(void *d, int v, size_t n) { return fill(d, v, n); }
cudaError_t cudaMemsetAsync(void *d, int v, size_t n, cudaStream_t) { return fill(d, v, n); }
cudaError_t cudaPointerGetAttributes(struct cudaPointerAttributes *a, const void *p) {
  size_t left;
  const Block *b = block_of(p, &left);
  std::memset(a, 0, sizeof *a);
  a->type = b ? cudaMemoryTypeDevice : cudaMemoryTypeUnregistered;
  a->device = b ? b->device : -1;
  return cudaSuccess;
}
static CUresult address_range(CUdeviceptr *base, size_t *size, CUdeviceptr p) {
  size_t left;
  const Block *b = block_of(reinterpret_cast<const void *>(p), &left);
  if (!b) return CUDA_ERROR_NOT_FOUND;
  *base = p + left - b->bytes;
  *size = b->bytes;
  return CUDA_SUCCESS;
}
cudaError_t cudaGetDriverEntryPointByVersion(const char *symbol, void **f, unsigned, unsigned long long,
                                             enum cudaDriverEntryPointQueryResult *) {
  *f = std::strcmp(symbol, "cuMemGetAddressRange") ? nullptr : reinterpret_cast<void *>(address_range);
  return cudaSuccess;
}
cudaError_t cudaGetSymbolAddress(void **p, const void *s) {
  *p = const_cast<void *>(s);
  return cudaSuccess;
}
cudaError_t cudaStreamCreateWithFlags(cudaStream_t *s, unsigned) {
  *s = reinterpret_cast<cudaStream_t>(std::malloc(1));
  return cudaSuccess;
}
cudaError_t cudaStreamDestroy(cudaStream_t s) {
  std::free(s);
  return cudaSuccess;
}
cudaError_t cudaStreamSynchronize(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaEventCreate(cudaEvent_t *e) {
  *e = reinterpret_cast<cudaEvent_t>(new double(0));
  return cudaSuccess;
}
cudaError_t cudaEventDestroy(cudaEvent_t e) {
  delete reinterpret_cast<double *>(e);
  return cudaSuccess;
}
cudaError_t cudaEventRecord(cudaEvent_t e, cudaStream_t) {
  *reinterpret_cast<double *>(e) = g_clock;
  return cudaSuccess;
}
cudaError_t cudaEventSynchronize(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventElapsedTime(float *ms, cudaEvent_t a, cudaEvent_t b) {
  *ms = (float)(*reinterpret_cast<double *>(b) - *reinterpret_cast<double *>(a));
  return cudaSuccess;
}
cudaError_t cudaStreamBeginCapture(cudaStream_t s, enum cudaStreamCaptureMode) {
  if (!s) return fail(cudaErrorStreamCaptureUnsupported);  // the legacy stream
  g_capture = new std::vector<std::string>;
  return cudaSuccess;
}
cudaError_t cudaStreamEndCapture(cudaStream_t, cudaGraph_t *g) {
  *g = reinterpret_cast<cudaGraph_t>(g_capture);
  g_capture = nullptr;
  return cudaSuccess;
}
cudaError_t cudaGraphGetNodes(cudaGraph_t g, cudaGraphNode_t *, size_t *n) {
  *n = reinterpret_cast<std::vector<std::string> *>(g)->size();
  return cudaSuccess;
}
cudaError_t cudaGraphNodeGetType(cudaGraphNode_t, enum cudaGraphNodeType *t) {
  *t = cudaGraphNodeTypeKernel;
  return cudaSuccess;
}
cudaError_t cudaGraphInstantiate(cudaGraphExec_t *x, cudaGraph_t g, unsigned long long) {
  *x = reinterpret_cast<cudaGraphExec_t>(new std::vector<std::string>(*reinterpret_cast<std::vector<std::string> *>(g)));
  return cudaSuccess;
}
cudaError_t cudaGraphDestroy(cudaGraph_t g) {
  delete reinterpret_cast<std::vector<std::string> *>(g);
  return cudaSuccess;
}
cudaError_t cudaGraphExecDestroy(cudaGraphExec_t x) {
  delete reinterpret_cast<std::vector<std::string> *>(x);
  return cudaSuccess;
}
cudaError_t cudaGraphLaunch(cudaGraphExec_t x, cudaStream_t) {
  for (auto &n : *reinterpret_cast<std::vector<std::string> *>(x)) run(n);
  return cudaSuccess;
}
cudaError_t cudaFuncSetAttribute(const void *f, enum cudaFuncAttribute a, int v) {
  if (a == cudaFuncAttributeMaxDynamicSharedMemorySize) g_smem[{g_device, f}] = v;
  return cudaSuccess;
}
cudaError_t cudaOccupancyMaxActiveBlocksPerMultiprocessorWithFlags(int *n, const void *, int, size_t, unsigned) {
  *n = 2;
  return cudaSuccess;
}
cudaError_t cudaOccupancyMaxActiveClusters(int *n, const void *, const cudaLaunchConfig_t *) {
  *n = 4;
  return cudaSuccess;
}
cudaError_t cudaLaunchKernelExC(const cudaLaunchConfig_t *c, const void *f, void **args) {
  return launch(f, c->dynamicSmemBytes, args);
}
cudaError_t cudaLaunchCooperativeKernel(const void *f, dim3, dim3, void **args, size_t smem, cudaStream_t) {
  return launch(f, smem, args);
}

// ---------------------------------------------------------------- the compiler's calls
static struct {
  dim3 grid, block;
  size_t smem;
  void *stream;
} g_config;
unsigned __cudaPushCallConfiguration(dim3 grid, dim3 block, size_t smem, void *stream) {
  g_config = {grid, block, smem, stream};
  return 0;
}
cudaError_t __cudaPopCallConfiguration(dim3 *grid, dim3 *block, size_t *smem, void *stream) {
  *grid = g_config.grid;
  *block = g_config.block;
  *smem = g_config.smem;
  *static_cast<void **>(stream) = g_config.stream;
  return cudaSuccess;
}
cudaError_t __cudaGetKernel(cudaKernel_t *k, const void *f) {
  *k = reinterpret_cast<cudaKernel_t>(const_cast<void *>(f));
  return cudaSuccess;
}
cudaError_t __cudaLaunchKernel(cudaKernel_t k, dim3, dim3, void **args, size_t smem, cudaStream_t) {
  return launch(reinterpret_cast<const void *>(k), smem, args);
}
void **__cudaRegisterFatBinary(void *) {
  static void *handle;
  return &handle;
}
void __cudaRegisterFatBinaryEnd(void **) {}
void __cudaUnregisterFatBinary(void **) {}
void __cudaRegisterFunction(void **, const char *host, char *, const char *name, int, uint3 *, uint3 *, dim3 *, dim3 *,
                            int *) {
  g_name[host] = name;
}
void __cudaRegisterVar(void **, char *, char *, const char *, int, size_t, int, int) {}
}
