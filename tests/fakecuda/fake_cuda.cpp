// fake_cuda.cpp -- a CUDA runtime on the host for tests of the library's
// host-side code without a GPU (tests/fakecuda/__init__.py links it with the
// library's objects in place of the runtime).  Device memory is host memory,
// copies are memcpy, launches are recorded and not run, and the test plants
// failures of allocations, copies and attribute calls.  Like the real runtime,
// a launch with more than 48 KB of dynamic shared memory needs the kernel's
// attribute on the current device.
#include <cuda.h>
#include <cuda_runtime.h>

#include <cstdlib>
#include <cstring>
#include <map>
#include <set>
#include <string>
#include <vector>

// the paired stage kernels' argument (paired_work.cu)
extern "C" const int4 *paired_items(const void *work, int list, int *n);
extern "C" void paired_item(const int4 *packed, int *v);

namespace {

struct Launch {
  int list;                 // the kernel's (stage_pair_impl.cuh)
  std::vector<int4> items;  // the list it walks
};
constexpr int DEVICES = 3;
int sms = 148;
int device = 0;
cudaError_t last = cudaSuccess;
std::map<std::string, std::pair<int, int>> fail;  // call -> calls to pass, then the error
std::map<const void *, size_t> memory;
std::set<const void *> fresh;  // allocated (zeros) and not yet written
std::set<std::pair<int, const void *>> attrs;
std::vector<Launch> launches;
std::vector<std::pair<std::string, dim3>> grids;  // of every launch
std::map<const void *, std::string> names;  // kernels
dim3 cfg_grid, cfg_block;
size_t cfg_smem;
cudaStream_t cfg_stream;

cudaError_t ret(cudaError_t e) {
  if (e != cudaSuccess) last = e;
  return e;
}
cudaError_t planted(const char *call) {
  auto it = fail.find(call);
  if (it == fail.end() || it->second.first-- > 0) return cudaSuccess;
  const cudaError_t e = (cudaError_t)it->second.second;
  fail.erase(it);
  return e;
}
// a distinct non-null handle
void *handle() {
  static std::vector<char *> all;
  all.push_back(new char);
  return all.back();
}
CUresult encode(CUtensorMap *m, CUtensorMapDataType, cuuint32_t, void *, const cuuint64_t *,
                const cuuint64_t *, const cuuint32_t *, const cuuint32_t *,
                CUtensorMapInterleave, CUtensorMapSwizzle, CUtensorMapL2promotion,
                CUtensorMapFloatOOBfill) {
  std::memset(m, 0, sizeof(*m));
  return CUDA_SUCCESS;
}

}  // namespace

extern "C" {

// ------------------------------ the test's side ----------------------------
// (attributes stay: the library sets them once)
void fake_reset() {
  device = 0;
  last = cudaSuccess;
  fail.clear();
  launches.clear();
  grids.clear();
  sms = 148;
}
void fake_sms(int n) { sms = n; }
// the call after `pass` more of them fails once with error e
void fake_fail(const char *call, int pass, int e) { fail[call] = {pass, e}; }
int fake_blocks() { return (int)memory.size(); }
void fake_clear_launches() {
  launches.clear();
  grids.clear();
}
// grid.z of the launches of the kernel so named: all the same, or -1
int fake_grid_z(const char *kernel) {
  int z = -1;
  for (const auto &g : grids)
    if (g.first.find(kernel) != std::string::npos) {
      if (z >= 0 && z != (int)g.second.z) return -1;
      z = (int)g.second.z;
    }
  return z;
}
// launches of the paired stage kernels so far: list and items
// (i0, j0, z0, z1, model, part of each)
int fake_launches() { return (int)launches.size(); }
int fake_list(int q) { return launches[q].list; }
int fake_items(int q) { return (int)launches[q].items.size(); }
void fake_get_items(int q, int *v) {
  for (const int4 &t : launches[q].items) paired_item(&t, v), v += 6;
}
// the last (unread) error, as cudaPeekAtLastError
int fake_last() { return (int)last; }

// ------------------------------ the runtime --------------------------------
void **__cudaRegisterFatBinary(void *) { return (void **)handle(); }
void __cudaRegisterFatBinaryEnd(void **) {}
char __cudaInitModule(void **) { return 1; }
void __cudaUnregisterFatBinary(void **) {}
void __cudaRegisterVar(void **, char *, char *, const char *, int, size_t, int, int) {}
void __cudaRegisterFunction(void **, const char *f, char *, const char *name, int, uint3 *, uint3 *,
                            dim3 *, dim3 *, int *) {
  names[f] = name;
}
unsigned __cudaPushCallConfiguration(dim3 grid, dim3 block, size_t smem, cudaStream_t s) {
  cfg_grid = grid, cfg_block = block, cfg_smem = smem, cfg_stream = s;
  return 0;
}
cudaError_t __cudaPopCallConfiguration(dim3 *grid, dim3 *block, size_t *smem, void *s) {
  *grid = cfg_grid, *block = cfg_block, *smem = cfg_smem, *(cudaStream_t *)s = cfg_stream;
  return cudaSuccess;
}
const char *cudaGetErrorString(cudaError_t e) {
  return e == cudaSuccess                ? "no error"
         : e == cudaErrorMemoryAllocation ? "out of memory"
         : e == cudaErrorIllegalAddress   ? "an illegal memory access"
                                          : "another error";
}
cudaError_t cudaGetDeviceCount(int *n) { *n = DEVICES; return cudaSuccess; }
cudaError_t cudaGetDevice(int *d) { *d = device; return cudaSuccess; }
cudaError_t cudaSetDevice(int d) { device = d; return cudaSuccess; }
cudaError_t cudaGetLastError() {
  const cudaError_t e = last;
  last = cudaSuccess;
  return e;
}
cudaError_t cudaDeviceGetAttribute(int *v, cudaDeviceAttr, int) {
  *v = sms;  // (the one attribute the library reads)
  return cudaSuccess;
}
cudaError_t cudaMalloc(void **p, size_t n) {
  *p = nullptr;
  if (const cudaError_t e = planted("cudaMalloc")) return ret(e);
  void *q = std::calloc(1, n ? n : 1);
  if (!q) return ret(cudaErrorMemoryAllocation);
  memory[q] = n;
  fresh.insert(q);
  *p = q;
  return cudaSuccess;
}
cudaError_t cudaHostAlloc(void **p, size_t n, unsigned) {
  *p = std::calloc(1, n);
  return cudaSuccess;
}
cudaError_t cudaFree(void *p) {
  if (!p) return cudaSuccess;
  if (!memory.erase(p)) return ret(cudaErrorInvalidValue);  // not (or no longer) allocated
  fresh.erase(p);
  std::free(p);
  return cudaSuccess;
}
cudaError_t cudaMemcpy(void *d, const void *s, size_t n, cudaMemcpyKind) {
  if (const cudaError_t e = planted("cudaMemcpy")) return ret(e);
  fresh.erase(d);
  std::memcpy(d, s, n);
  return cudaSuccess;
}
cudaError_t cudaMemcpyAsync(void *d, const void *s, size_t n, cudaMemcpyKind,
                                   cudaStream_t) {
  fresh.erase(d);
  std::memcpy(d, s, n);
  return cudaSuccess;
}
cudaError_t cudaMemset(void *d, int v, size_t n) {
  // the first one of a block has nothing to do (and leaves its pages untouched)
  if (v != 0 || !fresh.erase(d)) std::memset(d, v, n);
  return cudaSuccess;
}
cudaError_t cudaPointerGetAttributes(cudaPointerAttributes *a, const void *p) {
  std::memset(a, 0, sizeof(*a));
  a->type = memory.count(p) ? cudaMemoryTypeDevice : cudaMemoryTypeUnregistered;
  return cudaSuccess;
}
cudaError_t cudaFuncSetAttribute(const void *f, cudaFuncAttribute, int) {
  if (const cudaError_t e = planted("cudaFuncSetAttribute")) return ret(e);
  attrs.insert({device, f});
  return cudaSuccess;
}
cudaError_t cudaOccupancyMaxActiveBlocksPerMultiprocessorWithFlags(int *n, const void *f,
                                                                          int, size_t smem,
                                                                          unsigned) {
  *n = (smem > 48 * 1024 && !attrs.count({device, f})) ? 0 : 3;
  return cudaSuccess;
}
cudaError_t cudaLaunchKernel(const void *f, dim3 grid, dim3, void **args, size_t smem,
                                    cudaStream_t) {
  if (grid.x == 0 || (smem > 48 * 1024 && !attrs.count({device, f})))
    return ret(cudaErrorInvalidValue);
  const std::string &n = names[f];
  grids.push_back({n, grid});
  if (n.find("pair_kernel") != std::string::npos) {
    // template arguments <T, X, Y, Z, KIND, batched, LIST>
    const int list = n[n.find("ELi", n.find("Lb")) + 3] - '0';
    int k = 0;
    const int4 *it = paired_items(args[3], list, &k);
    if (k < 1 || !memory.count(it)) return ret(cudaErrorInvalidValue);
    launches.push_back({list, {it, it + k}});
  }
  return cudaSuccess;
}
cudaError_t cudaGetDriverEntryPointByVersion(const char *, void **p, unsigned,
                                                    unsigned long long,
                                                    cudaDriverEntryPointQueryResult *q) {
  *p = (void *)encode;
  if (q) *q = cudaDriverEntryPointSuccess;
  return cudaSuccess;
}
cudaError_t cudaGetSymbolAddress(void **p, const void *s) {
  *p = const_cast<void *>(s);
  return cudaSuccess;
}
cudaError_t cudaStreamCreateWithFlags(cudaStream_t *s, unsigned) {
  *s = (cudaStream_t)handle();
  return cudaSuccess;
}
cudaError_t cudaStreamDestroy(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamQuery(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamWaitEvent(cudaStream_t, cudaEvent_t, unsigned) { return cudaSuccess; }
cudaError_t cudaEventCreate(cudaEvent_t *e) {
  *e = (cudaEvent_t)handle();
  return cudaSuccess;
}
cudaError_t cudaEventCreateWithFlags(cudaEvent_t *e, unsigned) {
  *e = (cudaEvent_t)handle();
  return cudaSuccess;
}
cudaError_t cudaEventDestroy(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaEventSynchronize(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventElapsedTime(float *ms, cudaEvent_t, cudaEvent_t) {
  *ms = 1.f;
  return cudaSuccess;
}
cudaError_t cudaStreamBeginCapture(cudaStream_t, cudaStreamCaptureMode) {
  return cudaSuccess;
}
cudaError_t cudaStreamEndCapture(cudaStream_t, cudaGraph_t *g) {
  *g = (cudaGraph_t)handle();
  return cudaSuccess;
}
cudaError_t cudaGraphInstantiate(cudaGraphExec_t *x, cudaGraph_t, unsigned long long) {
  *x = (cudaGraphExec_t)handle();
  return cudaSuccess;
}
cudaError_t cudaGraphLaunch(cudaGraphExec_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaGraphExecDestroy(cudaGraphExec_t) { return cudaSuccess; }
cudaError_t cudaGraphDestroy(cudaGraph_t) { return cudaSuccess; }

}  // extern "C"
