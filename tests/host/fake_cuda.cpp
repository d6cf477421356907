// A CUDA runtime without a GPU: "device" memory is host memory, copies are copies, kernels are noted down and not run.  The engines' host
// code is linked against it (device code as PTX that nothing loads) to test what it launches, in which order, and what it does
// when a call fails.  Which launch, attribute or tensor map fails is set by fake_fail.
#include <cuda.h>
#include <cuda_runtime.h>

#include <cstdlib>
#include <cstring>
#include <map>
#include <string>
#include <vector>

namespace {
int g_device = 0;
cudaError_t g_last = cudaSuccess;
// host stub -> mangled kernel name; made by the first registration, which may come before this file's own objects exist
std::map<const void*, std::string>& names() { static std::map<const void*, std::string> m; return m; }
struct Launch { const void* f; int device, overlaps; unsigned blocks; };
std::vector<Launch> g_launches;
std::map<std::pair<int, const void*>, int> g_smem;              // (device, kernel) -> opted in dynamic shared memory
constexpr int kKinds = 4;                                        // launches, attributes, tensor maps, copies to the host
long g_count[kKinds] = {}, g_fail[kKinds] = {-1, -1, -1, -1};    // how many so far, which one fails
std::map<void*, size_t> g_device_blocks;                         // what is taken of the device's memory
size_t g_used = 0, g_room = (size_t)1 << 40;
std::vector<int> g_pinned;                                       // devices on which results' memory was page-locked
int g_on_their_way = 0;                                         // copies to the host that nothing has waited for
// what a test has kernels leave on the device: copies to the host of exactly `bytes`, from the number `from` on, bring `value` at `at`
struct Planted { size_t bytes, at; int value; long from; };
std::vector<Planted> g_planted;
std::map<size_t, long> g_of_size, g_cleared;                     // copies to the host, memory set, by their size
// copies to the device since the last wait, whose sources have to stay as they were until it (a test asks for this)
struct Source { const void* at; std::string was; };
std::vector<Source> g_sources;
bool g_watching = false;
int g_changed = 0;
constexpr size_t kDefaultSmem = 48 * 1024, kMostSmem = 227 * 1024;

bool fails(int what) { return g_count[what]++ == g_fail[what]; }
cudaError_t last(cudaError_t e) { if (e != cudaSuccess) g_last = e; return e; }
cudaError_t launch(const void* f, dim3 grid, size_t smem, const cudaLaunchConfig_t* c = nullptr) {
  if (fails(0)) return last(cudaErrorLaunchFailure);
  const auto it = g_smem.find({g_device, f});
  if (smem > (it == g_smem.end() ? kDefaultSmem : (size_t)it->second)) return last(cudaErrorInvalidValue);
  int overlaps = 0;
  for (unsigned i = 0; c && i < c->numAttrs; ++i)
    if (c->attrs[i].id == cudaLaunchAttributeProgrammaticStreamSerialization) overlaps = c->attrs[i].val.programmaticStreamSerializationAllowed;
  g_launches.push_back({f, g_device, overlaps, grid.x});
  return cudaSuccess;
}
CUresult encode(CUtensorMap* m, CUtensorMapDataType, cuuint32_t, void* p, const cuuint64_t*, const cuuint64_t*, const cuuint32_t*,
                const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill) {
  if (fails(2)) return CUDA_ERROR_INVALID_VALUE;
  memset(m, 0, sizeof(*m));
  memcpy(m, &p, sizeof(p));
  return CUDA_SUCCESS;
}
}  // namespace

extern "C" {
// ---- what a test asks ---------------------------------------------------------------------------------------------------------------
void fake_reset() { g_launches.clear(); g_pinned.clear(); g_planted.clear(); g_of_size.clear(); g_cleared.clear(); for (int i = 0; i < kKinds; ++i) { g_count[i] = 0; g_fail[i] = -1; } g_last = cudaSuccess; }
void fake_fail(int what, long at) { g_count[what] = 0; g_fail[what] = at; }
long fake_count(int what) { return g_count[what]; }
void fake_room(long long bytes) { g_room = (size_t)bytes; }
long long fake_used() { return (long long)g_used; }
int fake_pinned() { return (int)g_pinned.size(); }
int fake_pinned_device(int i) { return g_pinned[i]; }
int fake_on_their_way() { return g_on_their_way; }
void fake_plant(long bytes, long at, int value, long from) { g_planted.push_back({(size_t)bytes, (size_t)at, value, from}); }
void fake_watch(int on) { g_watching = on != 0; g_sources.clear(); g_changed = 0; }
int fake_changed() { return g_changed; }
long fake_cleared(long bytes) { return g_cleared[(size_t)bytes]; }
int fake_launches() { return (int)g_launches.size(); }
const char* fake_launch_name(int i) { return names()[g_launches[i].f].c_str(); }
int fake_launch_device(int i) { return g_launches[i].device; }
int fake_launch_blocks(int i) { return (int)g_launches[i].blocks; }
int fake_launch_overlaps(int i) { return g_launches[i].overlaps; }

// ---- registration -------------------------------------------------------------------------------------------------------------------
void** __cudaRegisterFatBinary(void*) { static void* h; return &h; }
void __cudaRegisterFatBinaryEnd(void**) {}
void __cudaUnregisterFatBinary(void**) {}
void __cudaRegisterFunction(void**, const char* f, char*, const char* name, int, uint3*, uint3*, dim3*, dim3*, int*) { names()[f] = name; }
void __cudaRegisterVar(void**, char*, char*, const char*, int, size_t, int, int) {}
char __cudaInitModule(void**) { return 0; }
static dim3 g_grid, g_block; static size_t g_dyn; static cudaStream_t g_stream;
unsigned __cudaPushCallConfiguration(dim3 g, dim3 b, size_t s, cudaStream_t st) { g_grid = g; g_block = b; g_dyn = s; g_stream = st; return 0; }
cudaError_t __cudaPopCallConfiguration(dim3* g, dim3* b, size_t* s, void* st) { *g = g_grid; *b = g_block; *s = g_dyn; *(cudaStream_t*)st = g_stream; return cudaSuccess; }

// ---- runtime ------------------------------------------------------------------------------------------------------------------------
cudaError_t cudaGetDeviceCount(int* n) { *n = 2; return cudaSuccess; }
cudaError_t cudaSetDevice(int d) { g_device = d; return cudaSuccess; }
cudaError_t cudaGetDeviceProperties_v2(cudaDeviceProp* p, int) {
  memset(p, 0, sizeof(*p));
  p->major = 10; p->multiProcessorCount = 148;
  return cudaSuccess;
}
cudaError_t cudaDeviceGetAttribute(int* v, cudaDeviceAttr a, int) {
  *v = a == cudaDevAttrMaxSharedMemoryPerBlockOptin ? (int)kMostSmem : a == cudaDevAttrMultiProcessorCount ? 148 : a == cudaDevAttrClockRate ? 1965000 : 1;
  return cudaSuccess;
}
cudaError_t cudaOccupancyMaxActiveBlocksPerMultiprocessorWithFlags(int* n, const void*, int, size_t, unsigned) { *n = 1; return cudaSuccess; }
cudaError_t cudaMallocHost(void** p, size_t n) { *p = calloc(n ? n : 1, 1); return *p ? cudaSuccess : last(cudaErrorMemoryAllocation); }
cudaError_t cudaHostAlloc(void** p, size_t n, unsigned f) {
  if (f & cudaHostAllocPortable) g_pinned.push_back(g_device);
  return cudaMallocHost(p, n);
}
cudaError_t cudaMalloc(void** p, size_t n) {
  if (n > g_room - g_used) return last(cudaErrorMemoryAllocation);
  const cudaError_t e = cudaMallocHost(p, n);
  if (e == cudaSuccess) { g_device_blocks[*p] = n; g_used += n; }
  return e;
}
cudaError_t cudaMemGetInfo(size_t* left, size_t* all) { *left = g_room - g_used; *all = g_room; return cudaSuccess; }
cudaError_t cudaHostGetDevicePointer(void** d, void* p, unsigned) { *d = p; return cudaSuccess; }
cudaError_t cudaFree(void* p) {
  const auto it = g_device_blocks.find(p);
  if (it != g_device_blocks.end()) { g_used -= it->second; g_device_blocks.erase(it); }
  free(p);
  return cudaSuccess;
}
cudaError_t cudaFreeHost(void* p) { free(p); return cudaSuccess; }
cudaError_t cudaMemcpy(void* d, const void* s, size_t n, cudaMemcpyKind) { memcpy(d, s, n); return cudaSuccess; }
cudaError_t cudaMemcpyAsync(void* d, const void* s, size_t n, cudaMemcpyKind k, cudaStream_t) {
  if (k == cudaMemcpyDeviceToHost) {
    if (fails(3)) return last(cudaErrorInvalidValue);
    ++g_on_their_way;
  }
  memcpy(d, s, n);
  if (g_watching && k == cudaMemcpyHostToDevice) g_sources.push_back({s, std::string((const char*)s, n)});
  if (k == cudaMemcpyDeviceToHost) {
    const long number = g_of_size[n]++;
    for (const Planted& p : g_planted)
      if (p.bytes == n && number >= p.from) memcpy((char*)d + p.at, &p.value, sizeof(int));
  }
  return cudaSuccess;
}
cudaError_t cudaMemset(void* d, int v, size_t n) { memset(d, v, n); return cudaSuccess; }
cudaError_t cudaMemsetAsync(void* d, int v, size_t n, cudaStream_t) { ++g_cleared[n]; memset(d, v, n); return cudaSuccess; }
cudaError_t cudaStreamCreate(cudaStream_t* s) { *s = nullptr; return cudaSuccess; }
cudaError_t cudaStreamCreateWithFlags(cudaStream_t* s, unsigned) { *s = nullptr; return cudaSuccess; }
cudaError_t cudaStreamDestroy(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t) {
  g_on_their_way = 0;
  for (const Source& x : g_sources) g_changed += memcmp(x.at, x.was.data(), x.was.size()) != 0;
  g_sources.clear();
  return cudaSuccess;
}
cudaError_t cudaDeviceSynchronize() { return cudaSuccess; }
cudaError_t cudaEventCreate(cudaEvent_t* e) { *e = nullptr; return cudaSuccess; }
cudaError_t cudaEventDestroy(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaEventElapsedTime(float* ms, cudaEvent_t, cudaEvent_t) { *ms = 0.0f; return cudaSuccess; }
cudaError_t cudaGetLastError() { const cudaError_t e = g_last; g_last = cudaSuccess; return e; }
const char* cudaGetErrorString(cudaError_t e) { return e == cudaErrorInvalidValue ? "invalid argument" : e == cudaErrorLaunchFailure ? "launch refused" : "error"; }
cudaError_t cudaFuncGetAttributes(cudaFuncAttributes* a, const void*) { memset(a, 0, sizeof(*a)); return cudaSuccess; }
cudaError_t cudaFuncSetAttribute(const void* f, cudaFuncAttribute a, int v) {
  if (fails(1)) return last(cudaErrorInvalidValue);
  if (a == cudaFuncAttributeMaxDynamicSharedMemorySize) {
    if (v < 0 || (size_t)v > kMostSmem) return last(cudaErrorInvalidValue);
    g_smem[{g_device, f}] = v;
  }
  return cudaSuccess;
}
cudaError_t cudaLaunchKernel(const void* f, dim3 grid, dim3, void**, size_t smem, cudaStream_t) { return launch(f, grid, smem); }
cudaError_t cudaLaunchCooperativeKernel(const void* f, dim3 grid, dim3, void**, size_t smem, cudaStream_t) { return launch(f, grid, smem); }
cudaError_t cudaLaunchKernelExC(const cudaLaunchConfig_t* c, const void* f, void**) { return launch(f, c->gridDim, c->dynamicSmemBytes, c); }
cudaError_t cudaGetDriverEntryPoint(const char*, void** p, unsigned long long, cudaDriverEntryPointQueryResult* r) {
  *p = (void*)encode;
  *r = cudaDriverEntryPointSuccess;
  return cudaSuccess;
}
cudaError_t cudaDeviceCanAccessPeer(int* v, int, int) { *v = 0; return cudaSuccess; }
cudaError_t cudaDeviceEnablePeerAccess(int, unsigned) { return cudaErrorInvalidValue; }
cudaError_t cudaIpcGetMemHandle(cudaIpcMemHandle_t*, void*) { return cudaErrorInvalidValue; }
cudaError_t cudaIpcOpenMemHandle(void**, cudaIpcMemHandle_t, unsigned) { return cudaErrorInvalidValue; }
cudaError_t cudaIpcCloseMemHandle(void*) { return cudaErrorInvalidValue; }
}
