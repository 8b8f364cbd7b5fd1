// A CUDA runtime without a GPU, for tests of the library's host code: linked
// with the library's objects in place of the real runtime.  Device memory is
// host memory, kernels do not run, and every call is written to a log that the
// test reads (fake_log).  A call that a stream capture forbids returns the
// error that the real runtime gives.
#include <cuda_runtime_api.h>

#include <algorithm>
#include <cstdarg>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <map>
#include <set>
#include <string>

namespace {

std::string g_log;
std::map<char*, size_t> g_device;             // allocations, by address
std::map<char*, size_t> g_host;               // page-locked ones
std::map<const void*, int> g_device_of;       // allocations of another device (fake_set_device)
std::map<const void*, std::string> g_kernel;  // host stub -> device name
std::map<const void*, size_t> g_var;
std::set<cudaStream_t> g_capturing;
int g_fail_malloc = 0;                        // the n-th allocation from here on fails
size_t g_next = 1;

void note(const char* fmt, ...) {
  char line[512];
  va_list ap;
  va_start(ap, fmt);
  vsnprintf(line, sizeof line, fmt, ap);
  va_end(ap);
  g_log += line;
  g_log += '\n';
}

bool inside(const std::map<char*, size_t>& m, const void* p, const void** base = nullptr) {
  char* c = static_cast<char*>(const_cast<void*>(p));
  auto it = m.upper_bound(c);
  if (it == m.begin()) return false;
  --it;
  if (base) *base = it->first;
  return c < it->first + it->second;
}

}  // namespace

extern "C" {

// ---- test side -------------------------------------------------------------
const char* fake_log() { return g_log.c_str(); }
void fake_clear() { g_log.clear(); }
void fake_fail_malloc(int n) { g_fail_malloc = n; }
void fake_set_device(const void* p, int device) { g_device_of[p] = device; }
void fake_capture(void* stream, int on) {
  if (on) g_capturing.insert(static_cast<cudaStream_t>(stream));
  else g_capturing.erase(static_cast<cudaStream_t>(stream));
}
void* fake_stream() { return reinterpret_cast<void*>(0x1000 + 16 * g_next++); }

// ---- runtime ---------------------------------------------------------------
cudaError_t cudaGetDeviceCount(int* n) { *n = 1; return cudaSuccess; }
cudaError_t cudaGetDevice(int* d) { *d = 0; return cudaSuccess; }
cudaError_t cudaDeviceGetAttribute(int* v, cudaDeviceAttr a, int) {
  *v = a == cudaDevAttrMultiProcessorCount ? 148 : a == cudaDevAttrL2CacheSize ? 132644864 : 0;
  return cudaSuccess;
}
cudaError_t cudaGetLastError() { return cudaSuccess; }
const char* cudaGetErrorString(cudaError_t e) {
  return e == cudaErrorMemoryAllocation ? "out of memory"
         : e == cudaErrorStreamCaptureUnsupported ? "operation not permitted when stream is capturing" : "error";
}

cudaError_t cudaMalloc(void** p, size_t n) {
  if (!g_capturing.empty()) { note("malloc-in-capture"); return cudaErrorStreamCaptureUnsupported; }
  if (g_fail_malloc > 0 && --g_fail_malloc == 0) { note("malloc-failed"); return cudaErrorMemoryAllocation; }
  *p = aligned_alloc(256, (n + 255) / 256 * 256);
  memset(*p, 0, (n + 255) / 256 * 256);
  g_device[static_cast<char*>(*p)] = n;
  note("malloc %p %zu", *p, n);
  return cudaSuccess;
}
cudaError_t cudaFree(void* p) {
  if (!p) return cudaSuccess;
  if (!g_capturing.empty()) { note("free-in-capture"); return cudaErrorStreamCaptureUnsupported; }
  note("free %p", p);
  g_device.erase(static_cast<char*>(p));
  free(p);
  return cudaSuccess;
}
cudaError_t cudaHostAlloc(void** p, size_t n, unsigned) {
  *p = aligned_alloc(256, (n + 255) / 256 * 256);
  g_host[static_cast<char*>(*p)] = n;
  return cudaSuccess;
}
cudaError_t cudaMallocHost(void** p, size_t n) { return cudaHostAlloc(p, n, 0); }
cudaError_t cudaFreeHost(void* p) {
  g_host.erase(static_cast<char*>(p));
  free(p);
  return cudaSuccess;
}
cudaError_t cudaMemcpy(void* d, const void* s, size_t n, cudaMemcpyKind) {
  if (!g_capturing.empty()) { note("memcpy-in-capture"); return cudaErrorStreamCaptureUnsupported; }
  note("memcpy %p %zu", d, n);
  memcpy(d, s, n);
  return cudaSuccess;
}
cudaError_t cudaMemcpyAsync(void* d, const void* s, size_t n, cudaMemcpyKind, cudaStream_t st) {
  note("memcpy-async %p %zu stream %p", d, n, static_cast<void*>(st));
  if (!g_capturing.count(st)) memcpy(d, s, n);
  return cudaSuccess;
}
cudaError_t cudaMemset(void* p, int v, size_t n) { memset(p, v, n); return cudaSuccess; }
cudaError_t cudaMemsetAsync(void* p, int v, size_t n, cudaStream_t st) {
  note("memset-async %p %zu stream %p", p, n, static_cast<void*>(st));
  return cudaSuccess;
}
cudaError_t cudaPointerGetAttributes(cudaPointerAttributes* a, const void* p) {
  memset(a, 0, sizeof *a);
  const void* base = nullptr;
  a->type = cudaMemoryTypeUnregistered;
  if (inside(g_device, p, &base)) a->type = cudaMemoryTypeDevice;
  else if (inside(g_host, p)) a->type = cudaMemoryTypeHost;
  else return cudaSuccess;
  a->devicePointer = const_cast<void*>(p);
  a->device = base && g_device_of.count(base) ? g_device_of[base] : 0;
  return cudaSuccess;
}

cudaError_t cudaStreamCreateWithFlags(cudaStream_t* s, unsigned) { *s = static_cast<cudaStream_t>(fake_stream()); return cudaSuccess; }
cudaError_t cudaStreamDestroy(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t s) {
  if (g_capturing.count(s)) return cudaErrorStreamCaptureUnsupported;
  note("synchronize stream %p", static_cast<void*>(s));
  return cudaSuccess;
}
cudaError_t cudaStreamWaitEvent(cudaStream_t s, cudaEvent_t e, unsigned) {
  note("wait stream %p event %p", static_cast<void*>(s), static_cast<void*>(e));
  return cudaSuccess;
}
cudaError_t cudaStreamIsCapturing(cudaStream_t s, cudaStreamCaptureStatus* c) {
  *c = g_capturing.count(s) ? cudaStreamCaptureStatusActive : cudaStreamCaptureStatusNone;
  return cudaSuccess;
}
cudaError_t cudaStreamBeginCapture(cudaStream_t s, cudaStreamCaptureMode) { g_capturing.insert(s); return cudaSuccess; }
cudaError_t cudaStreamEndCapture(cudaStream_t s, cudaGraph_t* g) {
  g_capturing.erase(s);
  *g = static_cast<cudaGraph_t>(fake_stream());
  return cudaSuccess;
}
cudaError_t cudaGraphInstantiate(cudaGraphExec_t* x, cudaGraph_t, unsigned long long) {
  *x = static_cast<cudaGraphExec_t>(fake_stream());
  return cudaSuccess;
}
cudaError_t cudaGraphLaunch(cudaGraphExec_t, cudaStream_t) { note("graph-launch"); return cudaSuccess; }
cudaError_t cudaGraphDestroy(cudaGraph_t) { return cudaSuccess; }
cudaError_t cudaGraphExecDestroy(cudaGraphExec_t) { return cudaSuccess; }
cudaError_t cudaEventCreate(cudaEvent_t* e) { *e = static_cast<cudaEvent_t>(fake_stream()); return cudaSuccess; }
cudaError_t cudaEventCreateWithFlags(cudaEvent_t* e, unsigned) { return cudaEventCreate(e); }
cudaError_t cudaEventDestroy(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t e, cudaStream_t s) {
  note("record event %p stream %p", static_cast<void*>(e), static_cast<void*>(s));
  return cudaSuccess;
}
cudaError_t cudaEventSynchronize(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventElapsedTime(float* ms, cudaEvent_t, cudaEvent_t) { *ms = 0.f; return cudaSuccess; }

cudaError_t cudaFuncSetAttribute(const void*, cudaFuncAttribute, int) { return cudaSuccess; }
// The resources of an SM: 228 KB of shared memory (1 KB more than asked for per
// block), 64 K registers at 128 a thread, 2,048 threads.
cudaError_t cudaOccupancyMaxActiveBlocksPerMultiprocessorWithFlags(int* n, const void*, int threads, size_t smem,
                                                                  unsigned) {
  const int by_smem = static_cast<int>(228 * 1024 / (smem + 1024)), by_regs = 65536 / (128 * threads);
  *n = std::min(by_smem, by_regs);
  return cudaSuccess;
}
cudaError_t cudaLaunchKernel(const void* f, dim3 g, dim3 b, void** args, size_t smem, cudaStream_t s) {
  const std::string& name = g_kernel[f];
  note("launch %s grid %u block %u smem %zu stream %p", name.c_str(), g.x, b.x, smem, static_cast<void*>(s));
  // (natoms, energies, virials, partials, out, err, d_energy, d_virial)
  if (name.find("k_totals") != std::string::npos)
    note("totals energy %p virial %p", *static_cast<void**>(args[6]), *static_cast<void**>(args[7]));
  return cudaSuccess;
}
cudaError_t cudaGetSymbolAddress(void** p, const void* sym) {
  static std::map<const void*, void*> at;
  if (!at.count(sym)) {
    void* q = nullptr;
    cudaError_t e = cudaMalloc(&q, g_var[sym]);
    if (e != cudaSuccess) return e;
    at[sym] = q;
  }
  *p = at[sym];
  return cudaSuccess;
}

// ---- what the compiler's launch and registration code calls ------------------
static struct { dim3 g, b; size_t smem; cudaStream_t s; } g_cfg;
unsigned __cudaPushCallConfiguration(dim3 g, dim3 b, size_t smem, void* s) {
  g_cfg = {g, b, smem, static_cast<cudaStream_t>(s)};
  return 0;
}
cudaError_t __cudaPopCallConfiguration(dim3* g, dim3* b, size_t* smem, void* s) {
  *g = g_cfg.g;
  *b = g_cfg.b;
  *smem = g_cfg.smem;
  *static_cast<cudaStream_t*>(s) = g_cfg.s;
  return cudaSuccess;
}
void** __cudaRegisterFatBinary(void*) {
  static void* h;
  return &h;
}
void __cudaRegisterFatBinaryEnd(void**) {}
void __cudaUnregisterFatBinary(void**) {}
void __cudaRegisterFunction(void**, const char* stub, char*, const char* name, int, void*, void*, void*, void*, int*) {
  g_kernel[stub] = name;
}
void __cudaRegisterVar(void**, char* host, char*, const char*, int, size_t n, int, int) { g_var[host] = n; }

}  // extern "C"
