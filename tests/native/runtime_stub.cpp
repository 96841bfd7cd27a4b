// A CUDA runtime without a device, linked with the library's own objects in
// place of libcudart: device memory is zeroed host memory, copies run at once
// and kernels do nothing but be counted. The library's host side runs every
// entry point over it (all sums are zero, which is as good a transcript as any),
// so that what it enqueues and allocates can be looked at where there is no GPU.
//
// A kernel launched with programmatic stream serialization has to follow a kernel
// on its stream: stub_misplaced() lists those that follow a copy, a memset, an
// event wait or an allocation in stream order instead.
#include <cuda_runtime_api.h>

#include <cstdlib>
#include <cstring>
#include <map>
#include <mutex>
#include <set>
#include <string>
#include <vector>

namespace {

std::recursive_mutex mu;
std::map<const void*, std::string> names;     // host stub -> kernel name
std::map<std::string, int> launched;
std::map<cudaStream_t, std::string> last_op;  // "" after a kernel
std::set<std::string> misplaced;
std::map<void*, size_t> blocks;
std::vector<uint32_t*> flags;                 // pinned result buffers
size_t held = 0, most = 0;

// A mangled name's own part: the last identifier of its nested name.
std::string plain(const char* s) {
  std::string out = s;
  for (const char* p = s; *p;) {
    if (*p < '0' || *p > '9') {
      ++p;
      continue;
    }
    char* e;
    const unsigned long n = strtoul(p, &e, 10);
    if (n == 0 || n > strlen(e)) break;
    if (e[0] == 'k' && e[1] == '_') return std::string(e, n);
    p = e + n;
  }
  return out;
}

void did(cudaStream_t s, const char* what) {
  std::lock_guard<std::recursive_mutex> l(mu);
  last_op[s] = what;
}

void ran(cudaStream_t s, const void* fn, bool chained) {
  std::lock_guard<std::recursive_mutex> l(mu);
  const std::string& name = names[fn];
  ++launched[name];
  auto it = last_op.find(s);
  if (chained && it != last_op.end() && !it->second.empty()) misplaced.insert(name + " after " + it->second);
  last_op[s].clear();
}

void* take(size_t n) {
  std::lock_guard<std::recursive_mutex> l(mu);
  char* raw = static_cast<char*>(calloc(n + 512, 1));
  if (!raw) return nullptr;
  char* p = raw + 256 - reinterpret_cast<uintptr_t>(raw) % 256;
  reinterpret_cast<void**>(p)[-1] = raw;
  blocks[p] = n;
  held += n;
  if (held > most) most = held;
  return p;
}

void drop(void* p) {
  std::lock_guard<std::recursive_mutex> l(mu);
  auto it = blocks.find(p);
  if (it == blocks.end()) return;
  held -= it->second;
  blocks.erase(it);
  free(static_cast<void**>(p)[-1]);
}

struct Call {
  dim3 grid, block;
  size_t smem;
  cudaStream_t stream;
};
thread_local std::vector<Call> calls;
int handle;

}  // namespace

extern "C" {

// ---- what the tests ask ----
static size_t text(const std::string& s, char* out, size_t cap) {
  if (cap) {
    strncpy(out, s.c_str(), cap - 1);
    out[cap - 1] = 0;
  }
  return s.size();
}
size_t stub_misplaced(char* out, size_t cap) {
  std::string s;
  for (auto& m : misplaced) s += m + "\n";
  return text(s, out, cap);
}
size_t stub_launched(char* out, size_t cap) {
  std::string s;
  for (auto& m : launched) s += m.first + " " + std::to_string(m.second) + "\n";
  return text(s, out, cap);
}
void stub_reset() {
  launched.clear();
  misplaced.clear();
  most = held;
}
void stub_caller() {  // the caller queued work of its own on every stream
  for (auto& s : last_op) s.second = "the caller's work";
}
size_t stub_held() { return held; }
size_t stub_most() { return most; }

// ---- the runtime ----
void** __cudaRegisterFatBinary(void*) { return reinterpret_cast<void**>(&handle); }
void __cudaRegisterFatBinaryEnd(void**) {}
void __cudaUnregisterFatBinary(void**) {}
void __cudaRegisterFunction(void**, const char* host, char*, const char* name, int, void*, void*, void*, void*, int*) {
  names[host] = plain(name);
}
void __cudaRegisterVar(void**, char*, char*, const char*, int, size_t, int, int) {}
cudaError_t __cudaGetKernel(cudaKernel_t* k, const void* host) {
  *k = reinterpret_cast<cudaKernel_t>(const_cast<void*>(host));
  return cudaSuccess;
}
unsigned __cudaPushCallConfiguration(dim3 grid, dim3 block, size_t smem, void* stream) {
  calls.push_back({grid, block, smem, static_cast<cudaStream_t>(stream)});
  return 0;
}
cudaError_t __cudaPopCallConfiguration(dim3* grid, dim3* block, size_t* smem, void* stream) {
  const Call c = calls.back();
  calls.pop_back();
  *grid = c.grid, *block = c.block, *smem = c.smem;
  *static_cast<cudaStream_t*>(stream) = c.stream;
  return cudaSuccess;
}
cudaError_t __cudaLaunchKernel(cudaKernel_t k, dim3, dim3, void**, size_t, cudaStream_t s) {
  ran(s, k, false);
  return cudaSuccess;
}
cudaError_t cudaLaunchKernelExC(const cudaLaunchConfig_t* cfg, const void* fn, void**) {
  bool chained = false;
  for (unsigned i = 0; i < cfg->numAttrs; ++i)
    chained |= cfg->attrs[i].id == cudaLaunchAttributeProgrammaticStreamSerialization &&
               cfg->attrs[i].val.programmaticStreamSerializationAllowed;
  ran(cfg->stream, fn, chained);
  return cudaSuccess;
}

cudaError_t cudaGetDeviceCount(int* n) { return *n = 1, cudaSuccess; }
cudaError_t cudaGetDevice(int* d) { return *d = 0, cudaSuccess; }
cudaError_t cudaSetDevice(int) { return cudaSuccess; }
cudaError_t cudaDeviceGetAttribute(int* v, enum cudaDeviceAttr, int) { return *v = 152, cudaSuccess; }
cudaError_t cudaDeviceGetDefaultMemPool(cudaMemPool_t* p, int) { return *p = nullptr, cudaSuccess; }
cudaError_t cudaMemPoolSetAttribute(cudaMemPool_t, enum cudaMemPoolAttr, void*) { return cudaSuccess; }
cudaError_t cudaMemPoolGetAttribute(cudaMemPool_t, enum cudaMemPoolAttr, void* v) {
  return *static_cast<uint64_t*>(v) = 0, cudaSuccess;
}
cudaError_t cudaMemGetInfo(size_t* free_, size_t* total) {
  return *total = (size_t)280 << 30, *free_ = *total - held, cudaSuccess;
}
cudaError_t cudaGetLastError() { return cudaSuccess; }
const char* cudaGetErrorString(cudaError_t) { return "stub"; }
cudaError_t cudaFuncSetAttribute(const void*, enum cudaFuncAttribute, int) { return cudaSuccess; }
cudaError_t cudaOccupancyMaxActiveBlocksPerMultiprocessorWithFlags(int* n, const void*, int, size_t, unsigned) {
  return *n = 4, cudaSuccess;
}
cudaError_t cudaGetSymbolAddress(void** p, const void* symbol) { return *p = const_cast<void*>(symbol), cudaSuccess; }

cudaError_t cudaMalloc(void** p, size_t n) { return (*p = take(n)) ? cudaSuccess : cudaErrorMemoryAllocation; }
cudaError_t cudaFree(void* p) { return drop(p), cudaSuccess; }
cudaError_t cudaMallocAsync(void** p, size_t n, cudaStream_t s) { return did(s, "an allocation"), cudaMalloc(p, n); }
cudaError_t cudaFreeAsync(void* p, cudaStream_t) { return drop(p), cudaSuccess; }
cudaError_t cudaMallocHost(void** p, size_t n) {
  *p = calloc(n, 1);
  flags.push_back(static_cast<uint32_t*>(*p));
  return cudaSuccess;
}
cudaError_t cudaFreeHost(void* p) {
  for (auto& f : flags)
    if (f == p) f = flags.back(), flags.pop_back();
  return free(p), cudaSuccess;
}
cudaError_t cudaMemset(void* p, int v, size_t n) { return memset(p, v, n), cudaSuccess; }
cudaError_t cudaMemsetAsync(void* p, int v, size_t n, cudaStream_t s) {
  return did(s, "a memset"), memset(p, v, n), cudaSuccess;
}
cudaError_t cudaMemcpyAsync(void* to, const void* from, size_t n, enum cudaMemcpyKind, cudaStream_t s) {
  return did(s, "a copy"), memcpy(to, from, n), cudaSuccess;
}

cudaError_t cudaStreamCreateWithFlags(cudaStream_t* s, unsigned) {
  return *s = reinterpret_cast<cudaStream_t>(malloc(1)), cudaSuccess;
}
cudaError_t cudaStreamDestroy(cudaStream_t s) {
  last_op.erase(s);
  return free(s), cudaSuccess;
}
cudaError_t cudaStreamSynchronize(cudaStream_t) { return cudaSuccess; }
// The host asks while it waits for a kernel's flag: the next of its values (one a
// flagged kernel) is there.
cudaError_t cudaStreamQuery(cudaStream_t) {
  for (uint32_t* f : flags) ++*f;
  return cudaErrorNotReady;
}
cudaError_t cudaStreamWaitEvent(cudaStream_t s, cudaEvent_t, unsigned) { return did(s, "an event wait"), cudaSuccess; }
cudaError_t cudaEventCreate(cudaEvent_t* e) { return *e = reinterpret_cast<cudaEvent_t>(malloc(1)), cudaSuccess; }
cudaError_t cudaEventCreateWithFlags(cudaEvent_t* e, unsigned) { return cudaEventCreate(e); }
cudaError_t cudaEventDestroy(cudaEvent_t e) { return free(e), cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaEventSynchronize(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventElapsedTime(float* ms, cudaEvent_t, cudaEvent_t) { return *ms = 1.0f, cudaSuccess; }

}  // extern "C"
