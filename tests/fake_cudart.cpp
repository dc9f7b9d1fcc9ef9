// fake_cudart.cpp - the CUDA runtime calls of the library without a GPU, for tests
// of its host side: preloaded into a child process (fake_cuda.py).  Device memory
// is host memory, copies are made at once, kernels do nothing and are counted by
// name.  Streams, events and waits keep a record of what the host has waited for,
// so that a test can ask whether anything is still in flight; a call can be made
// to fail.
#include <cuda_runtime_api.h>

#include <cstdint>
#include <cstdlib>
#include <cstring>
#include <map>
#include <string>
#include <vector>

namespace {
using Clock = std::map<cudaStream_t, long>;  // operations by stream
struct State {
  Clock count;                               // submitted
  std::map<cudaStream_t, Clock> known;       // what a stream has waited for
  std::map<cudaEvent_t, Clock> event;
  std::map<cudaStream_t, bool> blocking;
  Clock done;                                // what the host has waited for
  std::map<const void *, std::string> kernel;
  std::vector<std::string> launched;
  std::map<void *, size_t> mem;
  long next = 0;
  cudaError_t last = cudaSuccess;
  std::string fail_what;
  long fail_after = -1;
  cudaError_t fail_code = cudaSuccess;
};
State &S() {
  static State *s = new State;
  return *s;
}
void join(Clock &a, const Clock &b) {
  for (auto &e : b) a[e.first] = a[e.first] > e.second ? a[e.first] : e.second;
}
Clock at(cudaStream_t st) {
  Clock c = S().known[st];
  c[st] = S().count[st];
  return c;
}
void legacy_sync() {  // the legacy stream waits for the blocking ones
  for (auto &b : S().blocking)
    if (b.second) join(S().done, at(b.first));
}
cudaError_t err(cudaError_t e) {
  if (e != cudaSuccess) S().last = e;
  return e;
}
// whether this call of `what` (a launch: of kernel `name`) is the one that was asked to fail
bool fails(const std::string &what, const std::string &name = "") {
  State &s = S();
  const bool is = name.empty() ? s.fail_what == what
                               : s.fail_what.rfind(what + " ", 0) == 0 &&
                                     name.find(s.fail_what.substr(what.size() + 1)) != std::string::npos;
  return s.fail_after >= 0 && is && s.fail_after-- == 0;
}
cudaError_t launch(const void *f, dim3 b, cudaStream_t st) {
  State &s = S();
  const std::string &name = s.kernel[f];
  if (fails("launch", name)) return err(s.fail_code);
  s.count[st]++;
  s.launched.push_back(name + " [" + std::to_string(b.x * b.y * b.z) + "]");
  return cudaSuccess;
}
int encode_ok(...) { return 0; }
}  // namespace

extern "C" {
// ---- what tests call ----
void fake_clear() { S().launched.clear(); }
// launches whose "name [threads]" holds `part`
long fake_launched(const char *part) {
  long n = 0;
  for (auto &l : S().launched) n += l.find(part) != std::string::npos;
  return n;
}
// operations that the host has not waited for
long fake_in_flight() {
  long n = 0;
  for (auto &c : S().count) n += c.second - S().done[c.first];
  return n;
}
// the call of `what` ("launch <part of a kernel's name>", "cudaMalloc", ...) after `after` more fails
void fake_fail(const char *what, long after, int code) {
  S().fail_what = what, S().fail_after = after, S().fail_code = (cudaError_t)code;
}
// writes v into every 4-byte allocation (the error flags of device waits)
void fake_set_flags(unsigned v) {
  for (auto &m : S().mem)
    if (m.second == 4) memcpy(m.first, &v, 4);
}

// ---- the runtime ----
void **__cudaRegisterFatBinary(void *) {
  static void *h;
  return &h;
}
void __cudaRegisterFatBinaryEnd(void **) {}
void __cudaUnregisterFatBinary(void **) {}
void __cudaRegisterFunction(void **, const char *host, char *, const char *name, int, uint3 *, uint3 *, dim3 *, dim3 *, int *) {
  S().kernel[host] = name;
}
void __cudaRegisterVar(void **, char *, char *, const char *, int, size_t, int, int) {}
static thread_local struct {
  dim3 g, b;
  size_t s;
  cudaStream_t st;
} call;
unsigned __cudaPushCallConfiguration(dim3 g, dim3 b, size_t s, cudaStream_t st) {
  call = {g, b, s, st};
  return 0;
}
cudaError_t __cudaPopCallConfiguration(dim3 *g, dim3 *b, size_t *s, void *st) {
  *g = call.g, *b = call.b, *s = call.s, *(cudaStream_t *)st = call.st;
  return cudaSuccess;
}
cudaError_t cudaLaunchKernel(const void *f, dim3, dim3 b, void **, size_t, cudaStream_t st) { return launch(f, b, st); }
cudaError_t cudaLaunchKernelExC(const cudaLaunchConfig_t *c, const void *f, void **) {
  return launch(f, c->blockDim, c->stream);
}
cudaError_t cudaGetLastError() {
  cudaError_t e = S().last;
  S().last = cudaSuccess;
  return e;
}
const char *cudaGetErrorString(cudaError_t) { return "fake error"; }
cudaError_t cudaGetDevice(int *d) { return *d = 0, cudaSuccess; }
cudaError_t cudaSetDevice(int) { return cudaSuccess; }
cudaError_t cudaDeviceGetAttribute(int *v, cudaDeviceAttr, int) { return *v = 148, cudaSuccess; }
cudaError_t cudaFuncSetAttribute(const void *, cudaFuncAttribute, int) { return cudaSuccess; }
cudaError_t cudaOccupancyMaxActiveBlocksPerMultiprocessorWithFlags(int *n, const void *, int, size_t, unsigned) {
  return *n = 2, cudaSuccess;
}
cudaError_t cudaGetSymbolAddress(void **, const void *) { return err(cudaErrorInvalidSymbol); }
cudaError_t cudaGetDriverEntryPoint(const char *name, void **p, unsigned long long, cudaDriverEntryPointQueryResult *q) {
  const bool ok = !strcmp(name, "cuTensorMapEncodeTiled");
  *p = ok ? (void *)encode_ok : nullptr;
  if (q) *q = ok ? cudaDriverEntryPointSuccess : cudaDriverEntryPointSymbolNotFound;
  return ok ? cudaSuccess : err(cudaErrorUnknown);
}
cudaError_t cudaMalloc(void **p, size_t n) {
  *p = nullptr;
  if (fails("cudaMalloc")) return err(S().fail_code);
  if (posix_memalign(p, 256, n ? n : 1)) return err(cudaErrorMemoryAllocation);
  memset(*p, 0, n);
  S().mem[*p] = n;
  return cudaSuccess;
}
cudaError_t cudaFree(void *p) {
  legacy_sync();
  if (p) S().mem.erase(p), free(p);
  return cudaSuccess;
}
cudaError_t cudaHostAlloc(void **p, size_t n, unsigned) { return (*p = malloc(n)) ? cudaSuccess : err(cudaErrorMemoryAllocation); }
cudaError_t cudaFreeHost(void *p) {
  free(p);
  return cudaSuccess;
}
cudaError_t cudaMemcpy(void *d, const void *s, size_t n, cudaMemcpyKind) {
  legacy_sync();
  memmove(d, s, n);
  return cudaSuccess;
}
cudaError_t cudaMemcpyAsync(void *d, const void *s, size_t n, cudaMemcpyKind, cudaStream_t st) {
  if (fails("cudaMemcpyAsync")) return err(S().fail_code);
  S().count[st]++;
  memmove(d, s, n);
  return cudaSuccess;
}
cudaError_t cudaMemcpy2DAsync(void *d, size_t dp, const void *s, size_t sp, size_t w, size_t h, cudaMemcpyKind, cudaStream_t st) {
  S().count[st]++;
  for (size_t k = 0; k < h; k++) memmove((char *)d + k * dp, (const char *)s + k * sp, w);
  return cudaSuccess;
}
cudaError_t cudaMemset(void *d, int v, size_t n) {
  memset(d, v, n);
  return cudaSuccess;
}
cudaError_t cudaMemsetAsync(void *d, int v, size_t n, cudaStream_t st) {
  S().count[st]++;
  memset(d, v, n);
  return cudaSuccess;
}
cudaError_t cudaStreamCreateWithFlags(cudaStream_t *st, unsigned flags) {
  *st = (cudaStream_t)(uintptr_t)(16 * ++S().next);
  S().blocking[*st] = !(flags & cudaStreamNonBlocking);
  return cudaSuccess;
}
cudaError_t cudaStreamCreate(cudaStream_t *st) { return cudaStreamCreateWithFlags(st, 0); }
cudaError_t cudaStreamDestroy(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t st) {
  join(S().done, at(st));
  return cudaSuccess;
}
cudaError_t cudaStreamWaitEvent(cudaStream_t st, cudaEvent_t e, unsigned) {
  join(S().known[st], S().event[e]);
  return cudaSuccess;
}
cudaError_t cudaEventCreateWithFlags(cudaEvent_t *e, unsigned) {
  *e = (cudaEvent_t)(uintptr_t)(16 * ++S().next);
  return cudaSuccess;
}
cudaError_t cudaEventCreate(cudaEvent_t *e) { return cudaEventCreateWithFlags(e, 0); }
cudaError_t cudaEventDestroy(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t e, cudaStream_t st) {
  S().event[e] = at(st);
  return cudaSuccess;
}
cudaError_t cudaEventSynchronize(cudaEvent_t e) {
  join(S().done, S().event[e]);
  return cudaSuccess;
}
cudaError_t cudaEventElapsedTime(float *ms, cudaEvent_t, cudaEvent_t) { return *ms = (float)++S().next, cudaSuccess; }
}
