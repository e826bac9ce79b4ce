// The trajectory analysis' host code over a CUDA runtime made of host memory, whose calls can be made to
// fail one at a time: no GPU, and kernels do nothing.  A stream is "busy" from the first work put on
// it to the next wait for it.
//   drains    for every runtime call of souffle_analysis_frames and _enqueue in turn, that call fails: the
//             function reports it and leaves no stream busy
//   grows     the candidate list overflows and allocations fail while it is grown: kernels get lists as
//             long as they are told, one lane is enough for the call to succeed, and later calls work
// Prints what went wrong and returns the number of failures.
#include <cuda_runtime.h>

#include <cstdint>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <map>
#include <set>
#include <string>
#include <vector>

#include "souffle_analysis.h"

namespace souffle {
void record_error(const std::string&) {}
}

namespace {
int g_fail_at = -1, g_calls = 0;     // the call that fails, calls so far
int g_allocs = 0, g_fail_alloc = -1, g_fail_allocs = 0;  // allocations so far; from which on and how many fail
int g_overflows = 0;                 // frames still to be reported as overflowing
int g_short_lists = 0;               // launches with a list shorter than its capacity
std::map<void*, size_t> g_sizes;     // device memory
std::map<const void*, std::string>& kernels() {  // (filled before main)
  static std::map<const void*, std::string> m;
  return m;
}
std::set<void*> g_busy;              // streams with work
cudaStream_t g_launch = nullptr;     // stream of the launch being configured
bool fails() { return g_calls++ == g_fail_at; }
cudaError_t on(cudaStream_t s) {
  if (fails()) return cudaErrorUnknown;
  g_busy.insert(s);
  return cudaSuccess;
}
}  // namespace

extern "C" {
cudaError_t cudaGetDeviceCount(int* n) { return *n = 1, cudaSuccess; }
cudaError_t cudaGetDevice(int* d) { return *d = 0, cudaSuccess; }
cudaError_t cudaSetDevice(int) { return cudaSuccess; }
cudaError_t cudaDeviceGetAttribute(int* v, cudaDeviceAttr, int) { return *v = 152, cudaSuccess; }
cudaError_t cudaGetLastError(void) { return cudaSuccess; }
const char* cudaGetErrorString(cudaError_t) { return "an error"; }
cudaError_t cudaFuncSetAttribute(const void*, cudaFuncAttribute, int) { return cudaSuccess; }
cudaError_t cudaMalloc(void** p, size_t n) {
  if (fails()) return cudaErrorMemoryAllocation;
  const int k = g_allocs++ - g_fail_alloc;
  if (g_fail_alloc >= 0 && k >= 0 && k < g_fail_allocs) return cudaErrorMemoryAllocation;
  *p = calloc(1, n);
  g_sizes[*p] = n;
  return cudaSuccess;
}
cudaError_t cudaFree(void* p) { return g_sizes.erase(p), free(p), cudaSuccess; }
cudaError_t cudaHostAlloc(void** p, size_t n, unsigned int) { return *p = calloc(1, n), cudaSuccess; }
cudaError_t cudaMallocHost(void** p, size_t n) { return *p = calloc(1, n), cudaSuccess; }
cudaError_t cudaFreeHost(void* p) { return free(p), cudaSuccess; }
cudaError_t cudaStreamCreateWithFlags(cudaStream_t* s, unsigned int) {
  return *s = reinterpret_cast<cudaStream_t>(malloc(1)), cudaSuccess;
}
cudaError_t cudaStreamDestroy(cudaStream_t s) { return free(s), cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t s) { return g_busy.erase(s), cudaSuccess; }
cudaError_t cudaEventCreateWithFlags(cudaEvent_t* e, unsigned int) {
  return *e = reinterpret_cast<cudaEvent_t>(malloc(1)), cudaSuccess;
}
cudaError_t cudaEventDestroy(cudaEvent_t e) { return free(e), cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t, cudaStream_t s) { return on(s); }
cudaError_t cudaStreamWaitEvent(cudaStream_t s, cudaEvent_t, unsigned int) { return on(s); }
cudaError_t cudaMemsetAsync(void* p, int v, size_t n, cudaStream_t s) {
  const cudaError_t e = on(s);
  if (e == cudaSuccess) memset(p, v, n);
  return e;
}
cudaError_t cudaMemcpyAsync(void* d, const void* s, size_t n, cudaMemcpyKind kind, cudaStream_t st) {
  const cudaError_t e = on(st);
  if (e == cudaSuccess) memcpy(d, s, n);
  if (kind == cudaMemcpyDeviceToHost && n == 16 && g_overflows > 0) {  // a frame's counters
    static_cast<unsigned*>(d)[1] = 100000;
    static_cast<unsigned*>(d)[3] = 1;
    g_overflows--;
  }
  return e;
}
// what the compiler's launch code calls
unsigned __cudaPushCallConfiguration(dim3, dim3, size_t, void* stream) {
  g_launch = static_cast<cudaStream_t>(stream);
  return 0;
}
cudaError_t __cudaPopCallConfiguration(dim3*, dim3*, size_t*, void* stream) {
  *static_cast<cudaStream_t*>(stream) = g_launch;
  return cudaSuccess;
}
cudaError_t __cudaGetKernel(cudaKernel_t* k, const void* fn) {
  *k = reinterpret_cast<cudaKernel_t>(const_cast<void*>(fn));
  return cudaSuccess;
}
struct Params {  // AnParams of csrc/analysis.cu
  double d[4];
  float f[9];
  int N, np, S, bins, pcf_type, so_type, image, cap;
};
cudaError_t cudaLaunchKernel(const void* fn, dim3, dim3, void** args, size_t, cudaStream_t s) {
  g_busy.insert(s);
  if (kernels()[fn].find("k_an_candidates") != std::string::npos) {  // (spheres, parameters, list, counters)
    const int cap = static_cast<Params*>(args[1])->cap;
    void* list = *static_cast<void**>(args[2]);
    if (cap > 0 && (!g_sizes.count(list) || g_sizes[list] < 8 * (size_t)cap)) g_short_lists++;
  }
  return cudaSuccess;
}
cudaError_t __cudaLaunchKernel(cudaKernel_t k, dim3 g, dim3 b, void** args, size_t n, cudaStream_t s) {
  return cudaLaunchKernel(reinterpret_cast<const void*>(k), g, b, args, n, s);
}
void** __cudaRegisterFatBinary(void*) {
  static void* h = nullptr;
  return &h;
}
void __cudaRegisterFatBinaryEnd(void**) {}
void __cudaUnregisterFatBinary(void**) {}
void __cudaRegisterFunction(void**, const char* fn, char*, const char* name, int, void*, void*, void*, void*, int*) {
  kernels()[fn] = name;
}
}

namespace {
constexpr int kBeads = 43 * 12, kSubs = 12, kFrames = 11;  // two chunks of frames
std::vector<double> g_pos(3 * kBeads * kFrames, 0.0);
std::vector<int32_t> g_types(kBeads * kFrames, 1);
std::vector<int64_t> g_pcf(100 * kFrames), g_olig(kSubs * kFrames), g_so(2 * kSubs * kFrames);

souffle_analysis* create() {
  souffle_analysis* h = nullptr;
  g_fail_at = -1;
  if (souffle_analysis_create(kBeads, 43, 40.0, nullptr, 0, &h) != SOUFFLE_OK) exit(100);
  return h;
}
souffle_status frames(souffle_analysis* h) {
  return souffle_analysis_frames(h, kFrames, g_pos.data(), g_types.data(), g_pcf.data(), g_olig.data(), g_so.data(), nullptr);
}

int drains() {
  int bad = 0;
  for (const bool device : {false, true})
    for (int k = 0;; k++) {
      souffle_analysis* h = create();
      if (frames(h) != SOUFFLE_OK) exit(101);  // (both lanes exist)
      g_calls = 0;
      g_fail_at = k;
      const souffle_status s = device ? souffle_analysis_enqueue(h, g_pos.data(), g_types.data(), g_pcf.data(), g_olig.data(),
                                                                 g_so.data(), nullptr)
                                      : frames(h);
      const bool reached = g_calls > k;
      g_fail_at = -1;
      if (reached && s == SOUFFLE_OK && ++bad) printf("call %d fails and is not reported\n", k);
      if (reached && !g_busy.empty() && ++bad)
        printf("%s: %zu streams busy after call %d failed\n", device ? "enqueue" : "frames", g_busy.size(), k);
      souffle_analysis_destroy(h);
      g_busy.clear();
      if (!reached) break;
    }
  return bad;
}

int grows() {
  int bad = 0;
  for (int fail = 0; fail < 6; fail++)       // the first, second, ... allocation of the call
    for (const int count : {1, 2, 100}) {    // and the ones after it
      souffle_analysis* h = create();
      if (frames(h) != SOUFFLE_OK) exit(102);
      g_overflows = 2;
      g_allocs = 0;
      g_fail_alloc = fail;
      g_fail_allocs = count;
      const souffle_status s = frames(h);
      const int failed = g_allocs - fail;
      g_fail_alloc = -1;
      g_overflows = 0;
      if (failed > 0 && count == 1 && s != SOUFFLE_OK && ++bad) printf("grow: one failure (%d) fails the call\n", fail);
      if (failed > 0 && count == 100 && fail == 0 && s == SOUFFLE_OK && ++bad) printf("grow: no memory, and no error\n");
      // types of the last frame, as a program goes on
      if (souffle_analysis_frames(h, kFrames, g_pos.data(), nullptr, g_pcf.data(), nullptr, nullptr, nullptr) != SOUFFLE_OK &&
          ++bad)
        printf("grow: the call after a failure (%d, %d) fails\n", fail, count);
      souffle_analysis_destroy(h);
    }
  if (g_short_lists && ++bad) printf("grow: %d launches with a list shorter than its capacity\n", g_short_lists);
  if (!g_sizes.empty() && ++bad) printf("grow: %zu allocations left\n", g_sizes.size());
  return bad;
}
}  // namespace

int main(int argc, char** argv) { return argc > 1 && !strcmp(argv[1], "grows") ? grows() : drains(); }
