// A CUDA runtime and NCCL for host-side tests: device memory is host memory, kernels do nothing, and every launch, copy, event
// and wait is logged.  Loaded in front of the real runtime (LD_PRELOAD), so that the library's host code runs without a GPU
// and a test can make any single call fail.
#include <dlfcn.h>
#include <stdint.h>
#include <stdio.h>
#include <stdlib.h>
#include <string.h>
#include <sys/mman.h>

#include <chrono>
#include <condition_variable>
#include <map>
#include <mutex>
#include <string>

namespace {
std::mutex m;
std::string log_text;
std::map<const void *, std::string> kernels;
std::map<const void *, size_t> symbols;
std::map<uintptr_t, size_t> device, pinned;
std::map<const void *, void *> symbol_mem;
uintptr_t next_handle = 0x1000;
long mallocs = 0, fail_malloc = -1, host_allocs = 0;
std::string fail_kernel;
long fail_kernel_after = 0;
int last_error = 0;
struct Config { unsigned g[3], b[3]; size_t smem; void *st; } pushed;

void note(const char *what, const std::string &rest) { log_text += std::string(what) + " " + rest + "\n"; }
std::string hex(const void *p) { char s[32]; snprintf(s, sizeof s, "%p", p); return s; }
void *take(size_t n) { return mmap(nullptr, n ? n : 1, PROT_READ | PROT_WRITE, MAP_PRIVATE | MAP_ANONYMOUS | MAP_NORESERVE, -1, 0); }
// zeros without holding the pages: most buffers are cleared and never touched
void fill(void *d, int v, size_t n) {
    const uintptr_t a = (reinterpret_cast<uintptr_t>(d) + 4095) & ~(uintptr_t)4095, e = (reinterpret_cast<uintptr_t>(d) + n) & ~(uintptr_t)4095;
    if (v || e <= a) { memset(d, v, n); return; }
    memset(d, 0, a - reinterpret_cast<uintptr_t>(d));
    madvise(reinterpret_cast<void *>(a), e - a, MADV_DONTNEED);
    memset(reinterpret_cast<void *>(e), 0, reinterpret_cast<uintptr_t>(d) + n - e);
}
std::map<const void *, int> smem_limit;
std::string meet_kernel;
int meeting = 0;
std::condition_variable met;
int launch(const void *f, void *st, unsigned gx, unsigned gy, unsigned gz, size_t smem) {
    std::lock_guard<std::mutex> l(m);
    const std::string &name = kernels[f];
    if (smem > (smem_limit.count(f) ? (size_t)smem_limit[f] : (size_t)48 << 10)) { note("refused", name + " " + hex(st)); return last_error = 1; }
    if (!fail_kernel.empty() && name.find(fail_kernel) != std::string::npos && fail_kernel_after-- == 0) { note("failed", name + " " + hex(st)); return last_error = 719; }
    note("launch", name + " " + hex(st) + " " + std::to_string(gx) + "," + std::to_string(gy) + "," + std::to_string(gz));
    return 0;
}
// refuses what is not aligned and what is not allocated any more
int encode_tiled(void *, int, uint32_t, void *base, const uint64_t *, const uint64_t *, const uint32_t *, const uint32_t *, int, int, int, int) {
    const uintptr_t p = reinterpret_cast<uintptr_t>(base);
    std::lock_guard<std::mutex> l(m);
    auto it = device.upper_bound(p);
    if ((p & 15) || it == device.begin()) return 1;
    --it;
    return p < it->first + it->second ? 0 : 1;
}
}  // namespace

extern "C" {
// ---- control ----
const char *fake_log() { return log_text.c_str(); }
void fake_clear() { log_text.clear(); }
void fake_fail_malloc(long nth) { fail_malloc = nth < 0 ? -1 : mallocs + nth; }       // 0: the next one
void fake_fail_kernel(const char *part, long after) { fail_kernel = part; fail_kernel_after = after; }
// the next two settings of this kernel's shared-memory limit meet, and the smaller one takes effect last
void fake_meet(const char *part) { meet_kernel = part; meeting = 0; }
long fake_mallocs() { return mallocs; }
long fake_host_allocs() { return host_allocs; }
long long fake_device_bytes() { long long n = 0; for (auto &d : device) n += (long long)d.second; return n; }
long long fake_pinned_bytes() { long long n = 0; for (auto &d : pinned) n += (long long)d.second; return n; }

// ---- runtime ----
int cudaMalloc(void **p, size_t n) {
    std::lock_guard<std::mutex> l(m);
    if (mallocs++ == fail_malloc) return 2;
    *p = take(n);
    device[reinterpret_cast<uintptr_t>(*p)] = n;
    return 0;
}
int cudaFree(void *p) {
    std::lock_guard<std::mutex> l(m);
    auto it = device.find(reinterpret_cast<uintptr_t>(p));
    if (it == device.end()) return p ? 1 : 0;
    mprotect(p, it->second ? it->second : 1, PROT_NONE);        // a later use of it is a fault here and now
    note("free", hex(p));
    device.erase(it);
    return 0;
}
int cudaHostAlloc(void **p, size_t n, unsigned) {
    std::lock_guard<std::mutex> l(m);
    host_allocs++;
    *p = take(n);
    pinned[reinterpret_cast<uintptr_t>(*p)] = n;
    return 0;
}
int cudaFreeHost(void *p) {
    std::lock_guard<std::mutex> l(m);
    auto it = pinned.find(reinterpret_cast<uintptr_t>(p));
    if (it == pinned.end()) return 1;
    munmap(p, it->second);
    pinned.erase(it);
    return 0;
}
int cudaMemcpyAsync(void *d, const void *s, size_t n, int, void *st) { memcpy(d, s, n); std::lock_guard<std::mutex> l(m); note("copy", hex(st)); return 0; }
int cudaMemcpy(void *d, const void *s, size_t n, int) { memcpy(d, s, n); return 0; }
int cudaMemset(void *d, int v, size_t n) { memset(d, v, n); return 0; }
int cudaMemsetAsync(void *d, int v, size_t n, void *st) { fill(d, v, n); std::lock_guard<std::mutex> l(m); note("memset", hex(st)); return 0; }
int cudaMemGetInfo(size_t *f, size_t *t) { *f = *t = (size_t)8 << 30; return 0; }
int cudaPointerGetAttributes(void *a, const void *) { memset(a, 0, 16); return 0; }
int cudaGetDeviceCount(int *n) { *n = 1; return 0; }
int cudaGetDevice(int *d) { *d = 0; return 0; }
int cudaSetDevice(int) { return 0; }
int cudaDeviceGetAttribute(int *v, int a, int) { *v = a == 75 ? 10 : (a == 16 ? 148 : 0); return 0; }
int cudaGetDriverEntryPoint(const char *, void **fn, unsigned long long, int *res) { *fn = (void *)encode_tiled; if (res) *res = 0; return 0; }
int cudaGetLastError() { const int e = last_error; last_error = 0; return e; }
const char *cudaGetErrorString(int e) { return e == 2 ? "out of memory" : "a failure the test asked for"; }
int cudaFuncSetAttribute(const void *f, int a, int v) {
    if (a != 8) return 0;
    std::unique_lock<std::mutex> l(m);
    const bool meet = !meet_kernel.empty() && kernels[f].find(meet_kernel) != std::string::npos;
    smem_limit[f] = meet && meeting ? (v < smem_limit[f] ? v : smem_limit[f]) : v;
    if (meet) {
        meeting++;
        met.notify_all();
        met.wait_for(l, std::chrono::seconds(2), [] { return meeting > 1; });
    }
    return 0;
}
int cudaOccupancyMaxActiveClusters(int *n, const void *, const void *) { *n = 74; return 0; }
int cudaGetSymbolAddress(void **p, const void *s) {
    std::lock_guard<std::mutex> l(m);
    if (!symbol_mem[s]) symbol_mem[s] = take(symbols[s]);
    *p = symbol_mem[s];
    return 0;
}
int cudaStreamCreateWithFlags(void **s, unsigned) { std::lock_guard<std::mutex> l(m); *s = (void *)(next_handle += 16); return 0; }
int cudaStreamDestroy(void *) { return 0; }
int cudaStreamSynchronize(void *s) { std::lock_guard<std::mutex> l(m); note("sync", hex(s)); return 0; }
int cudaStreamWaitEvent(void *s, void *e, unsigned) { std::lock_guard<std::mutex> l(m); note("wait", hex(s) + " " + hex(e)); return 0; }
int cudaEventCreateWithFlags(void **e, unsigned) { std::lock_guard<std::mutex> l(m); *e = (void *)(next_handle += 16); return 0; }
int cudaEventCreate(void **e) { return cudaEventCreateWithFlags(e, 0); }
int cudaEventDestroy(void *) { return 0; }
int cudaEventRecord(void *e, void *s) { std::lock_guard<std::mutex> l(m); note("record", hex(e) + " " + hex(s)); return 0; }
int cudaEventSynchronize(void *) { return 0; }
int cudaEventElapsedTime(float *t, void *, void *) { *t = 0; return 0; }
int cudaStreamBeginCapture(void *, int) { return 0; }
int cudaStreamEndCapture(void *, void **g) { *g = (void *)1; return 0; }
int cudaGraphInstantiate(void **e, void *, unsigned long long) { *e = (void *)1; return 0; }
int cudaGraphDestroy(void *) { return 0; }
int cudaGraphExecDestroy(void *) { return 0; }
int cudaGraphLaunch(void *, void *st) { std::lock_guard<std::mutex> l(m); note("graph", hex(st)); return 0; }
int cudaLaunchKernel(const void *f, uint64_t gxy, uint32_t gz, uint64_t, uint32_t, void **, size_t smem, void *st) { return launch(f, st, (unsigned)gxy, (unsigned)(gxy >> 32), gz, smem); }
int cudaLaunchKernelExC(const void *cfg, const void *f, void **) {
    const unsigned *g = static_cast<const unsigned *>(cfg);
    return launch(f, *reinterpret_cast<void *const *>(static_cast<const char *>(cfg) + 32), g[0], g[1], g[2], *reinterpret_cast<const size_t *>(static_cast<const char *>(cfg) + 24));
}

// ---- what the compiler's start-up code calls ----
void **__cudaRegisterFatBinary(void *) { static void *h; return &h; }
void __cudaRegisterFatBinaryEnd(void **) {}
void __cudaUnregisterFatBinary(void **) {}
void __cudaRegisterFunction(void **, const char *f, char *, const char *name, int, void *, void *, void *, void *, int *) { kernels[f] = name; }
void __cudaRegisterVar(void **, char *v, char *, const char *, int, size_t n, int, int) { symbols[v] = n; }
unsigned __cudaPushCallConfiguration(uint64_t gxy, uint32_t gz, uint64_t bxy, uint32_t bz, size_t smem, void *st) {
    pushed = Config{{(unsigned)gxy, (unsigned)(gxy >> 32), gz}, {(unsigned)bxy, (unsigned)(bxy >> 32), bz}, smem, st};
    return 0;
}
int __cudaPopCallConfiguration(void *g, void *b, size_t *smem, void **st) {
    memcpy(g, pushed.g, 12); memcpy(b, pushed.b, 12); *smem = pushed.smem; *st = pushed.st;
    return 0;
}

// ---- NCCL ----
int ncclGetUniqueId(void *id) { memset(id, 1, 128); return 0; }
struct fake_id { char b[128]; };
int ncclCommInitRank(void **c, int, fake_id, int) { *c = (void *)1; return 0; }
int ncclCommDestroy(void *) { return 0; }
const char *ncclGetErrorString(int) { return "nccl"; }
int ncclAllGather(const void *, void *, size_t, int, void *, void *) { return 0; }
int ncclBroadcast(const void *, void *, size_t, int, int, void *, void *) { return 0; }
int ncclAllReduce(const void *, void *, size_t, int, int, void *, void *) { return 0; }
int ncclGroupStart() { return 0; }
int ncclGroupEnd() { return 0; }
}
