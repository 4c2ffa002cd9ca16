// Device arenas, pinned blocks and copies into pageable memory (see egg_copy.cuh).
#include "egg_copy.cuh"

#include <string.h>

#include <atomic>
#include <mutex>
#include <thread>

namespace egg {

int DeviceArena::commit(void **base) {
    *base = nullptr;
    cudaError_t e = cudaMalloc(base, (size_t)(total > 0 ? total : 1));
    if (e != cudaSuccess) {
        *base = nullptr;
        set_error("cudaMalloc of %lld bytes failed: %s", (long long)total, cudaGetErrorString(e));
        return EGG_E_NOMEM;
    }
    place(*base);
    return EGG_OK;
}

namespace {
struct PinnedPool {
    std::mutex m;
    int users = 0, copy_slabs = 0;
    std::vector<uint8_t *> slabs, free_blocks, free_status;
    bool grow() {
        void *slab = nullptr;
        if (cudaHostAlloc(&slab, PIN_SLAB, cudaHostAllocPortable) != cudaSuccess) { cudaGetLastError(); return false; }
        slabs.push_back(static_cast<uint8_t *>(slab));
        for (int64_t o = PIN_SLAB - PIN_BLOCK; o >= 0; o -= PIN_BLOCK) free_blocks.push_back(static_cast<uint8_t *>(slab) + o);
        return true;
    }
    static constexpr int64_t PIN_SLAB = 4 << 20;
};
PinnedPool g_pins;
constexpr int PIN_MAX_SLABS = 64;
}  // namespace

void pinned_retain() {
    std::lock_guard<std::mutex> l(g_pins.m);
    g_pins.users++;
}
void pinned_release() {
    std::lock_guard<std::mutex> l(g_pins.m);
    if (--g_pins.users > 0) return;
    for (uint8_t *s : g_pins.slabs) cudaFreeHost(s);
    g_pins.slabs.clear();
    g_pins.free_blocks.clear();
    g_pins.free_status.clear();
    g_pins.copy_slabs = 0;
}
uint8_t *pinned_take() {
    std::lock_guard<std::mutex> l(g_pins.m);
    if (g_pins.free_blocks.empty()) {
        if (g_pins.copy_slabs >= PIN_MAX_SLABS || !g_pins.grow()) return nullptr;
        g_pins.copy_slabs++;
    }
    uint8_t *b = g_pins.free_blocks.back();
    g_pins.free_blocks.pop_back();
    return b;
}
void pinned_give(uint8_t *block) {
    if (!block) return;
    std::lock_guard<std::mutex> l(g_pins.m);
    g_pins.free_blocks.push_back(block);
}
uint8_t *pinned_take_status() {
    std::lock_guard<std::mutex> l(g_pins.m);
    if (g_pins.free_status.empty()) {
        if (g_pins.free_blocks.empty() && !g_pins.grow()) return nullptr;
        uint8_t *b = g_pins.free_blocks.back();
        g_pins.free_blocks.pop_back();
        for (int64_t o = PIN_BLOCK / PIN_STATUS - 1; o >= 0; o--) g_pins.free_status.push_back(b + o * PIN_STATUS);
    }
    uint8_t *b = g_pins.free_status.back();
    g_pins.free_status.pop_back();
    return b;
}
void pinned_give_status(uint8_t *block) {
    if (!block) return;
    std::lock_guard<std::mutex> l(g_pins.m);
    g_pins.free_status.push_back(block);
}

void host_stage_free(HostStage &h) {
    for (cudaEvent_t &e : h.ev)
        if (e) { cudaEventDestroy(e); e = nullptr; }
}

int download_to_host(HostStage &h, int device, cudaStream_t st, void *dst, const void *src, int64_t bytes) {
    // small copies are latency, and a pinned destination takes the copy engine's writes itself
    bool direct = bytes < 8 * PIN_BLOCK;
    if (!direct) {
        cudaPointerAttributes a;
        if (cudaPointerGetAttributes(&a, dst) == cudaSuccess) direct = a.type != cudaMemoryTypeUnregistered;
        else cudaGetLastError();
    }
    const int64_t chunks = (bytes + PIN_BLOCK - 1) / PIN_BLOCK;
    const int most = chunks / 4 < HostStage::THREADS ? (int)(chunks / 4) : HostStage::THREADS;     // four blocks and more pay for a thread
    uint8_t *block[2 * HostStage::THREADS] = {};
    int lent = 0;
    if (!direct)
        while (lent < 2 * most && (block[lent] = pinned_take())) lent++;
    struct Return {
        uint8_t **b; int n;
        ~Return() { for (int i = 0; i < n; i++) pinned_give(b[i]); }
    } give_back{block, lent};
    if (direct || lent < 2) {
        EGG_CUDA(cudaMemcpyAsync(dst, src, (size_t)bytes, cudaMemcpyDeviceToHost, st));
        EGG_CUDA(cudaStreamSynchronize(st));
        return EGG_OK;
    }
    for (cudaEvent_t &e : h.ev)
        if (!e) EGG_CUDA(cudaEventCreateWithFlags(&e, cudaEventDisableTiming));
    const int threads = lent / 2;
    std::atomic<int> bad{(int)cudaSuccess};
    auto work = [&](int t) {
        auto check = [&](cudaError_t e) { int ok = (int)cudaSuccess; if (e != cudaSuccess) bad.compare_exchange_strong(ok, (int)e); return e == cudaSuccess; };
        if (t > 0 && !check(cudaSetDevice(device))) return;
        auto size_of = [&](int64_t c) { return (size_t)(c + 1 < chunks ? PIN_BLOCK : bytes - c * PIN_BLOCK); };
        auto fetch = [&](int64_t c, int slot) {
            const int i = 2 * t + slot;
            return check(cudaMemcpyAsync(block[i], (const uint8_t *)src + c * PIN_BLOCK, size_of(c), cudaMemcpyDeviceToHost, st)) &&
                   check(cudaEventRecord(h.ev[i], st));
        };
        int64_t next = t;
        for (int s = 0; s < 2 && next < chunks; s++, next += threads)
            if (!fetch(next, s)) return;
        int slot = 0;
        for (int64_t c = t; c < chunks; c += threads, slot ^= 1) {
            const int i = 2 * t + slot;
            if (!check(cudaEventSynchronize(h.ev[i]))) return;
            memcpy((uint8_t *)dst + c * PIN_BLOCK, block[i], size_of(c));
            if (next < chunks) {
                if (!fetch(next, slot)) return;
                next += threads;
            }
        }
    };
    std::thread helpers[HostStage::THREADS];
    int started = 1;
    try {
        for (; started < threads; started++) helpers[started] = std::thread(work, started);
    } catch (...) {
    }
    work(0);
    for (int t = 1; t < started; t++) helpers[t].join();
    for (int t = started; t < threads; t++) work(t);           // a thread that could not be started: its chunks here
    if (bad != (int)cudaSuccess) {
        cudaStreamSynchronize(st);                             // nothing may still be writing into blocks that go back
        set_error("copy to the host failed: %s", cudaGetErrorString((cudaError_t)bad.load())); return EGG_E_CUDA; }
    return EGG_OK;
}

}  // namespace egg
