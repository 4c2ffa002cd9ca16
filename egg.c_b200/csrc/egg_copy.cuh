// Host and device memory of contexts: one device allocation for a context's buffers, pinned blocks shared by the contexts of a
// process, and device-to-host copies into ordinary (pageable) memory.
#pragma once

#include "egg_common.cuh"

#include <vector>

namespace egg {

// Buffers carved out of one cudaMalloc: an allocation costs about 0.36 ms whatever its size, and a context has some forty.
class DeviceArena {
    struct Want { void **p; int64_t bytes; };
    std::vector<Want> wants;
    int64_t total = 0;

public:
    template <typename T>
    void add(T **p, int64_t count) {
        const int64_t bytes = ((count > 0 ? count : 1) * (int64_t)sizeof(T) + 1023) & ~(int64_t)1023;
        wants.push_back({reinterpret_cast<void **>(p), bytes});
        total += bytes;
    }
    int64_t bytes() const { return total; }
    int commit(void **base);                       // EGG_OK or EGG_E_NOMEM; the caller frees *base
    void place(void *base) const {                 // in memory that is there, bytes() long
        uint8_t *at = static_cast<uint8_t *>(base);
        for (const Want &w : wants) { *w.p = at; at += w.bytes; }
    }
};

// Pinned host memory in blocks of PIN_BLOCK bytes.  Pinning costs milliseconds, so the blocks belong to the process: every context
// retains the pool, blocks are lent out and given back (any thread), and the memory is released with the last context.
constexpr int64_t PIN_BLOCK = 512 << 10;
void pinned_retain();
void pinned_release();
uint8_t *pinned_take();                            // for copies; null when these hold 256 MB or pinning fails
void pinned_give(uint8_t *block);
// A context's own block, as long as it lives: seven to a block of the pool, as many as there are contexts.
constexpr int64_t PIN_STATUS = 72 << 10;
uint8_t *pinned_take_status();                     // null when pinning fails
void pinned_give_status(uint8_t *block);

// Copies into pageable memory: the driver moves them through one staging buffer on one CPU thread, page faults of a fresh
// destination included: 4 to 7 GB/s, 2 to 3 ms for the 13 to 18 MB of a model.  Here a few threads each drain a pair of
// pinned blocks, so that the copy engine, the memory copies and the page faults overlap.  Blocks of 512 KB: the copy engine moves 64 KB
// at 11 GB/s, 256 KB at 31, 1 MB at 46 and 16 MB at 55.  Threads by blocks: 18.9 MB took 1.2 ms with 4 x 256 KB, 0.9 with 8 x 512 KB; 59 MB
// 6.3 and 3.7 (what remains are the page faults of the destination).  Below eight blocks the driver's own copy is as fast.
struct HostStage {
    static constexpr int THREADS = 8;
    cudaEvent_t ev[2 * THREADS] = {};
};
void host_stage_free(HostStage &h);
// After everything enqueued on the stream; returns when the bytes are in place.
int download_to_host(HostStage &h, int device, cudaStream_t st, void *dst, const void *src, int64_t bytes);

}  // namespace egg
