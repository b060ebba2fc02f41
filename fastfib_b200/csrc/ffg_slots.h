// Host copies of an entry point's operands and result, through four pinned slots in
// turn: the CPU fills or empties one while the DMA works on the others (the driver's
// own pageable copies wait for each other: 50001 x 48000 limbs, 1.6 MB of copies,
// 305 -> 200 us a product; 1 000 000 x 900 000, 13 ms -> 2.8; operands that are pinned
// already are no slower this way, 270 -> 176 us and 3.3 -> 2.8 ms).  Where the slots
// cannot be had (no 512 KB of pinned memory), the copies are the driver's own.
//
// Used under the layer's lock, on one stream that is idle when a call begins: a slot's
// earlier copies are over by then, also those of a call that failed midway.
#pragma once
#include <algorithm>
#include <cstddef>
#include <cstring>

#include <cuda_runtime_api.h>

namespace ffg {

struct HostSlots {
    static constexpr size_t kBytes = 128 << 10;
    static constexpr int kCount = 4;
    char *mem = nullptr;
    cudaEvent_t done[kCount] = {};
    int turn = 0; // chunks this call has sent up

    // At the start of a call's copies; makes the slots on first use.  Without them the
    // failure is not kept as the runtime's last error (launches look at it).
    bool ready() {
        turn = 0;
        if (mem) return true;
        cudaError_t e = cudaMallocHost((void **)&mem, kCount * kBytes);
        for (int k = 0; k < kCount && !e; k++) e = cudaEventCreateWithFlags(&done[k], cudaEventDisableTiming);
        if (!e) return true;
        release();
        cudaGetLastError();
        return false;
    }

    void release() {
        for (auto &e : done)
            if (e) cudaEventDestroy(e);
        if (mem) cudaFreeHost(mem);
        *this = HostSlots{};
    }

    // Queues the copy of n bytes of src to the device; src has been read when it returns.
    cudaError_t up(void *dst, const void *src, size_t n, cudaStream_t st) {
        if (!mem) return n ? cudaMemcpyAsync(dst, src, n, cudaMemcpyHostToDevice, st) : cudaSuccess;
        cudaError_t e = cudaSuccess;
        for (size_t at = 0; at < n && !e; at += kBytes) {
            const int k = turn++ % kCount;
            const size_t len = std::min(kBytes, n - at);
            char *slot = mem + k * kBytes;
            if (turn > kCount && (e = cudaEventSynchronize(done[k]))) break;
            memcpy(slot, (const char *)src + at, len);
            e = cudaMemcpyAsync((char *)dst + at, slot, len, cudaMemcpyHostToDevice, st);
            if (!e) e = cudaEventRecord(done[k], st);
        }
        return e;
    }

    // Copies n bytes from the device, queued behind all that st holds (without the
    // slots, complete once st is).
    cudaError_t down(void *dst, const void *src, size_t n, cudaStream_t st) {
        if (!mem) return n ? cudaMemcpyAsync(dst, src, n, cudaMemcpyDeviceToHost, st) : cudaSuccess;
        const size_t chunks = (n + kBytes - 1) / kBytes;
        cudaError_t e = cudaSuccess;
        for (size_t c = 0; c < chunks + kCount && !e; c++) {
            char *slot = mem + c % kCount * kBytes;
            cudaEvent_t ev = done[c % kCount];
            if (c >= (size_t)kCount) { // chunk c - kCount has its slot until here
                const size_t at = (c - kCount) * kBytes;
                if (at < n) {
                    if ((e = cudaEventSynchronize(ev))) break;
                    memcpy((char *)dst + at, slot, std::min(kBytes, n - at));
                }
            }
            if (c < chunks) {
                const size_t at = c * kBytes;
                e = cudaMemcpyAsync(slot, (const char *)src + at, std::min(kBytes, n - at), cudaMemcpyDeviceToHost, st);
                if (!e) e = cudaEventRecord(ev, st);
            }
        }
        return e;
    }
};

} // namespace ffg
