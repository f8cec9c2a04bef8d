// Two pinned chunks that device memory lands in on its way into a caller's array, and the events that say when.
#pragma once
#include <cuda_runtime.h>

#include <algorithm>
#include <cstddef>
#include <cstdint>

namespace oxrt {

struct Landing {
    static constexpr size_t kBytes = 256 * 1024;  // of a chunk
    uint8_t* pinned = nullptr;
    cudaEvent_t events[2] = {};

    Landing() = default;
    Landing(const Landing&) = delete;
    Landing& operator=(const Landing&) = delete;
    ~Landing() {
        if (pinned) cudaFreeHost(pinned);
        for (auto e : events)
            if (e) cudaEventDestroy(e);
    }

    // Makes what is not there yet. What could not be made is tried again the next time.
    cudaError_t open() {
        for (auto& e : events)
            if (!e)
                if (const cudaError_t err = cudaEventCreateWithFlags(&e, cudaEventDisableTiming)) return e = nullptr, err;
        if (!pinned)
            if (const cudaError_t err = cudaMallocHost((void**)&pinned, 2 * kBytes)) return pinned = nullptr, err;
        return cudaSuccess;
    }

    // `nbytes` from `src`, `take(offset, bytes, n)` called in order: one chunk is read while the other lands.
    template <class F> cudaError_t land(const uint8_t* src, size_t nbytes, cudaStream_t stream, F&& take) {
        if (const cudaError_t err = open()) return err;
        const size_t chunks = (nbytes + kBytes - 1) / kBytes;
        auto ask = [&](size_t i) {
            const cudaError_t err = cudaMemcpyAsync(pinned + (i & 1) * kBytes, src + i * kBytes, std::min(kBytes, nbytes - i * kBytes), cudaMemcpyDeviceToHost, stream);
            return err ? err : cudaEventRecord(events[i & 1], stream);
        };
        if (const cudaError_t err = ask(0)) return err;
        for (size_t i = 0; i < chunks; i++) {
            if (i + 1 < chunks)
                if (const cudaError_t err = ask(i + 1)) return err;
            if (const cudaError_t err = cudaEventSynchronize(events[i & 1])) return err;
            take(i * kBytes, pinned + (i & 1) * kBytes, std::min(kBytes, nbytes - i * kBytes));
        }
        return cudaSuccess;
    }
};

}  // namespace oxrt
