// A plain cudaMemcpy of pageable memory goes through the driver's staging buffer on one thread: 11
// GB/s up, 20 GB/s down, 2 GB/s down into pages never touched, whatever the number of streams (52 MB
// up in 2 to 16 slices on streams of their own: 4.3 to 4.9 ms; whole 4.4 to 4.9). Here LANES threads
// each copy through two pinned slots of their own, one filled or emptied while the other is on its
// way: 52 MB up 1.8 ms, 15 MB down into fresh pages 2.0 instead of 6.5 ms. 4 threads with slots of 1 MB, 8
// with 1 MB and 8 with 512 KB: a denoiser call (both copies) 4.02, 4.34 and 4.94 ms, a film of 50 MB read
// into fresh pages 3.8, 3.2 and 3.4 ms, into used ones 1.95, 1.85 and 2.3 ms. More threads down and fewer
// up would suit both.
#include "rtg_copy.h"

#include <algorithm>
#include <atomic>
#include <cstdint>
#include <cstring>
#include <exception>
#include <thread>

namespace rtg {
namespace {
constexpr int LANES = 4;
constexpr size_t SLOT = 1u << 20;
// Below this much a thread costs what it saves.
constexpr size_t LEAST = 4u << 20;
uint8_t* g_pinned = nullptr;  // 2 * LANES slots, kept until copy_release

cudaError_t plain(const CopyPart* parts, int n, bool to_device, cudaStream_t stream) {
    for (int k = 0; k < n; ++k) {
        const cudaError_t e = to_device ? cudaMemcpyAsync(parts[k].dev, parts[k].host, parts[k].bytes, cudaMemcpyHostToDevice, stream)
                                        : cudaMemcpyAsync(parts[k].host, parts[k].dev, parts[k].bytes, cudaMemcpyDeviceToHost, stream);
        if (e != cudaSuccess) return e;
    }
    return cudaStreamSynchronize(stream);
}

// Pageable memory that CUDA knows nothing of: everything else the copy engines reach themselves.
bool pageable(const void* p) {
    cudaPointerAttributes a;
    if (cudaPointerGetAttributes(&a, p) != cudaSuccess) { cudaGetLastError(); return false; }
    return a.type == cudaMemoryTypeUnregistered;
}

struct Events {
    cudaEvent_t e[2 * LANES] = {};
    bool create() {
        for (auto& v : e)
            if (cudaEventCreateWithFlags(&v, cudaEventDisableTiming) != cudaSuccess) { v = nullptr; return false; }
        return true;
    }
    ~Events() {
        for (auto v : e)
            if (v) cudaEventDestroy(v);
    }
};
}  // namespace

void copy_release() {
    if (g_pinned) cudaFreeHost(g_pinned);
    g_pinned = nullptr;
}

cudaError_t copy_planes(const CopyPart* parts, int n, bool to_device, cudaStream_t stream) {
    size_t total = 0;
    bool ours = true;
    for (int k = 0; k < n; ++k) {
        total += parts[k].bytes;
        ours = ours && (parts[k].bytes == 0 || pageable(parts[k].host));
    }
    cudaStreamCaptureStatus capture = cudaStreamCaptureStatusNone;
    int device = 0;
    // cudaStreamPerThread names another stream in each thread: its order is the calling thread's alone.
    if (total < LEAST || !ours || stream == cudaStreamPerThread || cudaStreamIsCapturing(stream, &capture) != cudaSuccess || capture != cudaStreamCaptureStatusNone ||
        cudaGetDevice(&device) != cudaSuccess) {
        cudaGetLastError();
        return plain(parts, n, to_device, stream);
    }
    if (!g_pinned) {
        // A read takes no memory otherwise, and may go on beside another thread's capture: so in the mode
        // that an allocation does not break one in.
        cudaStreamCaptureMode mode = cudaStreamCaptureModeRelaxed;
        cudaThreadExchangeStreamCaptureMode(&mode);
        if (cudaHostAlloc((void**)&g_pinned, 2 * LANES * SLOT, cudaHostAllocPortable) != cudaSuccess) g_pinned = nullptr;
        cudaThreadExchangeStreamCaptureMode(&mode);
    }
    Events ev;
    // A stream of another device takes no event of this one.
    if (!g_pinned || !ev.create() || cudaEventRecord(ev.e[0], stream) != cudaSuccess) {
        cudaGetLastError();
        return plain(parts, n, to_device, stream);
    }
    size_t pieces = 0;
    for (int k = 0; k < n; ++k) pieces += (parts[k].bytes + SLOT - 1) / SLOT;
    std::atomic<size_t> next{0};
    std::atomic<int> failed{(int)cudaSuccess};
    auto piece = [&](size_t c, uint8_t*& host, uint8_t*& dev, size_t& bytes) {
        for (int k = 0; k < n; ++k) {
            const size_t m = (parts[k].bytes + SLOT - 1) / SLOT;
            if (c < m) {
                host = (uint8_t*)parts[k].host + c * SLOT;
                dev = (uint8_t*)parts[k].dev + c * SLOT;
                bytes = std::min(SLOT, parts[k].bytes - c * SLOT);
                return;
            }
            c -= m;
        }
    };
    auto lane = [&](int id) {
        auto check = [&](cudaError_t e) {
            if (e != cudaSuccess) failed = (int)e;
            return e == cudaSuccess;
        };
        if (!check(cudaSetDevice(device))) return;
        uint8_t* slot[2] = {g_pinned + (2 * id) * SLOT, g_pinned + (2 * id + 1) * SLOT};
        cudaEvent_t* event = ev.e + 2 * id;
        uint8_t *host = nullptr, *dev = nullptr, *host_of[2] = {};
        size_t bytes = 0, bytes_of[2] = {};
        bool flying[2] = {false, false};
        // A slot's copy has ended; a copy down is then taken to its place.
        auto land = [&](int s) {
            if (!flying[s]) return true;
            flying[s] = false;
            if (!check(cudaEventSynchronize(event[s]))) return false;
            if (!to_device) std::memcpy(host_of[s], slot[s], bytes_of[s]);
            return true;
        };
        int s = 0;
        for (size_t c; failed == (int)cudaSuccess && (c = next++) < pieces; s ^= 1) {
            if (!land(s)) return;
            piece(c, host, dev, bytes);
            host_of[s] = host;
            bytes_of[s] = bytes;
            if (to_device) std::memcpy(slot[s], host, bytes);
            if (!check(to_device ? cudaMemcpyAsync(dev, slot[s], bytes, cudaMemcpyHostToDevice, stream)
                                 : cudaMemcpyAsync(slot[s], dev, bytes, cudaMemcpyDeviceToHost, stream)) ||
                !check(cudaEventRecord(event[s], stream)))
                return;
            flying[s] = true;
        }
        if (land(s)) land(s ^ 1);
    };
    std::thread more[LANES - 1];
    for (int k = 1; k < LANES; ++k) {
        try {
            more[k - 1] = std::thread(lane, k);
        } catch (const std::exception&) {  // no thread, or no memory for one
            break;  // the other lanes take its pieces
        }
    }
    lane(0);
    for (auto& t : more)
        if (t.joinable()) t.join();
    const cudaError_t end = cudaStreamSynchronize(stream);  // no slot is in use when it is left
    return failed != (int)cudaSuccess ? (cudaError_t)failed.load() : end;
}

}  // namespace rtg
