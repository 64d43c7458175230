// The staged copies (csrc/rtg_copy.cpp) against a CUDA runtime of the host's: a stream is a queue of work
// that runs in order when it is waited for, and cudaStreamPerThread names another queue in each
// thread. The program's argument names the case; it prints the number of wrong bytes.
#include "../repackshot_b200/csrc/rtg_copy.cpp"

#include <chrono>
#include <cstdio>
#include <cstdlib>
#include <functional>
#include <map>
#include <mutex>
#include <new>
#include <string>
#include <utility>
#include <vector>

namespace {
std::mutex g_lock;
std::atomic<bool> g_no_memory{false};
using Queue = std::vector<std::function<void()>>;
std::map<std::pair<cudaStream_t, std::thread::id>, Queue> g_streams;
std::map<cudaEvent_t, std::pair<cudaStream_t, std::thread::id>> g_events;

std::pair<cudaStream_t, std::thread::id> stream_of(cudaStream_t s) {
    return {s, s == cudaStreamPerThread ? std::this_thread::get_id() : std::thread::id()};
}
void enqueue(cudaStream_t s, std::function<void()> work) {
    std::lock_guard<std::mutex> lk(g_lock);
    g_streams[stream_of(s)].push_back(std::move(work));
}
// Streams run beside each other: a stream's work holds its own lock only.
std::map<std::pair<cudaStream_t, std::thread::id>, std::mutex> g_running;
void drain(const std::pair<cudaStream_t, std::thread::id>& s) {
    std::mutex* running;
    {
        std::lock_guard<std::mutex> lk(g_lock);
        running = &g_running[s];
    }
    std::lock_guard<std::mutex> run(*running);
    Queue work;
    {
        std::lock_guard<std::mutex> lk(g_lock);
        work.swap(g_streams[s]);
    }
    for (auto& w : work) w();
}
}  // namespace

// Another thread captures a stream of its own in the global mode: an allocation outside the relaxed mode
// breaks that capture.
static bool g_captured_elsewhere = false, g_capture_broken = false;
static thread_local cudaStreamCaptureMode t_capture_mode = cudaStreamCaptureModeGlobal;

// Memory for threads runs out on request; this program's own bookkeeping keeps its.
static thread_local bool t_mine = false;
struct Mine {
    bool was = t_mine;
    Mine() { t_mine = true; }
    ~Mine() { t_mine = was; }
};
void* operator new(size_t n) {
    if (g_no_memory && !t_mine) throw std::bad_alloc();
    if (void* p = std::malloc(n)) return p;
    throw std::bad_alloc();
}
void operator delete(void* p) noexcept { std::free(p); }
void operator delete(void* p, size_t) noexcept { std::free(p); }

extern "C" {
cudaError_t cudaMemcpyAsync(void* to, const void* from, size_t n, cudaMemcpyKind, cudaStream_t s) {
    Mine m;
    enqueue(s, [=] { std::memcpy(to, from, n); });
    return cudaSuccess;
}
cudaError_t cudaStreamSynchronize(cudaStream_t s) {
    Mine m;
    drain(stream_of(s));
    return cudaSuccess;
}
cudaError_t cudaEventCreateWithFlags(cudaEvent_t* e, unsigned) {
    Mine m;
    static std::atomic<uintptr_t> next{1};
    *e = (cudaEvent_t)next++;
    return cudaSuccess;
}
cudaError_t cudaEventDestroy(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t e, cudaStream_t s) {
    Mine m;
    std::lock_guard<std::mutex> lk(g_lock);
    g_events[e] = stream_of(s);
    return cudaSuccess;
}
cudaError_t cudaEventSynchronize(cudaEvent_t e) {
    Mine m;
    std::pair<cudaStream_t, std::thread::id> s;
    {
        std::lock_guard<std::mutex> lk(g_lock);
        s = g_events[e];
    }
    drain(s);
    return cudaSuccess;
}
cudaError_t cudaPointerGetAttributes(cudaPointerAttributes* a, const void*) {
    a->type = cudaMemoryTypeUnregistered;
    return cudaSuccess;
}
cudaError_t cudaGetLastError() { return cudaSuccess; }
cudaError_t cudaThreadExchangeStreamCaptureMode(cudaStreamCaptureMode* mode) {
    std::swap(t_capture_mode, *mode);
    return cudaSuccess;
}
cudaError_t cudaHostAlloc(void** p, size_t n, unsigned) {
    if (t_capture_mode != cudaStreamCaptureModeRelaxed) g_capture_broken = g_captured_elsewhere;
    *p = std::malloc(n);
    return cudaSuccess;
}
cudaError_t cudaFreeHost(void* p) {
    std::free(p);
    return cudaSuccess;
}
cudaError_t cudaStreamIsCapturing(cudaStream_t, cudaStreamCaptureStatus* status) {
    *status = cudaStreamCaptureStatusNone;
    return cudaSuccess;
}
cudaError_t cudaGetDevice(int* d) {
    *d = 0;
    return cudaSuccess;
}
cudaError_t cudaSetDevice(int) { return cudaSuccess; }
}

int main(int argc, char** argv) {
    const std::string mode = argc > 1 ? argv[1] : "stream";
    const size_t n = argc > 2 ? std::strtoull(argv[2], nullptr, 10) : (9u << 20) + 12345;
    const cudaStream_t stream = mode == "per-thread" ? cudaStreamPerThread : (cudaStream_t)(uintptr_t)64;
    g_captured_elsewhere = mode == "captured-elsewhere";
    size_t wrong = 0;
    for (const bool to_device : {false, true}) {
        std::vector<uint8_t> from(n, 1), to(n, 0);
        // A kernel in the stream writes what a copy down reads; one after a copy up reads what it wrote.
        if (!to_device) enqueue(stream, [&] { std::this_thread::sleep_for(std::chrono::milliseconds(100)); for (size_t k = 0; k < n; ++k) from[k] = (uint8_t)(k * 7 + k / 251); });
        else for (size_t k = 0; k < n; ++k) from[k] = (uint8_t)(k * 7 + k / 251);
        const size_t a = n / 3;
        const rtg::CopyPart parts[2] = {{to_device ? from.data() : to.data(), to_device ? to.data() : from.data(), a},
                                        {(to_device ? from.data() : to.data()) + a, (to_device ? to.data() : from.data()) + a, n - a}};
        g_no_memory = mode == "no-memory";
        const cudaError_t e = rtg::copy_planes(parts, 2, to_device, stream);
        g_no_memory = false;
        if (e != cudaSuccess) return 2;
        for (size_t k = 0; k < n; ++k) wrong += to[k] != (uint8_t)(k * 7 + k / 251);
    }
    rtg::copy_release();
    if (g_capture_broken || t_capture_mode != cudaStreamCaptureModeGlobal) return 3;
    std::printf("%zu\n", wrong);
    return 0;
}
