// hostcopy.cu -- copies from device memory to ordinary (pageable) host buffers.
//
// The driver's staging writes a buffer whose pages are there at 17 GB/s (10 MB), but a fresh one,
// such as a newly allocated result array, at 2.3 GB/s: its one thread takes a page fault every
// 4 KB.  Here several threads take those faults first, and the driver copies what is ready behind
// them: 10 MB into fresh pages 4.55 -> 2.3 ms, 2.5 MB 1.16 -> 0.8 ms, 40 MB 18.2 -> 6.4 ms.
// Nothing is allocated: pinned chunks of the framework's own reach the same rates, but pinning
// 8 MB of them cost the first copy after a handle's creation 4 to 8 ms.
#include <sched.h>
#include <sys/mman.h>
#include <unistd.h>

#include <algorithm>
#include <atomic>
#include <cstdint>
#include <exception>
#include <memory>
#include <new>
#include <thread>
#include <vector>

#include "sim.cuh"

namespace ariel {
namespace hostimpl {
namespace {

constexpr size_t kPart = 512 * 1024;  // what a thread makes ready at a time
// Fresh bytes below which the faults are left to the driver's thread (1 MB is level, 0.48 ms;
// 512 KB is 0.25 ms either way).
constexpr size_t kFresh = 1024 * 1024;
// Ready bytes that the caller copies at a time while others still work (the copies wait for
// the device one by one: 512 KB each reach 10.5 GB/s, 2.5 MB 15.8).
constexpr size_t kRun = 2 * 1024 * 1024;
// Host threads of one copy, the caller among them: at most four, and no more than the CPUs that the
// caller may run on, where more of them would only take turns with it.
int workers() {
    constexpr int kMost = 4;
    cpu_set_t may;
    if (sched_getaffinity(0, sizeof(may), &may) != 0)  // more CPUs than the set holds
        return kMost;
    return std::min(kMost, std::max(1, CPU_COUNT(&may)));
}

// Joins its threads when it goes.
struct Helpers {
    std::vector<std::thread> t;
    // up to `n` threads (fewer if they cannot be started) that run `work`
    template <class F>
    Helpers(int n, const F& work) {
        try {
            t.reserve((size_t)std::max(n, 0));
            for (int i = 0; i < n; ++i) t.emplace_back(work);
        } catch (const std::exception&) {
            // no memory or no thread: those that there are do the work, the caller at least
        }
    }
    ~Helpers() {
        for (auto& x : t) x.join();
    }
};

bool pinned_host(const void* p) {
    cudaPointerAttributes a{};
    if (cudaPointerGetAttributes(&a, p) != cudaSuccess) {
        cudaGetLastError();
        return false;
    }
    return a.type == cudaMemoryTypeHost || a.type == cudaMemoryTypeManaged;
}

// Whether most pages of [p, p + bytes) (at most kPart of it is looked at) are not mapped yet.
bool fresh_pages(const char* p, size_t bytes, size_t page) {
    unsigned char v[kPart / 4096 + 2];
    const uintptr_t a = (uintptr_t)p & ~(uintptr_t)(page - 1);
    const uintptr_t b = (uintptr_t)p + std::min(bytes, kPart);
    const size_t n = (b - a + page - 1) / page;
    if (page < 4096 || n > sizeof(v) || mincore((void*)a, b - a, v) != 0) return false;
    size_t out = 0;
    for (size_t i = 0; i < n; ++i) out += (v[i] & 1) == 0;
    return 2 * out > n;
}

bool fresh(const char* p, size_t bytes, size_t page) {
    const size_t tail = bytes > kPart ? bytes - kPart : 0;
    return !pinned_host(p) && (fresh_pages(p, bytes, page) || fresh_pages(p + tail, bytes - tail, page));
}

// A write fault on every page of [p, p + bytes); the bytes keep their values.
void touch(char* p, size_t bytes, size_t page) {
    for (size_t o = 0; o < bytes; o += page) __atomic_fetch_or(p + o, (char)0, __ATOMIC_RELAXED);
    __atomic_fetch_or(p + bytes - 1, (char)0, __ATOMIC_RELAXED);
}

// Device bytes to host int32 through a buffer of the bytes.
cudaError_t download_i32(cudaStream_t st, const HostPiece& h) {
    const std::unique_ptr<uint8_t[]> f(new (std::nothrow) uint8_t[h.bytes]);
    if (!f) return cudaErrorMemoryAllocation;
    const HostPiece bytes{f.get(), h.dev, h.bytes};
    cudaError_t e = download(st, &bytes, 1);
    if (e != cudaSuccess) return e;
    int32_t* const out = static_cast<int32_t*>(h.host);
    constexpr size_t kElems = kPart / sizeof(int32_t);
    const size_t n = (h.bytes + kElems - 1) / kElems;
    std::atomic<size_t> next{0};
    auto work = [&] {
        for (size_t i = next++; i < n; i = next++)
            for (size_t j = i * kElems, end = std::min(j + kElems, h.bytes); j < end; ++j) out[j] = f[j];
    };
    Helpers helpers((int)std::min<size_t>(workers(), n) - 1, work);
    work();
    return cudaSuccess;
}

}  // namespace

// Throws nothing: without memory for its lists every piece goes the driver's way alone.
cudaError_t download(cudaStream_t st, const HostPiece* pieces, int count) {
    struct Part {
        const HostPiece* h;
        size_t off, bytes;
    };
    const size_t page = (size_t)sysconf(_SC_PAGESIZE);
    size_t total = 0;
    for (int i = 0; i < count; ++i)
        if (!pieces[i].to_i32) total += pieces[i].bytes;
    std::vector<Part> parts;
    std::vector<std::atomic<bool>> ready;
    auto in_parts = [&](const HostPiece& h) {
        return std::any_of(parts.begin(), parts.end(), [&](const Part& p) { return p.h == &h; });
    };
    try {
        for (int i = 0; i < count; ++i) {
            const HostPiece& h = pieces[i];
            if (h.bytes == 0 || h.to_i32) continue;
            if (total >= kFresh && fresh(static_cast<const char*>(h.host), h.bytes, page))
                for (size_t o = 0; o < h.bytes; o += kPart) parts.push_back({&h, o, std::min(kPart, h.bytes - o)});
        }
        ready = std::vector<std::atomic<bool>>(parts.size());
    } catch (const std::bad_alloc&) {
        parts.clear();
    }
    const size_t n = parts.size();
    std::atomic<size_t> next{0};
    cudaError_t e = cudaSuccess;
    {
        auto take = [&] {
            const size_t i = next++;
            if (i >= n) return false;
            touch(static_cast<char*>(parts[i].h->host) + parts[i].off, parts[i].bytes, page);
            ready[i].store(true, std::memory_order_release);
            return true;
        };
        Helpers helpers((int)std::min<size_t>(workers(), (n + 1) / 2) - 1, [&] {
            while (take()) {
            }
        });
        size_t done = 0;  // parts copied so far
        // copies the parts from `done` on that are ready, a piece at a time
        auto flush = [&](bool all) {
            while (done < n && e == cudaSuccess) {
                const HostPiece* h = parts[done].h;
                size_t r = done, bytes = 0;
                for (; r < n && parts[r].h == h; ++r) {
                    while (all && !ready[r].load(std::memory_order_acquire)) std::this_thread::yield();
                    if (!ready[r].load(std::memory_order_acquire)) break;
                    bytes += parts[r].bytes;
                }
                if (bytes == 0 || (!all && bytes < kRun)) return;
                const size_t o = parts[done].off;
                e = cudaMemcpyAsync(static_cast<char*>(h->host) + o, static_cast<const char*>(h->dev) + o, bytes,
                                    cudaMemcpyDeviceToHost, st);
                done = r;
            }
        };
        while (take()) flush(false);
        flush(true);
    }
    for (int i = 0; i < count && e == cudaSuccess; ++i) {
        const HostPiece& h = pieces[i];
        if (h.bytes == 0) continue;
        if (h.to_i32)
            e = download_i32(st, h);
        else if (!in_parts(h))
            e = cudaMemcpyAsync(h.host, h.dev, h.bytes, cudaMemcpyDeviceToHost, st);
    }
    const cudaError_t se = cudaStreamSynchronize(st);
    return e != cudaSuccess ? e : se;
}

}  // namespace hostimpl
}  // namespace ariel
