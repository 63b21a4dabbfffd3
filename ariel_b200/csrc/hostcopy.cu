// hostcopy.cu -- copies between device memory and ordinary (pageable) host buffers.
//
// A plain cudaMemcpyAsync to pageable memory is staged by one thread inside the driver, which
// also takes the page faults of a fresh result array: 211,584 particles came out at 3 GB/s.
// Here the copy goes through pinned chunks: the device fills them at the link's rate while up to
// kWorkers host threads move the finished ones, so that the host's share (the memory copy and
// the first touch of the pages) runs in parallel and beside the transfer.
#include <algorithm>
#include <atomic>
#include <mutex>
#include <system_error>
#include <thread>
#include <vector>

#include "sim.cuh"

namespace ariel {
namespace hostimpl {
namespace {

constexpr size_t kChunk = 512 * 1024;
constexpr size_t kDirect = 192 * 1024;  // below this the driver's own staging is as fast
constexpr int kSlots = 16;              // chunks of one copy in flight
constexpr int kPool = 4 * kSlots;       // pinned chunks kept for the next copies: 32 MB at most
constexpr int kWorkers = 4;             // host threads of one copy, the caller among them

struct Slot {
    void* p = nullptr;
    cudaEvent_t ev = nullptr;
    int device = 0;
};

// Pinned chunks shared by all handles.  A copy takes what it needs and gives it back; chunks
// beyond kPool are freed at once, the others with the last handle.
struct Pool {
    std::mutex m;
    std::vector<Slot> free;
    int handles = 0;
};
Pool& pool() {
    static Pool* p = new Pool;  // never destroyed: threads may outlive static destruction
    return *p;
}

void drop(const Slot& s) {
    cudaEventDestroy(s.ev);
    cudaFreeHost(s.p);
}

struct Lease {
    std::vector<Slot> slots;
    // Up to `n` chunks for the current device; fewer (or none) when pinned memory is short.
    Lease(int device, int n) {
        Pool& P = pool();
        {
            std::lock_guard<std::mutex> l(P.m);
            for (size_t i = P.free.size(); i-- > 0 && (int)slots.size() < n;)
                if (P.free[i].device == device) {
                    slots.push_back(P.free[i]);
                    P.free.erase(P.free.begin() + (long)i);
                }
        }
        while ((int)slots.size() < n) {
            Slot s;
            s.device = device;
            if (cudaHostAlloc(&s.p, kChunk, cudaHostAllocDefault) != cudaSuccess) {
                cudaGetLastError();
                break;
            }
            if (cudaEventCreateWithFlags(&s.ev, cudaEventDisableTiming) != cudaSuccess) {
                cudaGetLastError();
                cudaFreeHost(s.p);
                break;
            }
            slots.push_back(s);
        }
    }
    ~Lease() {
        Pool& P = pool();
        std::lock_guard<std::mutex> l(P.m);
        for (const Slot& s : slots) {
            if (P.handles > 0 && (int)P.free.size() < kPool)
                P.free.push_back(s);
            else
                drop(s);
        }
    }
};

// Runs `work` on the caller and `extra` more threads (fewer if they cannot be started).
template <class F>
void on_threads(int device, int extra, F&& work) {
    std::vector<std::thread> t;
    t.reserve((size_t)extra);
    for (int i = 0; i < extra; ++i) {
        try {
            t.emplace_back([&work, device] {
                cudaSetDevice(device);
                work();
            });
        } catch (const std::system_error&) {
            break;
        }
    }
    work();
    for (auto& x : t) x.join();
}

bool pinned_host(const void* p) {
    cudaPointerAttributes a{};
    if (cudaPointerGetAttributes(&a, p) != cudaSuccess) {
        cudaGetLastError();
        return false;
    }
    return a.type == cudaMemoryTypeHost || a.type == cudaMemoryTypeManaged;
}

}  // namespace

void host_pool_retain() {
    std::lock_guard<std::mutex> l(pool().m);
    ++pool().handles;
}

void host_pool_release() {
    Pool& P = pool();
    std::lock_guard<std::mutex> l(P.m);
    if (--P.handles > 0) return;
    for (const Slot& s : P.free) drop(s);
    P.free.clear();
}

cudaError_t download(cudaStream_t st, const std::vector<HostPiece>& pieces) {
    struct Part {
        const HostPiece* h;
        size_t off, bytes;
    };
    std::vector<Part> parts;
    cudaError_t e = cudaSuccess;
    size_t total = 0;
    for (const HostPiece& h : pieces) total += h.bytes;
    for (const HostPiece& h : pieces) {
        if (h.bytes == 0) continue;
        if (!h.to_i32 && (total < kDirect || pinned_host(h.host))) {
            e = cudaMemcpyAsync(h.host, h.dev, h.bytes, cudaMemcpyDeviceToHost, st);
            if (e != cudaSuccess) return e;
            continue;
        }
        for (size_t o = 0; o < h.bytes; o += kChunk) parts.push_back({&h, o, std::min(kChunk, h.bytes - o)});
    }
    if (parts.empty()) return cudaStreamSynchronize(st);
    int device = 0;
    cudaGetDevice(&device);
    const int n = (int)parts.size();
    Lease lease(device, std::min(n, kSlots));
    const int m = (int)lease.slots.size();
    if (m == 0) {
        // no pinned memory to be had: the driver's staging
        for (const HostPiece& h : pieces) {
            if (h.to_i32) {
                std::vector<uint8_t> f(h.bytes);
                e = copy_sync(st, f.data(), h.dev, h.bytes, cudaMemcpyDeviceToHost);
                if (e != cudaSuccess) return e;
                for (size_t i = 0; i < h.bytes; ++i) static_cast<int32_t*>(h.host)[i] = f[i];
            } else {
                e = copy_sync(st, h.host, h.dev, h.bytes, cudaMemcpyDeviceToHost);
                if (e != cudaSuccess) return e;
            }
        }
        return cudaStreamSynchronize(st);
    }
    std::atomic<int> err{0}, next{0};
    std::vector<std::atomic<int>> issued((size_t)m);  // the part whose copy into the slot is queued
    auto issue = [&](int i) {
        const Slot& s = lease.slots[(size_t)(i % m)];
        const Part& p = parts[(size_t)i];
        cudaError_t r = cudaMemcpyAsync(s.p, static_cast<const char*>(p.h->dev) + p.off, p.bytes, cudaMemcpyDeviceToHost, st);
        if (r == cudaSuccess) r = cudaEventRecord(s.ev, st);
        if (r != cudaSuccess) err = (int)r;
        issued[(size_t)(i % m)].store(i, std::memory_order_release);
    };
    for (auto& x : issued) x = -1;
    for (int i = 0; i < m; ++i) issue(i);
    on_threads(device, std::min(kWorkers, (n + 1) / 2) - 1, [&] {
        for (int i = next++; i < n; i = next++) {
            // (the part before it in its slot was taken earlier, so its issuer is at work)
            while (issued[(size_t)(i % m)].load(std::memory_order_acquire) != i) std::this_thread::yield();
            const Slot& s = lease.slots[(size_t)(i % m)];
            const Part& p = parts[(size_t)i];
            if (err == 0) {
                const cudaError_t r = cudaEventSynchronize(s.ev);
                if (r != cudaSuccess) err = (int)r;
            }
            if (err == 0) {
                if (p.h->to_i32) {
                    const uint8_t* f = static_cast<const uint8_t*>(s.p);
                    int32_t* o = static_cast<int32_t*>(p.h->host) + p.off;
                    for (size_t j = 0; j < p.bytes; ++j) o[j] = f[j];
                } else {
                    std::memcpy(static_cast<char*>(p.h->host) + p.off, s.p, p.bytes);
                }
            }
            if (i + m < n) issue(i + m);
        }
    });
    e = cudaStreamSynchronize(st);
    return err ? (cudaError_t)err.load() : e;
}

cudaError_t upload(cudaStream_t st, void* dev, const void* host, size_t bytes) {
    if (bytes < kDirect || pinned_host(host)) return copy_sync(st, dev, host, bytes, cudaMemcpyHostToDevice);
    int device = 0;
    cudaGetDevice(&device);
    const int n = (int)((bytes + kChunk - 1) / kChunk);
    Lease lease(device, std::min(n, kSlots));
    const int m = (int)lease.slots.size();
    if (m == 0) return copy_sync(st, dev, host, bytes, cudaMemcpyHostToDevice);
    std::atomic<int> err{0}, next{0};
    std::vector<std::atomic<int>> queued((size_t)m);  // the last part queued from the slot
    for (auto& x : queued) x = -1;
    on_threads(device, std::min(kWorkers, (n + 1) / 2) - 1, [&] {
        for (int i = next++; i < n; i = next++) {
            const Slot& s = lease.slots[(size_t)(i % m)];
            const size_t off = (size_t)i * kChunk, len = std::min(kChunk, bytes - off);
            cudaError_t r = cudaSuccess;
            if (i >= m) {
                while (queued[(size_t)(i % m)].load(std::memory_order_acquire) != i - m) std::this_thread::yield();
                r = cudaEventSynchronize(s.ev);
            }
            if (r == cudaSuccess && err == 0) {
                std::memcpy(s.p, static_cast<const char*>(host) + off, len);
                r = cudaMemcpyAsync(static_cast<char*>(dev) + off, s.p, len, cudaMemcpyHostToDevice, st);
                if (r == cudaSuccess) r = cudaEventRecord(s.ev, st);
            }
            if (r != cudaSuccess) err = (int)r;
            queued[(size_t)(i % m)].store(i, std::memory_order_release);
        }
    });
    const cudaError_t e = cudaStreamSynchronize(st);
    return err ? (cudaError_t)err.load() : e;
}

}  // namespace hostimpl
}  // namespace ariel
