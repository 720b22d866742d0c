// host_copy.h -- copies between the device and ordinary (pageable) host arrays.
// Not part of the C ABI.
//
// The driver moves a pageable array through its own staging buffer on the calling
// thread: one core copies at 8..16 GB/s and takes the page faults of a fresh result
// array, 10 to 70 ms for 148 MB on a link that needs 2.7.  Here up to kThreads threads
// move chunks through pinned buffers, each with one chunk on the link while it copies the
// other.  148 MB, 16 cores: to the device 14.2 -> 4.4 ms, back 9.5 -> 4.6 ms, into fresh
// pages 71 -> 10 ms; 4 threads need 17 ms there, 12 need 7 but 24 MB of buffers.
#pragma once
#include <cuda_runtime.h>

#include <atomic>
#include <cstring>
#include <memory>
#include <mutex>
#include <system_error>
#include <thread>

class HostCopy {
public:
    HostCopy() = default;
    HostCopy(const HostCopy &) = delete;
    HostCopy &operator=(const HostCopy &) = delete;
    ~HostCopy()
    {
        for (char *p : pin)
            if (p) cudaFreeHost(p);
    }

    // the caller's hold on the process's instance, taken if it has none: at most kThreads * 2
    // MB of pinned memory, shared by the handles that hold it and freed with the last of
    // them; null if it cannot be had.  Two threads may make their first copies with one
    // handle, so its hold is read and set under the instance's lock.
    static std::shared_ptr<HostCopy> get(std::shared_ptr<HostCopy> &hold) noexcept
    {
        try {
            static std::mutex mu;
            static std::weak_ptr<HostCopy> one;
            std::lock_guard<std::mutex> l(mu);
            if (!hold) hold = one.lock();
            if (!hold) one = hold = std::make_shared<HostCopy>();
            return hold;
        } catch (...) {
            return nullptr;
        }
    }

    // cudaMemcpyAsync(dst, src, n, kind, st), kind to or from the host, on device dev.  A
    // large pageable array is staged, and then the copy is complete on return (as the
    // driver's own is); anything else is the driver's.  hold: where the caller keeps its hold.
    static cudaError_t copy(std::shared_ptr<HostCopy> &hold, int dev, void *dst, const void *src, size_t n,
                            cudaMemcpyKind kind, cudaStream_t st) noexcept
    {
        // Below kMin the driver's copy is as fast: 6.9 MB back took 0.57 ms and varied little,
        // staged 0.43 to 0.59 with the threads' start; at 11 MB 1.04 to 1.22 and 0.99 to 1.14
        if (n >= kMin && pageable(kind == cudaMemcpyHostToDevice ? src : dst)) {
            cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
            const std::shared_ptr<HostCopy> hc = get(hold);
            if (hc && cudaStreamIsCapturing(st, &cap) == cudaSuccess && cap == cudaStreamCaptureStatusNone) {
                std::unique_lock<std::mutex> l(hc->busy, std::try_to_lock);   // in use by another thread: not waited for
                cudaError_t e = cudaSuccess;
                if (l.owns_lock() && hc->staged(dev, (char *)dst, (const char *)src, n, kind, st, e)) return e;
            }
        }
        return cudaMemcpyAsync(dst, src, n, kind, st);
    }

private:
    static constexpr size_t kChunk = 1 << 20, kMin = 16 << 20;
    static constexpr int kThreads = 8;
    char *pin[kThreads] = {};   // two chunks per thread, allocated when a copy first needs them
    std::mutex busy;

    static bool pageable(const void *p)
    {
        cudaPointerAttributes a{};
        if (cudaPointerGetAttributes(&a, p) != cudaSuccess) { cudaGetLastError(); return false; }
        return a.type == cudaMemoryTypeUnregistered;
    }

    // false: nothing was done (no buffers), the caller copies plainly
    bool staged(int dev, char *dst, const char *src, size_t n, cudaMemcpyKind kind, cudaStream_t st, cudaError_t &err)
    {
        const size_t nc = (n + kChunk - 1) / kChunk;
        int want = (int)std::thread::hardware_concurrency(), nt = 0;
        if (want < 1) want = 1;
        if (want > kThreads) want = kThreads;
        if ((size_t)want > (nc + 1) / 2) want = (int)((nc + 1) / 2);
        cudaEvent_t ev[kThreads][2] = {};
        for (; nt < want; nt++) {
            if (!pin[nt] && cudaHostAlloc((void **)&pin[nt], 2 * kChunk, cudaHostAllocPortable) != cudaSuccess) {
                pin[nt] = nullptr;
                break;
            }
            if (cudaEventCreateWithFlags(&ev[nt][0], cudaEventDisableTiming) != cudaSuccess ||
                cudaEventCreateWithFlags(&ev[nt][1], cudaEventDisableTiming) != cudaSuccess)
                break;
        }
        if (nt < want) cudaGetLastError();
        std::atomic<size_t> next{0};
        std::atomic<int> first{(int)cudaSuccess};
        auto work = [&](int w) noexcept {
            cudaError_t e = cudaSetDevice(dev);
            auto extent = [&](size_t c) { return c * kChunk + kChunk < n ? kChunk : n - c * kChunk; };
            if (kind == cudaMemcpyHostToDevice) {
                size_t c;
                for (int k = 0, used = 0; e == cudaSuccess && (c = next++) < nc; k ^= 1, used++) {
                    char *b = pin[w] + k * kChunk;
                    if (used > 1) e = cudaEventSynchronize(ev[w][k]);
                    if (e != cudaSuccess) break;
                    memcpy(b, src + c * kChunk, extent(c));
                    e = cudaMemcpyAsync(dst + c * kChunk, b, extent(c), kind, st);
                    if (e == cudaSuccess) e = cudaEventRecord(ev[w][k], st);
                }
            } else {
                size_t c[2];
                auto issue = [&](int k) {
                    c[k] = next++;
                    if (c[k] >= nc || e != cudaSuccess) return;
                    e = cudaMemcpyAsync(pin[w] + k * kChunk, src + c[k] * kChunk, extent(c[k]), kind, st);
                    if (e == cudaSuccess) e = cudaEventRecord(ev[w][k], st);
                };
                issue(0);
                issue(1);
                for (int k = 0; e == cudaSuccess && c[k] < nc; k ^= 1) {
                    e = cudaEventSynchronize(ev[w][k]);
                    if (e != cudaSuccess) break;
                    memcpy(dst + c[k] * kChunk, pin[w] + k * kChunk, extent(c[k]));
                    issue(k);
                }
            }
            if (e != cudaSuccess) {
                int none = (int)cudaSuccess;
                first.compare_exchange_strong(none, (int)e);
                next = nc;   // the others stop too
            }
        };
        if (nt > 0) {
            std::thread t[kThreads];
            for (int w = 1; w < nt; w++) {
                try {
                    t[w] = std::thread(work, w);
                } catch (const std::system_error &) {
                    break;   // the threads there are do it all
                }
            }
            work(0);
            for (auto &x : t)
                if (x.joinable()) x.join();
            err = (cudaError_t)first.load();
            // the buffers are free for the next copy only when the link has read them
            if (kind == cudaMemcpyHostToDevice || err != cudaSuccess) {
                const cudaError_t e = cudaStreamSynchronize(st);
                if (err == cudaSuccess) err = e;
            }
        }
        for (auto &p : ev)
            for (cudaEvent_t x : p)
                if (x) cudaEventDestroy(x);
        return nt > 0;
    }
};
