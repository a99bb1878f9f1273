// host_copy.h -- large copies between device memory and the caller's (pageable) host memory.
// The driver stages such a copy through its own pinned buffers on the calling thread, one memcpy deep: 9.5 MB take 484 us to the host where
// the link needs 175 (the memcpy alone 530).  Here the pieces go through a pinned ring and up to three threads move them between the ring and the
// caller's memory while the next pieces are on the link: 280 us, the threads' start included.  Smaller copies gain nothing and take
// the driver's way, and so does every copy where the ring or its events cannot be had.
#pragma once
#include <cuda_runtime.h>
#include <string.h>

#include <algorithm>
#include <atomic>
#include <thread>
#include <vector>

namespace lmrs {

// One ring per thread that copies (4 MB), given back when the thread ends.
class HostCopy {
  public:
    static constexpr size_t PIECE = 512 << 10, LEAST = 2 << 20;
    static constexpr int SLOTS = 8, HELPERS = 2;
    static HostCopy& of_this_thread() {
        static thread_local HostCopy c;
        return c;
    }
    ~HostCopy() {
        drop_events();
        if (ring) cudaFreeHost(ring);
    }
    // device -> host: the bytes are there on return (the stream's earlier work is waited for)
    cudaError_t to_host(void* dst, const void* src, size_t bytes, cudaStream_t st) {
        if (!ready(bytes)) {
            const cudaError_t e = cudaMemcpyAsync(dst, src, bytes, cudaMemcpyDeviceToHost, st);
            return e != cudaSuccess ? e : cudaStreamSynchronize(st);
        }
        const int n = (int)((bytes + PIECE - 1) / PIECE);
        auto len = [&](int i) { return std::min(PIECE, bytes - (size_t)i * PIECE); };
        std::vector<std::atomic<char>> done(n);
        for (auto& d : done) d.store(0);
        std::atomic<int> issued{0}, next{0};
        std::atomic<int> error{cudaSuccess};
        auto move = [&](int i) {   // piece i, whose copy has been issued
            cudaError_t e;
            while ((e = cudaEventQuery(event[i % SLOTS])) == cudaErrorNotReady) std::this_thread::yield();
            if (e != cudaSuccess) { error.store(e); return; }
            memcpy(static_cast<char*>(dst) + (size_t)i * PIECE, ring + (size_t)(i % SLOTS) * PIECE, len(i));
            done[i].store(1, std::memory_order_release);
        };
        auto helper = [&]() {
            cudaSetDevice(device);
            for (int i; (i = next.fetch_add(1)) < n;) {
                while (issued.load(std::memory_order_acquire) <= i)
                    if (error.load() != cudaSuccess) return; else std::this_thread::yield();
                move(i);
                if (error.load() != cudaSuccess) return;
            }
        };
        Helpers helpers(helper, n);
        for (int i = 0; error.load() == cudaSuccess;) {
            if (i < n && (i < SLOTS || done[i - SLOTS].load(std::memory_order_acquire))) {
                cudaError_t e = cudaMemcpyAsync(ring + (size_t)(i % SLOTS) * PIECE, static_cast<const char*>(src) + (size_t)i * PIECE, len(i), cudaMemcpyDeviceToHost, st);
                if (e == cudaSuccess) e = cudaEventRecord(event[i % SLOTS], st);
                if (e != cudaSuccess) { error.store(e); break; }
                issued.store(++i, std::memory_order_release);
                continue;
            }
            int mine = next.load();   // otherwise a piece that is on its way, if nobody has taken it
            if (mine < i && next.compare_exchange_strong(mine, mine + 1)) { move(mine); continue; }
            if (i == n && next.load() >= n) break;
            std::this_thread::yield();
        }
        helpers.join();
        if (error.load() != cudaSuccess) return finish((cudaError_t)error.load(), st);
        return cudaSuccess;
    }
    // host -> device, in the stream's order: the source has been read on return
    cudaError_t to_device(void* dst, const void* src, size_t bytes, cudaStream_t st) {
        if (!ready(bytes)) return cudaMemcpyAsync(dst, src, bytes, cudaMemcpyHostToDevice, st);
        const int n = (int)((bytes + PIECE - 1) / PIECE);
        auto len = [&](int i) { return std::min(PIECE, bytes - (size_t)i * PIECE); };
        std::vector<std::atomic<char>> filled(n);
        for (auto& f : filled) f.store(0);
        std::atomic<int> issued{0}, next{0};
        std::atomic<int> error{cudaSuccess};
        auto fill = [&](int i) {   // piece i, whose slot's last copy has been issued
            if (i >= SLOTS) {
                cudaError_t e;
                while ((e = cudaEventQuery(event[i % SLOTS])) == cudaErrorNotReady) std::this_thread::yield();
                if (e != cudaSuccess) { error.store(e); return; }
            }
            memcpy(ring + (size_t)(i % SLOTS) * PIECE, static_cast<const char*>(src) + (size_t)i * PIECE, len(i));
            filled[i].store(1, std::memory_order_release);
        };
        auto helper = [&]() {
            cudaSetDevice(device);
            for (int i; (i = next.fetch_add(1)) < n;) {
                while (issued.load(std::memory_order_acquire) <= i - SLOTS)
                    if (error.load() != cudaSuccess) return; else std::this_thread::yield();
                fill(i);
                if (error.load() != cudaSuccess) return;
            }
        };
        Helpers helpers(helper, n);
        for (int i = 0; i < n && error.load() == cudaSuccess;) {
            if (filled[i].load(std::memory_order_acquire)) {
                cudaError_t e = cudaMemcpyAsync(static_cast<char*>(dst) + (size_t)i * PIECE, ring + (size_t)(i % SLOTS) * PIECE, len(i), cudaMemcpyHostToDevice, st);
                if (e == cudaSuccess) e = cudaEventRecord(event[i % SLOTS], st);
                if (e != cudaSuccess) { error.store(e); break; }
                issued.store(++i, std::memory_order_release);
                continue;
            }
            int mine = next.load();
            if (mine < n && mine < i + SLOTS && next.compare_exchange_strong(mine, mine + 1)) { fill(mine); continue; }
            std::this_thread::yield();
        }
        helpers.join();
        if (error.load() != cudaSuccess) return finish((cudaError_t)error.load(), st);
        return cudaSuccess;
    }

  private:
    char* ring = nullptr;
    cudaEvent_t event[SLOTS] = {};
    int device = -1;   // the events'

    struct Helpers {   // threads for copies of several pieces; none where they cannot be started
        std::vector<std::thread> t;
        template <typename F> Helpers(F& f, int pieces) {
            const int n = std::min({HELPERS, pieces - 1, (int)std::thread::hardware_concurrency() - 1});
            try {
                for (int i = 0; i < n; i++) t.emplace_back(std::ref(f));
            } catch (...) {
            }
        }
        void join() { for (auto& x : t) if (x.joinable()) x.join(); }
        ~Helpers() { join(); }
    };
    void drop_events() {
        for (auto& e : event) { if (e) cudaEventDestroy(e); e = nullptr; }
        device = -1;
    }
    // after an error: nothing may still be using the ring
    cudaError_t finish(cudaError_t e, cudaStream_t st) { (void)cudaStreamSynchronize(st); return e; }
    // the ring and events of the current device, idle; false: the driver's way
    bool ready(size_t bytes) {
        if (bytes < LEAST) return false;
        int dev = 0;
        if (cudaGetDevice(&dev) != cudaSuccess) return false;
        if (!ring && cudaHostAlloc(reinterpret_cast<void**>(&ring), SLOTS * PIECE, cudaHostAllocPortable) != cudaSuccess) { ring = nullptr; (void)cudaGetLastError(); return false; }
        if (device != dev) {
            for (auto& e : event)
                if (e && cudaEventSynchronize(e) != cudaSuccess) return false;
            drop_events();
            for (auto& e : event)
                if (cudaEventCreateWithFlags(&e, cudaEventDisableTiming) != cudaSuccess) { e = nullptr; drop_events(); (void)cudaGetLastError(); return false; }
            device = dev;
        }
        for (auto& e : event)   // (copies of an earlier call, on whichever stream; an event never recorded is complete)
            if (cudaEventSynchronize(e) != cudaSuccess) { (void)cudaGetLastError(); return false; }
        return true;
    }
};

}  // namespace lmrs
