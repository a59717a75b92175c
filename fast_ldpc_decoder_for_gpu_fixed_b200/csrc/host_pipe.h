// Staging of pageable host buffers for the host decode calls.
//
// cudaMemcpyAsync from or to pageable memory is a copy through the driver's own staging buffer by
// the calling thread, which neither overlaps the decoding nor uses the memory bandwidth of the host.
// Here a few threads copy pieces of the caller's LLRs into a ring of pinned pieces and expand the
// packed decisions (an eighth of the bytes over PCIe) from another into the caller's 0/1 bytes,
// while the copy engines and the kernels work on the pieces before and after.
// 4000x2000, 4096 frames, 20 iterations, numpy buffers (16.4 MB each way), B200 with 16 cores:
// 2.7 to 3.9 ms a call with cudaMemcpyAsync on the caller's buffers, 0.96 ms through the pieces (the
// kernels alone take 0.63).
//
// A call takes a pipe for its time (HostPipes): pinned memory takes milliseconds to allocate, so at
// most two idle pipes are kept for later calls, of any decoder, until no decoder is left.
#pragma once
#include <algorithm>
#include <atomic>
#include <chrono>
#include <condition_variable>
#include <cstdint>
#include <cstring>
#include <exception>
#include <functional>
#include <mutex>
#include <new>
#include <thread>
#include <vector>

#include <cuda_runtime.h>
#include <unistd.h>

namespace ldpc {

// Threads that share a loop with the caller.  Asleep between calls; from wake() to rest() they spin on
// the loop counter, since a wake-up through the kernel takes as long as a piece's copy, but once CALL has
// passed since wake() only for SPIN without a new loop: then they sleep until there is one (the caller
// waits for the GPU, and other calls and processes need the cores).  16 cores, one caller, us a call and
// us of CPU time, spinning throughout / so: 4000x2000, 280 frames, 10 iterations 173, 950 / 172, 950; 4096
// frames, 20 iterations 930 to 950, 5440 to 5570 / 940, 5500; 200 iterations 7060, 42 200 / 7100, 20 200;
// 20000x10000, 1200 frames, 50 iterations, whose waits are the longest, 7240, 43 200 / 7390, 15 800.  With
// a SPIN of 100 us the 200 iterations take 14 800 us of CPU time, but one call in ten of 0.91 ms takes 0.12
// ms longer (a helper asleep when the last piece comes); without CALL calls of 0.2 ms take 2 to 4 % longer.
// Six callers at once, 4000x2000, 4096 frames: 1070 to 1630, 15 000 to 20 000 / 940, 10 600.
class HostTeam {
public:
    static constexpr std::chrono::microseconds SPIN{250}, CALL{500};
    explicit HostTeam(int helpers)
    {
        try {
            threads_.reserve(helpers);
            for (int i = 0; i < helpers; i++) threads_.emplace_back([this, i] { run(i + 1); });
        } catch (const std::exception&) {
            // no more threads or memory here: the caller and those that started do the work
        }
    }
    ~HostTeam()
    {
        {
            std::lock_guard<std::mutex> l(m_);
            stop_ = true;
            awake_.store(false);
        }
        cv_.notify_all();
        for (auto& t : threads_) t.join();
    }
    int size() const { return (int)threads_.size() + 1; }
    void wake()
    {
        {
            std::lock_guard<std::mutex> l(m_);
            awake_.store(true);
            wakes_++;
        }
        cv_.notify_all();
    }
    void rest() { awake_.store(false); }
    // f(part, parts) for every part, one a thread; returns when all are done
    void each(const std::function<void(int, int)>& f)
    {
        f_ = &f;
        done_.store(0, std::memory_order_relaxed);
        turn_.fetch_add(1);
        // a helper counts itself asleep before it looks at turn_ for the last time, under the lock: it
        // is seen here, or it sees the new turn (both sequentially consistent)
        if (asleep_.load()) {
            { std::lock_guard<std::mutex> l(m_); }
            cv_.notify_all();
        }
        f(0, size());
        while (done_.load(std::memory_order_acquire) < size() - 1) std::this_thread::yield();
    }

private:
    void run(int part)
    {
        unsigned seen = 0, woken = 0;
        for (;;) {
            bool called;
            {
                std::unique_lock<std::mutex> l(m_);
                asleep_.fetch_add(1);
                cv_.wait(l, [&] { return stop_ || wakes_ != woken || turn_.load() != seen; });
                asleep_.fetch_sub(1);
                if (stop_) return;
                called = wakes_ != woken;  // by wake(), not by a loop
                woken = wakes_;
            }
            // rest() comes after each() has returned: no turn is left undone
            auto last = std::chrono::steady_clock::now();
            if (called) last += CALL - SPIN;
            while (awake_.load(std::memory_order_acquire)) {
                const unsigned t = turn_.load(std::memory_order_acquire);
                if (t == seen) {
                    if (std::chrono::steady_clock::now() - last > SPIN) break;
                    std::this_thread::yield();
                    continue;
                }
                seen = t;
                (*f_)(part, size());
                done_.fetch_add(1, std::memory_order_release);
                last = std::max(last, std::chrono::steady_clock::now());
            }
        }
    }
    std::vector<std::thread> threads_;
    std::mutex m_;
    std::condition_variable cv_;
    bool stop_ = false;
    unsigned wakes_ = 0;
    std::atomic<bool> awake_{false};
    std::atomic<unsigned> turn_{0};
    std::atomic<int> asleep_{0};
    std::atomic<int> done_{0};
    const std::function<void(int, int)>* f_ = nullptr;
};

// frames [f0, f1) of packed decisions ((n + 7) / 8 bytes each, bit 0 first) to 0/1 bytes
inline void expand_bits(const uint8_t* in, uint8_t* out, int n, size_t f0, size_t f1)
{
    struct Table {
        uint64_t v[256];
        Table()
        {
            for (int b = 0; b < 256; b++) {
                uint8_t x[8];
                for (int i = 0; i < 8; i++) x[i] = (b >> i) & 1;
                memcpy(&v[b], x, 8);
            }
        }
    };
    static const Table table;
    const size_t nb = (size_t)(n + 7) / 8, whole = (size_t)n / 8;
    for (size_t f = f0; f < f1; f++) {
        const uint8_t* s = in + f * nb;
        uint8_t* o = out + f * (size_t)n;
        for (size_t b = 0; b < whole; b++) memcpy(o + 8 * b, &table.v[s[b]], 8);
        for (size_t i = 8 * whole; i < (size_t)n; i++) o[i] = (s[i / 8] >> (i & 7)) & 1;
    }
}

struct HostPipe {
    static constexpr size_t IN_BYTES = 512 << 10, OUT_BYTES = 128 << 10;  // of a piece
    static constexpr int IN = 4, OUT = 8;                               // pieces of a ring
    uint8_t* pinned = nullptr;
    cudaEvent_t in_ev[IN] = {}, out_ev[OUT] = {};
    cudaStream_t comp[2] = {};  // decode streams beside the decoder's own, so that chunks overlap
    cudaEvent_t chunk_ev = nullptr, dec_ev = nullptr;
    HostTeam team;
    int device;
    HostPipe(int helpers, int dev) : team(helpers), device(dev) {}
    ~HostPipe()
    {
        for (auto e : in_ev)
            if (e) cudaEventDestroy(e);
        for (auto e : out_ev)
            if (e) cudaEventDestroy(e);
        for (auto s : comp)
            if (s) cudaStreamDestroy(s);
        if (chunk_ev) cudaEventDestroy(chunk_ev);
        if (dec_ev) cudaEventDestroy(dec_ev);
        cudaFreeHost(pinned);
    }
    cudaError_t init()
    {
        cudaError_t e = cudaMallocHost((void**)&pinned, IN * IN_BYTES + OUT * OUT_BYTES);
        for (auto& x : in_ev)
            if (e == cudaSuccess) e = cudaEventCreateWithFlags(&x, cudaEventDisableTiming);
        for (auto& x : out_ev)
            if (e == cudaSuccess) e = cudaEventCreateWithFlags(&x, cudaEventDisableTiming);
        for (auto& x : comp)
            if (e == cudaSuccess) e = cudaStreamCreateWithFlags(&x, cudaStreamNonBlocking);
        if (e == cudaSuccess) e = cudaEventCreateWithFlags(&chunk_ev, cudaEventDisableTiming);
        if (e == cudaSuccess) e = cudaEventCreateWithFlags(&dec_ev, cudaEventDisableTiming);
        return e;
    }
    static HostPipe* make(int dev)  // null: no memory for it
    {
        const unsigned cores = std::thread::hardware_concurrency();
        HostPipe* p = new (std::nothrow) HostPipe(cores > 3 ? (int)(cores / 2 - 1 < 5 ? cores / 2 - 1 : 5) : 0, dev);
        if (p && p->init() == cudaSuccess) return p;
        cudaGetLastError();
        delete p;
        return nullptr;
    }
    uint8_t* in(int i) { return pinned + i * IN_BYTES; }
    uint8_t* out(int i) { return pinned + IN * IN_BYTES + i * OUT_BYTES; }
};

// The idle pipes of the process.  Safe from any thread; a pipe serves one call at a time.
class HostPipes {
public:
    static HostPipe* take(int device)
    {
        {
            std::lock_guard<std::mutex> l(lock());
            auto& v = idle();
            for (size_t i = 0; i < v.size(); i++)
                if (v[i]->device == device) {
                    HostPipe* p = v[i];
                    v.erase(v.begin() + i);
                    return p;
                }
        }
        return HostPipe::make(device);
    }
    static void give(HostPipe* p)
    {
        {
            std::lock_guard<std::mutex> l(lock());
            if (idle().size() < 2 && users() > 0) {
                idle().push_back(p);
                return;
            }
        }
        delete p;
    }
    // a decoder came (+1) or went (-1); the idle pipes go with the last one.  A forked child has
    // copies of the pipes without their threads: a decoder that it frees leaves them alone, as
    // joining those threads would wait for good.
    static void user(int change)
    {
        static const pid_t owner = getpid();
        if (getpid() != owner) return;
        std::vector<HostPipe*> gone;
        {
            std::lock_guard<std::mutex> l(lock());
            users() += change;
            if (users() <= 0) gone.swap(idle());
        }
        for (auto* p : gone) delete p;
    }

private:
    // never destroyed: a decoder may be freed after the process's static objects
    static std::mutex& lock() { static std::mutex* m = new std::mutex; return *m; }
    static std::vector<HostPipe*>& idle() { static auto* v = new std::vector<HostPipe*>; return *v; }
    static long& users() { static long n = 0; return n; }
};

}  // namespace ldpc
