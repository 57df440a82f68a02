// device_util.h -- device buffers with an HBM budget, error checks.
#pragma once
#include <cuda_runtime.h>

#include <algorithm>
#include <atomic>
#include <iterator>
#include <map>
#include <mutex>
#include <new>
#include <string>
#include <thread>
#include <vector>

#include "../../include/sgdg.h"
#include "sgdg_core.h"

namespace sgdg {

#define CK(call)                                                                                        \
    do {                                                                                                \
        cudaError_t e_ = (call);                                                                        \
        if (e_ != cudaSuccess)                                                                          \
            throw ::sgdg::Error(e_ == cudaErrorMemoryAllocation ? SGDG_ENOMEM_BUDGET : SGDG_ECUDA,     \
                                std::string(#call) + ": " + cudaGetErrorString(e_));                    \
    } while (0)

inline std::atomic<int64_t> g_budget{0};
inline std::atomic<int> g_budget_set{0};  // counts the calls that set it
inline std::atomic<int64_t> g_in_use{0};

inline void require_gpu() {
    static int state = -1;  // -1 unknown, 0 none, 1 ok
    if (state == 1) return;
    int n = 0;
    cudaError_t e = cudaGetDeviceCount(&n);
    if (e != cudaSuccess || n == 0) {
        cudaGetLastError();
        state = 0;
        throw Error(SGDG_ENOGPU,
                    std::string("no CUDA device: ") + (e != cudaSuccess ? cudaGetErrorString(e) : "0 devices"));
    }
    state = 1;
}

// Blocks handed back with DevBuf::recycle, kept for the next allocation of their
// size: a call that allocates its vectors, arenas or work list pays 10 to 100 us
// per block for cudaMalloc and cudaFree otherwise (an evolver's call 0.1 to 0.4
// ms).  Only a block whose work has finished is recycled (its owner has waited
// for every stream that used it), so any stream or thread may take it; the others
// are freed, and cudaFree waits.  At most kPoolBytes are kept; they count against
// the HBM budget, and are given back where an allocation or the budget needs them,
// when the last handle is destroyed (LiveHandle) or nothing else is held, and with
// every call of sgdg_set_hbm_budget.
class DevPool {
   public:
    static constexpr size_t kPoolBytes = size_t(1) << 30;
    static size_t rounded(size_t n) { return (n + 511) & ~size_t(511); }
    // a kept block of at least n bytes (at most an eighth more, or exactly n
    // rounded where a budget is set): its size in got, or null
    void* take(size_t n, bool exact, size_t& got) {
        const size_t want = rounded(n);
        std::lock_guard<std::mutex> g(mu_);
        auto& m = kept_[device()];
        const auto it = m.lower_bound(want);
        if (it == m.end() || it->first > (exact ? want : want + want / 8)) return nullptr;
        void* p = it->second;
        got = it->first;
        m.erase(it);
        held_ -= got;
        return p;
    }
    // keeps p (size bytes on device dev) or frees it
    void give(void* p, size_t size, int dev) {
        if (size <= kPoolBytes / 2 && dev == device()) {
            std::lock_guard<std::mutex> g(mu_);
            if (held_ + size <= kPoolBytes) {
                try {
                    kept_[dev].emplace(size, p);
                    held_ += size;
                    return;
                } catch (const std::bad_alloc&) {
                }
            }
        }
        cudaFree(p);
    }
    // frees kept blocks, the largest first, until at most `most` bytes are kept
    void trim(size_t most) {
        std::lock_guard<std::mutex> g(mu_);
        for (auto& d : kept_)
            while (held_ > most && !d.second.empty()) {
                const auto it = std::prev(d.second.end());
                cudaFree(it->second);
                held_ -= it->first;
                d.second.erase(it);
            }
    }
    size_t held() const { return held_.load(); }
    static int device() {
        int d = 0;
        cudaGetDevice(&d);
        return d;
    }

   private:
    std::mutex mu_;
    std::map<int, std::multimap<size_t, void*>> kept_;  // per device, by size
    std::atomic<size_t> held_{0};
};
inline DevPool& device_pool() {
    static DevPool* p = new DevPool;  // outlives the buffers of static objects
    return *p;
}

// Base of the handles: the blocks kept for reuse go with the last of them (tables
// kept for the process, of the point evaluation, may still be held then).
class LiveHandle {
   protected:
    LiveHandle() { count()++; }
    LiveHandle(const LiveHandle&) = delete;
    LiveHandle& operator=(const LiveHandle&) = delete;
    ~LiveHandle() {  // the last part of a handle to go: its own blocks are freed
        if (--count() == 0) device_pool().trim(0);
    }

   private:
    static std::atomic<int64_t>& count() {
        static std::atomic<int64_t> n{0};
        return n;
    }
};

// Device memory that its owner, a handle, can do without (an operator's second,
// faster form): given back where an allocation or the budget needs the room, so
// that holding it never refuses a call.  The owner holds a Use while it looks at
// that memory, changes it or launches with it; between its calls any thread may
// take it (its destructor calls retire() before anything else).
class Spare {
   public:
    // frees what idle handles can do without; false: there was nothing
    static bool give_back() {
        std::lock_guard<std::mutex> g(mutex());
        bool any = false;
        for (Spare* s : all()) {
            int idle = 0;
            if (!s->users_.compare_exchange_strong(idle, -1)) continue;
            any = s->drop_spare() || any;
            s->users_ = 0;
        }
        return any;
    }
    struct Use {
        explicit Use(Spare& s) : s_(s) {
            for (int u = s_.users_.load();;) {  // -1: being freed
                if (u < 0) {
                    std::this_thread::yield();
                    u = s_.users_.load();
                } else if (s_.users_.compare_exchange_weak(u, u + 1)) {
                    break;
                }
            }
        }
        ~Use() { s_.users_--; }
        Use(const Use&) = delete;
        Use& operator=(const Use&) = delete;

       private:
        Spare& s_;
    };

   protected:
    Spare() {
        std::lock_guard<std::mutex> g(mutex());
        all().push_back(this);
    }
    Spare(const Spare&) = delete;
    Spare& operator=(const Spare&) = delete;
    virtual ~Spare() { retire(); }
    void retire() {
        std::lock_guard<std::mutex> g(mutex());
        auto& a = all();
        a.erase(std::remove(a.begin(), a.end(), this), a.end());
    }
    // frees it (cudaFree waits for the launches that use it); whether there was any
    virtual bool drop_spare() = 0;

   private:
    static std::mutex& mutex() {
        static std::mutex* m = new std::mutex;
        return *m;
    }
    static std::vector<Spare*>& all() {
        static std::vector<Spare*>* a = new std::vector<Spare*>;
        return *a;
    }
    std::atomic<int> users_{0};  // -1 while give_back frees it
};

// Device allocation counted against the HBM budget (sgdg_set_hbm_budget).
struct DevBuf {
    void* p = nullptr;
    size_t bytes = 0;  // asked for
    size_t size = 0;   // of the block
    int dev = 0;       // it is on
    DevBuf() = default;
    explicit DevBuf(size_t n) { alloc(n); }
    DevBuf(const DevBuf&) = delete;
    DevBuf& operator=(const DevBuf&) = delete;
    DevBuf(DevBuf&& o) noexcept : p(o.p), bytes(o.bytes), size(o.size), dev(o.dev) {
        o.p = nullptr;
        o.bytes = o.size = 0;
    }
    DevBuf& operator=(DevBuf&& o) noexcept {
        if (this == &o) return *this;
        release();
        p = o.p;
        bytes = o.bytes;
        size = o.size;
        dev = o.dev;
        o.p = nullptr;
        o.bytes = o.size = 0;
        return *this;
    }
    void alloc(size_t n) {
        release();
        if (n == 0) n = 16;
        const int64_t b = g_budget.load();
        auto over = [&] { return b > 0 && g_in_use.load() + (int64_t)n > b; };
        if (over() && !(Spare::give_back() && !over()))
            throw Error(SGDG_ENOMEM_BUDGET, "HBM budget exceeded: requested " + std::to_string(n) + " bytes, " +
                                                std::to_string(g_in_use.load()) + " of " + std::to_string(b) +
                                                " in use");
        p = device_pool().take(n, b > 0, size);
        if (!p) {
            size = DevPool::rounded(n);
            if (b > 0) device_pool().trim((size_t)std::max<int64_t>(0, b - g_in_use.load() - (int64_t)n));
            cudaError_t e = cudaMalloc(&p, size);
            for (int more = 0; e == cudaErrorMemoryAllocation && more < 2; more++) {
                cudaGetLastError();
                if (more == 0 ? device_pool().held() == 0 : !Spare::give_back()) continue;
                device_pool().trim(0);
                e = cudaMalloc(&p, size);
            }
            if (e != cudaSuccess) {
                cudaGetLastError();
                p = nullptr;
                throw Error(SGDG_ENOMEM_BUDGET, std::string("cudaMalloc: ") + cudaGetErrorString(e));
            }
        }
        bytes = n;
        dev = DevPool::device();
        g_in_use += (int64_t)n;
    }
    void release() { drop(false); }
    // as release, where everything that used the buffer has finished
    void recycle() { drop(true); }
    ~DevBuf() { release(); }
    void drop(bool keep) {
        if (p) {
            if (keep)
                device_pool().give(p, size, dev);
            else
                cudaFree(p);
            if ((g_in_use -= (int64_t)bytes) == 0) device_pool().trim(0);
        }
        p = nullptr;
        bytes = size = 0;
    }
    template <class T>
    T* as() const {
        return static_cast<T*>(p);
    }
};

template <class T>
DevBuf upload(const std::vector<T>& v, cudaStream_t st) {
    DevBuf b(v.size() * sizeof(T));
    if (!v.empty()) CK(cudaMemcpyAsync(b.p, v.data(), v.size() * sizeof(T), cudaMemcpyHostToDevice, st));
    return b;
}

}  // namespace sgdg
