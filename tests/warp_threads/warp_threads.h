// warp_threads.h -- a block on the CPU: one thread per lane, for compiling the device
// code of csrc/*.cuh with the host compiler and running it under ThreadSanitizer.
//
// What orders memory here is what orders it on the device: __syncwarp and __syncthreads
// (barriers that the sanitizer sees) order the lanes' accesses before them against those
// after them; shuffles and votes exchange values but order nothing (the sanitizer is told
// to ignore their synchronisation).  So two lanes' accesses to one word of shared memory,
// one of them a write, with no barrier between them, are a reported race whatever order
// the threads happened to run in.
//
// Warp-collective calls take any lane mask (groups of a warp diverge in the advance's
// queue loop).
#pragma once

#include <algorithm>
#include <atomic>
#include <cfloat>
#include <climits>
#include <cmath>
#include <cstddef>
#include <cstdint>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <functional>
#include <thread>
#include <type_traits>
#include <utility>
#include <vector>

#if defined(__SANITIZE_THREAD__)
extern "C" void AnnotateIgnoreSyncBegin(const char*, int);
extern "C" void AnnotateIgnoreSyncEnd(const char*, int);
#else
inline void AnnotateIgnoreSyncBegin(const char*, int) {}
inline void AnnotateIgnoreSyncEnd(const char*, int) {}
#endif

#define __host__
#define __device__
#define __global__
#define __shared__
#define __constant__
#define __forceinline__ inline
#define __launch_bounds__(...)
#define __noinline__ __attribute__((noinline))

struct ulonglong2 {
    unsigned long long x, y;
};
struct Dim {
    unsigned x = 0, y = 0, z = 0;
};
inline thread_local Dim threadIdx, blockIdx;
inline Dim blockDim{32, 1, 1}, gridDim{1, 1, 1};

namespace warp {

constexpr int kLanes = 32;

// A barrier with an exchange of one word per lane, for the lanes of one mask.  Two sets
// of words: a lane may be at the next exchange while another still reads this one's.
struct Meeting {
    std::atomic<unsigned> arrived{0}, turn{0};
    std::atomic<uint64_t> word[2][kLanes];
    uint64_t meet(uint64_t mine, int lane, int lanes, const std::function<uint64_t(const std::atomic<uint64_t>*)>& get) {
        const unsigned t = turn.load(std::memory_order_acquire);
        word[t & 1][lane].store(mine, std::memory_order_relaxed);
        if (arrived.fetch_add(1, std::memory_order_acq_rel) + 1 == static_cast<unsigned>(lanes)) {
            arrived.store(0, std::memory_order_relaxed);
            turn.store(t + 1, std::memory_order_release);
            turn.notify_all();
        } else {
            turn.wait(t, std::memory_order_acquire);
        }
        return get(word[t & 1]);
    }
};
// one per warp and group of lanes (a mask is a run of lanes whose first and size identify it)
constexpr int kWarps = 16;
inline Meeting meetings[kWarps][6][kLanes];
inline Meeting& meeting(unsigned mask) {
    return meetings[threadIdx.x / kLanes][__builtin_ctz(static_cast<unsigned>(__builtin_popcount(mask)))]
                   [__builtin_ctz(mask)];
}
inline Meeting block;  // of all threads: word[.][0] is unused
inline int lane() { return static_cast<int>(threadIdx.x % kLanes); }

struct IgnoreSync {
    IgnoreSync() { AnnotateIgnoreSyncBegin(__FILE__, __LINE__); }
    ~IgnoreSync() { AnnotateIgnoreSyncEnd(__FILE__, __LINE__); }
};

template <class T>
uint64_t to_word(T v) {
    static_assert(sizeof(T) <= 8, "one word");
    uint64_t w = 0;
    std::memcpy(&w, &v, sizeof v);
    return w;
}
template <class T>
T from_word(uint64_t w) {
    T v;
    std::memcpy(&v, &w, sizeof v);
    return v;
}
template <class T>
T exchange(unsigned mask, T v, int from) {  // the value of lane `from`
    IgnoreSync s;
    return from_word<T>(meeting(mask).meet(to_word(v), lane(), __builtin_popcount(mask), [&](const auto* w) {
        return w[from].load(std::memory_order_relaxed);
    }));
}

// a kernel's body on one block of `warps` warps
inline void launch(const std::function<void()>& body, int warps = 1) {
    blockDim.x = static_cast<unsigned>(warps * kLanes);
    std::vector<std::thread> lanes;
    for (int l = 0; l < warps * kLanes; ++l)
        lanes.emplace_back([l, &body] {
            threadIdx.x = static_cast<unsigned>(l);
            body();
        });
    for (auto& t : lanes) t.join();
}

// The interpreter's shared-memory stores (coop::sts64).  Idle lanes all store into the
// write sink, which nothing reads; and a lane that stored a result in its own step
// (CTL_FLUSH) stores the same value to the same slot once more with the next step's.
// Neither is a conflict, so neither reaches the sanitizer.
inline std::function<bool(uint32_t)> is_sink = [](uint32_t) { return false; };
struct Stored {
    uint32_t at = 0;
    unsigned step = 0;
    uint64_t value = 0;
};
inline thread_local unsigned step = 0;  // barriers so far
inline thread_local Stored last[4];     // the lane's last stores: no step has more
inline thread_local unsigned last_n = 0;
inline void store(uint64_t* base, uint32_t addr, uint64_t v) {
    if (is_sink(addr)) return;
    for (const Stored& s : last)
        if (s.at == addr && s.value == v && s.step + 1 == step) return;
    last[last_n++ % 4] = {addr, step, v};
    base[addr / 8] = v;
}

}  // namespace warp

inline void __syncwarp(unsigned mask = 0xffffffffu) {
    warp::meeting(mask).meet(0, warp::lane(), __builtin_popcount(mask), [](const auto*) { return uint64_t{0}; });
    ++warp::step;
}
template <class T>
T __shfl_sync(unsigned mask, T v, int src, int width = 32) {
    return warp::exchange(mask, v, warp::lane() / width * width + src % width);
}
template <class T>
T __shfl_xor_sync(unsigned mask, T v, int off, int = 32) {
    return warp::exchange(mask, v, warp::lane() ^ off);
}
inline unsigned __ballot_sync(unsigned mask, int p) {
    warp::IgnoreSync s;
    return static_cast<unsigned>(
        warp::meeting(mask).meet(p != 0, warp::lane(), __builtin_popcount(mask), [&](const auto* w) {
            uint64_t m = 0;
            for (int l = 0; l < warp::kLanes; ++l)
                if ((mask >> l) & 1u) m |= w[l].load(std::memory_order_relaxed) << l;
            return m;
        }));
}
inline int __any_sync(unsigned mask, int p) { return __ballot_sync(mask, p) != 0; }
inline int __all_sync(unsigned mask, int p) { return __ballot_sync(mask, p) == mask; }
inline int __reduce_add_sync(unsigned mask, int v) {
    int sum = 0;
    for (int l = 0; l < warp::kLanes; ++l) sum += warp::exchange(mask, v, l);
    return sum;
}
using std::isfinite;
inline unsigned min(unsigned a, int b) { return std::min(a, static_cast<unsigned>(b)); }
inline int __popc(unsigned v) { return __builtin_popcount(v); }
inline int __ffs(unsigned v) { return v ? __builtin_ctz(v) + 1 : 0; }
inline void __syncthreads() {
    warp::block.meet(0, warp::lane(), static_cast<int>(blockDim.x), [](const auto*) { return uint64_t{0}; });
    ++warp::step;
}

inline double __longlong_as_double(long long v) { return warp::from_word<double>(static_cast<uint64_t>(v)); }
inline long long __double_as_longlong(double v) { return static_cast<long long>(warp::to_word(v)); }
inline double __fma_rn(double a, double b, double c) { return std::fma(a, b, c); }
inline float __double2float_rn(double v) { return static_cast<float>(v); }
inline unsigned __dp2a_lo(unsigned a, unsigned b, unsigned c) {
    return c + (a & 0xffffu) * (b & 0xffu) + (a >> 16) * ((b >> 8) & 0xffu);
}
template <class T, class U>
T atomicAdd(T* p, U v) {
    warp::IgnoreSync s;
    return __atomic_fetch_add(p, static_cast<T>(v), __ATOMIC_RELAXED);
}
inline int atomicCAS(int* p, int cmp, int v) {
    warp::IgnoreSync s;
    __atomic_compare_exchange_n(p, &cmp, v, false, __ATOMIC_RELAXED, __ATOMIC_RELAXED);
    return cmp;
}
inline unsigned long long atomicMin(unsigned long long* p, unsigned long long v) {
    unsigned long long old = *p;
    if (v < old) *p = v;
    return old;
}
// the fallback of wr_div_finish, counted
inline thread_local int native_divisions = 0;
inline double native_division(double a, double b) {
    ++native_divisions;
    return a / b;
}

// shared-window addresses: byte offsets from the program's slot array
inline uint64_t* slots = nullptr;
inline size_t __cvta_generic_to_shared(const uint64_t* p) { return static_cast<size_t>(p - slots) * 8; }
