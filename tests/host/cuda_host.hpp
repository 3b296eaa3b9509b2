// Compiles the library's device headers as host C++ (g++ with the CUDA toolkit's include path): the device
// functions that they use, and a warp of 32 host threads for code that votes or shuffles. The threads run
// one at a time, in lane order or from the last lane to the first, each until its next warp operation:
// whatever a lane does before an operation is done before the next lane begins, which is as far apart as the
// execution model lets lanes drift.
#pragma once

#include <cuda_runtime.h>

#include <algorithm>
#include <cfloat>
#include <cmath>
#include <condition_variable>
#include <cstdint>
#include <cstdio>
#include <cstring>
#include <mutex>
#include <thread>
#include <vector>

using std::max;
using std::min;

template <class T>
T __ldg(const T* p) { return *p; }
inline uint32_t __float_as_uint(float f)
{
    uint32_t u;
    memcpy(&u, &f, 4);
    return u;
}
inline float __uint_as_float(uint32_t u)
{
    float f;
    memcpy(&f, &u, 4);
    return f;
}
inline int __float_as_int(float f) { return (int) __float_as_uint(f); }
inline float __int_as_float(int i) { return __uint_as_float((uint32_t) i); }
inline int __clz(int v) { return v ? __builtin_clz((unsigned) v) : 32; }
inline int __ffs(int v) { return __builtin_ffs(v); }
inline int __popc(unsigned v) { return __builtin_popcount(v); }

// One thread runs at a time, so the atomics are plain.
template <class T, class F>
T host_atomic(T* p, F f)
{
    const T old = *p;
    *p = f(old);
    return old;
}
template <class T, class U>
T atomicAdd(T* p, U v) { return host_atomic(p, [v](T o) { return (T) (o + v); }); }
template <class T, class U>
T atomicOr(T* p, U v) { return host_atomic(p, [v](T o) { return (T) (o | v); }); }
template <class T, class U>
T atomicMin(T* p, U v) { return host_atomic(p, [v](T o) { return min(o, (T) v); }); }
template <class T, class U>
T atomicMax(T* p, U v) { return host_atomic(p, [v](T o) { return max(o, (T) v); }); }
template <class T, class U>
T atomicExch(T* p, U v) { return host_atomic(p, [v](T) { return (T) v; }); }
template <class T, class U, class V>
T atomicCAS(T* p, U c, V v) { return host_atomic(p, [c, v](T o) { return o == (T) c ? (T) v : o; }); }

class HostWarp {
public:
    // f(lane) on 32 lanes.
    template <class F>
    static void run(bool from_last, F f)
    {
        HostWarp w;
        w.step_ = from_last ? 31 : 1;
        w.turn_ = from_last ? 31 : 0;
        std::vector<std::thread> lanes;
        for (int i = 0; i < 32; ++i)
            lanes.emplace_back([&w, &f, i] {
                warp = &w;
                lane = i;
                w.take_turn();
                f(i);
                w.pass_turn();
            });
        for (auto& t : lanes)
            t.join();
    }

    // Every lane's word, once every lane has given one.
    static const uint32_t* exchange(uint32_t v)
    {
        HostWarp& w = *warp;
        uint32_t* words = w.words_[w.ops_[lane]++ & 1];
        words[lane] = v;
        w.pass_turn();
        w.take_turn();
        return words;
    }

    static thread_local int lane;

private:
    void take_turn()
    {
        std::unique_lock<std::mutex> l(mutex_);
        cv_[lane].wait(l, [this] { return turn_ == lane; });
    }
    void pass_turn()
    {
        std::lock_guard<std::mutex> l(mutex_);
        turn_ = (turn_ + step_) & 31;
        cv_[turn_].notify_one();
    }

    static thread_local HostWarp* warp;
    std::mutex mutex_;
    std::condition_variable cv_[32];
    int turn_ = 0, step_ = 1;
    unsigned ops_[32] = {};
    uint32_t words_[2][32];
};
inline thread_local int HostWarp::lane;
inline thread_local HostWarp* HostWarp::warp;

inline void __syncwarp() { HostWarp::exchange(0); }
inline unsigned __ballot_sync(unsigned, int p)
{
    const uint32_t* w = HostWarp::exchange(p != 0);
    unsigned b = 0;
    for (int i = 0; i < 32; ++i)
        b |= w[i] << i;
    return b;
}
inline int __any_sync(unsigned m, int p) { return __ballot_sync(m, p) != 0; }
template <class T>
T host_shuffle(T v, int src)
{
    static_assert(sizeof(T) == 4, "");
    uint32_t u;
    memcpy(&u, &v, 4);
    u = HostWarp::exchange(u)[src];
    memcpy(&v, &u, 4);
    return v;
}
template <class T>
T __shfl_sync(unsigned, T v, int src, int width = 32)
{
    return host_shuffle(v, (HostWarp::lane & ~(width - 1)) | (src & (width - 1)));
}
template <class T>
T __shfl_xor_sync(unsigned, T v, int mask) { return host_shuffle(v, HostWarp::lane ^ mask); }
