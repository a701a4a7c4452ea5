// One warp of device code on the CPU: its 32 lanes are coroutines that run in turn between shuffles, so
// that a device function that only uses the intrinsics below can be compiled with g++ and checked
// without a GPU.  Every lane must meet the same shuffles in the same order, as on the device.
#pragma once
#include <ucontext.h>

#include <cmath>
#include <cstdint>
#include <cstring>
#include <functional>
#include <vector>

#include <cuda_runtime.h>

#include <algorithm>

namespace host_warp {
constexpr int kLanes = 32;
struct Warp {
    ucontext_t main, lane[kLanes];
    std::vector<char> stack[kLanes];
    uint32_t slot[2][kLanes];  // values of the current shuffle and of the one before
    int phase[kLanes], cur;
    bool ended[kLanes];
    std::function<void(unsigned)> body;
};
inline Warp* warp = nullptr;
inline void enter()
{
    Warp* w = warp;
    w->body((unsigned)w->cur);
    w->ended[w->cur] = true;
    swapcontext(&w->lane[w->cur], &w->main);
}
// body(lane) on all lanes; false where the lanes did not meet the same number of shuffles.
inline bool run(std::function<void(unsigned)> body)
{
    Warp w;
    w.body = std::move(body);
    warp = &w;
    for (int l = 0; l < kLanes; ++l) {
        w.stack[l].resize(64 * 1024);
        w.phase[l] = 0;
        w.ended[l] = false;
        getcontext(&w.lane[l]);
        w.lane[l].uc_stack.ss_sp = w.stack[l].data();
        w.lane[l].uc_stack.ss_size = w.stack[l].size();
        w.lane[l].uc_link = nullptr;
        makecontext(&w.lane[l], enter, 0);
    }
    for (;;) {
        int done = 0;
        for (int l = 0; l < kLanes; ++l) {
            w.cur = l;
            swapcontext(&w.main, &w.lane[l]);
            done += w.ended[l];
        }
        if (done == kLanes) return true;
        if (done) return false;
    }
}
inline uint32_t shuffle(uint32_t v, int d)
{
    Warp* w = warp;
    const int l = w->cur, ph = w->phase[l]++ & 1, from = l + d;
    w->slot[ph][l] = v;
    swapcontext(&w->lane[l], &w->main);
    return w->slot[ph][from >= 0 && from < kLanes ? from : l];  // off the warp: the lane's own value
}
struct ThreadIdx {
    struct X {
        operator unsigned() const { return (unsigned)warp->cur; }
    } x;
};
}  // namespace host_warp

static const host_warp::ThreadIdx threadIdx{};
inline uint32_t __shfl_up_sync(unsigned, uint32_t v, int d) { return host_warp::shuffle(v, -d); }
inline uint32_t __shfl_down_sync(unsigned, uint32_t v, int d) { return host_warp::shuffle(v, d); }
double __shfl_xor_sync(unsigned, double, int);  // declared only: not used by what runs here
inline uint32_t __funnelshift_l(uint32_t lo, uint32_t hi, int s)
{
    return (uint32_t)((((uint64_t)hi << 32 | lo) << (s & 31)) >> 32);
}
inline uint32_t __funnelshift_r(uint32_t lo, uint32_t hi, int s)
{
    return (uint32_t)(((uint64_t)hi << 32 | lo) >> (s & 31));
}
inline unsigned __umulhi(unsigned a, unsigned b) { return (unsigned)((uint64_t)a * b >> 32); }
inline int __ffs(int v) { return __builtin_ffs(v); }
inline uint32_t atomicOr(uint32_t* p, uint32_t v)
{
    const uint32_t was = *p;
    *p |= v;
    return was;
}
unsigned long long atomicMax(unsigned long long*, unsigned long long);  // declared only
inline long long __double_as_longlong(double v)
{
    long long r;
    std::memcpy(&r, &v, 8);
    return r;
}
inline int __double2hiint(double v) { return (int)(__double_as_longlong(v) >> 32); }
inline int __double2loint(double v) { return (int)__double_as_longlong(v); }
inline double __hiloint2double(int hi, int lo)
{
    const uint64_t b = (uint64_t)(uint32_t)hi << 32 | (uint32_t)lo;
    double r;
    std::memcpy(&r, &b, 8);
    return r;
}
using std::abs;
using std::fma;
using std::sqrt;
