// 1D AWCM compressible-Euler path on one B200 (sm_100a), FP64: single instances and batches.
//
// A 1D instance is small (Nx = (nx_coarse-1) 2^(L-1) + 1 points, 1025 for the Sod case, up to
// 8193 in the uneven batch), so one CTA advances one instance through a whole RK3 step --
// PrepareEuler, CFL, three stages, residue removal -- separating the level-sequential phases with
// block barriers instead of kernel launches.  A batch is one persistent launch: CTAs pull instance
// ids from a queue (largest first), so hundreds of uneven instances share the GPU in one kernel;
// a single instance is the same launch with one queue entry.  Each step is captured once into a
// CUDA graph (queue reset + step kernel) and replayed.
//
// A step is a serial chain of short phases on one SM, so what it costs is the number of its
// phases and the latency of each.  Two representations keep both small:
//   - Masks and levels are bit planes while a step runs (one bit per point, the point i at bit
//     i & 31 of word (i >> 5) + 1).  A pass over a mask is a handful of shifts per 32-bit word in
//     one phase, where a point-per-thread pass walks every point of the line.  Levels are
//     bit-sliced (`nb` planes per level set) next to a plane of the finest-level points.
//   - The transforms and the stages run over compact lists of active points (16-bit entries where
//     the line allows it); the transform list is ordered by level, so that the points a level
//     predicts and the coarser points it updates are each one contiguous range.
//
// Per-instance layout in the pool (w = Nx + 6, ghost ring 3): doubles q[3][w] (conserved),
// qc[3][w] (stage-start copy), qt[3][w] (coarse-point flux derivatives of a stage), fl[3][w] (face
// fluxes, face i+1/2 at point i), then 2 (w + 32) doubles of list space; then the bit planes.
// Bytes mask[w] (bits 0..3 mask0..3, 4 previous mask0; 5..7 set on the ghost ring), then 16-byte
// aligned level[4][w]: the form in which masks and levels rest between launches.
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstring>
#include <mutex>
#include <numeric>
#include <vector>

#include "awcm1d_layout.cuh"
#include "awcm_b200.h"
#include "awcm_common.cuh"

namespace awcm {
namespace {

struct Inst1 {
    int nx, maxl, scheme, pad0;
    double x_min, dx, gamma, tol, cfl, t, t_end, dt_fixed;
    long long q_off;  // in doubles
    long long m_off;  // in bytes
    // results of the last step
    double dt, mv, alpha[3];
    int do_print, done, steps, err;
    unsigned mask_cnt[4];
    unsigned long long upd;
    // the enum-driven BOUNDARY_MANAGER_1D<T> when bc_generic: BOUNDARY_CONDITION of the ghost cells
    // -1, -2, -3 (bcg[0..2]) and N1+1, N1+2, N1+3 (bcg[3..5])
    int8_t bcg[6];
    int8_t bc_generic, pad1;
};

// BOUNDARY_CONDITION values of the generic manager (BOUNDARY_MANAGER_1D.h:4-13).
constexpr int kBcPeriodic1 = -3, kBcExtrapolation1 = -2;

// Threads per CTA: a caller may ask for up to 768, the step kernel runs at most 512, with 128 registers
// each.  At 768 threads and 80 registers it spills about 1.2 KB a thread in and around the faces, and
// every phase pays: a 1025-point step took 92 us against 75 us.
constexpr int kMaxLaunch1 = 768;
#ifndef AWCM_MAX_THREADS_1D
#define AWCM_MAX_THREADS_1D 512
#endif
constexpr int kMaxThreads1 = AWCM_MAX_THREADS_1D;

struct Pool {
    double* q;
    uint8_t* m;
    Weights W;
};

// The per-CTA workspace: class counters of the ordered list, list counters, reductions.
struct Work1 {
    Inst1 inst;                          // the instance's descriptor while its steps run
    unsigned cls[32], run[32], off[33];  // counts, write positions, starts of the level classes
    unsigned mask_cnt[4];                // |mask0..mask3|
    unsigned n_face[4], n_fin[4];        // of mask0..mask2: needed faces, finest-level points
    unsigned n_list[4][4];               // per mask: entries written so far (faces, finest, coarse points)
    unsigned long long red[3][2][32];    // per reduction of the step: two maxima, one value per warp
};

// A list of points (stored as i + kGhost) with 16- or 32-bit entries.
struct List {
    static constexpr bool kSome = false;
    void* p;
    bool half;
    __device__ __forceinline__ int get(unsigned e) const
    {
        return (half ? (int)static_cast<const uint16_t*>(p)[e] : (int)static_cast<const uint32_t*>(p)[e]) - kGhost;
    }
    __device__ __forceinline__ void put(unsigned e, int i) const
    {
        if (half) static_cast<uint16_t*>(p)[e] = (uint16_t)(i + kGhost);
        else static_cast<uint32_t*>(p)[e] = (uint32_t)(i + kGhost);
    }
    __device__ __forceinline__ List at(size_t e) const
    {
        return List{half ? (void*)(static_cast<uint16_t*>(p) + e) : (void*)(static_cast<uint32_t*>(p) + e), half};
    }
};

// Place of ghosted point x of a conserved plane in shared memory (mask m = 15; 0 in global memory: x
// itself).  The points of a level are a power of two apart, so in a linear plane the 32 lanes of a
// warp meet in one or a few of the 16 double-wide banks: every access of a level of spacing 16 or
// more took 32 turns.  Exchanging the 16 places of a bank row by the higher bits of x spreads any
// power-of-two stride over all banks.
__device__ __forceinline__ int place(int x, int m) { return x ^ (((x >> 4) ^ (x >> 8) ^ (x >> 12)) & m); }
struct Field1 {
    double *q0, *q1, *q2;  // conserved planes
    int m0, m12;           // place() masks of q0 and of q1, q2
    __device__ __forceinline__ double& at(int p, int i) const
    {
        return p == 0 ? q0[place(i + kGhost, m0)] : (p == 1 ? q1 : q2)[place(i + kGhost, m12)];
    }
};

// Views of one instance for a step or a pass.  Pointers are generic: in the step kernel the bit
// planes, the conserved planes and more point into the CTA's shared memory (staged in and out around
// the steps, see Layout1), elsewhere into the instance's global buffers.
struct Ctx {
    const Inst1& I;
    Field1 f;               // conserved planes
    double *qc, *qt, *fl;   // stage-start copy, coarse derivatives, face fluxes: x[p*w + i + 3]
    uint32_t* pl;           // bit planes
    uint32_t *m0, *aux;     // planes of mask0 and of the first work plane (they change places)
    uint8_t* ls;            // the two list regions in shared memory (cap entries each) ...
    uint8_t* lg;            // ... and in global memory (list_entries1 entries each)
    unsigned cap;
    Work1* wk;
    const Weights& W;
    int w, nx, N1, maxl, nb, nw;

    __device__ double& Q(int p, int i) const { return f.at(p, i); }
    __device__ double& QT(int p, int i) const { return qt[p * w + i + kGhost]; }
    __device__ double& QC(int p, int i) const { return qc[p * w + i + kGhost]; }
    __device__ uint32_t* plane(int k) const { return pl + (size_t)k * nw; }
    __device__ uint32_t* mask(int k) const { return k == 0 ? m0 : plane(k); }
    __device__ uint32_t* fine(int k) const { return plane(kPlFine + k); }
    __device__ uint32_t* slice(int k, int b) const { return plane(kPlLevel + k * nb + b); }
    __device__ static bool bit(const uint32_t* P, int i) { return (P[(i >> 5) + 1] >> (i & 31)) & 1u; }
    __device__ int level(int k, int i) const
    {
        int v = 0;
        for (int b = 0; b < nb; ++b) v |= (int)((slice(k, b)[(i >> 5) + 1] >> (i & 31)) & 1u) << b;
        return v;
    }
    __device__ int no_level() const { return (1 << nb) - 1; }
    // Bits of word x that are points lo .. N1 + hi_pad of the line.
    __device__ uint32_t upto(int x, int last) const
    {
        const int r = last - 32 * (x - 1);
        return r < 0 ? 0u : r >= 31 ? ~0u : (2u << r) - 1u;
    }
    __device__ uint32_t inside(int x) const { return x < 1 ? 0u : upto(x, N1); }  // points [0, N1]
    // Word x of a mask, everything off the ghosted line set / masked to the points [0, N1].
    __device__ uint32_t padded(const uint32_t* P, int x) const { return x < 0 || x >= nw ? ~0u : P[x]; }
    __device__ uint32_t points(const uint32_t* P, int x) const { return x < 1 || x >= nw ? 0u : P[x] & upto(x, N1); }
    __device__ int D(int lev) const { return 1 << (maxl - lev); }
    __device__ double w_(int cnt, int k) const { return W.w[cnt][k + 1]; }
    // One point into a plane; points off the ghosted line (only reachable from inconsistent user-set
    // masks/levels, where the reference writes out of bounds) are dropped.
    __device__ void push(uint32_t* P, int i) const
    {
        if (i < -kGhost || i > N1 + kGhost) return;
        atomicOr(&P[(i >> 5) + 1], 1u << (i & 31));
    }
    // The region r list of n entries: in shared memory where it fits.
    __device__ List list(int r, size_t n) const
    {
        const size_t eb = entry_bytes(w);
        return List{n <= cap ? ls + r * eb * cap : lg + r * eb * list_entries1(w), short_lists(w)};
    }
};

// Bits of a word whose point index is an odd multiple of 2^t (t < 5).
__device__ __forceinline__ uint32_t odd_bits(int t)
{
    return t == 0 ? 0xAAAAAAAAu : t == 1 ? 0x44444444u : t == 2 ? 0x10101010u : t == 3 ? 0x01000100u : 0x00010000u;
}
// (cur << s) with the top of the word below it shifted in, (cur >> s) with the bottom of the word above.
__device__ __forceinline__ uint32_t shl(uint32_t below, uint32_t cur, int s) { return __funnelshift_l(below, cur, s); }
__device__ __forceinline__ uint32_t shr(uint32_t cur, uint32_t above, int s) { return __funnelshift_r(cur, above, s); }

// Maximum of non-negative doubles over the warp by their bit patterns (which order like the values).
__device__ __forceinline__ unsigned long long warp_max_bits(unsigned long long v)
{
    const unsigned hi = (unsigned)(v >> 32), mh = __reduce_max_sync(0xffffffffu, hi);
    const unsigned ml = __reduce_max_sync(0xffffffffu, hi == mh ? (unsigned)v : 0u);
    return ((unsigned long long)mh << 32) | ml;
}
__device__ __forceinline__ void reduce_put(Work1* wk, int slot, int which, double v)
{
    const unsigned long long m = warp_max_bits((unsigned long long)__double_as_longlong(v));
    if ((threadIdx.x & 31) == 0) wk->red[slot][which][threadIdx.x >> 5] = m;
}
// After the barrier that follows every warp's reduce_put; all 32 lanes of the warp call it.
__device__ __forceinline__ double reduce_get(const Work1* wk, int slot, int which)
{
    const int lane = threadIdx.x & 31, n = (blockDim.x + 31) >> 5;
    return __longlong_as_double((long long)warp_max_bits(lane < n ? wk->red[slot][which][lane] : 0ull));
}

// ------------------------------------------------------------------ masks and levels, bytes <-> planes
// Sets of planes: bits 0..4 mask0..mask3 and the previous mask0 (as in a mask byte), bits 8..11 the levels.
constexpr unsigned kAllPlanes = 0xf1fu;
__host__ __device__ constexpr unsigned level_plane(int k) { return 0x100u << k; }
// One warp per word, one point per lane.
__device__ void load_planes(const Ctx& c, const uint8_t* mb, const int8_t* lb)
{
    const int lane = threadIdx.x & 31, nwarp = blockDim.x >> 5;
    for (int x = threadIdx.x >> 5; x < c.nw; x += nwarp) {
        const int i = 32 * (x - 1) + lane;
        const bool on = i >= -kGhost && i <= c.N1 + kGhost;
        const unsigned v = on ? mb[i + kGhost] : 0x1fu;
        for (int k = 0; k < 5; ++k) {
            const uint32_t b = __ballot_sync(0xffffffffu, (v >> k) & 1u);
            if (lane == 0) (k == kPlTemp ? c.plane(kPlTemp) : c.mask(k))[x] = b;
        }
        for (int k = 0; k < 4; ++k) {
            const int l = on && i >= 0 && i <= c.N1 ? lb[k * c.w + i + kGhost] : 0;
            const int s = l < 0 || l > c.maxl ? c.no_level() : l;
            const uint32_t f = __ballot_sync(0xffffffffu, s == c.maxl);
            if (lane == 0) c.fine(k)[x] = f;
            for (int b = 0; b < c.nb; ++b) {
                const uint32_t y = __ballot_sync(0xffffffffu, (s >> b) & 1);
                if (lane == 0) c.slice(k, b)[x] = y;
            }
        }
    }
}
// A level outside 0..maxl keeps its byte.
__device__ void store_planes(const Ctx& c, uint8_t* mb, int8_t* lb)
{
    const int lane = threadIdx.x & 31, nwarp = blockDim.x >> 5;
    for (int x = threadIdx.x >> 5; x < c.nw; x += nwarp) {
        const int i = 32 * (x - 1) + lane;
        if (i < -kGhost || i > c.N1 + kGhost) continue;
        const bool ghost = i < 0 || i > c.N1;
        unsigned v = ghost ? 0xe0u : 0u;
        for (int k = 0; k < 4; ++k) v |= ((c.mask(k)[x] >> lane) & 1u) << k;
        v |= ((c.plane(kPlTemp)[x] >> lane) & 1u) << kBitTemp;
        mb[i + kGhost] = (uint8_t)v;
        if (ghost) continue;
        for (int k = 0; k < 4; ++k) {
            int l = 0;
            for (int b = 0; b < c.nb; ++b) l |= (int)((c.slice(k, b)[x] >> lane) & 1u) << b;
            if (l != c.no_level()) lb[k * c.w + i + kGhost] = (int8_t)l;
        }
    }
}
// The planes `which` alone, U words of a warp at a time, so that the latencies of their loads overlap: a single
// pass's conversions, by warp `warp` of `nwarp`.  (A step, whose launch converts all planes once beside its
// twenty passes, keeps the short loops above: these cost a 257-point scalar step 41 us instead of 34.)
// The bits of the planes left out keep their values.
template <int U>
__device__ __forceinline__ void load_some(const Ctx& c, const uint8_t* mb, const int8_t* lb, unsigned which, int warp, int nwarp)
{
    const int lane = threadIdx.x & 31;
    for (int x0 = warp; x0 < c.nw; x0 += U * nwarp) {
        auto word = [&](int u) { return x0 + u * nwarp; };
        auto point = [&](int u) { return 32 * (word(u) - 1) + lane; };
        bool on[U], in[U];  // on the ghosted line, on the line
#pragma unroll
        for (int u = 0; u < U; ++u) {
            on[u] = point(u) >= -kGhost && point(u) <= c.N1 + kGhost;
            in[u] = point(u) >= 0 && point(u) <= c.N1;
        }
        if (which & 0x1fu) {
            unsigned v[U];
#pragma unroll
            for (int u = 0; u < U; ++u) v[u] = on[u] ? mb[point(u) + kGhost] : 0x1fu;
#pragma unroll
            for (int k = 0; k < 5; ++k) {
                if (!((which >> k) & 1u)) continue;
                uint32_t* P = k == kPlTemp ? c.plane(kPlTemp) : c.mask(k);
#pragma unroll
                for (int u = 0; u < U; ++u) {
                    const uint32_t b = __ballot_sync(0xffffffffu, (v[u] >> k) & 1u);
                    if (lane == 0 && word(u) < c.nw) P[word(u)] = b;
                }
            }
        }
        for (int k = 0; k < 4; ++k) {
            if (!(which & level_plane(k))) continue;
            int l[U];
#pragma unroll
            for (int u = 0; u < U; ++u)
                l[u] = in[u] ? lb[k * c.w + point(u) + kGhost] : 0;
#pragma unroll
            for (int u = 0; u < U; ++u) {
                const int s = l[u] < 0 || l[u] > c.maxl ? c.no_level() : l[u];
                const bool put = lane == 0 && word(u) < c.nw;
                const uint32_t f = __ballot_sync(0xffffffffu, s == c.maxl);
                if (put) c.fine(k)[word(u)] = f;
                for (int b = 0; b < c.nb; ++b) {
                    const uint32_t y = __ballot_sync(0xffffffffu, (s >> b) & 1);
                    if (put) c.slice(k, b)[word(u)] = y;
                }
            }
        }
    }
}
template <int U>
__device__ __forceinline__ void store_some(const Ctx& c, uint8_t* mb, int8_t* lb, unsigned which, int warp, int nwarp)
{
    const int lane = threadIdx.x & 31;
    const unsigned masks = which & 0x1fu;
    for (int x0 = warp; x0 < c.nw; x0 += U * nwarp) {
        auto word = [&](int u) { return x0 + u * nwarp; };
        auto point = [&](int u) { return 32 * (word(u) - 1) + lane; };
        bool on[U], in[U];
#pragma unroll
        for (int u = 0; u < U; ++u) {
            on[u] = point(u) >= -kGhost && point(u) <= c.N1 + kGhost;
            in[u] = point(u) >= 0 && point(u) <= c.N1;
        }
        if (masks) {
            unsigned v[U];
#pragma unroll
            for (int u = 0; u < U; ++u) {
                v[u] = in[u] ? 0u : 0xe0u;
                if (masks != 0x1fu && on[u]) v[u] = mb[point(u) + kGhost] & ~masks;
            }
#pragma unroll
            for (int k = 0; k < 5; ++k) {
                if (!((which >> k) & 1u)) continue;
                const uint32_t* P = k == kPlTemp ? c.plane(kPlTemp) : c.mask(k);
#pragma unroll
                for (int u = 0; u < U; ++u)
                    if (on[u]) v[u] |= ((P[word(u)] >> lane) & 1u) << k;
            }
#pragma unroll
            for (int u = 0; u < U; ++u)
                if (on[u]) mb[point(u) + kGhost] = (uint8_t)v[u];
        }
        for (int k = 0; k < 4; ++k) {
            if (!(which & level_plane(k))) continue;
            int l[U] = {};
            for (int b = 0; b < c.nb; ++b) {
                const uint32_t* P = c.slice(k, b);
#pragma unroll
                for (int u = 0; u < U; ++u)
                    if (in[u]) l[u] |= (int)((P[word(u)] >> lane) & 1u) << b;
            }
#pragma unroll
            for (int u = 0; u < U; ++u)
                if (in[u] && l[u] != c.no_level()) lb[k * c.w + point(u) + kGhost] = (int8_t)l[u];
        }
    }
}

// ------------------------------------------------------------------------------ lists of points
// The points of [0, N1] in plane P (and not in `without`), ordered by class: class 0 = the coarsest
// grid's nodes, class l + 1 = the details of level l (i = odd 2^t is a detail of level
// maxl-1-t).  wk->off[k] is the start of class k, off[maxl + 1] the length.  Order within a class
// is free: the points of one class neither read nor write one another.  Three barriers.
__device__ __forceinline__ int class_of(const Ctx& c, int t) { return t >= c.maxl ? 0 : c.maxl - t; }
__device__ List order_points(const Ctx& c, int region, const uint32_t* P, const uint32_t* without = nullptr)
{
    Work1* wk = c.wk;
    auto word = [&](int x) { return c.points(P, x) & (without ? ~without[x] : ~0u); };
    // a warp takes every nwarp-th word, so that neighbouring active words go to different warps.
    // Points of odd multiples of 1 .. 16 are counted per warp: n0 and n1 hold the packed counts.
    const int lane = threadIdx.x & 31, wp = threadIdx.x >> 5, nwarp = blockDim.x >> 5;
    auto counts = [&](uint32_t v, unsigned& n) {
        const unsigned a = __reduce_add_sync(0xffffffffu, (unsigned)__popc(v & odd_bits(0)) | (__popc(v & odd_bits(1)) << 10) |
                                                              (__popc(v & odd_bits(2)) << 20));
        const unsigned b = __reduce_add_sync(0xffffffffu, (unsigned)__popc(v & odd_bits(3)) | (__popc(v & odd_bits(4)) << 10));
        n = lane == 0 ? a & 1023u : lane == 1 ? (a >> 10) & 1023u : lane == 2 ? a >> 20 : lane == 3 ? b & 1023u : b >> 10;
        return (a | b) != 0;
    };
    auto class0 = [&](int x) { return x == 1 ? 0 : class_of(c, 5 + __ffs(x - 1) - 1); };  // of bit 0 of word x
    for (int x0 = 1 + wp; x0 < c.nw; x0 += 32 * nwarp) {
        const int x = x0 + nwarp * lane;
        const uint32_t v = x < c.nw ? word(x) : 0u;
        unsigned n;
        if (counts(v, n) && lane < 5 && n) atomicAdd(&wk->cls[class_of(c, lane)], n);
        if (v & 1u) atomicAdd(&wk->cls[class0(x)], 1u);
    }
    __syncthreads();
    if (threadIdx.x < 32) {
        const unsigned n = wk->cls[lane];
        unsigned s = n;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const unsigned y = __shfl_up_sync(0xffffffffu, s, o);
            if (lane >= o) s += y;
        }
        wk->cls[lane] = 0;
        wk->run[lane] = wk->off[lane] = s - n;
        if (lane == 31) wk->off[32] = s;
    }
    __syncthreads();
    const List L = c.list(region, wk->off[32]);
    // the warp reserves its ranges, then expands its non-empty words one by one, a point per lane
    const int t = lane ? __ffs(lane) - 1 : 5;
    const uint32_t group = lane ? odd_bits(t) : 0u;
    for (int x0 = 1 + wp; x0 < c.nw; x0 += 32 * nwarp) {
        const int xl = x0 + nwarp * lane;
        const uint32_t mine = xl < c.nw ? word(xl) : 0u;
        if (mine & 1u) L.put(atomicAdd(&wk->run[class0(xl)], 1u), 32 * (xl - 1));
        unsigned n, pos = 0;
        if (!counts(mine, n)) continue;
        if (lane < 5 && n) pos = atomicAdd(&wk->run[class_of(c, lane)], n);
        pos = __shfl_sync(0xffffffffu, pos, t < 5 ? t : 0);  // the next position of this lane's group
        unsigned todo = __ballot_sync(0xffffffffu, (mine & ~1u) != 0);
        while (todo) {
            const int j = __ffs(todo) - 1;
            todo &= todo - 1;
            const uint32_t v = __shfl_sync(0xffffffffu, mine, j) & group;
            if ((v >> lane) & 1u) L.put(pos + __popc(v & ((1u << lane) - 1u)), 32 * (x0 + nwarp * j - 1) + lane);
            pos += __popc(v);
        }
    }
    __syncthreads();
    return L;
}

// The lists of one stage over mask k: needed faces f in [-1, N1] (face f+1/2 is needed when a
// finest-level point of the mask lies on either side), then the finest-level points, then the
// coarse points.  Their lengths are known from count_masks1.  No barrier: the caller's next one
// publishes the lists; the positions wk->n_list[k] must be zero before.
struct StageLists {
    List faces, fin, crs;
    int nf, nfin, ncrs;
};
__device__ __forceinline__ StageLists stage_lists(const Ctx& c, int k, int region)
{
    const Work1* wk = c.wk;
    const unsigned n = wk->mask_cnt[k], nf = wk->n_face[k], nfin = wk->n_fin[k];
    const List L = c.list(region, (size_t)nf + n);
    return StageLists{L, L.at(nf), L.at(nf + nfin), (int)nf, (int)nfin, (int)(n - nfin)};
}
// Words x of the finest-level points of mask k and of the faces they need (bit i: face i+1/2).
__device__ __forceinline__ uint32_t fine_word(const Ctx& c, int k, int x)
{
    return x < 1 || x >= c.nw ? 0u : c.points(c.mask(k), x) & c.fine(k)[x];
}
__device__ void build_stage_lists(const Ctx& c, int k, int region)
{
    const StageLists L = stage_lists(c, k, region);
    unsigned* pos = c.wk->n_list[k];
    const int lane = threadIdx.x & 31, wp = threadIdx.x >> 5, nwarp = blockDim.x >> 5;
    const unsigned lt = (1u << lane) - 1u;
    // words to warps as in order_points
    for (int x0 = wp; x0 < c.nw; x0 += 32 * nwarp) {
        const int xl = x0 + nwarp * lane;
        uint32_t m = 0, f = 0, fa = 0;
        if (xl < c.nw) {
            m = c.points(c.mask(k), xl);
            f = fine_word(c, k, xl);
            fa = f | shr(f, fine_word(c, k, xl + 1), 1);
        }
        unsigned todo = __ballot_sync(0xffffffffu, (m | fa) != 0);
        if (!todo) continue;
        const unsigned nfa = __reduce_add_sync(0xffffffffu, __popc(fa));
        const unsigned nfc = __reduce_add_sync(0xffffffffu, __popc(f) | (__popc(m & ~f) << 16));
        unsigned base = 0;
        if (lane < 3) base = atomicAdd(&pos[lane], lane == 0 ? nfa : lane == 1 ? nfc & 0xffffu : nfc >> 16);
        unsigned bf = __shfl_sync(0xffffffffu, base, 0), bp = __shfl_sync(0xffffffffu, base, 1);
        unsigned bc = __shfl_sync(0xffffffffu, base, 2);
        while (todo) {
            const int j = __ffs(todo) - 1;
            todo &= todo - 1;
            const uint32_t mj = __shfl_sync(0xffffffffu, m, j), fj = __shfl_sync(0xffffffffu, f, j);
            const uint32_t faj = __shfl_sync(0xffffffffu, fa, j), cj = mj & ~fj;
            const int i = 32 * (x0 + nwarp * j - 1) + lane;
            if ((faj >> lane) & 1u) L.faces.put(bf + __popc(faj & lt), i);
            if ((fj >> lane) & 1u) L.fin.put(bp + __popc(fj & lt), i);
            if ((cj >> lane) & 1u) L.crs.put(bc + __popc(cj & lt), i);
            bf += __popc(faj);
            bp += __popc(fj);
            bc += __popc(cj);
        }
    }
}

// ------------------------------------------------------------------ PrepareEuler building blocks
// One phase of a transform over the entries [lo, hi) of an ordered list, on spacing D: the details of
// one level (predict) or the coarser points (update), forward or inverse.  temp: the inverse predict
// also interpolates momentum and energy of the points outside it.
// The weights away from the ends, -1/16 and 9/16 (make_weights gives them exactly).
constexpr double kInnerW0 = -0.0625, kInnerW1 = 0.5625;
enum Lift1 { kPredictF, kUpdateF, kUpdateI, kPredictI };
template <int OP, class Points>
__device__ __forceinline__ void lift1(const Ctx& c, const Points& L, unsigned lo, unsigned hi, int D,
                                      const uint32_t* temp = nullptr)
{
    constexpr bool predict = OP == kPredictF || OP == kPredictI;
    const double tol = c.I.tol;
    for (unsigned e = lo + threadIdx.x; e < hi; e += blockDim.x) {
        const int i = L.get(e);
        if (Points::kSome && i < 0) continue;
        if (!predict && (i == 0 || i == c.N1)) continue;
        int s, k;
        if (predict) predict_stencil(i, D, c.N1, s, k);
        else update_stencil(i, D, c.N1, s, k);
        double v = c.Q(0, i), w[4] = {kInnerW0, kInnerW1, kInnerW1, kInnerW0};
        if (k != 1)
#pragma unroll
            for (int n = 0; n < 4; ++n) w[n] = c.w_(n, k);
        if (OP == kPredictI) v *= 2;
#pragma unroll
        for (int n = 0; n < 4; ++n) {
            const double y = w[n] * c.Q(0, s + n * D);
            v = OP == kPredictF || OP == kUpdateI ? v - y : v + y;
        }
        if (OP == kPredictF) v *= 0.5;
        c.Q(0, i) = v;
        if (OP == kPredictF && absd(v) < tol) atomicAnd(&c.m0[(i >> 5) + 1], ~(1u << (i & 31)));
        if (OP == kPredictI && temp && !Ctx::bit(temp, i)) {
            double y = 0, z = 0;
#pragma unroll
            for (int n = 0; n < 4; ++n) {
                y += w[n] * c.Q(1, s + n * D);
                z += w[n] * c.Q(2, s + n * D);
            }
            c.Q(1, i) = y;
            c.Q(2, i) = z;
        }
    }
}

// ForwardWaveletTransformEuler (Wavelet/WAVELET_1D.h:282-335) over the points of mask0, listed by
// order_points: level by level the details of the level, then the coarser points.
__device__ void fwt1(const Ctx& c, const List& L)
{
    const unsigned* off = c.wk->off;
    for (int lev = c.maxl - 1; lev >= 0; --lev) {
        lift1<kPredictF>(c, L, off[lev + 1], off[lev + 2], c.D(lev));
        __syncthreads();
        lift1<kUpdateF>(c, L, 0, off[lev + 1], c.D(lev));
        __syncthreads();
    }
}

// The same without a list, for a pass on a short line: a thread per point of a level.
struct SomePoints {  // first, first + D, .. : those of plane P, else -1
    static constexpr bool kSome = true;
    const uint32_t* P;
    int first, D;
    __device__ __forceinline__ int get(unsigned e) const
    {
        const int i = first + (int)e * D;
        return Ctx::bit(P, i) ? i : -1;
    }
};
__device__ void fwt_short1(const Ctx& c)
{
    for (int lev = c.maxl - 1; lev >= 0; --lev) {
        const int D = c.D(lev), nd = c.N1 / D;
        lift1<kPredictF>(c, SomePoints{c.m0, D >> 1, D}, 0, nd, D);
        __syncthreads();
        lift1<kUpdateF>(c, SomePoints{c.m0, D, D}, 0, nd - 1, D);
        __syncthreads();
    }
}

// InverseWaveletTransformEuler(q, mask3) and InterpolateEuler(q, mask_temp, mask3)
// (Wavelet/WAVELET_1D.h:337-391, 393-431) over the points of mask3, listed by order_points.
// The interpolation of level l's new points (mask3 without mask_temp) reads the momentum and
// energy of coarser points, the transform the density: one phase does both.  The work mask that the
// reference closes first adds nothing here, because mask3 is closed under CheckReconstruction: the
// closure of a part of it lies inside it.
// The reference also sets the density to 0 at the points outside mask3, each in its level's phase.
// A level's update reads those points before that phase, and nothing reads them after it (the
// stencils of mask3's points lie in mask3), so the caller zeroes them at the end, or not at all
// where the residue removal does.
__device__ void iwt_interp1(const Ctx& c, const List& L, bool interp)
{
    const unsigned* off = c.wk->off;
    const uint32_t* temp = c.plane(kPlTemp);
    for (int lev = 0; lev < c.maxl; ++lev) {
        const unsigned lo = off[lev + 1], hi = off[lev + 2];
        const int D = c.D(lev);
        lift1<kUpdateI>(c, L, 0, lo, D);
        __syncthreads();
        lift1<kPredictI>(c, L, lo, hi, D, interp ? temp : nullptr);
        __syncthreads();
    }
}

// CheckReconstruction (Wavelet/AWCM_MANAGER_1D.h:45-71): every detail i of spacing h = 2^t in the
// mask marks its four coarse neighbours i -+ h, i -+ 3h, fine to coarse.  At the ends the stencil of
// the first detail h is that of the next one (0, 2h, 4h, 6h), and that of the last one N1 - h that of
// N1 - 3h, so those two count twice.  A level up to h = 16 is a few shifts of each word and its
// neighbours, and five levels reach at most 93 points: a warp holds 32 consecutive words, one per
// lane, takes the neighbours by shuffles through all five levels without a barrier, and keeps the 26
// words in the middle (three words of margin on either side).  A word that another warp has closed
// already only holds points that belong to the closure anyway, so words are closed in place.
// (One window of six words per thread took 2.7 us a mask of 1025 points with the coarse levels, a
// block barrier per level the same.)  The levels above are bit 0 of their words: up to 128 details on
// one warp, more on the whole block.
__device__ __forceinline__ void close_words(const Ctx& c, uint32_t* P)
{
    constexpr int kKeep = 26, kMargin = 3;
    const int lane = threadIdx.x & 31, nwarp = blockDim.x >> 5, top = min(c.maxl, 5);
    for (int x0 = 1 + (int)(threadIdx.x >> 5) * kKeep; x0 < c.nw; x0 += nwarp * kKeep) {
        const int x = x0 - kMargin + lane;
        const uint32_t in = x < c.nw ? c.inside(x) : 0u;
        uint32_t v = in ? P[x] & in : 0u;
        if (!__any_sync(0xffffffffu, v != 0)) continue;
        const uint32_t was = v;
        const int rl = c.N1 - 32 * (x - 1);  // bit of the last point, counted from this word
#pragma unroll
        for (int t = 0; t < 5; ++t) {
            if (t >= top) break;
            const int h = 1 << t;
            uint32_t d = v & odd_bits(t);
            // the detail h (in word 1) also as 3h, for h = 16 in the next word
            if (t < 4) {
                if (x == 1) d |= (d & (1u << h)) << (2 * h);
            } else {
                const uint32_t b = __shfl_up_sync(0xffffffffu, d, 1);
                if (x == 2) d |= b;
            }
            // the detail N1 - h also as N1 - 3h, in the same word or the one below
            {
                const int s = rl - h;
                const uint32_t e = s >= 0 && s < 32 ? d & (1u << s) : 0u;
                const uint32_t f = __shfl_down_sync(0xffffffffu, e, 1);
                d |= t < 4 ? shr(e, f, 2 * h) : f;
            }
            const uint32_t l = __shfl_up_sync(0xffffffffu, d, 1), r = __shfl_down_sync(0xffffffffu, d, 1);
            if (t < 4) {
                v |= (shl(l, d, h) | shr(d, r, h) | shl(l, d, 3 * h) | shr(d, r, 3 * h)) & in;
            } else {
                // bit 16 of a word marks bit 0 of the words at 0, +1, +2 and -1
                const uint32_t ll = __shfl_up_sync(0xffffffffu, d, 2);
                v |= ((l | d | r | ll) >> 16) & in;
            }
        }
        // (the shuffles' end lanes took their own words for their outer neighbours': margin only)
        if (lane >= kMargin && lane < kMargin + kKeep && v != was) P[x] |= v;
    }
}
__device__ __forceinline__ void close_point(const Ctx& c, uint32_t* P, int t, int a)
{
    const int h = 1 << t, D = 2 * h, i = h + a * D;
    if (!(P[(i >> 5) + 1] & 1u)) return;
    int s, k;
    predict_stencil(i, D, c.N1, s, k);
#pragma unroll
    for (int cnt = 0; cnt < 4; ++cnt) atomicOr(&P[((s + cnt * D) >> 5) + 1], 1u);
}
__device__ __forceinline__ void close1(const Ctx& c, uint32_t* P)
{
    close_words(c, P);
    __syncthreads();
    int t = 5;
    for (; t < c.maxl && (c.N1 >> (t + 1)) > 128; ++t) {
        for (int a = threadIdx.x; a < (c.N1 >> (t + 1)); a += blockDim.x) close_point(c, P, t, a);
        __syncthreads();
    }
    if (t < c.maxl) {
        if (threadIdx.x < 32)
            for (; t < c.maxl; ++t) {
                for (int a = threadIdx.x; a < (c.N1 >> (t + 1)); a += 32) close_point(c, P, t, a);
                __syncwarp();
            }
        __syncthreads();
    }
}

// AddAdjacentZone (Wavelet/AWCM_MANAGER_1D.h:14-43) of word x of the mask whose words word(y) gives
// (points [0, N1] only): the points that the word's own and the neighbouring details mark.  A detail
// i = odd 2^t marks i -+ max(1, 2^(t-1)).
template <class Word>
__device__ __forceinline__ uint32_t zone_word(const Ctx& c, int x, Word word)
{
    uint32_t s = 0;
    if (x >= 1) {
        const uint32_t l = word(x - 1), v = word(x), r = word(x + 1);
        if (l | v | r) {
            const uint32_t p01 = odd_bits(0) | (c.maxl > 1 ? odd_bits(1) : 0u);
            s |= shl(l & p01, v & p01, 1) | shr(v & p01, r & p01, 1);
#pragma unroll
            for (int t = 2; t < 5; ++t) {
                if (t >= c.maxl) break;
                const uint32_t p = odd_bits(t);
                s |= shl(l & p, v & p, 1 << (t - 1)) | shr(v & p, r & p, 1 << (t - 1));
            }
            if (c.maxl > 5) s |= ((x & 1) ? r & 1u : v & 1u) << 16;  // i = odd 32: bit 0 of an even word
        }
        // t >= 6: point 32 m' is marked by 32 (m' -+ 2^z), z = ctz(m'), if that is an odd multiple of 2^(z+1)
        const int m = x - 1;
        if (m > 0) {
            const int z = __ffs(m) - 1;
            if (z + 6 < c.maxl) {
                const int lo = m - (1 << z), hi = m + (1 << z);
                if (((lo >> (z + 1)) & 1) && (word(lo + 1) & 1u)) s |= 1u;
                if (((hi >> (z + 1)) & 1) && (word(hi + 1) & 1u)) s |= 1u;
            }
        }
    }
    return s;
}

// BadingBoundary (AWCM_1D.h:73-80: mask0 set on the three points at each end, i < 3 and i > N1 - 3).
__device__ __forceinline__ uint32_t band_word(const Ctx& c, int x)
{
    uint32_t b = x == 1 ? 7u : 0u;
    for (int i = c.N1 - 2; i <= c.N1; ++i)
        if ((i >> 5) + 1 == x) b |= 1u << (i & 31);
    return b;
}

// ComputeLevel (Wavelet/AWCM_MANAGER_1D.h:109-133) of word x of mask M into level set k: the points
// whose nearest neighbour in the mask is 2^j away get level maxl - j (the reference searches the
// distances one by one; here each distance is one shift of the whole word).  Off the ghosted line
// the mask reads as set.  A point without any such neighbour keeps its level.
// f(j, set): called for those points with their levels maxl - j, and with `all` for every level's.
__device__ __forceinline__ uint32_t end_bits(const Ctx& c, int x)
{
    return (x == 1 ? 1u : 0u) | ((c.N1 >> 5) + 1 == x ? 1u << (c.N1 & 31) : 0u);
}
// The points of word x (v, with its neighbours l and r) that have a neighbour in M at distance 2^j.
__device__ __forceinline__ uint32_t near_word(const Ctx& c, const uint32_t* M, int x, uint32_t l, uint32_t v, uint32_t r, int j)
{
    if (j < 5) return shl(l, v, 1 << j) | shr(v, r, 1 << j);
    return c.padded(M, x - (1 << (j - 5))) | c.padded(M, x + (1 << (j - 5)));
}
template <class F>
__device__ __forceinline__ void level_word(const Ctx& c, int k, const uint32_t* M, int x, F&& f, bool all = false)
{
    const uint32_t in = c.inside(x), ends = end_bits(c, x);  // the ends: the finest level, in the mask or not
    uint32_t todo = in ? M[x] & in & ~ends : 0u, fine = ends;
    uint32_t S[5];
#pragma unroll
    for (int b = 0; b < 5; ++b) S[b] = ((c.maxl >> b) & 1) ? fine : 0u;
    if (todo) {
        const uint32_t l = c.padded(M, x - 1), v = M[x], r = c.padded(M, x + 1);
        for (int j = 0; j <= c.maxl && todo; ++j) {
            const uint32_t got = todo & near_word(c, M, x, l, v, r, j);
            todo &= ~got;
            if (j == 0) fine |= got;
            else if (all && got) f(j, got);
            const int lev = c.maxl - j;
#pragma unroll
            for (int b = 0; b < 5; ++b)
                if ((lev >> b) & 1) S[b] |= got;
        }
        if (todo) {  // no neighbour found: the level stays as it was
            const uint32_t old = c.fine(k)[x] & todo;
            fine |= old;
            for (uint32_t u = todo; u; u &= u - 1) {
                const uint32_t one = u & (0u - u);
                int lev = 0;
#pragma unroll
                for (int b = 0; b < 5; ++b)
                    if (b < c.nb && (c.slice(k, b)[x] & one)) {
                        lev |= 1 << b;
                        S[b] |= one;
                    }
                if (lev != c.no_level()) f(c.maxl - lev, one);
            }
        }
    }
    if (all && in && (fine & M[x] & in)) f(0, fine & M[x] & in);
    c.fine(k)[x] = fine;
#pragma unroll
    for (int b = 0; b < 5; ++b)
        if (b < c.nb) c.slice(k, b)[x] = S[b];
}

// AddPointForDifferentiation (Wavelet/AWCM_MANAGER_1D.h:73-107) of the points `set` (points [0, N1])
// of word x, all of level maxl - j, into P: the finest level marks i-3 .. i+3, a coarser one
// the 5 points i-2D .. i+2D, or 6 points from the end it is near to.  own: the part that falls in
// the word itself.
__device__ __forceinline__ void stencil_push(const Ctx& c, uint32_t* P, int x, int j, uint32_t set, uint32_t& own)
{
    if (j == 0) {
        const uint32_t up = (set >> 31) | (set >> 30) | (set >> 29), dn = (set << 31) | (set << 30) | (set << 29);
        own |= set | (set << 1) | (set << 2) | (set << 3) | (set >> 1) | (set >> 2) | (set >> 3);
        if (up) atomicOr(&P[x + 1], up);
        if (dn) atomicOr(&P[x - 1], dn);
        return;
    }
    const int D = 1 << j, i0 = 32 * (x - 1);
    if (i0 <= 2 * D) {
        const uint32_t left = set & c.upto(x, 2 * D);
        if (left)
            for (int n = 0; n < 6; ++n) c.push(P, n * D);
        set &= ~left;
    }
    if (i0 + 31 >= c.N1 - 2 * D) {
        const uint32_t right = set & ~c.upto(x, c.N1 - 2 * D - 1);
        if (right)
            for (int n = 0; n < 6; ++n) c.push(P, c.N1 - n * D);
        set &= ~right;
    }
    if (!set) return;
    own |= set;
    if (j < 5) {
        // within the word and its two neighbours (2 D = 32 is the whole word)
        uint32_t up = set >> (32 - D), dn = set << (32 - D);
        own |= (set << D) | (set >> D);
        if (j < 4) {
            own |= (set << (2 * D)) | (set >> (2 * D));
            up |= set >> (32 - 2 * D);
            dn |= set << (32 - 2 * D);
        } else {
            up |= set;
            dn |= set;
        }
        if (up) atomicOr(&P[x + 1], up);
        if (dn) atomicOr(&P[x - 1], dn);
    } else {
        const int o = D >> 5;
        atomicOr(&P[x + o], set);
        atomicOr(&P[x - o], set);
        atomicOr(&P[x + 2 * o], set);
        atomicOr(&P[x - 2 * o], set);
    }
}

// ComputeLevel(level_{k-1}, mask_{k-1}), mask_k = mask_{k-1}, AddAdjacentZone(mask_k) (zone) and
// AddPointForDifferentiation(mask_k, level_{k-1}) in one phase.  All of them read mask_{k-1} only
// (the zone's points are not in it, so their level is 0), and mask_k (clear before) takes ORs.
// Lines of up to a few thousand points leave most warps idle at one word per thread.  There a warp takes
// 32 words and one job at a time -- the points of one distance, the zone, or the level planes -- so that
// the searches of the levels run side by side; each of them searches the nearer distances again, so
// with more words a thread goes through its word's distances in turn.  Steps by jobs / by words: 1025 points (34
// words) 52.0 / 57.0 us, 2049 64.2 / 68.9, 3073 (98 words) 71.3 / 74.6, 4097 (130) 84.5 / 86.4, 5121 (162) 79.0 / 79.8,
// 6145 (194) 93.6 / 91.6, 8193 114.4 / 110.8, 15361 193 / 172.
constexpr int kJobWords1 = 5;  // times 32 words
__device__ void next_mask1(const Ctx& c, int k, bool zone)
{
    const uint32_t* A = c.mask(k - 1);
    uint32_t* B = c.plane(k);
    auto pts = [&](int y) { return c.points(A, y); };
    const int lane = threadIdx.x & 31, nwarp = blockDim.x >> 5;
    const int nch = (c.nw + 31) >> 5, njobs = (c.maxl + 3) * nch;
    if (nch > kJobWords1) {
        for (int x = threadIdx.x; x < c.nw; x += blockDim.x) {
            const uint32_t a = A[x];
            const uint32_t fresh = zone ? zone_word(c, x, pts) & ~a : 0u;
            uint32_t own = a | fresh;
            level_word(c, k - 1, A, x, [&](int j, uint32_t set) { stencil_push(c, B, x, j, set, own); }, true);
            if (fresh) stencil_push(c, B, x, c.maxl, fresh, own);
            if (own) atomicOr(&B[x], own);
        }
        __syncthreads();
        return;
    }
    for (int job = threadIdx.x >> 5; job < njobs; job += nwarp) {
        const int j = job / nch, x = 32 * (job - j * nch) + lane;
        if (x >= c.nw) continue;
        const uint32_t a = A[x];  // ghosts and the bits off the line included
        uint32_t own = 0;
        if (j <= c.maxl) {
            const uint32_t ends = end_bits(c, x), on = a & c.inside(x);
            uint32_t got = on & ~ends;
            if (got) {
                // the points with a neighbour 2^j away and none nearer
                const uint32_t l = c.padded(A, x - 1), r = c.padded(A, x + 1);
                for (int i = 0; i < j; ++i) got &= ~near_word(c, A, x, l, a, r, i);
                if (got) got &= near_word(c, A, x, l, a, r, j);
            }
            if (j == 0) got |= ends & on;
            if (got) stencil_push(c, B, x, j, got, own);
        } else if (j == c.maxl + 1) {
            own = a;
            if (zone) {
                const uint32_t fresh = zone_word(c, x, pts) & ~a;
                own |= fresh;
                if (fresh) stencil_push(c, B, x, c.maxl, fresh, own);
            }
        } else {
            level_word(c, k - 1, A, x, [&](int jj, uint32_t set) { stencil_push(c, B, x, jj, set, own); });
        }
        if (own) atomicOr(&B[x], own);
    }
    __syncthreads();
}

// ComputeLevel alone.
__device__ void levels1(const Ctx& c, int k, const uint32_t* M)
{
    for (int x = threadIdx.x; x < c.nw; x += blockDim.x) level_word(c, k, M, x, [](int, uint32_t) {});
}

// Numbers of points of mask0..mask3 in [0, N1], and of the finest-level points and needed faces of
// mask0..mask2, into the workspace (zero before); no barrier.
__device__ void count_masks1(const Ctx& c)
{
    for (int x0 = 0; x0 < c.nw; x0 += blockDim.x) {
        const int x = x0 + (int)threadIdx.x;
        const bool head = (threadIdx.x & 31) == 0;
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            const unsigned n = __reduce_add_sync(0xffffffffu, x < c.nw ? __popc(c.points(c.mask(k), x)) : 0);
            if (n && head) atomicAdd(&c.wk->mask_cnt[k], n);
            if (k == 3) continue;
            const uint32_t f = fine_word(c, k, x);
            const uint32_t fa = x < c.nw ? f | shr(f, fine_word(c, k, x + 1), 1) : 0u;
            const unsigned nn = __reduce_add_sync(0xffffffffu, __popc(f) | (__popc(fa) << 16));
            if (nn && head) {
                atomicAdd(&c.wk->n_fin[k], nn & 0xffffu);
                atomicAdd(&c.wk->n_face[k], nn >> 16);
            }
        }
    }
}

// The mask and level chain and the transforms of AWCM_1D::PrepareEuler (Wavelet/AWCM_1D.h:86-120),
// or with euler false of AWCM_1D::Prepare (Wavelet/AWCM_1D.h:45-72: no mask_temp, no adjacent zones
// on mask1..mask3, no interpolation).  Leaves the ordered list of mask3 in region 0 and the counts
// of the masks, and does not zero the density outside mask3 (see iwt_interp1).  The start's mask0
// is in kPlTemp (euler) or kPlStart.
__device__ List prepare1(Ctx& c, bool euler)
{
    Work1* wk = c.wk;
    uint32_t* start = c.plane(euler ? kPlTemp : kPlStart);
    for (int x = threadIdx.x; x < c.nw; x += blockDim.x) {
        start[x] = c.m0[x];
        c.plane(1)[x] = c.plane(2)[x] = c.plane(3)[x] = 0;
    }
    if (threadIdx.x < 16) wk->n_list[threadIdx.x >> 2][threadIdx.x & 3] = 0;
    if (threadIdx.x < 4) wk->mask_cnt[threadIdx.x] = wk->n_face[threadIdx.x] = wk->n_fin[threadIdx.x] = 0;
    fwt1(c, order_points(c, 0, c.m0));
    for (int k = 0; k <= 3; ++k) {
        if (k == 0) {
            // banding and AddAdjacentZone of mask0, into the other plane
            const uint32_t* m = c.m0;
            auto band = [&](int y) { return y < 1 || y >= c.nw ? 0u : (m[y] | band_word(c, y)) & c.inside(y); };
            for (int x = threadIdx.x; x < c.nw; x += blockDim.x)
                c.aux[x] = m[x] | band_word(c, x) | zone_word(c, x, band);
            __syncthreads();
            uint32_t* t = c.m0;
            c.m0 = c.aux;
            c.aux = t;
        } else {
            next_mask1(c, k, euler);
        }
        close1(c, c.mask(k));
    }
    levels1(c, 3, c.plane(3));
    count_masks1(c);
    const List L3 = order_points(c, 0, c.plane(3));
    iwt_interp1(c, L3, euler);
    return L3;
}

// --------------------------------------------------------------------------------- RK3 stages
// The ghost cell fill of one component p and distance g (1..3) at both ends.
__device__ __forceinline__ void bc_cell1(const Ctx& c, int p, int g)
{
    if (!c.I.bc_generic) {
        // BOUNDARY_MANAGER::SetBoundaryCondition (Problems/1D/PROBLEM_SHOCKTUBE.h:86-107).
        c.Q(p, -g) = c.Q(p, 0);
        c.Q(p, c.N1 + g) = c.Q(p, c.N1);
    } else {
        // BOUNDARY_MANAGER_1D<T>::SetBoundaryCondition (BOUNDARY_MANAGER_1D.h:47-75): zero-order
        // extrapolation or the periodic image (ghost -g <- N1-(g-1), N1+g <- g-1) by the
        // condition of each ghost cell; other conditions leave it.
        const int kl = c.I.bcg[g - 1], kr = c.I.bcg[kGhost + g - 1];
        if (kl == kBcExtrapolation1) c.Q(p, -g) = c.Q(p, 0);
        else if (kl == kBcPeriodic1) c.Q(p, -g) = c.Q(p, c.N1 - (g - 1));
        if (kr == kBcExtrapolation1) c.Q(p, c.N1 + g) = c.Q(p, c.N1);
        else if (kr == kBcPeriodic1) c.Q(p, c.N1 + g) = c.Q(p, g - 1);
    }
}
__device__ __forceinline__ void bc1(const Ctx& c)
{
    if (threadIdx.x < 3 * kGhost) bc_cell1(c, threadIdx.x / kGhost, threadIdx.x % kGhost + 1);
}

// |u| + c (main_1d_euler.cpp:67-95); nf: set when it is NaN or infinite (NaN/Inf state, negative
// pressure or density).
__device__ __noinline__ double speed1_any(double q0, double q1, double q2, double gamma)
{
    return absd(q1 / q0) + sound1(q0, q1, q2, gamma);
}
__device__ __forceinline__ double speed1(double q0, double q1, double q2, double gamma, bool& nf)
{
    SharedDiv dv;
    double s = awcm::speed1(dv, q0, q1, q2, gamma);
    if (dv.bad) s = speed1_any(q0, q1, q2, gamma);
    nf |= !isfinite(s);
    return s;
}

// Coarse-level flux derivative (AWCM_1D::DifferentiateEuler*, Wavelet/AWCM_1D.h:142-189) with the
// driver's branch selection (main_1d_euler.cpp:111-133); right-boundary forms mirror the left ones.
// Reads the stage input Q, which no point update has touched yet when it runs.
template <class DV>
__device__ __forceinline__ void coarse_dF1(DV& dv, const Field1& q, int iend, int i, int d, double* dF)
{
    const double g = 1.4;  // EULER_EQUATION_1D euler_eqn(1.4) in the reference helpers
    auto F = [&](int ii, double* f) {
        const double s[3] = {q.at(0, ii), q.at(1, ii), q.at(2, ii)};
        flux1(dv, s, g, f);
    };
    double a[3], b[3], e[3], f[3], h[3];
    if (i - 2 * d > 0 && i + 2 * d < iend) {
        F(i - 2 * d, a), F(i - d, b), F(i + d, e), F(i + 2 * d, f);
        for (int p = 0; p < 3; ++p) dF[p] = kD1 * (e[p] - b[p]) + kD2 * (f[p] - a[p]);
    } else if (i - 2 * d < 0) {
        F(i - d, a), F(i, b), F(i + d, e), F(i + 2 * d, f);
        for (int p = 0; p < 3; ++p) dF[p] = kD01 * a[p] + kD11 * b[p] + kD21 * e[p] + kD31 * f[p];
    } else if (i == 2 * d) {
        F(i - 2 * d, a), F(i - d, b), F(i, e), F(i + d, f), F(i + 2 * d, h);
        for (int p = 0; p < 3; ++p) dF[p] = kD02 * a[p] + kD12 * b[p] + kD22 * e[p] + kD32 * f[p] + kD2 * h[p];
    } else if (i > iend - 2 * d) {
        F(i + d, a), F(i, b), F(i - d, e), F(i - 2 * d, f);
        for (int p = 0; p < 3; ++p) dF[p] = kD01 * a[p] + kD11 * b[p] + kD21 * e[p] + kD31 * f[p];
    } else {
        F(i + 2 * d, a), F(i + d, b), F(i, e), F(i - d, f), F(i - 2 * d, h);
        for (int p = 0; p < 3; ++p) dF[p] = kD02 * a[p] + kD12 * b[p] + kD22 * e[p] + kD32 * f[p] + kD2 * h[p];
    }
}

// A coarse point or a face whose operands are outside the range of SharedDiv, with IEEE divisions.
__device__ __noinline__ void coarse_any1(Field1 q, int N1, int i, int d, double* out, int w)
{
    IeeeDiv dv;
    double dF[3];
    coarse_dF1(dv, q, N1, i, d, dF);
    for (int k = 0; k < 3; ++k) out[k * w] = dF[k];
}
template <class DV>
__device__ __forceinline__ void face1(DV& dv, const Field1& q, int f, int scheme, double alpha, double gamma, double* out,
                                      int w)
{
    double s[6][3], o[3];
#pragma unroll
    for (int p = 0; p < 6; ++p)
#pragma unroll
        for (int k = 0; k < 3; ++k) s[p][k] = q.at(k, f - 2 + p);
    if (scheme == kWeno5) face_flux_1d<kWeno5>(dv, s, alpha, gamma, o);
    else face_flux_1d<kWenoZ>(dv, s, alpha, gamma, o);
#pragma unroll
    for (int k = 0; k < 3; ++k) out[k * w] = o[k];
}
__device__ __noinline__ void face_any1(Field1 q, int f, int scheme, double alpha, double gamma, double* out, int w)
{
    IeeeDiv dv;
    face1(dv, q, f, scheme, alpha, gamma, out, w);
}

// Spacing of the coarse point i in level set k, or 0: a level outside 0..maxl or a derivative
// stencil that leaves the ghosted line (the point then keeps its value).
__device__ __forceinline__ int coarse_spacing(const Ctx& c, int k, int i)
{
    const int lev = c.level(k, i);
    if (lev > c.maxl) return 0;
    const int d = c.D(lev);
    return (i - 2 * d < -kGhost || i + 2 * d > c.N1 + kGhost) ? 0 : d;
}

// One stage over mask k / level set k (main_1d_euler.cpp:97-245): kind 1..3 with k = 2, 1, 0.  Faces
// are computed once (face i+1/2 is shared by points i and i+1; the reference evaluates it for
// both, identically).  The faces and the coarse derivatives read the stage input Q and run in one
// phase (the coarse derivatives are parked in qt); the point updates follow in a second phase, so Q
// is never read after a point of this stage has been written and no copy of the stage input is
// needed.  Beside the faces the next stage's lists are built.  The update of a finest-level point
// of stages 1 and 2 also gives its speed: these points are exactly those of the next stage's
// Lax-Friedrichs scan (main_1d_euler.cpp:86-95), whose maximum over the block comes from slot
// `kind` of the reductions after the barrier that ends the stage.
__device__ __forceinline__ void stage1(const Ctx& c, int scheme, int kind, double alpha, double dt, bool& nf)
{
    const int k = 3 - kind, region = kind == 2 ? 0 : 1;
    const StageLists L = stage_lists(c, k, region);
    if (kind < 3) build_stage_lists(c, k - 1, 1 - region);
    for (int e = threadIdx.x; e < L.nf + L.ncrs; e += blockDim.x) {
        if (e < L.nf) {
            const int f = L.faces.get(e);
            SharedDiv dv;
            face1(dv, c.f, f, scheme, alpha, c.I.gamma, c.fl + f + kGhost, c.w);
            if (dv.bad) face_any1(c.f, f, scheme, alpha, c.I.gamma, c.fl + f + kGhost, c.w);
        } else {
            const int i = L.crs.get(e - L.nf), d = coarse_spacing(c, k, i);
            if (!d) continue;
            SharedDiv dv;
            double dF[3];
            coarse_dF1(dv, c.f, c.N1, i, d, dF);
#pragma unroll
            for (int q = 0; q < 3; ++q) c.QT(q, i) = dF[q];
            if (dv.bad) coarse_any1(c.f, c.N1, i, d, c.qt + i + kGhost, c.w);
        }
    }
    __syncthreads();
    double fast = 0;
    const double sc1 = dt / (c.I.dx * 1);
    for (int e = threadIdx.x; e < L.nfin + L.ncrs; e += blockDim.x) {
        int i, d;
        double dF[3];
        if (e < L.nfin) {
            i = L.fin.get(e);
            d = 1;
#pragma unroll
            for (int q = 0; q < 3; ++q) dF[q] = c.fl[q * c.w + i + kGhost] - c.fl[q * c.w + i - 1 + kGhost];
        } else {
            i = L.crs.get(e - L.nfin);
            d = coarse_spacing(c, k, i);
#pragma unroll
            for (int q = 0; q < 3; ++q) dF[q] = d ? c.QT(q, i) : 0.0;
        }
        // the stage-start copy: stages 2 and 3 read it on mask1 only
        const bool keep = kind == 1 && Ctx::bit(c.plane(1), i);
        // dt / (dx d): d is a power of two
        const double sc = sc1 * __hiloint2double((1023 - (31 - __clz(d | 1))) << 20, 0);
        double v[3];
#pragma unroll
        for (int q = 0; q < 3; ++q) {
            const double x = c.Q(q, i), start = kind == 1 ? 0.0 : c.QC(q, i);
            if (keep) c.QC(q, i) = x;
            const double r = x - sc * dF[q];
            v[q] = kind == 1 ? r : kind == 2 ? 0.75 * start + 0.25 * r : (start + 2.0 * r) / 3.0;
        }
        if (!d) continue;
#pragma unroll
        for (int q = 0; q < 3; ++q) c.Q(q, i) = v[q];
        if (kind < 3) {
            if (e < L.nfin) {
                const double s = speed1(v[0], v[1], v[2], c.I.gamma, nf);
                if (s > fast) fast = s;
            }
            if (!c.I.bc_generic && (i == 0 || i == c.N1)) {
                // the transmissive ghosts of the next stage's input
#pragma unroll
                for (int q = 0; q < 3; ++q)
                    for (int g = 1; g <= kGhost; ++g) c.Q(q, i == 0 ? -g : c.N1 + g) = v[q];
            }
        }
    }
    if (kind < 3) {
        reduce_put(c.wk, kind, 0, fast);
        __syncthreads();
        if (c.I.bc_generic) {
            bc1(c);
            __syncthreads();
        }
    }
}

// RemoveResidue (AWCM_MANAGER_1D.h:135-157): the first np components to 0 at the points [0, N1] off
// mask0; dense: all of them, else those that the step can have left a value at (the start's mask0
// and mask3; before the step the values off its mask0 were zero).  A warp per word.
__device__ void remove_residue1(const Ctx& c, const uint32_t* start, int np, bool dense)
{
    const int lane = threadIdx.x & 31, wp = threadIdx.x >> 5, nwarp = blockDim.x >> 5;
    for (int x0 = wp; x0 < c.nw; x0 += 32 * nwarp) {
        const int xl = x0 + nwarp * lane;
        const uint32_t z =
            xl < c.nw ? c.inside(xl) & ~c.m0[xl] & (dense ? ~0u : start[xl] | c.plane(3)[xl]) : 0u;
        unsigned todo = __ballot_sync(0xffffffffu, z != 0);
        while (todo) {
            const int j = __ffs(todo) - 1;
            todo &= todo - 1;
            const uint32_t zj = __shfl_sync(0xffffffffu, z, j);
            const int i = 32 * (x0 + nwarp * j - 1) + lane;
            if ((zj >> lane) & 1u)
                for (int p = 0; p < np; ++p) c.Q(p, i) = 0;
        }
    }
}

// The CFL step, the three stages and the residue removal after prepare1; L3: the list of mask3.
// dense: values may lie off the start's mask0.
__device__ __forceinline__ void stages1(Inst1& I, const Ctx& c, const List& L3, bool dense)
{
    Work1* wk = c.wk;
    // CFL over mask3 (main_1d_euler.cpp:67-81) and the first stage's LF speed over its finest-level
    // points; beside it the first fill of the ghosts and the first stage's lists
    double mv = 0, a1 = 0;
    bool nf = false;  // a NaN or infinite wave speed in the CFL or LF scans
    bc1(c);
    build_stage_lists(c, 2, 1);
    {
        const uint32_t* f3 = c.fine(3);
        const unsigned n3 = wk->off[32];
        for (unsigned e = threadIdx.x; e < n3; e += blockDim.x) {
            const int i = L3.get(e);
            const double s = speed1(c.Q(0, i), c.Q(1, i), c.Q(2, i), I.gamma, nf);
            if (s > mv) mv = s;  // a NaN speed is flagged and left out
            if (s > a1 && Ctx::bit(f3, i)) a1 = s;
        }
    }
    reduce_put(wk, 0, 0, mv);
    reduce_put(wk, 0, 1, a1);
    __syncthreads();
    mv = reduce_get(wk, 0, 0);
    a1 = reduce_get(wk, 0, 1);
    double dt = I.cfl * I.dx / mv;
    if (I.dt_fixed > 0) dt = I.dt_fixed;
    int do_print = 0;
    if (I.t + dt > I.t_end) {
        dt = I.t_end - I.t;
        do_print = 1;
    }
    double alpha = a1;
#pragma unroll 1
    for (int kind = 1; kind <= 3; ++kind) {
        if (threadIdx.x == 0) I.alpha[kind - 1] = alpha;
        stage1(c, I.scheme, kind, alpha, dt, nf);
        if (kind < 3) alpha = reduce_get(wk, kind, 0);
    }
    remove_residue1(c, c.plane(kPlTemp), 3, dense);
    const bool any_nf = __syncthreads_or(nf);
    if (threadIdx.x == 0) {
        I.dt = dt;
        I.mv = mv;
        I.do_print = do_print;
        for (int k = 0; k < 4; ++k) I.mask_cnt[k] = wk->mask_cnt[k];
        I.upd += wk->mask_cnt[0];
        I.steps += 1;
        I.t += dt;
        I.done = I.t >= I.t_end;
        if (any_nf) {
            // not a valid gas state: the instance stops and reports it (the reference carries
            // the NaN on)
            I.err = kErrNonFinite;
            I.done = 1;
        }
    }
    __syncthreads();
}

// ------------------------------------------------------------------- scalar AWCM (advection)
// The scalar path of Wavelet/main_1d_advect.cpp:48-224: one field q advected with unit speed at a
// fixed dt, on the same masks and levels.  q lives in plane 0 of the instance's field; the stage
// outputs q_2 and q_1 in the first two planes of the stage-start copy.

// Coarse-level derivative of the field with the driver's branch selection (main_1d_advect.cpp:
// 62-83): AWCM_1D::Differentiate and the 4-point DifferentiateAtLeftBoundary (Wavelet/AWCM_1D.h:
// 127-135), the right edge by the left form on the mirrored stencil as the driver calls it.  The
// driver's two 6-argument DifferentiateAtLeftBoundary calls (i == 2 dx_, i + 2 dx_ == i_end) name
// no scalar overload of AWCM_1D (the driver does not compile as shipped); they take the 5-point
// form of the vector counterpart, DifferentiateEulerAtLeftBoundary (AWCM_1D.h:174-185), with the
// identity flux of unit-speed advection.
__device__ double coarse_d1_scalar(const Ctx& c, const double* in, int m, int i, int d)
{
    auto Q = [&](int ii) { return in[place(ii + kGhost, m)]; };
    const int iend = c.N1;
    if (i - 2 * d > 0 && i + 2 * d < iend) return kD1 * (Q(i + d) - Q(i - d)) + kD2 * (Q(i + 2 * d) - Q(i - 2 * d));
    if (i - 2 * d < 0) return kD1 * (Q(i + d) - Q(i - d)) + kD2 * (Q(i + 2 * d) - Q(i - d));
    if (i == 2 * d)
        return kD02 * Q(i - 2 * d) + kD12 * Q(i - d) + kD22 * Q(i) + kD32 * Q(i + d) + kD2 * Q(i + 2 * d);
    if (i + 2 * d > iend) return kD1 * (Q(i - d) - Q(i + d)) + kD2 * (Q(i - 2 * d) - Q(i + d));
    return kD02 * Q(i + 2 * d) + kD12 * Q(i + d) + kD22 * Q(i) + kD32 * Q(i - d) + kD2 * Q(i - 2 * d);
}

// One scalar stage (main_1d_advect.cpp:50-99, :100-155, :164-212) over mask k (kind 1..3 with k =
// 2, 1, 0): the stage output is the stage input off the mask and in - dt (F_r - F_l) / (dx dx_) on
// the finest level, F_r = WENO5::ReconstructRight(in(i-2..i+2)) (WENO.h:101-104; the face i+1/2
// is shared by points i and i+1, which the reference evaluates twice identically), or in - dt /
// (dx dx_) dF below it, with the end points copied into the ghosts.  Only the points of the mask
// and the ghosts are written: the next stage's stencils lie in this stage's mask.
// Kind 2 then combines q_1 = 3/4 q + 1/4 q_1 (after q_1's ghost copies), kind 3 q = 1/3 q + 2/3 q_0.
__device__ __forceinline__ void stage1_scalar(const Ctx& c, int kind, const double* in, int m, double* out, double dt)
{
    auto In = [&](int i) { return in[place(i + kGhost, m)]; };
    const int k = 3 - kind, region = kind == 2 ? 0 : 1;
    const StageLists L = stage_lists(c, k, region);
    if (kind < 3) build_stage_lists(c, k - 1, 1 - region);
    for (int e = threadIdx.x; e < L.nf; e += blockDim.x) {
        const int f = L.faces.get(e);
        c.fl[f + kGhost] = recon_left<kWeno5>(In(f + 2), In(f + 1), In(f), In(f - 1), In(f - 2));
    }
    __syncthreads();
    for (int e = threadIdx.x; e < L.nfin + L.ncrs; e += blockDim.x) {
        const int i = e < L.nfin ? L.fin.get(e) : L.crs.get(e - L.nfin);
        double r = In(i);
        if (e < L.nfin) {
            r = r - dt * (c.fl[i + kGhost] - c.fl[i - 1 + kGhost]) / (c.I.dx * 1);
        } else {
            const int d = coarse_spacing(c, k, i);
            if (d) r = r - dt / (c.I.dx * d) * coarse_d1_scalar(c, in, m, i, d);
        }
        if (kind < 3 && (i == 0 || i == c.N1))
            for (int g = 1; g <= kGhost; ++g) out[(i == 0 ? -g : c.N1 + g) + kGhost] = r;
        if (kind == 1) out[i + kGhost] = r;
        else if (kind == 2) out[i + kGhost] = 0.75 * c.Q(0, i) + 0.25 * r;
        else c.Q(0, i) = kC1_3 * c.Q(0, i) + kD1 * r;
    }
    __syncthreads();
}

// One pass of the scalar driver loop after prepare1: the three stages at dt = dt_fixed (the driver's
// 0.5 dx is the caller's choice) with their combinations, and PostProcess (RemoveResidue on
// mask0).  The ghosts of q itself are never rewritten, as in the driver.
__device__ __forceinline__ void stages1_scalar(Inst1& I, const Ctx& c, bool dense)
{
    Work1* wk = c.wk;
    const double dt = I.dt_fixed;
    build_stage_lists(c, 2, 1);
    __syncthreads();
    double* s2 = c.qc;
    double* s1 = c.qc + c.w;
#pragma unroll 1
    for (int kind = 1; kind <= 3; ++kind)
        stage1_scalar(c, kind, kind == 1 ? c.f.q0 : kind == 2 ? s2 : s1, kind == 1 ? c.f.m0 : 0, kind == 1 ? s2 : s1, dt);
    remove_residue1(c, c.plane(kPlStart), 1, dense);
    if (threadIdx.x == 0) {
        I.dt = dt;
        I.mv = 0;
        I.alpha[0] = I.alpha[1] = I.alpha[2] = 0;
        I.do_print = 0;
        for (int k = 0; k < 4; ++k) I.mask_cnt[k] = wk->mask_cnt[k];
        I.upd += wk->mask_cnt[0];
        I.steps += 1;
        I.t += dt;
        I.done = I.t >= I.t_end;
    }
    __syncthreads();
}

// ------------------------------------------------------------------------------- one instance
// The global buffers of one instance.
struct Buffers1 {
    double *q, *qc, *qt, *fl;
    void* lists;        // 2 regions of list_entries1(w) entries
    uint32_t* planes;   // bit planes of an instance too large for shared memory (else unused)
    uint8_t* mask;
    int8_t* level;
};
__device__ __forceinline__ Ctx make_ctx(const Inst1& I, const Buffers1& g, Work1* wk, const Weights& W)
{
    const int w = I.nx + 2 * kGhost;
    uint32_t* pl = g.planes;
    const int nw = plane_words1(I.nx);
    return Ctx{I, Field1{g.q, g.q + w, g.q + 2 * w, 0, 0}, g.qc, g.qt, g.fl, pl, pl, pl + (size_t)kPlAux * nw, nullptr,
               static_cast<uint8_t*>(g.lists), 0, wk, W, w, I.nx, I.nx - 1, I.maxl, level_bits(I.maxl), nw};
}

// Up to nsteps RK3 steps of instance I (the caller has checked that it is not done), staged into
// shared memory once around them; the steps stop when the instance is done.
// Works on wk->inst (set by the caller, behind a barrier).
__device__ void step_inst(const Buffers1& g, const Weights& W, uint8_t* smem, size_t smem_bytes, Work1* wk, int nsteps)
{
    Inst1& I = wk->inst;
    const bool scalar = I.scheme == kScalarAdvection;
    const int w = I.nx + 2 * kGhost;
    const Layout1 lay = pick_layout(I.nx, I.maxl, smem_bytes, scalar);
    Ctx c = make_ctx(I, g, wk, W);
    uint8_t* p = smem;
    if (lay.tier >= kInPlanes) {
        c.pl = c.m0 = reinterpret_cast<uint32_t*>(p);
        c.aux = c.plane(kPlAux);
        p += plane_bytes1(I.nx, I.maxl);
        double* d = reinterpret_cast<double*>(p);
        p += align16(sizeof(double) * tier_doubles(lay.tier, scalar, w));
        const int np = lay.tier < kInDensity ? 0 : lay.tier == kInDensity || scalar ? 1 : 3, ws = row_doubles(w);
        for (int t = threadIdx.x; t < np * w; t += blockDim.x) d[t / w * ws + place(t % w, kPlaceMask)] = g.q[t];
        if (np) c.f.q0 = d, c.f.m0 = kPlaceMask;
        if (np == 3) c.f.q1 = d + ws, c.f.q2 = d + 2 * ws, c.f.m12 = kPlaceMask;
        d += np * ws;
        if (lay.tier == kInAll) {
            c.qc = d;
            d += (scalar ? 2 : 3) * w;
            if (!scalar) {
                c.qt = d;
                d += 3 * w;
            }
            c.fl = d;
        }
    }
    c.ls = p;
    c.cap = lay.cap;
    if (threadIdx.x < 32) wk->cls[threadIdx.x] = 0;
    load_planes(c, g.mask, g.level);
    __syncthreads();
    // Between steps the field is zero off mask0 (RemoveResidue); a field or masks set from outside
    // need not be, and then the first step removes the residue everywhere.
    bool off = false;
    for (int t = threadIdx.x; t < I.nx; t += blockDim.x)
        if (!Ctx::bit(c.m0, t))
            for (int k = 0; k < (scalar ? 1 : 3); ++k) off |= __double_as_longlong(c.Q(k, t)) != 0;
    bool dense = __syncthreads_or(off);
    for (int s = 0; s < nsteps; ++s) {
        // the step's end (thread 0, then a block barrier) sets done at t_end or on an error
        if (s > 0 && *reinterpret_cast<volatile int*>(&I.done)) break;
        const List L3 = prepare1(c, !scalar);
        if (scalar) stages1_scalar(I, c, dense);
        else stages1(I, c, L3, dense);
        dense = false;
    }
    store_planes(c, g.mask, g.level);
    for (int t = threadIdx.x; t < w; t += blockDim.x) {
        if (c.f.m0) g.q[t] = c.f.q0[place(t, kPlaceMask)];
        if (c.f.m12) {
            g.q[w + t] = c.f.q1[place(t, kPlaceMask)];
            g.q[2 * w + t] = c.f.q2[place(t, kPlaceMask)];
        }
    }
    __syncthreads();
}

// Doubles of the list space and offset of the bit planes behind an instance's 12 planes.
__host__ __device__ __forceinline__ size_t pool_list_doubles(int w) { return 2 * ((size_t)w + 32); }
__host__ __device__ __forceinline__ size_t pool_doubles(int nx, int maxl)
{
    const int w = nx + 2 * kGhost;
    const size_t n = 12 * (size_t)w + pool_list_doubles(w) + (plane_bytes1(nx, maxl) + 7) / 8;
    return (n + 31) & ~(size_t)31;
}
__device__ __forceinline__ Buffers1 pool_buffers(const Inst1& I, const Pool& P)
{
    const size_t w = (size_t)I.nx + 2 * kGhost;
    double* base = P.q + I.q_off;
    uint8_t* mb = P.m + I.m_off;
    return Buffers1{base, base + 3 * w, base + 6 * w, base + 9 * w, base + 12 * w,
                    reinterpret_cast<uint32_t*>(base + 12 * w + pool_list_doubles((int)w)), mb, (int8_t*)(mb + align16(w))};
}

// nsteps RK3 steps of every queued instance (fewer for an instance that reaches t_end).  CTAs pull
// queue slots until the queue is exhausted, and run each instance's steps back to back before
// taking the next: nsteps = 1 is one step of the whole batch (the per-step graph); a large
// nsteps runs every instance to its end in one launch, each CTA independently of the others.
// smem_bytes: the launch's dynamic shared memory.
// What bounds it: the latency of the step's phases on one SM.  Against one point per thread on mask
// bytes, the bit planes and lists took a step of one line from 99 to 94 us (1025 points) and from 555
// to 312 us (15361 points, a line whose bytes and levels did not fit in shared memory), and the
// 32769-point scalar line from 795 to 464 us.  Divisions by shared reciprocals, and 512 threads of
// 128 registers instead of 768 of 80, then took 1025 points to 78 us and 15361 points to 247 us.
// With the closures in a warp's registers and the bank rows permuted: 55, 181 and 395 us.
__global__ void __launch_bounds__(kMaxThreads1, 1) k_step1d(Inst1* insts, int n, const int* __restrict__ order, unsigned* queue, Pool P,
                         unsigned smem_bytes, int nsteps)
{
    extern __shared__ __align__(128) uint8_t smem[];
    __shared__ Work1 wk;
    __shared__ int cur;
    for (;;) {
        if (threadIdx.x == 0) cur = (int)atomicAdd(queue, 1u);
        __syncthreads();
        const int k = cur;
        __syncthreads();
        if (k >= n) break;
        Inst1& I = insts[order[k]];
        if (I.t >= I.t_end || I.err) {
            if (threadIdx.x == 0) I.done = 1;
        } else {
            static_assert(sizeof(Inst1) % 4 == 0, "copied by words");
            constexpr int nword = sizeof(Inst1) / 4;
            uint32_t *gl = reinterpret_cast<uint32_t*>(&I), *sh = reinterpret_cast<uint32_t*>(&wk.inst);
            for (int t = threadIdx.x; t < nword; t += blockDim.x) sh[t] = gl[t];
            __syncthreads();
            step_inst(pool_buffers(wk.inst, P), P.W, smem, smem_bytes, &wk, nsteps);
            for (int t = threadIdx.x; t < nword; t += blockDim.x) gl[t] = sh[t];
        }
        __syncthreads();
    }
}

// Single passes for the C-ABI manager surface (one CTA per instance), on planes in global memory.
constexpr int kPassThreads = 512;
// Points up to which a transform goes without lists (whole calls of the forward transform without / with, the
// host's share of 12 us a call and 20 us of parameters included: 257 points 35 / 37 us, 2049 41 / 43, 4097 46.5 / 46,
// 8193 55 / 52).
constexpr int kShortLine1 = 2100;
// The inverse transform of any mask: unlike in the step the mask need not be closed, so points
// outside it are zeroed in their level's own phase, as in the reference.
// on(i): whether point i is in the mask.
template <class On>
__device__ void iwt_any1(const Ctx& c, On&& on)
{
    for (int lev = 0; lev < c.maxl; ++lev) {
        const int D = c.D(lev), h = D >> 1, nd = c.N1 / D;
        for (int ph = 0; ph < 2; ++ph) {
            for (int a = threadIdx.x; a < (ph ? nd : nd - 1); a += blockDim.x) {
                const int i = ph ? h + a * D : D + a * D;
                double v = 0;
                if (on(i)) {
                    int s, k;
                    if (ph) predict_stencil(i, D, c.N1, s, k);
                    else update_stencil(i, D, c.N1, s, k);
                    v = c.Q(0, i);
                    if (ph) v *= 2;
                    for (int cnt = 0; cnt < 4; ++cnt) {
                        const double x = c.w_(cnt, k) * c.Q(0, s + cnt * D);
                        v = ph ? v + x : v - x;
                    }
                }
                c.Q(0, i) = v;
            }
            __syncthreads();
        }
    }
}
// InterpolateEuler(q, mra, from, to) (Wavelet/WAVELET_1D.h:393-431) for any two masks.
template <class Points>
__device__ __forceinline__ void interp_level1(const Ctx& c, const Points& L, unsigned lo, unsigned hi, int D, const uint32_t* from)
{
    for (unsigned e = lo + threadIdx.x; e < hi; e += blockDim.x) {
        const int i = L.get(e);
        if (Points::kSome && (i < 0 || Ctx::bit(from, i))) continue;
        int s, k;
        predict_stencil(i, D, c.N1, s, k);
        for (int p = 1; p < 3; ++p) {
            double v = 0;
            for (int cnt = 0; cnt < 4; ++cnt) v += c.w_(cnt, k) * c.Q(p, s + cnt * D);
            c.Q(p, i) = v;
        }
    }
    __syncthreads();
}
__device__ void interp_any1(const Ctx& c, const uint32_t* from, const uint32_t* to)
{
    for (int x = threadIdx.x; x < c.nw; x += blockDim.x) c.aux[x] = c.points(to, x) & ~from[x];
    __syncthreads();
    close1(c, c.aux);
    if (c.nx <= kShortLine1) {
        for (int lev = 0; lev < c.maxl; ++lev)
            interp_level1(c, SomePoints{c.aux, c.D(lev) >> 1, c.D(lev)}, 0, c.N1 / c.D(lev), c.D(lev), from);
        return;
    }
    const List L = order_points(c, 0, c.aux, from);
    const unsigned* off = c.wk->off;
    for (int lev = 0; lev < c.maxl; ++lev) interp_level1(c, L, off[lev + 1], off[lev + 2], c.D(lev), from);
}
// Density (or scalar field) to 0 at the interior points outside M (the inverse transform's zeros).
__device__ void zero_off1(const Ctx& c, const uint32_t* M)
{
    for (int i = 1 + (int)threadIdx.x; i < c.N1; i += blockDim.x)
        if (!Ctx::bit(M, i)) c.Q(0, i) = 0;
}

// A single pass converts the planes that it reads and the ones that it writes, no others: a step converts
// all of them once for some twenty passes, a pass alone would spend its time on them.  (With all of them, on
// one CTA, every pass over 32769 points took 420 to 600 us; now 11 to 117.)
struct PassPlanes {
    unsigned in, out;
};
PassPlanes pass_planes(int op, int bit, int level_id)
{
    const unsigned M = 1u << bit;
    switch (op) {
        case 0: case 1: return {M, M};
        case 2: return {M | level_plane(level_id), M};
        case 3: return {M, level_plane(level_id)};
        case 10: return {kAllPlanes, kAllPlanes};
        case 11: return {1u, 1u};
        case 13: return {M | 1u << level_id, 0u};
        default: return {0u, 0u};  // the passes that read or write single bits of the bytes
    }
}
// The conversions of a pass on all SMs.
__global__ void k_planes1d(Inst1* insts, int inst, Pool P, unsigned which, int store)
{
    const Inst1& I = insts[inst];
    const Buffers1 g = pool_buffers(I, P);
    const Ctx c = make_ctx(I, g, nullptr, P.W);
    const int per = blockDim.x >> 5, warp = blockIdx.x * per + (threadIdx.x >> 5), nwarp = gridDim.x * per;
    if (store) store_some<4>(c, g.mask, g.level, which, warp, nwarp);
    else load_some<4>(c, g.mask, g.level, which, warp, nwarp);
}
// in, out: the planes that the launch converts itself.
__global__ void __launch_bounds__(kPassThreads) k_pass1d(Inst1* insts, int inst, Pool P, int op, int bit, int level_id, unsigned in, unsigned out)
{
    __shared__ Work1 wk;
    Inst1& I = insts[inst];
    const Buffers1 g = pool_buffers(I, P);
    Ctx c = make_ctx(I, g, &wk, P.W);
    if (threadIdx.x < 32) wk.cls[threadIdx.x] = 0;
    const int warp = threadIdx.x >> 5, nwarp = kPassThreads / 32;
    if (in && c.nw <= nwarp) load_some<1>(c, g.mask, g.level, in, warp, nwarp);
    else if (in) load_some<4>(c, g.mask, g.level, in, warp, nwarp);
    __syncthreads();
    uint32_t* M = c.mask(bit);  // bit kBitTemp is plane kPlTemp
    auto on = [&](int i) { return (g.mask[i + kGhost] >> bit) & 1u; };
    switch (op) {
        case 0: {  // AddAdjacentZone
            for (int x = threadIdx.x; x < c.nw; x += blockDim.x)
                c.aux[x] = M[x] | zone_word(c, x, [&](int y) { return c.points(M, y); });
            __syncthreads();
            for (int x = threadIdx.x; x < c.nw; x += blockDim.x) M[x] = c.aux[x];
            break;
        }
        case 1: close1(c, M); break;
        case 2: {  // AddPointForDifferentiation
            for (int x = threadIdx.x; x < c.nw; x += blockDim.x) c.aux[x] = c.points(M, x);
            __syncthreads();
            for (int i = threadIdx.x; i <= c.N1; i += blockDim.x) {
                const int lev = c.level(level_id, i), x = (i >> 5) + 1;
                if (!Ctx::bit(c.aux, i) || lev > c.maxl) continue;
                uint32_t own = 0;
                stencil_push(c, M, x, c.maxl - lev, 1u << (i & 31), own);
                if (own) atomicOr(&M[x], own);
            }
            break;
        }
        case 3:
            // a point without any neighbour keeps its level: all ones in the planes keep the byte
            for (int x = threadIdx.x; x < c.nw; x += blockDim.x) {
                c.fine(level_id)[x] = 0;
                for (int b = 0; b < c.nb; ++b) c.slice(level_id, b)[x] = ~0u;
            }
            levels1(c, level_id, M);  // word x by the same thread
            break;
        case 4:
            for (int i = threadIdx.x; i <= c.N1; i += blockDim.x)
                if (!on(i)) c.Q(0, i) = c.Q(1, i) = c.Q(2, i) = 0;
            break;
        case 5:  // BadingBoundary
            if (threadIdx.x < 6) {
                const int t = (int)threadIdx.x, i = t < 3 ? t : c.N1 - (t - 3);
                if (t < 3 || i >= 3) g.mask[i + kGhost] |= (uint8_t)(1u << bit);
            }
            break;
        case 10:
            prepare1(c, I.scheme != kScalarAdvection);
            zero_off1(c, c.plane(3));
            break;
        case 11:
            if (c.nx <= kShortLine1) fwt_short1(c);
            else fwt1(c, order_points(c, 0, c.m0));
            break;
        case 12: iwt_any1(c, on); break;
        case 13: interp_any1(c, M, c.mask(level_id)); break;  // InterpolateEuler(from = bit, to = level_id as a bit)
        case 14: bc1(c); break;
        default: break;
    }
    __syncthreads();
    if (out && c.nw <= nwarp) store_some<1>(c, g.mask, g.level, out, warp, nwarp);
    else if (out) store_some<4>(c, g.mask, g.level, out, warp, nwarp);
    else if (c.m0 != c.plane(0)) {
        // the planes are stored by a launch of their own, which looks for mask0 at its own place
        for (int x = threadIdx.x; x < c.nw; x += blockDim.x) c.plane(0)[x] = c.m0[x];
    }
}

// EULER_EQUATION_1D batch entry points (EULER_EQUATION.h:16-26, 42-47): n states of 3 doubles.
__global__ void k_euler1d_flux(const double* __restrict__ q, double* __restrict__ f, int n, double gamma)
{
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= n) return;
    const double s[3] = {q[3 * t], q[3 * t + 1], q[3 * t + 2]};
    double o[3];
    IeeeDiv dv;
    flux1(dv, s, gamma, o);
    for (int k = 0; k < 3; ++k) f[3 * t + k] = o[k];
}

__global__ void k_euler1d_sr(const double* __restrict__ q, double* __restrict__ out, int n, double gamma)
{
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= n) return;
    const double q0 = q[3 * t], q1 = q[3 * t + 1], q2 = q[3 * t + 2];
    const double u = q1 / q0;
    out[t] = absd(u) + sound1(q0, q1, q2, gamma);
}

}  // namespace

// ====================================================================================== Batch1D
struct Batch1D {
    std::vector<Inst1> host;
    Inst1* d_inst = nullptr;
    int* d_order = nullptr;
    unsigned* d_queue = nullptr;
    double* d_q = nullptr;
    uint8_t* d_m = nullptr;
    size_t q_doubles = 0, m_bytes = 0;
    int max_w = 0;
    Pool P{};
    cudaStream_t stream = nullptr;
    cudaGraphExec_t graph = nullptr;
    int device = 0;
    int block = 256;
    int grid = 0;
    int n = 0;

    ~Batch1D()
    {
        if (graph) cudaGraphExecDestroy(graph);
        if (d_inst) cudaFree(d_inst);
        if (d_order) cudaFree(d_order);
        if (d_queue) cudaFree(d_queue);
        if (d_q) cudaFree(d_q);
        if (d_m) cudaFree(d_m);
        if (stream) cudaStreamDestroy(stream);
    }

    int create(int count, const int* num_levels, const int* nx_coarse, const double* x_min, const double* x_max,
               double gamma, int scheme)
    {
        if (count <= 0 || !num_levels || !nx_coarse || !x_min || !x_max) return kErrArg;
        if (scheme != kWenoZ && scheme != kWeno5 && scheme != kScalarAdvection) return kErrArg;
        AWCM_CUDA_TRY(cudaGetDevice(&device));
        n = count;
        host.assign(n, Inst1{});
        size_t qo = 0, mo = 0;
        for (int k = 0; k < n; ++k) {
            if (num_levels[k] < 2 || num_levels[k] > 20 || nx_coarse[k] < 5) return kErrArg;
            Inst1& I = host[k];
            I.nx = (nx_coarse[k] - 1) * (1 << (num_levels[k] - 1)) + 1;
            I.maxl = num_levels[k] - 1;
            I.scheme = scheme;
            I.x_min = x_min[k];
            I.dx = (x_max[k] - x_min[k]) / (I.nx - 1);
            I.gamma = gamma;
            I.t = 0;
            I.t_end = 0;
            const int w = I.nx + 2 * kGhost;
            max_w = std::max(max_w, w);
            I.q_off = (long long)qo;
            I.m_off = (long long)mo;
            qo += pool_doubles(I.nx, I.maxl);
            mo += align16((size_t)w) + (size_t)4 * w;  // mask bytes, then the levels 16-byte aligned
            mo = (mo + 255) & ~(size_t)255;
        }
        q_doubles = qo;
        m_bytes = mo;
        AWCM_CUDA_TRY(cudaStreamCreateWithFlags(&stream, cudaStreamNonBlocking));
        AWCM_CUDA_TRY(cudaMalloc(&d_inst, sizeof(Inst1) * n));
        AWCM_CUDA_TRY(cudaMalloc(&d_order, sizeof(int) * n));
        AWCM_CUDA_TRY(cudaMalloc(&d_queue, sizeof(unsigned)));
        AWCM_CUDA_TRY(cudaMalloc(&d_q, sizeof(double) * q_doubles));
        AWCM_CUDA_TRY(cudaMalloc(&d_m, m_bytes));
        AWCM_CUDA_TRY(cudaMemsetAsync(d_q, 0, sizeof(double) * q_doubles, stream));
        // AWCM_1D's constructor: mask0 true everywhere incl. ghosts, mask_temp and mask1..mask3
        // false everywhere, levels 0 (Wavelet/AWCM_1D.h:23-34).  Ghost bytes also carry the work
        // bits, which are never read there.
        std::vector<uint8_t> hm(m_bytes, 0);
        for (int k = 0; k < n; ++k) {
            const int w = host[k].nx + 2 * kGhost;
            uint8_t* mk = hm.data() + host[k].m_off;
            for (int a = 0; a < w; ++a) {
                const bool ghost = a < kGhost || a >= w - kGhost;
                mk[a] = ghost ? 0xe1 : 0x01;
            }
        }
        AWCM_CUDA_TRY(cudaMemcpy(d_m, hm.data(), m_bytes, cudaMemcpyHostToDevice));
        // Largest instances first in the queue.
        std::vector<int> order(n);
        std::iota(order.begin(), order.end(), 0);
        std::stable_sort(order.begin(), order.end(), [&](int a, int b) { return host[a].nx > host[b].nx; });
        AWCM_CUDA_TRY(cudaMemcpy(d_order, order.data(), sizeof(int) * n, cudaMemcpyHostToDevice));
        AWCM_CUDA_TRY(upload_inst());
        P.q = d_q;
        P.m = d_m;
        P.W = make_weights();
        return set_launch(kMaxThreads1, 0);
    }

    cudaError_t upload_inst()
    {
        return cudaMemcpy(d_inst, host.data(), sizeof(Inst1) * n, cudaMemcpyHostToDevice);
    }
    cudaError_t download_inst()
    {
        cudaError_t e = cudaStreamSynchronize(stream);
        if (e != cudaSuccess) return e;
        return cudaMemcpy(host.data(), d_inst, sizeof(Inst1) * n, cudaMemcpyDeviceToHost);
    }

    // Dynamic shared memory of the step kernel: what the instance that can use most takes, within the
    // share of the SM's shared memory that each of the CTAs resident on it can have.
    size_t smem_cap = 227 * 1024;
    size_t smem_bytes() const
    {
        size_t b = 0;
        for (const Inst1& I : host)
            b = std::max(b, pick_layout(I.nx, I.maxl, smem_cap, I.scheme == kScalarAdvection).bytes);
        return b;
    }

    // Launch shape: threads per CTA and CTAs per SM (0 = as many as fit).
    size_t smem = 0;
    int set_launch(int threads, int ctas_per_sm)
    {
        if (threads < 64 || threads > 1024 || threads % 32) return kErrArg;
        if (threads > kMaxLaunch1) {
            set_last_error("launch shape exceeds the step kernel's limit of 768 threads", __FILE__, __LINE__);
            return kErrArg;
        }
        cudaFuncAttributes fa{};
        AWCM_CUDA_TRY(cudaFuncGetAttributes(&fa, k_step1d));
        block = std::min(threads, kMaxThreads1);
        int sms = 148, occ = 1, optin = 227 * 1024, per_sm = 228 * 1024;
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device);
        cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, device);
        cudaDeviceGetAttribute(&per_sm, cudaDevAttrMaxSharedMemoryPerMultiprocessor, device);
        // the CTAs that registers and threads allow on an SM, as far as the batch fills them
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, k_step1d, block, 0);
        if (occ < 1) occ = 1;
        if (ctas_per_sm > 0) occ = std::min(occ, ctas_per_sm);
        occ = std::min(occ, (n + sms - 1) / sms);
        // 1 KB of each CTA's shared memory is the system's
        const int stat = (int)fa.sharedSizeBytes;
        smem_cap = (size_t)std::min(optin - stat, per_sm / occ - 1024 - stat) & ~(size_t)15;
        smem = smem_bytes();
        AWCM_CUDA_TRY(allow_dynamic_smem(reinterpret_cast<const void*>(k_step1d), optin - stat));
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, k_step1d, block, smem);
        if (occ < 1) occ = 1;
        if (ctas_per_sm > 0) occ = std::min(occ, ctas_per_sm);
        grid = std::min(n, sms * occ);
        if (graph) cudaGraphExecDestroy(graph);
        graph = nullptr;
        return kOk;
    }

    void enq_step(int nsteps = 1)
    {
        cudaMemsetAsync(d_queue, 0, sizeof(unsigned), stream);
        k_step1d<<<grid, block, smem, stream>>>(d_inst, n, d_order, d_queue, P, (unsigned)smem, nsteps);
    }

    int build_graph()
    {
        if (graph) return kOk;
        cudaGraph_t gr;
        AWCM_CUDA_TRY(cudaStreamBeginCapture(stream, cudaStreamCaptureModeThreadLocal));
        enq_step();
        cudaError_t e = cudaStreamEndCapture(stream, &gr);
        if (e != cudaSuccess) {
            set_last_error(cudaGetErrorString(e), __FILE__, __LINE__);
            return kErrCuda;
        }
        e = cudaGraphInstantiate(&graph, gr, 0);
        cudaGraphDestroy(gr);
        if (e != cudaSuccess) {
            set_last_error(cudaGetErrorString(e), __FILE__, __LINE__);
            return kErrCuda;
        }
        return kOk;
    }

    int set_run(const double* tol, const double* cfl, const double* t, const double* t_end, double dt_fixed)
    {
        AWCM_CUDA_TRY(download_inst());
        for (int k = 0; k < n; ++k) {
            Inst1& I = host[k];
            I.tol = tol[k];
            I.cfl = cfl[k];
            I.t = t[k];
            I.t_end = t_end[k];
            I.dt_fixed = dt_fixed;
            I.err = 0;
            I.done = I.t >= I.t_end;
        }
        AWCM_CUDA_TRY(upload_inst());
        return kOk;
    }

    int steps(int n_steps)
    {
        int rc = build_graph();
        if (rc) return rc;
        for (int s = 0; s < n_steps; ++s) AWCM_CUDA_TRY(cudaGraphLaunch(graph, stream));
        AWCM_CUDA_TRY(cudaGetLastError());
        return kOk;
    }

    // Every unfinished instance to its end time, at most max_steps steps each, in one launch.
    int run(int max_steps)
    {
        enq_step(max_steps);
        AWCM_CUDA_TRY(cudaGetLastError());
        return kOk;
    }

    // Attaches the enum-driven BOUNDARY_MANAGER_1D to instance k: bc = Nx+6 BOUNDARY_CONDITION
    // values in the FIELD_UNIFORM_1D layout (only the six ghost cells are read).
    int set_bc_field(int k, const int* bc)
    {
        const int nx = host[k].nx;
        const int idx[6] = {2, 1, 0, nx + 3, nx + 4, nx + 5};  // ghosts -1, -2, -3, N1+1, N1+2, N1+3
        for (int q = 0; q < 6; ++q)
            if (bc[idx[q]] < -4 || bc[idx[q]] > 0) {
                set_last_error("BOUNDARY_CONDITION values are -4 (SOLID_WALL) .. 0 (FLUID)", __FILE__, __LINE__);
                return kErrArg;
            }
        AWCM_CUDA_TRY(download_inst());
        for (int q = 0; q < 6; ++q) host[k].bcg[q] = (int8_t)bc[idx[q]];
        host[k].bc_generic = 1;
        AWCM_CUDA_TRY(upload_inst());
        return kOk;
    }

    // Threshold of instance k for a single-pass call (the step takes it from set_run).
    int set_tol(int k, double tol)
    {
        AWCM_CUDA_TRY(download_inst());
        host[k].tol = tol;
        AWCM_CUDA_TRY(upload_inst());
        return kOk;
    }

    // Plane words up to which a single pass converts its planes in its own launch: a launch more costs 3 us,
    // a CTA alone converts about 100 words in one.  Whole calls in one launch / with launches of their own:
    // CheckReconstruction of 8193 points 23 / 26 us, of 32769 points 37 / 24; PrepareEuler of 2049 points
    // 87 / 90, of 4097 points 114 / 108, of 32769 points 585 / 415.
    static constexpr int kPassWords = 1500;
    int pass(int inst, int op, int bit, int level_id)
    {
        if (inst < 0 || inst >= n) return kErrArg;
        PassPlanes p = pass_planes(op, bit, level_id), own{};
        const int nw = plane_words1(host[inst].nx);
        if (nw * (__builtin_popcount(p.in) + __builtin_popcount(p.out)) <= kPassWords) std::swap(p, own);
        const int blocks = std::min((nw + 7) / 8, 4 * 148);
        if (p.in) k_planes1d<<<blocks, 256, 0, stream>>>(d_inst, inst, P, p.in, 0);
        k_pass1d<<<1, kPassThreads, 0, stream>>>(d_inst, inst, P, op, bit, level_id, own.in, own.out);
        if (p.out) k_planes1d<<<blocks, 256, 0, stream>>>(d_inst, inst, P, p.out, 1);
        AWCM_CUDA_TRY(cudaGetLastError());
        AWCM_CUDA_TRY(cudaStreamSynchronize(stream));
        return kOk;
    }

    int w_of(int k) const { return host[k].nx + 2 * kGhost; }

    int set_q(int k, const double* aos)
    {
        const int w = w_of(k);
        std::vector<double> soa(3 * (size_t)w);
        for (int a = 0; a < w; ++a)
            for (int p = 0; p < 3; ++p) soa[p * w + a] = aos[a * 3 + p];
        AWCM_CUDA_TRY(cudaMemcpy(d_q + host[k].q_off, soa.data(), sizeof(double) * 3 * w, cudaMemcpyHostToDevice));
        return kOk;
    }

    int get_q(int k, double* aos)
    {
        const int w = w_of(k);
        std::vector<double> soa(3 * (size_t)w);
        AWCM_CUDA_TRY(cudaStreamSynchronize(stream));
        AWCM_CUDA_TRY(cudaMemcpy(soa.data(), d_q + host[k].q_off, sizeof(double) * 3 * w, cudaMemcpyDeviceToHost));
        for (int a = 0; a < w; ++a)
            for (int p = 0; p < 3; ++p) aos[a * 3 + p] = soa[p * w + a];
        return kOk;
    }

    int get_masks(int k, uint8_t* planes)
    {
        const int w = w_of(k);
        std::vector<uint8_t> mb(w);
        AWCM_CUDA_TRY(cudaStreamSynchronize(stream));
        AWCM_CUDA_TRY(cudaMemcpy(mb.data(), d_m + host[k].m_off, w, cudaMemcpyDeviceToHost));
        const int bits[5] = {kBitTemp, 0, 1, 2, 3};
        for (int r = 0; r < 5; ++r)
            for (int a = 0; a < w; ++a) planes[r * w + a] = (mb[a] >> bits[r]) & 1u;
        return kOk;
    }

    int set_masks(int k, const uint8_t* planes)
    {
        const int w = w_of(k);
        std::vector<uint8_t> mb(w);
        const int bits[5] = {kBitTemp, 0, 1, 2, 3};
        for (int a = 0; a < w; ++a) {
            const bool ghost = a < kGhost || a >= w - kGhost;
            unsigned v = ghost ? 0xe0u : 0u;
            for (int r = 0; r < 5; ++r) v |= (unsigned)(planes[r * w + a] != 0) << bits[r];
            mb[a] = (uint8_t)v;
        }
        AWCM_CUDA_TRY(cudaMemcpy(d_m + host[k].m_off, mb.data(), w, cudaMemcpyHostToDevice));
        return kOk;
    }

    int get_levels(int k, int* lv)
    {
        const int w = w_of(k), nx = host[k].nx;
        std::vector<int8_t> l(4 * (size_t)w);
        AWCM_CUDA_TRY(cudaStreamSynchronize(stream));
        AWCM_CUDA_TRY(cudaMemcpy(l.data(), d_m + host[k].m_off + align16((size_t)w), 4 * (size_t)w,
                                 cudaMemcpyDeviceToHost));
        for (int r = 0; r < 4; ++r)
            for (int i = 0; i < nx; ++i) lv[r * nx + i] = l[r * w + i + kGhost];
        return kOk;
    }

    int set_levels(int k, const int* lv)
    {
        const int w = w_of(k), nx = host[k].nx;
        std::vector<int8_t> l(4 * (size_t)w, 0);
        for (int r = 0; r < 4; ++r)
            for (int i = 0; i < nx; ++i) l[r * w + i + kGhost] = (int8_t)lv[r * nx + i];
        AWCM_CUDA_TRY(cudaMemcpy(d_m + host[k].m_off + align16((size_t)w), l.data(), 4 * (size_t)w,
                                 cudaMemcpyHostToDevice));
        return kOk;
    }

    // Sod-type states on the cell-centred grid x_min + i dx (SHOCKTUBE::Initialize,
    // Problems/1D/PROBLEM_SHOCKTUBE.h:14-54, with the interface and states as arguments).
    int init_riemann(int k, double x_interface, const double* left, const double* right)
    {
        const Inst1& I = host[k];
        const int w = w_of(k);
        std::vector<double> aos(3 * (size_t)w);
        for (int i = -kGhost; i < I.nx + kGhost; ++i) {
            const double x = I.x_min + I.dx * i;
            const double* s = x <= x_interface ? left : right;
            const double rho = s[0], u = s[1], p = s[2];
            double* o = &aos[3 * (size_t)(i + kGhost)];
            o[0] = rho;
            o[1] = rho * u;
            o[2] = p / (I.gamma - 1) + 0.5 * rho * (u * u);
        }
        return set_q(k, aos.data());
    }
};

// =========================================================================== allocation-free step
// One RK3 step of a single 1D instance whose conserved field and mask/level state live in device
// buffers the caller owns, with every other buffer the step needs -- the stage-start copy of the
// field, the coarse derivatives, the face fluxes and the lists -- placed in the file-scope array
// below or in shared memory instead of memory allocated per instance.  It
// is sized for instances of up to kNoAllocMaxNx points (Jmax 13 with 17 coarse points): 9 planes
// of 8199 doubles and two list regions of 16-bit entries, about 641 KiB,
// which every GPU that loads this library holds until the process exits.
constexpr int kNoAllocThreads = 512;
constexpr int kNoAllocMaxNx = 8193;
constexpr int kNoAllocMaxW = kNoAllocMaxNx + 2 * kGhost;
constexpr size_t kNoAllocLists = (size_t)kNoAllocMaxW + 32;  // 4 (w + 32) entries of 2 bytes
constexpr size_t kNoAllocDoubles = (size_t)9 * kNoAllocMaxW + kNoAllocLists;

static __device__ __align__(256) double g_noalloc_scratch[kNoAllocDoubles];

namespace {

// scratch: the device address of g_noalloc_scratch (resolved on the host once per device).  The
// bit planes of 8193 points (28 KB) are always in shared memory.
__global__ void __launch_bounds__(kNoAllocThreads, 1)
    k_step1d_noalloc(Inst1 param, double* q, uint8_t* state, double* scratch, double* out, Weights W, unsigned smem_bytes)
{
    extern __shared__ __align__(128) uint8_t smem[];
    __shared__ Work1 wk;
    Inst1& I = wk.inst;
    if (threadIdx.x == 0) I = param;
    __syncthreads();
    const int w = param.nx + 2 * kGhost;
    double* qc = scratch;
    const Buffers1 g{q, qc, qc + 3 * w, qc + 6 * w, qc + 9 * w, nullptr, state, (int8_t*)(state + w)};
    if (I.t < I.t_end) {
        step_inst(g, W, smem, smem_bytes, &wk, 1);
    } else if (threadIdx.x == 0) {
        I.done = 1;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        out[0] = I.t;
        out[1] = I.dt;
        out[2] = I.do_print;
        out[3] = I.done;
        out[4] = I.steps;
        for (int k = 0; k < 4; ++k) out[5 + k] = I.mask_cnt[k];
        out[9] = I.mv;
        out[10] = I.alpha[0];
        out[11] = I.alpha[1];
        out[12] = I.alpha[2];
        out[13] = (double)I.upd;
        out[14] = I.err;
        out[15] = 0;
    }
}

// Device address of the scratch array (host code must not use the symbol itself: on the host it is only
// a stand-in for the device copy) and the dynamic shared memory that a launch can take beside the
// kernel's static one (sizeof(Work1) and what the compiler pads it with), allowed and resolved once per
// device.
constexpr int kMaxDevices = 64;
struct NoAlloc {
    double* scratch;
    size_t smem;
};
std::mutex g_noalloc_mu;
NoAlloc g_noalloc[kMaxDevices] = {};

int noalloc_resources(int dev, NoAlloc* out)
{
    if (dev < 0 || dev >= kMaxDevices) return kErrArg;
    std::lock_guard<std::mutex> lock(g_noalloc_mu);
    NoAlloc& N = g_noalloc[dev];
    if (!N.scratch) {
        cudaFuncAttributes fa{};
        int optin = 0;
        AWCM_CUDA_TRY(cudaFuncGetAttributes(&fa, k_step1d_noalloc));
        AWCM_CUDA_TRY(cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev));
        void* p = nullptr;
        const cudaError_t e = cudaGetSymbolAddress(&p, g_noalloc_scratch);
        if (e != cudaSuccess || !p) {
            set_last_error(cudaGetErrorString(e), __FILE__, __LINE__);
            return kErrCuda;
        }
        N.smem = ((size_t)optin - fa.sharedSizeBytes) & ~(size_t)15;
        AWCM_CUDA_TRY(allow_dynamic_smem(reinterpret_cast<const void*>(k_step1d_noalloc), (int)N.smem));
        N.scratch = static_cast<double*>(p);
    }
    *out = N;
    return kOk;
}

}  // namespace

}  // namespace awcm

// ======================================================================================== C-ABI
using awcm::Batch1D;

struct awcm1d_batch_s {
    Batch1D b;
};

extern "C" {

int awcm1d_batch_create(int count, const int* num_levels, const int* nx_coarse, const double* x_min,
                        const double* x_max, double gamma, int scheme, awcm1d_batch_t* out)
{
    if (!out) return awcm::kErrArg;
    *out = nullptr;
    awcm1d_batch_s* h = new (std::nothrow) awcm1d_batch_s();
    if (!h) return awcm::kErrOom;
    const int rc = h->b.create(count, num_levels, nx_coarse, x_min, x_max, gamma, scheme);
    if (rc) {
        delete h;
        return rc;
    }
    *out = h;
    return awcm::kOk;
}

int awcm1d_batch_destroy(awcm1d_batch_t h)
{
    delete h;
    return awcm::kOk;
}

#define AWCM_B(h, k)                                                   \
    if (!(h) || (k) < 0 || (k) >= (h)->b.n) return awcm::kErrArg;     \
    cudaSetDevice((h)->b.device)

int awcm1d_batch_count(awcm1d_batch_t h, int* n)
{
    if (!h || !n) return awcm::kErrArg;
    *n = h->b.n;
    return awcm::kOk;
}
int awcm1d_batch_nx(awcm1d_batch_t h, int k, int* nx)
{
    AWCM_B(h, k);
    if (!nx) return awcm::kErrArg;
    *nx = h->b.host[k].nx;
    return awcm::kOk;
}
int awcm1d_batch_set_q(awcm1d_batch_t h, int k, const double* q)
{
    AWCM_B(h, k);
    return q ? h->b.set_q(k, q) : awcm::kErrArg;
}
int awcm1d_batch_get_q(awcm1d_batch_t h, int k, double* q)
{
    AWCM_B(h, k);
    return q ? h->b.get_q(k, q) : awcm::kErrArg;
}
int awcm1d_batch_get_masks(awcm1d_batch_t h, int k, uint8_t* m)
{
    AWCM_B(h, k);
    return m ? h->b.get_masks(k, m) : awcm::kErrArg;
}
int awcm1d_batch_set_masks(awcm1d_batch_t h, int k, const uint8_t* m)
{
    AWCM_B(h, k);
    return m ? h->b.set_masks(k, m) : awcm::kErrArg;
}
int awcm1d_batch_get_levels(awcm1d_batch_t h, int k, int* lv)
{
    AWCM_B(h, k);
    return lv ? h->b.get_levels(k, lv) : awcm::kErrArg;
}
int awcm1d_batch_set_levels(awcm1d_batch_t h, int k, const int* lv)
{
    AWCM_B(h, k);
    return lv ? h->b.set_levels(k, lv) : awcm::kErrArg;
}
int awcm1d_batch_init_riemann(awcm1d_batch_t h, int k, double x_interface, const double* left3,
                              const double* right3)
{
    AWCM_B(h, k);
    if (!left3 || !right3) return awcm::kErrArg;
    return h->b.init_riemann(k, x_interface, left3, right3);
}
int awcm1d_batch_set_run(awcm1d_batch_t h, const double* tol, const double* cfl, const double* t,
                         const double* t_end, double dt_fixed)
{
    if (!h || !tol || !cfl || !t || !t_end) return awcm::kErrArg;
    cudaSetDevice(h->b.device);
    return h->b.set_run(tol, cfl, t, t_end, dt_fixed);
}
int awcm1d_batch_steps(awcm1d_batch_t h, int n_steps)
{
    if (!h || n_steps < 0) return awcm::kErrArg;
    cudaSetDevice(h->b.device);
    return h->b.steps(n_steps);
}
int awcm1d_batch_run(awcm1d_batch_t h, int max_steps)
{
    if (!h || max_steps < 1) return awcm::kErrArg;
    cudaSetDevice(h->b.device);
    return h->b.run(max_steps);
}
int awcm1d_batch_sync(awcm1d_batch_t h)
{
    if (!h) return awcm::kErrArg;
    AWCM_CUDA_TRY(cudaStreamSynchronize(h->b.stream));
    return awcm::kOk;
}
// out[16]: t, dt, do_print, done, steps, |mask0..3|, max speed, alpha1..3, sum|mask0|, err, 0
int awcm1d_batch_status(awcm1d_batch_t h, int k, double* out)
{
    AWCM_B(h, k);
    if (!out) return awcm::kErrArg;
    AWCM_CUDA_TRY(h->b.download_inst());
    const auto& I = h->b.host[k];
    out[0] = I.t;
    out[1] = I.dt;
    out[2] = I.do_print;
    out[3] = I.done;
    out[4] = I.steps;
    for (int q = 0; q < 4; ++q) out[5 + q] = I.mask_cnt[q];
    out[9] = I.mv;
    out[10] = I.alpha[0];
    out[11] = I.alpha[1];
    out[12] = I.alpha[2];
    out[13] = (double)I.upd;
    out[14] = I.err;
    out[15] = 0;
    if (I.err == awcm::kErrNonFinite) {
        char msg[200];
        std::snprintf(msg, sizeof(msg),
                      "instance %d: non-finite state: a CFL or Lax-Friedrichs wave speed was NaN or infinite in "
                      "the step ending at t = %.17g (NaN/Inf values, negative pressure or density)",
                      k, I.t);
        awcm::set_last_error(msg, __FILE__, __LINE__);
        return I.err;
    }
    return awcm::kOk;
}
int awcm1d_batch_totals(awcm1d_batch_t h, double* out)
{
    if (!h || !out) return awcm::kErrArg;
    cudaSetDevice(h->b.device);
    AWCM_CUDA_TRY(h->b.download_inst());
    double upd = 0, steps = 0, done = 0;
    for (const auto& I : h->b.host) {
        upd += (double)I.upd;
        steps += I.steps;
        done += I.done;
    }
    out[0] = upd;
    out[1] = steps;
    out[2] = done;
    return awcm::kOk;
}
int awcm1d_batch_pass(awcm1d_batch_t h, int k, int op, int mask_id, int level_id)
{
    AWCM_B(h, k);
    const int bit = mask_id >= 0 && mask_id <= 3 ? mask_id : awcm::kBitTemp;
    if (level_id < 0 || level_id > 3) return awcm::kErrArg;
    return h->b.pass(k, op, bit, level_id);
}
static int bit_of_mask(int mask_id) { return mask_id >= 0 && mask_id <= 3 ? mask_id : awcm::kBitTemp; }
static bool mask_id_ok(int mask_id) { return mask_id >= 0 && mask_id <= 4; }

int awcm1d_batch_prepare(awcm1d_batch_t h, int k, double tol)
{
    AWCM_B(h, k);
    const int rc = h->b.set_tol(k, tol);
    return rc ? rc : h->b.pass(k, 10, 0, 0);
}
int awcm1d_batch_fwt(awcm1d_batch_t h, int k, double tol)
{
    AWCM_B(h, k);
    const int rc = h->b.set_tol(k, tol);
    return rc ? rc : h->b.pass(k, 11, 0, 0);
}
int awcm1d_batch_iwt(awcm1d_batch_t h, int k, int mask_id)
{
    AWCM_B(h, k);
    if (!mask_id_ok(mask_id)) return awcm::kErrArg;
    return h->b.pass(k, 12, bit_of_mask(mask_id), 0);
}
int awcm1d_batch_interpolate(awcm1d_batch_t h, int k, int from_id, int to_id)
{
    AWCM_B(h, k);
    if (!mask_id_ok(from_id) || !mask_id_ok(to_id)) return awcm::kErrArg;
    return h->b.pass(k, 13, bit_of_mask(from_id), bit_of_mask(to_id));
}
int awcm1d_batch_manager(awcm1d_batch_t h, int k, int op, int mask_id, int level_id)
{
    AWCM_B(h, k);
    if (op < AWCM_OP_ADD_ADJACENT_ZONE || op > AWCM_OP_BANDING || !mask_id_ok(mask_id) || level_id < 0 ||
        level_id > 3)
        return awcm::kErrArg;
    return h->b.pass(k, op, bit_of_mask(mask_id), level_id);
}
int awcm1d_batch_set_bc_field(awcm1d_batch_t h, int k, const int* bc)
{
    AWCM_B(h, k);
    if (!bc) return awcm::kErrArg;
    return h->b.set_bc_field(k, bc);
}
int awcm1d_batch_apply_bc(awcm1d_batch_t h, int k)
{
    AWCM_B(h, k);
    return h->b.pass(k, 14, 0, 0);
}

int euler1d_flux(const double* q_dev, double* f_dev, int n, double gamma, void* stream)
{
    if (n < 0 || (n && (!q_dev || !f_dev))) return awcm::kErrArg;
    if (!n) return awcm::kOk;
    awcm::k_euler1d_flux<<<(n + 255) / 256, 256, 0, (cudaStream_t)stream>>>(q_dev, f_dev, n, gamma);
    AWCM_CUDA_TRY(cudaGetLastError());
    return awcm::kOk;
}
int euler1d_spectral_radius(const double* q_dev, double* s_dev, int n, double gamma, void* stream)
{
    if (n < 0 || (n && (!q_dev || !s_dev))) return awcm::kErrArg;
    if (!n) return awcm::kOk;
    awcm::k_euler1d_sr<<<(n + 255) / 256, 256, 0, (cudaStream_t)stream>>>(q_dev, s_dev, n, gamma);
    AWCM_CUDA_TRY(cudaGetLastError());
    return awcm::kOk;
}

int awcm1d_batch_set_launch(awcm1d_batch_t h, int threads, int ctas_per_sm)
{
    if (!h) return awcm::kErrArg;
    cudaSetDevice(h->b.device);
    return h->b.set_launch(threads, ctas_per_sm);
}
int awcm1d_batch_stream(awcm1d_batch_t h, void** stream)
{
    if (!h || !stream) return awcm::kErrArg;
    *stream = (void*)h->b.stream;
    return awcm::kOk;
}

int awcm1d_step_noalloc(int num_levels, int nx_coarse, double x_min, double x_max, double gamma, int scheme,
                        double tol, double cfl, double t, double t_end, double* q_dev, uint8_t* state_dev,
                        double* out_dev, void* stream)
{
    using namespace awcm;
    if (num_levels < 2 || num_levels > 20 || nx_coarse < 5 || !q_dev || !state_dev || !out_dev) {
        set_last_error("awcm1d_step_noalloc: bad argument", __FILE__, __LINE__);
        return kErrArg;
    }
    if (scheme != kWenoZ && scheme != kWeno5) {
        set_last_error("awcm1d_step_noalloc: scheme must be 0 (WENO-Z) or 1 (WENO5)", __FILE__, __LINE__);
        return kErrArg;
    }
    const long long nx = (long long)(nx_coarse - 1) * (1LL << (num_levels - 1)) + 1;
    if (nx > kNoAllocMaxNx) {
        char msg[160];
        std::snprintf(msg, sizeof(msg),
                      "awcm1d_step_noalloc: Nx = %lld exceeds the static scratch limit of %d points", nx,
                      kNoAllocMaxNx);
        set_last_error(msg, __FILE__, __LINE__);
        return kErrArg;
    }
    int dev = 0;
    AWCM_CUDA_TRY(cudaGetDevice(&dev));
    NoAlloc N{};
    const int rc = noalloc_resources(dev, &N);
    if (rc) return rc;
    Inst1 I{};
    I.nx = (int)nx;
    I.maxl = num_levels - 1;
    I.scheme = scheme;
    I.x_min = x_min;
    I.dx = (x_max - x_min) / (double)(nx - 1);
    I.gamma = gamma;
    I.tol = tol;
    I.cfl = cfl;
    I.t = t;
    I.t_end = t_end;
    const unsigned smem = (unsigned)pick_layout((int)nx, num_levels - 1, N.smem, false).bytes;
    k_step1d_noalloc<<<1, kNoAllocThreads, smem, (cudaStream_t)stream>>>(I, q_dev, state_dev, N.scratch, out_dev, make_weights(),
                                                                         smem);
    AWCM_CUDA_TRY(cudaGetLastError());
    return kOk;
}

}  // extern "C"
