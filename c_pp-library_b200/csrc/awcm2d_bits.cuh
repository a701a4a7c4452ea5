// The mask bit planes of the 2D path: the passes of the mask and level chain as device functions.  Their
// kernels, and the byte passes that the comments name (ph_...), are in awcm2d.cu.
#pragma once
#include "awcm_b200.h"
#include "awcm2d_types.cuh"

namespace awcm {
namespace {

// u / d by the reciprocal inv = ceil(2^32 / d) (0: by division).  Exact while u (inv d - 2^32) < 2^32.
__device__ __forceinline__ unsigned quotient(unsigned u, unsigned d, unsigned inv)
{
    return inv ? __umulhi(u, inv) : u / d;
}
constexpr unsigned kLaneBits = 0x01010101u;  // bit 0 of each of the four bytes

// A virtual thread range: the first index and the stride.
struct Span {
    unsigned t0, stride;
};

// ---------------------------------------------------------------------------------- mask bit planes
// The mask and level chain of PrepareEuler between the two transforms (banding, AddAdjacentZone,
// CheckReconstruction, ComputeLevel, AddPointForDifferentiation: Wavelet/AWCM_2D.h:114-147) works on bit
// planes, one bit per point: a pass is a few shifts per 32 points, and a point takes what its
// neighbours push on it by reading them, where the byte form issues up to 19 atomics per active
// detail.  A plane has the mask's byte layout (bit (i+3) & 31 of word (i+3) >> 5 of row j+3, pitch / 32
// words a row), so a word is 32 aligned mask bytes.  Bits off the ghosted plane are set: ComputeLevel
// reads a mask as set there.
// live[k]: the points whose level_k byte may differ from 0 (all of them after a write from outside).
struct Bits2 {
    uint32_t* m[4];    // mask0..mask3
    uint32_t* aux;     // mask0 before its adjacent zone
    uint32_t* live[3];
    int nwx;            // words per row
    unsigned nwx_inv;   // ceil(2^32 / nwx) where that divides every word's index exactly, else 0
    int rpw, chunks;    // close_rows_per_warp, warps per row of a longer one
    unsigned chunks_inv;
};

__device__ __forceinline__ uint32_t bshl(uint32_t below, uint32_t cur, int s) { return __funnelshift_l(below, cur, s); }
__device__ __forceinline__ uint32_t bshr(uint32_t cur, uint32_t above, int s) { return __funnelshift_r(cur, above, s); }
// Bits of word x whose column lies in [lo, hi].
__device__ __forceinline__ uint32_t cols_in(int x, int lo, int hi)
{
    const int a = lo + kGhost - 32 * x, b = hi + kGhost - 32 * x;
    if (a > 31 || b < 0 || b < a) return 0u;
    const uint32_t up = b >= 31 ? ~0u : (2u << b) - 1u;
    return a <= 0 ? up : up & (~0u << a);
}
// Bits of word x whose column is a multiple of 2^t, and an odd multiple of it.
__device__ __forceinline__ uint32_t cols_mult(int x, int t)
{
    if (t >= 5) return (x & ((1 << (t - 5)) - 1)) == 0 ? 1u << kGhost : 0u;
    const uint32_t p = t == 0 ? ~0u : t == 1 ? 0x55555555u : t == 2 ? 0x11111111u : t == 3 ? 0x01010101u : 0x00010001u;
    return __funnelshift_l(p, p, kGhost);
}
__device__ __forceinline__ uint32_t cols_odd(int x, int t) { return cols_mult(x, t) & ~cols_mult(x, t + 1); }

// One bit of each byte of 32 mask bytes as a bit word, and back.
__device__ __forceinline__ uint32_t gather_bits(const uint32_t (&v)[8], int bit)
{
    uint32_t r = 0;
#pragma unroll
    for (int q = 0; q < 8; ++q) r |= ((((v[q] >> bit) & kLaneBits) * 0x01020408u) >> 24 & 15u) << (4 * q);
    return r;
}
__device__ __forceinline__ uint32_t spread4(uint32_t bits) { return (bits & 15u) * 0x00204081u & kLaneBits; }
__device__ __forceinline__ void load32(const uint8_t* p, uint32_t (&v)[8])
{
    const uint4 a = reinterpret_cast<const uint4*>(p)[0], b = reinterpret_cast<const uint4*>(p)[1];
    v[0] = a.x, v[1] = a.y, v[2] = a.z, v[3] = a.w, v[4] = b.x, v[5] = b.y, v[6] = b.z, v[7] = b.w;
}

// mask0 of the byte plane with the banding (see ph_band_copy) into aux; the other planes cleared.
__device__ void bits_pack(const Grid2& g, const Bits2& B, const uint8_t* __restrict__ m, Span sp, int done)
{
    const unsigned n = (unsigned)g.rows * (unsigned)B.nwx;
    for (unsigned w = sp.t0; w < n; w += sp.stride) {
        const int r = (int)quotient(w, (unsigned)B.nwx, B.nwx_inv), x = (int)w - r * B.nwx, j = r - kGhost;
        uint32_t v[8];
        load32(m + 32 * (size_t)w, v);
        if (done) return;
        uint32_t b = gather_bits(v, 0);
        if (j >= 0 && j < g.ny) {
            uint32_t inner = j >= 2 && j <= g.ny - 3 ? cols_in(x, 2, g.nx - 3) : 0u;
            if (g.bc_kind == AWCM_BC_WIND_TUNNEL) {
                if (abs(j - g.wt_j) <= 2) inner &= ~cols_in(x, g.wt_i - 2, g.nx - 1);
                if (j <= g.wt_j + 2) inner &= ~cols_in(x, g.wt_i - 2, g.wt_i + 2);
            }
            b |= cols_in(x, 0, g.nx - 1) & ~inner;
        }
        B.aux[w] = b | ~cols_in(x, -kGhost, g.nx - 1 + kGhost);
        B.m[0][w] = B.m[1][w] = B.m[2][w] = B.m[3][w] = 0;
    }
}

// The points `s` of word x of a row, shifted by +-d columns, into the row P (what falls off the row is
// dropped); own: the part in word x itself.
__device__ __forceinline__ void push_cols(uint32_t* P, int nwx, int x, uint32_t s, int d, bool lo, bool hi, uint32_t& own)
{
    if (d < 32) {
        if (hi) {
            own |= s << d;
            const uint32_t up = s >> (32 - d);
            if (up && x + 1 < nwx) atomicOr(&P[x + 1], up);
        }
        if (lo) {
            own |= s >> d;
            const uint32_t dn = s << (32 - d);
            if (dn && x > 0) atomicOr(&P[x - 1], dn);
        }
        return;
    }
    const int o = d >> 5;
    if (hi && x + o < nwx) atomicOr(&P[x + o], s);
    if (lo && x - o >= 0) atomicOr(&P[x - o], s);
}

// AddAdjacentZone (see ph_aaz) of aux into mask0 (clear before).
__device__ void bits_zone(const Grid2& g, const Bits2& B, Span sp, int done)
{
    const int NX = g.nx - 1, NY = g.ny - 1, nwx = B.nwx;
    const unsigned n = (unsigned)g.rows * (unsigned)nwx;
    for (unsigned w = sp.t0; w < n; w += sp.stride) {
        const uint32_t a = B.aux[w];
        if (done) return;
        if (!a) continue;
        const int r = (int)quotient(w, (unsigned)nwx, B.nwx_inv), x = (int)w - r * nwx, j = r - kGhost;
        uint32_t own = a;
        const uint32_t d = j >= 0 && j <= NY ? a & cols_in(x, 0, NX) : 0u;
        if (d) {
            uint32_t *M = B.m[0], *row = M + (size_t)r * nwx;
            auto push = [&](uint32_t s, int t) {
                const int h = 1 << t, q = t ? h >> 1 : 0;
                push_cols(row, nwx, x, s, h, true, true, own);
                atomicOr(&row[x - h * nwx], s);
                atomicOr(&row[x + h * nwx], s);
                if (q) {
                    push_cols(row, nwx, x, s, q, true, true, own);
                    atomicOr(&row[x - q * nwx], s);
                    atomicOr(&row[x + q * nwx], s);
                }
            };
            const int tj = j == 0 ? 64 : __ffs(j) - 1;
            if (j != 0 && j != NY)
                for (int t = 0; t < tj && t < g.maxl; ++t) {
                    const uint32_t s = d & cols_odd(x, t);
                    if (s) push(s, t);
                }
            if (tj < g.maxl) {
                const uint32_t s = d & cols_mult(x, tj) & cols_in(x, 1, NX - 1);
                if (s) push(s, tj);
            }
        }
        atomicOr(&B.m[0][w], own);
    }
}

// CheckReconstruction (AWCM_MANAGER_2D.h:63-158, see ph_cr) of the level of spacing h = 2^t of the plane
// whose row 0 is `base`.  done: nothing is written.  Up to h = 16 it is a gather:
//   an odd row takes, on its even columns, the columns -+h, -+3h of its own d3 points;
//   an even row takes from the odd rows -+h, -+3h their d3 points (marking d1 points there) and d2 points
//   (marking c points), and on its even columns the columns -+h, -+3h of those d3 points and of its own
//   d1 points.
// At the ends the stencil of the first detail h is that of the detail 3h, and likewise at the other end,
// so the first one counts as both.  A warp takes consecutive words of a row (two words of margin on
// either side; short rows several to a warp), so a word's neighbours come by shuffles.  Two words are what
// h = 16 needs: a detail marks the words at -1, 0, +1 and +2 of its own, and the last detail NX - 16, as
// NX - 48, marks NX - 96, two words below its own.
// A row's thread writes points of the row that no other thread of the pass reads, or (d1, d2 points
// set by a d3 point) whose marks lie among those of the d3 point.
// The coarser levels, whose columns are one bit of every (h / 32)-th word, push point by point.
constexpr int kCloseKeep = 28, kCloseLeft = 2;
__host__ __device__ __forceinline__ int close_rows_per_warp(int nwx) { return nwx <= 32 ? 32 / nwx : 1; }
__host__ __device__ __forceinline__ long close_warps(long nr, int nwx)
{
    if (nwx > 32) return nr * ((nwx + kCloseKeep - 1) / kCloseKeep);
    return (nr + close_rows_per_warp(nwx) - 1) / close_rows_per_warp(nwx);
}
__device__ void bits_close_level(const Grid2& g, const Bits2& B, uint32_t* base, int t, Span sp, int done)
{
    const int nwx = B.nwx;
    const int h = 1 << t, NX = g.nx - 1, NY = g.ny - 1;
    if (t >= 5) {
        const unsigned nc = (unsigned)(NX >> t) + 1u, n = ((unsigned)(NY >> t) + 1u) * nc;
        for (unsigned u = sp.t0; u < n; u += sp.stride) {
            const unsigned b = u / nc, a = u - b * nc;
            const bool io = a & 1u, jo = b & 1u;
            const int i = (int)a << t, j = (int)b << t, D = 2 * h;
            if (!io && (!jo || i == 0 || i == NX)) continue;
            if (!jo && (j == 0 || j == NY)) continue;
            if (!((base[(size_t)j * nwx + (i >> 5)] >> kGhost) & 1u) || done) continue;
            auto put = [&](int ii, int jj) { atomicOr(&base[(size_t)jj * nwx + (ii >> 5)], 1u << kGhost); };
            int is = 0, js = 0, k;
            if (io) predict_stencil(i, D, NX, is, k);
            if (jo) predict_stencil(j, D, NY, js, k);
            for (int c = 0; c < 4; ++c) {
                if (io) put(is + c * D, j);
                if (jo) put(i, js + c * D);
                if (io && jo)
                    for (int e = 0; e < 4; ++e) put(is + c * D, js + e * D);
            }
        }
        return;
    }
    const int nr = (NY >> t) + 1, lane = threadIdx.x & 31;
    const int lane_row = nwx <= 32 ? (lane * (65536 / nwx + 1)) >> 16 : 0;  // lane / nwx
    const int fa = h + kGhost, fb = 3 * h + kGhost, la = NX - h + kGhost;
    const unsigned n = nwx > 32 ? (unsigned)nr * (unsigned)B.chunks : (unsigned)((nr + B.rpw - 1) / B.rpw);
    for (unsigned it = sp.t0 >> 5; it < n; it += sp.stride >> 5) {
        int rr, x;
        bool keep;
        if (nwx <= 32) {
            x = lane - lane_row * nwx;
            rr = (int)it * B.rpw + lane_row;
            keep = lane_row < B.rpw && rr < nr;
        } else {
            rr = (int)quotient(it, (unsigned)B.chunks, B.chunks_inv);
            x = ((int)it - rr * B.chunks) * kCloseKeep - kCloseLeft + lane;
            keep = lane >= kCloseLeft && lane < kCloseLeft + kCloseKeep;
        }
        const bool on = x >= 0 && x < nwx && rr < nr && (nwx > 32 || keep);
        const int j = rr << t;
        const bool odd_row = rr & 1;
        uint32_t* R = base + (size_t)j * nwx + x;
        uint32_t own = 0, v = 0;  // this word; the rows around it (even rows)
        if (on) {
            own = *R;
            if (!odd_row) {
                const long st = (long)h * nwx;
#pragma unroll
                for (int k = -3; k <= 3; k += 2)
                    if (j + k * h > 0 && j + k * h < NY) v |= R[k * st];
                if (j == 6 * h) v |= R[-5 * st];
                if (j == NY - 6 * h) v |= R[5 * st];
            }
        }
        const uint32_t in = on ? cols_in(x, 0, NX) : 0u;
        const bool own_details = odd_row || (j != 0 && j != NY);
        uint32_t d = (v | (own_details ? own : 0u)) & cols_odd(x, t) & in;
        if (t < 4) {
            if (x == 0) d |= ((d >> fa) & 1u) << fb;
        } else {
            const uint32_t p = __shfl_up_sync(0xffffffffu, d, 1);
            if (x == 1) d |= p & (1u << fa);  // fb is bit fa of word 1
        }
        {
            const uint32_t e = x == la >> 5 ? d & (1u << (la & 31)) : 0u;
            uint32_t f = __shfl_down_sync(0xffffffffu, e, 1);
            if (x == nwx - 1) f = 0;
            d |= t < 4 ? bshr(e, f, 2 * h) : f;
        }
        uint32_t l = __shfl_up_sync(0xffffffffu, d, 1), r = __shfl_down_sync(0xffffffffu, d, 1);
        if (x == 0) l = 0;
        if (x == nwx - 1) r = 0;
        uint32_t mark;
        if (t < 4) {
            mark = bshl(l, d, h) | bshr(d, r, h) | bshl(l, d, 3 * h) | bshr(d, r, 3 * h);
        } else {
            // column 32 x' + 16 marks 32 x' - 32, 32 x', +32 and +64
            uint32_t ll = __shfl_up_sync(0xffffffffu, d, 2);
            if (x < 2) ll = 0;
            mark = (ll | l | d | r) >> 16;
        }
        mark &= cols_mult(x, t + 1);
        // the d3 and d2 points around (d2 points do not include the two end columns)
        mark |= v & cols_mult(x, t) & cols_in(x, 1, NX - 1);
        mark &= in;
        if (keep && on && (mark & ~own) && !done) *R = own | mark;
    }
}

// Word x of row r of M, everything off the plane set.
__device__ __forceinline__ uint32_t padded2(const Grid2& g, const uint32_t* M, int nwx, int r, int x)
{
    return r < 0 || r >= g.rows || x < 0 || x >= nwx ? ~0u : M[(size_t)r * nwx + x];
}

// ComputeLevel(level_{k-1}, mask_{k-1}), mask_k = mask_{k-1} and AddPointForDifferentiation(mask_k,
// level_{k-1}) (see ph_cl, ph_apd) into mask_k (clear before).  A distance of the level search is one shift of
// the word's row and a word of two other rows.
// (Fetching the words of four distances ahead of their use was slower: most words end at distance 1.)
__device__ void bits_next(const Grid2& g, const Bits2& B, int8_t* lvl, int k, Span sp, int done)
{
    const int NX = g.nx - 1, NY = g.ny - 1, nwx = B.nwx;
    const uint32_t* A = B.m[k - 1];
    uint32_t* M = B.m[k];
    const unsigned n = (unsigned)g.rows * (unsigned)nwx;
    for (unsigned w = sp.t0; w < n; w += sp.stride) {
        const uint32_t a = A[w], was = B.live[k - 1][w];
        if (done) return;
        if (!(a | was)) continue;
        const int r = (int)quotient(w, (unsigned)nwx, B.nwx_inv), x = (int)w - r * nwx, j = r - kGhost;
        const uint32_t in = j >= 0 && j <= NY ? cols_in(x, 0, NX) : 0u;
        const uint32_t on = a & in;
        uint32_t own = a;
        if (on | (was & in)) {
            uint32_t S[5] = {0, 0, 0, 0, 0};  // the level, bit-sliced
            const uint32_t mid = j >= 1 && j <= NY - 1 ? cols_in(x, 1, NX - 1) : 0u;
            uint32_t* row = M + (size_t)r * nwx;
            // the points `s` of level maxl - e: their levels, and their stencils into mask_k
            auto take = [&](uint32_t s, int e) {
                const int lev = g.maxl - e;
#pragma unroll
                for (int b = 0; b < 5; ++b)
                    if ((lev >> b) & 1) S[b] |= s;
                s &= mid;
                if (!s) return;
                if (e == 0) {
                    own |= (s << 1) | (s << 2) | (s << 3) | (s >> 1) | (s >> 2) | (s >> 3);
                    const uint32_t up = (s >> 31) | (s >> 30) | (s >> 29), dn = (s << 31) | (s << 30) | (s << 29);
                    if (up && x + 1 < nwx) atomicOr(&row[x + 1], up);
                    if (dn && x > 0) atomicOr(&row[x - 1], dn);
#pragma unroll
                    for (int c = 1; c <= 3; ++c) {
                        atomicOr(&row[x - c * nwx], s);
                        atomicOr(&row[x + c * nwx], s);
                    }
                    return;
                }
                const int D = 1 << e;
                const uint32_t left = s & cols_in(x, 0, 2 * D - 1), right = s & ~left & cols_in(x, NX - 2 * D + 1, NX);
                push_cols(row, nwx, x, s, D, true, true, own);
                push_cols(row, nwx, x, s & ~left, 2 * D, true, false, own);
                push_cols(row, nwx, x, s & ~right, 2 * D, false, true, own);
                const int lo = j - 2 * D < 0 ? -1 : -2, hi = lo == -2 && j + 2 * D > NY ? 1 : 2;
                for (int c = lo; c <= hi; ++c) {
                    const int rr = r + c * D;
                    if (c && rr >= 0 && rr < g.rows) atomicOr(&M[(size_t)rr * nwx + x], s);
                }
            };
            uint32_t todo = on;
            if (todo) {
                const uint32_t l = padded2(g, A, nwx, r, x - 1), rt = padded2(g, A, nwx, r, x + 1);
                // most points have a neighbour at distance 1
                const uint32_t got = todo & (padded2(g, A, nwx, r - 1, x) | padded2(g, A, nwx, r + 1, x) | bshl(l, a, 1) | bshr(a, rt, 1));
                todo &= ~got;
                if (got) take(got, 0);
                for (int e = 1; e <= g.maxl && todo; ++e) {
                    const int d = 1 << e;
                    uint32_t near = padded2(g, A, nwx, r - d, x) | padded2(g, A, nwx, r + d, x);
                    if (e < 5) near |= bshl(l, a, d) | bshr(a, rt, d);
                    else near |= padded2(g, A, nwx, r, x - (d >> 5)) | padded2(g, A, nwx, r, x + (d >> 5));
                    const uint32_t hit = todo & near;
                    todo &= ~hit;
                    if (hit) take(hit, e);
                }
            }
            int8_t* lp = lvl + 32 * (size_t)w;
            uint32_t odd = 0;  // the levels of the points without any neighbour stay as they were
            for (uint32_t u = todo; u; u &= u - 1) {
                const int b = __ffs(u) - 1, lev = lp[b];
                if (lev >= 0 && lev <= g.maxl) take(1u << b, g.maxl - lev);
                else odd |= 1u << b;
            }
            uint32_t* lw = reinterpret_cast<uint32_t*>(lp);
            uint32_t lev4[8];
#pragma unroll
            for (int q = 0; q < 8; ++q) {
                lev4[q] = 0;
#pragma unroll
                for (int b = 0; b < 5; ++b)
                    if (S[b]) lev4[q] |= spread4(S[b] >> (4 * q)) << b;
            }
            if (in == ~0u && !odd) {
                reinterpret_cast<uint4*>(lw)[0] = make_uint4(lev4[0], lev4[1], lev4[2], lev4[3]);
                reinterpret_cast<uint4*>(lw)[1] = make_uint4(lev4[4], lev4[5], lev4[6], lev4[7]);
            } else {
#pragma unroll
                for (int q = 0; q < 8; ++q) {
                    const uint32_t keep = ~(spread4((in & ~odd) >> (4 * q)) * 255u);  // ghosts keep theirs too
                    if (keep != ~0u) lw[q] = (lw[q] & keep) | lev4[q];
                }
            }
            B.live[k - 1][w] = on;
        } else if (was) {
            B.live[k - 1][w] = 0;
        }
        if (own) atomicOr(&M[w], own);
    }
}

// The planes mask0..mask3 back into the byte plane (its other bits stay).
__device__ void bits_unpack(const Grid2& g, const Bits2& B, uint8_t* m, Span sp, int done)
{
    const unsigned n = (unsigned)g.rows * (unsigned)B.nwx;
    for (unsigned w = sp.t0; w < n; w += sp.stride) {
        uint32_t v[8], o[8];
        load32(m + 32 * (size_t)w, v);
        const uint32_t b[4] = {B.m[0][w], B.m[1][w], B.m[2][w], B.m[3][w]};
        if (done) return;
        uint32_t diff = 0;
#pragma unroll
        for (int q = 0; q < 8; ++q) {
            o[q] = v[q] & 0xf0f0f0f0u;
#pragma unroll
            for (int k = 0; k < 4; ++k) o[q] |= spread4(b[k] >> (4 * q)) << k;
            diff |= o[q] ^ v[q];
        }
        if (!diff) continue;
        uint4* p = reinterpret_cast<uint4*>(m + 32 * (size_t)w);
        p[0] = make_uint4(o[0], o[1], o[2], o[3]);
        p[1] = make_uint4(o[4], o[5], o[6], o[7]);
    }
}

}  // namespace
}  // namespace awcm
