// The storage of a 1D instance: its bit planes and lists, and what of it a step keeps in shared memory.
#pragma once
#include "awcm_common.cuh"

namespace awcm {
namespace {

__host__ __device__ __forceinline__ size_t align16(size_t x) { return (x + 15) & ~(size_t)15; }

// ---------------------------------------------------------------------------------- bit planes
// Planes of an instance, in this order: mask0..mask3, the previous mask0 (mask_temp), two work
// planes, the finest-level points of level0..level3, then the nb slices of level0, of level1, ..
// The bits of a word outside the ghosted line are set in the mask planes: ComputeLevel reads a
// mask as set there, and every other pass ands with the words' valid bits.
enum Plane1 : int { kPlTemp = 4, kPlAux = 5, kPlStart = 6, kPlFine = 7, kPlLevel = 11 };
// Slices of a level value: enough for 0..maxl and one more value, all ones, which stands for a level
// outside that range (only set_levels can put one there; it rests in the bytes and is never used).
__host__ __device__ __forceinline__ int level_bits(int maxl)
{
    int b = 1;
    while ((1 << b) - 1 <= maxl) ++b;
    return b;
}
__host__ __device__ __forceinline__ int plane_words1(int nx) { return ((nx - 1 + kGhost + 32) >> 5) + 1; }
__host__ __device__ __forceinline__ size_t plane_bytes1(int nx, int maxl)
{
    // whole bank rows: the field follows in shared memory
    return (sizeof(uint32_t) * (size_t)(kPlLevel + 4 * level_bits(maxl)) * (size_t)plane_words1(nx) + 127) & ~(size_t)127;
}
// List space: two regions of 2 (w + 32) entries each (a stage's faces and points).
__host__ __device__ __forceinline__ size_t list_entries1(int w) { return 2 * ((size_t)w + 32); }
__host__ __device__ __forceinline__ bool short_lists(int w) { return w <= 0xffff; }
__host__ __device__ __forceinline__ size_t entry_bytes(int w) { return short_lists(w) ? 2 : 4; }

// ------------------------------------------------------------------------------- shared memory
// Doubles a step keeps per point of the line: the conserved planes, and the stage-start copy, the
// coarse derivatives and the face fluxes (one, two, none and one plane in the scalar path).
// What an instance keeps in the CTA's shared memory, the fullest that fits:
//   kInAll: the bit planes, every double above and the lists (lines of up to ~2000 points);
//   kInField: the bit planes, the conserved planes and as much of the lists as fits beside them
//     (an 8193-point tube: 28 KB of planes, 197 KB of field);
//   kInDensity: the bit planes, the density (or the scalar field) and lists;
//   kInPlanes: the bit planes and lists;  kInNone: lists.
enum Tier1 : int { kInNone = 0, kInPlanes = 1, kInDensity = 2, kInField = 3, kInAll = 4 };
struct Layout1 {
    int tier;
    unsigned cap;   // list entries per region
    size_t bytes;   // shared memory it takes
};
// Planes of the field are whole bank rows (16 doubles), see place().
constexpr int kPlaceMask = 15;
__host__ __device__ __forceinline__ int row_doubles(int w) { return (w + 15) & ~15; }
__host__ __device__ __forceinline__ size_t tier_doubles(int tier, bool scalar, int w)
{
    const size_t ws = (size_t)row_doubles(w);
    switch (tier) {
        case kInAll: return scalar ? ws + 3 * (size_t)w : 3 * ws + 9 * (size_t)w;
        case kInField: return scalar ? ws : 3 * ws;
        case kInDensity: return ws;
        default: return 0;
    }
}
__host__ __device__ __forceinline__ Layout1 pick_layout(int nx, int maxl, size_t avail, bool scalar)
{
    const int w = nx + 2 * kGhost;
    const size_t full = list_entries1(w), eb = 2 * entry_bytes(w), np = plane_bytes1(nx, maxl);
    // in whole eights like cap, so that the bytes of a layout give that layout again
    const size_t least = full < 512 ? full & ~(size_t)7 : 512;
    for (int tier = kInAll; tier >= kInNone; --tier) {
        const size_t fixed = tier == kInNone ? 0 : np + align16(sizeof(double) * tier_doubles(tier, scalar, w));
        if (tier != kInNone && fixed + eb * least > avail) continue;
        size_t cap = (avail - fixed) / eb;
        cap = cap < full ? cap : full;
        cap &= ~(size_t)7;
        return Layout1{tier, (unsigned)cap, fixed + eb * cap};
    }
    return Layout1{kInNone, 0, 0};
}

}  // namespace
}  // namespace awcm
