// Shared memory of the fixed-point nonlocal kernel (nonlocal_fx.cuh): one place for the size that a
// launch asks for and the offsets that the kernel uses. Plain C++, so that it also compiles
// without CUDA.
#pragma once

#ifdef __CUDACC__
#define SGPU_HD __host__ __device__
#else
#define SGPU_HD
#endif

namespace sgpu {
namespace nlfx {

constexpr int kPts = 128;      // covered points per range at most: 128 products of an item and of
                               // a point's rows fit the 64-bit sums in units of 2^57
constexpr int kLanes = 32;     // real columns per group
constexpr int kWarps = 8;
constexpr int kPitch = kLanes + 1;  // tile row, 8-byte elements

struct Layout {
    // byte offsets: alpha digits or projection sums [rows][kLanes] of 8 bytes, Chi digits
    // [entries][jp] of 8, an entry's point [entries] of 1, row and item tables [rows], [items] of 16,
    // first entries [items + 1] and warp splits [items][kWarps + 1] of 4. The tile, [kPts][kPitch]
    // of 8, is at 0.
    unsigned al, chi, lps, rows, items, ent0, wsplit, bytes;
};

// for ranges of at most max_rows projector rows, max_ent entries and max_items items
SGPU_HD inline Layout layout(int max_rows, int max_ent, int max_items, int jp)
{
    const unsigned r = max_rows, e = max_ent, i = max_items;
    Layout L{};
    L.al = 8u * kPts * kPitch;
    L.chi = L.al + 8u * kLanes * r;
    L.lps = L.chi + 8u * e * jp;
    L.rows = L.lps + (e + 15) / 16 * 16;
    L.items = L.rows + 16u * r;
    L.ent0 = L.items + 16u * i;
    L.wsplit = L.ent0 + 4u * (i + 1);
    L.bytes = (L.wsplit + 4u * i * (kWarps + 1) + 15) / 16 * 16;
    return L;
}

}  // namespace nlfx
}  // namespace sgpu
