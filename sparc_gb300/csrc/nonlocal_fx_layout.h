// Shared memory of the fixed-point nonlocal kernel (nonlocal_fx.cuh): one place for the size that a
// launch asks for and the offsets that the kernel uses. Plain C++, so that it also compiles
// without CUDA.
#pragma once

#include <cstddef>

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

// P: a byte pointer (the kernel's shared memory), or std::size_t for the offsets alone
template <typename P>
struct Regions {
    // the tile, [kPts][kPitch] of 8 bytes; alpha digits or projection sums [rows][kLanes] of 8; Chi
    // digits [entries][jp] of 8; an entry's point [entries] of 1; row and item tables [rows], [items]
    // of 16; first entries [items + 1] and warp splits [items][kWarps + 1] of 4
    P tile, al, chi, lps, rows, items, ent0, wsplit, end;
};

// for ranges of at most max_rows projector rows, max_ent entries and max_items items; jp even
template <typename P>
SGPU_HD inline Regions<P> regions(P base, int max_rows, int max_ent, int max_items, int jp)
{
    Regions<P> r;
    r.tile = base;
    r.al = r.tile + 8 * kPts * kPitch;
    r.chi = r.al + 8 * kLanes * max_rows;
    r.lps = r.chi + 8 * max_ent * jp;
    r.rows = r.lps + (max_ent + 15) / 16 * 16;
    r.items = r.rows + 16 * max_rows;
    r.ent0 = r.items + 16 * max_items;
    r.wsplit = r.ent0 + 4 * (max_items + 1);
    r.end = r.wsplit + 4 * max_items * (kWarps + 1);
    return r;
}

// bytes of shared memory for it
inline std::size_t shared_bytes(int max_rows, int max_ent, int max_items, int jp)
{
    return (regions<std::size_t>(0, max_rows, max_ent, max_items, jp).end + 15) / 16 * 16;
}

}  // namespace nlfx
}  // namespace sgpu
