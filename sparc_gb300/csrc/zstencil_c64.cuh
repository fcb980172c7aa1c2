// complex64 radius-6 stencil of Bloch columns, one point per thread; included by kpoint.cu.
//
// A block owns a TX x TY tile of an xy-plane for one column and marches along z. A thread keeps
// its point's planes k-6 .. k+6 in registers; the current plane and its halo stand in one of two
// shared buffers, one barrier per plane. In the step of plane k the block stores plane k+1 and
// loads the centre of plane k+8 and the halo of plane k+3; at the end of the step what the step
// before loaded gets its Bloch factor where it comes from outside the cell, in a loop that a warp
// enters only where a lane needs it (as predicated instructions the factors cost every value
// their issue slots; the halo entries of one side lie together, so most warps skip it).
//
// What bounds it: shared memory (65 % of the wavefronts: 24 eight-byte reads per point) and issue
// (56 %) at 24 warps per SM. 34^3, 20 blocks of 64 columns: 0.59 ms per launch; two x-neighbouring
// points per thread fed from a cp.async ring of planes took 0.88, with 132 registers, one block
// of ten warps per SM and twice the instructions per point. Loads one plane ahead instead of
// two: 0.60.
#pragma once

#include <type_traits>

#include "sgpu_internal.h"
#include "zmath.cuh"

namespace sgpu {
namespace {

struct ZTileConst {               // one launch: all its columns
    float wx[kMaxFDn + 1], wy[kMaxFDn + 1], wz[kMaxFDn + 1];
    int Nx, Ny, Nz, nslab, zlen;
    int TX, TY, P, hx, hy;        // tile, shared row length, halo entries of the x and y sides
};
struct ZTileCol {                 // one column
    const float2 *x, *z;
    float2 *out;
    const float *v;
    float c0, s1, s2;
    const double2 *bf;            // e^{i d k_a L_a}, index 3 a + d + 1
};

constexpr int kZTileThreads = 384, kZTileResident = 768;

__device__ __forceinline__ float2 ztile_mul(float2 a, float2 b)
{
    return make_float2(fmaf(a.x, b.x, -a.y * b.y), fmaf(a.x, b.y, a.y * b.x));
}
__device__ __forceinline__ float2 ztile_fma(float2 s, float w, float2 acc)
{
    return __ffma2_rn(s, make_float2(w, w), acc);
}
// v times f[i] in the warps where some lane's i is not 13, the index of a factor of one
__device__ __forceinline__ float2 ztile_turn(float2 v, const float2 *f, int i)
{
    bool turn = i != 13;
    while (__any_sync(0xffffffffu, turn)) {
        const float2 w = ztile_mul(v, f[i]);
        if (turn) v = w;
        turn = false;
    }
    return v;
}

template <int NS>
__device__ __forceinline__ void stencil_c64_tile(const ZTileConst &p, const ZTileCol &c, int slab,
                                                 unsigned char *smem)
{
    constexpr int R = kMaxFDn, UN = 2;
    __shared__ float2 s_f[27];                      // factors of the shifts, index 9 dz' + 3 dy' + dx'
    const int t = threadIdx.x, nthr = blockDim.x, P = p.P;
    const int ty = min(t / p.TX, p.TY - 1), tx = t % p.TX;
    const bool own = t < p.TX * p.TY;               // threads beyond the tile only load halos
    const int bufsz = P * (p.TY + 2 * R);
    float2 *const s0 = reinterpret_cast<float2 *>(smem);
    const int x0 = blockIdx.x * p.TX, y0 = blockIdx.y * p.TY;
    const int zs = slab * p.zlen, ze = min(zs + p.zlen, p.Nz);
    if (zs >= ze) return;
    auto bf = [&](int q) { return make_float2((float)c.bf[q].x, (float)c.bf[q].y); };
    if (t < 27)
        s_f[t] = t == 13 ? make_float2(1.f, 0.f)
                         : ztile_mul(ztile_mul(bf(t % 3), bf(3 + t / 3 % 3)), bf(6 + t / 9));
    const int i = x0 + tx, j = y0 + ty;
    const bool act = own && i < p.Nx && j < p.Ny;
    const unsigned plane = 8u * (unsigned)p.Nx * (unsigned)p.Ny;
    // unwrapped (x, y) -> byte offset in a plane and the index of its factor (the host has
    // checked that no position is a whole period or more away)
    auto place = [&](int px, int py, int &f) -> unsigned {
        const int dx = px < 0 ? 0 : px >= p.Nx ? 2 : 1, dy = py < 0 ? 0 : py >= p.Ny ? 2 : 1;
        f = 9 + 3 * dy + dx;
        return 8u * (unsigned)(px - (dx - 1) * p.Nx + (py - (dy - 1) * p.Ny) * p.Nx);
    };
    int of;
    const unsigned o = place(i, j, of);
    const int sc = (ty + R) * P + R + tx;
    unsigned ho[NS];
    int hs[NS], hf[NS];
#pragma unroll
    for (int u = 0; u < NS; u++) {
        const int e = t + u * nthr;
        ho[u] = 0u;
        hs[u] = -1;
        hf[u] = 13;
        if (e < p.hx) {  // the left side, then the right one
            const int side = e / (R * p.TY), q = e - side * R * p.TY, row = q / R;
            const int dx = q - row * R + (side ? p.TX : -R);
            ho[u] = place(x0 + dx, y0 + row, hf[u]);
            hs[u] = (row + R) * P + R + dx;
        } else if (e < p.hx + p.hy) {
            const int f = e - p.hx;
            const int row = f / p.TX, q = f - row * p.TX;
            const int dy = row < R ? row - R : p.TY + row - R;
            ho[u] = place(x0 + q, y0 + dy, hf[u]);
            hs[u] = (dy + R) * P + R + q;
        }
    }
    __syncthreads();
    auto is_one = [](float2 f) { return f.x == 1.f && f.y == 0.f; };
    if (is_one(s_f[of])) of = 13;
#pragma unroll
    for (int u = 0; u < NS; u++)
        if (is_one(s_f[hf[u]])) hf[u] = 13;
    const bool turn_z = !is_one(bf(8));
    auto ld = [&](unsigned off) {
        return __ldg(reinterpret_cast<const float2 *>(reinterpret_cast<const char *>(c.x) + off));
    };
    float2 q[2 * R + 2 + UN];                       // a slot per plane; the last one loaded ahead
    float2 h0[NS], h1[NS], zz = make_float2(0.f, 0.f);
    float vv = 0.f;
    // this thread's value at unwrapped plane kk, and its factor's index
    auto shift = [&](int kk) { return kk < 0 ? 0 : kk >= p.Nz ? 2 : 1; };
    auto centre = [&](int kk) { return ld(plane * (unsigned)(kk - (shift(kk) - 1) * p.Nz) + o); };
    auto turn_centre = [&](float2 v, int kk) {
        return ztile_turn(v, s_f, turn_z ? of + 9 * (shift(kk) - 1) : of);
    };
    auto load_halo = [&](float2 (&h)[NS], int kk) {
        const unsigned pk = plane * (unsigned)kk;
#pragma unroll
        for (int u = 0; u < NS; u++) h[u] = ld(pk + ho[u]);
    };
    auto turn_halo = [&](float2 (&h)[NS]) {
#pragma unroll
        for (int u = 0; u < NS; u++) h[u] = ztile_turn(h[u], s_f, hf[u]);
    };
    auto put_halo = [&](float2 *buf, const float2 (&h)[NS]) {
#pragma unroll
        for (int u = 0; u < NS; u++)
            if (hs[u] >= 0) buf[hs[u]] = h[u];
    };
    auto load_vz = [&](int kk) {
        const unsigned pk = plane * (unsigned)kk + o;
        if (c.v) vv = __ldg(reinterpret_cast<const float *>(reinterpret_cast<const char *>(c.v) + (pk >> 1)));
        if (c.z) zz = *reinterpret_cast<const float2 *>(reinterpret_cast<const char *>(c.z) + pk);
    };
    int k = zs;
    // hn: halo of plane k+1, reloaded with that of plane k+3; hm: halo of plane k+2, in flight
    auto step = [&](auto Uc, const float2 *buf, float2 *nb, float2 (&hn)[NS], float2 (&hm)[NS]) {
        constexpr int U = decltype(Uc)::value;
        __syncthreads();
        const float2 z = zz;
        const float v = vv;
        if (k + 1 < ze) {
            if (own) nb[sc] = q[U + R + 1];
            put_halo(nb, hn);
            if (k + 2 < ze) q[U + 2 * R + 2] = centre(k + R + 2);
            if (k + 3 < ze) load_halo(hn, k + 3);
            load_vz(k + 1);
        }
        const float2 cen = q[U + R];
        float2 rx = make_float2(c.c0 * cen.x, c.c0 * cen.y);
        float2 ry = make_float2(0.f, 0.f), rz = make_float2(0.f, 0.f);
#pragma unroll
        for (int r = 1; r <= R; r++) {
            rx = ztile_fma(__fadd2_rn(buf[sc - r], buf[sc + r]), p.wx[r], rx);
            ry = ztile_fma(__fadd2_rn(buf[sc - r * P], buf[sc + r * P]), p.wy[r], ry);
            rz = ztile_fma(__fadd2_rn(q[U + R - r], q[U + R + r]), p.wz[r], rz);
        }
        float2 res = __fadd2_rn(rx, __fadd2_rn(ry, rz));
        if (c.v) res = ztile_fma(cen, v, res);
        float2 y = make_float2(c.s1 * res.x, c.s1 * res.y);
        if (c.z) y = ztile_fma(z, c.s2, y);
        if (act)
            *reinterpret_cast<float2 *>(reinterpret_cast<char *>(c.out) + (plane * (unsigned)k + o)) = y;
        if (k + 1 < ze) q[U + 2 * R + 1] = turn_centre(q[U + 2 * R + 1], k + R + 1);
        if (k + 2 < ze) turn_halo(hm);
        k++;
    };
#pragma unroll
    for (int m = 0; m <= 2 * R; m++) q[m] = turn_centre(centre(k - R + m), k - R + m);
    load_vz(k);
    load_halo(h0, k);
    turn_halo(h0);
    if (own) s0[sc] = q[R];
    put_halo(s0, h0);
    if (k + 1 < ze) {
        q[2 * R + 1] = centre(k + R + 1);
        load_halo(h0, k + 1);
        turn_halo(h0);
    }
    if (k + 2 < ze) load_halo(h1, k + 2);
    while (true) {
        step(std::integral_constant<int, 0>{}, s0, s0 + bufsz, h0, h1);
        if (k >= ze) break;
        step(std::integral_constant<int, 1>{}, s0 + bufsz, s0, h1, h0);
        if (k >= ze) break;
#pragma unroll
        for (int m = 0; m <= 2 * R + 1; m++) q[m] = q[m + UN];
    }
}

}  // namespace
}  // namespace sgpu
