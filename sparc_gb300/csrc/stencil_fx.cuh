// FP64 radius-6 stencil in block fixed point (fixed64.cuh): the operation of k_stencil_orth,
//   out = s1 (a Lap + bv diag(v) + c) x + s2 z,
// with the 37-point sum and the potential term in integer arithmetic and two FP64 operations per
// point (the scale s1 and the recurrence term).
//
// A block owns a TX x TY tile of an xy-plane for one column and marches along z; a thread owns
// two x-neighbouring points. Digits of the planes k-6 .. k+8 sit in a register queue (15 slots,
// shifted by two every second plane), digits of the current plane and its halo in one of two
// shared-memory buffers, one barrier per plane. In the step of plane k the block converts plane
// k+1's halo and plane k+7's centre, which the previous step loaded, and loads the next ones; the
// largest exponent of what was loaded goes through the barrier one step ahead, so every thread
// knows before it converts whether the block scale still covers it. A larger value restarts the
// march at that plane with a new scale, the window's largest value, and so does a window without a
// value within 2^-4 of the scale: the scale follows the data along z both ways. (With a scale that
// only grew, a column that falls off into a vacuum was rounded to 2^-57 of its largest value
// everywhere: after 85 planes of exp(-0.35) that is 1e-5 of the values there.) Values that the
// fixed-point range does not cover (infinities, NaN, extreme exponents) send the rest of the slab
// through the FP64 path.
//
// What bounds it: instruction issue (58 % of the slots busy, 53 % of the shared-memory wavefronts,
// HBM 24 %) between barriers at 15 warps per SM. Per point about 36 integer adds, 24 wide
// multiply-adds and 7 high products (60 and 19 with three spacings), 21 instructions per converted
// value (2.5 of them on a 16 x 16 tile) and 40 for the way back, against 42 FP64 instructions at
// two lanes per clock in k_stencil_orth. 96^3, 512 columns: 37.3 -> 5.58 ms per launch (5.44 with
// ties rounded to one side, 5.29 without the lowering of the scale as well, 4.75 with coefficients of
// two digits: all cost a filter its accuracy).
#pragma once

#include <algorithm>
#include <cmath>
#include <type_traits>

#include "fixed64.cuh"
#include "sgpu_internal.h"

namespace sgpu {
namespace {

struct StencilFxParams {
    const double *__restrict__ x;
    double *__restrict__ out;
    const double *__restrict__ z;
    const double *__restrict__ v;
    const int2 *__restrict__ vd;  // digits of the potential (fx_potential)
    long ldx, ldo, ldz;
    int Nx, Ny, Nz, nslab, zlen;
    int TX, TY, hx, hy;      // tile; halo entries of the x sides (12 TY) and of the y sides
    int s;                   // unit of the coefficient digits: 2^-s
    int KW;                  // T 2^(KW + E) is the stencil sum (E the block exponent)
    int dv;                  // the potential's products count 2^-dv of the stencil's
    int c0h, c0l, c0r;       // digits of c0 and of a w_r
    int wh[3][kMaxFDn], wl[3][kMaxFDn], wr[3][kMaxFDn];
    double s2;
    // FP64 path of a block whose values the fixed-point range does not cover
    double c0, bv, s1;
    double w[3][kMaxFDn];
};

constexpr int kFxTile = 32;                        // largest tile edge
constexpr int kFxPitch = kFxTile + 2 * kMaxFDn;    // shared-memory row (points), 8 bytes each
constexpr int kFxThreads = 512;
constexpr int kFxUnroll = 2;                       // planes between two shifts of the queue

// planes k .. ze-1 of a block's tile in FP64, straight from global memory
__device__ __noinline__ void stencil_fx_slow(const StencilFxParams &p, const double *xc,
                                             const double *zc, double *oc, int i0, int j, int k,
                                             int ze)
{
    const long NxNy = (long)p.Nx * p.Ny;
    auto wr = [](int i, int n) { i %= n; return i < 0 ? i + n : i; };
    if (j >= p.Ny) return;
    for (; k < ze; k++) {
        for (int u = 0; u < 2; u++) {
            const int i = i0 + u;
            if (i >= p.Nx) break;
            const long o = i + (long)j * p.Nx + (long)k * NxNy;
            const double xo = xc[o];
            double rx = p.c0 * xo, ry = 0.0, rz = 0.0;
            for (int r = 1; r <= kMaxFDn; r++) {
                const long row = (long)j * p.Nx + (long)k * NxNy;
                rx = fma(xc[row + wr(i - r, p.Nx)] + xc[row + wr(i + r, p.Nx)], p.w[0][r - 1], rx);
                const long cy = i + (long)k * NxNy;
                ry = fma(xc[cy + (long)wr(j - r, p.Ny) * p.Nx] +
                         xc[cy + (long)wr(j + r, p.Ny) * p.Nx], p.w[1][r - 1], ry);
                const long cz = i + (long)j * p.Nx;
                rz = fma(xc[cz + (long)wr(k - r, p.Nz) * NxNy] +
                         xc[cz + (long)wr(k + r, p.Nz) * NxNy], p.w[2][r - 1], rz);
            }
            double res = rx + (ry + rz);
            if (p.v) res += p.bv * (p.v[o] * xo);
            double y = p.s1 * res;
            if (zc) y += p.s2 * zc[o];
            oc[o] = y;
        }
    }
}

// 8-byte load at an unsigned byte offset from a block-uniform base (one 32-bit register)
__device__ __forceinline__ double fx_ld(const double *__restrict__ base, unsigned off)
{
    return __ldg(reinterpret_cast<const double *>(reinterpret_cast<const char *>(base) + off));
}

template <int NS>
struct FxState {
    int4 q[2 * kMaxFDn + 1 + kFxUnroll];  // digits (h0, l0, h1, l1), one slot per plane
    double c0, c1, h[NS];      // loaded ahead: centre of plane k+7, halo of plane k+1
    double z0, z1;             // recurrence term and potential of the current plane
    int2 v0, v1;
    int E, k;
    unsigned pk;               // byte offset of plane k
    unsigned pc;               // byte offset of the next centre plane to load (wrapped)
    bool over;                 // the scale has to change: a value loaded ahead exceeds it, or none is near
};

// A block's scale is lowered when its window holds no value within 2^-kFxNear of it any more. Every
// second plane a thread that has just loaded such a value notes the plane in one of two slots, in
// turn, and all read the slot of two planes before: more than kFxQuiet planes without a note there
// restart the march, with the scale of a window that has left the noted planes behind. (A note of
// every plane, in the steps themselves, took 5.67 ms where this takes 5.44 and none 5.29.)
constexpr unsigned kFxNear = 4;
constexpr int kFxQuiet = 14;

// NS: halo values per thread. CUBE: equal weights in the three directions, so the six neighbours
// at one distance are added before the multiplication (24 wide multiply-adds per point, not 60).
template <int NS, bool CUBE>
__global__ void __launch_bounds__(kFxThreads, 1) k_stencil_fx(const StencilFxParams p)
{
    constexpr int R = kMaxFDn, P = kFxPitch;
    extern __shared__ __align__(16) unsigned char fx_smem[];
    __shared__ unsigned s_key;
    __shared__ int s_near[2];
    const int t = threadIdx.x, nthr = blockDim.x;
    const int TXP = p.TX >> 1;
    const int ty = min(t / TXP, p.TY - 1), tx = t % TXP;
    const bool own = t < TXP * p.TY;               // threads beyond the tile only load halos
    const int bufsz = P * (p.TY + 2 * R);
    int2 *const s0 = reinterpret_cast<int2 *>(fx_smem);
    const int x0 = blockIdx.x * p.TX, y0 = blockIdx.y * p.TY;
    const int col = blockIdx.z / p.nslab, slab = blockIdx.z - col * p.nslab;
    const int zs = slab * p.zlen, ze = min(zs + p.zlen, p.Nz);
    if (zs >= ze) return;
    auto wr = [](int i, int n) { i %= n; return i < 0 ? i + n : i; };
    const int i0 = x0 + 2 * tx, j = y0 + ty;
    const bool act0 = own && i0 < p.Nx && j < p.Ny, act1 = act0 && i0 + 1 < p.Nx;
    const unsigned plane = 8u * (unsigned)p.Nx * (unsigned)p.Ny, column = plane * (unsigned)p.Nz;
    const double *__restrict__ xc = p.x + (long)col * p.ldx;
    const double *__restrict__ zc = p.z ? p.z + (long)col * p.ldz : nullptr;
    double *__restrict__ oc = p.out + (long)col * p.ldo;
    // byte offsets in a plane of the two points
    const unsigned o0 = 8u * (unsigned)(wr(i0, p.Nx) + wr(j, p.Ny) * p.Nx);
    const unsigned o1 = 8u * (unsigned)(wr(i0 + 1, p.Nx) + wr(j, p.Ny) * p.Nx);
    const int sc = (ty + R) * P + R + 2 * tx;      // this thread's first point in a buffer

    // halo entries of this thread: byte offset in the plane, place in the buffer (-1: none)
    unsigned ho[NS];
    int hs[NS];
#pragma unroll
    for (int u = 0; u < NS; u++) {
        const int e = t + u * nthr;
        ho[u] = 0u;
        hs[u] = -1;
        if (e < p.hx) {
            const int row = e / (2 * R), c = e - row * 2 * R;
            const int dx = c < R ? c - R : p.TX + c - R;
            ho[u] = 8u * (unsigned)(wr(x0 + dx, p.Nx) + wr(y0 + row, p.Ny) * p.Nx);
            hs[u] = (row + R) * P + R + dx;
        } else if (e < p.hx + p.hy) {
            const int f = e - p.hx;
            const int row = f / p.TX, c = f - row * p.TX;
            const int dy = row < R ? row - R : p.TY + row - R;
            ho[u] = 8u * (unsigned)(wr(x0 + c, p.Nx) + wr(y0 + dy, p.Ny) * p.Nx);
            hs[u] = (dy + R) * P + R + c;
        }
    }

    FxState<NS> S;
    S.k = zs;
    S.pk = plane * (unsigned)zs;
    auto load_next = [&](unsigned ph) {  // centre of plane S.pc (advanced), halo of plane ph
        S.c0 = fx_ld(xc, S.pc + o0);
        S.c1 = fx_ld(xc, S.pc + o1);
        S.pc += plane;
        if (S.pc == column) S.pc = 0u;
#pragma unroll
        for (int u = 0; u < NS; u++) S.h[u] = fx_ld(xc, ph + ho[u]);
    };
    auto load_v = [&](unsigned pl) {
        if (p.vd) {
            const char *vb = reinterpret_cast<const char *>(p.vd);
            S.v0 = __ldg(reinterpret_cast<const int2 *>(vb + (pl + o0)));
            S.v1 = __ldg(reinterpret_cast<const int2 *>(vb + (pl + o1)));
        }
    };
    auto key_of_loaded = [&]() {
        unsigned key = max(fx::exp_key(S.c0), fx::exp_key(S.c1));
#pragma unroll
        for (int u = 0; u < NS; u++) key = max(key, fx::exp_key(S.h[u]));
        return key;
    };
    auto put_halo = [&](int2 *buf) {
#pragma unroll
        for (int u = 0; u < NS; u++)
            if (hs[u] >= 0) buf[hs[u]] = fx::to_digits(S.h[u], S.E);
    };

    // one plane; false: the march restarts at plane S.k (or has ended)
    auto step = [&](auto Uc, const int2 *buf, int2 *nb) -> bool {
        constexpr int U = decltype(Uc)::value;
        const unsigned pk = S.pk;
        const bool over = __syncthreads_or(S.over);
        const bool go_on = S.k + 1 < ze && !over;
        const double z0 = S.z0, z1 = S.z1;
        const int2 v0 = S.v0, v1 = S.v1;
        if (go_on) {
            const int2 a = fx::to_digits(S.c0, S.E), b = fx::to_digits(S.c1, S.E);
            S.q[U + 2 * R + 1] = make_int4(a.x, a.y, b.x, b.y);
            if (own) *reinterpret_cast<int4 *>(nb + sc) = S.q[U + R + 1];
            put_halo(nb);
            if (S.k + 2 < ze) load_next(pk + 2 * plane);
            if (zc) {
                const char *zb = reinterpret_cast<const char *>(zc);
                S.z0 = *reinterpret_cast<const double *>(zb + (pk + plane + o0));
                S.z1 = *reinterpret_cast<const double *>(zb + (pk + plane + o1));
            }
            load_v(pk + plane);
        }
        // ---- the 37-point sums of the two points; row window: points -6 .. 7 of the pair, point
        // m of it half m & 1 of L[m / 2]
        const int4 cen = S.q[U + R];
        int4 L[R + 1];
#pragma unroll
        for (int m = 0; m <= R; m++)
            L[m] = m == R / 2 ? cen : *reinterpret_cast<const int4 *>(buf + sc - R + 2 * m);
        auto ph = [&](int m) { return (m & 1) ? L[m >> 1].z : L[m >> 1].x; };
        auto pl = [&](int m) { return (m & 1) ? L[m >> 1].w : L[m >> 1].y; };
        long long hh0 = 0, mid0 = 0, hh1 = 0, mid1 = 0;
        int lo0 = 0, lo1 = 0;
        fx::mac(hh0, mid0, lo0, cen.x, cen.y, p.c0h, p.c0l, p.c0r);
        fx::mac(hh1, mid1, lo1, cen.z, cen.w, p.c0h, p.c0l, p.c0r);
#pragma unroll
        for (int r = 1; r <= R; r++) {
            const int4 a = S.q[U + R - r], b = S.q[U + R + r];
            const int4 c = *reinterpret_cast<const int4 *>(buf + sc - r * P);
            const int4 d = *reinterpret_cast<const int4 *>(buf + sc + r * P);
            const int wh = p.wh[0][r - 1], wl = p.wl[0][r - 1], wr = p.wr[0][r - 1];
            if constexpr (CUBE) {
                fx::mac(hh0, mid0, lo0, a.x + b.x + c.x + d.x + ph(R - r) + ph(R + r),
                        a.y + b.y + c.y + d.y + pl(R - r) + pl(R + r), wh, wl, wr);
                fx::mac(hh1, mid1, lo1, a.z + b.z + c.z + d.z + ph(R + 1 - r) + ph(R + 1 + r),
                        a.w + b.w + c.w + d.w + pl(R + 1 - r) + pl(R + 1 + r), wh, wl, wr);
            } else {
                const int uh = p.wh[1][r - 1], ul = p.wl[1][r - 1], ur = p.wr[1][r - 1];
                const int th = p.wh[2][r - 1], tl = p.wl[2][r - 1], tr = p.wr[2][r - 1];
                fx::mac(hh0, mid0, lo0, a.x + b.x, a.y + b.y, th, tl, tr);
                fx::mac(hh1, mid1, lo1, a.z + b.z, a.w + b.w, th, tl, tr);
                fx::mac(hh0, mid0, lo0, c.x + d.x, c.y + d.y, uh, ul, ur);
                fx::mac(hh1, mid1, lo1, c.z + d.z, c.w + d.w, uh, ul, ur);
                fx::mac(hh0, mid0, lo0, ph(R - r) + ph(R + r), pl(R - r) + pl(R + r), wh, wl, wr);
                fx::mac(hh1, mid1, lo1, ph(R + 1 - r) + ph(R + 1 + r), pl(R + 1 - r) + pl(R + 1 + r),
                        wh, wl, wr);
            }
        }
        long long T0 = fx::total(hh0, mid0, lo0), T1 = fx::total(hh1, mid1, lo1);
        if (p.vd) {
            long long a0 = 0, b0 = 0, a1 = 0, b1 = 0;
            fx::mac(a0, b0, cen.x, cen.y, v0.x, v0.y);
            fx::mac(a1, b1, cen.z, cen.w, v1.x, v1.y);
            // a half, ties up on even steps and down on odd ones
            const long long half = ((1ll << p.dv) >> 1) - (U == 1 && p.dv > 0);
            T0 += (fx::total(a0, b0) + half) >> p.dv;
            T1 += (fx::total(a1, b1) + half) >> p.dv;
        }
        const int K = p.KW + S.E;
        double y0v = fx::to_double(T0, K), y1v = fx::to_double(T1, K);
        if (zc) {
            y0v = fma(p.s1, y0v, p.s2 * z0);
            y1v = fma(p.s1, y1v, p.s2 * z1);
        } else if (p.s1 != 1.0) {
            y0v *= p.s1;
            y1v *= p.s1;
        }
        char *ob = reinterpret_cast<char *>(oc);
        if (act0) *reinterpret_cast<double *>(ob + (pk + o0)) = y0v;
        if (act1) *reinterpret_cast<double *>(ob + (pk + o1)) = y1v;
        // what was loaded in this step against the scale
        S.over = (key_of_loaded() >> 20) > (unsigned)S.E;
        S.k++;
        S.pk = pk + plane;
        return go_on;
    };

    while (S.k < ze) {
        // ---- (re)start at plane k: centres of planes k-6 .. k+6, halo of plane k, scale
        __syncthreads();  // the previous march's readers of the buffers, of s_key and s_near are done
        if (t == 0) s_key = 0u;
        double w0[2 * R + 1], w1[2 * R + 1];
        unsigned key = 0u;
        S.pc = plane * (unsigned)wr(S.k - R, p.Nz);
#pragma unroll
        for (int m = 0; m <= 2 * R; m++) {
            w0[m] = fx_ld(xc, S.pc + o0);
            w1[m] = fx_ld(xc, S.pc + o1);
            S.pc += plane;
            if (S.pc == column) S.pc = 0u;
            key = max(key, max(fx::exp_key(w0[m]), fx::exp_key(w1[m])));
        }
        S.z0 = S.z1 = 0.0;
        if (zc) {
            if (act0) S.z0 = zc[(S.pk + o0) >> 3];
            if (act1) S.z1 = zc[(S.pk + o1) >> 3];
        }
        S.v0 = S.v1 = make_int2(0, 0);
        load_v(S.pk);
        const unsigned pc7 = S.pc;
        load_next(S.pk);  // the halo of plane k (the centre that comes with it is loaded again)
        S.pc = pc7;
        key = __reduce_max_sync(0xffffffffu, max(key, key_of_loaded()));
        __syncthreads();
        if ((t & 31) == 0) atomicMax(&s_key, key);
        __syncthreads();
        const unsigned ke = s_key;
        S.E = (int)(ke >> 20);
        if (S.E >= fx::kMaxExp || (ke != 0u && S.E < fx::kMinExp)) {
            if (own) stencil_fx_slow(p, xc, zc, oc, i0, j, S.k, ze);
            return;
        }
        S.E = max(S.E, fx::kMinExp);
        if (t < 2) s_near[t] = S.E == fx::kMinExp ? 1 << 30 : S.k;
#pragma unroll
        for (int m = 0; m <= 2 * R; m++) {
            const int2 a = fx::to_digits(w0[m], S.E), b = fx::to_digits(w1[m], S.E);
            S.q[m] = make_int4(a.x, a.y, b.x, b.y);
        }
        if (own) *reinterpret_cast<int4 *>(s0 + sc) = S.q[R];
        put_halo(s0);
        S.over = false;
        if (S.k + 1 < ze) {
            load_next(S.pk + plane);
            S.over = (key_of_loaded() >> 20) > (unsigned)S.E;
        }
        while (true) {
            if (!step(std::integral_constant<int, 0>{}, s0, s0 + bufsz)) break;
            if (!step(std::integral_constant<int, 1>{}, s0 + bufsz, s0)) break;
#pragma unroll
            for (int m = 0; m <= 2 * R; m++) S.q[m] = S.q[m + kFxUnroll];
            S.over |= S.k - s_near[((S.k >> 1) & 1) ^ 1] > kFxQuiet;
            if ((key_of_loaded() >> 20) + kFxNear >= (unsigned)S.E) s_near[(S.k >> 1) & 1] = S.k;
        }
    }
}

// ---- host side

// block size of a tile: a thread per point pair, and enough for four halo values per thread
inline int fx_threads(int TX, int TY)
{
    const int halo = 2 * kMaxFDn * (TX + TY);
    return std::max((TX / 2 * TY + 31) / 32 * 32, (halo / 4 + 31) / 32 * 32);
}

// digits of w 2^s = h 2^29 + l + r 2^-30, rounded to nearest
inline void fx_coef(double w, int s, int &h, int &l, int &r)
{
    const double u = std::ldexp(w, s);
    const long long W = std::llrint(u);
    r = (int)std::llrint(std::ldexp(u - (double)W, 30));
    const long long H = (W + (1ll << (fx::kDigit - 1))) >> fx::kDigit;
    h = (int)H;
    l = (int)(W - H * (1ll << fx::kDigit));
}

// Tile edges and z slabs of a launch, by the time that a model of the kernel gives. A plane of a
// resident block costs 2.8 clocks per point and SM, plus 0.17 of a point per halo value
// (measured at 96^3: 16x16 tiles 3.34, 32x16 3.53, 32x32 4.17 clocks per point), a block alone
// on its SM 1.35 and two 1.1 of that (their barriers are exposed), and at least 2700 clocks (the
// latency of one step, from 14^3 and 26^3 launches); a slab starts with the 13 planes of its
// queue, about 5 planes' time.
// Many columns: whole columns in the tiles that pad least; few: enough slabs and small tiles to
// fill the SMs.
inline void fx_plan(int Nx, int Ny, int Nz, int ncol, int nsm, int &TX, int &TY, int &nslab)
{
    double best = 1e300;
    TX = TY = 2;
    nslab = 1;
    for (int ex = 4; ex <= kFxTile; ex += 2) {
        const int nx = (Nx + ex - 1) / ex, tx = 2 * ((Nx + 2 * nx - 1) / (2 * nx));
        if (tx != ex && ex != 4) continue;          // one candidate per tile count
        for (int ey = 4; ey <= kFxTile; ey++) {
            const int ny = (Ny + ey - 1) / ey, ty = (Ny + ny - 1) / ny;
            if (ty != ey && ey != 4) continue;
            const double halo = 2.0 * kMaxFDn * (tx + ty);
            const int thr = fx_threads(tx, ty);
            if (thr > kFxThreads) continue;
            const int fit = std::min(kFxThreads / thr, 8);
            static const double f[4] = {1.35, 1.35, 1.1, 1.04};
            for (int ns = 1; ns <= std::max(1, Nz / 3); ns *= 2) {
                const double nblk = (double)nx * ny * ncol * ns;
                const double waves = std::ceil(nblk / ((double)nsm * fit));
                const double res = std::min<double>(fit, std::ceil(nblk / nsm));
                const double work = res * (2.0 * thr + 0.17 * halo) * (res < 4 ? f[(int)res] : 1.0);
                const double t = waves * (5.0 + (Nz + ns - 1) / ns) * std::max(2700.0, 2.8 * work);
                if (t < 0.999 * best) { best = t; TX = tx; TY = ty; nslab = ns; }
            }
        }
    }
}

// Coefficient digits of a launch; vkey: exponent key of the largest |bv v| (0 without a
// potential). False when the coefficients do not fit: the caller takes the FP64 kernel, 37.3 ms per
// launch at 96^3 x 512 where this form takes 5.58. All terms of a point share one scale, the next
// power of two above the sum S of the coefficients' magnitudes, so a potential of 16 times that or
// more (it would take six bits of the scale from the points where it is small) goes there too,
// with all spins and columns of the launch.
inline bool fx_setup(StencilFxParams &p, int FDn, unsigned vkey)
{
    double S = std::fabs(p.c0);
    for (int d = 0; d < 3; d++)
        for (int r = 0; r < FDn; r++) S += 2.0 * std::fabs(p.w[d][r]);
    // a sum's last unit is 2^(eS + E - 60) biased: at least 2^29 for the smallest S and E taken here
    if (!(S > 1e-50 && S < 1e60) || !(std::fabs(p.s1) < 1e60)) return false;
    p.dv = 0;
    int eS = std::ilogb(S) + 1;                     // S < 2^eS
    const int ev = (int)(vkey >> 20) - 1023;        // |bv v| < 2^(ev + 1)
    if (vkey != 0u) {
        if (ev > eS + 3 || ev < -400) return false;
        eS = std::max(eS, ev + 3);
    }
    const int s = 2 * fx::kDigit + 1 - eS;          // S 2^s < 2^59: digits below 2^30
    p.s = s;
    fx_coef(p.c0, s, p.c0h, p.c0l, p.c0r);
    for (int d = 0; d < 3; d++)
        for (int r = 0; r < FDn; r++)
            fx_coef(p.w[d][r], s, p.wh[d][r], p.wl[d][r], p.wr[d][r]);
    // a potential value is V 2^(ev + 1 - kBits): its products are shifted to the unit 2^-s
    if (vkey != 0u) p.dv = std::min(fx::kBits - 1 - ev - s, 62);
    // T counts 2^(kDigit + kDrop) quanta x units; the quantum is 2^(E - 1023 + 1 - kBits)
    p.KW = fx::kDigit + fx::kDrop - s - 1023 + 1 - fx::kBits;
    return true;
}

// digits of bv v (n values) at the scale of their largest exponent key (*key)
__global__ void k_fx_key(const double *__restrict__ v, double bv, long n, unsigned *key)
{
    unsigned m = 0u;
    for (long i = blockIdx.x * (long)blockDim.x + threadIdx.x; i < n;
         i += (long)gridDim.x * blockDim.x)
        m = max(m, fx::exp_key(bv * v[i]));
    m = __reduce_max_sync(0xffffffffu, m);
    if ((threadIdx.x & 31) == 0) atomicMax(key, m);
}
__global__ void k_fx_digits(const double *__restrict__ v, double bv, long n,
                            const unsigned *__restrict__ key, int2 *__restrict__ out)
{
    const int E = (int)(*key >> 20);
    for (long i = blockIdx.x * (long)blockDim.x + threadIdx.x; i < n;
         i += (long)gridDim.x * blockDim.x)
        out[i] = fx::to_digits(bv * v[i], E);
}

}  // namespace
}  // namespace sgpu
