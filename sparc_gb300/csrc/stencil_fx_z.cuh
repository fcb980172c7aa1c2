// complex128 radius-6 stencil of Bloch columns in block fixed point: the scheme of stencil_fx.cuh (its
// header explains it) with one complex point per thread, the real and imaginary digits side by
// side, and the Bloch factor of a value's unwrapped position applied in FP64 before it becomes
// digits (only to values from outside the cell).
//
// What bounds it: latency at the 15 warps that 128 registers leave (47 % of the issue slots busy, the
// FP64 pipe, which has the output scale, the recurrence term and the factors, 35 %; with the
// factors as selects on every value it was the bound at 75 %, and 2.9 ms). 34^3, 20 blocks of 64
// columns: 12.6 ms per degree in k_stencil_zb<double2>, 2.08 here.
#pragma once

#include "stencil_fx.cuh"

namespace sgpu {
namespace {

struct FxZConst {              // one launch: all its columns
    int Nx, Ny, Nz, nslab, zlen;
    int TX, TY, hx, hy;
    int KW, dv;
    int wh[3][kMaxFDn], wl[3][kMaxFDn], wr[3][kMaxFDn];
    double w[3][kMaxFDn];      // FP64 path
};

struct FxZCol {                // one column
    const double2 *x, *z;
    double2 *out;
    const int2 *vd;            // digits of the potential, or null
    const double *v;
    int c0h, c0l, c0r;
    double c0, s1, s2;
    const double2 *bf;         // e^{i d k_a L_a}, index 3 a + d + 1
};

__device__ __forceinline__ double2 fxz_mul(double2 a, double2 b)
{
    return make_double2(fma(a.x, b.x, -a.y * b.y), fma(a.x, b.y, a.y * b.x));
}

// v times the factor f[i] in the warps where some lane's i is not one, the index of a factor of one.
// A loop, so that the branch stays: a conditional product becomes predicated instructions, which
// hold the FP64 pipe (16 clocks an instruction) also where every lane is off.
__device__ __forceinline__ double2 fxz_turn(double2 v, const double2 *f, int i, int one)
{
    bool turn = i != one;
    while (__any_sync(0xffffffffu, turn)) {
        v = fxz_mul(v, f[i]);
        turn = false;
    }
    return v;
}

// planes k .. ze-1 of a thread's point in FP64, straight from global memory
__device__ __noinline__ void stencil_fxz_slow(const FxZConst &p, const FxZCol &c, int i, int j, int k,
                                              int ze)
{
    const long NxNy = (long)p.Nx * p.Ny;
    if (i >= p.Nx || j >= p.Ny) return;
    const int N[3] = {p.Nx, p.Ny, p.Nz};
    for (; k < ze; k++) {
        const long o = i + (long)j * p.Nx + (long)k * NxNy;
        const double2 xo = c.x[o];
        double2 res = make_double2(c.c0 * xo.x, c.c0 * xo.y);
        for (int a = 0; a < 3; a++)
            for (int r = 1; r <= kMaxFDn; r++) {
                double2 s = make_double2(0.0, 0.0);
                for (int u = -1; u <= 1; u += 2) {
                    int q[3] = {i, j, k};
                    q[a] += u * r;
                    int d = 0;
                    while (q[a] < 0) { q[a] += N[a]; d--; }
                    while (q[a] >= N[a]) { q[a] -= N[a]; d++; }
                    double2 f = make_double2(1.0, 0.0);
                    for (int e = 0; e < (d < 0 ? -d : d); e++)
                        f = fxz_mul(f, c.bf[3 * a + (d < 0 ? 0 : 2)]);
                    const double2 y = c.x[q[0] + (long)q[1] * p.Nx + (long)q[2] * NxNy];
                    const double2 t = d ? fxz_mul(y, f) : y;
                    s.x += t.x;
                    s.y += t.y;
                }
                res.x = fma(s.x, p.w[a][r - 1], res.x);
                res.y = fma(s.y, p.w[a][r - 1], res.y);
            }
        if (c.v) {
            res.x = fma(c.v[o], xo.x, res.x);
            res.y = fma(c.v[o], xo.y, res.y);
        }
        double2 y = make_double2(c.s1 * res.x, c.s1 * res.y);
        if (c.z) {
            y.x = fma(c.s2, c.z[o].x, y.x);
            y.y = fma(c.s2, c.z[o].y, y.y);
        }
        c.out[o] = y;
    }
}

constexpr int kFxZTile = 24;                        // largest tile edge
constexpr int kFxZPitch = kFxZTile + 2 * kMaxFDn;   // shared-memory row (points), 16 bytes each
constexpr int kFxZThreads = 512;

template <int NS, bool CUBE>
__device__ __forceinline__ void stencil_fxz(const FxZConst &p, const FxZCol &c, int slab,
                                            unsigned char *smem)
{
    constexpr int R = kMaxFDn, P = kFxZPitch;
    __shared__ unsigned s_key;
    __shared__ int s_near[2];                       // as in stencil_fx.cuh
    __shared__ double2 s_f[27];                     // factors of the shifts, index 9 dz' + 3 dy' + dx'
    const int t = threadIdx.x, nthr = blockDim.x;
    const int ty = min(t / p.TX, p.TY - 1), tx = t % p.TX;
    const bool own = t < p.TX * p.TY;               // threads beyond the tile only load halos
    const int bufsz = P * (p.TY + 2 * R);
    int4 *const s0 = reinterpret_cast<int4 *>(smem);
    const int x0 = blockIdx.x * p.TX, y0 = blockIdx.y * p.TY;
    const int zs = slab * p.zlen, ze = min(zs + p.zlen, p.Nz);
    if (zs >= ze) return;
    if (t < 27)
        s_f[t] = t == 13 ? make_double2(1.0, 0.0)
                         : fxz_mul(fxz_mul(c.bf[t % 3], c.bf[3 + t / 3 % 3]), c.bf[6 + t / 9]);
    const int i = x0 + tx, j = y0 + ty;
    const bool act = own && i < p.Nx && j < p.Ny;
    const unsigned plane = 16u * (unsigned)p.Nx * (unsigned)p.Ny;
    // unwrapped (x, y) -> byte offset in a plane and the index of its factor (the host has
    // checked that no position is a whole period or more away)
    auto place = [&](int px, int py, int &f) -> unsigned {
        const int dx = px < 0 ? 0 : px >= p.Nx ? 2 : 1, dy = py < 0 ? 0 : py >= p.Ny ? 2 : 1;
        f = 9 + 3 * dy + dx;
        return 16u * (unsigned)(px - (dx - 1) * p.Nx + (py - (dy - 1) * p.Ny) * p.Nx);
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
        if (e < p.hx) {
            // all of the left side, then the right one: most warps hold values of one side, and
            // a warp without values from outside the cell skips the factors
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
    // a factor of one (a zero Bloch component) costs nothing
    auto is_one = [](double2 f) { return f.x == 1.0 && f.y == 0.0; };
    if (is_one(s_f[of])) of = 13;
#pragma unroll
    for (int u = 0; u < NS; u++)
        if (is_one(s_f[hf[u]])) hf[u] = 13;
    const bool turn_z = !is_one(c.bf[8]);
    auto ld = [&](const double2 *base, unsigned off) {
        return __ldg(reinterpret_cast<const double2 *>(reinterpret_cast<const char *>(base) + off));
    };
    int4 q[2 * R + 1 + kFxUnroll];                  // digits (re h, re l, im h, im l), a slot per plane
    double2 cc, h[NS], zz = make_double2(0.0, 0.0);
    int2 vv = make_int2(0, 0);
    int E = fx::kMinExp, k = zs, kc = 0;            // kc: unwrapped plane of the next centre to load
    bool over = false;
    int cf = 13;                                    // factor of the centre loaded ahead
    auto centre = [&](int kk, int &f) {             // this thread's value at unwrapped plane kk
        const int dz = kk < 0 ? 0 : kk >= p.Nz ? 2 : 1;
        f = turn_z ? of + 9 * (dz - 1) : of;
        return ld(c.x, plane * (unsigned)(kk - (dz - 1) * p.Nz) + o);
    };
    auto load_next = [&](int kh) {                  // centre of plane kc (advanced), halo of plane kh
        cc = kc < 2 * p.Nz ? centre(kc, cf) : make_double2(0.0, 0.0);
        kc++;
        const unsigned ph = plane * (unsigned)kh;
#pragma unroll
        for (int u = 0; u < NS; u++) h[u] = ld(c.x, ph + ho[u]);
    };
    auto turn_loaded = [&]() {                      // a step after the loads were issued
        cc = fxz_turn(cc, s_f, cf, 13);
#pragma unroll
        for (int u = 0; u < NS; u++) h[u] = fxz_turn(h[u], s_f, hf[u], 13);
    };
    auto load_vz = [&](int kk) {
        const unsigned pk = plane * (unsigned)kk + o;
        if (c.vd) vv = __ldg(reinterpret_cast<const int2 *>(reinterpret_cast<const char *>(c.vd) + (pk >> 1)));
        if (c.z) zz = *reinterpret_cast<const double2 *>(reinterpret_cast<const char *>(c.z) + pk);
    };
    auto key2 = [](double2 v) { return max(fx::exp_key(v.x), fx::exp_key(v.y)); };
    auto key_of_loaded = [&]() {
        unsigned key = key2(cc);
#pragma unroll
        for (int u = 0; u < NS; u++) key = max(key, key2(h[u]));
        return key;
    };
    auto dig = [&](double2 v) {
        const int2 a = fx::to_digits(v.x, E), b = fx::to_digits(v.y, E);
        return make_int4(a.x, a.y, b.x, b.y);
    };
    auto put_halo = [&](int4 *buf) {
#pragma unroll
        for (int u = 0; u < NS; u++)
            if (hs[u] >= 0) buf[hs[u]] = dig(h[u]);
    };
    auto step = [&](auto Uc, const int4 *buf, int4 *nb) -> bool {
        constexpr int U = decltype(Uc)::value;
        const bool any = __syncthreads_or(over);
        const bool go_on = k + 1 < ze && !any;
        const double2 z = zz;
        const int2 v = vv;
        if (go_on) {
            q[U + 2 * R + 1] = dig(cc);
            if (own) nb[sc] = q[U + R + 1];
            put_halo(nb);
            if (k + 2 < ze) load_next(k + 2);
            load_vz(k + 1);
        }
        const int4 cen = q[U + R];
        long long hr = 0, mr = 0, hi = 0, mi = 0;
        int lr = 0, li = 0;
        fx::mac(hr, mr, lr, cen.x, cen.y, c.c0h, c.c0l, c.c0r);
        fx::mac(hi, mi, li, cen.z, cen.w, c.c0h, c.c0l, c.c0r);
#pragma unroll
        for (int r = 1; r <= R; r++) {
            const int4 a = q[U + R - r], b = q[U + R + r];
            const int4 d = buf[sc - r * P], e = buf[sc + r * P];
            const int4 f = buf[sc - r], g = buf[sc + r];
            const int wh = p.wh[0][r - 1], wl = p.wl[0][r - 1], wr = p.wr[0][r - 1];
            if constexpr (CUBE) {
                fx::mac(hr, mr, lr, a.x + b.x + d.x + e.x + f.x + g.x, a.y + b.y + d.y + e.y + f.y + g.y,
                        wh, wl, wr);
                fx::mac(hi, mi, li, a.z + b.z + d.z + e.z + f.z + g.z, a.w + b.w + d.w + e.w + f.w + g.w,
                        wh, wl, wr);
            } else {
                const int uh = p.wh[1][r - 1], ul = p.wl[1][r - 1], ur = p.wr[1][r - 1];
                const int th = p.wh[2][r - 1], tl = p.wl[2][r - 1], tr = p.wr[2][r - 1];
                fx::mac(hr, mr, lr, a.x + b.x, a.y + b.y, th, tl, tr);
                fx::mac(hi, mi, li, a.z + b.z, a.w + b.w, th, tl, tr);
                fx::mac(hr, mr, lr, d.x + e.x, d.y + e.y, uh, ul, ur);
                fx::mac(hi, mi, li, d.z + e.z, d.w + e.w, uh, ul, ur);
                fx::mac(hr, mr, lr, f.x + g.x, f.y + g.y, wh, wl, wr);
                fx::mac(hi, mi, li, f.z + g.z, f.w + g.w, wh, wl, wr);
            }
        }
        long long Tr = fx::total(hr, mr, lr), Ti = fx::total(hi, mi, li);
        if (c.vd) {
            long long a0 = 0, b0 = 0, a1 = 0, b1 = 0;
            fx::mac(a0, b0, cen.x, cen.y, v.x, v.y);
            fx::mac(a1, b1, cen.z, cen.w, v.x, v.y);
            // a half, ties up on even steps and down on odd ones
            const long long half = ((1ll << p.dv) >> 1) - (U == 1 && p.dv > 0);
            Tr += (fx::total(a0, b0) + half) >> p.dv;
            Ti += (fx::total(a1, b1) + half) >> p.dv;
        }
        const int K = p.KW + E;
        double yr = fx::to_double(Tr, K), yi = fx::to_double(Ti, K);
        yr = fma(c.s1, yr, c.s2 * z.x);  // z is zero without a recurrence term
        yi = fma(c.s1, yi, c.s2 * z.y);
        if (act)
            *reinterpret_cast<double2 *>(reinterpret_cast<char *>(c.out) + (plane * (unsigned)k + o)) =
                make_double2(yr, yi);
        k++;
        if (go_on && k + 1 < ze) turn_loaded();
        over = (key_of_loaded() >> 20) > (unsigned)E;
        return go_on;
    };

    while (k < ze) {
        // ---- (re)start at plane k
        __syncthreads();
        if (t == 0) s_key = 0u;
        double2 w[2 * R + 1];
        unsigned key = 0u;
#pragma unroll
        for (int m = 0; m <= 2 * R; m++) {
            int f;
            w[m] = centre(k - R + m, f);
            w[m] = fxz_turn(w[m], s_f, f, 13);
            key = max(key, key2(w[m]));
        }
        if (act) load_vz(k);
        kc = k + R + 1;
        load_next(k);  // the halo of plane k (the centre that comes with it is loaded again)
        turn_loaded();
        key = __reduce_max_sync(0xffffffffu, max(key, key_of_loaded()));
        __syncthreads();
        if ((t & 31) == 0) atomicMax(&s_key, key);
        __syncthreads();
        const unsigned ke = s_key;
        E = (int)(ke >> 20);
        if (E >= fx::kMaxExp || (ke != 0u && E < fx::kMinExp)) {
            if (own) stencil_fxz_slow(p, c, i, j, k, ze);
            return;
        }
        E = max(E, fx::kMinExp);
        if (t < 2) s_near[t] = E == fx::kMinExp ? 1 << 30 : k;
#pragma unroll
        for (int m = 0; m <= 2 * R; m++) q[m] = dig(w[m]);
        if (own) s0[sc] = q[R];
        put_halo(s0);
        over = false;
        if (k + 1 < ze) {
            kc = k + R + 1;
            load_next(k + 1);
            turn_loaded();
            over = (key_of_loaded() >> 20) > (unsigned)E;
        }
        while (true) {
            if (!step(std::integral_constant<int, 0>{}, s0, s0 + bufsz)) break;
            if (!step(std::integral_constant<int, 1>{}, s0 + bufsz, s0)) break;
#pragma unroll
            for (int m = 0; m <= 2 * R; m++) q[m] = q[m + kFxUnroll];
            over |= k - s_near[((k >> 1) & 1) ^ 1] > kFxQuiet;
            if ((key_of_loaded() >> 20) + kFxNear >= (unsigned)E) s_near[(k >> 1) & 1] = k;
        }
    }
}

// ---- host side

// what fxz_plan weighs: largest tile edge, block and resident threads of an SM; of a step, the
// clocks per thread and per halo value, the factor on them where a thread has more than two
// halo values, the least that they come to, and what is added
struct FxZModel {
    int tile, threads, resident;
    double point, halo, more, least, add;
};
constexpr FxZModel kFxZModel = {kFxZTile, kFxZThreads, 512, 5.6, 0.95, 1.0, 2700.0, 0.0};

inline int fxz_threads(int TX, int TY)
{
    const int halo = 2 * kMaxFDn * (TX + TY);
    return std::max((TX * TY + 31) / 32 * 32, (halo / 4 + 31) / 32 * 32);
}

// Tile and slabs: the model of fx_plan with a complex point in the place of a point pair. False
// when a tile's halo would reach a whole period away (grids under a dozen points a side).
inline bool fxz_plan(const FxZModel &md, int Nx, int Ny, int Nz, long ncol, int nsm, int &TX, int &TY,
                     int &nslab)
{
    double best = 1e300;
    TX = TY = 0;
    for (int ex = 4; ex <= md.tile; ex++) {
        const int nx = (Nx + ex - 1) / ex, tx = (Nx + nx - 1) / nx;
        if ((tx != ex && ex != 4) || nx * tx + kMaxFDn > 2 * Nx) continue;
        for (int ey = 4; ey <= md.tile; ey++) {
            const int ny = (Ny + ey - 1) / ey, ty = (Ny + ny - 1) / ny;
            if ((ty != ey && ey != 4) || ny * ty + kMaxFDn > 2 * Ny) continue;
            const double halo = 2.0 * kMaxFDn * (tx + ty);
            const int thr = fxz_threads(tx, ty);
            if (thr > md.threads) continue;
            const int fit = std::min(md.resident / thr, 8);
            static const double f[4] = {1.35, 1.35, 1.1, 1.04};
            for (int ns = 1; ns <= std::max(1, Nz / 3); ns *= 2) {
                const double nblk = (double)nx * ny * ncol * ns;
                const double waves = std::ceil(nblk / ((double)nsm * fit));
                const double res = std::min<double>(fit, std::ceil(nblk / nsm));
                const double work = res * (md.point * thr + md.halo * halo) *
                                    (res < 4 ? f[(int)res] : 1.0) * (halo > 2 * thr ? md.more : 1.0);
                const double t = waves * (5.0 + (Nz + ns - 1) / ns) * (std::max(md.least, work) + md.add);
                // as good: the wider tile (rows are read along x; 34^3: 17 x 9 tiles take
                // 9 % less than 9 x 17)
                if (t < 0.999 * best || (t < 1.001 * best && tx > TX)) {
                    best = t; TX = tx; TY = ty; nslab = ns;
                }
            }
        }
    }
    return best < 1e299;
}

// the constants of a launch from the real kernel's digits (fx_setup with s1 = 1)
inline void fxz_const(FxZConst &g, const StencilFxParams &d)
{
    g.KW = d.KW;
    g.dv = d.dv;
    for (int a = 0; a < 3; a++)
        for (int r = 0; r < kMaxFDn; r++) {
            g.wh[a][r] = d.wh[a][r];
            g.wl[a][r] = d.wl[a][r];
            g.wr[a][r] = d.wr[a][r];
            g.w[a][r] = d.w[a][r];
        }
}

}  // namespace
}  // namespace sgpu
