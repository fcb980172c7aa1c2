// FP64 nonlocal projector apply and projection in block fixed point (fixed64.cuh).
//
// Reference: Vnl_vec_mult (src/nlocVecRoutines.c:798-886) and its k-point twin (:889-999).
//
// Both products are small contractions: alpha[row] = dV Gamma sum_points Chi[point][row] x[point]
// and Hx[point] += scale sum_rows Chi[point][row] alpha[row]. In FP64 they were bound by the
// FP64 pipe (two lanes per clock and SM); here the operands are 29-bit digit pairs and the sums
// are exact 64-bit integers (mad.wide.s32, 64 lanes per clock).
//
// Work: a range of at most 128 covered points, compact in space (the order of nonlocal_tc.cu), and
// 32 columns (16 complex ones) per block of eight warps; a lane is a column. The range's entries
// are grouped by atom image into items, by point within an item. Scales: each projector row's
// Chi values share one (fx_er; it is folded into the row's alpha), a column's values over the
// range share one, so no column loses to a larger one.
//   apply    the alpha rows of the items become digits in shared memory; a warp owns a run of the
//            range's points and walks the items, alpha digits in registers, adding each entry's
//            sum into the point's 64-bit accumulator in shared memory; then each accumulator
//            becomes a double and the output element is read, updated and written once
//   project  a warp converts whole columns of the range (largest exponent by warp reduction) into
//            shared memory; the warps share the entries evenly, each lane accumulating its
//            column's MAXJ sums in registers; the warps' integer sums of an item meet in shared
//            memory, and the range's sums go to a partial buffer that k_fx_reduce adds up per
//            projector row in a fixed order (the result does not depend on scheduling)
// With both, the finished output tile is projected for the next filter degree without reading it
// again. Chi digits are read at warp-uniform addresses of shared memory. A column whose values the
// fixed-point range does not cover (infinities, NaN, extreme exponents) sends the block's sums
// through FP64 arithmetic.
//
// What bounds it: the integer multiply pipe (60 % busy; 27 wide multiply-adds per entry, column
// and product of a 9-projector set) at 16 warps per SM; HBM 13 %. Chi digits staged in shared
// memory: read through L1 instead a launch waits for them (11.8 against 7.6 ms). 96^3, 512
// columns, 64 atoms of 9 projectors on 6 Bohr spheres: apply 17.6 + projection 11.0 ms per
// degree in FP64, 7.8 + 0.45 (reduction) ms here; 26^3, 32 columns: 78 + 163 us, 20 + 5 us here.
#pragma once

#include "fixed64.cuh"
#include "nonlocal_fx_layout.h"
#include "sgpu_internal.h"

namespace sgpu {
namespace nlfx {

constexpr int kPtRows = 128;   // projector rows over one point at most
constexpr int kRows = 128;     // projector rows per range (items' rows added up) at most
constexpr int kChiBytes = 32 * 1024;  // Chi digits per range at most (two blocks per SM)
constexpr int kChiBits = 56;   // |Chi digit value| < 2^kChiBits

struct Tables {
    const int *pt0;     // nrange + 1: first point of each range in pts
    const int *pts;     // grid point
    const int *item0;   // nrange + 1: first item of each range
    const int4 *items;  // (row offset in the range, first projector row, count, image)
    const int *ent0;    // nitem + 1: first entry of each item
    const int *wsplit;  // nitem x (kWarps + 1): an item's entries by the warp owning their point
    const unsigned char *lp;  // entry: point of the range
    const int4 *chi;    // entry: jp / 2 pairs of digits (h, l, h, l)
    const int4 *rows;   // row of a range: (alpha row, image, er), |Chi| of the row < 2^er
    const int *row0;    // nrange + 1: first row of each range (rows, partial buffer)
    int jp, max_rows, max_ent, max_items;
};

inline size_t shared_bytes(const Tables &T)
{
    return shared_bytes(T.max_rows, T.max_ent, T.max_items, T.jp);
}

// raw sum in units of 2^57. A product is below 2^113, so 128 of them end below 2^63 units (what an
// intermediate sum wraps, a later one wraps back); mid alone must not wrap: 64 products at most
__device__ __forceinline__ long long sum57(long long hh, long long mid)
{
    return (hh << 1) + ((mid + (1ll << 27)) >> 28);
}

__device__ __forceinline__ double chi_value(int2 c, int er)
{
    return ldexp((double)c.x * 536870912.0 + (double)c.y, er - kChiBits);
}

// Block (range r; column groups g0, g0 + gstep, ..., g0 among them) of x / out (column-major, ld in elements:
// doubles, or complex pairs when CPLX) with ncol columns in all; alpha: projector-major rows of
// lda elements; part: the ranges' projections (dV and Gamma not applied), rows of ldp elements.
// phase (CPLX): cos and sin of each image's phase.
template <bool CPLX, bool APPLY, bool PROJ, int MAXJ>
__device__ __forceinline__ void block(const Tables &T, int r, int g0, int gstep, int ncol,
                                      const double *__restrict__ alpha, double scale,
                                      double *out, const double *__restrict__ x, long ld,
                                      double *__restrict__ part, long lda, long ldp,
                                      const double2 *__restrict__ phase, unsigned char *smem)
{
    constexpr int NC = CPLX ? kLanes / 2 : kLanes;  // columns of a group
    constexpr int W = CPLX ? 2 : 1;                 // doubles per element
    constexpr int CW = NC / kWarps;                 // columns per warp
    constexpr int NV = kPts / 32;                   // points per lane
    constexpr int NA = kRows / kWarps;              // alpha rows per warp
    const int hp = T.jp >> 1;                                    // digit pairs per entry
    const auto R = regions(smem, T.max_rows, T.max_ent, T.max_items, T.jp);
    long long *tile = reinterpret_cast<long long *>(R.tile);     // [kPts][kPitch]
    int2 *al = reinterpret_cast<int2 *>(R.al);                   // [rows][kLanes]
    int4 *chi = reinterpret_cast<int4 *>(R.chi);
    unsigned char *lps = R.lps;
    int4 *rows = reinterpret_cast<int4 *>(R.rows);
    int4 *items = reinterpret_cast<int4 *>(R.items);
    int *ent0 = reinterpret_cast<int *>(R.ent0);
    int *wsplit = reinterpret_cast<int *>(R.wsplit);
    __shared__ unsigned s_key[kLanes];
    __shared__ int s_bad, s_E[kLanes];
    const int t = threadIdx.x, warp = t >> 5, lane = t & 31;
    const int p0 = T.pt0[r], npt = T.pt0[r + 1] - p0;
    const int i0 = T.item0[r], nit = T.item0[r + 1] - i0;
    const int q0 = T.row0[r], nrow = T.row0[r + 1] - q0;
    const int b0 = T.ent0[i0], nent = T.ent0[i0 + nit] - b0;
    const int ngroup = (ncol + NC - 1) / NC;

    // ---- the range's tables and Chi digits
    {
        const int4 *src = T.chi + (long)b0 * hp;
        const unsigned dst = (unsigned)__cvta_generic_to_shared(chi);
        for (int i = t; i < nent * hp; i += 32 * kWarps)
            asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(dst + 16u * i),
                         "l"(src + i)
                         : "memory");
        asm volatile("cp.async.commit_group;\n" ::: "memory");
        for (int i = t; i < nent; i += 32 * kWarps) lps[i] = T.lp[b0 + i];
        for (int i = t; i < nrow; i += 32 * kWarps) rows[i] = T.rows[q0 + i];
        for (int i = t; i < nit; i += 32 * kWarps) items[i] = T.items[i0 + i];
        for (int i = t; i <= nit; i += 32 * kWarps) ent0[i] = T.ent0[i0 + i] - b0;
        for (int i = t; i < nit * (kWarps + 1); i += 32 * kWarps)
            wsplit[i] = T.wsplit[(long)i0 * (kWarps + 1) + i] - b0;
    }
    int gp[NV];  // grid points of this lane
#pragma unroll
    for (int i = 0; i < NV; i++) gp[i] = 32 * i + lane < npt ? T.pts[p0 + 32 * i + lane] : -1;
    const int lo = (int)((long)nent * warp / kWarps), hi = (int)((long)nent * (warp + 1) / kWarps);

    for (int g = g0; g < ngroup; g += gstep) {
        const int n0 = g * NC;
        const int lcol = n0 + (CPLX ? lane >> 1 : lane);  // this lane's column
        const bool lin = lcol < ncol;
        // ---- the tile's elements, in flight until the apply's sums are done: this warp's columns
        double v[CW][NV][W];
#pragma unroll
        for (int c = 0; c < CW; c++) {
            const int n = n0 + warp + kWarps * c;
#pragma unroll
            for (int i = 0; i < NV; i++) {
#pragma unroll
                for (int u = 0; u < W; u++) v[c][i][u] = 0.0;
                if (n < ncol && gp[i] >= 0) {
                    const long o = (long)n * ld + gp[i];
                    if constexpr (CPLX) {
                        const double2 z = APPLY ? reinterpret_cast<const double2 *>(out)[o]
                                                : __ldg(reinterpret_cast<const double2 *>(x) + o);
                        v[c][i][0] = z.x;
                        v[c][i][W - 1] = z.y;
                    } else {
                        v[c][i][0] = APPLY ? out[o] : __ldg(x + o);
                    }
                }
            }
        }
        if (t < kLanes) s_key[t] = 0u;
        if (t == 0) s_bad = 0;
        if (g == g0) asm volatile("cp.async.wait_all;\n" ::: "memory");
        __syncthreads();  // tables staged; the previous group's readers of the tile are done
        // value of row k of the range in this lane's column, as the apply needs it
        auto alpha_at = [&](int k) -> double {
            if (!lin) return 0.0;
            const int4 q = rows[k];
            if constexpr (CPLX) {
                const double2 a =
                    __ldg(reinterpret_cast<const double2 *>(alpha) + (long)q.x * lda + lcol);
                const double2 ph = phase[q.y];  // e^{-i theta} alpha
                return (lane & 1) ? fma(a.y, ph.x, -a.x * ph.y) : fma(a.x, ph.x, a.y * ph.y);
            } else {
                return __ldg(alpha + (long)q.x * lda + lcol);
            }
        };

        if constexpr (APPLY) {
            // ---- alpha rows: column scales, digits; a row's Chi scale moves into it
            double a[NA];
            unsigned key = 0u;
#pragma unroll
            for (int i = 0; i < NA; i++) {
                const int k = warp + kWarps * i;
                a[i] = k < nrow ? alpha_at(k) : 0.0;
            }
#pragma unroll
            for (int i = 0; i < NA; i++) {
                const int k = warp + kWarps * i;
                const unsigned ex = fx::exp_key(a[i]) >> 20;
                // the exponent after the shift by er, saturated (infinities stay infinite)
                if (k < nrow && ex)
                    key = max(key, ex == 2047u ? 2047u
                                               : (unsigned)max(min((int)ex + rows[k].z, 2047), 1));
            }
            if (key) atomicMax(&s_key[CPLX ? lane & ~1 : lane], key);
            for (int i = t; i < npt * kPitch; i += 32 * kWarps) tile[i] = 0;
            __syncthreads();
            const int ck = (int)s_key[CPLX ? lane & ~1 : lane];
            const int E = max(ck, fx::kMinExp);
            if (ck && (ck >= fx::kMaxExp || ck < fx::kMinExp)) s_bad = 1;
            if (warp == 0) s_E[lane] = E;
#pragma unroll
            for (int i = 0; i < NA; i++) {
                const int k = warp + kWarps * i;
                if (k < nrow) al[k * kLanes + lane] = fx::to_digits(a[i], E - rows[k].z);
            }
            __syncthreads();
            // ---- each warp's points: sum of the entries' products
            const bool bad = s_bad != 0;
            for (int it = 0; it < nit; it++) {
                const int e0 = wsplit[it * (kWarps + 1) + warp];
                const int e1 = wsplit[it * (kWarps + 1) + warp + 1];
                if (e0 == e1) continue;
                const int4 I = items[it];
                if (!bad) {
                    int2 b[MAXJ];
#pragma unroll
                    for (int j = 0; j < MAXJ; j++)
                        b[j] = j < I.z ? al[(I.x + j) * kLanes + lane] : make_int2(0, 0);
#pragma unroll 2
                    for (int e = e0; e < e1; e++) {
                        const int4 *c = chi + e * hp;
                        // six chains: one chain of 2 MAXJ dependent adds left the pipe idle
                        long long hh[2] = {0, 0}, ma[2] = {0, 0}, mb[2] = {0, 0};
#pragma unroll
                        for (int j = 0; j < MAXJ; j++) {
                            const int4 q = c[j >> 1];
                            const int ch = (j & 1) ? q.z : q.x, cl = (j & 1) ? q.w : q.y;
                            hh[j & 1] = fx::mad_wide(b[j].x, ch, hh[j & 1]);
                            ma[j & 1] = fx::mad_wide(b[j].x, cl, ma[j & 1]);
                            mb[j & 1] = fx::mad_wide(b[j].y, ch, mb[j & 1]);
                        }
                        tile[lps[e] * kPitch + lane] +=
                            sum57(hh[0] + hh[1], (ma[0] + ma[1]) + (mb[0] + mb[1]));
                    }
                } else {
                    double *td = reinterpret_cast<double *>(tile);
                    for (int e = e0; e < e1; e++) {
                        const int2 *c = reinterpret_cast<const int2 *>(chi + e * hp);
                        double s = 0.0;
                        for (int j = 0; j < I.z; j++)
                            s += chi_value(c[j], rows[I.x + j].z) * alpha_at(I.x + j);
                        td[lps[e] * kPitch + lane] += s;
                    }
                }
            }
            __syncthreads();
            // ---- the finished elements of this warp's columns
#pragma unroll
            for (int c = 0; c < CW; c++) {
                const int cc = warp + kWarps * c, n = n0 + cc;
                const int K = s_E[W * cc] - 1023 + 1 - kChiBits;  // 2^57 units, 57-bit digits
#pragma unroll
                for (int i = 0; i < NV; i++) {
                    if (n < ncol && gp[i] >= 0) {
                        const long o = (long)n * ld + gp[i];
#pragma unroll
                        for (int u = 0; u < W; u++) {
                            const long long s = tile[(32 * i + lane) * kPitch + W * cc + u];
                            const double d = bad ? __longlong_as_double(s) : fx::to_double(s, K);
                            v[c][i][u] = fma(scale, d, v[c][i][u]);
                        }
                        if constexpr (CPLX)
                            reinterpret_cast<double2 *>(out)[o] =
                                make_double2(v[c][i][0], v[c][i][W - 1]);
                        else
                            out[o] = v[c][i][0];
                    }
                }
            }
        }
        if constexpr (PROJ) {
            if (APPLY) {
                __syncthreads();  // s_key, s_bad and the alpha digits are read
                if (t == 0) s_bad = 0;
                __syncthreads();
            }
            // ---- this warp's columns as digits
#pragma unroll
            for (int c = 0; c < CW; c++) {
                const int cc = warp + kWarps * c;
                unsigned key = 0u;
#pragma unroll
                for (int i = 0; i < NV; i++)
#pragma unroll
                    for (int u = 0; u < W; u++) key = max(key, fx::exp_key(v[c][i][u]));
                key = __reduce_max_sync(0xffffffffu, key) >> 20;
                const int E = max((int)key, fx::kMinExp);
                if (key && ((int)key >= fx::kMaxExp || (int)key < fx::kMinExp)) s_bad = 1;
                if (lane < W) s_key[W * cc + lane] = (unsigned)E;
#pragma unroll
                for (int i = 0; i < NV; i++)
                    if (gp[i] >= 0)
#pragma unroll
                        for (int u = 0; u < W; u++)
                            reinterpret_cast<int2 *>(tile)[(32 * i + lane) * kPitch + W * cc + u] =
                                fx::to_digits(v[c][i][u], E);
            }
            unsigned long long *red = reinterpret_cast<unsigned long long *>(al);  // [rows][kLanes]
            for (int i = t; i < nrow * kLanes; i += 32 * kWarps) red[i] = 0ull;
            __syncthreads();
            // ---- the entries in equal shares; an item's sums meet in shared memory
            const bool bad = s_bad != 0;
            const double *src = APPLY ? out : x;
            for (int it = 0; it < nit; it++) {
                int e = max(lo, ent0[it]);
                const int e1 = min(hi, ent0[it + 1]);
                if (e >= e1) continue;
                const int4 I = items[it];
                const int2 *td = reinterpret_cast<const int2 *>(tile) + lane;
                while (e < e1) {
                    const int ee = min(e + 64, e1);  // 64 products: the middle sum's bound
                    if (!bad) {
                        long long hh[MAXJ], mid[MAXJ];
#pragma unroll
                        for (int j = 0; j < MAXJ; j++) hh[j] = mid[j] = 0;
#pragma unroll 2
                        for (int k = e; k < ee; k++) {
                            const int2 xv = td[lps[k] * kPitch];
                            const int4 *c = chi + k * hp;
#pragma unroll
                            for (int j = 0; j < MAXJ; j += 2) {
                                const int4 q = c[j >> 1];
                                fx::mac(hh[j], mid[j], xv.x, xv.y, q.x, q.y);
                                if (j + 1 < MAXJ)
                                    fx::mac(hh[j + 1], mid[j + 1], xv.x, xv.y, q.z, q.w);
                            }
                        }
#pragma unroll
                        for (int j = 0; j < MAXJ; j++)
                            if (j < I.z)
                                atomicAdd(&red[(I.x + j) * kLanes + lane],
                                          (unsigned long long)sum57(hh[j], mid[j]));
                    } else {
                        for (int j = 0; j < I.z; j++) {
                            double s = 0.0;
                            for (int k = e; k < ee; k++) {
                                const long o = (long)lcol * ld + T.pts[p0 + lps[k]];
                                const double xv = !lin ? 0.0 : CPLX ? src[2 * o + (lane & 1)] : src[o];
                                s += chi_value(reinterpret_cast<const int2 *>(chi + k * hp)[j],
                                               rows[I.x + j].z) * xv;
                            }
                            atomicAdd(reinterpret_cast<double *>(&red[(I.x + j) * kLanes + lane]), s);
                        }
                    }
                    e = ee;
                }
            }
            __syncthreads();
            const int K = (int)s_key[lane] - 1023 + 1 - kChiBits;
            for (int k = warp; k < nrow; k += kWarps) {
                const int4 q = rows[k];
                const long long s = (long long)red[k * kLanes + lane];
                double y = bad ? __longlong_as_double(s) : fx::to_double(s, K + q.z);
                if constexpr (CPLX) {  // e^{i theta} (re + i im): this lane's part
                    const double2 ph = phase[q.y];
                    const double z = __shfl_xor_sync(0xffffffffu, y, 1);
                    y = fma(ph.x, y, ((lane & 1) ? ph.y : -ph.y) * z);
                }
                if (lin) part[W * ((long)(q0 + k) * ldp + lcol) + (CPLX ? lane & 1 : 0)] = y;
            }
        }
        if (g + gstep < ngroup) __syncthreads();  // tile, sums and keys are free again
    }
}

// out[c] = f times the sum over e in [e0, e1) of part[idx[e]][c] for the 32 doubles c from c0 (below
// n): the block's eight warps take every eighth row, and their sums are added in warp order, so
// the result is fixed by the tables alone. One thread per column instead waits for its rows one
// after another (26^3: 15 us for 144 rows).
__device__ __forceinline__ void reduce_row(int e0, int e1, const int *__restrict__ idx,
                                           const double *__restrict__ part, long ldp, int c0, int n,
                                           double f, double *__restrict__ out)
{
    __shared__ double sh[kWarps][32];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, c = c0 + lane;
    double s0 = 0.0, s1 = 0.0;
    if (c < n) {
        int e = e0 + warp;
        for (; e + kWarps < e1; e += 2 * kWarps) {
            s0 += __ldg(part + (long)__ldg(idx + e) * ldp + c);
            s1 += __ldg(part + (long)__ldg(idx + e + kWarps) * ldp + c);
        }
        if (e < e1) s0 += __ldg(part + (long)__ldg(idx + e) * ldp + c);
    }
    sh[warp][lane] = s0 + s1;
    __syncthreads();
    if (warp == 0 && c < n) {
        double s = sh[0][lane];
#pragma unroll
        for (int w = 1; w < kWarps; w++) s += sh[w][lane];
        out[c] = f * s;
    }
}

}  // namespace nlfx

nlfx::Tables nonlocal_fx_tables(const Nonlocal &nl, const NlFx &x);
const NlFx &nonlocal_fx_pick(const Nonlocal &nl, long groups);
// The partial rows (WS_NLPART) of `groups` column groups of group_bytes each, or of as many at a time
// as scratch_max and the device's free memory hold (*chunk); SGPU_ERR_NOMEM: not even one, and the
// caller takes the FP64 kernels, which need none
int nonlocal_fx_part(sgpu_ctx *ctx, size_t group_bytes, int groups, int *chunk, void **part);
}  // namespace sgpu
