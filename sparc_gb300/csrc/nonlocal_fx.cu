// FP64 nonlocal apply and projection in block fixed point: range tables and launches
// (the kernel body is in nonlocal_fx.cuh).
#include <algorithm>
#include <cmath>
#include <cstring>
#include <string>
#include <vector>

#include "nonlocal_fx.cuh"

namespace sgpu {
namespace {

template <bool APPLY, bool PROJ, int MAXJ>
__global__ void __launch_bounds__(32 * nlfx::kWarps, 2)
    k_nl_fx(const nlfx::Tables T, int ncol, const double *__restrict__ alpha, double scale,
            double *out, const double *__restrict__ x, long ld, double *__restrict__ part,
            long lda, long ldp)
{
    extern __shared__ __align__(16) unsigned char smem_nlfx[];
    nlfx::block<false, APPLY, PROJ, MAXJ>(T, blockIdx.y, blockIdx.x, gridDim.x, ncol, alpha, scale,
                                          out, x, ld, part, lda, ldp, nullptr, smem_nlfx);
}

// alpha[row] = dV Gamma[row] times the sum of the row's partial projections (nlfx::reduce_row)
__global__ void __launch_bounds__(256)
    k_fx_reduce(const int *__restrict__ ptr, const int *__restrict__ idx,
                const double *__restrict__ part, long ldp, int n, double dV,
                const double *__restrict__ gamma, double *__restrict__ alpha, long lda)
{
    const int row = blockIdx.x;  // x: more rows than a y dimension holds are in use
    nlfx::reduce_row(ptr[row], ptr[row + 1], idx, part, ldp, blockIdx.y * 32, n,
                     dV * __ldg(gamma + row), alpha + (long)row * lda);
}

// Chi digits of the entries: value j of entry e is chi[src[e].x + j * src[e].y] scaled by its row's
// 2^er, rounded to kChiBits bits
__global__ void k_fx_chi(const long2 *__restrict__ src, const int2 *__restrict__ rows, long nent,
                         int jp, const double *__restrict__ chi, const int *__restrict__ er,
                         int2 *__restrict__ out)
{
    for (long i = blockIdx.x * (long)blockDim.x + threadIdx.x; i < nent * jp;
         i += (long)gridDim.x * blockDim.x) {
        const long e = i / jp;
        const int j = (int)(i - e * jp);
        const int2 row = rows[e];  // (first projector row, count)
        int2 d = make_int2(0, 0);
        if (j < row.y) {
            const long long C =
                llrint(ldexp(chi[src[e].x + j * src[e].y], nlfx::kChiBits - er[row.x + j]));
            const long long H = (C + (1ll << (fx::kDigit - 1))) >> fx::kDigit;
            d = make_int2((int)H, (int)(C - (H << fx::kDigit)));
        }
        out[i] = d;
    }
}

template <bool APPLY, bool PROJ>
int launch(sgpu_ctx *ctx, int ncol, const double *alpha, double scale, double *out,
           const double *x, long ld, double *alpha_next, long lda, cudaStream_t st)
{
    const Nonlocal &nl = ctx->nl;
    const int groups = (ncol + nlfx::kLanes - 1) / nlfx::kLanes;
    const NlFx &X = nonlocal_fx_pick(nl, groups);
    const nlfx::Tables T = nonlocal_fx_tables(nl, X);
    const size_t smem = nlfx::shared_bytes(T);
    auto kern = nl.max_np <= 9 ? k_nl_fx<APPLY, PROJ, 9> : k_nl_fx<APPLY, PROJ, 18>;
    SGPU_CUDA_TRY(allow_smem(kern));
    double *part = nullptr;
    int chunk = groups;
    if (PROJ)
        SGPU_TRY(nonlocal_fx_part(ctx, sizeof(double) * (size_t)X.nrows * nlfx::kLanes, groups, &chunk,
                                  (void **)&part));
    const long ldp = (long)chunk * nlfx::kLanes;
    for (int g0 = 0; g0 < groups; g0 += chunk) {
        const int c0 = g0 * nlfx::kLanes, gn = std::min(chunk, groups - g0);
        const int n = std::min(ncol - c0, gn * nlfx::kLanes);
        {
            ProfScope ps(ctx, APPLY ? SGPU_KERNEL_NL_APPLY : SGPU_KERNEL_NL_PROJECT, st);
            for (int r0 = 0; r0 < X.nrange; r0 += 65535) {
                nlfx::Tables R = T;
                R.pt0 += r0;
                R.item0 += r0;
                R.row0 += r0;
                // blocks of few ranges split the column groups, so that there are at least 8 per SM
                const int gx = std::min(gn, std::max(1, 152 * 8 / X.nrange));
                const dim3 grid(gx, std::min(65535, X.nrange - r0));
                kern<<<grid, 32 * nlfx::kWarps, smem, st>>>(
                    R, n, APPLY ? alpha + c0 : nullptr, scale, APPLY ? out + (long)c0 * ld : nullptr,
                    APPLY ? nullptr : x + (long)c0 * ld, ld, part, lda, ldp);
            }
            SGPU_CUDA_TRY(cudaGetLastError());
        }
        if (PROJ) {
            ProfScope ps(ctx, SGPU_KERNEL_NL_PROJECT, st);
            k_fx_reduce<<<dim3(nl.ntot, gn), 256, 0, st>>>(X.sum_ptr, X.sum_idx, part, ldp, n, ctx->dV,
                                                           nl.gamma64, alpha_next + c0, lda);
            SGPU_CUDA_TRY(cudaGetLastError());
        }
    }
    return SGPU_OK;
}

// the projection in FP64, which adds up in alpha itself and needs no partial rows
int project_fp64(sgpu_ctx *ctx, int ncol, const double *x, long ldx, double *alpha, long lda,
                 cudaStream_t st)
{
    SGPU_CUDA_TRY(cudaMemsetAsync(alpha, 0, sizeof(double) * (size_t)ctx->nl.ntot * lda, st));
    return launch_nonlocal_project<double>(ctx, ncol, x, ldx, alpha, lda, st, false);
}

}  // namespace

nlfx::Tables nonlocal_fx_tables(const Nonlocal &nl, const NlFx &x)
{
    return {x.pt0, x.pts, x.item0, x.items, x.ent0, x.wsplit, x.lp, x.chi, x.rows, x.row0, nl.fx_jp,
            x.max_rows, x.max_ent, x.max_items};
}

// The large ranges when they and the column groups make two blocks per SM, else the small ones:
// 32-point ranges hold few entries per atom, so the rows' and columns' conversions weigh more
// (26^3, 32 columns: 28 large ranges leave most SMs idle; 34^3, 20 blocks of 64 complex columns:
// 80 large ranges against 310 small ones)
const NlFx &nonlocal_fx_pick(const Nonlocal &nl, long groups)
{
    return nl.fx[1].nrange > 0 && nl.fx[0].nrange * groups < 304 ? nl.fx[1] : nl.fx[0];
}

bool nonlocal_fx_ready(const sgpu_ctx *ctx)
{
    return ctx->fx_on && ctx->has_nl && ctx->nl.fx[0].nrange > 0;
}

void nonlocal_fx_free(Nonlocal &nl)
{
    for (NlFx &x : nl.fx) {
        if (x.mem) cudaFree(x.mem);
        x = NlFx();
    }
}

int nonlocal_fx_part(sgpu_ctx *ctx, size_t group_bytes, int groups, int *chunk, void **part)
{
    int c = (int)std::min<size_t>(std::min(groups, 32768), std::max<size_t>(1, scratch_max(ctx) / group_bytes));
    for (;; c = (c + 1) / 2) {
        const int rc = ws_get(ctx, WS_NLPART, group_bytes * c, part);
        *chunk = c;
        if (rc != SGPU_ERR_NOMEM || c == 1) return rc;
    }
}

int launch_nonlocal_fx_project(sgpu_ctx *ctx, int ncol, const double *x, long ldx, double *alpha,
                               long lda, cudaStream_t st)
{
    const int rc = launch<false, true>(ctx, ncol, nullptr, 0.0, nullptr, x, ldx, alpha, lda, st);
    return rc == SGPU_ERR_NOMEM ? project_fp64(ctx, ncol, x, ldx, alpha, lda, st) : rc;
}

int launch_nonlocal_fx_apply(sgpu_ctx *ctx, int ncol, const double *alpha, long lda, double scale,
                             double *out, long ldo, double *alpha_next, cudaStream_t st)
{
    if (alpha_next) {  // the partial rows are sought before anything is launched
        const int rc =
            launch<true, true>(ctx, ncol, alpha, scale, out, nullptr, ldo, alpha_next, lda, st);
        if (rc != SGPU_ERR_NOMEM) return rc;
    }
    SGPU_TRY((launch<true, false>(ctx, ncol, alpha, scale, out, nullptr, ldo, nullptr, lda, st)));
    return alpha_next ? project_fp64(ctx, ncol, out, ldo, alpha_next, lda, st) : SGPU_OK;
}

// Range tables. A range takes covered points in the order of 32 x 4 x 4 blocks of the grid until it
// holds `cap` of them or the next point's images would take its rows past kRows or its Chi digits
// past kChiBytes. No tables (and the FP64 kernels stay) for more than 18 projectors per atom, for a
// point under more than kPtRows projector rows (the 64-bit sums hold that many) and for Chi
// values outside 1e-40 .. 1e40. SGPU_ERR_NOMEM: no room for them.
static int build_ranges(sgpu_ctx *ctx, Nonlocal &nl, NlFx &x, int cap, const std::vector<int> &er,
                        const std::vector<int> &ord, const std::vector<int> &covpts,
                        const std::vector<int> &covptr, const std::vector<long> &ent_chi,
                        const std::vector<int4> &ent_meta)
{
    std::vector<int> pt0(1, 0), pts, item0(1, 0), ent0(1, 0), row0(1, 0), wsplit;
    std::vector<int4> items, rowinfo;
    std::vector<unsigned char> lp;
    std::vector<long2> src;
    std::vector<int2> rows;
    pts.reserve(nl.ncov);
    lp.reserve(nl.nent);
    src.reserve(nl.nent);
    rows.reserve(nl.nent);
    std::vector<int> slot(nl.nimg, -1);                 // image -> item of the current range
    std::vector<std::vector<std::pair<int, int>>> bucket;  // per item: (point, entry)
    const int max_ent = nlfx::kChiBytes / (8 * nl.fx_jp);
    int k = 0;
    x.max_rows = x.max_ent = x.max_items = 0;
    while (k < nl.ncov) {
        const int q0 = k;
        int nrow = 0, nitem = 0, nent = 0;
        std::vector<int> imgs;
        while (k < nl.ncov && k - q0 < cap) {
            const int c = ord[k];
            int add = 0, here = 0;
            for (int e = covptr[c]; e < covptr[c + 1]; e++) {
                here += ent_meta[e].y;
                if (slot[ent_meta[e].w] < 0) add += ent_meta[e].y;
            }
            if (here > nlfx::kPtRows) return SGPU_OK;
            if (nrow + add > nlfx::kRows || nent + covptr[c + 1] - covptr[c] > max_ent) break;
            nent += covptr[c + 1] - covptr[c];
            for (int e = covptr[c]; e < covptr[c + 1]; e++) {
                const int g = ent_meta[e].w;
                if (slot[g] < 0) {
                    slot[g] = nitem++;
                    imgs.push_back(g);
                    if ((int)bucket.size() < nitem) bucket.emplace_back();
                    bucket[slot[g]].clear();
                    nrow += ent_meta[e].y;
                }
                bucket[slot[g]].push_back({k - q0, e});
            }
            pts.push_back(covpts[c]);
            k++;
        }
        if (k == q0) return SGPU_OK;
        x.max_rows = std::max(x.max_rows, nrow);
        x.max_ent = std::max(x.max_ent, nent);
        x.max_items = std::max(x.max_items, nitem);
        // owner warps of the apply: runs of points with about equal entry counts
        int wb[nlfx::kWarps + 1];
        {
            long tot = 0, seen = 0;
            for (int q = q0; q < k; q++) tot += covptr[ord[q] + 1] - covptr[ord[q]];
            wb[0] = 0;
            int q = q0;
            for (int w = 1; w < nlfx::kWarps; w++) {
                while (q < k && seen < tot * w / nlfx::kWarps) {
                    seen += covptr[ord[q] + 1] - covptr[ord[q]];
                    q++;
                }
                wb[w] = q - q0;
            }
            wb[nlfx::kWarps] = k - q0;
        }
        int off = 0;
        for (int i = 0; i < nitem; i++) {
            const int4 m0 = ent_meta[bucket[i][0].second];
            items.push_back(make_int4(off, m0.x, m0.y, imgs[i]));
            off += m0.y;
            for (int j = 0; j < m0.y; j++)
                rowinfo.push_back(make_int4(m0.x + j, imgs[i], er[m0.x + j], 0));
            const int first = (int)lp.size();
            for (const auto &b : bucket[i]) {
                const int4 m = ent_meta[b.second];
                lp.push_back((unsigned char)b.first);
                src.push_back({ent_chi[b.second], (long)m.z});
                rows.push_back(make_int2(m.x, m.y));
            }
            for (int w = 0, e = first; w <= nlfx::kWarps; w++) {
                while (e < (int)lp.size() && (w == nlfx::kWarps || lp[e] < wb[w])) e++;
                wsplit.push_back(e);
            }
            ent0.push_back((int)lp.size());
            slot[imgs[i]] = -1;
        }
        pt0.push_back(k);
        item0.push_back((int)items.size());
        row0.push_back(row0.back() + nrow);
    }
    // per projector row, its rows of the partial buffer in range order
    x.nrows = row0.back();
    std::vector<int> sum_ptr(nl.ntot + 1, 0), sum_idx(x.nrows);
    for (const int4 &I : items)
        for (int j = 0; j < I.z; j++) sum_ptr[I.y + j + 1]++;
    for (int i = 0; i < nl.ntot; i++) sum_ptr[i + 1] += sum_ptr[i];
    {
        std::vector<int> at(sum_ptr.begin(), sum_ptr.end() - 1);
        for (size_t r = 0; r + 1 < item0.size(); r++)
            for (int i = item0[r]; i < item0[r + 1]; i++)
                for (int j = 0; j < items[i].z; j++)
                    sum_idx[at[items[i].y + j]++] = row0[r] + items[i].x + j;
    }
    // one allocation for the tables, another for what the Chi kernel reads
    struct Put {
        void **dst;
        const void *src;
        size_t at, bytes;
    };
    std::vector<Put> put;
    size_t size = 0, tsize = 0;
    auto table = [&](auto **dst, const auto &v, size_t &to) {
        const size_t at = (to + 255) / 256 * 256;
        to = at + sizeof(v[0]) * v.size();
        put.push_back({(void **)dst, v.data(), at, to - at});
    };
    long2 *dsrc = nullptr;
    int2 *drows = nullptr;
    table(&dsrc, src, tsize);
    table(&drows, rows, tsize);
    table(&x.pt0, pt0, size);
    table(&x.pts, pts, size);
    table(&x.item0, item0, size);
    table(&x.items, items, size);
    table(&x.ent0, ent0, size);
    table(&x.wsplit, wsplit, size);
    table(&x.lp, lp, size);
    table(&x.rows, rowinfo, size);
    table(&x.row0, row0, size);
    table(&x.sum_ptr, sum_ptr, size);
    table(&x.sum_idx, sum_idx, size);
    const size_t ochi = (size + 255) / 256 * 256;
    const size_t bytes = ochi + sizeof(int2) * (size_t)nl.nent * nl.fx_jp;
    char *base = nullptr, *temp = nullptr;
    int rc = SGPU_OK;
    if (dev_alloc(ctx, &base, ctx->inject & 2 ? (size_t)1 << 60 : bytes) != cudaSuccess ||
        dev_alloc(ctx, &temp, tsize) != cudaSuccess) {
        rc = SGPU_ERR_NOMEM;
    } else {
        // small tables in one copy (a copy takes about 10 us), large ones from where they are
        cudaError_t e = cudaSuccess;
        std::vector<char> host(size < ((size_t)4 << 20) ? size : 0);
        for (size_t p = 0; p < put.size() && e == cudaSuccess; p++) {
            const Put &q = put[p];
            *q.dst = (p < 2 ? temp : base) + q.at;
            if (p >= 2 && !host.empty()) std::memcpy(host.data() + q.at, q.src, q.bytes);
            else e = cudaMemcpy(*q.dst, q.src, q.bytes, cudaMemcpyHostToDevice);
        }
        if (e == cudaSuccess && !host.empty()) e = cudaMemcpy(base, host.data(), size, cudaMemcpyHostToDevice);
        x.chi = reinterpret_cast<int4 *>(base + ochi);
        if (e == cudaSuccess) {
            k_fx_chi<<<152 * 8, 256>>>(dsrc, drows, nl.nent, nl.fx_jp, nl.chi64, nl.fx_er,
                                       reinterpret_cast<int2 *>(x.chi));
            e = cudaDeviceSynchronize();
        }
        if (e != cudaSuccess) {
            set_error(std::string("set_nonlocal: the fixed-point tables: ") + cudaGetErrorString(e));
            rc = SGPU_ERR_CUDA;
        }
    }
    if (temp) cudaFree(temp);
    if (rc != SGPU_OK) {
        if (base) cudaFree(base);
        return rc;
    }
    x.mem = base;
    x.nrange = (int)pt0.size() - 1;
    return SGPU_OK;
}


int nonlocal_fx_build(sgpu_ctx *ctx, Nonlocal &nl, const std::vector<int> &ord, const std::vector<int> &covpts,
                      const std::vector<int> &covptr, const std::vector<long> &ent_chi,
                      const std::vector<int4> &ent_meta, const double *chi)
{
    if (nl.max_np > 18 || nl.max_np < 1 || nl.ncov == 0) return SGPU_OK;
    // exponent of each projector row's largest Chi value
    std::vector<int> er(nl.ntot, 0);
    {
        std::vector<double> mx(nl.ntot, 0.0);
        for (long e = 0; e < nl.nent; e++) {
            const int4 m = ent_meta[e];
            for (int j = 0; j < m.y; j++) {
                const double v = std::fabs(chi[ent_chi[e] + (long)j * m.z]);
                if (!(v < 1e40)) return SGPU_OK;  // NaN too
                mx[m.x + j] = std::max(mx[m.x + j], v);
            }
        }
        for (int i = 0; i < nl.ntot; i++) {
            if (mx[i] == 0.0) continue;
            if (mx[i] < 1e-40) return SGPU_OK;
            std::frexp(mx[i], &er[i]);
        }
    }
    if (dev_alloc(ctx, &nl.fx_er, sizeof(int) * er.size()) != cudaSuccess) return SGPU_ERR_NOMEM;
    SGPU_CUDA_TRY(cudaMemcpy(nl.fx_er, er.data(), sizeof(int) * er.size(), cudaMemcpyHostToDevice));
    nl.fx_jp = nl.max_np <= 9 ? 10 : 18;
    SGPU_TRY(build_ranges(ctx, nl, nl.fx[0], nlfx::kPts, er, ord, covpts, covptr, ent_chi, ent_meta));
    // small ranges where one column group in large ones leaves SMs without a block
    if (nl.fx[0].nrange > 0 && nl.fx[0].nrange < 304)
        SGPU_TRY(build_ranges(ctx, nl, nl.fx[1], nl.fx[0].nrange < 152 ? 32 : 64, er, ord, covpts, covptr,
                              ent_chi, ent_meta));
    return SGPU_OK;
}

}  // namespace sgpu
