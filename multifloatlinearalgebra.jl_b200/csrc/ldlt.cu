// Bunch-Kaufman LDL^T (1x1 and 2x2 pivots) with its solve and inertia.
//
// Follows src/factorizations/ldlt.jl of MultiFloatLinearAlgebra.jl:
//   * unblocked route (ldlt.jl:352-412): one cluster of CTAs runs the pivot
//     steps; each step's column scan, row scan, symmetric swap, column scaling
//     and rank-1 / rank-2 update are spread over the cluster's threads, the
//     pivot decisions are taken by every thread from the same values exactly
//     as ldlt.jl:183-219 orders them;
//   * blocked route (ldlt_gemmt.jl:36-73): per panel the same cluster kernel
//     runs the lazy panel (every entry evaluated against the earlier pivots of
//     the panel, ldlt.jl:414-593), then W = L21 * D (ldlt.jl:595-632), the
//     lower trailing update A22 = -1 * L21 W^T + 1 * A22 through the shared
//     mainloop (gemmt) and the upper mirror.
// Every per-element expression and its association is the reference's, so the
// result is bitwise the oracle's; the parallel loops only distribute
// independent elements.  When a step fails (info > 0) the factor content after
// that step is left as the parallel loop wrote it.
#include "cluster.cuh"
#include "mf_device.cuh"
#include "mflab_internal.h"

namespace mfl {

template <int N>
struct Ldlt {
    Mat A;
    int64_t n;
    double *dsub;  // dsub[l * lsd + k]
    int64_t lsd;
    int64_t *pivots;  // 1-based
    uint8_t *blocks;
    __device__ mf<N> at(int64_t r, int64_t c) const { return load_mf<N>(A.p, A.ld, A.ls, r, c); }
    __device__ void put(int64_t r, int64_t c, const mf<N> &v) const {
        store_mf<N>(A.p, A.ld, A.ls, r, c, v);
    }
    __device__ mf<N> ds(int64_t k) const {
        mf<N> v;
#pragma unroll
        for (int l = 0; l < N; ++l) v.v[l] = dsub[l * lsd + k];
        return v;
    }
    __device__ void set_ds(int64_t k, const mf<N> &v) const {
#pragma unroll
        for (int l = 0; l < N; ++l) dsub[l * lsd + k] = v.v[l];
    }
};

// ldlt.jl:65-101; returns nonsingular
template <int N>
__device__ __noinline__ bool solve_2x2(const mf<N> &d11, const mf<N> &d21, const mf<N> &d22, const mf<N> &first,
                          const mf<N> &second, mf<N> &x1, mf<N> &x2) {
    const mf<N> scale = max_mf(max_mf(abs_mf(d11), abs_mf(d21)), abs_mf(d22));
    x1 = from_double<N>(0.0);
    x2 = from_double<N>(0.0);
    if (iszero(scale) || !isfinite_mf(scale)) return false;
    const mf<N> a = div_call(d11, scale), b = div_call(d21, scale), c = div_call(d22, scale);
    const mf<N> r1 = div_call(first, scale), r2 = div_call(second, scale);
    if (ge(abs_mf(a), abs_mf(b))) {
        if (iszero(a)) return false;
        const mf<N> t = div_call(b, a);
        const mf<N> u = submul(c, t, b);
        if (iszero(u) || !isfinite_mf(u)) return false;
        const mf<N> y2 = div_call(submul(r2, t, r1), u);
        x1 = div_call(submul(r1, b, y2), a);
        x2 = y2;
        return true;
    }
    if (iszero(b)) return false;
    const mf<N> t = div_call(a, b);
    const mf<N> u = submul(b, t, c);
    if (iszero(u) || !isfinite_mf(u)) return false;
    const mf<N> y2 = div_call(submul(r1, t, r2), u);
    x1 = div_call(submul(r2, c, y2), b);
    x2 = y2;
    return true;
}

// ---------------------------------------------------- cluster kernel ------
// One launch runs a lazy panel (LAZY) or the whole unblocked factorization on
// one cluster.  A pivot step is a few dependent scans of a column with a
// decision after each, so its time is latency: the scans' chains and the
// cluster barriers.  What keeps both short:
//   * rows are dealt to the cluster's warps in groups of 32, so a scan is one
//     chain per thread and the rank updates use every CTA's FP64 pipe;
//   * in a lazy entry row r, column c (ldlt.jl:414-449),
//         v = A[r,c]; v -= A[r,q] * (D[q] * A[c,q]) over the panel's pivots q,
//     the inner product depends on the column alone: it is formed once per
//     column and CTA in shared memory, where it was formed anew in every
//     entry, and the pivots' D stay there too;
//   * candidates are written into every CTA of the cluster before the barrier
//     and read locally after it; a step takes two to four barriers;
//   * the symmetric swap is one pass over disjoint pairs.
// x3, n = 600: 215 us a 12-column panel (495 us on one CTA).
constexpr int LD_NT = 256, LD_WARPS = LD_NT / 32, LD_MAXC = MAX_CLUSTER, LD_PANEL = 66;

template <int N>
struct LdShared {
    double coef[2][LD_PANEL][N];  // D * A[col, panel] of the columns k and imax / k+1
    double rowi[LD_PANEL][N];     // A[imax, panel]
    double d[LD_PANEL][N], ds[LD_PANEL][N];
    double cand[2][LD_MAXC][N];   // every CTA's column / row maximum
    int candi[2][LD_MAXC];
    double red[LD_WARPS][N];
    int redi[LD_WARPS];
    double val[3][N];             // diagonal entries formed by single lanes
    double blk[6][N];             // the 2x2 block's scale, a, b, c, t, u (ld_block)
    int regular;                  // 0 singular, 1 |a| >= |b|, 2 |a| < |b|
    unsigned char type[LD_PANEL];
    int flag;
    int nan_at;                   // last NaN of the row scan, -1 without one
};

// coefficients D * A[col, pf + i], i < cnt, of one column's lazy entries
template <int N>
__device__ void ld_stage_coef(const Ldlt<N> &F, LdShared<N> &sh, double (*dst)[N], int64_t col,
                              int64_t pf, int cnt) {
    for (int i = threadIdx.x; i < cnt; i += LD_NT) {
        const mf<N> d = ld_get<N>(sh.d[i]), c = F.at(col, pf + i);
        if (sh.type[i] == 1) {
            ld_put<N>(dst[i], mul(d, c));
        } else if (sh.type[i] == 2) {
            const mf<N> cs = F.at(col, pf + i + 1), o = ld_get<N>(sh.ds[i]);
            ld_put<N>(dst[i], add(mul(d, c), mul(o, cs)));
            ld_put<N>(dst[i + 1], add(mul(o, c), mul(ld_get<N>(sh.d[i + 1]), cs)));
        }
    }
}

// entry (r, col), r >= col, from the column's staged coefficients; the panel
// values are fetched two terms ahead
template <int N>
__device__ __noinline__ mf<N> ld_entry(const Ldlt<N> &F, const LdShared<N> &sh, const double (*coef)[N],
                          int64_t r, int64_t col, int64_t pf, int cnt) {
    mf<N> v = F.at(r, col);
    if (cnt == 0) return v;
    auto fetch = [&](int i) { return i < cnt ? F.at(r, pf + i) : from_double<N>(0.0); };
    mf<N> a = fetch(0), b = fetch(1), c = fetch(2);
    // the product of term i, whose panel values are a (and b)
    auto term = [&](int i) {
        mf<N> p = mul(a, ld_get<N>(coef[i]));
        if (sh.type[i] != 1) p = add(p, mul(b, ld_get<N>(coef[i + 1])));
        return p;
    };
    mf<N> p = term(0);
    for (int i = 0;;) {
        const bool one = sh.type[i] == 1;
        const mf<N> n0 = fetch(i + 3);
        if (one) {
            a = b;
            b = c;
            c = n0;
            i += 1;
        } else {
            a = c;
            b = n0;
            c = fetch(i + 4);
            i += 2;
        }
        if (i >= cnt) return sub(v, p);
        const mf<N> q = term(i);  // the next product beside this subtraction
        v = sub(v, p);
        p = q;
    }
}

// entry (imax, c), c < imax: row imax staged, the coefficients are column c's own
template <int N>
__device__ __noinline__ mf<N> ld_row_entry(const Ldlt<N> &F, const LdShared<N> &sh, int64_t imax, int64_t c,
                              int64_t pf, int cnt) {
    mf<N> v = F.at(imax, c);
    if (cnt == 0) return v;
    auto fetch = [&](int i) { return i < cnt ? F.at(c, pf + i) : from_double<N>(0.0); };
    mf<N> a = fetch(0), b = fetch(1);
    auto term = [&](int i) {
        const mf<N> d = ld_get<N>(sh.d[i]);
        if (sh.type[i] == 1) return mul(ld_get<N>(sh.rowi[i]), mul(d, a));
        const mf<N> o = ld_get<N>(sh.ds[i]);
        const mf<N> c1 = add(mul(d, a), mul(o, b));
        const mf<N> c2 = add(mul(o, a), mul(ld_get<N>(sh.d[i + 1]), b));
        return add(mul(ld_get<N>(sh.rowi[i]), c1), mul(ld_get<N>(sh.rowi[i + 1]), c2));
    };
    mf<N> p = term(0);
    for (int i = 0;;) {
        const bool one = sh.type[i] == 1;
        const mf<N> n0 = fetch(i + 2);
        if (one) {
            a = b;
            b = n0;
            i += 1;
        } else {
            a = n0;
            b = fetch(i + 3);
            i += 2;
        }
        if (i >= cnt) return sub(v, p);
        const mf<N> q = term(i);
        v = sub(v, p);
        p = q;
    }
}

// cluster-wide best candidate, in every thread: buffer b of the candidates;
// one CTA barrier and one cluster barrier
template <int N>
__device__ void ld_reduce(LdShared<N> &sh, int b, uint32_t rank, int nc, mf<N> &v, int &i) {
    const int lane = threadIdx.x % 32, warp = threadIdx.x / 32;
    ld_lanes(v, i, 32);
    if (lane == 0) {
        ld_put<N>(sh.red[warp], v);
        sh.redi[warp] = i;
    }
    __syncthreads();
    if (warp == 0) {
        v = ld_get<N>(sh.red[lane % LD_WARPS]);
        i = sh.redi[lane % LD_WARPS];
        ld_lanes(v, i, LD_WARPS);
        if (lane < nc) {
#pragma unroll
            for (int l = 0; l < N; ++l)
                ld_remote_f64(ld_remote(&sh.cand[b][rank][l], (uint32_t)lane), v.v[l]);
            ld_remote_s32(ld_remote(&sh.candi[b][rank], (uint32_t)lane), i);
        }
    }
    ld_cluster_sync();
    v = lane < nc ? ld_get<N>(sh.cand[b][lane]) : from_double<N>(0.0);
    i = lane < nc ? sh.candi[b][lane] : -1;
    ld_lanes(v, i, 32);
}

// solve_2x2 in two parts with the same operations: what depends on the block
// alone, by one warp (the three quotients by the scale on a lane each), and a
// right-hand side's part given that.
template <int N>
__device__ __noinline__ void ld_block(LdShared<N> &sh, const mf<N> &d11, const mf<N> &d21,
                                      const mf<N> &d22) {
    const int lane = threadIdx.x % 32;
    const mf<N> scale = max_mf(max_mf(abs_mf(d11), abs_mf(d21)), abs_mf(d22));
    if (iszero(scale) || !isfinite_mf(scale)) {
        if (lane == 0) sh.regular = 0;
        return;
    }
    const mf<N> mine = div_call(lane == 0 ? d11 : lane == 1 ? d21 : d22, scale);
    mf<N> a, b, c;
#pragma unroll
    for (int l = 0; l < N; ++l) {
        a.v[l] = __shfl_sync(0xffffffffu, mine.v[l], 0);
        b.v[l] = __shfl_sync(0xffffffffu, mine.v[l], 1);
        c.v[l] = __shfl_sync(0xffffffffu, mine.v[l], 2);
    }
    const bool first = ge(abs_mf(a), abs_mf(b));
    const mf<N> lead = first ? a : b;
    int regular = 0;
    mf<N> t = lead, u = lead;
    if (!iszero(lead)) {
        t = div_call(first ? b : a, lead);
        u = first ? submul(c, t, b) : submul(b, t, c);
        if (!iszero(u) && isfinite_mf(u)) regular = first ? 1 : 2;
    }
    if (lane == 0) {
        const mf<N> out[6] = {scale, a, b, c, t, u};
#pragma unroll
        for (int i = 0; i < 6; ++i) ld_put<N>(sh.blk[i], out[i]);
        sh.regular = regular;
    }
}

template <int N>
__device__ __noinline__ void ld_block_solve(const LdShared<N> &sh, const mf<N> &r1, const mf<N> &r2,
                                            mf<N> &x1, mf<N> &x2) {
    const mf<N> a = ld_get<N>(sh.blk[1]), b = ld_get<N>(sh.blk[2]), c = ld_get<N>(sh.blk[3]);
    const mf<N> t = ld_get<N>(sh.blk[4]), u = ld_get<N>(sh.blk[5]);
    const bool first = sh.regular == 1;
    x2 = div_call(first ? submul(r2, t, r1) : submul(r1, t, r2), u);
    x1 = div_call(first ? submul(r1, b, x2) : submul(r2, c, x2), first ? a : b);
}

// P A P^T of rows / columns a < b on the active part plus the row swap of the
// earlier columns (ldlt.jl:155-181), as disjoint exchanges: rows a and b in
// every other column, columns a and b in every other row from `first` on, and
// the four entries where they cross
template <int N>
__device__ void ld_sym_swap(const Ldlt<N> &F, int64_t a, int64_t b, int64_t first, int64_t gt_,
                            int64_t total) {
    const int64_t ld = F.A.ld;
    for (int64_t c = gt_; c < F.n; c += total) {
        // all loads before the stores: x <-> y and, from `first` on, u <-> w
        const int64_t ix = c * ld + a, iy = c == a ? b * ld + b : c == b ? a * ld + b : c * ld + b;
        const bool cols = c != a && c != b && c >= first;
        const int64_t iu = a * ld + c, iw = b * ld + c;
        const mf<N> x = load_mf<N>(F.A.p, 0, F.A.ls, ix, 0), y = load_mf<N>(F.A.p, 0, F.A.ls, iy, 0);
        mf<N> u = x, w = y;
        if (cols) {
            u = load_mf<N>(F.A.p, 0, F.A.ls, iu, 0);
            w = load_mf<N>(F.A.p, 0, F.A.ls, iw, 0);
        }
        store_mf<N>(F.A.p, 0, F.A.ls, ix, 0, y);
        store_mf<N>(F.A.p, 0, F.A.ls, iy, 0, x);
        if (cols) {
            store_mf<N>(F.A.p, 0, F.A.ls, iu, 0, w);
            store_mf<N>(F.A.p, 0, F.A.ls, iw, 0, u);
        }
    }
}

template <int N, bool LAZY>
__global__ void __launch_bounds__(LD_NT)
    ldlt_cluster_kernel(Ldlt<N> F, scal<N> alpha_s, int64_t pf, int64_t requested_last, int *info,
                        int64_t *status) {
    __shared__ LdShared<N> sh;
    const int t = threadIdx.x, lane = t % 32, warp = t / 32;
    if (*info) {  // the same in every thread of the cluster
        if (LAZY && t == 0) status[1] = *info;
        return;
    }
    uint32_t rank, ncu;
    asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(rank));
    asm volatile("mov.u32 %0, %%cluster_nctarank;" : "=r"(ncu));
    const int nc = (int)ncu;
    const bool writer = rank == 0 && t == 0;
    const int64_t n = F.n, total = (int64_t)nc * LD_NT;
    // this thread's rows: group g of 32 goes to CTA g mod nc, warp (g / nc) mod 8
    const int64_t mine = 32 * (rank + (int64_t)nc * warp) + lane;
    const mf<N> alpha = alpha_s.get(), zero = from_double<N>(0.0);
    int64_t pl = LAZY ? requested_last : n - 1;
    int64_t k = LAZY ? pf : 0;
    if (t == 0) sh.flag = 0;
    // no CTA writes into another one before that one has started
    ld_cluster_sync();
    auto report = [&](int64_t failed) {  // {last column of the panel, failed column or 0}
        if (LAZY && writer) {
            status[0] = pl;
            status[1] = failed;
        }
    };
    auto fail = [&](int64_t kk) {
        if (writer) *info = (int)(kk + 1);
        report(kk + 1);
    };
    auto entry = [&](int which, int64_t r, int64_t col) {
        if constexpr (LAZY) return ld_entry<N>(F, sh, sh.coef[which], r, col, pf, (int)(k - pf));
        else return F.at(r, col);
    };
    while (k <= pl) {
        const int cnt = LAZY ? (int)(k - pf) : 0;
        if (t == 0) sh.nan_at = -1;
        if (LAZY) {
            ld_stage_coef<N>(F, sh, sh.coef[0], k, pf, cnt);
            __syncthreads();
        }
        // ---- pivot choice (ldlt.jl:183-219 / 451-508)
        int bs = 1;
        int64_t piv = k;
        mf<N> held = zero;  // the entry of this thread's first row below k
        int64_t held_row = -1;
        {
            mf<N> best = zero;
            int bi = -1;
            if (k < n - 1) {
                for (int64_t r = mine; r < n; r += total) {
                    if (r <= k) continue;
                    const mf<N> e = entry(0, r, k);
                    if (held_row < 0) {
                        held = e;
                        held_row = r;
                    }
                    // a NaN is never strictly larger; in the first row nothing
                    // is strictly larger than it
                    if (r == k + 1 || !isnan(e.v[0])) ld_better(best, bi, abs_mf(e), (int)r);
                }
            }
            if (t == LD_NT - 1) ld_put<N>(sh.val[0], entry(0, k, k));
            __syncwarp();
            ld_reduce<N>(sh, 0, rank, nc, best, bi);
            const mf<N> absakk = abs_mf(ld_get<N>(sh.val[0]));
            if (k == n - 1) {
                if (iszero(absakk)) bs = 0;
            } else if (iszero(max_mf(absakk, best))) {
                bs = 0;
            } else if (!ge(absakk, mul(alpha, best))) {
                const int64_t imax = bi;
                if (LAZY) {
                    ld_stage_coef<N>(F, sh, sh.coef[1], imax, pf, cnt);
                    for (int i = t; i < cnt; i += LD_NT) ld_put<N>(sh.rowi[i], F.at(imax, pf + i));
                    __syncthreads();
                }
                // max |entry| along row imax of the active matrix.  max(x, y)
                // is y where x is NaN (an elimination that overflowed), so the
                // fold of ldlt.jl:203-209 is the maximum of what follows the
                // last NaN: a second scan takes that.  The candidates carry
                // their positions: every pair then has one winner, whatever
                // the values, and all threads of the cluster agree on the
                // branches below.
                mf<N> rowmax;
                for (int from = -1;;) {
                    rowmax = zero;
                    int ri = -1, nan_at = -1;
                    for (int64_t c = mine; c < n; c += total) {
                        if (c < k || c == imax || c <= from) continue;
                        mf<N> e;
                        if (c > imax) e = entry(1, c, imax);
                        else if constexpr (LAZY) e = ld_row_entry<N>(F, sh, imax, c, pf, cnt);
                        else e = F.at(imax, c);
                        if (isnan(e.v[0])) nan_at = (int)c;
                        else ld_better(rowmax, ri, abs_mf(e), (int)c);
                    }
                    if (t == LD_NT - 1) ld_put<N>(sh.val[1], entry(1, imax, imax));
                    if (nan_at >= 0)
                        for (int q = 0; q < nc; ++q)
                            ld_remote_max(ld_remote(&sh.nan_at, (uint32_t)q), nan_at);
                    __syncwarp();
                    ld_reduce<N>(sh, 1, rank, nc, rowmax, ri);
                    if (ri < 0) rowmax = from_double<N>(nan(""));  // nothing follows the NaN
                    if (sh.nan_at == from) break;
                    from = sh.nan_at;
                    ld_cluster_sync();  // the readers of the candidates and of nan_at are done
                }
                if (!ge(absakk, mul(mul(alpha, best), div_call(best, rowmax)))) {
                    piv = imax;
                    bs = ge(abs_mf(ld_get<N>(sh.val[1])), mul(alpha, rowmax)) ? 1 : 2;
                }
            }
        }
        if (bs == 0) return fail(k);
        if (LAZY ? (bs == 2 && k == pl) : bs == 2) {
            if (!(k < n - 1)) return fail(k);
            if (LAZY) pl += 1;
        }
        if (bs == 1) {
            if (writer) {
                F.pivots[k] = piv + 1;
                F.blocks[k] = 1;
            }
            if (piv != k) {
                ld_sym_swap<N>(F, k, piv, k, rank * LD_NT + t, total);
                ld_cluster_sync();
                if (LAZY) {
                    ld_stage_coef<N>(F, sh, sh.coef[0], k, pf, cnt);
                    __syncthreads();
                }
                held_row = -1;
                for (int64_t r = mine; r < n && held_row < 0; r += total)
                    if (r > k) {
                        held = entry(0, r, k);
                        held_row = r;
                    }
                if (t == LD_NT - 1) ld_put<N>(sh.val[0], entry(0, k, k));
                __syncthreads();
            }
            const mf<N> d = ld_get<N>(sh.val[0]);
            if (iszero(d)) return fail(k);
            for (int64_t r = mine; r < n; r += total)
                if (r > k) F.put(r, k, div_call(r == held_row ? held : entry(0, r, k), d));
            if (LAZY && t == 0) {
                sh.type[cnt] = 1;
                ld_put<N>(sh.d[cnt], d);
            }
            ld_cluster_sync();
            if (LAZY) {
                if (writer) F.put(k, k, d);
            } else if (k < n - 1) {
                // rank-1 update of the lower active part with its mirror, one
                // column per warp
                for (int64_t col = k + 1 + rank + (int64_t)nc * warp; col < n; col += nc * LD_WARPS) {
                    const mf<N> coef = mul(d, F.at(col, k));
                    for (int64_t row = col + lane; row < n; row += 32) {
                        const mf<N> v = submul(F.at(row, col), F.at(row, k), coef);
                        F.put(row, col, v);
                        F.put(col, row, v);
                    }
                }
                ld_cluster_sync();
            }
            k += 1;
        } else {
            if (writer) {
                F.pivots[k] = piv + 1;
                F.blocks[k] = 2;
                F.blocks[k + 1] = 0;
            }
            if (piv != k + 1) {
                ld_sym_swap<N>(F, k + 1, piv, k, rank * LD_NT + t, total);
                ld_cluster_sync();
            }
            __syncthreads();  // the readers of val and coef[1] are done
            if (LAZY) {
                ld_stage_coef<N>(F, sh, sh.coef[1], k + 1, pf, cnt);
                __syncthreads();
            }
            // the block's three entries on a lane each, beside the rows' pairs
            if (lane == 31 && warp >= LD_WARPS - 3) {
                const int w = warp - (LD_WARPS - 3);
                ld_put<N>(sh.val[w], w == 0 ? entry(0, k, k)
                                            : w == 1 ? entry(0, k + 1, k) : entry(1, k + 1, k + 1));
            }
            __syncwarp();
            mf<N> e1 = zero, e2 = zero;
            held_row = -1;
            for (int64_t r = mine; r < n && held_row < 0; r += total)
                if (r > k + 1) {
                    e1 = entry(0, r, k);
                    e2 = entry(1, r, k + 1);
                    held_row = r;
                }
            __syncthreads();
            const mf<N> d11 = ld_get<N>(sh.val[0]), d21 = ld_get<N>(sh.val[1]),
                        d22 = ld_get<N>(sh.val[2]);
            // the block's quotients on the last warp, the first row's scaled
            // pair beside them
            const mf<N> scale = max_mf(max_mf(abs_mf(d11), abs_mf(d21)), abs_mf(d22));
            mf<N> r1 = zero, r2 = zero;
            if (warp == LD_WARPS - 1) ld_block<N>(sh, d11, d21, d22);
            __syncwarp();
            if (held_row >= 0) {
                r1 = div_call(e1, scale);
                r2 = div_call(e2, scale);
            }
            __syncthreads();
            const bool regular = sh.regular != 0;
            if (regular)
                for (int64_t r = mine; r < n; r += total) {
                    if (r <= k + 1) continue;
                    if (r != held_row) {
                        r1 = div_call(entry(0, r, k), scale);
                        r2 = div_call(entry(1, r, k + 1), scale);
                    }
                    mf<N> x1, x2;
                    ld_block_solve<N>(sh, r1, r2, x1, x2);
                    if (!(isfinite_mf(x1) && isfinite_mf(x2))) {
                        for (int q = 0; q < nc; ++q)
                            ld_remote_s32(ld_remote(&sh.flag, (uint32_t)q), 1);
                    } else {
                        F.put(r, k, x1);
                        F.put(r, k + 1, x2);
                    }
                }
            if (LAZY && t == 0) {
                sh.type[cnt] = 2;
                sh.type[cnt + 1] = 0;
                ld_put<N>(sh.d[cnt], d11);
                ld_put<N>(sh.d[cnt + 1], d22);
                ld_put<N>(sh.ds[cnt], d21);
            }
            ld_cluster_sync();
            if (writer) {
                if (LAZY) {
                    F.put(k, k, d11);
                    F.put(k + 1, k + 1, d22);
                }
                F.set_ds(k, d21);
            }
            if (!regular || sh.flag) return fail(k);
            if (!LAZY && k + 1 < n - 1) {
                // rank-2 update (ldlt.jl:261-326): rows in full groups of four
                // from the column use v - (f1 c1 + f2 c2), the remainder rows
                // (v - f1 c1) - f2 c2
                for (int64_t col = k + 2 + rank + (int64_t)nc * warp; col < n; col += nc * LD_WARPS) {
                    const mf<N> l1 = F.at(col, k), l2 = F.at(col, k + 1);
                    const mf<N> c1 = add(mul(d11, l1), mul(d21, l2));
                    const mf<N> c2 = add(mul(d21, l1), mul(d22, l2));
                    const int64_t grouped = col + 4 * ((n - col) / 4);
                    for (int64_t row = col + lane; row < n; row += 32) {
                        const mf<N> v0 = F.at(row, col), f1 = F.at(row, k), f2 = F.at(row, k + 1);
                        const mf<N> v = row < grouped
                                            ? sub(v0, add(mul(f1, c1), mul(f2, c2)))
                                            : submul(submul(v0, f1, c1), f2, c2);
                        F.put(row, col, v);
                        F.put(col, row, v);
                    }
                }
                ld_cluster_sync();
            }
            if (writer) {
                F.put(k + 1, k, zero);
                F.put(k, k + 1, zero);
            }
            k += 2;
        }
    }
    report(0);
}

// Cluster size: one CTA per 32 rows up to sixteen (the larger sizes that the
// device can place; eight where sixteen cannot be).
template <int N, bool LAZY>
static int launch_ldlt_cluster(const Ldlt<N> &F, const scal<N> &alpha, int64_t pf, int64_t req,
                               int *info, int64_t *status, int64_t rows, cudaStream_t s) {
    auto kern = ldlt_cluster_kernel<N, LAZY>;
    cudaLaunchConfig_t cfg = {};
    cfg.blockDim = dim3(LD_NT);
    cfg.stream = s;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    static std::atomic<unsigned long long> asked{0}, sixteen{0};
    int most = 0;
    if (int rc = largest_cluster((const void *)kern, LD_NT, 0, asked, sixteen, &most)) return rc;
    int nc = 1;
    while (nc < most && nc * 32 < rows) nc *= 2;
    cfg.gridDim = dim3((unsigned)nc);
    attr[0].val.clusterDim.x = (unsigned)nc;
    return record_cuda_error(cudaLaunchKernelEx(&cfg, kern, F, alpha, pf, req, info, status),
                             "sytrf cluster");
}

// W = L21 * D for the panel (ldlt.jl:595-632): one thread per trailing row
template <int N>
__global__ void ldlt_weighted_kernel(Ldlt<N> F, int64_t pf, int64_t pl, Mat W) {
    const int64_t lr = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    const int64_t row = pl + 1 + lr;
    if (row >= F.n) return;
    int64_t q = pf;
    while (q <= pl) {
        const int64_t lc = q - pf;
        if (F.blocks[q] == 1) {
            store_mf<N>(W.p, W.ld, W.ls, lr, lc, mul(F.at(row, q), F.at(q, q)));
            q += 1;
        } else {
            const mf<N> d11 = F.at(q, q), d21 = F.ds(q), d22 = F.at(q + 1, q + 1);
            const mf<N> f = F.at(row, q), s = F.at(row, q + 1);
            store_mf<N>(W.p, W.ld, W.ls, lr, lc, add(mul(f, d11), mul(s, d21)));
            store_mf<N>(W.p, W.ld, W.ls, lr, lc + 1, add(mul(f, d21), mul(s, d22)));
            q += 2;
        }
    }
}

// upper mirror of a square block: A(c, r) = A(r, c) for r > c
template <int N>
__global__ void mirror_kernel(int64_t n, Mat A, const int *info) {
    if (info && *info) return;
    const int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (e >= n * n) return;
    const int64_t r = e % n, c = e / n;
    if (r <= c) return;
#pragma unroll
    for (int l = 0; l < N; ++l) A.p[l * A.ls + r * A.ld + c] = A.p[l * A.ls + c * A.ld + r];
}

template <int N>
__global__ void ldlt_init_kernel(int64_t n, Mat A, double *dsub, int64_t lsd, int64_t *pivots,
                                 uint8_t *blocks, int *info) {
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    pivots[i] = i + 1;
    blocks[i] = 0;
#pragma unroll
    for (int l = 0; l < N; ++l) dsub[l * lsd + i] = 0.0;
}

template <int N>
__global__ void ldlt_lower_nonfinite_kernel(int64_t n, Mat A, int *info) {
    const int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (e >= n * n) return;
    const int64_t r = e % n, c = e / n;
    if (r < c) return;
    if (!isfinite_mf(load_mf<N>(A.p, A.ld, A.ls, r, c))) *info = -1;
}

template <int N>
__global__ void ldlt_alpha_kernel(double *out) {
    // (1 + sqrt(17)) / 8 in working precision (ldlt.jl:691)
    const mf<N> a = div(add(from_double<N>(1.0), sqrt_mf(from_double<N>(17.0))), from_double<N>(8.0));
#pragma unroll
    for (int l = 0; l < N; ++l) out[l] = a.v[l];
}

template <int N>
static int sytrf_n(mflab_handle *h, int64_t n, Mat A, double *dsub, int64_t lsd, int64_t *pivots,
                   uint8_t *blocks, int blocked, int64_t block, int *info, cudaStream_t s) {
    cudaError_t e = cudaMemsetAsync(info, 0, sizeof(int), s);
    if (e != cudaSuccess) return record_cuda_error(e, "sytrf info");
    if (n == 0) return MFLAB_OK;
    ldlt_init_kernel<N><<<(unsigned)((n + 255) / 256), 256, 0, s>>>(n, A, dsub, lsd, pivots, blocks, info);
    ldlt_lower_nonfinite_kernel<N><<<(unsigned)((n * n + 255) / 256), 256, 0, s>>>(n, A, info);
    mirror_kernel<N><<<(unsigned)((n * n + 255) / 256), 256, 0, s>>>(n, A, info);
    int rc = record_cuda_error(cudaGetLastError(), "sytrf prepare");
    if (rc) return rc;
    // alpha in working precision, read back once
    const size_t wbytes = sizeof(double) * (size_t)N * (size_t)n * (size_t)(block + 1);
    rc = mflab_reserve_scratch(h, wbytes + 256 + 64);
    if (rc) return rc;
    double *W = (double *)h->scratch;
    double *alpha_dev = (double *)((char *)h->scratch + (wbytes + 255) / 256 * 256);
    int64_t *st_dev = (int64_t *)(alpha_dev + 4);
    ldlt_alpha_kernel<N><<<1, 1, 0, s>>>(alpha_dev);
    scal<N> al{};
    double alpha_host[4] = {0, 0, 0, 0};
    e = cudaMemcpyAsync(alpha_host, alpha_dev, sizeof(double) * N, cudaMemcpyDeviceToHost, s);
    if (e == cudaSuccess) e = cudaStreamSynchronize(s);
    if (e != cudaSuccess) return record_cuda_error(e, "sytrf alpha");
    for (int l = 0; l < N; ++l) al.v[l] = alpha_host[l];
    Ldlt<N> F{A, n, dsub, lsd, pivots, blocks};
    if (!blocked) return launch_ldlt_cluster<N, false>(F, al, 0, n - 1, info, st_dev, n, s);
    const double mone[4] = {-1.0, 0.0, 0.0, 0.0}, one[4] = {1.0, 0.0, 0.0, 0.0};
    int64_t pf = 0;
    while (pf < n) {
        const int64_t req = pf + block - 1 < n - 1 ? pf + block - 1 : n - 1;
        rc = launch_ldlt_cluster<N, true>(F, al, pf, req, info, st_dev, n - pf, s);
        if (rc) return rc;
        int64_t status[2] = {0, 0};
        e = cudaMemcpyAsync(status, st_dev, sizeof(status), cudaMemcpyDeviceToHost, s);
        if (e == cudaSuccess) e = cudaStreamSynchronize(s);
        if (e != cudaSuccess) return record_cuda_error(e, "sytrf panel status");
        if (status[1]) return MFLAB_OK;
        const int64_t pl = status[0];
        if (pl < n - 1) {
            const int64_t tc = n - 1 - pl, pw = pl - pf + 1;
            Mat Wm{W, n, n * (block + 1)};
            ldlt_weighted_kernel<N><<<(unsigned)((tc + 127) / 128), 128, 0, s>>>(F, pf, pl, Wm);
            rc = record_cuda_error(cudaGetLastError(), "sytrf weighted");
            if (rc) return rc;
            rc = launch_mm(N, false, true, 1, false, tc, tc, pw, A.at(pl + 1, pf), Wm,
                           A.at(pl + 1, pl + 1), mone, one, s, info);
            if (rc) return rc;
            mirror_kernel<N><<<(unsigned)((tc * tc + 255) / 256), 256, 0, s>>>(tc, A.at(pl + 1, pl + 1), info);
            rc = record_cuda_error(cudaGetLastError(), "sytrf mirror");
            if (rc) return rc;
        }
        pf = pl + 1;
    }
    return MFLAB_OK;
}

// ------------------------------------------------------------ solve -------
// forward (reverse == 0) / reverse row interchanges (solve.jl:213-249);
// one thread per right-hand-side column
template <int N>
__global__ void ldlt_pivots_kernel(int64_t n, int64_t nrhs, Mat B, const int64_t *pivots,
                                   const uint8_t *blocks, int reverse) {
    const int64_t c = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (c >= nrhs) return;
    auto swap = [&](int64_t a, int64_t b) {
        if (a == b) return;
#pragma unroll
        for (int l = 0; l < N; ++l) {
            double *x = B.p + l * B.ls + c * B.ld;
            const double t = x[a];
            x[a] = x[b];
            x[b] = t;
        }
    };
    if (!reverse) {
        int64_t k = 0;
        while (k < n) {
            if (blocks[k] == 1) {
                swap(k, pivots[k] - 1);
                k += 1;
            } else {
                swap(k + 1, pivots[k] - 1);
                k += 2;
            }
        }
    } else {
        int64_t k = n - 1;
        while (k >= 0) {
            if (blocks[k] == 1) {
                swap(k, pivots[k] - 1);
                k -= 1;
            } else {
                swap(k, pivots[k - 1] - 1);
                k -= 2;
            }
        }
    }
}

// The same interchanges, one CTA per right-hand-side column: one thread replays
// them on an index array in shared memory (a swap there is two reads, not two
// rounds to L2), then the column is gathered.  x3, n = 600, 5 columns: 30 us
// (286 us with the swaps in the column itself).
constexpr int64_t LDLT_GATHER_MAXN = 12000;  // 16 bytes a row of shared memory

// Many short columns pay for a CTA each and take the kernel above, a thread per
// column.  us of a whole solve, gather / thread: x2, 8 rows 1000 columns 81 / 80,
// 10000 156 / 118; x2, 30 rows 3000 columns 184 / 183, 10000 306 / 272; x2, 150
// rows 10000 columns 4885 / 4920, 30000 5701 / 5535; x4, 100 rows 10000 columns
// 6666 / 6776, 30000 10369 / 10293.  Longer columns: within 1 % at any count.
static bool ldlt_gathers(int64_t n, int64_t nrhs) {
    if (n <= 8 || n > LDLT_GATHER_MAXN) return false;
    return n > 200 || nrhs <= (n <= 32 ? 3000 : 20000);
}

template <int N>
__global__ void __launch_bounds__(256)
    ldlt_gather_kernel(int64_t n, Mat B, const int64_t *pivots, const uint8_t *blocks, int reverse) {
    extern __shared__ double gather_raw[];
    double *buf = gather_raw;        // [n] one limb of the column
    int *idx = (int *)(buf + n);     // [n] source row of every row
    int *with = idx + n;             // [n] step k exchanges rows k and with[k]
    for (int64_t i = threadIdx.x; i < n; i += blockDim.x) {
        idx[i] = (int)i;
        // the second row of a 2x2 block is the one exchanged (marker 0)
        with[i] = (int)(blocks[i] == 1 ? pivots[i] - 1 : blocks[i] == 2 || i == 0 ? i : pivots[i - 1] - 1);
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        for (int64_t s = 0; s < n; ++s) {
            const int64_t k = reverse ? n - 1 - s : s;
            const int p = with[k];
            if (p != (int)k) {
                const int t = idx[k];
                idx[k] = idx[p];
                idx[p] = t;
            }
        }
    }
    for (int l = 0; l < N; ++l) {
        double *x = B.p + l * B.ls + (int64_t)blockIdx.x * B.ld;
        for (int64_t i = threadIdx.x; i < n; i += blockDim.x) buf[i] = x[i];
        __syncthreads();
        for (int64_t i = threadIdx.x; i < n; i += blockDim.x) x[i] = buf[idx[i]];
        __syncthreads();
    }
}

template <int N>
static int ldlt_interchange(int64_t n, int64_t nrhs, Mat B, const int64_t *pivots,
                            const uint8_t *blocks, int reverse, cudaStream_t s) {
    if (ldlt_gathers(n, nrhs)) {
        static std::atomic<unsigned long long> configured{0};
        if (int rc = set_smem_once((const void *)ldlt_gather_kernel<N>, (int)(16 * LDLT_GATHER_MAXN),
                                   configured, "sytrs interchange attribute"))
            return rc;
        ldlt_gather_kernel<N><<<(unsigned)nrhs, 256, (size_t)(16 * n), s>>>(n, B, pivots, blocks,
                                                                           reverse);
    } else {
        ldlt_pivots_kernel<N><<<(unsigned)((nrhs + 127) / 128), 128, 0, s>>>(n, nrhs, B, pivots,
                                                                             blocks, reverse);
    }
    return record_cuda_error(cudaGetLastError(), "sytrs interchange");
}

// D solve (solve.jl:251-296): independent per (block, column)
template <int N>
__global__ void ldlt_dsolve_kernel(int64_t n, int64_t nrhs, Mat F, const double *dsub,
                                   int64_t lsd, const uint8_t *blocks, Mat B, int *fail) {
    const int64_t k = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    const int64_t c = blockIdx.y;
    if (k >= n || c >= nrhs) return;
    if (blocks[k] == 1) {
        store_mf<N>(B.p, B.ld, B.ls, k, c,
                    div(load_mf<N>(B.p, B.ld, B.ls, k, c), load_mf<N>(F.p, F.ld, F.ls, k, k)));
    } else if (blocks[k] == 2) {
        mf<N> d21;
#pragma unroll
        for (int l = 0; l < N; ++l) d21.v[l] = dsub[l * lsd + k];
        mf<N> x1, x2;
        const bool ok = solve_2x2(load_mf<N>(F.p, F.ld, F.ls, k, k), d21,
                                  load_mf<N>(F.p, F.ld, F.ls, k + 1, k + 1),
                                  load_mf<N>(B.p, B.ld, B.ls, k, c),
                                  load_mf<N>(B.p, B.ld, B.ls, k + 1, c), x1, x2);
        if (!ok) {
            atomicMin(fail, (int)(k + 1));
        } else {
            store_mf<N>(B.p, B.ld, B.ls, k, c, x1);
            store_mf<N>(B.p, B.ld, B.ls, k + 1, c, x2);
        }
    }
}

// ----------------------------------------------------- diagnostics --------
// One thread: inertia, block counts and block quality of an LDLT factor
// (diagnostics.jl:109-246).  out: [0] positive [1] negative [2] zero
// [3] 1x1 count [4] 2x2 count [5] has-min-block, then N-limb values
// min block eigenvalue magnitude, max block entry.
template <int N>
__global__ void ldlt_diag_kernel(int64_t n, Mat F, const double *dsub, int64_t lsd,
                                 const uint8_t *blocks, const double *omax, double *out) {
    int64_t pos = 0, neg = 0, zer = 0, one = 0, two = 0;
    bool have_min = false;
    mf<N> minb = from_double<N>(0.0), maxe = from_double<N>(0.0);
    const mf<N> z = from_double<N>(0.0);
    int64_t k = 0;
    while (k < n) {
        const uint8_t b = blocks[k];
        if (b == 1) {
            const mf<N> v = load_mf<N>(F.p, F.ld, F.ls, k, k);
            if (gt(v, z)) pos++;
            else if (lt(v, z)) neg++;
            else zer++;
            one++;
            const mf<N> bv = abs_mf(v);
            minb = have_min ? min_mf(minb, bv) : bv;
            have_min = true;
            maxe = max_mf(maxe, bv);
            k += 1;
        } else if (b == 2 && k < n - 1) {
            two++;
            const mf<N> d11 = load_mf<N>(F.p, F.ld, F.ls, k, k);
            const mf<N> d22 = load_mf<N>(F.p, F.ld, F.ls, k + 1, k + 1);
            mf<N> d21;
#pragma unroll
            for (int l = 0; l < N; ++l) d21.v[l] = dsub[l * lsd + k];
            const mf<N> scale = max_mf(max_mf(abs_mf(d11), abs_mf(d21)), abs_mf(d22));
            // inertia of the 2x2 block (diagnostics.jl:118-134)
            if (iszero(scale)) {
                zer += 2;
            } else {
                const mf<N> a = div(d11, scale), bb = div(d21, scale), c = div(d22, scale);
                const mf<N> det = sub(mul(a, c), mul(bb, bb));
                const mf<N> tr = add(a, c);
                if (lt(det, z)) {
                    pos++;
                    neg++;
                } else if (gt(det, z)) {
                    if (gt(tr, z)) pos += 2;
                    else neg += 2;
                } else {
                    if (gt(tr, z)) {
                        pos++;
                        zer++;
                    } else if (lt(tr, z)) {
                        neg++;
                        zer++;
                    } else {
                        zer += 2;
                    }
                }
            }
            // smallest |eigenvalue| of the block (diagnostics.jl:136-154)
            mf<N> bv = z;
            if (!iszero(scale)) {
                const mf<N> a = div(d11, scale), bb = div(d21, scale), c = div(d22, scale);
                const mf<N> amc = sub(a, c);
                const mf<N> disc = sqrt_mf(add(mul(amc, amc), mul(mul(from_double<N>(4.0), bb), bb)));
                const mf<N> first = div(add(add(a, c), disc), from_double<N>(2.0));
                const mf<N> second = div(sub(add(a, c), disc), from_double<N>(2.0));
                const mf<N> largest = max_mf(abs_mf(first), abs_mf(second));
                if (!iszero(largest)) {
                    const mf<N> det = abs_mf(sub(mul(a, c), mul(bb, bb)));
                    bv = mul(scale, div(det, largest));
                }
            }
            minb = have_min ? min_mf(minb, bv) : bv;
            have_min = true;
            maxe = max_mf(max_mf(max_mf(maxe, abs_mf(d11)), abs_mf(d21)), abs_mf(d22));
            k += 2;
        } else {
            break;
        }
    }
    out[0] = (double)pos;
    out[1] = (double)neg;
    out[2] = (double)zer;
    out[3] = (double)one;
    out[4] = (double)two;
    out[5] = have_min ? 1.0 : 0.0;
    mf<N> om;
#pragma unroll
    for (int l = 0; l < N; ++l) om.v[l] = omax ? omax[l] : 0.0;
    const bool omz = iszero(om);
    const mf<N> scaled = (omz || !have_min) ? z : div(minb, om);
    const mf<N> growth = omz ? z : div(maxe, om);
#pragma unroll
    for (int l = 0; l < N; ++l) {
        out[6 + l] = minb.v[l];
        out[6 + N + l] = maxe.v[l];
        out[6 + 2 * N + l] = scaled.v[l];
        out[6 + 3 * N + l] = growth.v[l];
    }
}

}  // namespace mfl

using mfl::Mat;

extern "C" int mflab_sytrf(mflab_handle *h, void *stream, int limbs, int64_t n, double *A,
                           int64_t lda, int64_t lsa, double *dsub, int64_t lsd, int64_t *pivots,
                           uint8_t *blocks, int blocked, int64_t block, int *info) {
    MFLAB_RANGE("mflab_sytrf");
    if (!h || !mfl::valid_limbs(limbs)) return MFLAB_ERR_UNSUPPORTED;
    if (n < 0 || (n > 0 && (lda < n || !dsub || !pivots || !blocks || lsd < n)) || !info)
        return MFLAB_ERR_ARG;
    if (blocked && block < 2) block = 2;
    if (block > 64) return MFLAB_ERR_UNSUPPORTED;
    Mat a{A, lda, lsa};
    cudaStream_t s = (cudaStream_t)stream;
    switch (limbs) {
    case 2: return mfl::sytrf_n<2>(h, n, a, dsub, lsd, pivots, blocks, blocked, block, info, s);
    case 3: return mfl::sytrf_n<3>(h, n, a, dsub, lsd, pivots, blocks, blocked, block, info, s);
    default: return mfl::sytrf_n<4>(h, n, a, dsub, lsd, pivots, blocks, blocked, block, info, s);
    }
}

extern "C" int mflab_sytrs(mflab_handle *h, void *stream, int limbs, int64_t n, int64_t nrhs,
                           const double *F, int64_t ldf, int64_t lsf, const double *dsub,
                           int64_t lsd, const int64_t *pivots, const uint8_t *blocks, double *B,
                           int64_t ldb, int64_t lsb, int *fail) {
    MFLAB_RANGE("mflab_sytrs");
    if (!h || !mfl::valid_limbs(limbs)) return MFLAB_ERR_UNSUPPORTED;
    if (n < 0 || nrhs < 0 || (n > 0 && (ldf < n || ldb < n)) || !fail) return MFLAB_ERR_ARG;
    if (n == 0 || nrhs == 0) return MFLAB_OK;
    if (nrhs > 65535) return MFLAB_ERR_UNSUPPORTED;
    const double one[4] = {1.0, 0.0, 0.0, 0.0};
    cudaStream_t s = (cudaStream_t)stream;
    Mat f{(double *)F, ldf, lsf}, b{B, ldb, lsb};
    cudaError_t e = cudaMemsetAsync(fail, 0x7f, sizeof(int), s);  // 0x7f7f7f7f = no failure
    if (e != cudaSuccess) return mfl::record_cuda_error(e, "sytrs flag");
    const dim3 gd((unsigned)((n + 127) / 128), (unsigned)nrhs);
    auto interchange = [&](int reverse) {
        switch (limbs) {
        case 2: return mfl::ldlt_interchange<2>(n, nrhs, b, pivots, blocks, reverse, s);
        case 3: return mfl::ldlt_interchange<3>(n, nrhs, b, pivots, blocks, reverse, s);
        default: return mfl::ldlt_interchange<4>(n, nrhs, b, pivots, blocks, reverse, s);
        }
    };
    int rc = interchange(0);
    if (rc) return rc;
    rc = mfl::launch_trsm_info(limbs, 0, 0, 0, 1, n, nrhs, f, b, one, s, nullptr, h->solve_order);
    if (rc) return rc;
    switch (limbs) {
    case 2: mfl::ldlt_dsolve_kernel<2><<<gd, 128, 0, s>>>(n, nrhs, f, dsub, lsd, blocks, b, fail); break;
    case 3: mfl::ldlt_dsolve_kernel<3><<<gd, 128, 0, s>>>(n, nrhs, f, dsub, lsd, blocks, b, fail); break;
    default: mfl::ldlt_dsolve_kernel<4><<<gd, 128, 0, s>>>(n, nrhs, f, dsub, lsd, blocks, b, fail); break;
    }
    rc = mfl::launch_trsm_info(limbs, 0, 0, 1, 1, n, nrhs, f, b, one, s, nullptr, h->solve_order);
    if (rc) return rc;
    rc = mfl::record_cuda_error(cudaGetLastError(), "sytrs");
    return rc ? rc : interchange(1);
}

extern "C" int mflab_ldlt_diagnostics(mflab_handle *h, void *stream, int limbs, int64_t n,
                                      const double *F, int64_t ldf, int64_t lsf,
                                      const double *dsub, int64_t lsd, const uint8_t *blocks,
                                      const double *omax, double *out) {
    MFLAB_RANGE("mflab_ldlt_diagnostics");
    if (!h || !mfl::valid_limbs(limbs)) return MFLAB_ERR_UNSUPPORTED;
    if (n < 0 || !out) return MFLAB_ERR_ARG;
    Mat f{(double *)F, ldf, lsf};
    cudaStream_t s = (cudaStream_t)stream;
    switch (limbs) {
    case 2: mfl::ldlt_diag_kernel<2><<<1, 1, 0, s>>>(n, f, dsub, lsd, blocks, omax, out); break;
    case 3: mfl::ldlt_diag_kernel<3><<<1, 1, 0, s>>>(n, f, dsub, lsd, blocks, omax, out); break;
    default: mfl::ldlt_diag_kernel<4><<<1, 1, 0, s>>>(n, f, dsub, lsd, blocks, omax, out); break;
    }
    return mfl::record_cuda_error(cudaGetLastError(), "ldlt diagnostics");
}
