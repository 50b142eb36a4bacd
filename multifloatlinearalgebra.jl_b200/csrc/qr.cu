// Householder QR, rank-revealing QR, apply_q! and numerical_rank
// (src/factorizations/qr.jl of MultiFloatLinearAlgebra.jl).
//
// Every result is the reference's element by element: column norms are the
// sequential scaled sum of squares (qr.jl:96-122), each reflector
// application is one ascending projection chain per column (qr.jl:624-642),
// and the rank-revealing path follows the reference's two routes, the
// hybrid pivot search for small problems (qr.jl:192-224, 364-398) and the
// DLAQPS-style panel with delayed updates, norm downdates and panel breaks
// (qr.jl:450-604), whose end-of-panel update is the matched GEMM kernel.
//
// Parallel structure: what the reference's order makes sequential is the
// additions of a column norm and of each projection chain; one lane adds while
// the other warps form the quotients, squares and products it adds next.
// Norm state lives in device planes and a panel break is a device word that
// the panel's later steps read first, so the host waits once per panel.
#include "mf_device.cuh"
#include "mflab_internal.h"

namespace mfl {

constexpr int QR_BLOCK = 16;          // _QR_BLOCK_SIZE, qr.jl:306
constexpr int QR_CTA = 256;           // single-CTA kernels
constexpr int QR_COLS_PER_CTA = 64;   // one column per thread

template <int N>
struct QRNorms {
    double *scale;  // N planes of n
    double *sum;    // N planes of n
    int *dirty;     // n
    int64_t n;
    __device__ mf<N> sc(int64_t c) const {
        mf<N> x;
#pragma unroll
        for (int l = 0; l < N; ++l) x.v[l] = scale[l * n + c];
        return x;
    }
    __device__ mf<N> su(int64_t c) const {
        mf<N> x;
#pragma unroll
        for (int l = 0; l < N; ++l) x.v[l] = sum[l * n + c];
        return x;
    }
    __device__ void set(int64_t c, const mf<N> &s, const mf<N> &u) const {
#pragma unroll
        for (int l = 0; l < N; ++l) {
            scale[l * n + c] = s.v[l];
            sum[l * n + c] = u.v[l];
        }
    }
    __device__ void set_sum(int64_t c, const mf<N> &u) const {
#pragma unroll
        for (int l = 0; l < N; ++l) sum[l * n + c] = u.v[l];
    }
    __device__ void swap(int64_t a, int64_t b) const {
        if (a == b) return;
#pragma unroll
        for (int l = 0; l < N; ++l) {
            double t = scale[l * n + a];
            scale[l * n + a] = scale[l * n + b];
            scale[l * n + b] = t;
            t = sum[l * n + a];
            sum[l * n + a] = sum[l * n + b];
            sum[l * n + b] = t;
        }
        const int d = dirty[a];
        dirty[a] = dirty[b];
        dirty[b] = d;
    }
};

// _qr_column_norm_state / _qr_delayed_column_norm_state (qr.jl:96-122,
// 226-262): rows r0..m-1 of column c, each value first corrected by
// value -= A[row, bs + p] * F[p, c] for p < prior
template <int N>
__device__ void norm_state(const Mat &A, int64_t m, int64_t r0, int64_t c, const Mat &F,
                           int64_t bs, int64_t prior, mf<N> &scale, mf<N> &sum) {
    const mf<N> one = from_double<N>(1.0);
    scale = from_double<N>(0.0);
    sum = one;
    bool seen = false;
    for (int64_t r = r0; r < m; ++r) {
        mf<N> v = load_mf<N>(A.p, A.ld, A.ls, r, c);
        for (int64_t p = 0; p < prior; ++p)
            v = submul(v, load_mf<N>(A.p, A.ld, A.ls, r, bs + p), load_mf<N>(F.p, F.ld, F.ls, p, c));
        const mf<N> mag = abs_mf(v);
        if (iszero(mag)) continue;
        if (!seen) {
            scale = mag;
            sum = one;
            seen = true;
        } else if (gt(mag, scale)) {
            const mf<N> ratio = div(scale, mag);
            sum = add(one, mul(mul(sum, ratio), ratio));
            scale = mag;
        } else {
            const mf<N> ratio = div(mag, scale);
            sum = add(sum, mul(ratio, ratio));
        }
    }
}

// The same scaled sum of squares computed by one warp, bit for bit: per chunk
// of 32 rows the lanes load their magnitudes, a warp scan gives every row the
// running maximum before it (the reference's `scale` at that row: the scale
// only ever moves to a new maximum), each lane forms its ratio and square in
// parallel, and lane 0 folds the chunk in row order with the reference's own
// operations (sum += ratio^2, or sum = 1 + sum*ratio*ratio at a new maximum,
// or sum = 1 at the first nonzero).  The divisions and products leave the
// sequential path; only the additions stay on it.  All 32 lanes must call it;
// buf is this warp's shared scratch of QR_NORM_BUF(N) doubles.
#define QR_NORM_BUF(N) (32 * (3 * (N) + 1))
template <int N>
__device__ void norm_state_warp(const Mat &A, int64_t m, int64_t r0, int64_t c, double *buf,
                                mf<N> &scale, mf<N> &sum) {
    const unsigned FULL = 0xffffffffu;
    const int lane = threadIdx.x & 31;
    const mf<N> one = from_double<N>(1.0), zero = from_double<N>(0.0);
    scale = zero;
    sum = one;
    bool seen = false;
    double *bmag = buf, *brat = buf + 32 * N, *bsq = buf + 64 * N;
    int *bflag = (int *)(buf + 96 * N);
    for (int64_t base = r0; base < m; base += 32) {
        const int64_t r = base + lane;
        const mf<N> mag = r < m ? abs_mf(load_mf<N>(A.p, A.ld, A.ls, r, c)) : zero;
        const bool nz = !iszero(mag);
        // inclusive running maximum over the lanes, then shifted by one and
        // merged with the scale carried from the previous chunks
        mf<N> pm = mag;
#pragma unroll
        for (int off = 1; off < 32; off <<= 1) {
            mf<N> o;
#pragma unroll
            for (int l = 0; l < N; ++l) o.v[l] = __shfl_up_sync(FULL, pm.v[l], off);
            if (lane >= off && gt(o, pm)) pm = o;
        }
        mf<N> before;
#pragma unroll
        for (int l = 0; l < N; ++l) before.v[l] = __shfl_up_sync(FULL, pm.v[l], 1);
        if (lane == 0 || gt(scale, before)) before = scale;
        const bool isnew = nz && gt(mag, before);
        mf<N> ratio = zero, sq = zero;
        if (nz && !iszero(before)) {
            ratio = isnew ? div(before, mag) : div(mag, before);
            sq = mul(ratio, ratio);
        }
#pragma unroll
        for (int l = 0; l < N; ++l) {
            bmag[l * 32 + lane] = mag.v[l];
            brat[l * 32 + lane] = ratio.v[l];
            bsq[l * 32 + lane] = sq.v[l];
        }
        bflag[lane] = (nz ? 1 : 0) | (isnew ? 2 : 0);
        __syncwarp();
        if (lane == 0) {
            for (int i = 0; i < 32; ++i) {
                const int f = bflag[i];
                if (!(f & 1)) continue;
                mf<N> mi, ri, si;
#pragma unroll
                for (int l = 0; l < N; ++l) {
                    mi.v[l] = bmag[l * 32 + i];
                    ri.v[l] = brat[l * 32 + i];
                    si.v[l] = bsq[l * 32 + i];
                }
                if (!seen) {
                    scale = mi;
                    sum = one;
                    seen = true;
                } else if (f & 2) {
                    sum = add(one, mul(mul(sum, ri), ri));
                    scale = mi;
                } else {
                    sum = add(sum, si);
                }
            }
        }
        __syncwarp();
#pragma unroll
        for (int l = 0; l < N; ++l) {
            scale.v[l] = __shfl_sync(FULL, scale.v[l], 0);
            sum.v[l] = __shfl_sync(FULL, sum.v[l], 0);
        }
        seen = __shfl_sync(FULL, seen ? 1 : 0, 0) != 0;
    }
}

// _qr_norm_from_state (qr.jl:157-165)
template <int N>
__device__ __forceinline__ mf<N> norm_value(const mf<N> &scale, const mf<N> &sum) {
    return iszero(scale) ? from_double<N>(0.0) : mul(scale, sqrt_mf(sum));
}

__global__ void qr_finite_kernel_init(int *flag) { *flag = 0; }

template <int N>
__global__ void qr_finite_kernel(int64_t m, int64_t n, Mat A, int *flag) {
    bool bad = false;
    const int64_t total = m * n;
    for (int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; e < total;
         e += (int64_t)gridDim.x * blockDim.x) {
        const int64_t c = e / m, r = e % m;
#pragma unroll
        for (int l = 0; l < N; ++l) bad = bad || !isfinite(A.p[l * A.ls + c * A.ld + r]);
    }
    if (__syncthreads_or(bad) && threadIdx.x == 0) atomicExch(flag, 1);
}

// _qr_make_reflector! (qr.jl:606-622) for column s; tau at tau[l * lt + s].
// blocked != 0 (the DLAQPS panel, qr.jl:513-515): afterwards save A[s,s] to
// diag and set A[s,s] = 1.
//
// The bound is the norm's chain of m - s additions (90 cycles each in x2), so
// nothing else is left on it.  The reference's running scale is the running
// maximum of the magnitudes, which eight warps find with a scan: each of 256
// rows then has its ratio and square at once, and what its row does to the sum
// is a flag.  The ninth warp's first lane folds tile t in row order while the
// eight form tile t + 1.  x2, m = 500: 37 us a column, 23 of them the chain;
// 127 us with one warp for both and the projections on the earlier panel
// columns behind it (these are now column chains beside the trailing ones).
constexpr int QRR_TILE = 256, QRR_NT = QRR_TILE + 32;
enum : unsigned char { QRR_SKIP = 0, QRR_ADD = 1, QRR_RAISE = 2, QRR_FIRST = 3 };

// scale and sum of squares of rows r0..m-1 of column c by a CTA of QRR_NT
// threads; the first thread of the last warp has the result
template <int N>
__device__ __forceinline__ void cta_norm(const Mat &A, int64_t m, int64_t r0, int64_t c,
                                         mf<N> &scale, mf<N> &sum) {
    __shared__ double val[2][N][QRR_TILE];  // squares (QRR_ADD) or ratios (QRR_RAISE)
    __shared__ unsigned char flag[2][QRR_TILE];
    __shared__ unsigned plain[2][QRR_TILE / 32];  // rows of a group that only add
    __shared__ double wmax[QRR_TILE / 32][N], carry[2][N];
    const unsigned FULL = 0xffffffffu;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const mf<N> one = from_double<N>(1.0), zero = from_double<N>(0.0);
    const int64_t tiles = (m - r0 + QRR_TILE - 1) / QRR_TILE;
    if (tid < N) carry[0][tid] = 0.0;
    __syncthreads();

    auto produce = [&](int64_t t) {  // warps 0 .. 7
        const int b = (int)(t & 1);
        const int64_t r = r0 + t * QRR_TILE + tid;
        const mf<N> mag = r < m ? abs_mf(load_mf<N>(A.p, A.ld, A.ls, r, c)) : zero;
        const bool nz = !iszero(mag);
        mf<N> pm = mag;  // running maximum within the warp
#pragma unroll
        for (int off = 1; off < 32; off <<= 1) {
            mf<N> o;
#pragma unroll
            for (int l = 0; l < N; ++l) o.v[l] = __shfl_up_sync(FULL, pm.v[l], off);
            if (lane >= off && gt(o, pm)) pm = o;
        }
        if (lane == 31)
#pragma unroll
            for (int l = 0; l < N; ++l) wmax[warp][l] = pm.v[l];
        asm volatile("bar.sync 1, %0;" ::"n"(QRR_TILE) : "memory");
        mf<N> base;  // the maximum before this warp's rows
#pragma unroll
        for (int l = 0; l < N; ++l) base.v[l] = carry[b][l];
        for (int w = 0; w < warp; ++w) {
            mf<N> o;
#pragma unroll
            for (int l = 0; l < N; ++l) o.v[l] = wmax[w][l];
            if (gt(o, base)) base = o;
        }
        mf<N> before;
#pragma unroll
        for (int l = 0; l < N; ++l) before.v[l] = __shfl_up_sync(FULL, pm.v[l], 1);
        if (lane == 0 || gt(base, before)) before = base;
        unsigned char f = QRR_SKIP;
        mf<N> x = zero;
        if (nz) {
            if (iszero(before)) {
                f = QRR_FIRST;
            } else if (gt(mag, before)) {
                f = QRR_RAISE;
                x = div(before, mag);
            } else {
                f = QRR_ADD;
                x = div(mag, before);
                x = mul(x, x);
            }
        }
#pragma unroll
        for (int l = 0; l < N; ++l) val[b][l][tid] = x.v[l];
        flag[b][tid] = f;
        const unsigned p = __ballot_sync(FULL, f == QRR_ADD);
        if (lane == 0) plain[b][warp] = p;
        if (tid == QRR_TILE - 1) {
            if (gt(base, pm)) pm = base;
#pragma unroll
            for (int l = 0; l < N; ++l) carry[b ^ 1][l] = pm.v[l];
        }
    };

    sum = one;
    if (warp < QRR_TILE / 32) produce(0);
    for (int64_t t = 0; t < tiles; ++t) {
        __syncthreads();
        if (warp == QRR_TILE / 32) {
            if (lane == 0) {
                const int b = (int)(t & 1);
                for (int g = 0; g < QRR_TILE / 32; ++g) {
                    auto get = [&](int i) {
                        mf<N> x;
#pragma unroll
                        for (int l = 0; l < N; ++l) x.v[l] = val[b][l][g * 32 + i];
                        return x;
                    };
                    if (plain[b][g] == FULL) {
#pragma unroll 8
                        for (int i = 0; i < 32; ++i) sum = add(sum, get(i));
                    } else {
                        for (int i = 0; i < 32; ++i) {
                            const unsigned char f = flag[b][g * 32 + i];
                            if (f == QRR_SKIP) continue;
                            const mf<N> x = get(i);
                            if (f == QRR_FIRST) sum = one;
                            else if (f == QRR_RAISE) sum = add(one, mul(mul(sum, x), x));
                            else sum = add(sum, x);
                        }
                    }
                }
            }
        } else if (t + 1 < tiles) {
            produce(t + 1);
        }
    }
    __syncthreads();
#pragma unroll
    for (int l = 0; l < N; ++l) scale.v[l] = carry[tiles & 1][l];
}

// Columns of fewer than QRR_ROWS rows (TALL false) leave the norm to the last
// warp: the nine warps' scan and barriers cost more than the chain.  us a step,
// whole factorization, TALL / not: 40 rows and fewer 21 / 13, 80 rows 29 / 27,
// 90 rows 31 / 31, 120 rows 32 / 36 (x2); x4 5 rows 58 / 48, 80 rows 76 / 76, 120
// rows 90 / 100.
constexpr int64_t QRR_ROWS = 88;

template <int N, bool TALL>
__global__ void __launch_bounds__(QRR_NT)
    qr_reflector_kernel(int64_t m, int64_t s, Mat A, double *tau, int64_t lt, int blocked,
                        double *diag, const int *stop) {
    // every step's kernels are programmatic dependents of one another: wait
    // for the previous grid, let the next one be placed
    asm volatile("griddepcontrol.wait;" ::: "memory");
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    if (stop && *stop != 0 && *stop <= (int)s) return;
    __shared__ double slead[N];
    __shared__ int go;
    const mf<N> one = from_double<N>(1.0), zero = from_double<N>(0.0);
    const int tid = threadIdx.x;
    mf<N> scale, sum;
    if constexpr (TALL) {
        cta_norm<N>(A, m, s, s, scale, sum);
    } else {
        __shared__ double nbuf[QR_NORM_BUF(N)];
        if (tid >= QRR_TILE) norm_state_warp<N>(A, m, s, s, nbuf, scale, sum);
    }
    if (tid == QRR_TILE) {
        const mf<N> nrm = norm_value(scale, sum);
        mf<N> t = zero;
        go = 0;
        if (!iszero(nrm)) {
            const mf<N> alpha = load_mf<N>(A.p, A.ld, A.ls, s, s);
            const mf<N> beta = ge(alpha, zero) ? neg(nrm) : nrm;
            const mf<N> lead = sub(alpha, beta);
            t = div(sub(beta, alpha), beta);
#pragma unroll
            for (int l = 0; l < N; ++l) slead[l] = lead.v[l];
            store_mf<N>(A.p, A.ld, A.ls, s, s, beta);
            go = 1;
        }
#pragma unroll
        for (int l = 0; l < N; ++l) tau[l * lt + s] = t.v[l];
    }
    __syncthreads();
    if (go) {
        mf<N> lead;
#pragma unroll
        for (int l = 0; l < N; ++l) lead.v[l] = slead[l];
        for (int64_t r = s + 1 + tid; r < m; r += QRR_NT)
            store_mf<N>(A.p, A.ld, A.ls, r, s, div(load_mf<N>(A.p, A.ld, A.ls, r, s), lead));
    }
    if (blocked && tid == 0) {
        const mf<N> d = load_mf<N>(A.p, A.ld, A.ls, s, s);
#pragma unroll
        for (int l = 0; l < N; ++l) diag[l] = d.v[l];
        store_mf<N>(A.p, A.ld, A.ls, s, s, one);
    }
}

// acc folded over rows r0..m-1 in ascending order, acc = acc + X[r,cx] *
// Y[r,cy], by one warp: the lanes form 32 products at a time, lane 0 adds
// them in row order (the reference's chain; only the additions are
// sequential) while the next 32 rows' operands are on their way.  All 32
// lanes call it; buf holds 32 N doubles of this warp; the result is returned
// in every lane.  U additions are unrolled: a kernel that runs one reflector of
// a short column spends more on fetching the longer x4 loop than it saves.
template <int N, int U>
__device__ mf<N> chain_warp(mf<N> acc, int64_t r0, int64_t m, const Mat &X, int64_t cx,
                            const Mat &Y, int64_t cy, double *buf) {
    const unsigned FULL = 0xffffffffu;
    const int lane = threadIdx.x & 31;
    mf<N> x = from_double<N>(0.0), y = x;
    auto fetch = [&](int64_t r) {
        if (r < m) {
            x = load_mf<N>(X.p, X.ld, X.ls, r, cx);
            y = load_mf<N>(Y.p, Y.ld, Y.ls, r, cy);
        }
    };
    fetch(r0 + lane);
    for (int64_t base = r0; base < m; base += 32) {
        const mf<N> pr = mul(x, y);  // of a row past the end: never added
#pragma unroll
        for (int l = 0; l < N; ++l) buf[l * 32 + lane] = pr.v[l];
        __syncwarp();
        fetch(base + 32 + lane);
        if (lane == 0) {
            auto term = [&](int i) {
                mf<N> p;
#pragma unroll
                for (int l = 0; l < N; ++l) p.v[l] = buf[l * 32 + i];
                acc = add(acc, p);
            };
            const int cnt = m - base < 32 ? (int)(m - base) : 32;
            if (cnt == 32) {
#pragma unroll U
                for (int i = 0; i < 32; ++i) term(i);
            } else {
                for (int i = 0; i < cnt; ++i) term(i);
            }
        }
        __syncwarp();
    }
#pragma unroll
    for (int l = 0; l < N; ++l) acc.v[l] = __shfl_sync(FULL, acc.v[l], 0);
    return acc;
}

// reflector s of V (implicit one at row s) applied to column c of D by one
// warp (qr.jl:624-642): the projection chain, then the rank-one update with
// the rows spread over the lanes
template <int N, int U = 8>
__device__ __forceinline__ void apply_reflector_col_warp(int64_t m, int64_t s, const Mat &V,
                                                         const mf<N> &t, const Mat &D, int64_t c,
                                                         double *buf) {
    const int lane = threadIdx.x & 31;
    mf<N> proj = chain_warp<N, U>(load_mf<N>(D.p, D.ld, D.ls, s, c), s + 1, m, V, s, D, c, buf);
    proj = mul(proj, t);
    if (lane == 0) store_mf<N>(D.p, D.ld, D.ls, s, c, sub(load_mf<N>(D.p, D.ld, D.ls, s, c), proj));
    for (int64_t r = s + 1 + lane; r < m; r += 32)
        store_mf<N>(D.p, D.ld, D.ls, r, c,
                    submul(load_mf<N>(D.p, D.ld, D.ls, r, c), load_mf<N>(V.p, V.ld, V.ls, r, s), proj));
    __syncwarp();
}

constexpr int QR_COL_WARPS = 4;  // columns (one warp each) per CTA

static inline unsigned warp_col_grid(int64_t cols) {
    return (unsigned)((cols + QR_COL_WARPS - 1) / QR_COL_WARPS);
}

// x4 columns of fewer than QR_SHORT_ROWS rows (SHORT) unroll less: 64 x 20
// 1367 -> 1318 us, 300 x 300 30.9 -> 30.6 ms; 1000 x 100 would take 42.8 ms, not
// 42.5.
constexpr int64_t QR_SHORT_ROWS = 300;

template <int N, bool SHORT>
__global__ void __launch_bounds__(32 * QR_COL_WARPS)
    qr_apply_kernel(int64_t m, int64_t s, Mat V, const double *tau, int64_t lt, Mat D, int64_t c0,
                    int64_t nd) {
    asm volatile("griddepcontrol.wait;" ::: "memory");
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    __shared__ double buf[QR_COL_WARPS][32 * N];
    const int w = threadIdx.x >> 5;
    const int64_t j = (int64_t)blockIdx.x * QR_COL_WARPS + w;
    if (j >= nd) return;  // whole warps leave together
    mf<N> t;
#pragma unroll
    for (int l = 0; l < N; ++l) t.v[l] = tau[l * lt + s];
    if (iszero(t)) return;
    apply_reflector_col_warp<N, SHORT ? 2 : 8>(m, s, V, t, D, c0 + j, buf[w]);
}

// apply_q! (qr.jl:890-956): every reflector in order on one column of D
template <int N>
__global__ void __launch_bounds__(32 * QR_COL_WARPS)
    qr_apply_all_warp_kernel(int64_t m, int64_t r, Mat V, const double *tau, int64_t lt, Mat D,
                             int64_t nd, int trans) {
    __shared__ double buf[QR_COL_WARPS][32 * N];
    const int w = threadIdx.x >> 5;
    const int64_t c = (int64_t)blockIdx.x * QR_COL_WARPS + w;
    if (c >= nd) return;
    for (int64_t i = 0; i < r; ++i) {
        const int64_t s = trans ? i : r - 1 - i;
        mf<N> t;
#pragma unroll
        for (int l = 0; l < N; ++l) t.v[l] = tau[l * lt + s];
        if (iszero(t)) continue;
        apply_reflector_col_warp<N>(m, s, V, t, D, c, buf[w]);
    }
}

// The same, one CTA per column.  r reflectors are r chains of m - s additions
// one after another; the ninth warp's first lane runs them while eight warps
// form the next 256 products, and all nine apply the update.  Taken for up to
// QR_APPLY_CTAS columns: the chains of CTAs that share an SM share one of its
// four schedulers (40 of a chain's 90 cycles an addition are issue in x2), so
// beyond two of them the warp kernel above is the faster one.  x2, m = 500,
// 40 reflectors, 3 columns: 977 us (1257 us with a warp per column).
constexpr int64_t QR_APPLY_CTAS = 2 * 148;

template <int N>
__global__ void __launch_bounds__(QRR_NT)
    qr_apply_all_kernel(int64_t m, int64_t r, Mat V, const double *tau, int64_t lt, Mat D,
                        int trans) {
    __shared__ double buf[2][N][QRR_TILE];
    __shared__ double sproj[N];
    const int tid = threadIdx.x, warp = tid >> 5;
    const int64_t c = blockIdx.x;
    for (int64_t i = 0; i < r; ++i) {
        const int64_t s = trans ? i : r - 1 - i;
        mf<N> t;
#pragma unroll
        for (int l = 0; l < N; ++l) t.v[l] = tau[l * lt + s];
        if (iszero(t)) continue;  // the same in every thread
        const int64_t r0 = s + 1, tiles = (m - r0 + QRR_TILE - 1) / QRR_TILE;
        auto produce = [&](int64_t b) {
            const int64_t row = r0 + b * QRR_TILE + tid;
            if (row >= m) return;
            const mf<N> p = mul(load_mf<N>(V.p, V.ld, V.ls, row, s),
                                load_mf<N>(D.p, D.ld, D.ls, row, c));
#pragma unroll
            for (int l = 0; l < N; ++l) buf[b & 1][l][tid] = p.v[l];
        };
        mf<N> acc;
        if (tid == QRR_TILE) acc = load_mf<N>(D.p, D.ld, D.ls, s, c);
        if (warp < QRR_TILE / 32 && tiles > 0) produce(0);
        for (int64_t b = 0; b < tiles; ++b) {
            __syncthreads();
            if (tid == QRR_TILE) {
                auto term = [&](int k) {
                    mf<N> p;
#pragma unroll
                    for (int l = 0; l < N; ++l) p.v[l] = buf[b & 1][l][k];
                    acc = add(acc, p);
                };
                const int64_t left = m - r0 - b * QRR_TILE;
                const int cnt = left < QRR_TILE ? (int)left : QRR_TILE;
                int k = 0;
                for (; k + 8 <= cnt; k += 8)
#pragma unroll
                    for (int q = 0; q < 8; ++q) term(k + q);
                for (; k < cnt; ++k) term(k);
            } else if (warp < QRR_TILE / 32 && b + 1 < tiles) {
                produce(b + 1);
            }
        }
        if (tid == QRR_TILE) {
            const mf<N> proj = mul(acc, t);
#pragma unroll
            for (int l = 0; l < N; ++l) sproj[l] = proj.v[l];
            store_mf<N>(D.p, D.ld, D.ls, s, c, sub(load_mf<N>(D.p, D.ld, D.ls, s, c), proj));
        }
        __syncthreads();
        mf<N> proj;
#pragma unroll
        for (int l = 0; l < N; ++l) proj.v[l] = sproj[l];
        for (int64_t row = r0 + tid; row < m; row += QRR_NT)
            store_mf<N>(D.p, D.ld, D.ls, row, c,
                        submul(load_mf<N>(D.p, D.ld, D.ls, row, c),
                               load_mf<N>(V.p, V.ld, V.ls, row, s), proj));
        __syncthreads();  // the column and sproj before the next reflector
    }
}

// norm state of columns c0..n-1 from rows r0 (qr.jl:143-155, 417-448): a CTA per
// column from QR_NORM_ROWS rows on, where the column's own chain bounds it, else
// a warp per column.  Many columns fill the FP64 pipe with either, and the
// warp's divisions, 32 at a time, then cost less: the line lies at two columns
// per SM in x2, one in x3 and x4.  us, CTA / warp:
//   x2  32 x 40 15 / 7, 128 x 40 18 / 21, 500 x 40 34 / 79, 500 x 296 43 / 80,
//       500 x 592 79 / 81, 500 x 1200 124 / 94;
//   x4  128 x 40 40 / 51, 500 x 148 109 / 189, 500 x 296 217 / 194.
// rrqr 500 x 40 in x2 3.42 -> 3.30 ms, 2000 x 40 10.35 -> 9.82 ms.
constexpr int QR_NORM_WARPS = 4, QR_NORM_ROWS = 128;

template <int N>
__global__ void __launch_bounds__(QRR_NT)
    qr_norm_init_kernel(int64_t m, int64_t r0, int64_t c0, Mat A, QRNorms<N> S) {
    const int64_t c = c0 + blockIdx.x;
    mf<N> scale, sum;
    cta_norm<N>(A, m, r0, c, scale, sum);
    if (threadIdx.x == QRR_TILE) {
        S.set(c, scale, sum);
        S.dirty[c] = 0;
    }
}

template <int N>
__global__ void __launch_bounds__(32 * QR_NORM_WARPS)
    qr_norm_init_warp_kernel(int64_t m, int64_t r0, int64_t c0, Mat A, QRNorms<N> S) {
    __shared__ double nbuf[QR_NORM_WARPS][QR_NORM_BUF(N)];
    const int w = threadIdx.x >> 5;
    const int64_t c = c0 + (int64_t)blockIdx.x * QR_NORM_WARPS + w;
    if (c >= S.n) return;  // whole warps leave together
    mf<N> scale, sum;
    norm_state_warp<N>(A, m, r0, c, nbuf[w], scale, sum);
    if ((threadIdx.x & 31) == 0) {
        S.set(c, scale, sum);
        S.dirty[c] = 0;
    }
}

template <int N>
static void launch_norm_init(int64_t m, int64_t r0, int64_t c0, const Mat &A, const QRNorms<N> &S,
                             cudaStream_t s) {
    const int64_t cols = S.n - c0;
    if (m - r0 >= QR_NORM_ROWS && cols <= (N == 2 ? 2 * 148 : 148))
        qr_norm_init_kernel<N><<<(unsigned)cols, QRR_NT, 0, s>>>(m, r0, c0, A, S);
    else
        qr_norm_init_warp_kernel<N><<<(unsigned)((cols + QR_NORM_WARPS - 1) / QR_NORM_WARPS),
                                      32 * QR_NORM_WARPS, 0, s>>>(m, r0, c0, A, S);
}

// _qr_update_norm_state! for one column (qr.jl:264-304)
template <int N>
__device__ void update_norm_col(int64_t m, int64_t step, int64_t c, const Mat &A,
                                const QRNorms<N> &S, const mf<N> &floor_, const Mat &F,
                                int64_t bs, int64_t prior) {
    if (S.dirty[c]) return;
    const mf<N> scale = S.sc(c);
    const mf<N> removed = abs_mf(load_mf<N>(A.p, A.ld, A.ls, step, c));
    if (iszero(scale)) {
        S.dirty[c] = !iszero(removed);
        return;
    }
    const mf<N> ratio = div(removed, scale);
    const mf<N> ns = sub(S.su(c), mul(ratio, ratio));
    if (!isfinite_mf(ns) || ge(floor_, ns)) {
        mf<N> sc, su;
        norm_state<N>(A, m, step + 1, c, F, bs, prior, sc, su);
        S.set(c, sc, su);
        S.dirty[c] = 0;
    } else {
        S.set_sum(c, ns);
    }
}

template <int N>
__global__ void __launch_bounds__(QR_COLS_PER_CTA)
    qr_update_norms_kernel(int64_t m, int64_t step, Mat A, const double *tau, int64_t lt,
                           QRNorms<N> S, scal<N> floor_) {
    asm volatile("griddepcontrol.wait;" ::: "memory");
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    const int64_t c = step + 1 + (int64_t)blockIdx.x * QR_COLS_PER_CTA + threadIdx.x;
    if (c >= S.n) return;
    mf<N> t;
#pragma unroll
    for (int l = 0; l < N; ++l) t.v[l] = tau[l * lt + step];
    if (iszero(t)) return;
    const Mat none{nullptr, 1, 1};
    update_norm_col<N>(m, step, c, A, S, floor_.get(), none, 0, 0);
}

template <int N>
__device__ void swap_columns_cta(int64_t m, const Mat &A, int64_t a, int64_t b) {
    if (a == b) return;
    for (int64_t r = threadIdx.x; r < m; r += blockDim.x)
#pragma unroll
        for (int l = 0; l < N; ++l) {
            double *pa = A.p + l * A.ls + a * A.ld + r, *pb = A.p + l * A.ls + b * A.ld + r;
            const double t = *pa;
            *pa = *pb;
            *pb = t;
        }
}

// _qr_select_pivot_hybrid! (qr.jl:192-224) on thread 0, then the column,
// permutation and norm-state swaps (qr.jl:376-386)
template <int N>
__global__ void __launch_bounds__(QR_CTA)
    qr_hybrid_pivot_kernel(int64_t m, int64_t step, Mat A, int64_t *perm, QRNorms<N> S,
                           scal<N> one_minus_margin) {
    asm volatile("griddepcontrol.wait;" ::: "memory");
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    __shared__ int64_t sp;
    __shared__ double nbuf[QR_NORM_BUF(N)];
    if (threadIdx.x < 32) {
        // warp 0 walks the columns in order; every lane takes the same
        // branches (the state it reads is the same), lane 0 writes
        const bool w0 = threadIdx.x == 0;
        const mf<N> om = one_minus_margin.get();
        int64_t piv = step;
        mf<N> sc, su;
        norm_state_warp<N>(A, m, step, step, nbuf, sc, su);
        if (w0) {
            S.set(step, sc, su);
            S.dirty[step] = 0;
        }
        __syncwarp();
        mf<N> pn = norm_value(sc, su);
        for (int64_t c = step + 1; c < S.n; ++c) {
            mf<N> cn = norm_value(S.sc(c), S.su(c));
            if (S.dirty[c] || iszero(pn) || ge(cn, mul(om, pn))) {
                norm_state_warp<N>(A, m, step, c, nbuf, sc, su);
                __syncwarp();
                if (w0) {
                    S.set(c, sc, su);
                    S.dirty[c] = 0;
                }
                __syncwarp();
                cn = norm_value(sc, su);
            }
            bool eq = true;
#pragma unroll
            for (int l = 0; l < N; ++l) eq = eq && cn.v[l] == pn.v[l];
            if (gt(cn, pn) || (eq && perm[c] < perm[piv])) {
                piv = c;
                pn = cn;
            }
        }
        if (w0) sp = piv;
    }
    __syncthreads();
    const int64_t piv = sp;
    swap_columns_cta<N>(m, A, step, piv);
    if (threadIdx.x == 0 && piv != step) {
        const int64_t t = perm[step];
        perm[step] = perm[piv];
        perm[piv] = t;
        S.swap(step, piv);
    }
}

constexpr int QR_PIVOT_CTA = 1024;

// DLAQPS step head (qr.jl:478-511): downdated pivot choice (largest norm
// from the state, smallest original column on ties), the column swap with
// its F entries, permutation and norm state, then the delayed prefix on the
// chosen column
template <int N>
__global__ void __launch_bounds__(QR_PIVOT_CTA)
    qr_dlaqps_pivot_kernel(int64_t m, int64_t step, int64_t bs, int64_t ls, Mat A, int64_t *perm,
                           QRNorms<N> S, Mat F, const int *stop) {
    asm volatile("griddepcontrol.wait;" ::: "memory");
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    if (*stop != 0 && *stop <= (int)step) return;
    __shared__ double sval[N][QR_PIVOT_CTA];
    __shared__ int64_t sidx[QR_PIVOT_CTA];
    const int tid = threadIdx.x;
    int64_t bi = -1;
    mf<N> bv = from_double<N>(0.0);
    for (int64_t c = step + tid; c < S.n; c += QR_PIVOT_CTA) {
        const mf<N> v = norm_value(S.sc(c), S.su(c));
        bool eq = true;
#pragma unroll
        for (int l = 0; l < N; ++l) eq = eq && v.v[l] == bv.v[l];
        if (bi < 0 || gt(v, bv) || (eq && perm[c] < perm[bi])) {
            bi = c;
            bv = v;
        }
    }
#pragma unroll
    for (int l = 0; l < N; ++l) sval[l][tid] = bv.v[l];
    sidx[tid] = bi;
    __syncthreads();
    int width = 32;  // threads that hold a column
    while (width < QR_PIVOT_CTA && width < S.n - step) width <<= 1;
    for (int s = width / 2; s > 0; s >>= 1) {
        if (tid < s && sidx[tid + s] >= 0) {
            const int64_t ia = sidx[tid], ib = sidx[tid + s];
            mf<N> va, vb;
#pragma unroll
            for (int l = 0; l < N; ++l) {
                va.v[l] = sval[l][tid];
                vb.v[l] = sval[l][tid + s];
            }
            bool eq = true;
#pragma unroll
            for (int l = 0; l < N; ++l) eq = eq && va.v[l] == vb.v[l];
            if (ia < 0 || gt(vb, va) || (eq && perm[ib] < perm[ia])) {
#pragma unroll
                for (int l = 0; l < N; ++l) sval[l][tid] = vb.v[l];
                sidx[tid] = ib;
            }
        }
        __syncthreads();
    }
    const int64_t piv = sidx[0];
    swap_columns_cta<N>(m, A, step, piv);
    if (piv != step) {
        for (int64_t e = tid; e < ls * N; e += QR_PIVOT_CTA) {
            const int64_t p = e / N;
            const int l = (int)(e % N);
            double *fa = F.p + l * F.ls + step * F.ld + p, *fb = F.p + l * F.ls + piv * F.ld + p;
            const double t = *fa;
            *fa = *fb;
            *fb = t;
        }
    }
    __syncthreads();
    if (tid == 0 && piv != step) {
        const int64_t t = perm[step];
        perm[step] = perm[piv];
        perm[piv] = t;
        S.swap(step, piv);
    }
    if (ls > 0)
        for (int64_t r = step + tid; r < m; r += QR_PIVOT_CTA) {
            mf<N> corr = from_double<N>(0.0);
#pragma unroll 4
            for (int64_t p = 0; p < ls; ++p)
                corr = mac<N, false>(corr, load_mf<N>(A.p, A.ld, A.ls, r, bs + p),
                                     load_mf<N>(F.p, F.ld, F.ls, p, step));
            store_mf<N>(A.p, A.ld, A.ls, r, step, sub(load_mf<N>(A.p, A.ld, A.ls, r, step), corr));
        }
}

// DLAQPS step body after the column chains acc[j] = sum_r A[r, bs+j] v[r]
// (gemv! trans = :T), one trailing column per thread (qr.jl:517-576): aux[p]
// = -tau acc[p] of the earlier panel columns, the new F row, the R row and
// the norm downdate.  A column left unreliable ends the panel after this
// step: *stop = step + 1, read by every later step of the panel.
template <int N>
__global__ void __launch_bounds__(QR_COLS_PER_CTA)
    qr_dlaqps_columns_kernel(int64_t m, int64_t step, int64_t bs, int64_t ls, Mat A,
                             const double *tau, int64_t lt, const double *chains, Mat F,
                             QRNorms<N> S, scal<N> floor_, int *stop) {
    asm volatile("griddepcontrol.wait;" ::: "memory");
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    if (*stop != 0 && *stop <= (int)step) return;
    // the panel's entries the correction loops read, staged so that no load
    // waits inside a chain
    __shared__ double aux[QR_BLOCK][N], row[QR_BLOCK][N];
    __shared__ double Fs[QR_BLOCK][N][QR_COLS_PER_CTA];
    const int tid = threadIdx.x;
    const int64_t c = step + 1 + (int64_t)blockIdx.x * QR_COLS_PER_CTA + tid;
    mf<N> t;
#pragma unroll
    for (int l = 0; l < N; ++l) t.v[l] = tau[l * lt + step];
    if (tid <= ls) {
        const mf<N> x = load_mf<N>(A.p, A.ld, A.ls, step, bs + tid);
#pragma unroll
        for (int l = 0; l < N; ++l) row[tid][l] = x.v[l];
    }
    if (tid < ls) {
        const mf<N> a = mul(neg(t), load_mf<N>(chains, 0, S.n, tid, 0));
#pragma unroll
        for (int l = 0; l < N; ++l) aux[tid][l] = a.v[l];
    }
    mf<N> chain = from_double<N>(0.0), old = chain;
    if (c < S.n) {
        chain = load_mf<N>(chains, 0, S.n, c - bs, 0);
        old = load_mf<N>(A.p, A.ld, A.ls, step, c);
#pragma unroll 4
        for (int64_t p = 0; p < ls; ++p) {
            const mf<N> f = load_mf<N>(F.p, F.ld, F.ls, p, c);
#pragma unroll
            for (int l = 0; l < N; ++l) Fs[p][l][tid] = f.v[l];
        }
    }
    __syncthreads();
    if (c >= S.n) return;
    auto Fat = [&](int64_t p) {
        mf<N> f;
#pragma unroll
        for (int l = 0; l < N; ++l) f.v[l] = Fs[p][l][tid];
        return f;
    };
    auto get = [&](const double *v) {
        mf<N> x;
#pragma unroll
        for (int l = 0; l < N; ++l) x.v[l] = v[l];
        return x;
    };
    mf<N> f = mul(t, chain);
    if (ls > 0) {
        mf<N> corr = from_double<N>(0.0);
        for (int64_t p = 0; p < ls; ++p) corr = mac<N, false>(corr, Fat(p), get(aux[p]));
        f = add(f, corr);
    }
    store_mf<N>(F.p, F.ld, F.ls, ls, c, f);
    mf<N> corr = from_double<N>(0.0);
    for (int64_t p = 0; p < ls; ++p) corr = mac<N, false>(corr, get(row[p]), Fat(p));
    corr = mac<N, false>(corr, get(row[ls]), f);
    store_mf<N>(A.p, A.ld, A.ls, step, c, sub(old, corr));
    if (!iszero(t)) update_norm_col<N>(m, step, c, A, S, floor_.get(), F, bs, ls + 1);
    if (S.dirty[c]) atomicExch(stop, (int)step + 1);
}

// the panel's diagonal entries back in place of the ones, for the steps that ran
__global__ void qr_restore_diag_kernel(int N, Mat A, int64_t bs, int64_t req, const double *diag,
                                       const int *stop) {
    const int64_t actual = *stop ? *stop - bs : req;
    const int64_t i = threadIdx.x;
    if (i >= actual) return;
    for (int l = 0; l < N; ++l) A.p[l * A.ls + (bs + i) * A.ld + bs + i] = diag[i * N + l];
}

__global__ void qr_identity_kernel(int64_t n, int64_t *perm) {
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) perm[i] = i + 1;
}

// numerical_rank (qr.jl:863-888)
template <int N>
__global__ void qr_rank_kernel(int64_t r, Mat F, scal<N> atol, scal<N> rtol, int64_t *rank) {
    mf<N> largest = from_double<N>(0.0);
    for (int64_t i = 0; i < r; ++i)
        largest = max_mf(largest, abs_mf(load_mf<N>(F.p, F.ld, F.ls, i, i)));
    const mf<N> thr = max_mf(atol.get(), mul(rtol.get(), largest));
    int64_t k = 0;
    for (; k < r; ++k)
        if (!gt(abs_mf(load_mf<N>(F.p, F.ld, F.ls, k, k)), thr)) break;
    *rank = k;
}

static inline unsigned col_grid(int64_t cols) {
    return (unsigned)((cols + QR_COLS_PER_CTA - 1) / QR_COLS_PER_CTA);
}

template <int N>
static int qr_n(mflab_handle *h, cudaStream_t s, int pivoted, int64_t m, int64_t n, Mat A,
                double *tau, int64_t lt, int64_t *perm, int *info) {
    const int64_t r = m < n ? m : n;
    // scratch: norm planes, F (QR_BLOCK x n), column chains, panel diagonal, flags
    const size_t nn = (size_t)(n > 0 ? n : 1);
    const size_t doubles = 2 * N * nn + (size_t)N * QR_BLOCK * nn + N * nn + QR_BLOCK * N;
    const size_t bytes = doubles * sizeof(double) + (nn + 4) * sizeof(int);
    int rc = mflab_reserve_scratch(h, bytes);
    if (rc) return rc;
    double *base = (double *)h->scratch;
    QRNorms<N> S{base, base + N * nn, nullptr, n};
    double *Fp = base + 2 * N * nn;
    const Mat F{Fp, QR_BLOCK, (int64_t)(QR_BLOCK * nn)};
    double *chains = Fp + (size_t)N * QR_BLOCK * nn;
    double *diag = chains + N * nn;
    S.dirty = (int *)(diag + QR_BLOCK * N);
    int *flag = S.dirty + nn;

    cudaError_t e = cudaSuccess;
    for (int l = 0; l < N; ++l) {
        e = cudaMemsetAsync(tau + l * lt, 0, r * sizeof(double), s);
        if (e != cudaSuccess) return record_cuda_error(e, "qr tau");
    }
    // identity permutation, finiteness
    {
        if (n > 0) qr_identity_kernel<<<(unsigned)((n + 255) / 256), 256, 0, s>>>(n, perm);
        qr_finite_kernel_init<<<1, 1, 0, s>>>(flag);
        const int64_t g = (m * n + 255) / 256;
        qr_finite_kernel<N><<<(unsigned)(g < 1184 ? (g > 0 ? g : 1) : 1184), 256, 0, s>>>(m, n, A, flag);
        int fin = 0;
        e = cudaMemcpyAsync(&fin, flag, sizeof(int), cudaMemcpyDeviceToHost, s);
        if (e == cudaSuccess) e = cudaStreamSynchronize(s);
        if (e != cudaSuccess) return record_cuda_error(e, "qr finiteness");
        if (fin) {
            const int neg1 = -1;
            e = cudaMemcpyAsync(info, &neg1, sizeof(int), cudaMemcpyHostToDevice, s);
            if (e == cudaSuccess) e = cudaStreamSynchronize(s);
            return record_cuda_error(e, "qr info");
        }
    }
    auto apply = [&](int64_t st) {
        return N == 4 && m - st < QR_SHORT_ROWS ? qr_apply_kernel<N, N == 4> : qr_apply_kernel<N, false>;
    };
    auto reflector = [&](int64_t st) {
        return m - st >= QRR_ROWS ? qr_reflector_kernel<N, true> : qr_reflector_kernel<N, false>;
    };
    if (!pivoted) {
        // each step's kernels are programmatic dependent launches
        for (int64_t st = 0; st < r; ++st) {
            int rc = launch_programmatic(reflector(st), dim3(1), dim3(QRR_NT), 0, s,
                                         "qr reflector", m, st, A, tau, lt, 0, nullptr, nullptr);
            if (rc) return rc;
            if (st + 1 < n) {
                rc = launch_programmatic(apply(st), dim3(warp_col_grid(n - st - 1)),
                                         dim3(32 * QR_COL_WARPS), 0, s, "qr apply", m, st, A,
                                         (const double *)tau, lt, A, st + 1, n - st - 1);
                if (rc) return rc;
            }
        }
    } else {
        // constants of rrqr! (qr.jl:736-737): margin = sqrt(eps), floor = 16 eps,
        // eps = 2^(-52 N); sqrt and the products are exact powers of two
        scal<N> om{}, fl{};
        om.v[0] = 1.0;
        if (N == 2) {
            om.v[0] = 1.0 - ldexp(1.0, -52);
        } else {
            om.v[1] = -ldexp(1.0, -26 * N);
        }
        fl.v[0] = ldexp(1.0, 4 - 52 * N);
        if (n > 0)
            launch_norm_init<N>(m, 0, 0, A, S, s);
        const bool blocked = r >= QR_BLOCK && m * n >= 16384;
        if (!blocked) {
            for (int64_t st = 0; st < r; ++st) {
                int rc = launch_programmatic(qr_hybrid_pivot_kernel<N>, dim3(1), dim3(QR_CTA), 0,
                                             s, "qr pivot", m, st, A, perm, S, om);
                if (rc == MFLAB_OK)
                    rc = launch_programmatic(reflector(st), dim3(1), dim3(QRR_NT), 0, s,
                                             "qr reflector", m, st, A, tau, lt, 0, nullptr,
                                             nullptr);
                if (rc == MFLAB_OK && st + 1 < n) {
                    rc = launch_programmatic(apply(st), dim3(warp_col_grid(n - st - 1)),
                                             dim3(32 * QR_COL_WARPS), 0, s, "qr apply", m, st, A,
                                             (const double *)tau, lt, A, st + 1, n - st - 1);
                    if (rc == MFLAB_OK)
                        rc = launch_programmatic(
                            qr_update_norms_kernel<N>, dim3(col_grid(n - st - 1)),
                            dim3(QR_COLS_PER_CTA), 0, s, "qr norms", m, st, A,
                            (const double *)tau, lt, S, fl);
                }
                if (rc) return rc;
            }
        } else {
            int64_t bs = 0;
            rc = MFLAB_OK;
            while (bs < r && rc == MFLAB_OK) {
                const int64_t req = (r - bs) < QR_BLOCK ? (r - bs) : QR_BLOCK;
                for (int l = 0; l < N && e == cudaSuccess; ++l)
                    e = cudaMemsetAsync(Fp + l * F.ls, 0, QR_BLOCK * nn * sizeof(double), s);
                if (e == cudaSuccess) e = cudaMemsetAsync(flag, 0, sizeof(int), s);
                if (e != cudaSuccess) {
                    rc = record_cuda_error(e, "qr F");
                    break;
                }
                // the whole panel is issued; after a break its later steps
                // return at once, and the host reads how far it came
                for (int64_t ls = 0; ls < req && rc == MFLAB_OK; ++ls) {
                    const int64_t st = bs + ls;
                    rc = launch_programmatic(qr_dlaqps_pivot_kernel<N>, dim3(1), dim3(QR_PIVOT_CTA),
                                             0, s, "qr panel pivot", m, st, bs, ls, A, perm, S, F,
                                             (const int *)flag);
                    if (rc == MFLAB_OK)
                        rc = launch_programmatic(reflector(st), dim3(1), dim3(QRR_NT), 0,
                                                 s, "qr panel reflector", m, st, A, tau, lt, 1,
                                                 diag + ls * N, (const int *)flag);
                    if (rc == MFLAB_OK && st + 1 < n) {
                        // every panel and trailing column (the step's own is unused)
                        rc = launch_column_chains(N, n - bs, m - st, A.at(st, bs), A.at(st, st),
                                                  Mat{chains, n, n}, s, flag, (int)st);
                        if (rc == MFLAB_OK)
                            rc = launch_programmatic(
                                qr_dlaqps_columns_kernel<N>, dim3(col_grid(n - st - 1)),
                                dim3(QR_COLS_PER_CTA), 0, s, "qr panel columns", m, st, bs, ls, A,
                                (const double *)tau, lt, (const double *)chains, F, S, fl, flag);
                    }
                }
                if (rc) break;
                qr_restore_diag_kernel<<<1, QR_BLOCK, 0, s>>>(N, A, bs, req, diag, flag);
                int stopped = 0;
                e = cudaMemcpyAsync(&stopped, flag, sizeof(int), cudaMemcpyDeviceToHost, s);
                if (e == cudaSuccess) e = cudaStreamSynchronize(s);
                if (e != cudaSuccess) {
                    rc = record_cuda_error(e, "qr panel flag");
                    break;
                }
                const int64_t actual = stopped ? stopped - bs : req;
                const int64_t be = bs + actual;
                if (be < m && be < n) {
                    const double mone[4] = {-1.0, 0.0, 0.0, 0.0}, one[4] = {1.0, 0.0, 0.0, 0.0};
                    rc = launch_mm(N, 0, false, 0, N == 3, m - be, n - be, actual, A.at(be, bs),
                                   Mat{Fp + be * F.ld, F.ld, F.ls}, A.at(be, be), mone, one, s);
                    if (rc) break;
                }
                if (be < n)
                    launch_norm_init<N>(m, be, be, A, S, s);
                bs = be;
            }
            if (rc) return rc;
        }
    }
    e = cudaMemsetAsync(info, 0, sizeof(int), s);
    if (e != cudaSuccess) return record_cuda_error(e, "qr info");
    return record_cuda_error(cudaGetLastError(), "qr launch");
}

template <int N>
static int apply_q_n(int64_t m, int64_t r, Mat F, const double *tau, int64_t lst, Mat D, int64_t nd,
                     int trans, cudaStream_t s) {
    if (nd <= QR_APPLY_CTAS)
        qr_apply_all_kernel<N><<<(unsigned)nd, QRR_NT, 0, s>>>(m, r, F, tau, lst, D, trans);
    else
        qr_apply_all_warp_kernel<N><<<warp_col_grid(nd), 32 * QR_COL_WARPS, 0, s>>>(
            m, r, F, tau, lst, D, nd, trans);
    return record_cuda_error(cudaGetLastError(), "apply_q launch");
}

}  // namespace mfl

using mfl::Mat;

extern "C" int mflab_qr(mflab_handle *h, void *stream, int limbs, int pivoted, int64_t m,
                        int64_t n, double *A, int64_t lda, int64_t lsa, double *tau, int64_t lst,
                        int64_t *perm, int *info) {
    MFLAB_RANGE("mflab_qr");
    if (!h || !mfl::valid_limbs(limbs)) return MFLAB_ERR_UNSUPPORTED;
    if (pivoted & ~1) return MFLAB_ERR_FLAG;
    if (m < 0 || n < 0 || !tau || !perm || !info) return MFLAB_ERR_ARG;
    const int64_t r = m < n ? m : n;
    if ((m > 0 && lda < m) || lst < r) return MFLAB_ERR_ARG;
    const Mat Am{A, lda, lsa};
    cudaStream_t s = (cudaStream_t)stream;
    switch (limbs) {
    case 2: return mfl::qr_n<2>(h, s, pivoted, m, n, Am, tau, lst, perm, info);
    case 3: return mfl::qr_n<3>(h, s, pivoted, m, n, Am, tau, lst, perm, info);
    default: return mfl::qr_n<4>(h, s, pivoted, m, n, Am, tau, lst, perm, info);
    }
}

extern "C" int mflab_apply_q(mflab_handle *h, void *stream, int limbs, int trans, int64_t m,
                             int64_t r, const double *F, int64_t ldf, int64_t lsf,
                             const double *tau, int64_t lst, double *D, int64_t ldd, int64_t lsd,
                             int64_t nd) {
    MFLAB_RANGE("mflab_apply_q");
    if (!h || !mfl::valid_limbs(limbs)) return MFLAB_ERR_UNSUPPORTED;
    if (trans & ~1) return MFLAB_ERR_FLAG;
    if (m < 0 || r < 0 || nd < 0 || r > m) return MFLAB_ERR_ARG;
    if (m == 0 || nd == 0 || r == 0) return MFLAB_OK;
    if (ldf < m || ldd < m || lst < r) return MFLAB_ERR_ARG;
    if (mfl::views_overlap(D, ldd, lsd, m, nd, limbs, F, ldf, lsf, m, r)) return MFLAB_ERR_ALIAS;
    const Mat Fm{(double *)F, ldf, lsf}, Dm{D, ldd, lsd};
    cudaStream_t s = (cudaStream_t)stream;
    switch (limbs) {
    case 2: return mfl::apply_q_n<2>(m, r, Fm, tau, lst, Dm, nd, trans, s);
    case 3: return mfl::apply_q_n<3>(m, r, Fm, tau, lst, Dm, nd, trans, s);
    default: return mfl::apply_q_n<4>(m, r, Fm, tau, lst, Dm, nd, trans, s);
    }
}

extern "C" int mflab_qr_numerical_rank(mflab_handle *h, void *stream, int limbs, int64_t m,
                                       int64_t n, const double *F, int64_t ldf, int64_t lsf,
                                       const double *atol, const double *rtol, int64_t *rank) {
    MFLAB_RANGE("mflab_qr_numerical_rank");
    if (!h || !mfl::valid_limbs(limbs)) return MFLAB_ERR_UNSUPPORTED;
    if (m < 0 || n < 0 || !atol || !rtol || !rank) return MFLAB_ERR_ARG;
    const int64_t r = m < n ? m : n;
    if (r > 0 && ldf < m) return MFLAB_ERR_ARG;
    const Mat Fm{(double *)F, ldf, lsf};
    cudaStream_t s = (cudaStream_t)stream;
    switch (limbs) {
    case 2: {
        mfl::scal<2> a{}, b{};
        for (int l = 0; l < 2; ++l) a.v[l] = atol[l], b.v[l] = rtol[l];
        mfl::qr_rank_kernel<2><<<1, 1, 0, s>>>(r, Fm, a, b, rank);
        break;
    }
    case 3: {
        mfl::scal<3> a{}, b{};
        for (int l = 0; l < 3; ++l) a.v[l] = atol[l], b.v[l] = rtol[l];
        mfl::qr_rank_kernel<3><<<1, 1, 0, s>>>(r, Fm, a, b, rank);
        break;
    }
    default: {
        mfl::scal<4> a{}, b{};
        for (int l = 0; l < 4; ++l) a.v[l] = atol[l], b.v[l] = rtol[l];
        mfl::qr_rank_kernel<4><<<1, 1, 0, s>>>(r, Fm, a, b, rank);
        break;
    }
    }
    return mfl::record_cuda_error(cudaGetLastError(), "numerical_rank launch");
}
