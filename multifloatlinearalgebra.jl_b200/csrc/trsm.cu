// Multi-double triangular solves, src/kernels/trsm.jl:1-302 and trsv.jl:19-73
// of MultiFloatLinearAlgebra.jl.
//
// Order contract: the reference computes, for every unknown,
//     v = B[i]; for k in the substitution order: v -= coef(i,k) * X[k]; v /= A[i,i]
// (left side; right side uses B[i,k] * coef(k,j)).  Each kernel below keeps that
// exact per-element chain:
//   * trsm_left_cta: forward substitution, one CTA per right-hand-side column.
//     The column's running values live in registers (rows distributed
//     cyclically over the threads).  Step k finalises X[k] (owner divides by
//     the diagonal), broadcasts it through shared memory, and every later row
//     applies its term k.  Each row thus receives its terms in the reference's
//     ascending order while the rows progress in parallel.
//   * trsm_left_warp: the same with the rows over the lanes of a warp, for
//     triangles of at most 64 rows and up to some thousand columns.
//   * trsm_left_backward_cta, trsm_left_backward_rows: backward substitution, one
//     CTA per column.
//   * trsm_left_thread: one thread per right-hand-side column, the plain
//     serial loop (many columns).
//   * trsm_right_thread: one thread per row of B, the plain serial loop (the
//     Cholesky panel solve A21 <- A21 / L11^T).
#include "mf_device.cuh"
#include "mflab_internal.h"

namespace mfl {

constexpr int TRSM_SMS = 148;

template <int N>
__device__ __forceinline__ mf<N> tri_coef(const Mat &A, int64_t r, int64_t c, bool transposed) {
    return transposed ? load_mf<N>(A.p, A.ld, A.ls, c, r) : load_mf<N>(A.p, A.ld, A.ls, r, c);
}

template <int N>
__global__ void scale_kernel(int64_t m, int64_t n, Mat B, scal<N> alpha) {
    int64_t idx = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (idx >= m * n) return;
    int64_t r = idx % m, c = idx / m;
    mf<N> v = load_mf<N>(B.p, B.ld, B.ls, r, c);
    store_mf<N>(B.p, B.ld, B.ls, r, c, mul(v, alpha.get()));
}

// one CTA per column; NT threads; each thread owns up to MAXR rows.  A step is
// a division, a CTA barrier and the rows' multiply-subtracts.  AHEAD loads the
// coefficients of the next step (the diagonal among them, for the row it
// finalises) behind the ones just used, which shortens the step and costs the
// registers of a CTA per SM.  x2, n = 2048, 64 columns: 4200 us (4711 us with
// the loads inside the step).
template <int N, int NT, int MAXR, bool AHEAD>
__global__ void __launch_bounds__(NT) trsm_left_cta(int64_t m, int64_t n, Mat A, Mat B,
                                                    bool eff_lower, bool transposed, bool unit,
                                                    const int *info) {
    if (info && *info) return;
    __shared__ double xs[2][N];
    const int64_t col = blockIdx.x;
    if (col >= n) return;
    const int t = threadIdx.x;
    mf<N> v[MAXR], coef[AHEAD ? MAXR : 1];
    auto fetch = [&](int q, int64_t k) {
        if constexpr (AHEAD) {
            const int64_t r = t + (int64_t)q * NT;
            if (r < m && (eff_lower ? r >= k && k < m : r <= k && k >= 0) && !(unit && r == k))
                coef[q] = tri_coef<N>(A, r, k, transposed);
        }
    };
    const int64_t k0 = eff_lower ? 0 : m - 1;
#pragma unroll
    for (int q = 0; q < MAXR; ++q) {
        int64_t r = t + (int64_t)q * NT;
        v[q] = r < m ? load_mf<N>(B.p, B.ld, B.ls, r, col) : from_double<N>(0.0);
        if constexpr (AHEAD) coef[q] = from_double<N>(1.0);
        fetch(q, k0);
    }
    for (int64_t s = 0; s < m; ++s) {
        const int64_t k = eff_lower ? s : m - 1 - s;  // row finalised at this step
        const int64_t kn = eff_lower ? k + 1 : k - 1;
        const int slot = (int)(s & 1);
        if ((k % NT) == t) {
            const int qk = (int)(k / NT);
            mf<N> x, d;
#pragma unroll
            for (int q = 0; q < MAXR; ++q)
                if (q == qk) {
                    x = v[q];
                    if constexpr (AHEAD) d = coef[q];
                }
            if constexpr (!AHEAD)
                if (!unit) d = load_mf<N>(A.p, A.ld, A.ls, k, k);
            if (!unit) x = div(x, d);
            store_mf<N>(B.p, B.ld, B.ls, k, col, x);
#pragma unroll
            for (int l = 0; l < N; ++l) xs[slot][l] = x.v[l];
        }
        __syncthreads();
        mf<N> xk;
#pragma unroll
        for (int l = 0; l < N; ++l) xk.v[l] = xs[slot][l];
#pragma unroll
        for (int q = 0; q < MAXR; ++q) {
            const int64_t r = t + (int64_t)q * NT;
            const bool later = eff_lower ? (r > k) : (r < k);
            if (r < m && later) {
                if constexpr (AHEAD) v[q] = submul(v[q], coef[q], xk);
                else v[q] = submul(v[q], tri_coef<N>(A, r, k, transposed), xk);
                fetch(q, kn);
            }
        }
    }
}

// AHEAD is the faster form for as long as it takes no more rounds of CTAs over
// the chip.  CTAs per SM (AHEAD / not): up to 2048 rows x2 2 / 3, x3 and x4
// 1 / 2; beyond x2 1 / 2, x3 1 / 1; x4 spills there (35.5 / 28.0 ms at 3000
// rows).  us, 300 rows: x2 296 columns 371 / 413, 444 columns 685 / 440, 3000
// columns 3798 / 2962; x4 148 columns 1113 / 1210, 222 columns 1975 / 1217, 3000
// columns 20554 / 12481.
template <int N>
static bool trsm_ahead(int64_t m, int64_t n) {
    if (N == 1) return true;  // no registers to win
    const bool tall = m > 256 * 8;
    if (N == 4 && tall) return false;
    const int64_t with = TRSM_SMS * (N == 2 && !tall ? 2 : 1);
    const int64_t without = TRSM_SMS * (N == 2 && !tall ? 3 : N == 3 && tall ? 1 : 2);
    return (n + with - 1) / with <= (n + without - 1) / without;
}

// Forward substitution of a triangle of at most 64 rows: W lanes per column, RPL
// rows per lane, the triangle staged in shared memory row-contiguous.  Row k's
// lane finalises X[k] and broadcasts it; the rows below apply their term k.
// A column of 16 rows is 16 steps of a broadcast and a multiply-subtract.
// x4, 16 unit rows, 685 columns: about 7 us (77 us with a thread per column
// whose 120 terms wait for their loads one by one).
constexpr int TRSW_NT = 128;

// Its line against the thread kernel: a column costs the warp kernel m steps of
// issue, an unknown's division for 16 or 32 lanes alone, so its time grows with
// the columns, while the thread kernel's, bound by its chains, is the same up to
// some 20 000 columns.  They meet in proportion to m, by the lanes and rows per
// lane.  us, warp / thread: x2, 16 rows 10000 44 / 52, 100000 261 / 170; x2, 64
// rows 10000 322 / 510, 20000 630 / 717, 100000 2988 / 1889; x3, 32 rows 4000
// 183 / 255, 8000 334 / 255; x4, 8 rows 2000 45 / 49, 4000 71 / 48; x4, 64 rows
// 4000 1336 / 1347, 100000 31900 / 4225.
template <int N>
static int64_t trsw_columns(int64_t m) {
    constexpr int per_row[3][3] = {{640, 270, 200}, {300, 145, 125}, {200, 90, 60}};
    return m * per_row[N - 2][m <= 16 ? 0 : m <= 32 ? 1 : 2];
}

template <int N, int W, int RPL>
__global__ void __launch_bounds__(TRSW_NT)
    trsm_left_warp(int m, int64_t n, Mat A, Mat B, bool transposed, bool unit, const int *info) {
    if (info && *info) return;
    extern __shared__ double tri[];  // [N][m][m]: tri[(l*m + k)*m + row], row >= k
    for (int e = threadIdx.x; e < m * m; e += TRSW_NT) {
        const int i = e % m, j = e / m;
        const int row = transposed ? j : i, k = transposed ? i : j;  // op(A)[row, k]
        if (row < k || (unit && row == k)) continue;
        const mf<N> a = tri_coef<N>(A, row, k, transposed);
#pragma unroll
        for (int l = 0; l < N; ++l) tri[(l * m + k) * m + row] = a.v[l];
    }
    __syncthreads();
    const int sub = threadIdx.x % W;
    const int64_t col = (int64_t)blockIdx.x * (TRSW_NT / W) + threadIdx.x / W;
    const bool in = col < n;  // the lanes of a warp stay together
    auto coef = [&](int row, int k) {
        mf<N> a;
#pragma unroll
        for (int l = 0; l < N; ++l) a.v[l] = tri[(l * m + k) * m + row];
        return a;
    };
    mf<N> v[RPL];
#pragma unroll
    for (int q = 0; q < RPL; ++q) {
        const int row = sub + q * W;
        v[q] = in && row < m ? load_mf<N>(B.p, B.ld, B.ls, row, col) : from_double<N>(0.0);
    }
#pragma unroll
    for (int qk = 0; qk < RPL; ++qk) {
        for (int kl = 0; kl < W; ++kl) {
            const int k = qk * W + kl;
            if (k >= m) break;
            if (!unit && sub == kl) v[qk] = div(v[qk], coef(k, k));
            mf<N> x;
#pragma unroll
            for (int l = 0; l < N; ++l) x.v[l] = __shfl_sync(0xffffffffu, v[qk].v[l], kl, W);
#pragma unroll
            for (int q = 0; q < RPL; ++q) {
                const int row = sub + q * W;
                if (q >= qk && row > k && row < m) v[q] = submul(v[q], coef(row, k), x);
            }
        }
    }
#pragma unroll
    for (int q = 0; q < RPL; ++q) {
        const int row = sub + q * W;
        if (in && row < m) store_mf<N>(B.p, B.ld, B.ls, row, col, v[q]);
    }
}

template <int N>
static int run_trsm_left_warp(int64_t m, int64_t n, Mat A, Mat B, bool transposed, bool unit,
                              cudaStream_t s, const int *info) {
    const size_t smem = (size_t)N * m * m * sizeof(double);
    const int w = m <= 16 ? 16 : 32;
    const int64_t grid = (n + TRSW_NT / w - 1) / (TRSW_NT / w);
    if (grid > 2147483647LL) return MFLAB_ERR_UNSUPPORTED;
    auto launch = [&](auto kern, std::atomic<unsigned long long> &configured) -> int {
        if (int rc = set_smem_once((const void *)kern, N * 64 * 64 * (int)sizeof(double),
                                   configured, "trsm left warp attribute"))
            return rc;
        kern<<<(unsigned)grid, TRSW_NT, smem, s>>>((int)m, n, A, B, transposed, unit, info);
        return record_cuda_error(cudaGetLastError(), "trsm left warp");
    };
    static std::atomic<unsigned long long> done[3];
    if (m <= 16) return launch(trsm_left_warp<N, 16, 1>, done[0]);
    if (m <= 32) return launch(trsm_left_warp<N, 32, 1>, done[1]);
    return launch(trsm_left_warp<N, 32, 2>, done[2]);
}

// Backward substitution (effective upper, left side) in the reference order:
// row r's chain v = B[r]; v -= coef(r,k) * X[k] for k = r+1..m-1 ascending.
// X[r+1] enters row r's chain first, so a column is one chain of m(m-1)/2
// subtractions (about 92 / 220 / 340 cycles each in x2 / x3 / x4): nothing but
// that chain is left on the critical path.  One CTA per column; one warp's
// first lane runs the chain and the divisions, eight warps form the products
// of the next 256 terms, across the row's end too: only the product with the
// unknown just found is the chain's own (its slot holds the coefficient).  The
// chain warp's place rotates over the schedulers with the CTA.  x2, n = 2048,
// 64 columns: 101 ms (105.2 ms with the products of a row formed between
// two barriers before its chain).
constexpr int TRSB_TILE = 256, TRSB_NT = TRSB_TILE + 32, TRSR_NT = 256;

template <int N>
__global__ void __launch_bounds__(TRSB_NT)
    trsm_left_backward_cta(int64_t m, int64_t n, Mat A, Mat B, bool transposed, bool unit,
                           const int *info) {
    if (info && *info) return;
    __shared__ double prod[2][TRSB_TILE][N];
    __shared__ double head[2][2][N];  // right-hand side and diagonal of a row
    const int64_t col = blockIdx.x;
    if (col >= n) return;
    const int warp = threadIdx.x / 32, lane = threadIdx.x % 32;
    const int chain = (int)((blockIdx.x + blockIdx.x / TRSM_SMS) % 4);
    const int slot = (warp - (warp > chain ? 1 : 0)) * 32 + lane;  // of a producing thread
    auto slabs = [&](int64_t r) { return (m - 1 - r + TRSB_TILE - 1) / TRSB_TILE; };
    auto produce = [&](int64_t r, int64_t j, int b) {
        const int64_t k = r + 1 + j * TRSB_TILE + slot;
        if (k < m) {
            mf<N> p = tri_coef<N>(A, r, k, transposed);
            if (k > r + 1) p = mul(p, load_mf<N>(B.p, B.ld, B.ls, k, col));
#pragma unroll
            for (int l = 0; l < N; ++l) prod[b][slot][l] = p.v[l];
        }
        if (j == 0 && slot >= TRSB_TILE - 2) {
            const int which = slot - (TRSB_TILE - 2);
            if (which == 0 || !unit) {
                const mf<N> x = which == 0 ? load_mf<N>(B.p, B.ld, B.ls, r, col)
                                           : load_mf<N>(A.p, A.ld, A.ls, r, r);
#pragma unroll
                for (int l = 0; l < N; ++l) head[b][which][l] = x.v[l];
            }
        }
    };
    mf<N> v = from_double<N>(0.0), x = v, d = v;
    int64_t r = m - 1, j = 0;
    if (warp != chain) produce(r, 0, 0);
    for (int b = 0;; b ^= 1) {
        __syncthreads();
        const bool last = j + 1 >= slabs(r);
        const int64_t rn = last ? r - 1 : r, jn = last ? 0 : j + 1;
        if (warp != chain) {
            if (rn >= 0) produce(rn, jn, b ^ 1);
        } else if (lane == 0) {
            const int64_t left = m - 1 - r - j * TRSB_TILE;
            const int cnt = left < TRSB_TILE ? (int)left : TRSB_TILE;
            auto get = [&](const double *q) {
                mf<N> p;
#pragma unroll
                for (int l = 0; l < N; ++l) p.v[l] = q[l];
                return p;
            };
            int i = 0;
            if (j == 0) {
                v = get(head[b][0]);
                if (!unit) d = get(head[b][1]);
                if (cnt > 0) {
                    v = sub(v, mul(get(prod[b][0]), x));
                    i = 1;
                }
            }
            // terms unrolled together: a loop end costs about 13 cycles, the
            // longer networks fill the instruction cache sooner
            constexpr int U = N == 2 ? 32 : N == 3 ? 16 : 8;
            for (; i + U <= cnt; i += U)
#pragma unroll
                for (int q = 0; q < U; ++q) v = sub(v, get(prod[b][i + q]));
            for (; i < cnt; ++i) v = sub(v, get(prod[b][i]));
            if (last) {
                if (!unit) v = div(v, d);
                store_mf<N>(B.p, B.ld, B.ls, r, col, v);
                x = v;
            }
        }
        if (last && r == 0) break;
        r = rn;
        j = jn;
    }
}

// The same, less of it at once: the products of row r are formed by all threads
// into shared memory between two barriers, thread 0 runs the chain.  An SM
// holds more of these CTAs, and their chains then hide one another's barriers.
template <int N>
__global__ void __launch_bounds__(TRSR_NT)
    trsm_left_backward_rows(int64_t m, int64_t n, Mat A, Mat B, bool transposed, bool unit,
                            const int *info) {
    if (info && *info) return;
    extern __shared__ double row_prod[];  // [m][N]
    const int64_t col = blockIdx.x;
    if (col >= n) return;
    const int t = threadIdx.x;
    auto get = [&](int64_t k) {
        mf<N> p;
#pragma unroll
        for (int l = 0; l < N; ++l) p.v[l] = row_prod[k * N + l];
        return p;
    };
    for (int64_t r = m - 1; r >= 0; --r) {
        for (int64_t k = r + 1 + t; k < m; k += TRSR_NT) {
            const mf<N> p = mul(tri_coef<N>(A, r, k, transposed), load_mf<N>(B.p, B.ld, B.ls, k, col));
#pragma unroll
            for (int l = 0; l < N; ++l) row_prod[k * N + l] = p.v[l];
        }
        __syncthreads();
        if (t == 0) {
            // the next term is read from shared memory while the current one
            // is subtracted
            mf<N> v = load_mf<N>(B.p, B.ld, B.ls, r, col), next = v;
            if (r + 1 < m) next = get(r + 1);
            for (int64_t k = r + 1; k < m; ++k) {
                const mf<N> p = next;
                if (k + 1 < m) next = get(k + 1);
                v = sub(v, p);
            }
            if (!unit) v = div(v, load_mf<N>(A.p, A.ld, A.ls, r, r));
            store_mf<N>(B.p, B.ld, B.ls, r, col, v);
        }
        __syncthreads();
    }
}

template <int N>
__global__ void trsm_left_thread(int64_t m, int64_t n, Mat A, Mat B, bool eff_lower,
                                 bool transposed, bool unit, const int *info) {
    if (info && *info) return;
    const int64_t c = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (c >= n) return;
    if (eff_lower) {
        for (int64_t row = 0; row < m; ++row) {
            mf<N> v = load_mf<N>(B.p, B.ld, B.ls, row, c);
            for (int64_t k = 0; k < row; ++k)
                v = submul(v, tri_coef<N>(A, row, k, transposed), load_mf<N>(B.p, B.ld, B.ls, k, c));
            if (!unit) v = div(v, load_mf<N>(A.p, A.ld, A.ls, row, row));
            store_mf<N>(B.p, B.ld, B.ls, row, c, v);
        }
    } else {
        for (int64_t row = m - 1; row >= 0; --row) {
            mf<N> v = load_mf<N>(B.p, B.ld, B.ls, row, c);
            for (int64_t k = row + 1; k < m; ++k)
                v = submul(v, tri_coef<N>(A, row, k, transposed), load_mf<N>(B.p, B.ld, B.ls, k, c));
            if (!unit) v = div(v, load_mf<N>(A.p, A.ld, A.ls, row, row));
            store_mf<N>(B.p, B.ld, B.ls, row, c, v);
        }
    }
}

// Which of the three kernels solves n columns backward.  The slab kernel wins
// while its CTAs have an SM to themselves (in x2 up to 256 rows two share one),
// the row kernel after that, and a thread per column where either takes too
// many rounds: beyond four (x4 three) CTAs per SM for short triangles and for
// those whose row exceeds the row kernel's buffer, else from 4096 columns on.
// us, slab / row / thread kernel: x2, 64 rows 148 columns 160 / 182 / 518, 296
// 172 / 185 / 518, 444 217 / 185 / 518, 800 337 / 342 / 517, 2400 780 / 668 /
// 519; x2, 300 rows 148 columns 2357 / 2548, 444 3589 / 2580, 4095 20501 / 15911;
// x4, 300 rows 148 columns 8201 / 8354, 222 13261 / 8398, 4095 106437 / 83817;
// x4, 8 rows 444 columns 68 / 47 / 46, 592 77 / 71 / 48.
constexpr size_t TRSR_SMEM = 200 * 1024;

template <int N>
static int run_trsm_left_backward(int64_t m, int64_t n, Mat A, Mat B, bool transposed, bool unit,
                                  cudaStream_t s, const int *info) {
    const size_t smem = (size_t)m * N * sizeof(double);
    const bool fits = smem <= TRSR_SMEM;
    const int64_t most = m > 64 && fits ? 4095 : (N == 4 ? 3 : 4) * TRSM_SMS;
    if (n > most) {
        trsm_left_thread<N><<<(unsigned)((n + 127) / 128), 128, 0, s>>>(m, n, A, B, false, transposed,
                                                                        unit, info);
    } else if (!fits || n <= (N == 2 && m <= 256 ? 2 : 1) * TRSM_SMS) {
        trsm_left_backward_cta<N><<<(unsigned)n, TRSB_NT, 0, s>>>(m, n, A, B, transposed, unit, info);
    } else {
        static std::atomic<unsigned long long> configured{0};
        if (int rc = set_smem_once((const void *)trsm_left_backward_rows<N>, (int)TRSR_SMEM, configured,
                                   "trsm backward attribute"))
            return rc;
        trsm_left_backward_rows<N><<<(unsigned)n, TRSR_NT, smem, s>>>(m, n, A, B, transposed, unit,
                                                                    info);
    }
    return record_cuda_error(cudaGetLastError(), "trsm left backward");
}

template <int N>
__global__ void trsm_right_thread(int64_t m, int64_t n, Mat A, Mat B, bool eff_lower,
                                  bool transposed, bool unit, const int *info) {
    if (info && *info) return;
    const int64_t r = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (r >= m) return;
    if (eff_lower) {
        for (int64_t col = n - 1; col >= 0; --col) {
            mf<N> v = load_mf<N>(B.p, B.ld, B.ls, r, col);
            for (int64_t k = col + 1; k < n; ++k)
                v = submul(v, load_mf<N>(B.p, B.ld, B.ls, r, k), tri_coef<N>(A, k, col, transposed));
            if (!unit) v = div(v, load_mf<N>(A.p, A.ld, A.ls, col, col));
            store_mf<N>(B.p, B.ld, B.ls, r, col, v);
        }
    } else {
        for (int64_t col = 0; col < n; ++col) {
            mf<N> v = load_mf<N>(B.p, B.ld, B.ls, r, col);
            for (int64_t k = 0; k < col; ++k)
                v = submul(v, load_mf<N>(B.p, B.ld, B.ls, r, k), tri_coef<N>(A, k, col, transposed));
            if (!unit) v = div(v, load_mf<N>(A.p, A.ld, A.ls, col, col));
            store_mf<N>(B.p, B.ld, B.ls, r, col, v);
        }
    }
}

// Binary64 diagonal-block solve of the blocked left solve below: one CTA
// per right-hand-side column, the jb x jb block (jb <= 64) in shared memory,
// row t of the column in thread t.
constexpr int TRSM64_NB = 64;

__global__ void __launch_bounds__(TRSM64_NB)
    trsm64_diag_kernel(int64_t jb, Mat A, Mat B, bool lower, bool unit) {
    __shared__ double a[TRSM64_NB][TRSM64_NB + 1];
    __shared__ double xk;
    const int t = threadIdx.x;
    const int64_t col = blockIdx.x;
    for (int c = 0; c < jb; ++c)
        if (t < jb) a[t][c] = A.p[(int64_t)c * A.ld + t];
    double v = t < jb ? B.p[col * B.ld + t] : 0.0;
    __syncthreads();
    for (int s = 0; s < jb; ++s) {
        const int k = lower ? s : (int)jb - 1 - s;
        if (t == k) {
            if (!unit) v = __ddiv_rn(v, a[k][k]);
            xk = v;
        }
        __syncthreads();
        if (t < jb && (lower ? t > k : t < k)) v = __dsub_rn(v, __dmul_rn(a[t][k], xk));
        __syncthreads();
    }
    if (t < jb) B.p[col * B.ld + t] = v;
}

// Blocked left solve op(A) X = B for binary64 (no reference order to keep):
// 64 x 64 diagonal blocks solved from shared memory, the rows below (forward)
// or above (backward) updated with the FP64 GEMM kernel.  A not transposed.
static int trsm64_blocked(int64_t m, int64_t n, Mat A, Mat B, bool lower, bool unit,
                          cudaStream_t s, const int *info) {
    const double mone[1] = {-1.0}, one[1] = {1.0};
    const int64_t nblk = (m + TRSM64_NB - 1) / TRSM64_NB;
    for (int64_t bi = 0; bi < nblk; ++bi) {
        const int64_t blk = lower ? bi : nblk - 1 - bi;
        const int64_t j0 = blk * TRSM64_NB;
        const int64_t jb = m - j0 < TRSM64_NB ? m - j0 : TRSM64_NB;
        trsm64_diag_kernel<<<(unsigned)n, TRSM64_NB, 0, s>>>(jb, A.at(j0, j0), B.at(j0, 0), lower,
                                                             unit);
        int rc = record_cuda_error(cudaGetLastError(), "trsm64 diagonal");
        if (rc) return rc;
        if (lower && j0 + jb < m) {
            rc = launch_mm(1, false, false, 0, false, m - j0 - jb, n, jb, A.at(j0 + jb, j0),
                           B.at(j0, 0), B.at(j0 + jb, 0), mone, one, s, info);
        } else if (!lower && j0 > 0) {
            rc = launch_mm(1, false, false, 0, false, j0, n, jb, A.at(0, j0), B.at(j0, 0),
                           B.at(0, 0), mone, one, s, info);
        }
        if (rc) return rc;
    }
    return MFLAB_OK;
}

template <int N>
static int run_trsm(int side, int uplo, int trans, int diag, int64_t m, int64_t n, Mat A, Mat B,
                    const double *alpha, cudaStream_t s, const int *info, int order) {
    if (m <= 0 || n <= 0) return MFLAB_OK;
    bool one = alpha[0] == 1.0;
    for (int l = 1; l < N; ++l) one = one && alpha[l] == 0.0;
    if (!one) {
        scal<N> al{};
        for (int l = 0; l < N; ++l) al.v[l] = alpha[l];
        int64_t tot = m * n;
        scale_kernel<N><<<(unsigned)((tot + 255) / 256), 256, 0, s>>>(m, n, B, al);
        int rc = record_cuda_error(cudaGetLastError(), "trsm scale");
        if (rc) return rc;
    }
    const bool transposed = trans == 1;
    const bool eff_lower = (uplo == 0) == !transposed;
    const bool unit = diag == 1;
    if (side == 1) {
        trsm_right_thread<N><<<(unsigned)((m + 127) / 128), 128, 0, s>>>(m, n, A, B, eff_lower,
                                                                         transposed, unit, info);
        return record_cuda_error(cudaGetLastError(), "trsm right");
    }
    // The wavefront kernel applies row r's terms as the unknowns are finalised.
    // That is the reference's ascending-k chain only for forward substitution
    // (effective lower): in backward substitution the reference's chain for
    // row r starts with X[r+1], the last unknown finalised before X[r], so each
    // row's chain is serial after its predecessor; those solves use the
    // product-parallel CTA kernel (or the per-column loop for short triangles).
    // The binary64 instance (N == 1) has no reference order to keep and uses
    // the wavefront in both directions.
    // the fast order applies every term as soon as its unknown is final, in both
    // directions (deterministic, not the reference's association)
    const bool wavefront_ok = eff_lower || N == 1 || order == MFLAB_ORDER_FAST;
    if (N == 1 && !transposed && m > 2 * TRSM64_NB && n <= 65535 && !info)
        return trsm64_blocked(m, n, A, B, eff_lower, unit, s, info);
    if constexpr (N >= 2) {
        if (eff_lower && m <= 64 && n <= trsw_columns<N>(m))
            return run_trsm_left_warp<N>(m, n, A, B, transposed, unit, s, info);
        if (!wavefront_ok) return run_trsm_left_backward<N>(m, n, A, B, transposed, unit, s, info);
    }
    if (m <= 64 || n >= 4096) {
        trsm_left_thread<N><<<(unsigned)((n + 127) / 128), 128, 0, s>>>(m, n, A, B, eff_lower,
                                                                        transposed, unit, info);
        return record_cuda_error(cudaGetLastError(), "trsm left thread");
    }
    if (n > 2147483647LL) return MFLAB_ERR_UNSUPPORTED;
    if (m > 256 * 16) {
        trsm_left_thread<N><<<(unsigned)((n + 127) / 128), 128, 0, s>>>(m, n, A, B, eff_lower,
                                                                        transposed, unit, info);
        return record_cuda_error(cudaGetLastError(), "trsm left thread");
    }
    const bool ahead = trsm_ahead<N>(m, n);
    auto kern = m <= 256 * 8 ? (ahead ? trsm_left_cta<N, 256, 8, true> : trsm_left_cta<N, 256, 8, false>)
                             : (ahead ? trsm_left_cta<N, 256, 16, true> : trsm_left_cta<N, 256, 16, false>);
    kern<<<(unsigned)n, 256, 0, s>>>(m, n, A, B, eff_lower, transposed, unit, info);
    return record_cuda_error(cudaGetLastError(), "trsm left cta");
}

int launch_trsm_info(int N, int side, int uplo, int trans, int diag, int64_t m, int64_t n, Mat A,
                     Mat B, const double *alpha, cudaStream_t s, const int *info, int order) {
    switch (N) {
    case 1: return run_trsm<1>(side, uplo, trans, diag, m, n, A, B, alpha, s, info, order);
    case 2: return run_trsm<2>(side, uplo, trans, diag, m, n, A, B, alpha, s, info, order);
    case 3: return run_trsm<3>(side, uplo, trans, diag, m, n, A, B, alpha, s, info, order);
    case 4: return run_trsm<4>(side, uplo, trans, diag, m, n, A, B, alpha, s, info, order);
    default: return MFLAB_ERR_UNSUPPORTED;
    }
}

int launch_trsm(int N, int side, int uplo, int trans, int diag, int64_t m, int64_t n, Mat A, Mat B,
                const double *alpha, cudaStream_t s) {
    return launch_trsm_info(N, side, uplo, trans, diag, m, n, A, B, alpha, s, nullptr);
}

}  // namespace mfl

extern "C" int mflab_trsm(mflab_handle *h, void *stream, int limbs, int side, int uplo, int trans,
                          int diag, int64_t m, int64_t n, const double *A, int64_t lda,
                          int64_t lsa, double *B, int64_t ldb, int64_t lsb, const double *alpha) {
    MFLAB_RANGE("mflab_trsm");
    if (!h || !mfl::valid_limbs(limbs)) return MFLAB_ERR_UNSUPPORTED;
    if (side < 0 || side > 1 || uplo < 0 || uplo > 1 || trans < 0 || trans > 1 || diag < 0 ||
        diag > 1)
        return MFLAB_ERR_FLAG;
    if (m < 0 || n < 0 || !alpha) return MFLAB_ERR_ARG;
    const int64_t na = side == 0 ? m : n;
    if ((na > 0 && lda < na) || (m > 0 && ldb < m)) return MFLAB_ERR_ARG;
    return mfl::launch_trsm_info(limbs, side, uplo, trans, diag, m, n,
                                 mfl::Mat{(double *)A, lda, lsa}, mfl::Mat{B, ldb, lsb}, alpha,
                                 (cudaStream_t)stream, nullptr, h->solve_order);
}
