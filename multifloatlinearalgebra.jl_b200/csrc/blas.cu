// Matched-order multi-double GEMM / SYRK / GEMMT on the FP64 pipe.
//
// Reduction-order contract (src/kernels/gemm.jl:138-265, syrk.jl:1-50,
// gemmt.jl:1-52 of MultiFloatLinearAlgebra.jl): every output element is ONE
// serial chain acc = 0; for k ascending: acc = acc + a(i,k)*b(k,j), followed
// by alpha*acc (beta == 0: C is never read) or alpha*acc + beta*C.  No split-k
// and no tree reduction, so with the same scalar networks the result is
// bitwise the reference's.
//
// Mapping: a CTA owns a BM x BN output tile; each thread owns TM x TN outputs
// strided by the thread grid so shared-memory reads are conflict-free
// broadcasts.  k-slabs of BK columns of every limb plane are staged in shared
// memory with cp.async into a double buffer while the previous slab is
// consumed.  The kernel is FP64-issue bound: per k step a thread reads
// (TM + TN)*N doubles and executes TM*TN*ops(N) FP64 instructions.  Tile
// shapes trade that ratio against the number of CTAs (mm_tile below); a
// matrix-vector product is a chain per row and has a kernel of its own
// (mv_kernel).
#include "mf_device.cuh"
#include "mflab_internal.h"

#include <algorithm>

MFLAB_DEBUG_RECORD(blas)

namespace mfl {

__device__ __forceinline__ void cp_async8(void *smem, const void *gmem, bool pred) {
    unsigned s = (unsigned)__cvta_generic_to_shared(smem);
    int src_size = pred ? 8 : 0;
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;\n" ::"r"(s), "l"(gmem),
                 "r"(src_size)
                 : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }
template <int n>
__device__ __forceinline__ void cp_async_wait() {
    asm volatile("cp.async.wait_group %0;\n" ::"n"(n) : "memory");
}

// column tiles in a grid's y dimension; wider products take several launches, up
// to as many columns as a grid of the widest tiles (64 columns, 32 in x4) holds
constexpr int64_t MM_GRID_Y = 65535;
template <int N>
struct MMColumns {
    static constexpr int64_t most = MM_GRID_Y * (N == 4 ? 32 : 64);
};

template <int N, int BM, int BN, int BK, int TM, int TN>
struct MMShape {
    static constexpr int TX = BM / TM;
    static constexpr int TY = BN / TN;
    static constexpr int NT = TX * TY;
    static constexpr size_t smem_bytes = sizeof(double) * 2 * N * BK * (BM + BN);
};

// TA: 0 a(i,k) = A[i,k]; 1 a(i,k) = A[k,i]; 2 symmetric from the lower
// triangle (k <= i ? A[i,k] : A[k,i]); 3 symmetric from the upper triangle.
// mode bits: MM_PACKED C is a packed lower triangle (column-major
// (0,0),(1,0)..(n-1,0),(1,1)..), limb stride C.ls; with TRMM the chain of
// C(i,j) runs over k <= idx (or k >= idx with MM_KGE), idx = i (or j with
// MM_RIGHT), and with MM_UNIT its diagonal term k == idx adds the other
// operand's entry instead of a product (trmm.jl:1-80).
// UNR: k steps unrolled together (threads with one output need several steps
// in flight to hide the shared-memory reads behind the accumulation chain).
template <int N, int BM, int BN, int BK, int TM, int TN, int UNR, int TA, bool TB, bool TRI,
          bool FUSED, bool TRMM>
__global__ void __launch_bounds__(MMShape<N, BM, BN, BK, TM, TN>::NT)
    mm_kernel(int64_t m, int64_t n, int64_t K, Mat A, Mat B, Mat C, scal<N> alpha, scal<N> beta,
              int overwrite, const int *info, int mode) {
    using S = MMShape<N, BM, BN, BK, TM, TN>;
    constexpr int NT = S::NT, TX = S::TX, TY = S::TY;
    // a kernel launched after this one as a programmatic dependent (the
    // blocked Cholesky's next step) may be placed now; it waits for this
    // grid's completion before reading (no effect otherwise)
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    extern __shared__ double smem[];
    double *As = smem;                   // [2][N][BK][BM]
    double *Bs = smem + 2 * N * BK * BM;  // [2][N][BK][BN]
    const int tid = threadIdx.x;
    const int tx = tid % TX, ty = tid / TX;
    const int64_t row0 = (int64_t)blockIdx.x * BM, col0 = (int64_t)blockIdx.y * BN;
    if (TRI && row0 + BM - 1 < col0) return;  // tile strictly above the diagonal
    // debug builds: C's column stride holds its rows
    if (!(mode & MM_PACKED) && !MFLAB_IDX_OK(C.ld >= m, 6, C.ld, m)) return;
    if (info && *info) return;                 // an earlier factorization step failed
    // reduction range of this tile: all of K, or the triangular part TRMM needs
    int64_t kbeg = 0, kend = K;
    if (TRMM) {
        const bool right = mode & MM_RIGHT;
        const int64_t lo = right ? col0 : row0, hi = right ? col0 + BN : row0 + BM;
        if (mode & MM_KGE) kbeg = lo < K ? lo : K;
        else kend = hi < K ? hi : K;
    }

    mf<N> acc[TM][TN];
#pragma unroll
    for (int i = 0; i < TM; ++i)
#pragma unroll
        for (int j = 0; j < TN; ++j) acc[i][j] = from_double<N>(0.0);

    auto load_tile = [&](int buf, int64_t k0) {
        for (int e = tid; e < BM * BK; e += NT) {
            int i, kk;
            if (TA != 1) {
                i = e % BM;
                kk = e / BM;
            } else {
                kk = e % BK;
                i = e / BK;
            }
            int64_t gi = row0 + i, gk = k0 + kk;
            bool ok = gi < m && gk < kend;
            bool tr = TA == 1 || (TA == 2 && gk > gi) || (TA == 3 && gk < gi);
            const double *src = ok ? (tr ? A.p + gi * A.ld + gk : A.p + gk * A.ld + gi) : A.p;
#pragma unroll
            for (int l = 0; l < N; ++l)
                cp_async8(&As[((buf * N + l) * BK + kk) * BM + i], src + (ok ? l * A.ls : 0), ok);
        }
        for (int e = tid; e < BN * BK; e += NT) {
            int j, kk;
            if (!TB) {
                kk = e % BK;
                j = e / BK;
            } else {
                j = e % BN;
                kk = e / BN;
            }
            int64_t gj = col0 + j, gk = k0 + kk;
            bool ok = gj < n && gk < kend;
            const double *src = ok ? (TB ? B.p + gk * B.ld + gj : B.p + gj * B.ld + gk) : B.p;
#pragma unroll
            for (int l = 0; l < N; ++l)
                cp_async8(&Bs[((buf * N + l) * BK + kk) * BN + j], src + (ok ? l * B.ls : 0), ok);
        }
    };

    auto step = [&](int buf, int kk, int64_t gk) {
        mf<N> a[TM], b[TN];
#pragma unroll
        for (int i = 0; i < TM; ++i)
#pragma unroll
            for (int l = 0; l < N; ++l) a[i].v[l] = As[((buf * N + l) * BK + kk) * BM + tx + i * TX];
#pragma unroll
        for (int j = 0; j < TN; ++j)
#pragma unroll
            for (int l = 0; l < N; ++l) b[j].v[l] = Bs[((buf * N + l) * BK + kk) * BN + ty + j * TY];
        if constexpr (!TRMM) {
#pragma unroll
            for (int i = 0; i < TM; ++i)
#pragma unroll
                for (int j = 0; j < TN; ++j) acc[i][j] = mac<N, FUSED>(acc[i][j], a[i], b[j]);
        } else {
            const bool right = mode & MM_RIGHT, kge = mode & MM_KGE, unit = mode & MM_UNIT;
#pragma unroll
            for (int i = 0; i < TM; ++i)
#pragma unroll
                for (int j = 0; j < TN; ++j) {
                    const int64_t idx = right ? col0 + ty + j * TY : row0 + tx + i * TX;
                    if (gk == idx) {
                        if (unit) acc[i][j] = add(acc[i][j], right ? a[i] : b[j]);
                        else acc[i][j] = mac<N, false>(acc[i][j], a[i], b[j]);
                    } else if (kge ? gk > idx : gk < idx) {
                        acc[i][j] = mac<N, false>(acc[i][j], a[i], b[j]);
                    }
                }
        }
    };

    const int64_t nk = kend > kbeg ? (kend - kbeg + BK - 1) / BK : 0;
    if (nk > 0) {
        load_tile(0, kbeg);
        cp_async_commit();
    }
    for (int64_t kt = 0; kt < nk; ++kt) {
        const int buf = (int)(kt & 1);
        const int64_t k0 = kbeg + kt * BK;
        if (kt + 1 < nk) load_tile(buf ^ 1, k0 + BK);
        cp_async_commit();
        cp_async_wait<1>();
        __syncthreads();
        const int64_t rem = kend - k0;
        if (rem >= BK) {
#pragma unroll UNR
            for (int kk = 0; kk < BK; ++kk) step(buf, kk, k0 + kk);
        } else {
            for (int kk = 0; kk < (int)rem; ++kk) step(buf, kk, k0 + kk);
        }
        __syncthreads();
    }

    const mf<N> al = alpha.get(), be = beta.get();
#pragma unroll
    for (int i = 0; i < TM; ++i) {
#pragma unroll
        for (int j = 0; j < TN; ++j) {
            const int64_t gi = row0 + tx + i * TX, gj = col0 + ty + j * TY;
            if (gi < m && gj < n && (!TRI || gi >= gj)) {
                mf<N> r = mul(al, acc[i][j]);
                if (mode & MM_PACKED) {
                    double *c = C.p + gj * (2 * n - gj + 1) / 2 + (gi - gj);
                    if (!overwrite) {
                        mf<N> old;
#pragma unroll
                        for (int l = 0; l < N; ++l) old.v[l] = c[l * C.ls];
                        r = add(r, mul(be, old));
                    }
#pragma unroll
                    for (int l = 0; l < N; ++l) c[l * C.ls] = r.v[l];
                } else {
                    if (!overwrite) r = add(r, mul(be, load_mf<N>(C.p, C.ld, C.ls, gi, gj)));
                    store_mf<N>(C.p, C.ld, C.ls, gi, gj, r);
                }
            }
        }
    }
}

template <int N, int BM, int BN, int BK, int TM, int TN, int UNR, int TA, bool TB, bool TRI,
          bool FUSED, bool TRMM>
static int run_mm(int64_t m, int64_t n, int64_t k, Mat A, Mat B, Mat C, const double *alpha,
                  const double *beta, cudaStream_t s, const int *info, int mode) {
    using S = MMShape<N, BM, BN, BK, TM, TN>;
    auto kern = mm_kernel<N, BM, BN, BK, TM, TN, UNR, TA, TB, TRI, FUSED, TRMM>;
    static std::atomic<unsigned long long> configured{0};
    if (int rc = set_smem_once((const void *)kern, (int)S::smem_bytes, configured,
                               "mm_kernel attribute"))
        return rc;
    scal<N> al{}, be{};
    int overwrite = 1;
    for (int l = 0; l < N; ++l) {
        al.v[l] = alpha[l];
        be.v[l] = beta[l];
        if (beta[l] != 0.0) overwrite = 0;
    }
    if (m <= 0 || n <= 0) return MFLAB_OK;
    if (n > MMColumns<N>::most) return MFLAB_ERR_UNSUPPORTED;
    // the columns' own indices matter to a triangular or packed result and to a
    // triangle on the right, which no memory holds at that many columns
    if (n > MM_GRID_Y * BN && (TRI || (mode & (MM_PACKED | MM_RIGHT)))) return MFLAB_ERR_UNSUPPORTED;
    for (int64_t c0 = 0; c0 < n; c0 += MM_GRID_Y * BN) {
        const int64_t cols = std::min(n - c0, MM_GRID_Y * BN);
        const dim3 grid((unsigned)((m + BM - 1) / BM), (unsigned)((cols + BN - 1) / BN));
        kern<<<grid, S::NT, S::smem_bytes, s>>>(m, cols, k, A, TB ? B.at(c0, 0) : B.at(0, c0),
                                                C.at(0, c0), al, be, overwrite, info, mode);
        if (int rc = record_cuda_error(cudaGetLastError(), "mm_kernel launch")) return rc;
    }
    return MFLAB_OK;
}

// Tile shapes.  Every output is the same chain in every shape, so the choice
// is free.  One CTA of at least two outputs per thread keeps an SM's FP64 pipe
// busy by itself, so a launch takes about
//     ceil(tiles / SMs) * BM * BN / rate
// with the tile's measured rate (10^12 FP64 instructions/s on a full chip).
// Measured, us (x2: 64x64 of 4x4 outputs per thread / 32x16 of 2x1 / 16x8 of 1):
//     48 x 56 x 40       49.2 / 13.2 / 9.2
//     256 x 256 x 256     276 / 50.2 / 50.1
//     515 x 777, k 389    416 /  336 / 330
//     1000 cubed         2063 / 1911 / 1993
//     2048 x 2048, k 512 3642 / 3825 / 4147
// x3 (64x64 / 32x32 / 16x16): 515 x 777, k 389: 1371 / 1018 / 964;
// 2048 x 2048, k 512: 12494 / 12172 / 12478.  x4 (64x32 / 16x16 / 16x8):
// 48 x 56 x 40: 197 / 27.6 / 20.5; 515 x 777, k 389: 3075 / 2101 / 2125;
// 2048 x 2048, k 512: 27455 / 27549 / 27719.
constexpr int MM_SMS = 148;
enum { MM_TINY = 0, MM_MID = 1, MM_WIDE = 2 };

static double mm_cost(int64_t m, int64_t n, bool tri, int bm, int bn, double rate, int least) {
    const int64_t tr = (m + bm - 1) / bm, tc = (n + bn - 1) / bn;
    int64_t tiles = tr * tc;
    if (tri) tiles = tiles / 2 + (tr + tc) / 4 + 1;  // tiles above the diagonal return at once
    const int64_t rounds = std::max<int64_t>((tiles + MM_SMS - 1) / MM_SMS, least);
    return (double)(rounds * bm * bn) / rate;
}

// the shape with the smallest estimate; a lone 16 x 8 CTA (one chain per
// scheduler) leaves the pipe half idle, hence at least two rounds for it.  The
// small x2 tiles of a triangle run below their rate: every other CTA returns at
// once, and a transposed left operand (TA 1) is staged across its columns.  k =
// 256, mid / wide, us: P^T P n = 1600 777 / 843, 2000 1191 / 1111, 3500 3477 /
// 2980; A B^T 2000 977 / 1032, 3500 2854 / 2773.
template <int N, int TA>
static int mm_tile(int64_t m, int64_t n, bool tri) {
    const double slow = N == 2 && tri ? (TA == 1 ? 1.18 : 1.035) : 1.0;
    const double tiny = slow * mm_cost(m, n, tri, 16, 8, N == 2 ? 14.6 : 16.8, 2);
    const double mid = N == 2 ? slow * mm_cost(m, n, tri, 32, 16, 15.6, 1)
                              : mm_cost(m, n, tri, 16, 16, N == 3 ? 17.0 : 17.7, 1);
    const double wide = N == 2   ? mm_cost(m, n, tri, 64, 64, 16.5, 1)
                        : N == 3 ? mm_cost(m, n, tri, 32, 32, 17.4, 1)
                                 : 1e300;
    if (wide <= mid && wide <= tiny) return MM_WIDE;
    return mid <= tiny ? MM_MID : MM_TINY;
}

template <int N, int TA, bool TB, bool TRI, bool FUSED, bool TRMM = false>
static int run_mm_n(int64_t m, int64_t n, int64_t k, Mat A, Mat B, Mat C, const double *alpha,
                    const double *beta, cudaStream_t s, const int *info, int mode) {
    if constexpr (N == 1) {
        return run_mm<1, 64, 64, 16, 4, 4, 2, TA, TB, TRI, FUSED, TRMM>(m, n, k, A, B, C, alpha, beta, s, info, mode);
    } else {
        const int tile = mm_tile<N, TA>(m, n, TRI);
        if (tile == MM_TINY)
            return run_mm<N, 16, 8, 16, 1, 1, (N == 2 ? 8 : N == 3 ? 4 : 2), TA, TB, TRI, FUSED, TRMM>(
                m, n, k, A, B, C, alpha, beta, s, info, mode);
        if constexpr (N == 2) {
            // one 32 x 16 tile per SM: sixteen warps of one output each hide the
            // chains better than eight of two (256 cubed: 43.5 us, 47.8)
            if (tile == MM_MID && !TRI && (m + 31) / 32 * ((n + 15) / 16) <= MM_SMS)
                return run_mm<2, 32, 16, 32, 1, 1, 8, TA, TB, TRI, FUSED, TRMM>(m, n, k, A, B, C, alpha, beta, s, info, mode);
            if (tile == MM_MID)
                return run_mm<2, 32, 16, 16, 2, 1, 4, TA, TB, TRI, FUSED, TRMM>(m, n, k, A, B, C, alpha, beta, s, info, mode);
            return run_mm<2, 64, 64, 16, 4, 4, 2, TA, TB, TRI, FUSED, TRMM>(m, n, k, A, B, C, alpha, beta, s, info, mode);
        } else if constexpr (N == 3) {
            if (tile == MM_MID)
                return run_mm<3, 16, 16, 16, 1, 1, 4, TA, TB, TRI, FUSED, TRMM>(m, n, k, A, B, C, alpha, beta, s, info, mode);
            return run_mm<3, 32, 32, 8, 2, 2, 2, TA, TB, TRI, FUSED, TRMM>(m, n, k, A, B, C, alpha, beta, s, info, mode);
        } else {
            return run_mm<4, 16, 16, 8, 1, 1, 4, TA, TB, TRI, FUSED, TRMM>(m, n, k, A, B, C, alpha, beta, s, info, mode);
        }
    }
}

// Matrix-vector product y = alpha op(A) x + beta y: row i is one ascending
// chain acc = acc + a(i,k) x(k), so a launch cannot end before K dependent
// additions have (about 90 cycles each in x2, 220 in x3, 350 in x4).  A CTA
// owns 32 rows: one warp runs their chains and does nothing else, six warps on
// the other three schedulers load A and form the products of the next slab of
// columns into shared memory (two slabs, one CTA barrier per slab).  The
// second warp on the chain's own scheduler stays idle, and the chain warp's
// place rotates over the schedulers with the CTA so that CTAs that share an
// SM do not share a scheduler.  TA as in mm_kernel.  2500 x 3100 in
// x2: 154 us, 96 cycles a term (590 us on mm_kernel's 32 x 16 tile, of whose
// sixteen columns one was used; 298 us on 32 x 1 tiles that load and multiply
// in the chain's own warp; 167 us with slabs of 32 columns).
constexpr int MV_ROWS = 32, MV_NT = 256, MV_HELPERS = 6;

// columns per slab: a slab costs the chain a barrier and a loop end
template <int N>
struct MVSlab {
    static constexpr int value = N == 2 ? 64 : 32;
};

template <int N>
struct MVStride {  // odd: the columns of one row fall on all banks
    static constexpr int value = N * MV_ROWS + 1;
};

// RAW stores the chains themselves (no alpha, no beta).  The kernel returns at
// once when an earlier step of its factorization stopped: *info != 0 and
// *info <= last.
template <int N, int TA, bool RAW>
__global__ void __launch_bounds__(MV_NT)
    mv_kernel(int64_t m, int64_t K, Mat A, Mat X, Mat Y, scal<N> alpha, scal<N> beta, int overwrite,
              const int *info, int last) {
    // may be launched as a programmatic dependent (no effect otherwise)
    asm volatile("griddepcontrol.wait;" ::: "memory");
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    if (info && *info != 0 && *info <= last) return;
    extern __shared__ double prod[];  // [2][MV_KB][ST]
    constexpr int ST = MVStride<N>::value, MV_KB = MVSlab<N>::value;
    const int lane = threadIdx.x % 32, warp = threadIdx.x / 32;
    const int chain = (int)((blockIdx.x + blockIdx.x / MM_SMS) % 4);
    const int side = (warp - chain) & 3;                        // scheduler beside the chain's
    const int helper = side == 0 ? -1 : 2 * (side - 1) + warp / 4;  // 0 .. 5
    const int64_t row0 = (int64_t)blockIdx.x * MV_ROWS;
    const int64_t slabs = (K + MV_KB - 1) / MV_KB;
    constexpr int PER = (MV_KB + MV_HELPERS - 1) / MV_HELPERS;

    auto produce = [&](int64_t s) {
        double *out = prod + (s & 1) * MV_KB * ST;
        const int64_t k0 = s * MV_KB;
        // is the slab read down its rows (A[i,k]) or across (A[k,i])?  A slab on
        // the diagonal of a symmetric matrix decides entry by entry.
        const bool across = TA == 1 || (TA == 2 && k0 > row0 + MV_ROWS - 1) ||
                            (TA == 3 && k0 + MV_KB - 1 < row0);
        mf<N> a[PER];
        if (!across) {
            const int64_t row = row0 + lane;
#pragma unroll
            for (int q = 0; q < PER; ++q) {
                const int kk = helper + MV_HELPERS * q;
                const int64_t k = k0 + kk;
                const bool ok = kk < MV_KB && k < K && row < m;
                const bool tr = (TA == 2 && k > row) || (TA == 3 && k < row);
                a[q] = !ok  ? from_double<N>(0.0)
                       : tr ? load_mf<N>(A.p, A.ld, A.ls, k, row)
                            : load_mf<N>(A.p, A.ld, A.ls, row, k);
            }
#pragma unroll
            for (int q = 0; q < PER; ++q) {
                const int kk = helper + MV_HELPERS * q;
                if (kk >= MV_KB || k0 + kk >= K) break;
                const mf<N> p = mul(a[q], load_mf<N>(X.p, 0, X.ls, k0 + kk, 0));
#pragma unroll
                for (int l = 0; l < N; ++l) out[kk * ST + l * MV_ROWS + lane] = p.v[l];
            }
        } else {
#pragma unroll
            for (int half = 0; half < MV_KB; half += 32) {
                const int64_t k = k0 + half + lane;
                const bool kin = k < K;
                constexpr int RPER = (MV_ROWS + MV_HELPERS - 1) / MV_HELPERS;
#pragma unroll
                for (int q = 0; q < RPER; ++q) {
                    const int64_t row = row0 + helper + MV_HELPERS * q;
                    const bool ok = kin && helper + MV_HELPERS * q < MV_ROWS && row < m;
                    a[q] = ok ? load_mf<N>(A.p, A.ld, A.ls, k, row) : from_double<N>(0.0);
                }
                const mf<N> x = kin ? load_mf<N>(X.p, 0, X.ls, k, 0) : from_double<N>(0.0);
#pragma unroll
                for (int q = 0; q < RPER; ++q) {
                    const int i = helper + MV_HELPERS * q;
                    if (i >= MV_ROWS) break;
                    const mf<N> p = mul(a[q], x);
#pragma unroll
                    for (int l = 0; l < N; ++l) out[(half + lane) * ST + l * MV_ROWS + i] = p.v[l];
                }
            }
        }
    };

    mf<N> acc = from_double<N>(0.0);
    if (slabs > 0 && helper >= 0) produce(0);
    for (int64_t s = 0; s < slabs; ++s) {
        __syncthreads();
        if (warp == chain) {
            const double *in = prod + (s & 1) * MV_KB * ST + lane;
            auto term = [&](int kk) {
                mf<N> p;
#pragma unroll
                for (int l = 0; l < N; ++l) p.v[l] = in[kk * ST + l * MV_ROWS];
                acc = add(acc, p);
            };
            const int64_t left = K - s * MV_KB;
            if (left >= MV_KB) {
#pragma unroll (N == 2 ? 32 : 8)
                for (int kk = 0; kk < MV_KB; ++kk) term(kk);
            } else {
                for (int kk = 0; kk < (int)left; ++kk) term(kk);
            }
        } else if (helper >= 0 && s + 1 < slabs) {
            produce(s + 1);
        }
    }
    const int64_t row = row0 + lane;
    if (warp != chain || row >= m) return;
    if constexpr (RAW) {
        store_mf<N>(Y.p, 0, Y.ls, row, 0, acc);
        return;
    }
    mf<N> r = mul(alpha.get(), acc);
    if (!overwrite) r = add(r, mul(beta.get(), load_mf<N>(Y.p, 0, Y.ls, row, 0)));
    store_mf<N>(Y.p, 0, Y.ls, row, 0, r);
}

template <int N, int TA>
static int run_mv(int64_t m, int64_t k, Mat A, Mat X, Mat Y, const double *alpha,
                  const double *beta, cudaStream_t s, const int *info) {
    constexpr size_t smem = sizeof(double) * 2 * MVSlab<N>::value * MVStride<N>::value;
    auto kern = mv_kernel<N, TA, false>;
    static std::atomic<unsigned long long> configured{0};
    if (int rc = set_smem_once((const void *)kern, (int)smem, configured, "mv_kernel attribute"))
        return rc;
    scal<N> al{}, be{};
    int overwrite = 1;
    for (int l = 0; l < N; ++l) {
        al.v[l] = alpha[l];
        be.v[l] = beta[l];
        if (beta[l] != 0.0) overwrite = 0;
    }
    const int64_t grid = (m + MV_ROWS - 1) / MV_ROWS;
    if (grid > 2147483647LL) return MFLAB_ERR_UNSUPPORTED;
    kern<<<(unsigned)grid, MV_NT, smem, s>>>(m, k, A, X, Y, al, be, overwrite, info, 0x7fffffff);
    return record_cuda_error(cudaGetLastError(), "mv_kernel launch");
}

template <int N>
static int run_column_chains(int64_t cols, int64_t k, Mat A, Mat X, Mat Y, cudaStream_t s,
                             const int *stop, int last) {
    constexpr size_t smem = sizeof(double) * 2 * MVSlab<N>::value * MVStride<N>::value;
    auto kern = mv_kernel<N, 1, true>;
    static std::atomic<unsigned long long> configured{0};
    if (int rc = set_smem_once((const void *)kern, (int)smem, configured, "column chains attribute"))
        return rc;
    if (cols <= 0) return MFLAB_OK;
    const int64_t grid = (cols + MV_ROWS - 1) / MV_ROWS;
    if (grid > 2147483647LL) return MFLAB_ERR_UNSUPPORTED;
    return launch_programmatic(kern, dim3((unsigned)grid), dim3(MV_NT), smem, s, "column chains",
                               cols, k, A, X, Y, scal<N>{}, scal<N>{}, 1, stop, last);
}

int launch_column_chains(int N, int64_t cols, int64_t k, Mat A, Mat X, Mat Y, cudaStream_t s,
                         const int *stop, int last) {
    switch (N) {
    case 2: return run_column_chains<2>(cols, k, A, X, Y, s, stop, last);
    case 3: return run_column_chains<3>(cols, k, A, X, Y, s, stop, last);
    case 4: return run_column_chains<4>(cols, k, A, X, Y, s, stop, last);
    default: return MFLAB_ERR_UNSUPPORTED;
    }
}

template <int N>
static int dispatch_mm(int ta, bool tb, int tri, bool fused3, int64_t m, int64_t n, int64_t k,
                       Mat A, Mat B, Mat C, const double *alpha, const double *beta,
                       cudaStream_t s, const int *info, int mode) {
    if (n == 1 && m > 0 && !tb && !tri && !mode && !(N == 3 && fused3)) {
        // one column: every output is a chain over a row (the fused x3 step
        // has no separate product and stays with the tiles).  A lone row of
        // adjacent entries transposed is a column, whose loads all lanes share
        // (x3, 300 000 entries: 84 us as a row).
        if (ta == 1 && k == 1 && A.ld == 1) ta = 0;
        if (ta == 0) return run_mv<N, 0>(m, k, A, B, C, alpha, beta, s, info);
        if (ta == 1) return run_mv<N, 1>(m, k, A, B, C, alpha, beta, s, info);
        if (ta == 2) return run_mv<N, 2>(m, k, A, B, C, alpha, beta, s, info);
        if (ta == 3) return run_mv<N, 3>(m, k, A, B, C, alpha, beta, s, info);
    }
    if (ta == 0 && !tb && !tri) {
        if (N == 3 && fused3)
            return run_mm_n<N, 0, false, false, true>(m, n, k, A, B, C, alpha, beta, s, info, mode);
        return run_mm_n<N, 0, false, false, false>(m, n, k, A, B, C, alpha, beta, s, info, mode);
    }
    if (ta == 1 && !tb && tri) return run_mm_n<N, 1, false, true, false>(m, n, k, A, B, C, alpha, beta, s, info, mode);
    if (ta == 1 && !tb && !tri) return run_mm_n<N, 1, false, false, false>(m, n, k, A, B, C, alpha, beta, s, info, mode);
    if (ta == 0 && tb && tri) return run_mm_n<N, 0, true, true, false>(m, n, k, A, B, C, alpha, beta, s, info, mode);
    if (ta == 2 && !tb && !tri) return run_mm_n<N, 2, false, false, false>(m, n, k, A, B, C, alpha, beta, s, info, mode);
    if (ta == 3 && !tb && !tri) return run_mm_n<N, 3, false, false, false>(m, n, k, A, B, C, alpha, beta, s, info, mode);
    return MFLAB_ERR_UNSUPPORTED;
}

int launch_mm(int N, int ta, bool tb, int tri, bool fused3, int64_t m, int64_t n, int64_t k,
              Mat A, Mat B, Mat C, const double *alpha, const double *beta, cudaStream_t s,
              const int *info, int mode) {
    switch (N) {
    case 1:
        if (ta == 0 && !tb && !tri)
            return run_mm_n<1, 0, false, false, false>(m, n, k, A, B, C, alpha, beta, s, info, mode);
        return MFLAB_ERR_UNSUPPORTED;
    case 2: return dispatch_mm<2>(ta, tb, tri, fused3, m, n, k, A, B, C, alpha, beta, s, info, mode);
    case 3: return dispatch_mm<3>(ta, tb, tri, fused3, m, n, k, A, B, C, alpha, beta, s, info, mode);
    case 4: return dispatch_mm<4>(ta, tb, tri, fused3, m, n, k, A, B, C, alpha, beta, s, info, mode);
    default: return MFLAB_ERR_UNSUPPORTED;
    }
}

// C = alpha * a * b with the triangular chain of the mode bits (beta = 0):
// left products a = op(A) (ta 0/1), b = the saved B; right products a = the
// saved B, b = op(A) (tb 0/1).
template <int N>
static int dispatch_trmm(int ta, bool tb, int64_t m, int64_t n, int64_t k, Mat A, Mat B, Mat C,
                         const double *alpha, const double *zero, cudaStream_t s, int mode) {
    if (ta == 0 && !tb) return run_mm_n<N, 0, false, false, false, true>(m, n, k, A, B, C, alpha, zero, s, nullptr, mode);
    if (ta == 1 && !tb) return run_mm_n<N, 1, false, false, false, true>(m, n, k, A, B, C, alpha, zero, s, nullptr, mode);
    if (ta == 0 && tb) return run_mm_n<N, 0, true, false, false, true>(m, n, k, A, B, C, alpha, zero, s, nullptr, mode);
    return MFLAB_ERR_UNSUPPORTED;
}

int launch_trmm_mm(int N, int ta, bool tb, int mode, int64_t m, int64_t n, int64_t k, Mat A, Mat B,
                   Mat C, const double *alpha, cudaStream_t s) {
    const double zero[4] = {0.0, 0.0, 0.0, 0.0};
    switch (N) {
    case 2: return dispatch_trmm<2>(ta, tb, m, n, k, A, B, C, alpha, zero, s, mode);
    case 3: return dispatch_trmm<3>(ta, tb, m, n, k, A, B, C, alpha, zero, s, mode);
    case 4: return dispatch_trmm<4>(ta, tb, m, n, k, A, B, C, alpha, zero, s, mode);
    default: return MFLAB_ERR_UNSUPPORTED;
    }
}

}  // namespace mfl

using mfl::Mat;

extern "C" int mflab_gemm(mflab_handle *h, void *stream, int limbs, int route, int64_t m,
                          int64_t n, int64_t k, const double *A, int64_t lda, int64_t lsa,
                          const double *B, int64_t ldb, int64_t lsb, double *C, int64_t ldc,
                          int64_t lsc, const double *alpha, const double *beta);

extern "C" int mflab_gemm_ozaki_route(mflab_handle *h, void *stream, int limbs, int64_t m,
                                      int64_t n, int64_t k, const double *A, int64_t lda,
                                      int64_t lsa, const double *B, int64_t ldb, int64_t lsb,
                                      double *C, int64_t ldc, int64_t lsc, const double *alpha,
                                      const double *beta);

extern "C" int mflab_gemm(mflab_handle *h, void *stream, int limbs, int route, int64_t m,
                          int64_t n, int64_t k, const double *A, int64_t lda, int64_t lsa,
                          const double *B, int64_t ldb, int64_t lsb, double *C, int64_t ldc,
                          int64_t lsc, const double *alpha, const double *beta) {
    MFLAB_RANGE("mflab_gemm");
    if (!h || !mfl::valid_limbs(limbs)) return MFLAB_ERR_UNSUPPORTED;
    if (m < 0 || n < 0 || k < 0 || !alpha || !beta) return MFLAB_ERR_ARG;
    if (m == 0 || n == 0) return MFLAB_OK;
    if (lda < (m > 0 ? m : 1) || ldb < (k > 0 ? k : 1) || ldc < m) return MFLAB_ERR_ARG;
    if (mfl::views_overlap(C, ldc, lsc, m, n, limbs, A, lda, lsa, m, k) ||
        mfl::views_overlap(C, ldc, lsc, m, n, limbs, B, ldb, lsb, k, n))
        return MFLAB_ERR_ALIAS;
    cudaStream_t s = (cudaStream_t)stream;
    if (route == MFLAB_GEMM_OZAKI)
        return mflab_gemm_ozaki_route(h, stream, limbs, m, n, k, A, lda, lsa, B, ldb, lsb, C, ldc,
                                      lsc, alpha, beta);
    if (route != MFLAB_GEMM_AUTO && route != MFLAB_GEMM_DIRECT) return MFLAB_ERR_FLAG;
    bool fused = (limbs == 3 && route == MFLAB_GEMM_AUTO);
    return mfl::launch_mm(limbs, false, false, 0, fused, m, n, k, Mat{(double *)A, lda, lsa},
                          Mat{(double *)B, ldb, lsb}, Mat{C, ldc, lsc}, alpha, beta, s);
}

// y = alpha * op(A) x + beta * y (gemv.jl:1-167): one ascending chain per
// output (columns for trans = 0, rows for trans = 1), the plain network (no
// fused Float64x3 step), y unread when beta == 0; the GEMM kernel with one
// right-hand column.  x and y are contiguous vectors with limb strides lsx, lsy.
extern "C" int mflab_gemv(mflab_handle *h, void *stream, int limbs, int trans, int64_t m,
                          int64_t n, const double *A, int64_t lda, int64_t lsa, const double *x,
                          int64_t lsx, double *y, int64_t lsy, const double *alpha,
                          const double *beta) {
    MFLAB_RANGE("mflab_gemv");
    if (!h || !mfl::valid_limbs(limbs)) return MFLAB_ERR_UNSUPPORTED;
    if (trans != 0 && trans != 1) return MFLAB_ERR_FLAG;
    if (m < 0 || n < 0 || !alpha || !beta) return MFLAB_ERR_ARG;
    if (m > 0 && lda < m) return MFLAB_ERR_ARG;
    const int64_t rows = trans ? n : m, len = trans ? m : n;
    if (rows == 0) return MFLAB_OK;
    if (mfl::views_overlap(y, rows, lsy, rows, 1, limbs, A, lda, lsa, m, n) ||
        mfl::views_overlap(y, rows, lsy, rows, 1, limbs, x, len > 0 ? len : 1, lsx, len, 1))
        return MFLAB_ERR_ALIAS;
    return mfl::launch_mm(limbs, trans, false, 0, false, rows, 1, len, Mat{(double *)A, lda, lsa},
                          Mat{(double *)x, len > 0 ? len : 1, lsx}, Mat{y, rows, lsy}, alpha, beta,
                          (cudaStream_t)stream);
}

// y = alpha * A x + beta * y with A symmetric, read only from its uplo
// triangle (symv.jl:1-89): row r's chain runs over ascending columns, taking
// A[r, c] from the authoritative triangle and A[c, r] across it.
extern "C" int mflab_symv(mflab_handle *h, void *stream, int limbs, int uplo, int64_t n,
                          const double *A, int64_t lda, int64_t lsa, const double *x, int64_t lsx,
                          double *y, int64_t lsy, const double *alpha, const double *beta) {
    MFLAB_RANGE("mflab_symv");
    if (!h || !mfl::valid_limbs(limbs)) return MFLAB_ERR_UNSUPPORTED;
    if (uplo != 0 && uplo != 1) return MFLAB_ERR_FLAG;
    if (n < 0 || !alpha || !beta) return MFLAB_ERR_ARG;
    if (n == 0) return MFLAB_OK;
    if (lda < n) return MFLAB_ERR_ARG;
    if (mfl::views_overlap(y, n, lsy, n, 1, limbs, A, lda, lsa, n, n) ||
        mfl::views_overlap(y, n, lsy, n, 1, limbs, x, n, lsx, n, 1))
        return MFLAB_ERR_ALIAS;
    return mfl::launch_mm(limbs, 2 + uplo, false, 0, false, n, 1, n, Mat{(double *)A, lda, lsa},
                          Mat{(double *)x, n, lsx}, Mat{y, n, lsy}, alpha, beta,
                          (cudaStream_t)stream);
}

namespace mfl {
// sum over the column-major linear index of x .* y, one ascending chain
// (dot.jl:1-22) by one thread
template <int N>
__global__ void dot_kernel(int64_t m, int64_t n, Mat X, Mat Y, double *out) {
    mf<N> acc = from_double<N>(0.0);
    for (int64_t c = 0; c < n; ++c)
        for (int64_t r = 0; r < m; ++r)
            acc = add(acc, mul(load_mf<N>(X.p, X.ld, X.ls, r, c), load_mf<N>(Y.p, Y.ld, Y.ls, r, c)));
#pragma unroll
    for (int l = 0; l < N; ++l) out[l] = acc.v[l];
}
}  // namespace mfl

// out (device, limbs doubles) = mfdot(x, y) for two m x n arrays (vectors:
// n = 1), in ascending column-major order (dot.jl:1-22).  One serial chain,
// as the reference's.
extern "C" int mflab_dot(mflab_handle *h, void *stream, int limbs, int64_t m, int64_t n,
                         const double *x, int64_t ldx, int64_t lsx, const double *y, int64_t ldy,
                         int64_t lsy, double *out) {
    MFLAB_RANGE("mflab_dot");
    if (!h || !mfl::valid_limbs(limbs)) return MFLAB_ERR_UNSUPPORTED;
    if (m < 0 || n < 0 || !out || (m > 0 && (ldx < m || ldy < m))) return MFLAB_ERR_ARG;
    cudaStream_t s = (cudaStream_t)stream;
    Mat X{(double *)x, ldx, lsx}, Y{(double *)y, ldy, lsy};
    switch (limbs) {
    case 2: mfl::dot_kernel<2><<<1, 1, 0, s>>>(m, n, X, Y, out); break;
    case 3: mfl::dot_kernel<3><<<1, 1, 0, s>>>(m, n, X, Y, out); break;
    default: mfl::dot_kernel<4><<<1, 1, 0, s>>>(m, n, X, Y, out); break;
    }
    return mfl::record_cuda_error(cudaGetLastError(), "dot");
}

// packed lower(C) = alpha * P[k0:k1, :]^T P[k0:k1, :] + beta * packed lower(C)
// (syrk.jl:110-254): the SYRK chains over the reduction rows k0 .. k1-1, stored
// column-major packed, (0,0),(1,0)..(n-1,0),(1,1)..; limb stride lsc.
extern "C" int mflab_syrk_packed(mflab_handle *h, void *stream, int limbs, int64_t n, int64_t kp,
                                 int64_t k0, int64_t k1, const double *P, int64_t ldp, int64_t lsp,
                                 double *C, int64_t lsc, const double *alpha, const double *beta) {
    MFLAB_RANGE("mflab_syrk_packed");
    if (!h || !mfl::valid_limbs(limbs)) return MFLAB_ERR_UNSUPPORTED;
    if (n < 0 || kp < 0 || !alpha || !beta) return MFLAB_ERR_ARG;
    if (!(0 <= k0 && k0 < k1 && k1 <= kp)) return MFLAB_ERR_ARG;
    if (n == 0) return MFLAB_OK;
    const int64_t len = n * (n + 1) / 2;
    if (ldp < kp || lsc < len) return MFLAB_ERR_ARG;
    if (mfl::views_overlap(C, len, lsc, len, 1, limbs, P, ldp, lsp, kp, n)) return MFLAB_ERR_ALIAS;
    return mfl::launch_mm(limbs, true, false, 1, false, n, n, k1 - k0,
                          Mat{(double *)P + k0, ldp, lsp}, Mat{(double *)P + k0, ldp, lsp},
                          Mat{C, len, lsc}, alpha, beta, (cudaStream_t)stream, nullptr,
                          mfl::MM_PACKED);
}

// B = alpha * op(A) * B (side 0) or alpha * B * op(A) (side 1), in place
// (trmm.jl:82-131).  Each B(i,j) is one ascending chain over the triangle of
// op(A) (trmm.jl:1-80): left lower k = 0..i, left upper k = i..m-1, right
// lower k = j..n-1, right upper k = 0..j, the diagonal term B(i,j) itself for
// diag = unit.  B is saved to the handle's scratch and the product written
// back, so every chain reads the original B.
extern "C" int mflab_trmm(mflab_handle *h, void *stream, int limbs, int side, int uplo, int trans,
                          int diag, int64_t m, int64_t n, const double *A, int64_t lda,
                          int64_t lsa, double *B, int64_t ldb, int64_t lsb, const double *alpha) {
    MFLAB_RANGE("mflab_trmm");
    if (!h || !mfl::valid_limbs(limbs)) return MFLAB_ERR_UNSUPPORTED;
    if ((side | uplo | trans | diag) & ~1) return MFLAB_ERR_FLAG;
    if (m < 0 || n < 0 || !alpha) return MFLAB_ERR_ARG;
    const int64_t na = side ? n : m;
    if (m == 0 || n == 0) return MFLAB_OK;
    if (lda < na || ldb < m) return MFLAB_ERR_ARG;
    if (mfl::views_overlap(B, ldb, lsb, m, n, limbs, A, lda, lsa, na, na)) return MFLAB_ERR_ALIAS;
    cudaStream_t s = (cudaStream_t)stream;
    const size_t plane = (size_t)m * n;
    int rc = mflab_reserve_scratch(h, plane * limbs * sizeof(double));
    if (rc) return rc;
    double *saved = (double *)h->scratch;
    for (int l = 0; l < limbs; ++l) {
        cudaError_t e = cudaMemcpy2DAsync(saved + l * plane, m * sizeof(double), B + l * lsb,
                                          ldb * sizeof(double), m * sizeof(double), n,
                                          cudaMemcpyDeviceToDevice, s);
        if (e != cudaSuccess) return mfl::record_cuda_error(e, "trmm save");
    }
    const Mat Bs{saved, m, (int64_t)plane}, Am{(double *)A, lda, lsa}, Bm{B, ldb, lsb};
    const bool eff_lower = (uplo == 0) == (trans == 0);
    const int unit = diag ? mfl::MM_UNIT : 0;
    if (side == 0)
        return mfl::launch_trmm_mm(limbs, trans, false, (eff_lower ? 0 : mfl::MM_KGE) | unit, m,
                                   n, m, Am, Bs, Bm, alpha, s);
    return mfl::launch_trmm_mm(limbs, 0, trans != 0,
                               mfl::MM_RIGHT | (eff_lower ? mfl::MM_KGE : 0) | unit, m, n, n, Bs,
                               Am, Bm, alpha, s);
}

extern "C" int mflab_syrk_lower(mflab_handle *h, void *stream, int limbs, int64_t n, int64_t k,
                                const double *P, int64_t ldp, int64_t lsp, double *C, int64_t ldc,
                                int64_t lsc, const double *alpha, const double *beta) {
    MFLAB_RANGE("mflab_syrk_lower");
    if (!h || !mfl::valid_limbs(limbs)) return MFLAB_ERR_UNSUPPORTED;
    if (n < 0 || k < 0 || !alpha || !beta) return MFLAB_ERR_ARG;
    if (n == 0) return MFLAB_OK;
    if (ldp < (k > 0 ? k : 1) || ldc < n) return MFLAB_ERR_ARG;
    if (mfl::views_overlap(C, ldc, lsc, n, n, limbs, P, ldp, lsp, k, n)) return MFLAB_ERR_ALIAS;
    return mfl::launch_mm(limbs, true, false, 1, false, n, n, k, Mat{(double *)P, ldp, lsp},
                          Mat{(double *)P, ldp, lsp}, Mat{C, ldc, lsc}, alpha, beta,
                          (cudaStream_t)stream);
}

extern "C" int mflab_gemmt_lower(mflab_handle *h, void *stream, int limbs, int64_t n, int64_t k,
                                 const double *A, int64_t lda, int64_t lsa, const double *B,
                                 int64_t ldb, int64_t lsb, double *C, int64_t ldc, int64_t lsc,
                                 const double *alpha, const double *beta) {
    MFLAB_RANGE("mflab_gemmt_lower");
    if (!h || !mfl::valid_limbs(limbs)) return MFLAB_ERR_UNSUPPORTED;
    if (n < 0 || k < 0 || !alpha || !beta) return MFLAB_ERR_ARG;
    if (n == 0) return MFLAB_OK;
    if (lda < n || ldb < n || ldc < n) return MFLAB_ERR_ARG;
    if (mfl::views_overlap(C, ldc, lsc, n, n, limbs, A, lda, lsa, n, k) ||
        mfl::views_overlap(C, ldc, lsc, n, n, limbs, B, ldb, lsb, n, k))
        return MFLAB_ERR_ALIAS;
    return mfl::launch_mm(limbs, false, true, 1, false, n, n, k, Mat{(double *)A, lda, lsa},
                          Mat{(double *)B, ldb, lsb}, Mat{C, ldc, lsc}, alpha, beta,
                          (cudaStream_t)stream);
}
