// Panel and block-row kernels of the blocked multi-double LU (lu.jl:34-195):
// per panel of at most 16 columns one cluster launch factors the panel, one
// launch applies its interchanges to the other columns and solves U12.  Every
// entry receives the reference's operations in its order: the pivot is the
// first strictly larger |A[r,k]|, the multipliers are A[r,k] * (1 / A[k,k]),
// the panel's entries take one rank-1 term per step.
#include "cluster.cuh"
#include "mf_device.cuh"
#include "mflab_internal.h"

#include <algorithm>

namespace mfl {

// The panel's rows stay in registers, one row per thread, dealt to the
// cluster's warps in groups of 32; register j holds column k + j at step k (the
// rank-1 term writes its result one register down).  Interchanges are logical:
// a thread knows its row's current position, and the panel is written back at
// the end.  Per step:
//   * every CTA reduces its candidates for column k + 1 as soon as that column
//     has its term; the last warp then forms the candidate's reciprocal (a
//     serial chain of about 0.35 us in x2 and 2.4 us in x4) while the others
//     apply the term to the remaining columns;
//   * the candidate's row and reciprocal are written into every CTA of the
//     cluster, one cluster barrier, and every warp picks the same winner from
//     its own shared memory.
// Two buffers alternate: a CTA overwrites a buffer only after the barrier of
// the step in between.  x4, n = 701: 121 us a panel (31 launches of a
// one-CTA pivot search and a rank-1 update: 270 us); its interchanges and U12:
// 12 us (39 us in two launches, one thread per column for the swaps).
constexpr int LP_NT = 256, LP_WARPS = LP_NT / 32;

template <int N>
struct LpCand {
    double u[LU_PANEL_W][N];  // the candidate row, columns k ..
    double inv[N];
    int row, pad;             // its position, -1 without an active row
};

template <int N>
struct LpShared {
    LpCand<N> recv[2][MAX_CLUSTER];
    double stage[LU_PANEL_W][N], inv[N];
    double red[LP_WARPS][N];
    int redi[LP_WARPS];
};

// best candidate over groups of `width` lanes by |v|, in every lane
template <int N>
__device__ __forceinline__ void lp_lanes(mf<N> &v, int &i, int width) {
    for (int off = width / 2; off > 0; off >>= 1) {
        mf<N> o;
#pragma unroll
        for (int l = 0; l < N; ++l) o.v[l] = __shfl_xor_sync(0xffffffffu, v.v[l], off);
        const int oi = __shfl_xor_sync(0xffffffffu, i, off);
        const mf<N> a = abs_mf(v), b = abs_mf(o);
        bool take = oi >= 0;
        if (take && i >= 0) take = gt(b, a) ? true : gt(a, b) ? false : oi < i;
        if (take) {
            v = o;
            i = oi;
        }
    }
}

template <int N>
__global__ void __launch_bounds__(LP_NT)
    lu_panel_kernel(int64_t m, Mat A, int64_t first, int w, int64_t *ipiv, int *info) {
    if (*info) return;  // the same in every thread of the cluster
    extern __shared__ double lp_fin[];  // [w][LP_NT][N] final values of each thread's row
    __shared__ LpShared<N> sh;
    const int t = threadIdx.x, lane = t % 32, warp = t / 32;
    uint32_t rank, ncu;
    asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(rank));
    asm volatile("mov.u32 %0, %%cluster_nctarank;" : "=r"(ncu));
    const int nc = (int)ncu;
    const int64_t orig = first + 32 * (rank + (int64_t)nc * warp) + lane;
    const bool has = orig < m;
    int cur = (int)orig;
    bool act = has;
    mf<N> row[LU_PANEL_W];
#pragma unroll
    for (int j = 0; j < LU_PANEL_W; ++j)
        row[j] = has && j < w ? load_mf<N>(A.p, A.ld, A.ls, orig, first + j) : from_double<N>(0.0);
    ld_cluster_sync();  // every CTA has started and holds its rows

    mf<N> l = from_double<N>(0.0);
    const LpCand<N> *win = nullptr;
    auto final_value = [&](int c, const mf<N> &v) {
        ld_put<N>(&lp_fin[((size_t)c * LP_NT + t) * N], v);
    };
    int c = -1;  // the column whose term is being applied; -1 before the first
    for (;; ++c) {
        if (c >= 0) {
            // the winner of column c among the cluster's candidates
            const int64_t k = first + c;
            const LpCand<N> *cand = sh.recv[c & 1];
            mf<N> v = lane < nc ? ld_get<N>(cand[lane].u[0]) : from_double<N>(0.0);
            const int mine = lane < nc ? cand[lane].row : -1;
            int prow = mine;
            lp_lanes(v, prow, 32);
            const unsigned q = __ballot_sync(0xffffffffu, lane < nc && mine == prow);
            win = &cand[__ffs(q) - 1];
            if (rank == 0 && t == 0) ipiv[k] = (int64_t)prow + 1;
            if (iszero(v)) {  // the same in every thread of the cluster
                if (rank == 0 && t == 0) *info = (int)(k + 1);
                break;
            }
            if (act && cur == prow) {  // the pivot row is final: its part of U
#pragma unroll
                for (int j = 0; j < LU_PANEL_W; ++j)
                    if (c + j < w) final_value(c + j, row[j]);
                cur = (int)k;
                act = false;
            } else if (act && cur == (int)k) {
                cur = prow;  // the row the pivot row displaces
            }
            if (__any_sync(0xffffffffu, act)) {
                l = mul(row[0], ld_get<N>(win->inv));
                if (act) final_value(c, l);
                if (c + 1 < w) row[0] = submul(row[1], l, ld_get<N>(win->u[1]));
            }
            if (c + 1 == w) {
                c = w;
                break;
            }
        }
        // this CTA's candidate for column c + 1
        mf<N> best = row[0];
        int bi = act ? cur : -1;
        lp_lanes(best, bi, 32);
        if (lane == 0) {
            ld_put<N>(sh.red[warp], best);
            sh.redi[warp] = bi;
        }
        __syncthreads();
        best = ld_get<N>(sh.red[lane % LP_WARPS]);
        bi = sh.redi[lane % LP_WARPS];
        lp_lanes(best, bi, LP_WARPS);
        if (warp == LP_WARPS - 1 && bi >= 0 && !iszero(best)) {
            const mf<N> iv = inv(best);
            if (lane == 0) ld_put<N>(sh.inv, iv);
        }
        __syncwarp();
        // the term on the remaining columns
        if (c >= 0 && __any_sync(0xffffffffu, act)) {
#pragma unroll
            for (int j = 1; j < LU_PANEL_W - 1; ++j)
                if (c + 1 + j < w) row[j] = submul(row[j + 1], l, ld_get<N>(win->u[j + 1]));
        }
        const int left = w - (c + 1);  // columns of the candidate row
        if (act && cur == bi) {
#pragma unroll
            for (int j = 0; j < LU_PANEL_W; ++j)
                if (j < left) ld_put<N>(sh.stage[j], row[j]);
        }
        __syncthreads();
        LpCand<N> *to = &sh.recv[(c + 1) & 1][rank];
        const int per = (left + 1) * N;  // doubles: the row and the reciprocal
        for (int e = t; e < nc * per; e += LP_NT) {
            const int target = e / per, x = e % per;
            const bool isinv = x >= left * N;
            const double v = isinv ? sh.inv[x - left * N] : (&sh.stage[0][0])[x];
            ld_remote_f64(ld_remote(isinv ? &to->inv[x - left * N] : &to->u[0][0] + x, target), v);
        }
        if (t < nc) ld_remote_s32(ld_remote(&to->row, (uint32_t)t), bi);
        ld_cluster_sync();
    }
    // a zero pivot at column c leaves the active rows as they are
    if (act && c < w) {
#pragma unroll
        for (int j = 0; j < LU_PANEL_W; ++j)
            if (c + j < w) final_value(c + j, row[j]);
    }
    if (!has) return;
    for (int j = 0; j < w; ++j)
        store_mf<N>(A.p, A.ld, A.ls, cur, first + j, ld_get<N>(&lp_fin[((size_t)j * LP_NT + t) * N]));
}

// The interchanges of panel steps first .. first + w - 1 (ipiv, ascending, as
// the sequential row swaps of lu.jl) on every column outside the panel and, on
// columns first + w .. solve_hi - 1, the block row U12 = inv(L11) A12 (unit
// lower, each row its ascending chain).  The swaps move at most 2w rows: one
// warp per CTA replays them on its lanes' row numbers, then a column is one
// gather by a warp and a solve over its lanes.  Only the steps that ran are
// replayed: after a zero pivot at step info-1 (no interchange there) the later
// ones did not, and nothing is solved.
constexpr int LSW_WARPS = 4;

template <int N>
__global__ void __launch_bounds__(32 * LSW_WARPS)
    lu_swap_solve_kernel(int64_t n, int64_t solve_hi, Mat A, int64_t first, int w,
                         const int64_t *ipiv, const int *info) {
    const int st = *info;
    if (st < 0) return;
    const int steps = st == 0 ? w : (int)(st - 1 - first < w ? st - 1 - first : w);
    if (steps <= 0 && st != 0) return;
    __shared__ int rows[32], src[32], count;
    __shared__ double L[N][LU_PANEL_W][LU_PANEL_W];  // L[.][k][row]
    const int lane = threadIdx.x % 32, warp = threadIdx.x / 32;
    if (warp == 0) {
        int row = lane < w ? (int)first + lane : -1, content = lane, cnt = w;
        for (int i = 0; i < steps; ++i) {
            const int p = (int)(ipiv[first + i] - 1);
            int b = p - (int)first;
            if (b >= w) {
                const unsigned hit = __ballot_sync(0xffffffffu, lane >= w && row == p);
                b = hit ? __ffs(hit) - 1 : cnt;
                if (!hit) {
                    if (lane == cnt) row = p;
                    ++cnt;
                }
            }
            const int ci = __shfl_sync(0xffffffffu, content, i);
            const int cb = __shfl_sync(0xffffffffu, content, b);
            if (lane == i) content = cb;
            if (lane == b) content = ci;
        }
        const int from = __shfl_sync(0xffffffffu, row, content & 31);
        rows[lane] = row;
        src[lane] = from;
        if (lane == 0) count = cnt;
    } else {
        for (int e = threadIdx.x - 32; e < w * w; e += 32 * (LSW_WARPS - 1)) {
            const int i = e % w, k = e / w;
            if (i <= k) continue;
            const mf<N> a = load_mf<N>(A.p, A.ld, A.ls, first + i, first + k);
#pragma unroll
            for (int l = 0; l < N; ++l) L[l][k][i] = a.v[l];
        }
    }
    __syncthreads();
    const bool in = lane < count;
    const int to = rows[lane], from = src[lane];
    for (int64_t j = (int64_t)blockIdx.x * LSW_WARPS + warp; j < n - w;
         j += (int64_t)gridDim.x * LSW_WARPS) {
        const int64_t col = j < first ? j : j + w;
        const bool solve = st == 0 && col >= first && col < solve_hi;
        mf<N> v = in ? load_mf<N>(A.p, A.ld, A.ls, from, col) : from_double<N>(0.0);
        __syncwarp();
        if (solve) {
            for (int k = 0; k + 1 < w; ++k) {
                mf<N> x, a;
#pragma unroll
                for (int l = 0; l < N; ++l) x.v[l] = __shfl_sync(0xffffffffu, v.v[l], k);
                if (lane > k && lane < w) {
#pragma unroll
                    for (int l = 0; l < N; ++l) a.v[l] = L[l][k][lane];
                    v = submul(v, a, x);
                }
            }
        }
        if (in) store_mf<N>(A.p, A.ld, A.ls, to, col, v);
    }
}

// MFLAB_ERR_UNSUPPORTED: more rows than the largest cluster holds
template <int N>
static int lu_panel_n(int64_t m, Mat A, int64_t first, int w, int64_t *ipiv, int *info,
                      cudaStream_t s) {
    auto kern = lu_panel_kernel<N>;
    constexpr size_t smem = sizeof(double) * LU_PANEL_W * LP_NT * N;
    static std::atomic<unsigned long long> configured{0}, asked{0}, sixteen{0};
    int rc = set_smem_once((const void *)kern, (int)smem, configured, "getrf panel attribute");
    if (rc) return rc;
    int most = 0;
    rc = largest_cluster((const void *)kern, LP_NT, smem, asked, sixteen, &most);
    if (rc) return rc;
    const int64_t rows = m - first;
    if (rows > (int64_t)most * LP_NT || m > 0x7fffffff) return MFLAB_ERR_UNSUPPORTED;
    int nc = 1;
    while (nc < most && nc * 32 < rows) nc *= 2;
    cudaLaunchConfig_t cfg = {};
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = (unsigned)nc;
    attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
    cfg.gridDim = dim3((unsigned)nc);
    cfg.blockDim = dim3(LP_NT);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    return record_cuda_error(cudaLaunchKernelEx(&cfg, kern, m, A, first, w, ipiv, info),
                             "getrf panel");
}

template <int N>
static int lu_swap_solve_n(int64_t n, int64_t solve_hi, Mat A, int64_t first, int w,
                           const int64_t *ipiv, const int *info, cudaStream_t s) {
    if (n <= w) return MFLAB_OK;
    const int64_t grid = std::min<int64_t>((n - w + LSW_WARPS - 1) / LSW_WARPS, 148 * 8);
    lu_swap_solve_kernel<N><<<(unsigned)grid, 32 * LSW_WARPS, 0, s>>>(n, solve_hi, A, first, w, ipiv,
                                                                     info);
    return record_cuda_error(cudaGetLastError(), "getrf block row");
}

int launch_lu_panel(int N, int64_t m, Mat A, int64_t first, int w, int64_t *ipiv, int *info,
                    cudaStream_t s) {
    switch (N) {
    case 2: return lu_panel_n<2>(m, A, first, w, ipiv, info, s);
    case 3: return lu_panel_n<3>(m, A, first, w, ipiv, info, s);
    case 4: return lu_panel_n<4>(m, A, first, w, ipiv, info, s);
    default: return MFLAB_ERR_UNSUPPORTED;
    }
}

int launch_lu_swap_solve(int N, int64_t n, int64_t solve_hi, Mat A, int64_t first, int w,
                         const int64_t *ipiv, const int *info, cudaStream_t s) {
    switch (N) {
    case 2: return lu_swap_solve_n<2>(n, solve_hi, A, first, w, ipiv, info, s);
    case 3: return lu_swap_solve_n<3>(n, solve_hi, A, first, w, ipiv, info, s);
    case 4: return lu_swap_solve_n<4>(n, solve_hi, A, first, w, ipiv, info, s);
    default: return MFLAB_ERR_UNSUPPORTED;
    }
}

}  // namespace mfl
