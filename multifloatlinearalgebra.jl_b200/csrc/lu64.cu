// Repeated binary64 LU solves with inverted diagonal blocks (the correction
// solves of the mixed-precision LU solver: one binary64 factor, many solves
// with a few right-hand sides each).
//
// No reference counterpart and no reference order to keep: the binary64
// factor only drives iterative refinement, whose Float64xN residuals decide
// the accuracy.  A forward or backward substitution with a few right-hand
// sides is a chain of dependent steps; done row by row or in 64-row blocks
// with a triangular solve and a GEMM per block it is launch- and
// latency-bound (hundreds of small kernels per solve).  Here the 128 x 128
// diagonal blocks of L (unit lower) and U are inverted once after the
// factorization, the row interchanges are turned into one permutation, and
// every off-diagonal block column is premultiplied by its inverted diagonal
// block, M_{r,i} = L_{r,i} inv(DL_i) (rows below block i) and
// U_{r,i} inv(DU_i) (rows above it), all stored in a caller-owned workspace.
// A solve is then one gather and one kernel per block row and direction,
// whose CTAs share the work without redundancy and without waiting for one
// another: with b_i the block's current right-hand side rows,
//   the block's rows:      y_i = inv(D_i) b_i          (a few CTAs)
//   every remaining row r: W_r -= M_{r,i} b_i          (= L_{r,i} y_i)
//
// Workspace: perm[n] int32 (rounded up to 256 bytes), then the inverted L
// blocks and the inverted U blocks, nblk = ceil(n / 128) of 128 x 128
// doubles each (column-major, ld 128; a last partial block is padded), then
// ML and MU, n x n column-major (ld n) each, of which the blocks below /
// above the diagonal are used.
#include <algorithm>

#include "mflab_internal.h"

MFLAB_DEBUG_RECORD(lu64)

namespace mfl {

namespace {

constexpr int IB = 128;        // diagonal block size
constexpr int64_t PIVOT_PERM_MAXN_LU64 = 24576;  // indices and pivots in shared memory (192 KB)

size_t perm_bytes(int64_t n) { return ((size_t)n * 4 + 255) / 256 * 256; }
int64_t nblocks(int64_t n) { return (n + IB - 1) / IB; }

// In-place inversion of one diagonal block (jb x jb, jb <= 128) in shared
// memory: unit lower L (which = 0) or upper U (which = 1); block b of the
// factor goes to inv + b * IB * IB (ld IB).  One CTA per (block, which).
//   L: for j = jb-1 .. 0, column j of inv(L) below the diagonal is
//      -inv(L)[j+1:, j+1:] L[j+1:, j];
//   U: for j = 0 .. jb-1, inv(U)[j][j] = 1 / U[j][j] and the column above it
//      is -inv(U)[:j, :j] U[:j, j] inv(U)[j][j].
__global__ void __launch_bounds__(IB)
    lu64_inv_diag_kernel(int64_t n, const double *__restrict__ LU, int64_t ldl, double *invL,
                         double *invU) {
    extern __shared__ double sm[];  // [IB][IB + 1] block, then [IB] column copy
    double *blk = sm;
    double *v = sm + IB * (IB + 1);
    const int b = blockIdx.x, which = blockIdx.y, t = threadIdx.x;
    const int64_t j0 = (int64_t)b * IB;
    const int jb = (int)(n - j0 < IB ? n - j0 : IB);
    // column c of the block at blk[c * (IB + 1) + r]
    for (int c = 0; c < jb; ++c)
        if (t < jb) blk[c * (IB + 1) + t] = LU[(j0 + c) * ldl + j0 + t];
    __syncthreads();
    if (which == 0) {
        for (int j = jb - 1; j >= 0; --j) {
            if (t < jb) v[t] = t > j ? blk[j * (IB + 1) + t] : 0.0;  // L[:, j] below j
            __syncthreads();
            if (t > j && t < jb) {
                // row t of inv(L)[j+1:, j+1:] (final) times L[j+1:, j]
                double acc = v[t];  // inv(L)[t][t] = 1
                for (int i = j + 1; i < t; ++i) acc = fma(blk[i * (IB + 1) + t], v[i], acc);
                blk[j * (IB + 1) + t] = -acc;
            }
            __syncthreads();
        }
    } else {
        for (int j = 0; j < jb; ++j) {
            if (t <= j) v[t] = blk[j * (IB + 1) + t];  // U[:j+1, j]
            __syncthreads();
            const double djj = 1.0 / v[j];
            if (t < j) {
                // row t of inv(U)[:j, :j] (final) times U[:j, j]
                double acc = 0.0;
                for (int i = t; i < j; ++i) acc = fma(blk[i * (IB + 1) + t], v[i], acc);
                blk[j * (IB + 1) + t] = -acc * djj;
            } else if (t == j) {
                blk[j * (IB + 1) + t] = djj;
            }
            __syncthreads();
        }
    }
    // store with zeros outside the triangle and the unit diagonal of inv(L)
    double *dst = (which == 0 ? invL : invU) + (int64_t)b * IB * IB;
    for (int c = 0; c < IB; ++c) {
        double x = 0.0;
        if (t < jb && c < jb) {
            if (which == 0) x = t > c ? blk[c * (IB + 1) + t] : (t == c ? 1.0 : 0.0);
            else x = t <= c ? blk[c * (IB + 1) + t] : 0.0;
        }
        dst[c * IB + t] = x;
    }
}

// perm[i] = the original row that ends up in row i after the interchanges
// ipiv[0..n) (1-based, applied in ascending order): replayed by one thread on
// index and pivot arrays in shared memory
__global__ void lu64_perm_kernel(int64_t n, const int64_t *ipiv, int *perm) {
    extern __shared__ int sidx[];  // [n] indices, [n] pivots
    int *spiv = sidx + n;
    for (int64_t i = threadIdx.x; i < n; i += blockDim.x) {
        sidx[i] = (int)i;
        spiv[i] = (int)(ipiv[i] - 1);
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        for (int64_t k = 0; k < n; ++k) {
            const int p = spiv[k];
            if (p != k) {
                const int x = sidx[k];
                sidx[k] = sidx[p];
                sidx[p] = x;
            }
        }
    }
    __syncthreads();
    for (int64_t i = threadIdx.x; i < n; i += blockDim.x) perm[i] = sidx[i];
}

// W[i, c] = B[perm[i], c]
__global__ void lu64_gather_kernel(int64_t n, int64_t nrhs, const double *B, int64_t ldb,
                                   const int *perm, double *W, int64_t ldw) {
    const int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (e >= n * nrhs) return;
    const int64_t i = e % n, c = e / n;
    W[c * ldw + i] = B[c * ldb + perm[i]];
}

// One block step of a triangular solve.  Block i spans rows [j0, j0 + jb)
// and b = W[j0 : j0 + jb, :] holds its final right-hand side rows.
//   CTA k < ceil(jb / 32):  Out[j0 + 32k + r, c] = (inv(D_i) b)[32k + r, c]
//   the other CTAs, 32 rows r of [r_begin, r_end) each:
//                           W[r, c] -= (M[r, block i] b)[r, c]
// The rows written to W are outside the block, so no CTA reads what another
// writes.  A CTA stages its 32 x jb slice of inv(D_i) or M (k-major) and b
// (16 right-hand sides at a time) in shared memory; thread (row, warp)
// accumulates two right-hand sides over the jb columns.
constexpr int MS_ROWS = 32, MS_NT = 256, MS_RHS = 16;

__global__ void __launch_bounds__(MS_NT)
    lu64_mstep_kernel(int64_t nrhs, int64_t j0, int jb, const double *__restrict__ M, int64_t ldm,
                      const double *__restrict__ inv, double *W, int64_t ldw, double *Out,
                      int64_t ldo, int64_t r_begin, int64_t r_end) {
    static_assert(MS_NT / 32 * 2 == MS_RHS, "two right-hand sides per warp");
    __shared__ double tile[IB][MS_ROWS];             // [k][row]
    __shared__ __align__(16) double bT[IB][MS_RHS];  // [k][rhs]
    const int t = threadIdx.x, lane = t % 32, warp = t / 32;
    const int ndiag = (jb + MS_ROWS - 1) / MS_ROWS;
    const bool diag = (int)blockIdx.x < ndiag;
    // diag: the first row inside the block; else the first absolute row of R
    const int64_t rb = diag ? (int64_t)blockIdx.x * MS_ROWS
                            : r_begin + ((int64_t)blockIdx.x - ndiag) * MS_ROWS;
    const int64_t left = diag ? (int64_t)jb - rb : r_end - rb;
    const int nrows = (int)(left < MS_ROWS ? left : MS_ROWS);
    // launched as a programmatic dependent of the previous step: the next
    // step may start its prologue now, and this one stages its slice of M
    // or inv(D_i) (written before the solve) before waiting for the
    // previous step's results
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    // all loads of a thread in flight together (unrolled, then stored)
    {
        const double *src = diag ? inv + rb : M + j0 * ldm + rb;
        const int64_t ld = diag ? IB : ldm;
        double x[IB * MS_ROWS / MS_NT];
#pragma unroll
        for (int u = 0; u < IB * MS_ROWS / MS_NT; ++u) {
            const int e = t + u * MS_NT, r = e % MS_ROWS, k = e / MS_ROWS;
            x[u] = (r < nrows && k < jb &&
                    MFLAB_IDX_OK(rb + r < (diag ? (int64_t)IB : ldm), 7, rb + r, k))
                       ? src[(int64_t)k * ld + r]
                       : 0.0;
        }
#pragma unroll
        for (int u = 0; u < IB * MS_ROWS / MS_NT; ++u) {
            const int e = t + u * MS_NT;
            tile[e / MS_ROWS][e % MS_ROWS] = x[u];
        }
    }
    // the previous steps have completed and their writes are visible
    asm volatile("griddepcontrol.wait;" ::: "memory");
    for (int64_t c0 = 0; c0 < nrhs; c0 += MS_RHS) {
        const int cw = (int)(nrhs - c0 < MS_RHS ? nrhs - c0 : MS_RHS);
        double y[IB * MS_RHS / MS_NT];
#pragma unroll
        for (int u = 0; u < IB * MS_RHS / MS_NT; ++u) {
            const int e = t + u * MS_NT, k = e % IB, c = e / IB;
            y[u] = (k < jb && c < cw) ? W[(c0 + c) * ldw + j0 + k] : 0.0;
        }
#pragma unroll
        for (int u = 0; u < IB * MS_RHS / MS_NT; ++u) {
            const int e = t + u * MS_NT;
            bT[e % IB][e / IB] = y[u];
        }
        __syncthreads();
        double a0 = 0.0, a1 = 0.0;
#pragma unroll 8
        for (int k = 0; k < IB; ++k) {
            const double m = tile[k][lane];
            const double2 bb = *(const double2 *)&bT[k][2 * warp];
            a0 = fma(m, bb.x, a0);
            a1 = fma(m, bb.y, a1);
        }
        const int c = 2 * warp;
        if (lane < nrows) {
            if (diag) {
                if (c < cw) Out[(c0 + c) * ldo + j0 + rb + lane] = a0;
                if (c + 1 < cw) Out[(c0 + c + 1) * ldo + j0 + rb + lane] = a1;
            } else {
                if (c < cw) W[(c0 + c) * ldw + rb + lane] -= a0;
                if (c + 1 < cw) W[(c0 + c + 1) * ldw + rb + lane] -= a1;
            }
        }
        __syncthreads();
    }
}

// one step, launched with programmatic stream serialization (its prologue
// overlaps the previous step); grid: the block's row groups, then R's
int mstep_launch(cudaStream_t s, int64_t nrhs, int64_t j0, int jb, const double *M, int64_t ldm,
                 const double *inv, double *W, int64_t ldw, double *Out, int64_t ldo,
                 int64_t r_begin, int64_t r_end) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)((jb + MS_ROWS - 1) / MS_ROWS +
                                  (r_end - r_begin + MS_ROWS - 1) / MS_ROWS));
    cfg.blockDim = dim3(MS_NT);
    cfg.dynamicSmemBytes = 0;
    cfg.stream = s;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    return record_cuda_error(cudaLaunchKernelEx(&cfg, lu64_mstep_kernel, nrhs, j0, jb, M, ldm,
                                                inv, W, ldw, Out, ldo, r_begin, r_end),
                             "lu64 solve step");
}

// The same solve in one cooperative launch, every CTA 32 rows of the right-hand
// side in registers.  A step of the block kernel above is bound by launch and
// load latency (7.2 us a step at n = 4096, 64 steps); here the owners of block
// i publish its rows and every CTA that still needs them reads them, applies its
// 32 x 128 slice of M (or inv(D_i), an owner) and goes on to the next block.
// The rows are their own flags: the buffer starts as all ones (a NaN no value
// is written as), and a reader polls its own words until none of them is, so a
// step costs one store and one load through L2 instead of a fence, a flag and
// then the load.  The rows are written LS_COPIES times: copy 0 is for the
// owners of the block itself and of the next one, the only CTAs the chain of
// steps waits for, and the others' polls are spread over the rest.  The slices
// do not depend on the solve: two are prefetched into shared memory ahead of
// the rows.  Arithmetic and results are the block kernel's.  All CTAs are
// co-resident (cooperative launch); a wait that runs out (LS_SPIN polls, or the
// handle's limit) records error 6 in the handle's status word and the CTA leaves
// at its next barrier, the others as their waits run out or see the abort word.
// B is then not solved: a caller reads the status word before it uses the
// result.  n = 4096, 16 right-hand sides: 220 us (460 us as 64 launches, 348 us
// with flags, 286 us before the 2 x 2 tiles below).
constexpr int LS_STAGES = 3, LS_ERR_TIMEOUT = 6;
constexpr long long LS_SPIN = 1LL << 21;
constexpr int64_t LS_MAX_RHS = 32;  // more right-hand sides: the block kernel
constexpr unsigned long long LS_UNSET = ~0ULL;
constexpr int LS_COPIES = 4;

__device__ __forceinline__ void ls_cp_async(void *dst, const void *src, int bytes, bool pred) {
    const unsigned d = (unsigned)__cvta_generic_to_shared(dst);
    if (bytes == 16)
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(d), "l"(src),
                     "r"(pred ? 16 : 0)
                     : "memory");
    else
        asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;" ::"r"(d), "l"(src),
                     "r"(pred ? 8 : 0)
                     : "memory");
}
__device__ __forceinline__ unsigned long long ls_word(double v) {
    const unsigned long long w = (unsigned long long)__double_as_longlong(v);
    return w == LS_UNSET ? 0x7ff8000000000000ULL : w;
}

struct LsShared {
    double tile[LS_STAGES][IB][MS_ROWS];  // slices of M or inv(D), [k][row]
    double b[IB][MS_RHS];                 // the block's rows
};

// pub: [chunk][2][nblk][LS_COPIES][IB][MS_RHS] words, all LS_UNSET at the start
__global__ void __launch_bounds__(MS_NT)
    lu64_solve_kernel(int64_t n, int64_t nrhs, const int *perm, const double *__restrict__ invL,
                      const double *__restrict__ invU, const double *__restrict__ ML,
                      const double *__restrict__ MU, double *B, int64_t ldb,
                      unsigned long long *pub, int *abort_word, int *err, long long spin) {
    extern __shared__ __align__(16) uint8_t ls_raw[];
    LsShared &sh = *reinterpret_cast<LsShared *>(ls_raw);
    __shared__ int s_stop;
    const int t = threadIdx.x, lane = t % 32, warp = t / 32;
    const int nb = (int)((n + IB - 1) / IB);
    const int64_t rb = (int64_t)blockIdx.x * MS_ROWS;
    const int nrows = (int)(n - rb < MS_ROWS ? n - rb : MS_ROWS);
    const int own = (int)(rb / IB), inner = (int)(rb % IB);
    // blocks 0 .. own forward, then nb-1 .. own backward
    const int fwd = own + 1, steps = fwd + nb - own;
    auto block_of = [&](int s) { return s < fwd ? s : nb - 1 - (s - fwd); };
    auto rows_of = [&](int i) { return (int)(n - (int64_t)i * IB < IB ? n - (int64_t)i * IB : IB); };
    // 16-byte copies where every column of the slice starts on 16 bytes
    const bool wide = nrows == MS_ROWS && (n & 1) == 0 &&
                      (((uintptr_t)invL | (uintptr_t)invU | (uintptr_t)ML | (uintptr_t)MU) & 15) == 0;
    auto prefetch = [&](int s) {
        if (s < steps) {
            const int i = block_of(s), jb = rows_of(i);
            const bool forward = s < fwd;
            const double *src = i == own ? (forward ? invL : invU) + (int64_t)i * IB * IB + inner
                                         : (forward ? ML : MU) + (int64_t)i * IB * n + rb;
            const int64_t ld = i == own ? IB : n;
            double(*tile)[MS_ROWS] = sh.tile[s % LS_STAGES];
            if (wide) {
                const int r = 2 * (t % 16), k0 = t / 16;
                const double *p = src + k0 * ld + r;
#pragma unroll
                for (int u = 0; u < IB / 16; ++u, p += 16 * ld)
                    ls_cp_async(&tile[k0 + 16 * u][r], k0 + 16 * u < jb ? p : src, 16,
                                k0 + 16 * u < jb);
            } else {
                const double *p = src + warp * ld + lane;
#pragma unroll
                for (int u = 0; u < IB / 8; ++u, p += 8 * ld) {
                    const bool ok = lane < nrows && warp + 8 * u < jb;
                    ls_cp_async(&tile[warp + 8 * u][lane], ok ? p : src, 8, ok);
                }
            }
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    if (t == 0) s_stop = 0;
    __syncthreads();
    // Warps 0-3 hold the right-hand sides, 2 rows x 2 columns per thread (16 x 8
    // per warp): a k step is then one 16-byte read of the slice and one of the
    // rows, a wavefront each, for four products; one row per lane and two
    // columns per warp over eight warps made three wavefronts for two.
    const bool holds = warp < 4;
    const int r0 = 16 * (warp & 1) + 2 * (lane % 8), q0 = 8 * (warp >> 1 & 1) + 2 * (lane / 8);
    bool stop = false;
    for (int64_t c0 = 0; c0 < nrhs && !stop; c0 += MS_RHS, pub += 2 * (int64_t)nb * LS_COPIES * IB * MS_RHS) {
        double w[2][2];
#pragma unroll
        for (int a = 0; a < 2; ++a)
#pragma unroll
            for (int c = 0; c < 2; ++c) {
                const bool in = holds && r0 + a < nrows && c0 + q0 + c < nrhs;
                w[a][c] = in ? B[(c0 + q0 + c) * ldb + perm[rb + r0 + a]] : 0.0;
            }
        for (int s = 0; s < LS_STAGES - 1; ++s) prefetch(s);
        for (int s = 0; s < steps; ++s) {
            const int i = block_of(s), dir = s < fwd ? 0 : 1, jb = rows_of(i);
            unsigned long long *rows = pub + ((int64_t)dir * nb + i) * LS_COPIES * IB * MS_RHS;
            if (i == own && holds) {  // this CTA's rows of the block are final
#pragma unroll
                for (int c = 0; c < LS_COPIES; ++c)
#pragma unroll
                    for (int a = 0; a < 2; ++a)
                        if (r0 + a < nrows)
                            asm volatile("st.volatile.global.v2.u64 [%0], {%1, %2};" ::"l"(
                                             rows + (int64_t)(c * IB + inner + r0 + a) * MS_RHS + q0),
                                         "l"(ls_word(w[a][0])), "l"(ls_word(w[a][1]))
                                         : "memory");
            }
            const int far = dir == 0 ? own - i : i - own;  // blocks until this CTA's own
            if (far > 1) rows += (int64_t)(1 + blockIdx.x % (LS_COPIES - 1)) * IB * MS_RHS;
            prefetch(s + LS_STAGES - 1);
            // the block's rows: every thread polls its own words
            constexpr int PER = IB * MS_RHS / (2 * MS_NT);
            unsigned long long y[PER][2];
            bool open = true;
            for (long long polls = 0; open; ++polls) {
                open = false;
#pragma unroll
                for (int u = 0; u < PER; ++u) {
                    const int e = 2 * (t + u * MS_NT);
                    y[u][0] = y[u][1] = 0;
                    if (e / MS_RHS < jb)
                        asm volatile("ld.volatile.global.v2.u64 {%0, %1}, [%2];"
                                     : "=l"(y[u][0]), "=l"(y[u][1])
                                     : "l"(rows + e)
                                     : "memory");
                }
#pragma unroll
                for (int u = 0; u < PER; ++u)
                    open = open || y[u][0] == LS_UNSET || y[u][1] == LS_UNSET;
                if (open && (polls >= spin ||
                             ((polls & 255) == 255 && *(volatile int *)abort_word))) {
                    if (atomicExch(abort_word, 1) == 0) atomicExch(err, LS_ERR_TIMEOUT);
                    s_stop = 1;
                    break;
                }
            }
#pragma unroll
            for (int u = 0; u < PER; ++u) {
                double2 v;
                v.x = __longlong_as_double((long long)y[u][0]);
                v.y = __longlong_as_double((long long)y[u][1]);
                *(double2 *)(&sh.b[0][0] + 2 * (t + u * MS_NT)) = v;
            }
            // the slice of step s has landed (the two newer groups may be open)
            asm volatile("cp.async.wait_group %0;" ::"n"(LS_STAGES - 1) : "memory");
            __syncthreads();
            stop = s_stop != 0;
            if (stop) break;
            const double(*tile)[MS_ROWS] = sh.tile[s % LS_STAGES];
            if (holds) {
                double x[2][2] = {{0.0, 0.0}, {0.0, 0.0}};
#pragma unroll 16
                for (int k = 0; k < IB; ++k) {
                    const double2 m = *(const double2 *)&tile[k][r0];
                    const double2 bb = *(const double2 *)&sh.b[k][q0];
                    x[0][0] = fma(m.x, bb.x, x[0][0]);
                    x[0][1] = fma(m.x, bb.y, x[0][1]);
                    x[1][0] = fma(m.y, bb.x, x[1][0]);
                    x[1][1] = fma(m.y, bb.y, x[1][1]);
                }
#pragma unroll
                for (int a = 0; a < 2; ++a)
#pragma unroll
                    for (int c = 0; c < 2; ++c) w[a][c] = i == own ? x[a][c] : w[a][c] - x[a][c];
            }
            __syncthreads();  // tile and b before they are written again
        }
        asm volatile("cp.async.wait_group 0;" ::: "memory");
        if (stop) break;
        // every CTA has read its right-hand side: this one's last block waited
        // for rows that depend on all of them
#pragma unroll
        for (int a = 0; a < 2; ++a)
#pragma unroll
            for (int c = 0; c < 2; ++c)
                if (holds && r0 + a < nrows && c0 + q0 + c < nrhs)
                    B[(c0 + q0 + c) * ldb + rb + r0 + a] = w[a][c];
        __syncthreads();
    }
}

// Scratch of the one-launch solve, or 0 where the block kernel is taken: more
// right-hand sides than two rounds are worth, or more CTAs than fit at once.
size_t solve_bytes(int64_t n, int64_t nrhs) {
    if (nrhs > LS_MAX_RHS) return 0;
    static std::atomic<unsigned long long> configured{0};
    if (set_smem_once((const void *)lu64_solve_kernel, (int)sizeof(LsShared), configured,
                      "lu64 solve attribute"))
        return 0;
    int dev = 0, sms = 0, per = 0;
    if (cudaGetDevice(&dev) != cudaSuccess ||
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess ||
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, lu64_solve_kernel, MS_NT,
                                                      sizeof(LsShared)) != cudaSuccess)
        return 0;
    if ((n + MS_ROWS - 1) / MS_ROWS > (int64_t)sms * per) return 0;
    const size_t chunks = (size_t)((nrhs + MS_RHS - 1) / MS_RHS), nb = (size_t)nblocks(n);
    return sizeof(double) * chunks * 2 * nb * LS_COPIES * IB * MS_RHS + 256;
}

std::atomic<unsigned long long> g_inv_configured{0};

}  // namespace
}  // namespace mfl

extern "C" int mflab_lu64_work_bytes(int64_t n, size_t *bytes) {
    if (n < 0 || !bytes) return MFLAB_ERR_ARG;
    *bytes = mfl::perm_bytes(n) + 2 * (size_t)mfl::nblocks(n) * mfl::IB * mfl::IB * sizeof(double) +
             2 * (size_t)n * n * sizeof(double);
    return MFLAB_OK;
}

extern "C" int mflab_lu64_prepare(mflab_handle *h, void *stream, int64_t n, const double *LU,
                                  int64_t ldl, const int64_t *ipiv, void *work) {
    MFLAB_RANGE("mflab_lu64_prepare");
    if (!h) return MFLAB_ERR_UNSUPPORTED;
    if (n < 0 || (n > 0 && (!LU || !ipiv || !work || ldl < n))) return MFLAB_ERR_ARG;
    if (n == 0) return MFLAB_OK;
    if (n > mfl::PIVOT_PERM_MAXN_LU64) return MFLAB_ERR_UNSUPPORTED;
    cudaStream_t s = (cudaStream_t)stream;
    int *perm = (int *)work;
    double *invL = (double *)((char *)work + mfl::perm_bytes(n));
    double *invU = invL + (size_t)mfl::nblocks(n) * mfl::IB * mfl::IB;
    const int smem = (mfl::IB * (mfl::IB + 1) + mfl::IB) * (int)sizeof(double);
    int rc = mfl::set_smem_once((const void *)mfl::lu64_inv_diag_kernel, smem,
                                mfl::g_inv_configured, "lu64 inverse attribute");
    if (rc) return rc;
    static std::atomic<unsigned long long> perm_configured{0};
    rc = mfl::set_smem_once((const void *)mfl::lu64_perm_kernel,
                            (int)(2 * mfl::PIVOT_PERM_MAXN_LU64 * sizeof(int)), perm_configured,
                            "lu64 perm attribute");
    if (rc) return rc;
    mfl::lu64_perm_kernel<<<1, 256, 2 * (size_t)n * sizeof(int), s>>>(n, ipiv, perm);
    mfl::lu64_inv_diag_kernel<<<dim3((unsigned)mfl::nblocks(n), 2), mfl::IB, smem, s>>>(
        n, LU, ldl, invL, invU);
    rc = mfl::record_cuda_error(cudaGetLastError(), "lu64 prepare");
    if (rc) return rc;
    // ML = L_{r,i} inv(DL_i) below block i, MU = U_{r,i} inv(DU_i) above it
    // (binary64 GEMMs of the library)
    double *ML = invU + (size_t)mfl::nblocks(n) * mfl::IB * mfl::IB, *MU = ML + (size_t)n * n;
    const size_t wsb = (size_t)32 << 20;
    rc = mflab_reserve_scratch(h, wsb);
    if (rc) return rc;
    for (int64_t i = 0; i < mfl::nblocks(n) && rc == MFLAB_OK; ++i) {
        const int64_t j0 = i * mfl::IB, jb = std::min<int64_t>(mfl::IB, n - j0);
        const double *iL = invL + i * mfl::IB * mfl::IB, *iU = invU + i * mfl::IB * mfl::IB;
        if (j0 + jb < n)
            rc = mfl::dgemm_lt(n - j0 - jb, jb, jb, LU + j0 * ldl + j0 + jb, ldl, iL, mfl::IB,
                               ML + j0 * n + j0 + jb, n, 1.0, 0.0, h->scratch, wsb, s);
        if (rc == MFLAB_OK && j0 > 0)
            rc = mfl::dgemm_lt(j0, jb, jb, LU + j0 * ldl, ldl, iU, mfl::IB, MU + j0 * n, n, 1.0,
                               0.0, h->scratch, wsb, s);
    }
    return rc;
}

extern "C" int mflab_lu64_solve(mflab_handle *h, void *stream, int64_t n, int64_t nrhs,
                                const double *LU, int64_t ldl, const void *work, double *B,
                                int64_t ldb) {
    MFLAB_RANGE("mflab_lu64_solve");
    if (!h) return MFLAB_ERR_UNSUPPORTED;
    if (n < 0 || nrhs < 0 || (n > 0 && (!LU || !work || !B || ldl < n || ldb < n)))
        return MFLAB_ERR_ARG;
    if (n == 0 || nrhs == 0) return MFLAB_OK;
    cudaStream_t s = (cudaStream_t)stream;
    const int *perm = (const int *)work;
    const double *invL = (const double *)((const char *)work + mfl::perm_bytes(n));
    const double *invU = invL + (size_t)mfl::nblocks(n) * mfl::IB * mfl::IB;
    const double *ML = invU + (size_t)mfl::nblocks(n) * mfl::IB * mfl::IB, *MU = ML + (size_t)n * n;
    if (const size_t bytes = mfl::solve_bytes(n, nrhs)) {
        int rc = mflab_reserve_scratch(h, bytes);
        if (rc) return rc;
        unsigned long long *pub = (unsigned long long *)h->scratch;
        int *abort_word = (int *)((char *)h->scratch + bytes - 256), *err = h->dev_flags + 1;
        cudaError_t e = cudaMemsetAsync(pub, 0xff, bytes - 256, s);
        if (e == cudaSuccess) e = cudaMemsetAsync(abort_word, 0, sizeof(int), s);
        if (e != cudaSuccess) return mfl::record_cuda_error(e, "lu64 solve rows");
        long long spin = h->tc_limit > 0 ? h->tc_limit : mfl::LS_SPIN;
        void *args[] = {&n,   &nrhs, &perm, &invL, &invU,       &ML,  &MU,
                        &B,   &ldb,  &pub,  &abort_word, &err, &spin};
        e = cudaLaunchCooperativeKernel((const void *)mfl::lu64_solve_kernel,
                                        dim3((unsigned)((n + mfl::MS_ROWS - 1) / mfl::MS_ROWS)),
                                        dim3(mfl::MS_NT), args, sizeof(mfl::LsShared), s);
        return mfl::record_cuda_error(e, "lu64 solve");
    }
    // W: the permuted right-hand sides, then the forward solution
    int rc = mflab_reserve_scratch(h, (size_t)n * nrhs * sizeof(double));
    if (rc) return rc;
    double *W = (double *)h->scratch;
    const int64_t tot = n * nrhs;
    mfl::lu64_gather_kernel<<<(unsigned)((tot + 255) / 256), 256, 0, s>>>(n, nrhs, B, ldb, perm, W,
                                                                         n);
    rc = mfl::record_cuda_error(cudaGetLastError(), "lu64 gather");
    if (rc) return rc;
    const int64_t nb = mfl::nblocks(n);
    // forward: L y = P b, y written into B, W updated below each block
    for (int64_t i = 0; i < nb && rc == MFLAB_OK; ++i) {
        const int64_t j0 = i * mfl::IB;
        const int jb = (int)std::min<int64_t>(mfl::IB, n - j0);
        rc = mfl::mstep_launch(s, nrhs, j0, jb, ML, n, invL + i * mfl::IB * mfl::IB, W, n, B, ldb,
                               j0 + jb, n);
    }
    // backward: U x = y, x written into W, B (holding y) updated above each block
    for (int64_t i = nb - 1; i >= 0 && rc == MFLAB_OK; --i) {
        const int64_t j0 = i * mfl::IB;
        const int jb = (int)std::min<int64_t>(mfl::IB, n - j0);
        rc = mfl::mstep_launch(s, nrhs, j0, jb, MU, n, invU + i * mfl::IB * mfl::IB, B, ldb, W, n,
                               0, j0);
    }
    if (rc) return rc;
    rc = mfl::record_cuda_error(cudaGetLastError(), "lu64 solve");
    if (rc) return rc;
    // the solution (in W) back into B
    cudaError_t e = cudaMemcpy2DAsync(B, ldb * sizeof(double), W, n * sizeof(double),
                                      n * sizeof(double), nrhs, cudaMemcpyDeviceToDevice, s);
    return mfl::record_cuda_error(e, "lu64 solve copy");
}
