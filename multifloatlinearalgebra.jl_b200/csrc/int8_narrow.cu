// Residue products of the modular route with few columns (at most 32) on the
// tcgen05 tensor cores: the residuals of a refinement with a few right-hand
// sides.
//
// Such a product is bound by reading the residue planes of A once.  The 256 x
// 256 tiles of int8_tc.cu pad its columns to 256 and read A's first digit once
// per level.  Here a task is 128 rows of one modulus over all digits of A, and
// all levels are formed while a K step is in shared memory (A digit d times B
// digit e adds to level d + e; levels Q and above are dropped):
//   digit 0 of A   one MMA of N = Q NC columns against [B digit 0 | B digit 1]
//                  writes level 0 and adds to level 1 side by side;
//   digit 1 of A   one MMA of N = NC columns against B digit 0 adds to level 1.
// Persistent CTAs of six warps: a TMA producer, an MMA issuer (owner of two
// alternating accumulators of Q NC columns), four epilogue warps that store
// the sums modulo crt_modulus(z) as bytes.  8 stages of 128 A rows (16 KiB) and
// up to 64 B rows keep 128 KiB of A in flight per SM.  Bounded waits and the
// abort path are those of int8_tc.cu.  x4, m = k = 4096, n = 16, 32 moduli (1.07
// GB of A residues): 226 us, against 396 us for the two level launches on
// 256 x 256 tiles.
#include "int8_tc_common.cuh"

#include <algorithm>

namespace mfl {

constexpr int TN_BM = 128, TN_STAGES = 8, TN_THREADS = 192;
constexpr uint32_t TN_A_BYTES = TN_BM * TC_BK;  // 16 KiB

template <int Q, int NC>
struct TnShape {
    static constexpr uint32_t b_bytes = NC * TC_BK;                      // one digit's box
    static constexpr uint32_t stage = TN_A_BYTES + Q * b_bytes;
    static constexpr uint32_t smem = TN_STAGES * stage + 1024 + 256;
    static constexpr uint32_t cols = Q * NC;                             // one accumulator
    static constexpr uint32_t alloc = 2 * cols < 32 ? 32 : 2 * cols;     // a power of two
};

template <int Q, int NC>
__global__ void __launch_bounds__(TN_THREADS, 1)
    int8_narrow_kernel(const __grid_constant__ CUtensorMap tmA,
                       const __grid_constant__ CUtensorMap tmB, int kp, uint8_t *R, int64_t ldr,
                       int64_t plane, int mp, int nz, int *err, TcDebug dbg) {
    using S = TnShape<Q, NC>;
    extern __shared__ uint8_t smem_raw[];
    uint8_t *smem = (uint8_t *)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
    uint64_t *full = (uint64_t *)(smem + TN_STAGES * S::stage);
    uint64_t *empty = full + TN_STAGES;
    uint64_t *tfull = empty + TN_STAGES;  // [2] accumulator ready (MMA -> epilogue)
    uint64_t *tempty = tfull + 2;         // [2] accumulator drained (epilogue -> MMA)
    uint64_t *drain = tempty + 2;
    uint64_t *never = drain + 1;          // injected timeouts wait here (no arrivals)
    uint32_t *tmem_slot = (uint32_t *)(never + 1);
    int *abort_flag = (int *)(tmem_slot + 1);

    const int warp = threadIdx.x / 32, lane = threadIdx.x % 32;
    const int kd = kp / TC_BK, ksteps = Q * kd;  // K steps per digit, per task
    const int tiles_m = mp / TN_BM, total = tiles_m * nz;
    const long long lim = dbg.limit;

    if (threadIdx.x == 0) {
        for (int s = 0; s < TN_STAGES; ++s) {
            mbar_init(&full[s], 1);
            mbar_init(&empty[s], 1);
        }
        for (int a = 0; a < 2; ++a) {
            mbar_init(&tfull[a], 1);
            mbar_init(&tempty[a], 4);  // one arrival per epilogue warp
        }
        mbar_init(drain, 1);
        mbar_init(never, 1);
        *abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                         smem_u32(tmem_slot)),
                     "r"(S::alloc)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem = *tmem_slot;
    auto give_up = [&](int code) {
        if (!*(volatile int *)abort_flag) atomicExch(err, code);
        atomicExch(abort_flag, 1);
    };

    if (warp == 0) {
        if (lane == 0) {
            // ---------------- TMA producer; digit d of B sits at (Q-1-d) kp
            int ks = 0;
            bool ok = true;
            for (int tile = blockIdx.x; tile < total && ok && !*(volatile int *)abort_flag;
                 tile += gridDim.x) {
                const int z = tile / tiles_m, am0 = z * mp + (tile % tiles_m) * TN_BM;
                for (int kb = 0; kb < ksteps; ++kb, ++ks) {
                    const int s = ks % TN_STAGES;
                    if (ks >= TN_STAGES &&
                        !mbar_wait(&empty[s], ((ks / TN_STAGES) - 1) & 1, lim, abort_flag)) {
                        give_up(TC_ERR_PRODUCER);
                        ok = false;
                        break;
                    }
                    uint8_t *sa = smem + s * S::stage, *sb = sa + TN_A_BYTES;
                    const int kk = (kb % kd) * TC_BK;
                    const bool both = Q == 2 && kb < kd;
                    mbar_expect_tx(&full[s], TN_A_BYTES + (both ? 2 : 1) * S::b_bytes);
                    tma_load_2d(sa, &tmA, kb * TC_BK, am0, &full[s]);
                    tma_load_2d(sb, &tmB, (Q - 1) * kp + kk, z * NC, &full[s]);
                    if (both) tma_load_2d(sb + S::b_bytes, &tmB, kk, z * NC, &full[s]);
                }
            }
            // the copies of the last issued steps land before the CTA exits
            for (int i = ks - TN_STAGES > 0 ? ks - TN_STAGES : 0; i < ks; ++i)
                if (!mbar_wait(&full[i % TN_STAGES], (i / TN_STAGES) & 1, TC_DRAIN_LIMIT))
                    atomicExch(err, TC_ERR_DRAIN);
        }
    } else if (warp == 1) {
        if (lane == 0) {
            // ---------------- MMA issuer
            constexpr uint32_t id_all = idesc_i8(TN_BM, Q * NC), id_one = idesc_i8(TN_BM, NC);
            if (dbg.inject && !mbar_wait(never, 0, TC_INJECT_POLLS)) give_up(TC_ERR_MMA);
            int ks = 0, it = 0;
            bool ok = true;
            for (int tile = blockIdx.x; tile < total && ok && !*(volatile int *)abort_flag;
                 tile += gridDim.x, ++it) {
                const int a = it & 1;
                if (it > 1 && !mbar_wait(&tempty[a], ((it >> 1) - 1) & 1, lim, abort_flag)) {
                    give_up(TC_ERR_MMA);
                    break;
                }
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                const uint32_t acc = tmem + a * S::cols;
                for (int kb = 0; kb < ksteps; ++kb, ++ks) {
                    const int s = ks % TN_STAGES;
                    if (!mbar_wait(&full[s], (ks / TN_STAGES) & 1, lim, abort_flag)) {
                        give_up(TC_ERR_MMA);
                        ok = false;
                        break;
                    }
                    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                    const uint32_t sa = smem_u32(smem + s * S::stage), sb = sa + TN_A_BYTES;
#pragma unroll
                    for (int kk = 0; kk < TC_BK / 32; ++kk) {
                        const uint64_t ad = smem_desc_sw128(sa + kk * 32);
                        const uint64_t bd = smem_desc_sw128(sb + kk * 32);
                        if (kb < kd) mma_i8(acc, ad, bd, id_all, (kb > 0 || kk > 0) ? 1u : 0u);
                        else mma_i8(acc + NC, ad, bd, id_one, 1u);
                    }
                    mma_commit(&empty[s]);
                }
                mma_commit(&tfull[a]);  // also on abort: the epilogue then sees the flag
            }
            // every MMA issued by this thread has completed once `drain` flips
            mma_commit(drain);
            if (!mbar_wait(drain, 0, TC_DRAIN_LIMIT)) atomicExch(err, TC_ERR_DRAIN);
        }
    } else {
        // ---------------- epilogue: TMEM -> residue bytes of every level
        const int q = warp & 3;  // TMEM lane quarter of this warp
        int it = 0;
        for (int tile = blockIdx.x; tile < total; tile += gridDim.x, ++it) {
            const int a = it & 1;
            if (!mbar_wait(&tfull[a], (it >> 1) & 1, lim, abort_flag)) {
                give_up(TC_ERR_EPILOGUE);
                break;
            }
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            if (*(volatile int *)abort_flag) break;
            const int z = tile / tiles_m, row = (tile % tiles_m) * TN_BM + q * 32 + lane;
            const int pz = crt_modulus(z);
            const double pzinv = 1.0 / (double)pz;
#pragma unroll 1
            for (int c0 = 0; c0 < Q * NC; c0 += 16) {
                uint32_t v[16];
                tmem_ld16(tmem + ((uint32_t)(q * 32) << 16) + (uint32_t)(a * S::cols + c0), v);
                uint8_t *Rl = R + ((int64_t)(c0 / NC) * nz + z) * plane;
                tc_store16<1>(Rl, ldr, row, c0 % NC, v, pz, pzinv);
            }
            asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
            __syncwarp();
            if (lane == 0) mbar_arrive(&tempty[a]);
        }
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (warp == 1) {
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem),
                     "r"(S::alloc)
                     : "memory");
    }
}

template <int Q, int NC>
static int launch_narrow(int64_t mp, int64_t kp, const int8_t *A8, const int8_t *B8, uint8_t *R,
                         int64_t ldr, size_t plane, int nz, int *err, cudaStream_t s,
                         const TcOpts &o) {
    using S = TnShape<Q, NC>;
    CUtensorMap ta, tb;
    int rc = tc_make_map(&ta, A8, mp * nz, Q * kp, Q * kp, TN_BM);
    if (!rc) rc = tc_make_map(&tb, B8, (int64_t)NC * nz, Q * kp, Q * kp, NC);
    if (rc) return rc;
    auto kern = int8_narrow_kernel<Q, NC>;
    static std::atomic<unsigned long long> configured{0};
    rc = set_smem_once((const void *)kern, (int)S::smem, configured, "int8 narrow attribute");
    if (rc) return rc;
    int dev = 0, sms = 0;
    cudaGetDevice(&dev);
    if (cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || sms <= 0)
        sms = 148;
    TcDebug dbg;
    dbg.limit = o.limit > 0 ? o.limit : TC_ROLE_LIMIT;
    dbg.inject = o.inject;
    const int64_t tiles = mp / TN_BM * nz;
    kern<<<(unsigned)std::min<int64_t>(tiles, sms), TN_THREADS, S::smem, s>>>(
        ta, tb, (int)kp, R, ldr, (int64_t)plane, (int)mp, nz, err, dbg);
    return record_cuda_error(cudaGetLastError(), "int8 narrow");
}

// Residue bytes R[L][z][col][row] (levels plane * nz apart, problems `plane`
// apart, columns ldr apart) of nz stacked problems: A8 holds mp rows of Q kp
// bytes per problem (digit 0 first), B8 nc = 16 or 32 rows (digit Q-1 first).
// mp and kp are multiples of 128.
int int8_gemm_narrow(int Q, int nc, int64_t mp, int64_t kp, const int8_t *A8, const int8_t *B8,
                     uint8_t *R, int64_t ldr, size_t plane, int nz, int *err, cudaStream_t s,
                     const TcOpts &o) {
    if (mp <= 0 || mp % TN_BM || kp <= 0 || kp % TC_BK || nz < 1 || nz > CRT_TABLE_SIZE || ldr < mp)
        return MFLAB_ERR_ARG;
    if (mp * nz > 0x7fffffff || Q * kp > 0x7fffffff) return MFLAB_ERR_UNSUPPORTED;
    if (Q == 1 && nc == 16) return launch_narrow<1, 16>(mp, kp, A8, B8, R, ldr, plane, nz, err, s, o);
    if (Q == 1 && nc == 32) return launch_narrow<1, 32>(mp, kp, A8, B8, R, ldr, plane, nz, err, s, o);
    if (Q == 2 && nc == 16) return launch_narrow<2, 16>(mp, kp, A8, B8, R, ldr, plane, nz, err, s, o);
    if (Q == 2 && nc == 32) return launch_narrow<2, 32>(mp, kp, A8, B8, R, ldr, plane, nz, err, s, o);
    return MFLAB_ERR_UNSUPPORTED;
}

}  // namespace mfl
