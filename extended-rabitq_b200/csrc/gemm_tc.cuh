// C = A * B^T on the 5th-generation tensor cores (tcgen05, sm_100a).
//
// A [M][Kd] and B [N][Kd] are BF16, K-major (the split-BF16 operands of
// gemm.cuh: [hi | hi | lo] x [hi | lo | hi] gives hi.hi + hi.lo + lo.hi), the
// accumulators are FP32 in tensor memory.  The kernel is persistent: one CTA
// per SM walks the 128 x 256 output tiles (row-major tile order, so the CTAs
// running at the same time share A tiles in L2), and the shared ring runs on
// across tiles:
//   warp 0   (one thread)  TMA: 64-wide K slices of A (128 rows) and B (256
//            rows), 128-byte swizzled, into a kTcStages-deep shared ring;
//   warp 1   (one thread)  allocates 2 x 256 TMEM columns (two accumulators),
//            issues tcgen05.mma.cta_group::1.kind::f16 (M 128, N 256, K 16)
//            four times per slice into the accumulator of the tile, frees
//            each slot with tcgen05.commit, and commits the accumulator;
//   warps 2-9              read an accumulator back (tcgen05.ld 32x32b, each
//            warp the 32 TMEM lanes of its quadrant in half of the columns,
//            so that two warps hide each other's latencies), release it, and apply
//            the epilogue of gemm.cuh (plain, distance ranking, bias + ReLU)
//            while the MMAs of the next tile fill the other accumulator.
// Barriers: full/empty per ring slot, tfull/tempty per accumulator, and a
// drain barrier the MMA thread commits to last.  Every mbarrier wait is
// bounded; a wait that runs out sets bit 0 of *status, and the CTA stops
// issuing work, lets its TMA copies land and its MMAs finish, frees its TMEM
// and exits.  Every TMA load reads this GPU's own memory into this CTA's own
// shared memory.
#pragma once

#include <cuda.h>

#include "gemm.cuh"
#include "mbarrier.cuh"

namespace erq {

constexpr int kTcBM = 128, kTcBN = 256, kTcBK = 64, kTcStages = 4;
constexpr int kTcThreads = 320;
constexpr int kTcEpiWarps = kTcThreads / 32 - 2;  // two per TMEM lane quadrant, half of the columns each
constexpr uint32_t kTcABytes = kTcBM * kTcBK * 2;   // 16 KB
constexpr uint32_t kTcBBytes = kTcBN * kTcBK * 2;   // 32 KB
constexpr uint32_t kTcStageBytes = kTcABytes + kTcBBytes;
constexpr uint32_t kTcWaitLimit = 1u << 26;  // polls per pipeline wait (the default)


__device__ __forceinline__ void tma_load_2d(uint32_t dst, const CUtensorMap* map, int x, int y,
                                            uint32_t bar) {
    asm volatile(
        "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];"
        ::"r"(dst), "l"(reinterpret_cast<uint64_t>(map)), "r"(x), "r"(y), "r"(bar)
        : "memory");
}

// Shared-memory matrix descriptor: K-major, 128-byte swizzle, rows of 128
// bytes, 8-row groups 1024 bytes apart (leading offset unused: 1).
__device__ __forceinline__ uint64_t umma_desc_sw128(uint32_t saddr) {
    return (uint64_t)((saddr >> 4) & 0x3FFFu) | (1ull << 16) | (64ull << 32) | (1ull << 46) |
           (2ull << 61);
}

// Instruction descriptor: F32 accumulator, BF16 A and B, both K-major.
__host__ __device__ constexpr uint32_t umma_idesc_bf16(int M, int N) {
    return (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(N >> 3) << 17) | ((uint32_t)(M >> 4) << 24);
}

__device__ __forceinline__ void tc_fence_before() {
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
}
__device__ __forceinline__ void tc_fence_after() {
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
}

constexpr int kTpAccumCols = 256;  // columns per accumulator (two of them)

// A warp's 32 x 32 block of the accumulator on its way to memory, the 16-byte
// piece p of row r at p ^ (r & 7): 8 rows' pieces are in different banks.
constexpr size_t kTcSlabBytes = 32 * 32 * sizeof(float);
__device__ __forceinline__ float* tc_slab_at(float* slab, int r, int p) {
    return slab + 32 * r + 4 * (p ^ (r & 7));
}

// 1024 bytes of alignment slack + the ring + barriers and the TMEM address +
// the epilogue warps' blocks
__host__ __device__ constexpr size_t gemm_tc_smem_bytes() {
    return 1024 + (size_t)kTcStages * kTcStageBytes + 256 + kTcEpiWarps * kTcSlabBytes;
}

// Rows row0 .. row0+31 and columns col0 .. col0+31 of the output, lane l
// holding row row0 + l.  The block is turned around in shared memory, so that 8
// lanes store 128 contiguous bytes of a row and the norms are read once per
// block: stored as held, each instruction wrote 16 bytes of 32 rows.  With four
// warps as held, four turned around, eight turned around: 10,000 x 4096 x 4608
// 307, 290, 283 us; 10,000 x 1536 x 4608 135, 128.6, 125 us; 2000 x 4096 x 4608 83,
// 76, 72 us; 1000 x 1024 x 384 25, 21, 16.8 us.
__device__ __forceinline__ void gemm_epilogue_store(const uint32_t (&v)[32], float* slab,
                                                    float* __restrict__ Cout, int M, int N, int row0,
                                                    int col0, const GemmEpilogue& epi) {
    const int lane = threadIdx.x & 31;
#pragma unroll
    for (int j = 0; j < 32; j += 4)
        *reinterpret_cast<uint4*>(tc_slab_at(slab, lane, j / 4)) =
            make_uint4(v[j], v[j + 1], v[j + 2], v[j + 3]);
    __syncwarp();
    const int col = col0 + 4 * (lane & 7);
    float cn[4], bias[4];
#pragma unroll
    for (int e = 0; e < 4; ++e) {
        const int cc = min(col + e, N - 1);
        cn[e] = epi.row_norm ? epi.col_norm[cc] : 0.f;
        bias[e] = epi.bias ? epi.bias[cc] : 0.f;
    }
    const bool whole = col + 3 < N && (N & 3) == 0;
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        const int lr = 4 * i + (lane >> 3), row = row0 + lr;
        if (row >= M) continue;
        const float4 y = *reinterpret_cast<const float4*>(tc_slab_at(slab, lr, lane & 7));
        float x[4] = {y.x, y.y, y.z, y.w};
        const float rn = epi.row_norm ? epi.row_norm[row] : 0.f;
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            if (epi.row_norm) x[e] = rn + cn[e] - 2.f * x[e];
            if (epi.bias) x[e] += bias[e];
            if (epi.relu) x[e] = fmaxf(x[e], 0.f);
        }
        float* out = Cout + (size_t)row * N + col;
        if (whole) {
            *reinterpret_cast<float4*>(out) = make_float4(x[0], x[1], x[2], x[3]);
        } else {
#pragma unroll
            for (int e = 0; e < 4; ++e)
                if (col + e < N) out[e] = x[e];
        }
    }
    __syncwarp();
}

// The norms of columns col0 .. col0+31 (infinity past the last), asked for before
// the accumulator is read so that the two waits overlap.
__device__ __forceinline__ void load_col_norms(const float* __restrict__ col_norm, int N, int col0,
                                               float (&cn)[32]) {
    if (col0 + 31 < N) {
#pragma unroll
        for (int j = 0; j < 32; j += 4) {
            const float4 c = __ldg(reinterpret_cast<const float4*>(col_norm + col0 + j));
            cn[j] = c.x, cn[j + 1] = c.y, cn[j + 2] = c.z, cn[j + 3] = c.w;
        }
    } else {
#pragma unroll
        for (int j = 0; j < 32; ++j) cn[j] = col0 + j < N ? __ldg(col_norm + col0 + j) : INFINITY;
    }
}

// The smallest ranking value of columns col0 .. col0+31 and its column (the
// first of equal ones), on top of (best, at) of the columns before, for the row
// this lane holds.  The minimum of the 32 is a tree; its column is looked for
// only where some row's minimum fell.
__device__ __forceinline__ void gemm_epilogue_nearest(const uint32_t (&v)[32], const float (&cn)[32], int col0,
                                                      float rn, float& best, int& at) {
    float x[32], m[4];
#pragma unroll
    for (int j = 0; j < 32; j += 4) {
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            x[j + e] = rn + cn[j + e] - 2.f * __uint_as_float(v[j + e]);
            m[e] = j ? fminf(m[e], x[j + e]) : x[j + e];
        }
    }
    const float least = fminf(fminf(m[0], m[1]), fminf(m[2], m[3]));
    const bool less = least < best;
    if (!__any_sync(0xffffffffu, less)) return;
    int c = 0;
#pragma unroll
    for (int j = 31; j >= 0; --j) c = x[j] == least ? j : c;
    if (less) {
        best = least;
        at = col0 + c;
    }
}

// NEAREST: the epilogue keeps each row's smallest ranking value instead of
// storing the block (kmeans.cuh).  200,000 x 1024 x 128 dims: the 819 MB of
// rankings cost 680 us to write and 116 us to read for the minimum; this takes 148
// us (with the four warps and the serial minimum that were tried first, 252).
template <bool NEAREST>
__global__ void __launch_bounds__(kTcThreads, 1) gemm_tc_kernel(
    const __grid_constant__ CUtensorMap tma_a, const __grid_constant__ CUtensorMap tma_b,
    float* __restrict__ Cout, int M, int N, int Kd, GemmEpilogue epi, uint32_t* status,
    uint32_t wait_limit) {
    extern __shared__ uint8_t smem_raw[];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const uint32_t raw = (uint32_t)__cvta_generic_to_shared(smem_raw);
    const uint32_t ring = (raw + 1023u) & ~1023u;
    const uint32_t bars = ring + kTcStages * kTcStageBytes;
    const uint32_t full0 = bars, empty0 = bars + 8 * kTcStages;
    const uint32_t tfull0 = bars + 16 * kTcStages, tempty0 = tfull0 + 16, drain = tempty0 + 16;
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(smem_raw + (drain + 8 - raw));
    volatile uint32_t* flag = tmem_slot + 1;  // set when any wait of this CTA ran out
    const int tiles_n = (N + kTcBN - 1) / kTcBN;
    const int tiles = ((M + kTcBM - 1) / kTcBM) * tiles_n;
    const int nk = Kd / kTcBK;

    if (tid == 0) {
        for (int s = 0; s < kTcStages; ++s) {
            mbar_init(full0 + 8 * s, 1);
            mbar_init(empty0 + 8 * s, 1);
        }
        for (int b = 0; b < 2; ++b) {
            mbar_init(tfull0 + 8 * b, 1);
            mbar_init(tempty0 + 8 * b, kTcEpiWarps);  // one arrival per epilogue warp
        }
        mbar_init(drain, 1);
        *flag = 0u;
        mbar_init_fence();
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                         (uint32_t)__cvta_generic_to_shared(tmem_slot)),
                     "r"((uint32_t)(2 * kTpAccumCols))
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = *tmem_slot;

    uint32_t issued = 0;  // ring slices the TMA thread started
    if (warp == 0) {
        if (lane == 0) {
            for (int t = blockIdx.x; t < tiles && !*flag; t += gridDim.x) {
                const int m0 = (t / tiles_n) * kTcBM, n0 = (t % tiles_n) * kTcBN;
                for (int kt = 0; kt < nk; ++kt) {
                    const uint32_t s = issued % kTcStages, r = issued / kTcStages;
                    if (r > 0 && !mbar_wait(empty0 + 8 * s, (r - 1) & 1u, wait_limit)) {
                        *flag = 1u;
                        break;
                    }
                    if (*flag) break;
                    const uint32_t sa = ring + s * kTcStageBytes, sb = sa + kTcABytes;
                    mbar_expect_tx(full0 + 8 * s, kTcStageBytes);
                    tma_load_2d(sa, &tma_a, kt * kTcBK, m0, full0 + 8 * s);
                    tma_load_2d(sb, &tma_b, kt * kTcBK, n0, full0 + 8 * s);
                    ++issued;
                }
            }
        }
    } else if (warp == 1) {
        if (lane == 0) {
            const uint32_t idesc = umma_idesc_bf16(kTcBM, kTcBN);
            uint32_t g = 0;  // ring slices consumed
            int i = 0;       // tiles of this CTA
            for (int t = blockIdx.x; t < tiles && !*flag; t += gridDim.x, ++i) {
                const int b = i & 1;
                const uint32_t u = (uint32_t)(i >> 1);
                if (u > 0 && !mbar_wait(tempty0 + 8 * b, (u - 1) & 1u, wait_limit)) {
                    *flag = 1u;
                    break;
                }
                tc_fence_after();
                const uint32_t acc_tmem = tmem + (uint32_t)(b * kTpAccumCols);
                bool ok = true;
                for (int kt = 0; kt < nk; ++kt, ++g) {
                    const uint32_t s = g % kTcStages, r = g / kTcStages;
                    if (!mbar_wait(full0 + 8 * s, r & 1u, wait_limit) || *flag) {
                        *flag = 1u;
                        ok = false;
                        break;
                    }
                    tc_fence_after();
                    const uint32_t sa = ring + s * kTcStageBytes, sb = sa + kTcABytes;
#pragma unroll
                    for (int kk = 0; kk < kTcBK / 16; ++kk) {
                        const uint64_t ad = umma_desc_sw128(sa + 32 * kk);
                        const uint64_t bd = umma_desc_sw128(sb + 32 * kk);
                        const uint32_t acc = (kt | kk) ? 1u : 0u;
                        asm volatile(
                            "{\n\t.reg .pred p;\n\t"
                            "setp.ne.b32 p, %4, 0;\n\t"
                            "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}"
                            ::"r"(acc_tmem), "l"(ad), "l"(bd), "r"(idesc), "r"(acc)
                            : "memory");
                    }
                    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];"
                                 ::"r"(empty0 + 8 * s)
                                 : "memory");
                }
                if (!ok) break;
                // the accumulator is complete once every MMA above has finished
                asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];"
                             ::"r"(tfull0 + 8 * b)
                             : "memory");
            }
            // every MMA this thread issued has finished once this arrives
            asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];"
                         ::"r"(drain)
                         : "memory");
            mbar_wait(drain, 0, kTcWaitLimit);
        }
    } else {
        const int q = warp & 3;  // TMEM lane quadrant this warp may read
        const int cb = warp < 6 ? 0 : kTcBN / 2;  // its columns of the tile
        float* slab = reinterpret_cast<float*>(smem_raw + (bars + 256 - raw) + (warp - 2) * kTcSlabBytes);
        int i = 0;
        for (int t = blockIdx.x; t < tiles; t += gridDim.x, ++i) {
            const int b = i & 1;
            const uint32_t u = (uint32_t)(i >> 1);
            const int m0 = (t / tiles_n) * kTcBM, n0 = (t % tiles_n) * kTcBN;
            const int row = m0 + 32 * q + lane;
            const float rn = NEAREST && row < M ? epi.row_norm[row] : 0.f;
            if (!mbar_wait(tfull0 + 8 * b, u & 1u, wait_limit) || *flag) {
                *flag = 1u;
                break;
            }
            tc_fence_after();
            float best = INFINITY;
            int at = 0;
            for (int c0 = cb; c0 < cb + kTcBN / 2; c0 += 32) {
                float cn[32];
                if constexpr (NEAREST) load_col_norms(epi.col_norm, N, n0 + c0, cn);
                uint32_t v[32];
                const uint32_t taddr = tmem + ((uint32_t)(32 * q) << 16) + (uint32_t)(b * kTpAccumCols + c0);
                asm volatile(
                    "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,"
                    "%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%32];"
                    : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]),
                      "=r"(v[7]), "=r"(v[8]), "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]),
                      "=r"(v[13]), "=r"(v[14]), "=r"(v[15]), "=r"(v[16]), "=r"(v[17]), "=r"(v[18]),
                      "=r"(v[19]), "=r"(v[20]), "=r"(v[21]), "=r"(v[22]), "=r"(v[23]), "=r"(v[24]),
                      "=r"(v[25]), "=r"(v[26]), "=r"(v[27]), "=r"(v[28]), "=r"(v[29]), "=r"(v[30]),
                      "=r"(v[31])
                    : "r"(taddr));
                asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
                if (c0 + 32 >= cb + kTcBN / 2) {
                    // the last columns are in registers: the accumulator is free
                    tc_fence_before();
                    __syncwarp();
                    if (lane == 0) mbar_arrive(tempty0 + 8 * b);
                }
                if constexpr (NEAREST) gemm_epilogue_nearest(v, cn, n0 + c0, rn, best, at);
                else gemm_epilogue_store(v, slab, Cout, M, N, m0 + 32 * q, n0 + c0, epi);
            }
            if (NEAREST && row < M && best < INFINITY) {
                const uint32_t u = __float_as_uint(best + 0.f);  // -0 orders as 0
                const uint32_t key = u ^ ((u >> 31) ? 0xffffffffu : 0x80000000u);
                atomicMin(epi.nearest + row, ((unsigned long long)key << 32) | (uint32_t)at);
            }
        }
    }
    // A CTA that gave up still lets its TMA copies land before it exits (its
    // MMAs finished above: the MMA thread always waits for the drain commit).
    if (warp == 0 && lane == 0 && *flag) {
        for (uint32_t g = issued > (uint32_t)kTcStages ? issued - kTcStages : 0u; g < issued; ++g)
            mbar_wait(full0 + 8 * (g % kTcStages), (g / kTcStages) & 1u, kTcWaitLimit);
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 1) {
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem),
                     "r"((uint32_t)(2 * kTpAccumCols))
                     : "memory");
    }
    if (tid == 0 && *flag && status) atomicOr(status, 1u);
}

}  // namespace erq
