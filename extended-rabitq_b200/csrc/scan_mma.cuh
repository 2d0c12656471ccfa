// FastScan on the 5th-generation tensor cores (tcgen05 kind::i8, sm_100a).
//
// S_v = <x_b(v), qq> is an exact integer dot product of a 0/1 vector and a
// 14-bit signed one (scan.cuh), so the sums of one cluster's vectors against
// the queries that probe it are a small matrix product over 8-bit integers:
// qq = 128 * hi + lo with hi in [-64, 63] and lo in [0, 127], the 1-bit codes
// as bytes 0 or 128, int32 accumulators; S = acc_hi + acc_lo / 128, exactly.
//
// scan_quantize_kernel writes hi and lo of every (query, probe) pair once, in
// the order of the cluster-sorted pairs, so the rows of one cluster's queries
// are consecutive.  scan_mma_kernel is persistent: work items - one cluster,
// up to kMmaQueries of the queries that probe it, a chunk of up to CB of its
// 32-vector blocks - come from a counter (scan_batch.cuh's work list), and its
// warps run as a pipeline over them:
//   warp 9      claims items, writes their records (two in flight) and loads
//               the queries' rows by TMA (B operand, K-major, 128-byte swizzle);
//   warps 0-3   expand codes, a block (32 vectors, a lane each) per warp: 16
//               bytes of a lane hold 16 groups of 6 dims (layout.cuh); a shift
//               and a mask turn each 4-byte word into six registers of four
//               bytes 0 / 128, and tcgen05.st puts 96 of them per chunk into
//               the lane's row of a ring of A operands in tensor memory;
//   warp 8      one thread issues three tcgen05.mma (M 128 = four blocks,
//               N = 2 * queries, K 32) per chunk;
//   warps 4-7   read a finished accumulator back (tcgen05.ld, a lane per
//               vector), write S and each block's smallest lower bound.
// B's bytes follow the order in which the expansion leaves the dims: within
// 24 dims, dim 6b + j is byte 4j + b.
//
// Barriers: full/empty per ring slot, tfull/tempty per accumulator (two),
// full/empty per record, one per K block of B, bfree when an item's products
// are done.  Every wait is bounded (wait_limit polls); a role whose wait runs out
// sets the block's flag and leaves, the others run out of theirs (a product warp
// that gives up never frees B, whose copies may still be landing), copies and
// products in flight are waited for, and bit kScanTimeoutBit of the status word
// is set.
#pragma once

#include "common.cuh"
#include "gemm_tc.cuh"
#include "scan.cuh"
#include "scan_batch.cuh"

namespace erq {

constexpr int kMmaQueries = 32;      // queries per item: N = 64 accumulator columns
constexpr int kMmaThreads = 320;     // 4 expansion, 4 read-back, MMA, claim + TMA warps
constexpr int kMmaRing = 5;          // A operands (96 dims each) in tensor memory
constexpr int kMmaChunkCols = 24;    // 32-bit columns of one A operand
constexpr int kMmaAccCols = 64;      // columns of one accumulator (two of them)
constexpr int kMmaTmemCols = 256;
constexpr uint32_t kMmaBBlock = 2u * kMmaQueries * 128u;  // bytes of one K block of B
constexpr int kMmaPrefetch = 8;      // code loads in flight per expansion warp
constexpr int kMmaMaxKBlocks = 17;   // of 128 dims (D <= 2048)
constexpr int kMmaBars = (2 * kMmaRing + 10 + kMmaMaxKBlocks + 1) & ~1;  // even: what follows is 16-byte aligned
static_assert(2 * kMmaAccCols + kMmaRing * kMmaChunkCols <= kMmaTmemCols, "tensor memory");

__host__ __device__ constexpr int mma_k_blocks(int D) { return (hex_chunks(D) * 96 + 127) / 128; }
static_assert(mma_k_blocks(kMaxD) <= kMmaMaxKBlocks, "K blocks");
// Bytes of one quantized row (hi or lo) in global memory.
__host__ __device__ constexpr uint32_t mma_row_bytes(int D) { return (uint32_t)mma_k_blocks(D) * 128u; }
__host__ __device__ constexpr uint32_t mma_b_bytes(int D) {
    return (uint32_t)mma_k_blocks(D) * kMmaBBlock;
}

// An item as its claiming warp hands it to the other roles.
struct MmaItem {
    uint32_t end;                 // no more items
    uint32_t fblock, b0, b1;      // the cluster's first block; the chunk's blocks
    uint32_t csize, qn;           // vectors of the cluster, queries of the item
    uint32_t pad[2];
    uint64_t soff[kMmaQueries];   // offsets into S
    float4 k0[kMmaQueries / 2];   // of two queries: delta, delta, -c1, -c1
    float4 k1[kMmaQueries / 2];   // c2, c2, c3, c3
};

static_assert(alignof(MmaItem) == 16 && (kMmaBars * 8 + 16) % 16 == 0, "items after the barriers");

// [pad to 1024][B][bars][flag, tensor-memory address][two items]
__host__ __device__ constexpr size_t mma_smem_bytes(int D) {
    const size_t need = 1024 + (size_t)mma_b_bytes(D) + kMmaBars * 8 + 16 + 2 * sizeof(MmaItem);
    // at least a third of an SM's shared memory, so that no more than two
    // blocks (512 tensor-memory columns) share an SM
    return need < 80 * 1024 ? 80 * 1024 : need;
}

// Instruction descriptor: S32 accumulator, unsigned 8-bit A, signed 8-bit B.
__host__ __device__ constexpr uint32_t umma_idesc_u8s8(int M, int N) {
    return (2u << 4) | (1u << 10) | ((uint32_t)(N >> 3) << 17) | ((uint32_t)(M >> 4) << 24);
}

__device__ __forceinline__ void tmem_st8(uint32_t addr, const uint32_t* r) {
    asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8};" ::"r"(addr),
                 "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7])
                 : "memory");
}
__device__ __forceinline__ void tmem_ld8(uint32_t addr, uint32_t (&r)[8]) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]),
                   "=r"(r[7])
                 : "r"(addr));
}
// D[128][N] (+)= A * B^T of 32 dims: A in tensor memory (u8), B by its shared
// descriptor (s8); `add` 0 starts the accumulator.
__device__ __forceinline__ void mma_u8s8(uint32_t d, uint32_t a, uint64_t b, uint32_t idesc, uint32_t add) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::i8 [%0], [%1], %2, %3, p;\n\t}" ::"r"(d),
        "r"(a), "l"(b), "r"(idesc), "r"(add)
        : "memory");
}
// One lane of the (converged) warp.
__device__ __forceinline__ bool elect_one() {
    uint32_t p;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "elect.sync _|p, 0xffffffff;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(p));
    return p != 0;
}
__device__ __forceinline__ void tc_commit(uint32_t bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar)
                 : "memory");
}
// Smallest value over the warp (NaN lanes are ignored), in every lane.
__device__ __forceinline__ float redux_min(float v) {
    float r;
    asm volatile("redux.sync.min.f32 %0, %1, 0xffffffff;" : "=f"(r) : "f"(v));
    return r;
}

// ------------------------------------------------------------ quantization
struct QuantizeArgs {
    const float* qrot;
    const float* centroids;
    const uint32_t* probe_cid;
    const float* probe_sqy;
    const uint32_t* order_pairs;  // pairs sorted by cluster
    const uint32_t* bucket_end;   // [K + 1]
    uint8_t* rows;                // [2][cap][mma_row_bytes(D)]: hi, then lo, by sorted position
    float* qp_delta;              // [nq][nprobe]
    float* qp_sumq;
    uint64_t cap;                 // rows per half (the batch's pairs)
    int K, D, nprobe;
};
constexpr int kQuantizeWarps = 8;
__host__ __device__ constexpr int quantize_floats(int D) { return (D + 23) / 24 * 24; }
__host__ __device__ constexpr size_t quantize_smem_bytes(int D) {
    return (size_t)kQuantizeWarps * quantize_floats(D) * 4;
}

// unit_q, delta, sumq of a (query, cluster) pair exactly as hex_prepare
// (scan.cuh), and its quantized dims as two byte rows, a warp per pair.
// round-half-away(fl(u / delta)): with inv = fl(1 / delta), t = fl(u * inv) is
// within 3.01 * 2^-24 |t| of fl(u / delta); unless that reaches over a half
// (or something is not finite), rounding t gives the same integer, otherwise
// the division is made.  Adding 1.5 * 2^23 + 8192 rounds t and leaves
// v + 8192 = 128 * (hi + 64) + lo in the low bits.
__global__ void __launch_bounds__(kQuantizeWarps * 32) scan_quantize_kernel(QuantizeArgs a) {
    extern __shared__ __align__(16) float quant_smem[];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const uint64_t i = (uint64_t)blockIdx.x * kQuantizeWarps + warp;
    if (i >= a.bucket_end[a.K - 1]) return;  // whole warp; nothing below waits across warps
    const int D = a.D;
    float* u = quant_smem + warp * quantize_floats(D);
    const uint32_t pair = a.order_pairs[i];
    const uint32_t q = pair / (uint32_t)a.nprobe;
    const float4* qv = reinterpret_cast<const float4*>(a.qrot + (size_t)q * D);
    const float4* cv = reinterpret_cast<const float4*>(a.centroids + (size_t)a.probe_cid[pair] * D);
    const float y = __fsqrt_rn(a.probe_sqy[pair]);
    const bool normal = y > kNormEps;
    const float fac = normal ? recip_via_double(y) : 0.f;
    const float fill = recip_via_double(__fsqrt_rn((float)D));
    float vmax = 0.f;
#pragma unroll 4
    for (int g = lane; g < D / 4; g += 32) {
        float4 v = make_float4(fill, fill, fill, fill);
        if (normal) {
            const float4 x = __ldg(qv + g), c = __ldg(cv + g);
            v.x = __fmul_rn(__fsub_rn(x.x, c.x), fac);
            v.y = __fmul_rn(__fsub_rn(x.y, c.y), fac);
            v.z = __fmul_rn(__fsub_rn(x.z, c.z), fac);
            v.w = __fmul_rn(__fsub_rn(x.w, c.w), fac);
        }
        reinterpret_cast<float4*>(u)[g] = v;
        vmax = fmaxf(vmax, fmaxf(fmaxf(fabsf(v.x), fabsf(v.y)), fmaxf(fabsf(v.z), fabsf(v.w))));
    }
    for (int d = D + lane; d < quantize_floats(D); d += 32) u[d] = 0.f;
    vmax = __uint_as_float(__reduce_max_sync(0xffffffffu, __float_as_uint(vmax)));
    __syncwarp();
    const float delta = __fdiv_rn(vmax, 8191.f);
    const float inv = __frcp_rn(delta);
    uint32_t* hi_row = reinterpret_cast<uint32_t*>(a.rows + i * mma_row_bytes(D));
    uint32_t* lo_row = reinterpret_cast<uint32_t*>(a.rows + (a.cap + i) * mma_row_bytes(D));
    constexpr float kRound = 12582912.f + 8192.f;
    for (int w = lane; w < quantize_floats(D) / 4; w += 32) {
        const int g = w / 6, d = 24 * g + (w - 6 * g);  // byte b of the word: dim d + 6b
        uint32_t x[4];
        bool sure = true;
        float uu[4];
#pragma unroll
        for (int b = 0; b < 4; ++b) {
            uu[b] = u[d + 6 * b];
            const float t = __fmul_rn(uu[b], inv);
            const float m = __fadd_rn(t, kRound);
            const float frac = fabsf(__fsub_rn(t, __fsub_rn(m, kRound)));  // exact, at most 1/2
            sure = sure && __fmaf_rn(fabsf(t), 2.5e-7f, frac) < 0.5f;
            x[b] = __float_as_uint(m);
        }
        if (!sure) {
#pragma unroll
            for (int b = 0; b < 4; ++b)
                x[b] = (uint32_t)((int)(int16_t)quantize_round(__fdiv_rn(uu[b], delta)) + 8192);
        }
        // two 16-bit v + 8192 per word; bits 0-6 are lo, bits 7-13 hi + 64
        const uint32_t p01 = __byte_perm(x[0], x[1], 0x5410), p23 = __byte_perm(x[2], x[3], 0x5410);
        const uint32_t h = __byte_perm(p01 << 1, p23 << 1, 0x7531);
        hi_row[w] = ((h | 0x80808080u) - 0x40404040u) ^ 0x80808080u;  // h - 64 in each byte
        lo_row[w] = __byte_perm(p01, p23, 0x6420) & 0x7F7F7F7Fu;
    }
    // sumq: 16 ordered chains and the reduce tree
    float acc = 0.f;
    if (lane < 16) {
#pragma unroll 8
        for (int d = lane; d < D; d += 16) acc = __fadd_rn(acc, u[d]);
    }
    const float s = tree16_sum(acc);
    if (lane == 0) {
        a.qp_delta[pair] = delta;
        a.qp_sumq[pair] = normal ? s : __fmul_rn((float)D, fill);
    }
}

// ---------------------------------------------------------------- products
// First query of group g of a run of m queries split evenly into
// ceil(m / kMmaQueries) groups.
__device__ __forceinline__ uint32_t mma_group_start(uint32_t m, uint32_t g) {
    const uint32_t G = (m + kMmaQueries - 1) / kMmaQueries;
    return (uint32_t)(((uint64_t)m * g) / G);
}

// LIMITED: waits give up after `polls` instead of kScanWaitLimit, which as an
// argument costs the kernel 3 % (erq_debug_set_scan_wait_limit).
template <bool LIMITED>
__global__ void __launch_bounds__(kMmaThreads, 2)
scan_mma_kernel(const __grid_constant__ CUtensorMap rows, uint32_t cap, ScanBatchArgs a, uint32_t polls) {
    const uint32_t wait_limit = LIMITED ? polls : kScanWaitLimit;
    extern __shared__ uint8_t smem_raw[];
    const int D = a.D;
    const int tid = threadIdx.x, lane = tid & 31;
    const int warp = __shfl_sync(0xffffffffu, tid >> 5, 0);  // known uniform to the compiler
    const uint32_t raw = (uint32_t)__cvta_generic_to_shared(smem_raw);
    const uint32_t bop = (raw + 1023u) & ~1023u;  // B operand
    uint64_t* bars_p = reinterpret_cast<uint64_t*>(smem_raw + (bop - raw) + mma_b_bytes(D));
    volatile uint32_t* flag = reinterpret_cast<volatile uint32_t*>(bars_p + kMmaBars);
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars_p + kMmaBars) + 1;
    MmaItem* items = reinterpret_cast<MmaItem*>(reinterpret_cast<uint8_t*>(bars_p + kMmaBars) + 16);
    const uint32_t bars = (uint32_t)__cvta_generic_to_shared(bars_p);
    const uint32_t full0 = bars, empty0 = full0 + 8 * kMmaRing;
    const uint32_t tfull0 = empty0 + 8 * kMmaRing, tempty0 = tfull0 + 16;
    const uint32_t rfull0 = tempty0 + 16, rempty0 = rfull0 + 16;
    const uint32_t bfree = rempty0 + 16, drain = bfree + 8, bfull0 = drain + 8;
    const uint32_t nc = hex_chunks(D), nkb = mma_k_blocks(D);

    if (tid == 0) {
        for (int s = 0; s < kMmaRing; ++s) {
            mbar_init(full0 + 8 * s, 4);  // one arrival per expansion warp
            mbar_init(empty0 + 8 * s, 1);
        }
        for (int b = 0; b < 2; ++b) {
            mbar_init(tfull0 + 8 * b, 1);
            mbar_init(tempty0 + 8 * b, 4);  // one arrival per read-back warp
            mbar_init(rfull0 + 8 * b, 1);
            mbar_init(rempty0 + 8 * b, 9);  // expansion, read-back and MMA warps
        }
        mbar_init(bfree, 1);
        mbar_init(drain, 1);
        for (uint32_t s = 0; s < nkb; ++s) mbar_init(bfull0 + 8 * s, 1);
        *flag = 0u;
        mbar_init_fence();
    }
    if (warp == 8) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                         (uint32_t)__cvta_generic_to_shared(tmem_slot)),
                     "r"((uint32_t)kMmaTmemCols)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = *tmem_slot;
    const uint32_t ring = tmem + 2 * kMmaAccCols;
    // the consumers' wait for item n (its record slot is n & 1); uniform
    const auto next_item = [&](uint32_t n) -> const MmaItem* {
        if (!__all_sync(0xffffffffu, mbar_wait(rfull0 + 8 * (n & 1u), (n >> 1) & 1u, wait_limit))) {
            *flag = 1u;
            return nullptr;
        }
        const MmaItem* m = items + (n & 1u);
        return m->end ? nullptr : m;
    };

    if (warp < 4) {
        const uint32_t bb = code_block_bytes(D);
        const uint32_t lane_base = (uint32_t)(32 * warp) << 16;
        uint32_t slot = 0, phase = 1;  // the first round of the ring waits for nothing
        for (uint32_t n = 0;; ++n) {
            const MmaItem* m = next_item(n);
            if (!m) break;
            const uint32_t b1 = m->b1;
            uint32_t ld_b = m->b0 + warp, ld_c = 0;  // next load: block, chunk
            const uint32_t todo = ((b1 - m->b0 + 3) >> 2) * nc;
            const uint8_t* src = a.codes + (size_t)(m->fblock + ld_b) * bb + lane * 16;
            __syncwarp();
            if (lane == 0) mbar_arrive(rempty0 + 8 * (n & 1u));
            // blocks past the chunk's end load nothing (their rows are not read back)
            auto load_next = [&]() -> uint4 {
                uint4 v = make_uint4(0u, 0u, 0u, 0u);
                if (ld_b < b1) v = __ldg(reinterpret_cast<const uint4*>(src));
                src += 512;
                if (++ld_c == nc) {
                    ld_c = 0;
                    ld_b += 4;
                    src += (size_t)3 * bb;
                }
                return v;
            };
            uint4 buf[kMmaPrefetch];
#pragma unroll
            for (int i = 0; i < kMmaPrefetch; ++i) buf[i] = load_next();
            bool ok = true;
            for (uint32_t g0 = 0; g0 < todo && ok; g0 += kMmaPrefetch) {
#pragma unroll
                for (int u = 0; u < kMmaPrefetch; ++u) {
                    if (g0 + u < todo && ok) {
                        const uint4 w = buf[u];
                        buf[u] = load_next();
                        ok = __all_sync(0xffffffffu, mbar_wait(empty0 + 8 * slot, phase, wait_limit));
                        if (ok) {
                            tc_fence_after();
                            uint32_t e[kMmaChunkCols];
                            const uint32_t ww[4] = {w.x, w.y, w.z, w.w};
#pragma unroll
                            for (int i = 0; i < 4; ++i)
#pragma unroll
                                for (int j = 0; j < 6; ++j)  // bit j + 1 of each byte to bit 7
                                    e[6 * i + j] = (ww[i] * (1u << (6 - j))) & 0x80808080u;
                            const uint32_t at = ring + lane_base + slot * kMmaChunkCols;
                            tmem_st8(at, e);
                            tmem_st8(at + 8, e + 8);
                            tmem_st8(at + 16, e + 16);
                            asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
                            tc_fence_before();
                            __syncwarp();
                            if (lane == 0) mbar_arrive(full0 + 8 * slot);
                            if (++slot == (uint32_t)kMmaRing) {
                                slot = 0;
                                phase ^= 1u;
                            }
                        }
                    }
                }
            }
            if (!ok) {
                *flag = 1u;
                break;
            }
        }
    } else if (warp < 8) {
        const int w = warp - 4;
        uint32_t acc = 0, phase = 0;
        bool ok = true;
        for (uint32_t n = 0; ok; ++n) {
            const MmaItem* m = next_item(n);
            if (!m) break;
            const uint32_t b1 = m->b1, csize = m->csize, fblock = m->fblock;
            const int qn = (int)m->qn, qp = (qn + 7) & ~7;
            for (uint32_t bt = m->b0; bt < b1; bt += 4) {
                const uint32_t b = bt + w;
                const bool mine = b < b1;
                const float on = mine ? __ldg(a.onorm + (size_t)(fblock + b) * 32 + lane) : 0.f;
                // lanes past the cluster's end get an infinite lower bound
                const float on2 = 32 * b + lane < csize ? __fmul_rn(on, on) : INFINITY;
                ok = __all_sync(0xffffffffu, mbar_wait(tfull0 + 8 * acc, phase, wait_limit));
                if (!ok) {
                    *flag = 1u;
                    break;
                }
                tc_fence_after();
                if (mine) {
                    const uint32_t at = tmem + acc * kMmaAccCols + ((uint32_t)(32 * w) << 16);
                    const float2 on_2 = make_float2(on, on), on2_2 = make_float2(on2, on2);
                    int32_t* sb = a.S + (32 * b + lane);
                    float bm = 0.f;
                    for (int j0 = 0; j0 < qp; j0 += 8) {
                        uint32_t hi[8], lo[8];
                        tmem_ld8(at + j0, hi);
                        tmem_ld8(at + qp + j0, lo);
                        asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
                        for (int i = 0; i < 8; i += 2) {
                            const int j = j0 + i;
                            if (j < qn) {
                                const int s0 = (int)hi[i] + ((int)lo[i] >> 7);
                                const int s1 = (int)hi[i + 1] + ((int)lo[i + 1] >> 7);
                                sb[m->soff[j]] = s0;
                                if (j + 1 < qn) sb[m->soff[j + 1]] = s1;
                                // lower_bound (common.cuh) of two queries
                                const float4 k0 = m->k0[j >> 1], k1 = m->k1[j >> 1];
                                float2 t = fmul2(make_float2(__int2float_rn(s0), __int2float_rn(s1)),
                                                 make_float2(k0.x, k0.y));
                                t = fadd2(t, make_float2(k0.z, k0.w));
                                t = fmul2(fmul2(t, make_float2(k1.x, k1.y)), on_2);
                                t = fadd2(fadd2(t, make_float2(k1.z, k1.w)), on2_2);
                                const float m0 = redux_min(t.x), m1 = redux_min(t.y);
                                if (lane == j) bm = m0;
                                if (lane == j + 1) bm = m1;
                            }
                        }
                    }
                    if (lane < qn && a.bmin) a.bmin[m->soff[lane] / 32 + b] = bm;
                }
                tc_fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive(tempty0 + 8 * acc);
                acc ^= 1u;
                phase ^= acc ^ 1u;
            }
            __syncwarp();
            if (lane == 0) mbar_arrive(rempty0 + 8 * (n & 1u));
        }
    } else if (warp == 8) {
        // the whole warp keeps to one control flow (so that operands stay in
        // uniform registers), one lane issues
        const bool leader = elect_one();
        uint32_t slot = 0, phase = 0, acc = 0, aphase = 1;
        bool ok = true;
        for (uint32_t n = 0; ok; ++n) {
            const MmaItem* m = next_item(n);
            if (!m) break;
            const uint32_t tiles = __shfl_sync(0xffffffffu, (m->b1 - m->b0 + 3) >> 2, 0);
            const uint32_t qp = __shfl_sync(0xffffffffu, (m->qn + 7u) & ~7u, 0);
            if (leader) mbar_arrive(rempty0 + 8 * (n & 1u));
            const uint32_t idesc = umma_idesc_u8s8(128, (int)(2 * qp));
            const uint64_t bdesc = umma_desc_sw128(bop);
            for (uint32_t t = 0; t < tiles; ++t) {
                ok = __all_sync(0xffffffffu, mbar_wait(tempty0 + 8 * acc, aphase, wait_limit));
                if (!ok) break;
                tc_fence_after();
                const uint32_t d = tmem + acc * kMmaAccCols;
                uint32_t step = 0;  // of 32 dims
                for (uint32_t k = 0; k < nc; ++k) {
                    if (t == 0) {  // the K blocks of B this chunk is the first to read
                        const uint32_t f0 = (96 * k + 127) >> 7, f1 = (96 * k + 95) >> 7;
                        for (uint32_t f = f0; f <= f1 && ok; ++f)
                            ok = __all_sync(0xffffffffu, mbar_wait(bfull0 + 8 * f, n & 1u, wait_limit));
                    }
                    ok = ok && __all_sync(0xffffffffu, mbar_wait(full0 + 8 * slot, phase, wait_limit));
                    if (!ok) break;
                    tc_fence_after();
                    if (leader) {
                        const uint32_t at = ring + slot * kMmaChunkCols;
#pragma unroll
                        for (uint32_t i = 0; i < 3; ++i) {
                            const uint32_t st = step + i;
                            mma_u8s8(d, at + 8 * i, bdesc + (st >> 2) * (kMmaBBlock >> 4) + (st & 3u) * 2, idesc,
                                     st);
                        }
                        tc_commit(empty0 + 8 * slot);
                    }
                    step += 3;
                    if (++slot == (uint32_t)kMmaRing) {
                        slot = 0;
                        phase ^= 1u;
                    }
                }
                if (!ok) break;
                if (leader) tc_commit(tfull0 + 8 * acc);
                acc ^= 1u;
                aphase ^= acc ^ 1u;
            }
            if (!ok) break;
            if (leader) tc_commit(bfree);
        }
        if (leader && !ok) *flag = 1u;
        // every product of this block has finished once this arrives
        if (leader) {
            tc_commit(drain);
            mbar_wait(drain, 0, kTcWaitLimit);
        }
        __syncwarp();
    } else {
        const uint32_t total = a.item_off[a.K];
        const float one_over_sqrtD = recip_via_double(__fsqrt_rn((float)D));
        uint32_t n = 0;  // items handed out
        bool ok = true;
        for (;;) {
            uint32_t it = 0;
            if (lane == 0) it = atomicAdd(a.item_counter, 1u);
            it = __shfl_sync(0xffffffffu, it, 0);
            uint32_t row = 0, qn = 0, b0 = 0, b1 = 0, fblock = 0, csize = 0;
            if (it < total) {
                const uint32_t j = item_cluster(a.item_off, a.K, it, lane);
                const uint32_t c = a.c_order[j];
                const uint32_t start = c ? a.bucket_end[c - 1] : 0u;
                const uint32_t m_c = a.bucket_end[c] - start;
                const uint32_t nb = a.c_nblocks[c];
                const uint32_t nch = max(1u, (nb + a.CB - 1) / a.CB);
                const uint32_t local = it - a.item_off[j], g = local / nch;
                const uint32_t g0 = mma_group_start(m_c, g);
                qn = mma_group_start(m_c, g + 1) - g0;
                row = start + g0;
                b0 = (local - g * nch) * a.CB;
                b1 = min(nb, b0 + (uint32_t)a.CB);
                fblock = a.c_first_block[c];
                csize = a.c_size[c];
                if (b1 <= b0) continue;  // an empty cluster: no sums
            }
            MmaItem* m = items + (n & 1u);
            if (n >= 2) {
                ok = __all_sync(0xffffffffu,
                                mbar_wait(rempty0 + 8 * (n & 1u), ((n >> 1) - 1u) & 1u, wait_limit));
                if (!ok) break;
            }
            if (lane == 0) {
                m->end = it >= total ? 1u : 0u;
                m->fblock = fblock;
                m->b0 = b0;
                m->b1 = b1;
                m->csize = csize;
                m->qn = qn;
            }
            if ((uint32_t)lane < qn) {
                const uint32_t pair = a.order_pairs[row + lane];
                const LbConsts k = lb_consts(a.qp_sumq[pair], __fsqrt_rn(a.probe_sqy[pair]), one_over_sqrtD);
                m->soff[lane] = a.s_off[pair];
                float* k0 = reinterpret_cast<float*>(m->k0 + (lane >> 1)) + (lane & 1);
                float* k1 = reinterpret_cast<float*>(m->k1 + (lane >> 1)) + (lane & 1);
                k0[0] = a.qp_delta[pair];
                k0[2] = -k.c1;
                k1[0] = k.c2;
                k1[2] = k.c3;
            }
            __syncwarp();
            if (lane == 0) mbar_arrive(rfull0 + 8 * (n & 1u));
            if (it >= total) break;
            // the queries' rows, once the item before has been multiplied
            if (lane == 0) {
                if (n >= 1) ok = mbar_wait(bfree, (n - 1u) & 1u, wait_limit);
                if (ok) {
                    const uint32_t qp = (qn + 7u) & ~7u;
                    for (uint32_t f = 0; f < nkb; ++f) {
                        uint32_t dst = bop + f * kMmaBBlock;  // hi rows, then lo rows
                        mbar_expect_tx(bfull0 + 8 * f, 2 * qp * 128u);
                        for (uint32_t h = 0; h < 2; ++h)
                            for (uint32_t r = 0; r < qp; r += 8, dst += 1024)
                                tma_load_2d(dst, &rows, (int)(f * 128u), (int)(h * cap + row + r),
                                            bfull0 + 8 * f);
                    }
                }
            }
            ok = __shfl_sync(0xffffffffu, ok ? 1 : 0, 0) != 0;
            if (!ok) break;
            ++n;
        }
        if (lane == 0) {
            if (!ok) *flag = 1u;
            // the last item's copies land before the block exits, whoever left early
            if (n >= 1)
                for (uint32_t f = 0; f < nkb; ++f) mbar_wait(bfull0 + 8 * f, (n - 1u) & 1u, kScanDrainLimit);
        }
        __syncwarp();
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 8) {
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem),
                     "r"((uint32_t)kMmaTmemCols)
                     : "memory");
    }
    if (tid == 0 && *flag && a.status) atomicOr(a.status, kScanTimeoutBit);
}

}  // namespace erq
