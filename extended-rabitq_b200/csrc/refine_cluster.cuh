// The refinement with a window per cluster: a window of blocks ends with the
// cluster it lies in, candidates are listed in any order, and every pool is
// merged in shared memory (refine.cuh has windows across clusters and pools in
// registers; arguments, results and statistics are the same).
//
// Where it is the faster of the two (refine_by_cluster in erq_capi.cu): it needs
// 64 registers and 12 to 26 KB a block, so 8 blocks of 4 warps share an SM where
// refine.cuh's row ring allows 6, and its windows have one barrier and one chain
// of dependent loads less.  That decides where a window is all there is to a
// cluster - a few probes of clusters of a few blocks, small rows - and where the
// replay by one warp bounds the kernel (pools above kSmallPool).  10,000 queries,
// here / across clusters: 64 dims, 9 bits, nprobe 1: k = 1 98 / 160 us, k = 100 207 /
// 285; nprobe 16, k = 1000 14.8 / 19.4 ms; 1536 dims, nprobe 16, k = 1000 14.7 / 21.1;
// Zipf clusters of 256 dims, k = 257, nprobe 2 4.74 / 6.29 ms.
#pragma once

#include "refine.cuh"

namespace erq {

constexpr int kClusterWarps = 4;
constexpr int kClusterPerSm = 8;         // blocks of the 4-warp form an SM holds
constexpr int kClusterWindow = 16;       // blocks whose candidates are refined together
constexpr int kClusterFirstWindow = 8;   // the same in the query's first probed cluster
// Wide form for small batches (a query per SM): more warps, longer windows.
constexpr int kClusterWideWarps = 32;
constexpr int kClusterWideWindow = 128;

// Shared memory of one block: unit_q[D] | per window lane: lb, ipq, onorm,
// ex_dist, id, list | pool_d[kpad] | pool_id[kpad] | misc | window blocks
__host__ __device__ constexpr size_t refine_cluster_smem_bytes(int D, int kpad, int wb) {
    return (size_t)D * 4 + (size_t)wb * 32 * (5 * 4 + 2) + (size_t)kpad * 8 + 64 + 128 + (size_t)wb * 4;
}

// One block of WARPS warps per query (4, or 32 in the wide form).  Per window
// of up to WB blocks of the current cluster (16, or 128; 8 in a query's first
// cluster in the 4-warp form): the warps compute the lower bounds of the
// window's blocks, dealt round robin, and list the lanes below the threshold
// as it stands at the window's start (a superset of the exact candidates,
// because the threshold only falls); the quads compute the listed candidates'
// exact distances (8 quads per warp; warps without a candidate skip the
// round); warp 0 then replays the window in the reference's order -
// each block's mask against the threshold at that block's start, the block's
// candidates merged into the pool as inserting them in lane order would.
template <int EX, int WARPS, int WB>
__global__ void __launch_bounds__(WARPS * 32, WARPS == kClusterWarps ? kClusterPerSm : 1)
    refine_cluster_kernel(RefineArgs a) {
    constexpr int kThreads = WARPS * 32, kLanes = WB * 32;
    static_assert(WB % WARPS == 0 && kLanes <= 65536, "window lanes are listed as u16");
    extern __shared__ __align__(16) uint8_t smem_raw[];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int q = a.order ? (int)a.order[blockIdx.x] : (int)blockIdx.x;
    const int D = a.D, k = a.k;
    const int kpad = (k + 31) & ~31;
    float* uq = reinterpret_cast<float*>(smem_raw);
    float* w_lb = uq + D;
    float* w_ipq = w_lb + kLanes;
    float* w_on = w_ipq + kLanes;
    float* w_ed = w_on + kLanes;
    uint32_t* w_id = reinterpret_cast<uint32_t*>(w_ed + kLanes);
    uint16_t* w_list = reinterpret_cast<uint16_t*>(w_id + kLanes);
    float* pool_d = reinterpret_cast<float*>(w_list + kLanes);
    uint32_t* pool_id = reinterpret_cast<uint32_t*>(pool_d + kpad);
    int* misc = reinterpret_cast<int*>(pool_id + kpad);  // [0] list count [1] pool size
    float* s_distk = reinterpret_cast<float*>(misc + 2);
    float* cs = reinterpret_cast<float*>(misc + 16);  // 32 floats of merge scratch
    uint32_t* w_blk = reinterpret_cast<uint32_t*>(cs + 32);  // the window's blocks
    const int fac_rescale = 1 << EX;
    const float one_over_sqrtD = recip_via_double(__fsqrt_rn((float)D));
    const float* qv = a.qrot + (size_t)q * D;

    for (int i = tid; i < kpad; i += blockDim.x) {
        pool_d[i] = 0.f;
        pool_id[i] = 0u;
    }
    if (tid == 0) {
        *s_distk = FLT_MAX;
        misc[1] = 0;  // pool size as seen by all warps
    }
    int size = 0;         // pool state, maintained by warp 0
    float distk = FLT_MAX;
    uint32_t st_cand = 0, st_refined = 0, st_windows = 0, st_blocks = 0;  // with a.stats
    __syncthreads();

    const int np_q = a.q_nprobe ? a.q_nprobe[q] : a.nprobe;
    for (int p = 0; p < np_q; ++p) {
        const size_t qp = (size_t)q * a.nprobe + p;
        const uint32_t cid = a.probe_cid[qp];
        const float sqy = a.probe_sqy[qp];
        const float y = __fsqrt_rn(sqy);
        const float delta = a.qp_delta[qp];
        const float sumq = a.qp_sumq[qp];
        // lower-bound constants (inc/index/fastscan/FastScan.hpp:297-303)
        const LbConsts lbk = lb_consts(sumq, y, one_over_sqrtD);
        const double ex_sub = __dmul_rn((double)fac_rescale - 0.5, (double)sumq);
        const uint32_t n = a.c_size[cid];
        const uint32_t fb = a.c_first_block[cid];
        const uint32_t first_vec = a.c_first_vec[cid];
        const int32_t* S = a.S + a.s_off[qp];
        const float* bmin = a.bmin ? a.bmin + a.s_off[qp] / 32 : nullptr;
        const uint32_t nblocks = (n + 31) >> 5;
        bool uq_ready = false;
        // The first cluster's threshold falls fast (the pool fills, then
        // tightens), so a long window there lists many lanes that its replay
        // drops; later clusters' thresholds barely move and long windows save
        // barriers.
        const int wcap = (WARPS == kClusterWarps && p == 0) ? kClusterFirstWindow : WB;
        for (uint32_t wb = 0; wb < nblocks;) {
            const float d0 = *s_distk;
            const int filled = misc[1];
            // While the pool is filling every lane is a candidate: take just
            // enough blocks to fill it, so few lanes are refined in vain.
            const int want = filled < k ? min(wcap, max(1, (k - filled + 31) / 32))
                                        : wcap;
            __syncthreads();
            // warp 0 picks the window: the next `want` blocks from wb whose
            // smallest lower bound is below the threshold (a block above it
            // has no candidate now or later: the threshold only falls)
            if (warp == 0) {
                int got = 0;
                uint32_t pos = wb, next = nblocks;
                while (got < want && pos < nblocks) {
                    const uint32_t bb = pos + lane;
                    const bool take = bb < nblocks && (!bmin || bmin[bb] < d0);
                    const uint32_t m = __ballot_sync(0xffffffffu, take);
                    const int rank = __popc(m & ((1u << lane) - 1u));
                    if (take && got + rank < want) w_blk[got + rank] = bb;
                    const int nm = __popc(m);
                    if (got + nm >= want) {
                        // the want-th taken block ends the window
                        const uint32_t endm = __ballot_sync(0xffffffffu, take && rank == want - got - 1);
                        next = pos + (uint32_t)(__ffs(endm) - 1) + 1;
                        got = want;
                        break;
                    }
                    got += nm;
                    pos += 32;
                }
                if (lane == 0) {
                    misc[0] = 0;
                    misc[5] = got;
                    misc[6] = (int)next;
                }
            }
            __syncthreads();
            const int nbw = misc[5];
            const uint32_t wnext = (uint32_t)misc[6];
            // lower bounds and the candidate superset, 4 blocks per warp
#pragma unroll
            for (int i = 0; i < WB / (kThreads / 32); ++i) {
                const int b = i * (kThreads / 32) + warp;  // round robin: short windows use every warp
                if (b < nbw) {  // uniform per warp
                    const uint32_t blk = w_blk[b];
                    const float ipq = __fmul_rn(__int2float_rn(S[32 * blk + lane]), delta);
                    const float on = a.onorm[(size_t)(fb + blk) * 32 + lane];
                    const float t = lower_bound(ipq, on, lbk);
                    const bool valid = 32 * blk + lane < n;
                    // padding lanes never pass (NaN compares false)
                    w_lb[32 * b + lane] = valid ? t : __int_as_float(0x7fc00000);
                    w_ipq[32 * b + lane] = ipq;
                    w_on[32 * b + lane] = on;
                    const uint32_t m = __ballot_sync(0xffffffffu, valid && t < d0);
                    int base = 0;
                    if (lane == 0 && m) base = atomicAdd(&misc[0], __popc(m));
                    base = __shfl_sync(0xffffffffu, base, 0);
                    if ((m >> lane) & 1u) {
                        w_list[base + __popc(m & ((1u << lane) - 1u))] = (uint16_t)(32 * b + lane);
                        // start the candidate's EX-code row on its way to L2
                        const size_t pos = (size_t)first_vec + 32 * blk + lane;
                        asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(
                                         a.excode + pos * a.ex_row),
                                     "r"((uint32_t)a.ex_row)
                                     : "memory");
                    }
                }
            }
            __syncthreads();
            const int cnt = misc[0];
            if (a.stats) {
                st_refined += cnt;
                st_windows += 1;
                st_blocks += nbw;
            }
            if (cnt == 0) {  // uniform: nothing in this window can pass
                wb = wnext;
                continue;
            }
            if (!uq_ready) {
                const float* cv = a.centroids + (size_t)cid * D;
                if (y > kNormEps) {
                    const float fac = recip_via_double(y);
                    for (int i = tid; i < D; i += blockDim.x) uq[i] = __fmul_rn(__fsub_rn(qv[i], cv[i]), fac);
                } else {
                    const float fill = recip_via_double(__fsqrt_rn((float)D));
                    for (int i = tid; i < D; i += blockDim.x) uq[i] = fill;
                }
                uq_ready = true;
                __syncthreads();
            }
            // refine the listed candidates: quad g (lanes 4g..4g+3) takes two
            // per round while more than one per quad remain, else one; within a warp
            // that has work, quads past the end repeat the list's first so
            // the warp stays converged
            {
                const int g = tid >> 2, r = tid & 3;
                const float4* uq4 = reinterpret_cast<const float4*>(uq);
                for (int base = 0; base < cnt;) {
                    const int two = cnt - base > kThreads / 4;
                    const int step = two ? kThreads / 2 : kThreads / 4;
                    // per warp: skip when none of its slots holds a candidate,
                    // one candidate per quad when its second slots are empty
                    if (base + 8 * warp >= cnt) {
                        base += step;
                        continue;
                    }
                    const int wtwo = two && base + kThreads / 4 + 8 * warp < cnt;
                    const int i0 = base + g, i1 = base + kThreads / 4 + g;
                    const int s0 = w_list[i0 < cnt ? i0 : 0];
                    const int s1 = w_list[wtwo && i1 < cnt ? i1 : 0];
                    const size_t pos0 = (size_t)first_vec + 32 * w_blk[s0 >> 5] + (s0 & 31);
                    const size_t pos1 = (size_t)first_vec + 32 * w_blk[s1 >> 5] + (s1 & 31);
                    const uint4* row0 = reinterpret_cast<const uint4*>(a.excode + pos0 * a.ex_row);
                    const uint4* row1 = reinterpret_cast<const uint4*>(a.excode + pos1 * a.ex_row);
                    // lane 0 of the quad finishes the first, lane 1 the second
                    const int i = r == 0 ? i0 : i1;
                    const bool fin = r < 2 && (r == 0 || wtwo) && i < cnt;
                    const int slot = r == 0 ? s0 : s1;
                    const size_t pos = r == 0 ? pos0 : pos1;
                    float xipn = 0.f;
                    uint32_t vid = 0u;
                    if (fin) {
                        xipn = __ldg(a.xipnorm + pos);
                        vid = __ldg(a.ids + pos);
                    }
                    float ip[2];
                    if (wtwo)
                        ex_ip_quad<ex_storage_bits(EX), 2>(uq4, row0, row1, r, D / 16, ip);
                    else
                        ex_ip_quad<ex_storage_bits(EX), 1>(uq4, row0, row0, r, D / 16, ip);
                    if (fin) {
                        // inc/index/HASearcher.hpp:225-232
                        const float on = w_on[slot];
                        const float sqr_x = __fmul_rn(on, on);
                        const float t = __fadd_rn(__fmul_rn((float)fac_rescale, w_ipq[slot]), r == 0 ? ip[0] : ip[1]);
                        const double br = __dsub_rn((double)t, ex_sub);
                        const float xy = __fmul_rn(xipn, y);
                        const float f = __fadd_rn(sqr_x, sqy);
                        // as refine_kernel
                        w_ed[slot] = fminf(__double2float_rn(__dsub_rn((double)f, __dmul_rn((double)xy, br))), INFINITY);
                        w_id[slot] = vid;
                    }
                    base += step;
                }
            }
            __syncthreads();
            if (warp == 0) {
                for (int b = 0; b < nbw; ++b) {
                    // candidates of the block against the threshold at its
                    // start; those above a full pool's k-th cannot enter
                    const float ed = w_ed[32 * b + lane];
                    const bool below = w_lb[32 * b + lane] < distk;
                    if (a.stats) st_cand += __popc(__ballot_sync(0xffffffffu, below));
                    const bool enter = below && (size < k || !(ed > distk));
                    if (__ballot_sync(0xffffffffu, enter))
                        pool_merge_block(pool_d, pool_id, size, k, distk, enter, ed,
                                         w_id[32 * b + lane], cs, lane, p > 0);
                }
                if (lane == 0) {
                    *s_distk = distk;
                    misc[1] = size;
                }
            }
            __syncthreads();
            wb = wnext;
        }
    }
    if (warp == 0) {
        if (a.stats && lane == 0) {
            atomicAdd(a.stats + 0, (unsigned long long)st_cand);
            atomicAdd(a.stats + 1, (unsigned long long)st_refined);
            atomicAdd(a.stats + 2, (unsigned long long)st_windows);
            atomicAdd(a.stats + 3, (unsigned long long)st_blocks);
        }
        uint32_t* oid = a.out_ids + (size_t)q * k;
        for (int i = lane; i < k; i += 32) {
            oid[i] = i < size ? pool_id[i] : 0u;
            if (a.out_dists)
                a.out_dists[(size_t)q * k + i] = i < size ? pool_d[i] : __int_as_float(0x7f800000);
        }
    }
}

}  // namespace erq
