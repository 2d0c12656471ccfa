// Lower-bound test, EX-bit refinement and the per-query top-k pool.
//
// One block per query replays the reference's sequential scan order
// (inc/index/IVF.hpp:313-321, inc/index/HASearcher.hpp:82-112,187-236):
// clusters in probe order, blocks in storage order, candidates of a block in
// ascending lane order.  The block's candidate mask is taken against the
// top-k threshold as it stands when the block starts; every candidate is
// offered to the pool in order and the threshold is refreshed after each
// insertion.  The integer sums S come from the scan kernels; everything that
// depends on the threshold happens here, so the candidate sets and the
// returned ids and distances equal the reference's.
//
//   lower bound  accumulate_one_block_high_acc  inc/index/fastscan/FastScan.hpp:295-323
//   ex-IP        IP16_fxu8 / IP32_fxu4 / IP64_fxu{2,3,6,7}  inc/utils/space.hpp
//   distance     inc/index/HASearcher.hpp:225-232
//   pool         ResultPool::insert / distk    inc/index/Pool.hpp:15-31
#pragma once

#include <cfloat>

#include "common.cuh"
#include "layout.cuh"

namespace erq {

struct RefineArgs {
    const float* qrot;            // [nq][D]
    const float* centroids;       // [K][D]
    const uint32_t* probe_cid;    // [nq][nprobe]
    const float* probe_sqy;       // [nq][nprobe]
    const uint64_t* s_off;        // [nq][nprobe]
    const int32_t* S;
    const float* qp_delta;        // [nq][nprobe]
    const float* qp_sumq;         // [nq][nprobe]
    const float* onorm;           // [blocks*32]
    const uint8_t* excode;        // [N][ex_row] device layout (layout.cuh)
    uint64_t ex_row;              // bytes per EX-code row
    const float* xipnorm;         // [N]
    const uint32_t* ids;          // [N]
    const uint32_t* c_first_block; // [K]
    const uint32_t* c_first_vec;   // [K]
    const uint32_t* c_size;        // [K]
    uint32_t* out_ids;            // [nq][k]
    float* out_dists;             // [nq][k] or null
    const int* q_nprobe;          // optional [nq]: clusters probed by each query
    const uint32_t* order;        // optional: block i refines query order[i]
    const float* bmin;            // optional: smallest lower bound per scanned block, at
                                  // s_off/32 + block (blocks above the threshold are skipped)
    unsigned long long* stats;    // optional [4], added to once per query: the reference's
                                  // exact candidates (lower bound below the threshold at
                                  // their block's start), lanes refined (the windows'
                                  // supersets), windows, window blocks
    int nq, D, EX, nprobe, k;
};


// Codes of bytes (lo, lo+1) of w as floats.  SCALED: the byte v in bits 16-23
// of a float is exactly v * 2^-133 (subnormal below 128, and the exponent's
// lowest bit carries on the same spacing above): one instruction per code.
// Otherwise exact integers: 0x4B0000vv is 2^23 + v.
template <bool SCALED>
__device__ __forceinline__ float2 code_pair(uint32_t w, int lo) {
    if (SCALED)
        return make_float2(__int_as_float((int)__byte_perm(w, 0u, 0x4044u | ((uint32_t)lo << 8))),
                           __int_as_float((int)__byte_perm(w, 0u, 0x4044u | ((uint32_t)(lo + 1) << 8))));
    const float2 big = make_float2(__int_as_float((int)__byte_perm(w, 0x4B000000u, 0x7540u | (uint32_t)lo)),
                                   __int_as_float((int)__byte_perm(w, 0x4B000000u, 0x7540u | (uint32_t)(lo + 1))));
    return fsub2(big, make_float2(8388608.f, 8388608.f));
}

// Codes of step t (0 <= t < 32/SB) of a lane's uint4 as 4 bytes.
template <int SB>
__device__ __forceinline__ uint32_t step_word(const uint4& v, int t) {
    const uint32_t c[4] = {v.x, v.y, v.z, v.w};
    if (SB == 8) return c[t];
    if (SB == 4) return (c[t >> 1] >> (4 * (t & 1))) & 0x0F0F0F0Fu;
    return (c[t >> 2] >> (2 * (t & 3))) & 0x03030303u;
}

// One step of one candidate: accumulators 4r+0..4r+3 of the reference's 16
// (as two pairs) take fma(unit_q[16s + 4r + i], code, acc).
template <bool SCALED>
__device__ __forceinline__ void ip_step(float2 acc[2], const float4& u, uint32_t w) {
    acc[0] = ffma2(make_float2(u.x, u.y), code_pair<SCALED>(w, 0), acc[0]);
    acc[1] = ffma2(make_float2(u.z, u.w), code_pair<SCALED>(w, 2), acc[1]);
}

// The reduce tree over a quad's 16 accumulators: acc[l] + acc[l+8], then + 4,
// then (0 + 2) + (1 + 3); the sum in every lane of the quad.
__device__ __forceinline__ float ip_tree(const float2 acc[2]) {
    float t3[4], t6[4];
    const float a4[4] = {acc[0].x, acc[0].y, acc[1].x, acc[1].y};
#pragma unroll
    for (int i = 0; i < 4; ++i) t3[i] = __fadd_rn(__shfl_xor_sync(0xffffffffu, a4[i], 2), a4[i]);
#pragma unroll
    for (int i = 0; i < 4; ++i) t6[i] = __fadd_rn(__shfl_xor_sync(0xffffffffu, t3[i], 1), t3[i]);
    return __fadd_rn(__fadd_rn(t6[0], t6[2]), __fadd_rn(t6[1], t6[3]));
}

// <unit_q, ex code> of NC (1 or 2) candidates by the 4 lanes r = 0..3 of a
// quad, in the reference's order (IP*_fxu* in inc/utils/space.hpp): the 16
// accumulators acc[l] take the dims l, l+16, l+32, ... in turn; lane r holds
// acc[4r..4r+3].  Rows are in the lane-interleaved layout of layout.cuh;
// each lane streams its own uint4s one ahead (a loop unrolled by 3, then the
// last pass, which fetches nothing).  uq4 = unit_q as float4.  Returns the
// sums in every lane of the quad.
template <int SB, int NC>
__device__ __forceinline__ void ex_ip_quad(const float4* __restrict__ uq4, const uint4* __restrict__ row0,
                                           const uint4* __restrict__ row1, int r, int steps,
                                           float out[2]) {
    constexpr int SPU = 32 / SB;  // steps per uint4
    const int U = (steps + SPU - 1) / SPU;
    float2 acc[NC][2];
#pragma unroll
    for (int c = 0; c < NC; ++c) acc[c][0] = acc[c][1] = make_float2(0.f, 0.f);
    // running pointers: each pass advances them by a constant, so the loads
    // of a pass take immediate offsets
    const uint4* rp[NC];
    rp[0] = row0 + r;
    if (NC > 1) rp[NC - 1] = row1 + r;
    const float4* qp = uq4 + r;
    uint4 cur[NC];
#pragma unroll
    for (int c = 0; c < NC; ++c) cur[c] = __ldg(rp[c]);
    const int Uf = steps / SPU;      // uint4s whose steps are all real
    const int Upf = min(Uf, U - 1);  // passes that fetch the next uint4
    int u = 0;
#pragma unroll 3
    for (; u < Upf; ++u) {
        uint4 nn[NC];
#pragma unroll
        for (int c = 0; c < NC; ++c) {
            rp[c] += 4;
            nn[c] = __ldg(rp[c]);
        }
#pragma unroll
        for (int t = 0; t < SPU; ++t) {
            const float4 q = qp[4 * t];
#pragma unroll
            for (int c = 0; c < NC; ++c) ip_step<false>(acc[c], q, step_word<SB>(cur[c], t));
        }
        qp += 4 * SPU;
#pragma unroll
        for (int c = 0; c < NC; ++c) cur[c] = nn[c];
    }
    for (; u < Uf; ++u) {  // the last pass: nothing left to fetch
#pragma unroll
        for (int t = 0; t < SPU; ++t) {
            const float4 q = qp[4 * t];
#pragma unroll
            for (int c = 0; c < NC; ++c) ip_step<false>(acc[c], q, step_word<SB>(cur[c], t));
        }
        qp += 4 * SPU;
    }
    for (int t = 0; t < steps - Uf * SPU; ++t) {  // a partly filled last uint4
        const float4 q = qp[4 * t];
#pragma unroll
        for (int c = 0; c < NC; ++c) ip_step<false>(acc[c], q, step_word<SB>(cur[c], t));
    }
#pragma unroll
    for (int c = 0; c < NC; ++c) out[c] = ip_tree(acc[c]);
}

// The same for two candidates (or one) of a quad whose rows come through a
// ring of kRowRing stages of asynchronous 16-byte copies, every lane copying
// and reading its own words: with one register-fed row word in flight per lane
// a pass waited for L2 (about 700 cycles for 16 codes a lane).  U: uint4s per
// lane of a row; uq4 = unit_q * 2^127, zero past D up to U whole uint4s, so
// every sum is the plain one times 2^-6; ring: this lane's 16 bytes of stage 0,
// candidate 0 (stages 1024 bytes apart, candidates 512).
constexpr int kRowRing = 4;
__device__ __forceinline__ void row_copy(uint32_t dst, const uint4* src) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src) : "memory");
}
__device__ __forceinline__ void row_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int SB, int NC>
__device__ __forceinline__ void ex_ip_ring(const float4* __restrict__ uq4, const uint4* __restrict__ row0,
                                           const uint4* __restrict__ row1, int r, int U, uint32_t ring,
                                           float out[2]) {
    constexpr int SPU = 32 / SB;  // steps per uint4
    float2 acc[NC][2];
#pragma unroll
    for (int c = 0; c < NC; ++c) acc[c][0] = acc[c][1] = make_float2(0.f, 0.f);
    const uint4* rp[NC];
    rp[0] = row0 + r;
    if (NC > 1) rp[NC - 1] = row1 + r;
    const float4* qp = uq4 + r;
#pragma unroll
    for (int s = 0; s < kRowRing - 1; ++s) {
        if (s < U) {
#pragma unroll
            for (int c = 0; c < NC; ++c) row_copy(ring + s * 1024 + c * 512, rp[c] + 4 * s);
        }
        row_commit();
    }
    const auto next_words = [&](int u, uint4 (&cur)[NC]) {
        asm volatile("cp.async.wait_group %0;" ::"n"(kRowRing - 2) : "memory");
#pragma unroll
        for (int c = 0; c < NC; ++c) cur[c] = lds128(ring + (u % kRowRing) * 1024 + c * 512);
        if (u + kRowRing - 1 < U) {
#pragma unroll
            for (int c = 0; c < NC; ++c)
                row_copy(ring + ((u + kRowRing - 1) % kRowRing) * 1024 + c * 512, rp[c] + 4 * (u + kRowRing - 1));
        }
        row_commit();
    };
#pragma unroll 4
    for (int u = 0; u < U; ++u) {
        uint4 cur[NC];
        next_words(u, cur);
#pragma unroll
        for (int t = 0; t < SPU; ++t) {
            const float4 q = qp[4 * t];
#pragma unroll
            for (int c = 0; c < NC; ++c) ip_step<true>(acc[c], q, step_word<SB>(cur[c], t));
        }
        qp += 4 * SPU;
    }
#pragma unroll
    for (int c = 0; c < NC; ++c) out[c] = __fmul_rn(ip_tree(acc[c]), 64.f);  // the scale: exact
}

// One candidate with the plain codes (kUnitScale below), a step at a time.
template <int SB>
__device__ __forceinline__ float ex_ip_plain(const float4* __restrict__ uq4, const uint4* __restrict__ row, int r,
                                             int steps) {
    constexpr int SPW = 8 / SB;  // steps per 32-bit word
    const uint32_t* words = reinterpret_cast<const uint32_t*>(row + r);
    float2 acc[2] = {make_float2(0.f, 0.f), make_float2(0.f, 0.f)};
#pragma unroll 1
    for (int t = 0; t < steps; ++t) {
        const int j = t / SPW;  // word j of this lane: word j % 4 of its uint4 j / 4
        const uint32_t w = __ldg(words + 16 * (j >> 2) + (j & 3)) >> (SB * (t % SPW));
        ip_step<false>(acc, uq4[4 * t + r], SB == 8 ? w : w & (0x01010101u * ((1u << SB) - 1u)));
    }
    return ip_tree(acc);
}

// unit_q is staged times 2^127 for the scaled codes.  With every non-zero
// |unit_q| in [2^-96, 2) the products and sums are multiples of 2^-125 below
// 2^128 in the scaled form, so each rounding is that of the plain one; a
// cluster whose unit query leaves that range (never, for data of ordinary
// magnitudes: its norm is 1) takes the plain codes.
constexpr float kUnitScale = 1.7014118346046923e38f;  // 2^127
__device__ __forceinline__ bool unit_scales(float u) {
    const float a = fabsf(u);
    return a == 0.f || (a >= 1.262177448e-29f && a < 2.f);  // 2^-96; false for NaN
}

constexpr int kRefineThreads = 128;     // 4 warps per query
// Three forms by the warps of a query's block.  The 4-warp form has the best
// rate (6 blocks an SM hide each other's replays); a query alone in its block
// waits for every window, and windows of more clusters and candidates, computed
// by more warps, are fewer and shorter.
constexpr int kMidWarps = 8;
constexpr int kWideWarps = 16;
constexpr int kWideTuning = 32;  // erq_plan_tuning's refine_warps of the wide form

// Window capacities: blocks (a lane each), listed candidates, clusters whose unit
// queries are staged at once (at most), block minima tested per thread.
template <int WARPS>
struct RefineForm {
    static constexpr bool kNarrow = WARPS == 4, kWide = WARPS == kWideWarps;
    static constexpr int kBlocks = kNarrow ? 16 : 32;
    // 8 warps, 444 slots of one wave: 2,000 queries of 1536 dims at nprobe 64 take
    // 730 us with 16 blocks and 256 candidates, 680 with 32 and 512, 668 with 384
    static constexpr int kEntries = kNarrow ? 256 : (kWide ? 1024 : 384);
    static constexpr int kSlots = kNarrow ? 8 : (kWide ? 16 : 12);
    static constexpr int kPerThread = kWide ? 2 : 4;
    static constexpr int kWords = WARPS * kPerThread;  // 32 blocks each
    static constexpr int kProbes = kWide ? 256 : 128;  // probes whose clusters are kept
    // shared memory of a block: 6 blocks of the 4-warp form per SM (1,284 us of
    // learned refinement with 5, 1,191 with 6; with 8 the ring does not fit,
    // 1,233), 3 of the 8-warp form (with 2, 4.69 ms where 3 take 4.22), one of
    // the wide form
    static constexpr int kRoom = kNarrow ? 36 * 1024 + 512 : (kWide ? 220 * 1024 : 73 * 1024 + 512);
    static constexpr int kPerSm = kNarrow ? 6 : (kWide ? 1 : 3);
};
template <int WARPS>
struct RefineShared {
    using F = RefineForm<WARPS>;
    uint4 ring[WARPS][kRowRing][2][32];  // EX-code words (ex_ip_ring)
    // slots: clusters whose unit queries are staged
    double ex_sub[F::kSlots];
    float y[F::kSlots], fac[F::kSlots], sqy[F::kSlots], delta[F::kSlots];
    uint32_t cid[F::kSlots], plain[F::kSlots];
    // blocks of the window
    float4 k[F::kBlocks];           // delta, c1, c2, c3 (LbConsts)
    uint32_t block[F::kBlocks];     // among the query's blocks
    uint32_t probe[F::kBlocks];
    uint32_t vec[F::kBlocks];       // position of lane 0's vector
    uint32_t on[F::kBlocks];        // index of its block factor
    uint32_t cid_of[F::kBlocks];
    float sqy_of[F::kBlocks], sumq_of[F::kBlocks];
    uint32_t lanes[F::kBlocks];     // vectors of the block
    uint32_t mask[F::kBlocks];      // lanes below the threshold
    uint32_t slot[F::kBlocks];
    uint32_t words[32];                // block minima below the threshold
    uint32_t start[F::kProbes], pcid[F::kProbes], psize[F::kProbes];  // first block, cluster, its size
    // the listed candidates, in scan order; a block's list is padded to an
    // even length (kNoEntry)
    float d[F::kEntries];
    uint32_t id[F::kEntries];
    uint16_t list[F::kEntries];        // 32 * window block + lane
    float lb[F::kBlocks * 32];         // lower bounds of the window's lanes
    float merge[32];                   // scratch of pool_merge_block
    int got, size;
    uint32_t next;
    float distk;
};
constexpr uint16_t kNoEntry = 0xffff;

__host__ __device__ constexpr int refine_pool_bytes(int kpad) { return kpad * 8; }  // distance, id
// Row length of a staged unit query: D up to whole uint4s of 8-, 4- or 2-bit codes.
__host__ __device__ constexpr int refine_row(int D) { return (D + 255) & ~255; }
// Unit queries staged at once: what the block's shared memory leaves, at least one.
template <int WARPS>
__host__ __device__ constexpr int refine_slots(int D, int kpad) {
    const int fixed = (int)sizeof(RefineShared<WARPS>) + refine_pool_bytes(kpad);
    const int room = RefineForm<WARPS>::kRoom - fixed;
    const int n = room / (4 * refine_row(D));
    return n < 1 ? 1 : (n > RefineForm<WARPS>::kSlots ? RefineForm<WARPS>::kSlots : n);
}
// [RefineShared][pool][unit queries]
template <int WARPS>
__host__ __device__ constexpr size_t refine_smem_bytes(int D, int kpad) {
    return sizeof(RefineShared<WARPS>) + (size_t)refine_pool_bytes(kpad) + (size_t)refine_slots<WARPS>(D, kpad) * refine_row(D) * 4;
}

// Order key: ascending distance (-0 equal to +0, as float compares see it);
// among equal distances the higher lane, offered to the pool later, first.
// Non-candidates sort last.
__device__ __forceinline__ uint64_t merge_key(float d, int lane, bool cand) {
    const uint32_t b = __float_as_uint(d == 0.f ? 0.f : d);
    const uint32_t o = (b & 0x80000000u) ? ~b : (b | 0x80000000u);
    return cand ? (((uint64_t)o << 32) | (uint32_t)(31 - lane)) : ~0ull;
}

// Offers one block's candidates (lanes with `cand`, distance d, id) to the
// pool in ascending lane order, as ResultPool::insert does one at a time
// (inc/index/Pool.hpp:15-26), in one parallel step.  Each insert keeps the k
// smallest entries under the order (distance, newer first): lower_bound
// places a new value before equal ones, an equal value still enters a full
// pool and pushes the last one out, a larger one is rejected.  A sequence of
// inserts therefore leaves the k smallest of (pool + sequence) in that order:
// sort the candidates by (distance, later lane first); pool entry i moves to
// i + #(candidates <= it), candidate j goes to j + #(pool entries < it), and
// ranks >= k fall off.  Executed by one whole warp; `cs` is 32 floats of
// scratch.  The caller may drop candidates that cannot enter a full pool
// (distance > its k-th): they would rank >= k and move no other entry.
__device__ __forceinline__ void pool_merge_block(float* pool_d, uint32_t* pool_id, int& size, int k,
                                                 float& distk, bool cand, float d, uint32_t id,
                                                 float* cs, int lane, bool count_all = false) {
    const uint32_t cm = __ballot_sync(0xffffffffu, cand);
    const int nc = __popc(cm);
    // each candidate's place among the pool entries: those below it (a new
    // value goes before equal ones), by binary search on the sorted pool
    const auto place = [&](bool m, float v) {
        int l = 0;
        if (m) {
            int hi = size;
            while (l < hi) {
                const int mid = (l + hi) >> 1;
                if (pool_d[mid] < v) l = mid + 1; else hi = mid;
            }
        }
        return l;
    };
    // Up to kFew candidates (any number with count_all) stay on their lanes:
    // a candidate's rank among the block's candidates is counted by broadcast,
    // and each pool entry counts the candidates below it.  More are sorted
    // (bitonic, lane j then holds the j-th).  Sorting pays while the pool fills
    // (blocks of up to 32 candidates spread over the whole pool); in a query's
    // later clusters counting is cheaper at any number.
    constexpr int kFew = 4;
    const bool few = count_all || nc <= kFew;
    int lo = 0;
    float dv = d;
    uint32_t val = id;
    bool mine = cand;
    int rk = 0;
    if (few) {
        lo = place(cand, d);
        const uint64_t key = merge_key(d, lane, cand);
        for (uint32_t m = cm; m; m &= m - 1u) {
            const int src = __ffs(m) - 1;
            rk += merge_key(__shfl_sync(0xffffffffu, d, src), src, true) < key;
        }
    } else {
        uint64_t key = merge_key(d, lane, cand);
#pragma unroll
        for (int sz = 2; sz <= 32; sz <<= 1) {
#pragma unroll
            for (int st = sz >> 1; st > 0; st >>= 1) {
                const uint64_t ok = __shfl_xor_sync(0xffffffffu, key, st);
                const uint32_t ov = __shfl_xor_sync(0xffffffffu, val, st);
                const float od = __shfl_xor_sync(0xffffffffu, dv, st);
                const bool take_min = ((lane & st) == 0) == ((lane & sz) == 0);
                if (take_min ? (ok < key) : (ok > key)) {
                    key = ok;
                    val = ov;
                    dv = od;
                }
            }
        }
        rk = lane;
        mine = lane < nc;
        cs[lane] = dv;
        lo = place(mine, dv);
    }
    // entries below the smallest candidate's place stay put
    const int first = (int)__reduce_min_sync(0xffffffffu, mine ? (uint32_t)lo : 0xffffffffu);
    const int rc = mine ? rk + lo : k;
    __syncwarp();
    // move pool entries, top chunk first: entry i goes to i + c(i) >= i, and
    // i + c(i) strictly increases with i, so no chunk overwrites an entry
    // that has not been read or one already moved
    for (int i0 = ((size - 1) >> 5) << 5; i0 >= 0 && i0 + 31 >= first; i0 -= 32) {
        const int i = i0 + lane;
        float pd = 0.f;
        uint32_t pid = 0u;
        if (i < size) {
            pd = pool_d[i];
            pid = pool_id[i];
        }
        int c = 0;
        if (few) {
            for (uint32_t m = cm; m; m &= m - 1u) c += __shfl_sync(0xffffffffu, d, __ffs(m) - 1) <= pd;
        } else if (i < size) {
            int h2 = nc;
            while (c < h2) {
                const int mid = (c + h2) >> 1;
                if (cs[mid] <= pd) c = mid + 1; else h2 = mid;
            }
        }
        const int pr = i < size ? i + c : k;
        __syncwarp();
        if (pr < k) {
            pool_d[pr] = pd;
            pool_id[pr] = pid;
        }
        __syncwarp();
    }
    if (rc < k) {
        pool_d[rc] = dv;
        pool_id[rc] = val;
    }
    __syncwarp();
    size = min(k, size + nc);
    distk = size == k ? pool_d[k - 1] : FLT_MAX;
}

// pool_merge_block on a pool whose size and threshold lie in shared memory,
// out of line: only pools above kSmallPool entries use it.
__device__ __noinline__ void pool_merge_shared(float* pool_d, uint32_t* pool_id, int* size_s, float* distk_s,
                                               int k, bool cand, float d, uint32_t id, float* cs, int lane,
                                               bool count_all) {
    int size = *size_s;
    float distk = *distk_s;
    __syncwarp();
    pool_merge_block(pool_d, pool_id, size, k, distk, cand, d, id, cs, lane, count_all);
    if (lane == 0) {
        *size_s = size;
        *distk_s = distk;
    }
    __syncwarp();
}

// The query's top-k pool.  ResultPool (inc/index/Pool.hpp:10-50) keeps the k
// smallest under the order (distance, newer first): a new value goes before
// equal ones, an equal value still enters a full pool and pushes the last one
// out, a larger one is rejected.  Up to kSmallPool entries warp 0 keeps a full
// pool sorted in registers, place p in lane p % 32: the order of the distance
// and the id, at the top places; those below hold order 0.  An insertion moves
// the entries not below the new one up a place, the largest out: about 45
// instructions without a branch (merging each block's candidates into a sorted
// pool in shared memory took about 600 per block).  Larger pools stay in shared
// memory (pool_merge_block).
constexpr int kSmallPool = 256;
// Order of a distance as an unsigned number (-0 as +0, as float compares see it).
__device__ __forceinline__ uint32_t float_order(float x) {
    const uint32_t b = __float_as_uint(x == 0.f ? 0.f : x);
    return (b & 0x80000000u) ? ~b : (b | 0x80000000u);
}
__device__ __forceinline__ float order_float(uint32_t o) {
    return __uint_as_float((o & 0x80000000u) ? (o & 0x7fffffffu) : ~o);
}
struct SmallPool {
    static constexpr int kRows = kSmallPool / 32;
    uint32_t v[kRows], id[kRows];  // the first R rows, R = 1, 4 or 8 by k

    // n entries (distance and id in d and ids, entry e the e-th insertion),
    // sorted by counting.  scratch: 64 * R words.  (A loop over the entries: a
    // sorting network in registers is 1,400 instructions run once a query.)
    template <int R>
    __device__ __forceinline__ void fill(const float* d, const uint32_t* ids, int n, int lane, uint32_t* scratch) {
        uint32_t* sid = scratch + 32 * R;
        int at[R];
#pragma unroll
        for (int j = 0; j < R; ++j) {
            const int e = lane + 32 * j;
            v[j] = e < n ? float_order(d[e]) : 0u;
            id[j] = e < n ? ids[e] : 0u;
            at[j] = 32 * R - n;
            scratch[e] = v[j];
        }
        __syncwarp();
#pragma unroll(R == 8 ? 4 : 8)
        for (int e = 0; e < n; ++e) {
            const uint32_t x = scratch[e];
#pragma unroll
            for (int j = 0; j < R; ++j)  // of equal ones the newer comes first
                at[j] += x < v[j] + (uint32_t)(e > lane + 32 * j);
        }
        __syncwarp();
#pragma unroll
        for (int j = 0; j < R; ++j) {
            const int e = lane + 32 * j, to = e < n ? at[j] : e - n;
            scratch[to] = v[j];
            sid[to] = id[j];
        }
        __syncwarp();
#pragma unroll
        for (int j = 0; j < R; ++j) {
            v[j] = scratch[lane + 32 * j];
            id[j] = sid[lane + 32 * j];
        }
        __syncwarp();
    }
    // Order of the k-th distance (of a full pool).
    template <int R>
    __device__ __forceinline__ uint32_t last() const {
        return __shfl_sync(0xffffffffu, v[R - 1], 31);
    }
    // Inserts (x, vid), x the order of its distance: before equal ones, the
    // largest entry leaves (x itself when it is larger than all).
    template <int R>
    __device__ __forceinline__ void insert(uint32_t x, uint32_t vid, int lane) {
        uint32_t rv[R], ri[R];
#pragma unroll
        for (int j = 0; j < R; ++j) {  // the entries one place down (lane 0: one row up)
            rv[j] = __shfl_sync(0xffffffffu, v[j], (lane + 31) & 31);
            ri[j] = __shfl_sync(0xffffffffu, id[j], (lane + 31) & 31);
        }
#pragma unroll
        for (int j = 0; j < R; ++j) {
            const uint32_t dv = lane ? rv[j] : (j ? rv[j > 0 ? j - 1 : 0] : 0u);
            const uint32_t di = lane ? ri[j] : (j ? ri[j > 0 ? j - 1 : 0] : 0u);
            const bool stays = v[j] < x, here = dv < x;
            id[j] = stays ? id[j] : (here ? vid : di);
            v[j] = stays ? v[j] : (here ? x : dv);
        }
    }
};

// What a warp needs to replay a window (below).
struct Replay {
    const uint16_t* list;
    const float* d;
    const float* lb;
    const uint32_t* ids;
    float* pool_d;      // the entries of a pool that is not full
    uint32_t* pool_id;
    uint32_t* scratch;
    int entries, k;
    bool all;           // count every candidate (RefineArgs::stats)
};

// Replays a window's list in the reference's order: each block's candidates
// against the threshold at that block's start, those that can enter inserted
// one by one.  worst: order of the threshold, order of FLT_MAX while the pool
// fills.
template <int R>
__device__ __forceinline__ void replay_window(const Replay& w, SmallPool& sp, int& size, uint32_t& worst,
                                              uint32_t& st_cand, int lane) {
    const uint32_t lt = (1u << lane) - 1u;
    int cur = -1;  // block the replay is in, and the threshold at its start
    uint32_t at_start = worst;
    uint32_t most = worst;  // the pool's largest is no more (infinite ones may be among those that fill it)
#pragma unroll 1
    for (int e0 = 0; e0 < w.entries; e0 += 32) {
        const int e = e0 + lane;
        const uint32_t l = e < w.entries ? w.list[e] : kNoEntry;
        const bool valid = l != kNoEntry;
        const float d = valid ? w.d[e] : 0.f;
        const uint32_t od = float_order(d), ol = float_order(valid ? w.lb[l] : 0.f);
        const uint32_t vid = valid ? w.ids[e] : 0u;
        const int blk = (int)(l >> 5);
        // those above a full pool's k-th cannot enter
        uint32_t todo = __ballot_sync(0xffffffffu, valid && (w.all || size < w.k || od <= worst));
        if (size < w.k && todo) {
            // the pool fills: its blocks started without a threshold, so
            // every listed lane is a candidate
            const int at = size + __popc(todo & lt);
            const bool take = ((todo >> lane) & 1u) && at < w.k;
            if (take) {
                w.pool_d[at] = d;
                w.pool_id[at] = vid;
            }
            const uint32_t taken = __ballot_sync(0xffffffffu, take);
            cur = __shfl_sync(0xffffffffu, blk, 31 - __clz((int)taken));
            size += __popc(taken);
            if (w.all) st_cand += __popc(taken);
            todo &= ~taken;
            __syncwarp();
            if (size == w.k) {
                sp.fill<R>(w.pool_d, w.pool_id, w.k, lane, w.scratch);
                worst = sp.last<R>();
                most = max(most, worst);
                todo &= __ballot_sync(0xffffffffu, w.all || od <= worst);
            }
        }
#pragma unroll 1
        while (todo) {  // a block at a time
            const int b = __shfl_sync(0xffffffffu, blk, __ffs(todo) - 1);
            if (b != cur) {
                cur = b;
                at_start = most = sp.last<R>();
            }
            const bool mine = ((todo >> lane) & 1u) && blk == b;
            const bool candidate = mine && ol < at_start;
            todo &= ~__ballot_sync(0xffffffffu, mine);
            if (w.all) st_cand += __popc(__ballot_sync(0xffffffffu, candidate));
            // a larger distance than the largest leaves the pool as it is
            uint32_t in = __ballot_sync(0xffffffffu, candidate && od <= most);
#pragma unroll 1
            while (in) {
                const int src = __ffs(in) - 1;
                in &= in - 1u;
                sp.insert<R>(__shfl_sync(0xffffffffu, od, src), __shfl_sync(0xffffffffu, vid, src), lane);
            }
        }
        if (size == w.k) worst = sp.last<R>();
    }
}

// The sorted pool to the query's results.
template <int R>
__device__ __forceinline__ void pool_out(SmallPool& sp, const Replay& w, int size, uint32_t* oid, float* od,
                                         int lane) {
    if (size < w.k) sp.fill<R>(w.pool_d, w.pool_id, size, lane, w.scratch);
#pragma unroll
    for (int j = 0; j < R; ++j) {
        const int i = lane + 32 * j - (32 * R - size);
        if (i >= 0) {
            oid[i] = sp.id[j];
            if (od) od[i] = order_float(sp.v[j]);
        }
    }
}

// One block of WARPS warps per query (4, 8 or 16).  The query's
// blocks - of all its probed clusters, in probe order - form one sequence; a
// window is the next of them whose smallest lower bound (from the scan) is
// below the threshold at the window's start (a block above it has no candidate
// then or later), whatever clusters they belong to.  The warps compute the
// lower bounds of the window's blocks and list the lanes below the threshold -
// a superset of the exact candidates, because the threshold only falls; the
// quads compute the listed candidates' exact distances against the staged unit
// queries; warp 0 then replays the window in the reference's order: each
// block's candidates against the threshold at that block's start, those that
// can enter inserted one by one.
// A window ends early when its list is full, when its candidates come from
// more clusters than unit queries fit, or, while the pool fills (every lane is
// a candidate), once it can fill it; its length never changes a result.
// Windows across clusters keep the quads busy where a cluster has a few
// candidates: with a window per cluster (and up to 16 of its blocks) 2,047
// queries at nprobe 96 over Zipf clusters took 109 windows each and 5.41 ms, now
// 40 and 4.45 ms; 64 queries at nprobe 128 129 and 1.12 ms, now 14 and 0.56 ms;
// 2,000 queries at nprobe 64 over even clusters 67 and 1.47 ms, now 4 and 0.92 ms;
// one query of 128 dims at nprobe 32 88 us, now 35 us.
template <int EX, int WARPS>
__global__ void __launch_bounds__(WARPS * 32, RefineForm<WARPS>::kPerSm) refine_kernel(RefineArgs a) {
    using F = RefineForm<WARPS>;
    constexpr int kThreads = WARPS * 32;
    constexpr int kOwn = F::kBlocks / WARPS;  // window blocks per warp
    constexpr int SB = ex_storage_bits(EX);
    extern __shared__ __align__(16) uint8_t smem_raw[];
    RefineShared<WARPS>& sh = *reinterpret_cast<RefineShared<WARPS>*>(smem_raw);
    const int tid = threadIdx.x, lane = tid & 31;
    // through a shuffle, so that the compiler knows it uniform over the warp and
    // the warp-wide operations of the branches on it need no resynchronisation
    const int warp = __shfl_sync(0xffffffffu, tid >> 5, 0);
    const uint32_t lt = (1u << lane) - 1u;
    const int q = a.order ? (int)a.order[blockIdx.x] : (int)blockIdx.x;
    const int D = a.D, k = a.k, kpad = (k + 31) & ~31;
    const int nslots = refine_slots<WARPS>(D, kpad), row_len = refine_row(D);
    const int row_words = (int)ex_row_uint4(D, EX);
    float* pool_d = reinterpret_cast<float*>(smem_raw + sizeof(RefineShared<WARPS>));
    uint32_t* pool_id = reinterpret_cast<uint32_t*>(pool_d + kpad);
    float* uq = reinterpret_cast<float*>(pool_id + kpad);
    const uint32_t ring = (uint32_t)__cvta_generic_to_shared(&sh.ring[warp][0][0][lane]);
    // warp 0's ring is free while it replays
    Replay rp{sh.list, sh.d, sh.lb, sh.id, pool_d, pool_id, reinterpret_cast<uint32_t*>(&sh.ring[0][0][0][0]), 0, k,
              a.stats != nullptr};
    SmallPool sp;            // with size and distk, maintained by warp 0
    int size = 0;
    uint32_t worst = float_order(FLT_MAX);  // order of the threshold
    const float one_over_sqrtD = recip_via_double(__fsqrt_rn((float)D));
    const float* qv = a.qrot + (size_t)q * D;
    const size_t q0 = (size_t)q * a.nprobe;
    const int np_q = a.q_nprobe ? a.q_nprobe[q] : a.nprobe;
    const uint64_t s_base = a.s_off[q0];
    const int32_t* S = a.S + s_base;
    const float* bmin = a.bmin ? a.bmin + s_base / 32 : nullptr;
    const auto start_of = [&](int p) -> uint32_t {
        return p < F::kProbes ? sh.start[p] : (uint32_t)((a.s_off[q0 + p] - s_base) >> 5);
    };
    const auto cid_of = [&](int p) -> uint32_t { return p < F::kProbes ? sh.pcid[p] : a.probe_cid[q0 + p]; };
    const auto size_of = [&](int p) -> uint32_t { return p < F::kProbes ? sh.psize[p] : a.c_size[cid_of(p)]; };
#pragma unroll 1
    for (int p = tid; p < np_q && p < F::kProbes; p += kThreads) {
        const uint32_t c = a.probe_cid[q0 + p];
        sh.pcid[p] = c;
        sh.start[p] = (uint32_t)((a.s_off[q0 + p] - s_base) >> 5);
        sh.psize[p] = a.c_size[c];
    }
    if (tid == 0) {
        sh.distk = FLT_MAX;
        sh.size = 0;
    }
    uint32_t st_cand = 0, st_refined = 0, st_windows = 0, st_blocks = 0;  // with a.stats
    uint32_t held_probe = 0xffffffffu;  // the last staged cluster's probe, and its slot
    int held_slot = 0;
    __syncthreads();
    const uint32_t first_size = sh.psize[0];
    const uint32_t total = start_of(np_q - 1) + ((size_of(np_q - 1) + 31u) >> 5);

    for (uint32_t pos = 0; pos < total;) {
        const float d0 = sh.distk;
        const int need = k - sh.size;  // entries the pool lacks
        // the next blocks' minima against the threshold
        const bool open = !bmin || d0 == FLT_MAX;
#pragma unroll
        for (int i = 0; i < F::kPerThread; ++i) {
            const uint32_t bb = pos + i * kThreads + tid;
            // (without a threshold every block may have candidates: no need to look)
            const uint32_t m = __ballot_sync(0xffffffffu, bb < total && (open || bmin[bb] < d0));
            if (lane == 0) sh.words[i * WARPS + warp] = m;
        }
        __syncthreads();
        // warp 0 takes the window's blocks and reads what they need, a lane each
        if (warp == 0) {
            const int want = need > 0 && first_size >= (uint32_t)k ? min(F::kBlocks, (need + 31) >> 5) : F::kBlocks;
            uint32_t w = lane < F::kWords ? sh.words[lane] : 0u;
            int incl = __popc(w);
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const int v = __shfl_up_sync(0xffffffffu, incl, o);
                if (lane >= o) incl += v;
            }
            const int all = __shfl_sync(0xffffffffu, incl, 31);
#pragma unroll 1
            for (int e = incl - __popc(w); w && e < want; ++e, w &= w - 1u)
                sh.block[e] = pos + 32 * lane + __ffs(w) - 1;
            __syncwarp();
            const int got = min(all, want);
            if (lane < got) {
                const uint32_t b = sh.block[lane];
                int lo = 0, n = np_q;  // the last probe that starts at or before b
#pragma unroll 1
                while (n > 1) {
                    const int h = n >> 1;
                    if (start_of(lo + h) <= b) {
                        lo += h;
                        n -= h;
                    } else {
                        n = h;
                    }
                }
                const uint32_t cid = cid_of(lo);
                const float delta = a.qp_delta[q0 + lo], sumq = a.qp_sumq[q0 + lo], sqy = a.probe_sqy[q0 + lo];
                sh.cid_of[lane] = cid;
                sh.sqy_of[lane] = sqy;
                sh.sumq_of[lane] = sumq;
                // constants of inc/index/fastscan/FastScan.hpp:297-303
                const LbConsts kc = lb_consts(sumq, __fsqrt_rn(sqy), one_over_sqrtD);
                const uint32_t r = b - start_of(lo);
                sh.probe[lane] = (uint32_t)lo;
                sh.vec[lane] = a.c_first_vec[cid] + 32 * r;
                sh.on[lane] = (a.c_first_block[cid] + r) * 32;
                sh.lanes[lane] = min(32u, size_of(lo) - 32 * r);
                sh.k[lane] = make_float4(delta, kc.c1, kc.c2, kc.c3);
            }
            if (lane == 0) {
                sh.got = got;
                sh.next = all > want ? sh.block[want - 1] + 1 : min(total, pos + 32u * F::kWords);
            }
        }
        __syncthreads();
        const int got = sh.got;
        uint32_t next = sh.next;
        if (got == 0) {  // uniform
            pos = next;
            continue;
        }
        // lower bounds, blocks dealt to the warps round robin
#pragma unroll 4
        for (int i = 0; i < kOwn; ++i) {
            const int b = i * WARPS + warp;
            if (b < got) {  // uniform per warp
                const float4 kc = sh.k[b];
                const float on = a.onorm[(size_t)sh.on[b] + lane];
                const float ipq = __fmul_rn(__int2float_rn(S[32 * (size_t)sh.block[b] + lane]), kc.x);
                const float lb = lower_bound(ipq, on, LbConsts{kc.y, kc.z, kc.w});
                const uint32_t m = __ballot_sync(0xffffffffu, lane < (int)sh.lanes[b] && lb < d0);
                sh.lb[32 * b + lane] = lb;
                if (lane == 0) sh.mask[b] = m;
            }
        }
        __syncthreads();
        // every warp: where each block's candidates go, and where the window ends
        const uint32_t bmask = lane < got ? sh.mask[lane] : 0u;
        const uint32_t bprobe = lane < got ? sh.probe[lane] : 0u;
        const int cnt = __popc(bmask), even = (cnt + 1) & ~1;
        int end = even, seen = cnt;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int v = __shfl_up_sync(0xffffffffu, end, o), u = __shfl_up_sync(0xffffffffu, seen, o);
            if (lane >= o) {
                end += v;
                seen += u;
            }
        }
        const uint32_t has = __ballot_sync(0xffffffffu, cnt > 0);
        const int before = 31 - __clz((int)(has & lt));  // the block with candidates before this one
        const uint32_t pprobe = __shfl_sync(0xffffffffu, bprobe, before & 31);
        const bool fresh = cnt > 0 && (before < 0 || pprobe != bprobe);
        const uint32_t freshm = __ballot_sync(0xffffffffu, fresh);
        const int rank = __popc(freshm & (lt | (1u << lane))) - 1;  // of this block's cluster
        const bool fits = end <= F::kEntries && rank < nslots && (need <= 0 || seen - cnt < need);
        const uint32_t out = __ballot_sync(0xffffffffu, !fits && lane < got);
        const int nb = out ? __ffs(out) - 1 : got;  // blocks of the window, at least one
        if (nb < got) next = sh.block[nb];
        const int entries = __shfl_sync(0xffffffffu, end, nb - 1);
        const uint32_t inm = freshm & (nb < 32 ? (1u << nb) - 1u : 0xffffffffu);
        const int ns = __popc(inm);  // clusters with candidates
        // the first one may be staged already, from the window before
        const uint32_t probe0 = __shfl_sync(0xffffffffu, bprobe, inm ? __ffs(inm) - 1 : 0);
        const bool held = ns > 0 && probe0 == held_probe;
        const int slot0 = held ? held_slot : 0;
        const int slot = rank < 0 ? 0 : (slot0 + rank) % nslots;
        if (warp == 0 && lane < nb) {
            sh.slot[lane] = (uint32_t)slot;
            if (fresh && !(held && rank == 0)) {
                const float sumq = sh.sumq_of[lane], sqy = sh.sqy_of[lane];
                sh.cid[slot] = sh.cid_of[lane];
                sh.plain[slot] = 0u;
                const float y = __fsqrt_rn(sqy);
                sh.y[slot] = y;
                sh.fac[slot] = recip_via_double(y);
                sh.sqy[slot] = sqy;
                sh.delta[slot] = sh.k[lane].x;
                sh.ex_sub[slot] = __dmul_rn((double)(1 << EX) - 0.5, (double)sumq);
            }
        }
        if (ns > 0) {
            const int lastb = 31 - __clz((int)inm);
            held_probe = __shfl_sync(0xffffffffu, bprobe, lastb);
            held_slot = (slot0 + ns - 1) % nslots;
        }
#pragma unroll 2
        for (int i = 0; i < kOwn; ++i) {
            const int b = i * WARPS + warp;
            if (b < nb) {
                const int base = __shfl_sync(0xffffffffu, end - even, b);
                const uint32_t m = __shfl_sync(0xffffffffu, bmask, b);
                if ((m >> lane) & 1u) {
                    const int e = base + __popc(m & lt);
                    sh.list[e] = (uint16_t)(32 * b + lane);
                    // start the candidate's EX-code row on its way to L2
                    asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(
                                     a.excode + ((size_t)sh.vec[b] + lane) * a.ex_row),
                                 "r"((uint32_t)a.ex_row)
                                 : "memory");
                }
                if (lane == 0 && (__popc(m) & 1)) sh.list[base + __popc(m)] = kNoEntry;
            }
        }
        if (a.stats) {
            st_refined += __shfl_sync(0xffffffffu, seen, nb - 1);
            st_windows += 1;
            st_blocks += nb;
        }
        __syncthreads();
        if (entries == 0) {  // uniform: nothing in this window can pass
            pos = next;
            continue;
        }
        // unit queries of the clusters not staged yet, scaled; if one of them
        // leaves the range (never, for ordinary data), all the window's plain
        bool plain = false;
        for (bool scaled = true;; scaled = false) {
            const int r0 = scaled && held ? 1 : 0, g4 = row_len >> 2;
#pragma unroll 1
            for (int i = tid; i < (ns - r0) * g4; i += kThreads) {
                const int r = i / g4, g = i - r * g4, s = (slot0 + r0 + r) % nslots;
                float4 u = make_float4(0.f, 0.f, 0.f, 0.f);  // past D
                if (4 * g < D) {
                    const float fac = sh.fac[s];
                    if (sh.y[s] > kNormEps) {
                        const float4 x = reinterpret_cast<const float4*>(qv)[g];
                        const float4 c = __ldg(reinterpret_cast<const float4*>(a.centroids + (size_t)sh.cid[s] * D) + g);
                        u = make_float4(__fmul_rn(__fsub_rn(x.x, c.x), fac), __fmul_rn(__fsub_rn(x.y, c.y), fac),
                                        __fmul_rn(__fsub_rn(x.z, c.z), fac), __fmul_rn(__fsub_rn(x.w, c.w), fac));
                    } else {  // (float)(1.0 / sqrt(D))
                        u = make_float4(one_over_sqrtD, one_over_sqrtD, one_over_sqrtD, one_over_sqrtD);
                    }
                }
                if (scaled) {
                    if (!(unit_scales(u.x) && unit_scales(u.y) && unit_scales(u.z) && unit_scales(u.w)))
                        sh.plain[s] = 1u;
                    u = make_float4(__fmul_rn(u.x, kUnitScale), __fmul_rn(u.y, kUnitScale),
                                    __fmul_rn(u.z, kUnitScale), __fmul_rn(u.w, kUnitScale));
                }
                reinterpret_cast<float4*>(uq + (size_t)s * row_len)[g] = u;
            }
            __syncthreads();
            if (!scaled) break;
#pragma unroll 1
            for (int r = 0; r < ns; ++r) plain |= sh.plain[(slot0 + r) % nslots] != 0u;
            if (!plain) break;  // uniform
            held_probe = 0xffffffffu;  // nothing scaled will be left
            __syncthreads();  // sh.plain is rewritten below for the next window
        }
        // exact distances: quad g (lanes 4g..4g+3) takes one candidate while
        // there are no more than quads, else two of a block; quads past the
        // end repeat the first so that the warp stays converged
        {
            const int g = tid >> 2, r = tid & 3;
            const bool two = entries > kThreads / 4;
            const int tasks = two ? entries >> 1 : entries;
#pragma unroll 1
            for (int base = 0; base + 8 * warp < tasks; base += kThreads / 4) {
                const int t = base + g;
                const int i0 = t < tasks ? (two ? 2 * t : t) : 0;
                const int s0 = sh.list[i0] == kNoEntry ? sh.list[0] : sh.list[i0];
                const int i1 = two ? i0 + 1 : i0;
                const int s1 = two && sh.list[i1] != kNoEntry ? sh.list[i1] : s0;
                const size_t pos0 = (size_t)sh.vec[s0 >> 5] + (s0 & 31);
                const size_t pos1 = (size_t)sh.vec[s1 >> 5] + (s1 & 31);
                const uint4* row0 = reinterpret_cast<const uint4*>(a.excode + pos0 * a.ex_row);
                const uint4* row1 = reinterpret_cast<const uint4*>(a.excode + pos1 * a.ex_row);
                // lane 0 of the quad finishes the first, lane 1 the second
                const int mine = r == 0 ? i0 : i1, sl = r == 0 ? s0 : s1;
                const int wb = sl >> 5;
                const bool fin = t < tasks && (r == 0 || (r == 1 && two)) && sh.list[mine] != kNoEntry;
                const uint32_t cs = sh.slot[wb];
                float xipn = 0.f, on = 0.f;
                int sum = 0;
                uint32_t vid = 0u;
                if (fin) {
                    const size_t at = r == 0 ? pos0 : pos1;
                    xipn = __ldg(a.xipnorm + at);
                    vid = __ldg(a.ids + at);
                    on = a.onorm[(size_t)sh.on[wb] + (sl & 31)];
                    sum = S[32 * (size_t)sh.block[wb] + (sl & 31)];
                }
                const float4* uq4 = reinterpret_cast<const float4*>(uq + (size_t)cs * row_len);
                float ip[2];
                if (plain) {
                    ip[0] = ex_ip_plain<SB>(uq4, row0, r, D / 16);
                    ip[1] = ex_ip_plain<SB>(uq4, row1, r, D / 16);
                } else if (two) {
                    ex_ip_ring<SB, 2>(uq4, row0, row1, r, row_words, ring, ip);
                } else {
                    ex_ip_ring<SB, 1>(uq4, row0, row0, r, row_words, ring, ip);
                }
                if (fin) {
                    // inc/index/HASearcher.hpp:225-232
                    const float y = sh.y[cs];
                    const float ipq = __fmul_rn(__int2float_rn(sum), sh.delta[cs]);
                    const float sqr_x = __fmul_rn(on, on);
                    const float tt = __fadd_rn(__fmul_rn((float)(1 << EX), ipq), r == 0 ? ip[0] : ip[1]);
                    const double br = __dsub_rn((double)tt, sh.ex_sub[cs]);
                    const float xy = __fmul_rn(xipn, y);
                    const float f = __fadd_rn(sqr_x, sh.sqy[cs]);
                    // what is not a number (the factor of a damaged file) counts as
                    // infinite: the pools order numbers only
                    sh.d[mine] = fminf(__double2float_rn(__dsub_rn((double)f, __dmul_rn((double)xy, br))), INFINITY);
                    sh.id[mine] = vid;
                }
            }
        }
        __syncthreads();
        if (k > kSmallPool) {
            if (warp == 0) {
#pragma unroll 1
                for (int b = 0; b < nb; ++b) {
                    // candidates of the block against the threshold at its
                    // start; those above a full pool's k-th cannot enter
                    const uint32_t m = __shfl_sync(0xffffffffu, bmask, b);
                    const int e = __shfl_sync(0xffffffffu, end - even, b) + __popc(m & lt);
                    const bool listed = (m >> lane) & 1u;
                    const float d = listed ? sh.d[e] : 0.f;
                    const bool below = listed && sh.lb[32 * b + lane] < sh.distk;
                    if (a.stats) st_cand += __popc(__ballot_sync(0xffffffffu, below));
                    const bool enter = below && (sh.size < k || !(d > sh.distk));
                    if (__ballot_sync(0xffffffffu, enter))
                        pool_merge_shared(pool_d, pool_id, &sh.size, &sh.distk, k, enter, d, listed ? sh.id[e] : 0u,
                                          sh.merge, lane, pos >= ((first_size + 31u) >> 5));
                }
            }
        } else if (warp == 0) {
            rp.entries = entries;
            if (k <= 32) replay_window<1>(rp, sp, size, worst, st_cand, lane);
            else if (k <= 128) replay_window<4>(rp, sp, size, worst, st_cand, lane);
            else replay_window<8>(rp, sp, size, worst, st_cand, lane);
        }
        if (tid == 0 && k <= kSmallPool) {
            sh.distk = order_float(worst);
            sh.size = size;
        }
        __syncthreads();
        pos = next;
    }
    // the pool's entries in order: ascending distance, newer first
    if (a.stats && tid == 0) {
        atomicAdd(a.stats + 0, (unsigned long long)st_cand);
        atomicAdd(a.stats + 1, (unsigned long long)st_refined);
        atomicAdd(a.stats + 2, (unsigned long long)st_windows);
        atomicAdd(a.stats + 3, (unsigned long long)st_blocks);
    }
    size = sh.size;
    uint32_t* oid = a.out_ids + (size_t)q * k;
    float* od = a.out_dists ? a.out_dists + (size_t)q * k : nullptr;
    if (k > kSmallPool) {  // sorted already
#pragma unroll 1
        for (int i = tid; i < size; i += kThreads) {
            oid[i] = pool_id[i];
            if (od) od[i] = pool_d[i];
        }
    } else if (warp == 0) {
        if (k <= 32) pool_out<1>(sp, rp, size, oid, od, lane);
        else if (k <= 128) pool_out<4>(sp, rp, size, oid, od, lane);
        else pool_out<8>(sp, rp, size, oid, od, lane);
    }
#pragma unroll 1
    for (int i = size + tid; i < k; i += kThreads) {
        oid[i] = 0u;
        if (od) od[i] = __int_as_float(0x7f800000);
    }
}

}  // namespace erq
