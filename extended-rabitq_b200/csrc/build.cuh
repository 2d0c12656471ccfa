// Index construction on the GPU: IVF::construct (inc/index/IVF.hpp:116-153)
// with DataQuantizer::quantize (inc/index/Quantizer.hpp:233-311) for every
// cluster, HIGH_ACC_FAST_SCAN format, writing the bytes the reference's
// create_index writes for the same data, centroids, cluster ids and rotation.
//
// Vectors are processed in file order: clusters in order, each cluster's
// members by ascending data index (IVF::construct's IDLists).  Per vector:
//   build_rotate_kernel   XP = pad(x) P - pad(c) P, every product summed in
//                         ascending k with separate multiply and add
//                         (data_transformation, Quantizer.hpp:316-362, whose
//                         matrix product accumulates that way)
//   build_rows_kernel     ||XP|| in double (ascending dims), XP / ||XP|| in
//                         float, the sign bits (XP > 0)
//   build_x2_kernel       L2Sqr(x, c) over DIM (16 FMA chains + the reduce
//                         tree, then the tail in order) and ||o - c|| =
//                         sqrt((double) that) (rabitq_factor, Quantizer.hpp:386-437)
//   fast_quantize_kernel  the EX-bit code: fast_quantize's sweep over the
//                         critical rescaling factors (Quantizer.hpp:138-219),
//                         a block per vector: windows of the factors sorted in
//                         shared memory, every double value as the reference
//                         computes it (fast_quantize_serial_kernel, one thread
//                         with a heap, for vectors outside its terms)
//   build_long_kernel     codes flipped on negative dims, store_compacted_code
//                         (Quantizer.hpp:491-631), xipnorm = ipnorm * 2 * ||o - c||
//   build_short_kernel    the 1-bit FastScan blocks (pack_binary + pack_codes,
//                         Quantizer.hpp:371-384, fastscan/pack_codes.hpp:33-98)
//                         and the block factor ||o - c||; lanes past the
//                         cluster's end hold zero codes and factor 0 (the
//                         reference leaves those factors unset)
#pragma once

#include <cstdint>

#include "common.cuh"

namespace erq {

constexpr int kBuildBM = 64, kBuildBN = 64, kBuildBK = 16;

// out[r][j] = sum_{k < D} xp[r][k] P[k][j] (ascending k, multiply then add),
// xp = row order[r] of x padded with zeros from DIM to D; minus sub[cid[r]][j]
// when sub is given.  64 x 64 output tile per 256-thread block, 4 x 4 per
// thread.
__global__ void __launch_bounds__(256) build_rotate_kernel(const float* __restrict__ x, int DIM,
                                                           const uint32_t* __restrict__ order, int n,
                                                           const float* __restrict__ P, int D,
                                                           const float* __restrict__ sub,
                                                           const uint32_t* __restrict__ cid,
                                                           float* __restrict__ out) {
    __shared__ float As[kBuildBK][kBuildBM + 4];
    __shared__ float Bs[kBuildBK][kBuildBN + 4];
    const int tid = threadIdx.x;
    const int tx = tid & 15, ty = tid >> 4;
    const int row0 = blockIdx.y * kBuildBM, col0 = blockIdx.x * kBuildBN;
    float acc[4][4];
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) acc[i][j] = 0.f;
    for (int k0 = 0; k0 < D; k0 += kBuildBK) {
        for (int i = tid; i < kBuildBM * kBuildBK; i += 256) {
            const int m = i / kBuildBK, kk = i % kBuildBK;
            const int r = row0 + m, k = k0 + kk;
            float v = 0.f;
            if (r < n && k < DIM) v = x[(size_t)(order ? order[r] : (uint32_t)r) * DIM + k];
            As[kk][m] = v;
        }
        for (int i = tid; i < kBuildBK * kBuildBN; i += 256) {
            const int kk = i / kBuildBN, c = i % kBuildBN;
            Bs[kk][c] = (col0 + c < D) ? P[(size_t)(k0 + kk) * D + col0 + c] : 0.f;
        }
        __syncthreads();
#pragma unroll
        for (int kk = 0; kk < kBuildBK; ++kk) {
            float a[4], b[4];
#pragma unroll
            for (int i = 0; i < 4; ++i) a[i] = As[kk][ty * 4 + i];
#pragma unroll
            for (int j = 0; j < 4; ++j) b[j] = Bs[kk][tx * 4 + j];
#pragma unroll
            for (int i = 0; i < 4; ++i)
#pragma unroll
                for (int j = 0; j < 4; ++j) acc[i][j] = __fadd_rn(acc[i][j], __fmul_rn(a[i], b[j]));
        }
        __syncthreads();
    }
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const int r = row0 + ty * 4 + i;
        if (r >= n) continue;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const int c = col0 + tx * 4 + j;
            if (c >= D) continue;
            float v = acc[i][j];
            if (sub) v = __fsub_rn(v, sub[(size_t)cid[r] * D + c]);
            out[(size_t)r * D + c] = v;
        }
    }
}

// One thread per row of xp [n][D]: sq = sum of double(x)^2 in ascending
// dims, norm = (float)sqrt(sq); xp becomes x / norm (unchanged when sq = 0,
// rowwise().normalized()); bits[r][w] bit i = (x_{64w+i} > 0).
__global__ void build_rows_kernel(float* __restrict__ xp, int n, int D, uint64_t* __restrict__ bits) {
    const int r = blockIdx.x * blockDim.x + threadIdx.x;
    if (r >= n) return;
    float* row = xp + (size_t)r * D;
    double sq = 0.0;
    for (int j = 0; j < D; ++j) {
        const double v = (double)row[j];
        sq = __dadd_rn(sq, __dmul_rn(v, v));
    }
    const float norm = __double2float_rn(__dsqrt_rn(sq));
    for (int w = 0; w < D / 64; ++w) {
        uint64_t b = 0;
        for (int i = 0; i < 64; ++i) {
            const float v = row[64 * w + i];
            b |= (uint64_t)(v > 0.f) << i;
            if (sq > 0.0) row[64 * w + i] = __fdiv_rn(v, norm);
        }
        bits[(size_t)r * (D / 64) + w] = b;
    }
}

// ||o - c|| of each row: L2Sqr (inc/utils/space.hpp:18-51) over DIM of the
// raw vector and its raw centroid, then sqrt in double rounded to float.
// One half-warp per row.
__global__ void build_x2_kernel(const float* __restrict__ x, const uint32_t* __restrict__ order,
                                const float* __restrict__ cent, const uint32_t* __restrict__ cid,
                                int n, int DIM, float* __restrict__ onorm) {
    const int hw = (blockIdx.x * blockDim.x + threadIdx.x) >> 4, l = threadIdx.x & 15;
    const int r = min(hw, n - 1);
    const float* a = x + (size_t)order[r] * DIM;
    const float* c = cent + (size_t)cid[r] * DIM;
    const int num16 = DIM - (DIM & 15);
    float acc = 0.f;
    for (int i = l; i < num16; i += 16) {
        const float t = __fsub_rn(a[i], c[i]);
        acc = __fmaf_rn(t, t, acc);
    }
    float s = tree16_sum(acc);
    if (l == 0 && hw < n) {
        for (int i = num16; i < DIM; ++i) {
            const float t = __fsub_rn(a[i], c[i]);
            s = __fadd_rn(s, __fmul_rn(t, t));
        }
        onorm[hw] = __double2float_rn(__dsqrt_rn((double)s));
    }
}

// fast_quantize (inc/index/Quantizer.hpp:138-219) for the rows listed in
// list[0 .. T) of xn, one thread per row.  The thread's priority queue of (t, dim),
// ordered by t then dim as std::priority_queue<pair, ..., greater> pops them,
// and its current codes live in global memory, entry e of thread j at
// e * T + j.  code[r][i] = the EX-bit magnitude code of |xn[r][i]|,
// ipnorm[r] = 1 / sum (code + 0.5) |xn| (1 when not finite).
__global__ void fast_quantize_serial_kernel(const float* __restrict__ xn, const uint32_t* __restrict__ list,
                                            int T, int D, int EX, double* __restrict__ heap_t,
                                            uint16_t* __restrict__ heap_i, uint8_t* __restrict__ cur,
                                            uint8_t* __restrict__ code, float* __restrict__ ipnorm) {
    const int j = blockIdx.x * blockDim.x + threadIdx.x;
    if (j >= T) return;
    const size_t r = list[j];
    const float* o = xn + (size_t)r * D;
    const double eps = 1e-5;
    const int cap = (1 << EX) - 1;
    double max_o = -1.0;
    for (int i = 0; i < D; ++i) {
        const double v = (double)fabsf(o[i]);
        if (v > max_o) max_o = v;
    }
    const double t_start = __ddiv_rn((double)(cap / 3), max_o);
    const double t_end = __ddiv_rn((double)(cap + 10), max_o);
    double sqr_den = (double)D * 0.25;
    double num = 0.0;
    auto ht = [&](int e) -> double& { return heap_t[(size_t)e * T + j]; };
    auto hi = [&](int e) -> uint16_t& { return heap_i[(size_t)e * T + j]; };
    auto less = [](double ta, int ia, double tb, int ib) { return ta < tb || (ta == tb && ia < ib); };
    for (int i = 0; i < D; ++i) {
        const double v = (double)fabsf(o[i]);
        const int c = __double2int_rz(__dadd_rn(__dmul_rn(t_start, v), eps));
        cur[(size_t)i * T + j] = (uint8_t)c;
        sqr_den = __dadd_rn(sqr_den, (double)(c * c + c));
        num = __dadd_rn(num, __dmul_rn((double)c + 0.5, v));
        ht(i) = __ddiv_rn((double)(c + 1), v);
        hi(i) = (uint16_t)i;
    }
    // heapify (the pop order of distinct keys does not depend on the layout)
    int size = D;
    auto sift = [&](int e) {
        const double t0 = ht(e);
        const int i0 = hi(e);
        while (true) {
            const int a = 2 * e + 1;
            if (a >= size) break;
            int m = a;
            double tm = ht(a);
            int im = hi(a);
            if (a + 1 < size) {
                const double tb = ht(a + 1);
                const int ib = hi(a + 1);
                if (less(tb, ib, tm, im)) {
                    m = a + 1;
                    tm = tb;
                    im = ib;
                }
            }
            if (!less(tm, im, t0, i0)) break;
            ht(e) = tm;
            hi(e) = (uint16_t)im;
            e = m;
        }
        ht(e) = t0;
        hi(e) = (uint16_t)i0;
    };
    for (int e = size / 2 - 1; e >= 0; --e) sift(e);
    double max_ip = 0.0, t = 0.0;
    while (size > 0) {
        const double cur_t = ht(0);
        const int id = hi(0);
        const int c = (int)cur[(size_t)id * T + j] + 1;
        cur[(size_t)id * T + j] = (uint8_t)c;
        const double v = (double)fabsf(o[id]);
        sqr_den = __dadd_rn(sqr_den, (double)(2 * c));
        num = __dadd_rn(num, v);
        const double ip = __ddiv_rn(num, __dsqrt_rn(sqr_den));
        if (ip > max_ip) {
            max_ip = ip;
            t = cur_t;
        }
        bool again = false;
        double tn = 0.0;
        if (c < cap) {
            tn = __ddiv_rn((double)(c + 1), v);
            again = tn < t_end;
        }
        if (again) {  // pop then push = the new entry at the root, sifted down
            ht(0) = tn;
            hi(0) = (uint16_t)id;
        } else {
            --size;
            if (size == 0) break;
            ht(0) = ht(size);
            hi(0) = hi(size);
        }
        sift(0);
    }
    double num2 = 0.0;
    uint8_t* out = code + (size_t)r * D;
    for (int i = 0; i < D; ++i) {
        const double v = (double)fabsf(o[i]);
        int b = __double2int_rz(__dadd_rn(__dmul_rn(t, v), eps));
        if (b >= (1 << EX)) b = cap;
        num2 = __dadd_rn(num2, __dmul_rn((double)b + 0.5, v));
        out[i] = (uint8_t)b;
    }
    float ipn = __double2float_rn(__ddiv_rn(1.0, num2));
    if (!isfinite(ipn)) ipn = 1.f;
    ipnorm[r] = ipn;
}

// The same sweep, a block per vector.
//
// fast_quantize visits the critical factors t = c / |o_i| of all dims in
// ascending (t, i), adds |o_i| to a numerator and 2c to a squared denominator
// at each, and keeps the t of the first largest quotient num / sqrt(den).  The
// block takes the factors in windows of ascending t, each bounded so that its
// factors fit shared memory (a dim has at most w |o_i| + 1 of them in a window
// of width w); a window is sorted by a counting sort over uniform bins of t and
// a rank inside each bin, then the running sums are a block-wide scan and every
// quotient is taken in parallel.
//
// The running numerator is a double and rounds in the reference's order.  Its
// terms are multiples of 2^(lsb-1), lsb the last bit of the smallest non-zero
// |o_i|: while it stays below 2^(52+lsb) no addition rounds and any order gives
// the same doubles (and a sum in any order that ends below it was exact).  Past
// that one thread adds in order.  The denominators are integers.  Vectors
// without a finite positive largest |o_i|, or with more factors in a window than
// fit, go to `slow` for the serial kernel.
//
// What bounds it: instructions issued (some 1700 per warp and window: counting,
// sorting, scanning), 8 warps a block and 4 blocks an SM hiding each other's
// barriers (4 warps a block: 12.0 ms below).  The divisions are two products
// and four fused steps, the square roots only one per thread and window.
// 20,000 vectors of 768 dims, EX = 7: 168.3 -> 7.0 ms (the serial kernel's heap
// steps are chains of some 20 dependent global loads, 20,000 threads in all).
constexpr int kFqThreads = 256;
template <int CAP>
struct FqShared {
    double t[CAP];
    union {
        struct {
            uint32_t bin[CAP];      // counts, then first places
            uint16_t arrival[CAP];  // of a factor within its bin
            uint16_t binned[CAP];   // factors by bin
        } s;
        double num[CAP];            // terms, then running sums, in sorted order
    } u;
    uint32_t item[CAP];             // dim | count << 16
    uint16_t sorted[CAP];
    double red[kFqThreads / 32], red2[kFqThreads / 32];
    uint32_t scan[kFqThreads / 32], at[kFqThreads / 32];
    double num, best, best_t;
    uint32_t den;
    int n;
};
template <int CAP>
__host__ __device__ constexpr size_t fq_smem_bytes(int D) {
    return sizeof(FqShared<CAP>) + (size_t)D * (8 + 4 + 2);
}
// CAP - D - 64 bounds a window's factors beyond one per dim
__host__ __device__ constexpr int fq_cap(int D) { return D <= 1024 ? 2048 : 4096; }

// Exclusive prefix of v over the block and its total; two barriers.
template <typename T>
__device__ __forceinline__ T fq_scan(T v, T* red, T* total) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    T incl = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const T x = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += x;
    }
    if (lane == 31) red[warp] = incl;
    __syncthreads();
    T before = 0, all = 0;
#pragma unroll
    for (int w = 0; w < kFqThreads / 32; ++w) {
        if (w < warp) before += red[w];
        all += red[w];
    }
    __syncthreads();
    *total = all;
    return before + incl - v;
}

// c / x correctly rounded from y = 1 / x correctly rounded, two corrected
// steps (Markstein, IBM J. Res. Dev. 34(1), 1990); x a float, so nothing here
// under- or overflows; c / 0 = infinity.
__device__ __forceinline__ double fq_quotient(int c, double x, double y) {
    const double a = (double)c;
    double q = __dmul_rn(a, y);
    if (x > 0.0) {
        q = __fma_rn(__fma_rn(-x, q, a), y, q);
        q = __fma_rn(__fma_rn(-x, q, a), y, q);
    }
    return q;
}

template <int CAP>
__global__ void __launch_bounds__(kFqThreads) fast_quantize_kernel(const float* __restrict__ xn, int D,
                                                                   int EX, uint8_t* __restrict__ code,
                                                                   float* __restrict__ ipnorm,
                                                                   uint32_t* __restrict__ slow,
                                                                   uint32_t* __restrict__ slow_n) {
    extern __shared__ __align__(16) uint8_t smem_raw[];
    FqShared<CAP>& sh = *reinterpret_cast<FqShared<CAP>*>(smem_raw);
    double* inv = reinterpret_cast<double*>(smem_raw + sizeof(FqShared<CAP>));  // 1 / |o_i|
    float* v = reinterpret_cast<float*>(inv + D);
    uint16_t* cn = reinterpret_cast<uint16_t*>(v + D);  // count at the next factor of a dim, 0: none left
    const int r = blockIdx.x, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const float* o = xn + (size_t)r * D;
    const double eps = 1e-5;
    const int cap = (1 << EX) - 1;
    // largest, smallest non-zero, sum
    float mx = 0.f, mn = INFINITY;
    double sum = 0.0;
    bool finite = true;
    for (int i = tid; i < D; i += kFqThreads) {
        const float x = fabsf(o[i]);
        v[i] = x;
        finite = finite && x < INFINITY;  // false for NaN
        mx = fmaxf(mx, x);
        if (x > 0.f) mn = fminf(mn, x);
        sum += (double)x;
    }
    mx = __uint_as_float(__reduce_max_sync(0xffffffffu, __float_as_uint(mx)));
    mn = __uint_as_float(__reduce_min_sync(0xffffffffu, __float_as_uint(mn)));
#pragma unroll
    for (int s = 16; s > 0; s >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, s);
    if (lane == 0) {
        sh.red[warp] = sum;
        sh.scan[warp] = __float_as_uint(mx);
        sh.at[warp] = __float_as_uint(mn);
    }
    if (tid == 0) {
        sh.n = 0;
        sh.best = 0.0;
        sh.best_t = 0.0;
    }
    finite = __syncthreads_and(finite);
    sum = 0.0;
#pragma unroll
    for (int w = 0; w < kFqThreads / 32; ++w) {
        sum += sh.red[w];
        mx = fmaxf(mx, __uint_as_float(sh.scan[w]));
        mn = fminf(mn, __uint_as_float(sh.at[w]));
    }
    const double t_start = __ddiv_rn((double)(cap / 3), (double)mx);
    const double t_end = __ddiv_rn((double)(cap + 10), (double)mx);
    if (!finite || !(mx > 0.f) || !(t_end < 1e300)) {  // uniform
        if (tid == 0) slow[atomicAdd(slow_n, 1u)] = (uint32_t)r;
        return;
    }
    const int lsb = max((int)(__float_as_uint(mn) >> 23), 1) - 127 - 23;
    const double limit = __longlong_as_double((long long)(52 + lsb + 1023) << 52);  // sums below are exact
    __syncthreads();  // red, scan and at are reused
    // the state at t_start
    double num0 = 0.0;
    uint32_t den0 = 0;
    for (int i = tid; i < D; i += kFqThreads) {
        const double x = (double)v[i];
        const int c = __double2int_rz(__dadd_rn(__dmul_rn(t_start, x), eps));
        const double term = __dmul_rn((double)c + 0.5, x);
        num0 = __dadd_rn(num0, term);
        sh.u.num[i] = term;
        den0 += (uint32_t)(c * c + c);
        inv[i] = __drcp_rn(x);
        cn[i] = (uint16_t)(c + 1);
    }
    {
        double all = 0.0;
        uint32_t alld = 0;
        fq_scan<double>(num0, sh.red, &all);
        fq_scan<uint32_t>(den0, sh.scan, &alld);
        if (tid == 0) {
            if (!(all < limit)) {
                all = 0.0;
                for (int i = 0; i < D; ++i) all = __dadd_rn(all, sh.u.num[i]);
            }
            sh.num = all;
            sh.den = alld + (uint32_t)(D / 4);
        }
    }
    const double width = (double)(CAP - D - 64) / sum;
    double lo = t_start;
    for (bool tail = false;;) {
        const double hi = tail ? INFINITY : fmin(lo + width, t_end);
        const double scale = (double)CAP / width;
        // the bin of a factor (non-decreasing in t); past t_end, 32 per octave
        const auto bin_of = [&](double t) -> int {
            if (tail) {
                const long long d = (__double_as_longlong(t) - __double_as_longlong(t_end)) >> 47;
                return (int)(d < 0 ? 0 : (d < CAP ? d : CAP - 1));
            }
            const int b = __double2int_rz((t - lo) * scale);
            return b < 0 ? 0 : (b < CAP ? b : CAP - 1);
        };
        __syncthreads();  // the window before has been read
        for (int b = tid; b < CAP; b += kFqThreads) sh.u.s.bin[b] = 0u;
        __syncthreads();
        // this window's factors: counted by dim, listed, then placed one by one
        for (int i0 = 0; i0 < D; i0 += kFqThreads) {
            const int i = i0 + tid, c0 = i < D ? cn[i] : 0;
            int m = 0;
            if (c0 > 0) {
                const double x = (double)v[i], y = inv[i];
                if (tail) {
                    m = 1;
                } else {
                    int last = min(__double2int_rz(hi * x) + 1, cap);
                    while (last >= c0 && !(fq_quotient(last, x, y) < hi)) --last;
                    m = max(last + 1 - c0, 0);
                    if (m > 0) cn[i] = last < cap && fq_quotient(last + 1, x, y) < t_end ? last + 1 : 0;
                }
            }
            int incl = m;
#pragma unroll
            for (int s = 1; s < 32; s <<= 1) {
                const int x = __shfl_up_sync(0xffffffffu, incl, s);
                if (lane >= s) incl += x;
            }
            int at = 0;
            if (lane == 31 && incl > 0) at = atomicAdd(&sh.n, incl);
            at = __shfl_sync(0xffffffffu, at, 31) + incl - m;
            for (int j = 0; j < m && at + j < CAP; ++j)
                sh.item[at + j] = (uint32_t)i | ((uint32_t)(c0 + j) << 16);
        }
        __syncthreads();
        const int n = sh.n;
        if (n > CAP) {  // uniform
            if (tid == 0) slow[atomicAdd(slow_n, 1u)] = (uint32_t)r;
            return;
        }
        for (int e = tid; e < n; e += kFqThreads) {
            const uint32_t it = sh.item[e], i = it & 0xffffu;
            const double t = fq_quotient((int)(it >> 16), (double)v[i], inv[i]);
            sh.t[e] = t;
            sh.u.s.arrival[e] = (uint16_t)atomicAdd(&sh.u.s.bin[bin_of(t)], 1u);
        }
        __syncthreads();
        // first places of the bins
        {
            constexpr int PER = CAP / kFqThreads / 4;
            uint4* mine = reinterpret_cast<uint4*>(sh.u.s.bin) + tid * PER;
            uint4 c[PER];
            uint32_t own = 0, all = 0;
#pragma unroll
            for (int b = 0; b < PER; ++b) {
                c[b] = mine[b];
                own += c[b].x + c[b].y + c[b].z + c[b].w;
            }
            uint32_t run = fq_scan<uint32_t>(own, sh.scan, &all);
#pragma unroll
            for (int b = 0; b < PER; ++b) {
                uint4 f;
                f.x = run;
                f.y = f.x + c[b].x;
                f.z = f.y + c[b].y;
                f.w = f.z + c[b].z;
                run = f.w + c[b].w;
                mine[b] = f;
            }
        }
        __syncthreads();
        for (int e = tid; e < n; e += kFqThreads)
            sh.u.s.binned[sh.u.s.bin[bin_of(sh.t[e])] + sh.u.s.arrival[e]] = (uint16_t)e;
        __syncthreads();
        // a factor's rank within its bin, by (t, dim)
        for (int e = tid; e < n; e += kFqThreads) {
            const double t = sh.t[e];
            const int b = bin_of(t);
            const uint32_t first = sh.u.s.bin[b], last = b + 1 < CAP ? sh.u.s.bin[b + 1] : (uint32_t)n;
            const uint32_t dim = sh.item[e] & 0xffffu;
            uint32_t at = first;
            for (uint32_t k = first; k < last; ++k) {
                const int f = sh.u.s.binned[k];
                at += sh.t[f] < t || (sh.t[f] == t && (sh.item[f] & 0xffffu) < dim);
            }
            sh.sorted[at] = (uint16_t)e;
        }
        __syncthreads();
        // running sums and quotients, each thread a stretch of the sequence
        const int per = (n + kFqThreads - 1) / kFqThreads;
        const int k0 = min(n, tid * per), k1 = min(n, k0 + per);
        double own = 0.0;
        uint32_t ownd = 0;
        for (int k = k0; k < k1; ++k) {
            const uint32_t it = sh.item[sh.sorted[k]];
            const double x = (double)v[it & 0xffffu];
            sh.u.num[k] = x;
            own = __dadd_rn(own, x);
            ownd += 2u * (it >> 16);
        }
        double all = 0.0;
        uint32_t alld = 0;
        double num = fq_scan<double>(own, sh.red, &all);
        uint32_t den = fq_scan<uint32_t>(ownd, sh.scan, &alld) + sh.den;
        num = __dadd_rn(num, sh.num);
        all = __dadd_rn(all, sh.num);
        const bool exact = all < limit;
        if (!exact) {  // uniform: in order, by one thread
            if (tid == 0) {
                double x = sh.num;
#pragma unroll 4
                for (int k = 0; k < n; ++k) {
                    x = __dadd_rn(x, sh.u.num[k]);
                    sh.u.num[k] = x;
                }
                all = x;
            }
            __syncthreads();
        }
        // The squared quotients compared by their cross products: where those
        // differ by 1e-14, some 20 times what the rounded quotient can be off,
        // the rounded quotients are in the same order.
        double bnum = 0.0, bden = 1.0;
        int best_k = -1;
        for (int k = k0; k < k1; ++k) {
            num = exact ? __dadd_rn(num, sh.u.num[k]) : sh.u.num[k];
            den += 2u * (sh.item[sh.sorted[k]] >> 16);
            const double a = num * num * bden, b = bnum * bnum * (double)den;
            bool more = a > b;
            if (fabs(a - b) <= 1e-14 * b)
                more = __ddiv_rn(num, __dsqrt_rn((double)den)) > __ddiv_rn(bnum, __dsqrt_rn(bden));
            if (more) {
                bnum = num;
                bden = (double)den;
                best_k = k;
            }
        }
        double best = best_k < 0 ? -1.0 : __ddiv_rn(bnum, __dsqrt_rn(bden));
        // the first largest quotient of the window
#pragma unroll
        for (int s = 16; s > 0; s >>= 1) {
            const double ob = __shfl_xor_sync(0xffffffffu, best, s);
            const int ok = __shfl_xor_sync(0xffffffffu, best_k, s);
            if (ob > best || (ob == best && ok < best_k)) {
                best = ob;
                best_k = ok;
            }
        }
        if (lane == 0) {
            sh.red2[warp] = best;
            sh.at[warp] = (uint32_t)best_k;
        }
        __syncthreads();  // sh.num and sh.den have been read
        if (tid == 0) {
#pragma unroll
            for (int w = 0; w < kFqThreads / 32; ++w)  // the warps' stretches are in order
                if (sh.red2[w] > sh.best) {
                    sh.best = sh.red2[w];
                    sh.best_t = sh.t[sh.sorted[sh.at[w]]];
                }
            sh.num = all;
            sh.den += alld;
            sh.n = 0;
        }
        if (tail) break;
        tail = hi >= t_end;
        lo = hi;
    }
    __syncthreads();
    // the codes at the best factor, and 1 / sum (code + 0.5) |o|
    const double t = sh.best_t;
    uint8_t* out = code + (size_t)r * D;
    double own = 0.0, all = 0.0;
    for (int i = tid; i < D; i += kFqThreads) {
        const double x = (double)v[i];
        int b = __double2int_rz(__dadd_rn(__dmul_rn(t, x), eps));
        if (b >= (1 << EX)) b = cap;
        const double term = __dmul_rn((double)b + 0.5, x);
        own = __dadd_rn(own, term);
        sh.u.num[i] = term;
        out[i] = (uint8_t)b;
    }
    fq_scan<double>(own, sh.red, &all);
    if (tid == 0) {
        if (!(all < limit)) {
            all = 0.0;
            for (int i = 0; i < D; ++i) all = __dadd_rn(all, sh.u.num[i]);
        }
        float ipn = __double2float_rn(__ddiv_rn(1.0, all));
        if (!isfinite(ipn)) ipn = 1.f;
        ipnorm[r] = ipn;
    }
}

// Per row: codes flipped where the sign bit is 0, compacted to D*EX/8 bytes
// (store_compacted_code), xipnorm = (ipnorm * 2) * onorm.  One thread per
// (row, 64-dim group).
__global__ void build_long_kernel(const uint8_t* __restrict__ code, const uint64_t* __restrict__ bits,
                                  const float* __restrict__ ipnorm, const float* __restrict__ onorm,
                                  int rows, int D, int EX, uint8_t* __restrict__ lng,
                                  float* __restrict__ xipnorm) {
    const int G = D / 64;
    const size_t t = blockIdx.x * (size_t)blockDim.x + threadIdx.x;
    if (t >= (size_t)rows * G) return;
    const int r = (int)(t / G), g = (int)(t - (size_t)r * G);
    const uint8_t mask = (uint8_t)((1 << EX) - 1);
    const uint64_t sb = bits[(size_t)r * G + g];
    uint8_t v[64];
    for (int i = 0; i < 64; ++i) {
        const uint8_t c = code[(size_t)r * D + 64 * g + i];
        v[i] = ((sb >> i) & 1) ? c : (uint8_t)(~c & mask);
    }
    const size_t row_bytes = (size_t)D * EX / 8;
    uint8_t* o = lng + (size_t)r * row_bytes + (size_t)g * 8 * EX;
    if (EX == 8) {
        for (int i = 0; i < 64; ++i) o[i] = v[i];
    } else if (EX == 4) {
        for (int h = 0; h < 2; ++h)
            for (int i = 0; i < 16; ++i) o[16 * h + i] = v[32 * h + i] | (uint8_t)(v[32 * h + 16 + i] << 4);
    } else if (EX == 2 || EX == 3) {
        for (int i = 0; i < 16; ++i)
            o[i] = (v[i] & 3) | ((v[16 + i] & 3) << 2) | ((v[32 + i] & 3) << 4) | ((v[48 + i] & 3) << 6);
        if (EX == 3)  // top byte m, bit j = bit 2 of dim 8j + m
            for (int m = 0; m < 8; ++m) {
                uint8_t b = 0;
                for (int jj = 0; jj < 8; ++jj) b |= (uint8_t)(((v[8 * jj + m] >> 2) & 1) << jj);
                o[16 + m] = b;
            }
    } else {  // 6 or 7
        const uint8_t lo = EX == 7 ? 0x3F : 0xFF;
        for (int i = 0; i < 16; ++i) {
            o[i] = (v[i] & lo) | (uint8_t)((v[32 + i] << 2) & 0xC0);
            o[16 + i] = (v[16 + i] & lo) | (uint8_t)((v[48 + i] << 2) & 0xC0);
            o[32 + i] = (v[32 + i] & 0x0F) | (uint8_t)((v[48 + i] & 0x0F) << 4);
        }
        if (EX == 7)  // top byte m, bit j = bit 6 of dim 8j + m
            for (int m = 0; m < 8; ++m) {
                uint8_t b = 0;
                for (int jj = 0; jj < 8; ++jj) b |= (uint8_t)(((v[8 * jj + m] >> 6) & 1) << jj);
                o[48 + m] = b;
            }
    }
    if (g == 0) xipnorm[r] = __fmul_rn(__fmul_rn(ipnorm[r], 2.f), onorm[r]);
}

// FastScan blocks: block b covers rows [vfirst[b], vfirst[b] + vnum[b]) (at
// most 32, zero codes past the end).  Group q (dims 4q..4q+3) is 16 bytes;
// byte j holds vector perm0[j]'s nibble low and vector perm0[j] + 16's high,
// perm0 = {0, 8, 1, 9, ..., 7, 15}, nibble bit 3 = dim 4q.  Then 32 floats of
// ||o - c||.  One thread per output byte of the code part.
__global__ void build_short_kernel(const uint64_t* __restrict__ bits, const float* __restrict__ onorm,
                                   const uint32_t* __restrict__ vfirst, const uint32_t* __restrict__ vnum,
                                   uint64_t nblocks, int D, uint8_t* __restrict__ shrt) {
    const uint64_t code_bytes = 4ull * D, bb = code_bytes + 128;
    const uint64_t total = nblocks * bb;
    const int G = D / 64;
    for (uint64_t t = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; t < total;
         t += (uint64_t)gridDim.x * blockDim.x) {
        const uint64_t b = t / bb;
        const uint32_t rem = (uint32_t)(t - b * bb);
        const uint32_t nv = vnum[b], f = vfirst[b];
        if (rem < code_bytes) {
            const uint32_t q = rem >> 4, jb = rem & 15;
            const uint32_t pv = (jb & 1) ? 8 + (jb >> 1) : (jb >> 1);
            uint8_t byte = 0;
            for (int h = 0; h < 2; ++h) {
                const uint32_t v = pv + 16 * h;
                if (v >= nv) continue;
                const uint64_t w = bits[(size_t)(f + v) * G + (4 * q) / 64];
                const uint32_t s = (4 * q) & 63;
                const uint32_t nib = (uint32_t)(((w >> s) & 1) << 3 | ((w >> (s + 1)) & 1) << 2 |
                                                ((w >> (s + 2)) & 1) << 1 | ((w >> (s + 3)) & 1));
                byte |= (uint8_t)(nib << (4 * h));
            }
            shrt[t] = byte;
        } else {
            const uint32_t v = (rem - (uint32_t)code_bytes) >> 2, by = (rem - (uint32_t)code_bytes) & 3;
            const float fv = v < nv ? onorm[f + v] : 0.f;
            shrt[t] = (uint8_t)(__float_as_uint(fv) >> (8 * by));
        }
    }
}

}  // namespace erq
