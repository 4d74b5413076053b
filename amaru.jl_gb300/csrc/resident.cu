// Block-Jacobi PCG of a small model, or of the parts of a batch, with the matrix kept in shared memory.
//
// A part (a contiguous range of nodes that no element leaves; a small model is one part) is solved by a cluster of
// 1 to 16 CTAs in one launch: solve_system! (src/solver.jl:5-79) by the mixed-precision method of solver.cu, FP32 PCG
// with FP64 true-residual refreshes.  CTA r owns a contiguous slice of the rows, of about equal numbers of blocks (so
// that nodes no element uses change nothing).  Its blocks of K32, with 16-bit
// column offsets, stay in its shared memory over all iterations, beside the direction p over the slice's column
// window; x, r, q and the block inverses of its rows are in registers.
//
// The matrix product is bound by shared-memory wavefronts.  Its rows are sorted by their number of blocks and laid out
// lane by lane (one thread per row, or 2 or 4 where the rows are few): 32 blocks then take 7 wavefronts in 2-D, 4 of
// them the values, without conflicts or shuffles.  8 lanes per row over the rows' own layout took 4.9 times as long
// (9 430 cycles for 586 rows and 8 568 blocks).
//
// Two forms.  For a model alone (Exact) the operations are those of solve_mixed's launch-per-step kernels in solver.cu,
// in the same order: the eight partial sums of a row and their tree, the rows' products by warps and CTAs of 32, 64
// and 256 rows, the refresh's FP64 sums over CTAs.  Only an iteration's sums over CTAs are not FP64 numbers; what they
// give, alpha and beta, is the nearest FP32 number to the quotient of the exact sums, which FP64 sums miss once in some
// hundred million.  So which form a model's size selects shows in its time and hardly ever in a bit of its result.  For a
// batch's parts, which other CTAs summed anyway, the order is free: one sum per row, one per thread, a warp's in FP32.
//
// What else bounds it is the chain of an iteration, two cluster-wide sums (p.q, then r.z and r.r).  So:
//   * the direction needs no sum of its own: a CTA pushes the z of its rows into the windows of the CTAs that read them,
//     and after the second sum each forms p = z + beta p over its whole window;
//   * what a CTA sends, its partial sums and its z, goes by st.async into the others' shared memory and is counted by
//     their mbarriers, so a sum is one way across the cluster, with no fence; every CTA adds the cluster's partials
//     itself.  As each CTA waits for all, a sum is a barrier of the cluster: the slots and windows are never written
//     while they may be read;
//   * nothing in an iteration takes the FP64 pipe (two lanes a clock per SM; FP64 trees and quotients took as long as the
//     rest of an iteration): the partials, FP32 as in solver.cu, are added as pairs of FP32 numbers, and in the few cases
//     where 48 bits do not settle alpha's or beta's rounding again as integers (in all cases: batch below 63 ms).
// Measured, three launches per iteration over all SMs before: 26 us an iteration, now 3.2 us with Exact
// (1 613 QUAD8 nodes, 8 CTAs); a batch of 64 QUAD8 models of 10 to 60 cells a side 230 ms, now 49 ms.
#include <algorithm>
#include <climits>
#include <cmath>
#include <mutex>
#include <type_traits>

#include <cooperative_groups.h>

#include "amr_internal.h"

namespace cg = cooperative_groups;

namespace {

constexpr int kT = 512;             // threads of a CTA
constexpr int kW = kT / 32;
constexpr int kRowsPerThread = 2;   // rows a thread keeps in registers
constexpr int kMaxC = 16;           // CTAs of a cluster at most (above 8 where the device allows it)
constexpr size_t kMaxDyn = 221 * 1024, kMaxDynExact = 206 * 1024;  // beside the sums' slots (Exact: and the rows' values)
constexpr int kMaxGroups = kMaxC * kT * kRowsPerThread / 32;        // groups of 32 rows of a part

struct Args {
    const int64_t *slices, *first;   // the parts' slice bounds, and where a part's begin (null: 0)
    const uint16_t *perm;            // per node: at n0 + i the i-th row of its slice by descending length, as n - n0
    const int64_t *list;             // the launch's parts, a cluster each (null: part 0)
    const uint8_t *active;           // null: every part
    int64_t nb;
    const int64_t *rp;
    const int32_t *cj;
    const float *K32;
    const double *K64;
    const float *Minv;
    const uint8_t *fm;
    const double *b;
    double *x, *reac;
    double *rows64;                  // Exact: 2 x nnodes, r.r and r.z of each row at a refresh
    int64_t nnodes;
    AmrPartStat *stat;
    unsigned long long *t0, *t1;     // null: no timing
    double tol2;
    int max_iters, force_every;
    int kcap, wcap;                  // slots of blocks and window nodes of a slice at most
    unsigned long long wait_ns;      // a wait for a sum gives up after this time
    int withhold;                    // tests: the rank that never sends its part of p.q, and every rank reports its status
                                     // at stat[rank] (-1: none)
};
constexpr unsigned long long kWaitNs = 2000000000ull;  // a sum takes microseconds

// Sums over the cluster and their quotients alpha and beta, which an iteration takes rounded to FP32.  Added as pairs
// hi + lo of FP32 numbers (48 bits), they give that FP32 number in all but a few of a thousand cases: where the
// quotient is not within 2^-34 of the middle between two.  There, and outside of 2^-100 to 2^100 after a scaling by the
// last refresh's, the sums are taken again as integers and divided exactly.  So alpha and beta are the nearest FP32
// numbers, as with FP64 sums.
struct Pair {
    float h, l;
};
__device__ __forceinline__ Pair pair_add(Pair a, Pair b) {
    const float s = __fadd_rn(a.h, b.h);
    const float t = __fsub_rn(s, a.h);
    const float e = __fadd_rn(__fsub_rn(a.h, __fsub_rn(s, t)), __fsub_rn(b.h, t));
    const float l = __fadd_rn(__fadd_rn(a.l, b.l), e);
    const float h = __fadd_rn(s, l);
    return Pair{h, __fsub_rn(l, __fsub_rn(h, s))};
}
__device__ __forceinline__ Pair pair(double v) {
    const float h = (float)v;
    return Pair{h, (float)(v - (double)h)};
}
// a power of two near 1 / v
__device__ __forceinline__ float scale_of(double v) {
    return __int_as_float((127 + max(-120, min(120, 1023 - ((int)(__double_as_longlong(v) >> 52) & 0x7ff)))) << 23);
}
__device__ __forceinline__ bool in_range(float v) { return v > 0x1p-100f && v < 0x1p100f; }  // (false with NaN)
// a / b rounded to FP32; sure: it is the nearest to the sums' quotient
__device__ __forceinline__ float pair_div(Pair a, Pair b, bool &sure) {
    const float q = __fdiv_rn(a.h, b.h);
    const float r = __fadd_rn(__fmaf_rn(-q, b.h, a.h), __fmaf_rn(-q, b.l, a.l));
    const float c = __fdiv_rn(r, b.h), d = q * 0x1p-34f;
    sure = in_range(a.h) && in_range(b.h) && in_range(q) &&
           __fadd_rn(q, __fadd_rn(c, d)) == __fadd_rn(q, __fsub_rn(c, d));
    return __fadd_rn(q, c);
}
// the sum of get(0 .. n - 1), n <= 512, the same in every lane
template <int K, class F>
__device__ __forceinline__ Pair pair_sum(F get) {
    Pair p[K];
#pragma unroll
    for (int i = 0; i < K; i++) p[i] = Pair{get(32 * i + (int)(threadIdx.x & 31)), 0.0f};
#pragma unroll
    for (int o = K / 2; o > 0; o >>= 1)
#pragma unroll
        for (int i = 0; i < o; i++) p[i] = pair_add(p[i], p[i + o]);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1)
        p[0] = pair_add(p[0], Pair{__shfl_xor_sync(0xffffffffu, p[0].h, o), __shfl_xor_sync(0xffffffffu, p[0].l, o)});
    return p[0];
}
template <class F>
__device__ __forceinline__ Pair pair_sum(int n, F get) {
    if (n <= 32) return pair_sum<1>(get);
    if (n <= 64) return pair_sum<2>(get);
    if (n <= 128) return pair_sum<4>(get);
    if (n <= 256) return pair_sum<8>(get);
    return pair_sum<16>(get);
}

// A number (neg ? -1 : 1) m 2^e, the top bit of m set; m = 0: zero, or with e = kNoNumber NaN
struct Num {
    unsigned long long m;
    int e;
    bool neg;
};
constexpr int kNoNumber = INT_MIN, kInfinite = 1 << 20;
__device__ __forceinline__ Num number(double v) {
    const unsigned long long b = (unsigned long long)__double_as_longlong(v);
    const int ex = (int)(b >> 52 & 0x7ff);
    unsigned long long m = b & 0xfffffffffffffULL;
    const bool neg = b >> 63;
    if (ex == 0x7ff) return m ? Num{0, kNoNumber, false} : Num{1ULL << 63, kInfinite, neg};
    if (ex > 0) m |= 1ULL << 52;
    if (m == 0) return Num{0, 0, false};
    const int up = __clzll((long long)m);
    return Num{m << up, max(ex, 1) - 1075 - up, neg};
}
// a > b of numbers that are not negative (false with NaN)
__device__ __forceinline__ bool greater(const Num &a, const Num &b) {
    if (a.m == 0 || a.neg) return false;
    if (b.m == 0) return b.e != kNoNumber;
    return a.e != b.e ? a.e > b.e : a.m > b.m;
}
// the leading 24 bits as a float in [1, 2)
__device__ __forceinline__ float leading(const Num &a) { return __int_as_float(0x3f800000 | ((int)(a.m >> 40) & 0x7fffff)); }
// a / b rounded to FP32: a quotient of the leading bits, corrected by its exact remainder (long division)
__device__ __noinline__ float quotient(Num a, Num b) {
    if (a.m == 0 || b.m == 0) return a.m == 0 && a.e != kNoNumber && b.m != 0 ? 0.0f : __int_as_float(0x7fc00000);
    // a.m 2^up / b.m has 24 bits, or those of a denormal
    const int up = min(a.m >= b.m ? 23 : 24, a.e - b.e + 149);
    if (up < 0) return 0.0f;
    const unsigned long long n = a.m >> 4, d = b.m >> 4;  // 60 bits, so that remainders of some d fit 64
    int q = __float2int_rn(__fdiv_rn(leading(a), leading(b)) * (float)(1 << up));
    long long r = (long long)((n << up) - (unsigned long long)q * d);  // |r| < 4 d, exact modulo 2^64
    const int k = __float2int_rn(__fdiv_rn((float)(int)(r >> 32), (float)(int)(d >> 32)));
    q += k;
    r -= (long long)k * (long long)d;
    if (2 * r > (long long)d) q++;
    if (2 * r < -(long long)d) q--;
    const float v = ldexpf((float)q, a.e - b.e - up);
    return a.neg != b.neg ? -v : v;
}
// The sum of v[0 .. n), n <= 512, the same in every lane: as integers of a unit 2^-52 of the largest value's exponent, in
// which FP32 values down to 2^-29 of it are exact.  eights: the values of eight neighbours are added first, in FP32.
__device__ __noinline__ Num exact_sum(const float *v, int n, bool eights) {
    constexpr int kUp = 29;
    const int lane = threadIdx.x & 31;
    auto get = [&](int i) {
        float t = i + lane < n ? v[i + lane] : 0.0f;
        if (eights) {
            t += __shfl_xor_sync(0xffffffffu, t, 4);
            t += __shfl_xor_sync(0xffffffffu, t, 2);
            t += __shfl_xor_sync(0xffffffffu, t, 1);
            if (lane & 7) t = 0.0f;
        }
        return t;
    };
    int top = 1;
    for (int i = 0; i < n; i += 32) top = max(top, __float_as_int(get(i)) >> 23 & 0xff);
    top = (int)__reduce_max_sync(0xffffffffu, (unsigned)top);
    if (top == 255) {  // infinite or NaN
        float f = 0.0f;
        for (int i = 0; i < n; i += 32) f += get(i);
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) f += __shfl_xor_sync(0xffffffffu, f, o);
        return number((double)f);
    }
    long long s = 0;  // |s| < 16 2^53 in a lane, 2^62 in all
    for (int i = 0; i < n; i += 32) {
        const int b = __float_as_int(get(i)), ex = b >> 23 & 0xff;
        const unsigned long long m = (unsigned long long)((b & 0x7fffff) | (ex ? 0x800000 : 0)) << kUp;
        const int down = top - max(ex, 1);  // rounded where bits go
        const unsigned long long w = down > 53 ? 0 : (m + (down > kUp ? 1ULL << (down - 1) : 0)) >> down;
        s += b < 0 ? -(long long)w : (long long)w;
    }
    // three parts whose sums over the lanes fit 32 bits
    const unsigned p0 = __reduce_add_sync(0xffffffffu, (unsigned)(s & 0x3ffffff)),
                   p1 = __reduce_add_sync(0xffffffffu, (unsigned)(s >> 26 & 0x3ffffff));
    const int p2 = __reduce_add_sync(0xffffffffu, (int)(s >> 52));
    s = ((long long)p2 << 52) + ((long long)p1 << 26) + (long long)p0;
    if (s == 0) return Num{0, 0, false};
    const unsigned long long m = s < 0 ? 0ULL - (unsigned long long)s : (unsigned long long)s;
    const int up = __clzll((long long)m);
    return Num{m << up, top - 150 - kUp - up, s < 0};
}

template <int B>
size_t slice_bytes(int64_t slots, int64_t rows, int64_t window) {
    (void)rows;
    return (size_t)slots * (B * B * 4 + 2) + (size_t)window * 2 * B * 4;
}
// threads per row of a part whose slices have at most `rows` rows with blocks
__host__ __device__ inline int threads_per_row(int64_t rows) { return rows * 4 <= kT ? 4 : rows * 2 <= kT ? 2 : 1; }

__device__ __forceinline__ unsigned long long global_ns() {
    unsigned long long t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}

__device__ __forceinline__ uint32_t shared_addr(const void *p) { return (uint32_t)__cvta_generic_to_shared(p); }
__device__ __forceinline__ uint32_t cluster_addr(uint32_t local, int r) {  // the same place in rank r's shared memory
    uint32_t remote;
    asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(remote) : "r"(local), "r"(r));
    return remote;
}
// v to a place in a CTA's shared memory, counted by an mbarrier there
__device__ __forceinline__ void store_async(uint32_t to, float v, uint32_t bar) {
    asm volatile("st.async.weak.shared::cluster.mbarrier::complete_tx::bytes.f32 [%0], %1, [%2];" ::"r"(to), "f"(v), "r"(bar)
                 : "memory");
}
__device__ __forceinline__ void store_async4(uint32_t to, float4 v, uint32_t bar) {
    asm volatile("st.async.weak.shared::cluster.mbarrier::complete_tx::bytes.v4.f32 [%0], {%1, %2, %3, %4}, [%5];" ::"r"(to),
                 "f"(v.x), "f"(v.y), "f"(v.z), "f"(v.w), "r"(bar)
                 : "memory");
}
__device__ __forceinline__ void store_async2(uint32_t to, float v, float w, uint32_t bar) {
    asm volatile("st.async.weak.shared::cluster.mbarrier::complete_tx::bytes.v2.f32 [%0], {%1, %2}, [%3];" ::"r"(to), "f"(v),
                 "f"(w), "r"(bar)
                 : "memory");
}
// waits for the phase of an mbarrier to complete; false after `limit` nanoseconds (a try may suspend the thread for a time
// that the device sets, so tries alone would not bound it).  A pause between two looks at the clock counts for 20 ms at
// most: while another process has the GPU, nobody here could have sent anything.
__device__ __forceinline__ bool wait_phase(uint32_t bar, unsigned parity, unsigned long long limit) {
    unsigned long long last = 0, waited = 0;
    for (int i = 0; i < (1 << 28); i++) {
        uint32_t done;
        asm volatile("{\n.reg .pred p;\nmbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n"
                     "selp.u32 %0, 1, 0, p;\n}"
                     : "=r"(done)
                     : "r"(bar), "r"(parity)
                     : "memory");
        if (done) return true;
        if (i % 16 == 15) {
            const unsigned long long now = global_ns();
            if (last) waited += min(now - last, 20000000ull);
            if (waited > limit) break;
            last = now;
        }
    }
    return false;
}

template <int B>
__device__ __forceinline__ void load_node(const float *p, float *v) {
    if constexpr (B == 2) {
        const float2 f = *reinterpret_cast<const float2 *>(p);
        v[0] = f.x;
        v[1] = f.y;
    } else {
#pragma unroll
        for (int d = 0; d < B; d++) v[d] = p[d];
    }
}

// sum of n doubles as solver.cu's grid_sum adds its CTAs' partials: thread j of 256 has partials j, j + 256, .., a
// shuffle tree per warp, then the warps'; levels and warps that would add zeros left out.  One warp; get(i): partial i.
template <class F>
__device__ __forceinline__ double tree_sum(int n, F get) {
    const int lane = threadIdx.x & 31;
    double w[8];
    const int nw = min(8, (n + 31) / 32);
#pragma unroll
    for (int q = 0; q < 8; q++) {
        w[q] = 0.0;
        if (q < nw) {
            double v = 0.0;
            for (int i = 32 * q + lane; i < n; i += 256) v += get(i);
#pragma unroll
            for (int o = 16; o > 0; o >>= 1)
                if (o < n) v += __shfl_xor_sync(0xffffffffu, v, o);
            w[q] = v;
        }
    }
    return nw == 1 ? w[0] : ((w[0] + w[4]) + (w[2] + w[6])) + ((w[1] + w[5]) + (w[3] + w[7]));
}
// One row's product (or this thread's part of it): the thread's share of the eight sums of k_spmv32v's lanes, which take
// four blocks each in turn, then the lanes' tree
template <int B, int S>
__device__ __forceinline__ void exact_row(const float4 *val4, const float *val1, const uint16_t *cols, int kcap, int e,
                                          int chunks, const float *pwin, float *q) {
    constexpr int BB = B * B, A = 8 / S;
    float acc[A][B];
#pragma unroll
    for (int i = 0; i < A; i++)
#pragma unroll
        for (int c = 0; c < B; c++) acc[i][c] = 0.0f;
    for (int t0 = 0; t0 < chunks; t0 += A)
#pragma unroll
        for (int i = 0; i < A; i++) {
            if (t0 + i >= chunks) break;  // (uniform over the warp)
#pragma unroll
            for (int u = 0; u < 4; u++, e += 32) {
                const int j = (int)cols[e] * B;
                float v[BB], pv[B];
#pragma unroll
                for (int w = 0; w < BB / 4; w++) {
                    const float4 f = val4[w * kcap + e];
                    v[4 * w] = f.x; v[4 * w + 1] = f.y; v[4 * w + 2] = f.z; v[4 * w + 3] = f.w;
                }
                if (BB % 4) v[BB - 1] = val1[e];
                load_node<B>(pwin + j, pv);
#pragma unroll
                for (int c = 0; c < B; c++)
#pragma unroll
                    for (int d = B - 1; d >= 0; d--) acc[i][c] = fmaf(v[c * B + d], pv[d], acc[i][c]);
            }
        }
#pragma unroll
    for (int c = 0; c < B; c++) {
        if constexpr (S == 1) {
            q[c] = ((acc[0][c] + acc[4][c]) + (acc[2][c] + acc[6][c])) + ((acc[1][c] + acc[5][c]) + (acc[3][c] + acc[7][c]));
        } else if constexpr (S == 2) {
            const float x = (acc[0][c] + acc[2][c]) + (acc[1][c] + acc[3][c]);
            q[c] = x + __shfl_xor_sync(0xffffffffu, x, 1);
        } else {
            float x = acc[0][c] + acc[1][c];
            x += __shfl_xor_sync(0xffffffffu, x, 2);
            q[c] = x + __shfl_xor_sync(0xffffffffu, x, 1);
        }
    }
}

template <int B, bool Exact>
__global__ void __launch_bounds__(kT, 1) k_resident_pcg(Args a) {
    constexpr int BB = B * B, M = kRowsPerThread;
    constexpr int XR = Exact ? kT * kRowsPerThread : 1;
    __shared__ float s_row[2][XR];                                  // Exact: a value of each row of the slice
    // the cluster's sums of 32 rows, or of warps: p.q, r.r, and r.z of this iteration and the last by turns
    __shared__ __align__(16) float s_warp[2][kW];
    __shared__ __align__(16) float s_grp[4][Exact ? kMaxGroups : kMaxC * kW];
    __shared__ double s_grpd[2][Exact ? kMaxGroups / 2 + 1 : 1];    // Exact: the sums of 64 rows at a refresh
    extern __shared__ __align__(16) float dyn[];  // read as float4
    __shared__ int s_off[M * kW + 1];       // first slot of each 32 rows' (row parts') blocks
    __shared__ double s_slotd[2][kMaxC], s_dwarp[2][kW], s_dtot[2], s_um[kMaxC];
    __shared__ __align__(8) uint64_t s_bar[2];                      // the two sums' arrivals
    __shared__ int s_w0, s_w1, s_win[kMaxC][2], s_bytes, s_abort, s_late, s_stop;
    __shared__ float s_alpha, s_beta;
    cg::cluster_group cl = cg::this_cluster();
    const int C = (int)cl.num_blocks(), rank = (int)cl.block_rank();
    const long long part = a.list ? a.list[blockIdx.x / C] : 0;
    if (a.active && !a.active[part]) return;  // (uniform over the cluster)
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    if (a.t0 && tid == 0) atomicMin(a.t0, global_ns());
    // Another CTA's shared memory may be touched only once that CTA runs: all arrive here and wait before the first remote
    // store below, so that the set-up of the slice hides the wait.
    if (C > 1) asm volatile("barrier.cluster.arrive.release;" ::: "memory");
    auto barrier = [&]() {
        if (C > 1) cl.sync();
        else __syncthreads();
    };

    // ---- the slice: rows [n0, n1), their blocks and the window of their columns
    const int64_t *bound = a.slices + (a.first ? a.first[part] : 0);
    const int64_t n0 = bound[rank], n1 = bound[rank + 1];
    const int R = (int)(n1 - n0);
    const int64_t k0 = a.rp[n0];
    const int nk = (int)(a.rp[n1] - k0);
    float4 *val4 = reinterpret_cast<float4 *>(dyn);           // [BB / 4][kcap]: the blocks' first 4 or 8 values
    float *val1 = dyn + (size_t)(BB / 4) * 4 * a.kcap;        // [kcap] the ninth (3-D)
    float *pwin = val1 + (size_t)(BB % 4) * a.kcap;           // [window][B]
    float *zwin = pwin + (size_t)B * a.wcap;                  // [window][B], own rows and what the others push
    uint16_t *cols = (uint16_t *)(zwin + (size_t)B * a.wcap); // [kcap]
    if (tid == 0) {
        s_w0 = (int)n0;
        s_w1 = (int)n1;
        s_bytes = s_abort = s_late = 0;
        for (int i = 0; i < 2; i++)
            asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(shared_addr(&s_bar[i])), "r"(1) : "memory");
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    __syncthreads();
    {
        int lo = (int)n0, hi = (int)n1;
        for (int k = tid; k < nk; k += kT) {
            const int j = a.cj[k0 + k];
            lo = min(lo, j);
            hi = max(hi, j + 1);
        }
        lo = __reduce_min_sync(0xffffffffu, lo);
        hi = __reduce_max_sync(0xffffffffu, hi);
        if (lane == 0) { atomicMin(&s_w0, lo); atomicMax(&s_w1, hi); }
    }
    __syncthreads();
    const int w0 = s_w0, W = s_w1 - w0, own = (int)n0 - w0;
    // the rows with blocks, sorted: thread tid has the parts sub of the rows at (tid + m kT) / S
    int most = 0, Rn = 0;  // (over the part's slices, so that S belongs to the part)
    for (int r = 0; r < C; r++) {
        const int64_t b0 = bound[r], b1 = bound[r + 1];
        int lo = 0, hi = (int)(b1 - b0);  // rows without blocks are sorted last
        while (lo < hi) {
            const int mid = (lo + hi) >> 1;
            const int64_t n = b0 + a.perm[b0 + mid];
            if (a.rp[n + 1] > a.rp[n]) lo = mid + 1;
            else hi = mid;
        }
        most = max(most, lo);
        if (r == rank) Rn = lo;
    }
    const int S = threads_per_row(most), sub = tid & (S - 1);
    int row[M], width[M];  // row: -1 none
#pragma unroll
    for (int m = 0; m < M; m++) {
        const int i = (tid + m * kT) / S;
        row[m] = i < Rn ? (int)a.perm[n0 + i] : -1;
        int n = row[m] >= 0 ? (int)(a.rp[n0 + row[m] + 1] - a.rp[n0 + row[m]]) : 0;
        if (Exact && n > 0) n = ((int)(a.rp[n0 + row[m]] & 3) + n + 3) / 4;  // runs of four from a multiple of four
        width[m] = __reduce_max_sync(0xffffffffu, (n + S - 1) / S);
        if (lane == 0) s_off[m * kW + warp + 1] = 32 * (Exact ? 4 : 1) * width[m];
    }
    __syncthreads();
    if (tid == 0) {
        s_off[0] = 0;
        for (int i = 0; i < M * kW; i++) s_off[i + 1] += s_off[i];
    }
    __syncthreads();
    int slot0[M];
#pragma unroll
    for (int m = 0; m < M; m++) {
        slot0[m] = s_off[m * kW + warp] + lane;
        const int64_t ks = row[m] >= 0 ? a.rp[n0 + row[m]] : 0, ke = row[m] >= 0 ? a.rp[n0 + row[m] + 1] : 0;
        for (int t = 0; t < width[m] * (Exact ? 4 : 1); t++) {
            const int64_t k = Exact ? (ks & ~int64_t(3)) + 4 * ((t >> 2) * S + sub) + (t & 3) : ks + t * S + sub;
            const bool in = k >= ks && k < ke;
            float v[BB];
#pragma unroll
            for (int q = 0; q < BB; q++) v[q] = in ? a.K32[(int64_t)q * a.nb + k] : 0.0f;
            const int e = slot0[m] + 32 * t;
            cols[e] = in ? (uint16_t)(a.cj[k] - w0) : (uint16_t)own;
#pragma unroll
            for (int q = 0; q < BB / 4; q++)
                val4[q * a.kcap + e] = make_float4(v[4 * q], v[4 * q + 1], v[4 * q + 2], v[4 * q + 3]);
            if (BB % 4) val1[e] = v[BB - 1];
        }
    }
    // the bytes of z the others push here: their rows with blocks in this window
    {
        int got = 0;
        for (int i = tid; i < W; i += kT) {
            const int64_t n = w0 + i;
            if ((n < n0 || n >= n1) && a.rp[n + 1] > a.rp[n]) got += B * 4;
        }
        got = __reduce_add_sync(0xffffffffu, got);
        if (lane == 0) atomicAdd(&s_bytes, got);
    }
    for (int i = tid; i < W * B; i += kT) pwin[i] = zwin[i] = 0.0f;
    if constexpr (Exact)  // (rows without blocks keep their zeros)
        for (int i = tid; i < XR; i += kT) s_row[0][i] = s_row[1][i] = 0.0f;
    if (sub != 0)  // from here on a row's first thread owns it
#pragma unroll
        for (int m = 0; m < M; m++) row[m] = -1;
    float xr[M][B], rv[M][B], mi[M][BB];
#pragma unroll
    for (int m = 0; m < M; m++) {
#pragma unroll
        for (int c = 0; c < B; c++) xr[m][c] = rv[m][c] = 0.0f;
#pragma unroll
        for (int q = 0; q < BB; q++) mi[m][q] = row[m] >= 0 ? a.Minv[(n0 + row[m]) * BB + q] : 0.0f;
    }

    // every CTA's window; the ranks (bits) whose windows hold a row of this thread
    if (C > 1) asm volatile("barrier.cluster.wait.acquire;" ::: "memory");
    if (tid < C) {
        *cl.map_shared_rank(&s_win[rank][0], tid) = w0;
        *cl.map_shared_rank(&s_win[rank][1], tid) = w0 + W;
    }
    barrier();  // (also: every CTA's mbarriers and zero window exist before a neighbour writes there)
    unsigned to[M];
#pragma unroll
    for (int m = 0; m < M; m++) {
        to[m] = 0;
        const int n = (int)n0 + row[m];
        if (row[m] >= 0)
            for (int r = 0; r < C; r++)
                if (r != rank && n >= s_win[r][0] && n < s_win[r][1]) to[m] |= 1u << r;
    }
    // z of this thread's row m into its window and the others'; counted (st.async) by their second mbarrier, or plain
    // stores that a barrier of the cluster follows
    auto push_z = [&](auto counted, int m, const float *z) {
        float *mine = zwin + (own + row[m]) * B;
#pragma unroll
        for (int c = 0; c < B; c++) mine[c] = z[c];
        for (unsigned t = to[m]; t; t &= t - 1) {
            const int r = __ffs(t) - 1;
            const uint32_t z_to = cluster_addr(shared_addr(zwin + ((int)n0 + row[m] - s_win[r][0]) * B), r);
            if constexpr (decltype(counted)::value) {
                const uint32_t bar = cluster_addr(shared_addr(&s_bar[1]), r);
                if constexpr (B == 2) {
                    store_async2(z_to, z[0], z[1], bar);
                } else {
#pragma unroll
                    for (int c = 0; c < B; c++) store_async(z_to + 4 * c, z[c], bar);
                }
            } else {
#pragma unroll
                for (int c = 0; c < B; c++)
                    asm volatile("st.shared::cluster.f32 [%0], %1;" ::"r"(z_to + 4 * c), "f"(z[c]) : "memory");
            }
        }
    };
    const int half = lane >> 4, hl = lane & 15;
    // Sums over the cluster: the sums of 32 rows, or of warps, go to all CTAs.  Two sums share their steps, one in each half
    // of a warp.  Warp 0 (and 1, the second sum) waits for what arrives here, adds it and tells the CTA; without its
    // __syncwarp the lanes would go on one by one (the beam below: 111 ms).
    // A wait that gives up: the CTA goes on, with values that mean nothing but stay in bounds, to the end of the iteration,
    // where it leaves the loop as one.  The others learn of it (s_abort) at the next barrier of the cluster, before they
    // store into another CTA again, and none has left by then.
    unsigned parity = 0;  // bit i: the phase of s_bar[i] to wait for
    int turn = 0;         // the last r.z are s_grp[2 + turn]
    const int senders = rank == a.withhold ? 0 : C;
    auto arrived = [&](int set, int bytes) {
        if (tid == 0)
            asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(shared_addr(&s_bar[set])), "r"(bytes)
                         : "memory");
        if (warp <= set && !wait_phase(shared_addr(&s_bar[set]), (parity >> set) & 1u, a.wait_ns)) s_late = 1;
        __syncwarp();
        parity ^= 1u << set;
    };
    // the sums of v0 (and v1) over the threads, a warp's in FP32; a CTA's 16 sums as four stores to each CTA (16 of four
    // bytes: 58 ms for the batch below instead of 49)
    auto push_warps = [&](auto two, int set, float v0, float v1) {
        constexpr bool two_sums = decltype(two)::value;
        float t;
        if (two_sums) t = (half ? v1 : v0) + __shfl_xor_sync(0xffffffffu, half ? v0 : v1, 16);
        else t = v0 + __shfl_xor_sync(0xffffffffu, v0, 16);
#pragma unroll
        for (int o = 8; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
        if (hl == 0 && (two_sums || half == 0)) s_warp[half][warp] = t;
        __syncthreads();
        if (warp < (two_sums ? 2 : 1)) {
            const int q = 4 * (lane & 3);
            const uint32_t slot = shared_addr(&s_grp[two_sums ? (warp ? 1 : 3 - turn) : 0][rank * kW + q]);
            const float4 sums = *reinterpret_cast<const float4 *>(&s_warp[warp][q]);
            for (int r = lane >> 2; r < (two_sums ? C : senders); r += 8)
                store_async4(cluster_addr(slot, r), sums, cluster_addr(shared_addr(&s_bar[set]), r));
        }
        arrived(set, two_sums ? s_bytes + 8 * C * kW : 4 * C * kW);
    };
    // Exact: sums over 32 rows of the slice's values s_row[0] (s_row[1]), pushed to every CTA; of p.q by the lane bits 2, 1,
    // then 16, 8, 4, as the warps of 4 rows and CTAs of 32 add them, the others in natural order
    const int64_t P0 = bound[0];
    const int groups = (int)((bound[C] - P0 + 31) / 32), g0 = (int)((n0 - P0) / 32);
    auto push_groups = [&](auto two, int set) {
        constexpr bool two_sums = decltype(two)::value;
        __syncthreads();
        for (int g = warp; g * 32 < R; g += kW) {
            const int i = 32 * g + lane;
            float t = i < R ? s_row[0][i] : 0.0f;
            if (two_sums) {
                const float v1 = i < R ? s_row[1][i] : 0.0f;
                t = (half ? v1 : t) + __shfl_xor_sync(0xffffffffu, half ? t : v1, 16);
#pragma unroll
                for (int o = 8; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
            } else {
                t += __shfl_xor_sync(0xffffffffu, t, 2);
                t += __shfl_xor_sync(0xffffffffu, t, 1);
                t += __shfl_xor_sync(0xffffffffu, t, 16);
                t += __shfl_xor_sync(0xffffffffu, t, 8);
                t += __shfl_xor_sync(0xffffffffu, t, 4);
            }
            if (hl < (two_sums ? C : senders) && (two_sums || half == 0))  // lane r (and 16 + r) to CTA r
                store_async(cluster_addr(shared_addr(&s_grp[two_sums ? (half ? 1 : 3 - turn) : 0][g0 + g]), hl), t,
                            cluster_addr(shared_addr(&s_bar[set]), hl));
        }
        arrived(set, two_sums ? s_bytes + 8 * groups : 4 * groups);
    };
    // FP64 sums (a refresh only), valid in every thread
    auto cluster_sum64 = [&](double v0, double v1, double &t0, double &t1) {
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            v0 += __shfl_down_sync(0xffffffffu, v0, o);
            v1 += __shfl_down_sync(0xffffffffu, v1, o);
        }
        if (lane == 0) { s_dwarp[0][warp] = v0; s_dwarp[1][warp] = v1; }
        __syncthreads();
        if (warp == 0) {
            double u0 = lane < kW ? s_dwarp[0][lane] : 0.0, u1 = lane < kW ? s_dwarp[1][lane] : 0.0;
#pragma unroll
            for (int o = kW / 2; o > 0; o >>= 1) {
                u0 += __shfl_xor_sync(0xffffffffu, u0, o);
                u1 += __shfl_xor_sync(0xffffffffu, u1, o);
            }
            if (lane < C) {
                *cl.map_shared_rank(&s_slotd[0][rank], lane) = u0;
                *cl.map_shared_rank(&s_slotd[1][rank], lane) = u1;
            }
        }
        barrier();
        if (warp == 0) {
            double u0 = lane < C ? s_slotd[0][lane] : 0.0, u1 = lane < C ? s_slotd[1][lane] : 0.0;
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) {
                u0 += __shfl_xor_sync(0xffffffffu, u0, o);
                u1 += __shfl_xor_sync(0xffffffffu, u1, o);
            }
            if (lane == 0) { s_dtot[0] = u0; s_dtot[1] = u1; }
        }
        __syncthreads();
        t0 = s_dtot[0];
        t1 = s_dtot[1];
    };
    // the FP64 true residual of the slice from a.x (published by a barrier before): r, z = Minv r, r.z and |r|^2
    auto residual64 = [&](double &rz, double &rr) {
        constexpr int G = Exact ? 4 : 8;  // lanes per row
        const int gl = tid % G, grp = tid / G;
        const unsigned gmask = ((1u << G) - 1u) << (G * ((tid & 31) / G));
        if constexpr (Exact) __syncthreads();
        double srr = 0.0, srz = 0.0;
        for (int i = grp; i < R; i += kT / G) {
            const int64_t n = n0 + i;
            double acc[B];
#pragma unroll
            for (int c = 0; c < B; c++) acc[c] = 0.0;
            for (int64_t k = a.rp[n] + gl; k < a.rp[n + 1]; k += G) {
                const int64_t j = a.cj[k];
                double u[B];
#pragma unroll
                for (int d = 0; d < B; d++) u[d] = __ldcg(a.x + j * B + d);
#pragma unroll
                for (int c = 0; c < B; c++)
#pragma unroll
                    for (int d = 0; d < B; d++) acc[c] = fma(__ldg(a.K64 + (int64_t)(c * B + d) * a.nb + k), u[d], acc[c]);
            }
#pragma unroll
            for (int o = G / 2; o > 0; o >>= 1)
#pragma unroll
                for (int c = 0; c < B; c++) acc[c] += __shfl_xor_sync(gmask, acc[c], o, G);
            if (gl == 0) {
                double row_rr = 0.0;
#pragma unroll
                for (int c = 0; c < B; c++) {
                    double res = 0.0;
                    if (a.fm[n * B + c]) res = a.b[n * B + c] - acc[c];
                    else if (a.reac) a.reac[n * B + c] = acc[c];
                    zwin[(own + i) * B + c] = (float)res;
                    row_rr = fma(res, res, row_rr);
                }
                if constexpr (Exact) a.rows64[n] = row_rr;
                else srr += row_rr;
            }
        }
        __syncthreads();
#pragma unroll
        for (int m = 0; m < M; m++) {
            const int i = row[m];
            if (i < 0) continue;
#pragma unroll
            for (int c = 0; c < B; c++) rv[m][c] = zwin[(own + i) * B + c];
            float z[B];
            double row_rz = 0.0;
#pragma unroll
            for (int c = 0; c < B; c++) {
                z[c] = 0.0f;
#pragma unroll
                for (int d = 0; d < B; d++) z[c] = fmaf(mi[m][c * B + d], rv[m][d], z[c]);
                row_rz = fma((double)rv[m][c], (double)z[c], row_rz);
            }
            if constexpr (Exact) a.rows64[a.nnodes + n0 + i] = row_rz;
            else srz += row_rz;
            push_z(std::false_type(), m, z);
        }
        if constexpr (Exact) {
            // sums over 64 rows (the slices are whole groups of 64): row bits 4, 2, 1, then 32, 16, 8
            __syncthreads();
            for (int g = warp; g * 64 < R; g += kW)
#pragma unroll
                for (int w = 0; w < 2; w++) {
                    double h[2];
#pragma unroll
                    for (int u = 0; u < 2; u++) {
                        const int i = 64 * g + 32 * u + lane;
                        // (a row without blocks has no owner, and no r)
                        const bool in = i < R && a.rp[n0 + i + 1] > a.rp[n0 + i];
                        h[u] = in ? __ldcg(a.rows64 + (w ? a.nnodes : 0) + n0 + i) : 0.0;
                        h[u] += __shfl_xor_sync(0xffffffffu, h[u], 4);
                        h[u] += __shfl_xor_sync(0xffffffffu, h[u], 2);
                        h[u] += __shfl_xor_sync(0xffffffffu, h[u], 1);
                    }
                    double t = h[0] + h[1];
                    t += __shfl_xor_sync(0xffffffffu, t, 16);
                    t += __shfl_xor_sync(0xffffffffu, t, 8);
                    if (lane < C) *cl.map_shared_rank(&s_grpd[w][(n0 - P0) / 64 + g], lane) = t;
                }
            barrier();
            if (warp == 0) {
                const int n = (groups + 1) / 2;
                const double trr = tree_sum(n, [&](int i) { return s_grpd[0][i]; });
                const double trz = tree_sum(n, [&](int i) { return s_grpd[1][i]; });
                if (lane == 0) { s_dtot[0] = trz; s_dtot[1] = trr; }
            }
            __syncthreads();
            rz = s_dtot[0];
            rr = s_dtot[1];
        } else {
            cluster_sum64(srz, srr, rz, rr);
        }
    };

    double rz64, rr_true;
    residual64(rz64, rr_true);
    const double bnorm2 = rr_true;
    const double stop_rr = 0.0625 * a.tol2 * bnorm2;
    float scale = scale_of(rz64);
    Pair gam = pair(rz64 * (double)scale);
    bool fresh = true;  // the last r.z is a refresh's
    auto last_rz = [&]() { return fresh ? number(rz64) : exact_sum(s_grp[2 + turn], Exact ? groups : C * kW, Exact); };
    // the next refresh: after a 10x drop, or, where that would end within the tolerance, at a quarter of the
    // tolerance (a refresh just inside it would return the solution with up to four times the residual; not with
    // Exact, which refreshes where solve_mixed does)
    auto threshold = [&]() {
        return Exact || 1e-2 * rr_true > a.tol2 * bnorm2 ? fmax(stop_rr, 1e-2 * rr_true) : stop_rr;
    };
    double thr = threshold();
    float scale_rr = scale_of(thr), stop_at = (float)(thr * (double)scale_rr), beta = 0.0f;
    int iters = 0, refreshes = 0, status = 0, since = 0;
    bool done = !(bnorm2 > 0.0) || rr_true <= a.tol2 * bnorm2;
    if (isnan(rr_true)) { status = AMR_ENOCONV; done = true; }
    while (!done) {
        if (iters >= a.max_iters) { status = AMR_ENOCONV; break; }
        // p = z + beta p over the window
#pragma unroll 4
        for (int i = tid; i < W * B; i += kT) pwin[i] = fmaf(beta, pwin[i], zwin[i]);
        __syncthreads();
        // q = K32 p, p.q
        float q[M][B], dot = 0.0f;
#pragma unroll
        for (int m = 0; m < M; m++) {
#pragma unroll
            for (int c = 0; c < B; c++) q[m][c] = 0.0f;
            int e = slot0[m];
            if constexpr (Exact) {  // (S is uniform)
                if (S == 1) exact_row<B, 1>(val4, val1, cols, a.kcap, e, width[m], pwin, q[m]);
                else if (S == 2) exact_row<B, 2>(val4, val1, cols, a.kcap, e, width[m], pwin, q[m]);
                else exact_row<B, 4>(val4, val1, cols, a.kcap, e, width[m], pwin, q[m]);
                if (row[m] >= 0) {
                    float d = 0.0f;
#pragma unroll
                    for (int c = 0; c < B; c++) d = fmaf(pwin[(own + row[m]) * B + c], q[m][c], d);
                    s_row[0][row[m]] = d;
                }
            } else {
#pragma unroll 4
            for (int t = 0; t < width[m]; t++, e += 32) {
                const int j = (int)cols[e] * B;
                float v[BB], pv[B];
#pragma unroll
                for (int u = 0; u < BB / 4; u++) {
                    const float4 f = val4[u * a.kcap + e];
                    v[4 * u] = f.x; v[4 * u + 1] = f.y; v[4 * u + 2] = f.z; v[4 * u + 3] = f.w;
                }
                if (BB % 4) v[BB - 1] = val1[e];
                load_node<B>(pwin + j, pv);
#pragma unroll
                for (int c = 0; c < B; c++)
#pragma unroll
                    for (int d = 0; d < B; d++) q[m][c] = fmaf(v[c * B + d], pv[d], q[m][c]);
            }
            if (S > 1)  // (uniform)
#pragma unroll
                for (int c = 0; c < B; c++) {
                    q[m][c] += __shfl_xor_sync(0xffffffffu, q[m][c], 1);
                    if (S > 2) q[m][c] += __shfl_xor_sync(0xffffffffu, q[m][c], 2);
                }
            if (row[m] >= 0)
#pragma unroll
                for (int c = 0; c < B; c++) dot = fmaf(pwin[(own + row[m]) * B + c], q[m][c], dot);
            }
        }
        if constexpr (Exact) push_groups(std::false_type(), 0);
        else push_warps(std::false_type(), 0, dot, 0.0f);
        const int parts = Exact ? groups : C * kW;
        if (warp == 0) {
            const Pair pq = pair_sum(parts, [&](int i) { return i < parts ? s_grp[0][i] * scale : 0.0f; });
            bool sure;
            float al = pair_div(gam, pq, sure);
            if (!sure) {  // (the same in all lanes)
                const Num e = exact_sum(s_grp[0], parts, false);
                al = e.m == 0 || e.neg ? __int_as_float(0x7fc00000) : quotient(last_rz(), e);
            }
            if (lane == 0) s_alpha = al;
            __syncwarp();
        }
        __syncthreads();
        const bool broken = isnan(s_alpha);  // ends the solve below, where the CTA knows of waits that gave up
        const float alpha = broken ? 0.0f : s_alpha;
        // x += alpha p ; r -= alpha q ; z = Minv r
        float v0 = 0.0f, v1 = 0.0f;
#pragma unroll
        for (int m = 0; m < M; m++) {
            const int i = row[m];
            if (i < 0) continue;
#pragma unroll
            for (int c = 0; c < B; c++) {
                xr[m][c] = fmaf(alpha, pwin[(own + i) * B + c], xr[m][c]);
                rv[m][c] = fmaf(-alpha, q[m][c], rv[m][c]);
            }
            float z[B];
            if (Exact) v0 = v1 = 0.0f;
#pragma unroll
            for (int c = 0; c < B; c++) {
                z[c] = 0.0f;
#pragma unroll
                for (int d = 0; d < B; d++) z[c] = fmaf(mi[m][c * B + d], rv[m][d], z[c]);
                v0 = fmaf(rv[m][c], z[c], v0);
                v1 = fmaf(rv[m][c], rv[m][c], v1);
            }
            push_z(std::true_type(), m, z);
            if constexpr (Exact) {
                s_row[0][i] = v0;
                s_row[1][i] = v1;
            }
        }
        if constexpr (Exact) push_groups(std::true_type(), 1);
        else push_warps(std::true_type(), 1, v0, v1);
        const float *rz = s_grp[3 - turn];
        if (warp < 2) {
            const float *v = warp == 0 ? rz : s_grp[1], sc = warp == 0 ? scale : scale_rr;
            const Pair t = pair_sum(parts, [&](int i) {
                float x = i < parts ? v[i] : 0.0f;
                if constexpr (Exact) {  // CTAs of 256 rows: eight warps' sums by bits 4, 2, 1
                    x += __shfl_xor_sync(0xffffffffu, x, 4);
                    x += __shfl_xor_sync(0xffffffffu, x, 2);
                    x += __shfl_xor_sync(0xffffffffu, x, 1);
                    if (lane & 7) x = 0.0f;
                }
                return x * sc;
            });
            if (warp == 0) {
                bool sure;
                float be = pair_div(t, gam, sure);
                if (!sure) be = quotient(exact_sum(rz, parts, Exact), last_rz());
                gam = t;
                if (lane == 0) s_beta = be;
            } else {
                bool more = t.h > stop_at;  // r.r above the threshold: no refresh yet
                if (!(in_range(t.h) && fabsf(t.h - stop_at) > 0x1p-20f * stop_at))
                    more = greater(exact_sum(v, parts, Exact), number(thr));
                if (lane == 0) s_stop = !more;
            }
            __syncwarp();
        }
        turn ^= 1;
        fresh = false;
        __syncthreads();
        if (s_late) { status = AMR_ETIMEOUT; break; }
        if (broken) { status = AMR_ENOCONV; break; }
        beta = s_beta;
        iters++;
        since++;
        if (Exact && iters >= a.max_iters) { status = AMR_ENOCONV; break; }
        if (s_stop || since >= a.force_every) {
            // refresh: fold the FP32 correction into the FP64 solution and recompute the true residual
#pragma unroll
            for (int m = 0; m < M; m++) {
                const int i = row[m];
                if (i < 0) continue;
#pragma unroll
                for (int c = 0; c < B; c++) {
                    const int64_t g = (n0 + i) * B + c;
                    if (a.fm[g]) a.x[g] += (double)xr[m][c];
                    xr[m][c] = 0.0f;
                }
            }
            __threadfence();
            barrier();
            if (__syncthreads_or(s_abort)) { status = AMR_ETIMEOUT; break; }
            residual64(rz64, rr_true);
            scale = scale_of(rz64);
            gam = pair(rz64 * (double)scale);
            fresh = true;
            thr = threshold();
            scale_rr = scale_of(thr);
            stop_at = (float)(thr * (double)scale_rr);
            refreshes++;
            since = 0;
            if (isnan(rr_true)) { status = AMR_ENOCONV; break; }
            if (rr_true <= a.tol2 * bnorm2) done = true;
        }
    }
    if (status == AMR_ETIMEOUT && tid < C) *cl.map_shared_rank(&s_abort, tid) = 1;  // (every CTA is still there)
    barrier();
    const bool aborted = __syncthreads_or(s_abort);  // from here on no store into another CTA
    // the largest |x| at free slots (NaN as +inf), and the part's statistics
    double um = 0.0;
    for (int64_t i = n0 * B + tid; i < n1 * B; i += kT)
        if (a.fm[i]) {
            const double v = fabs(a.x[i]);
            um = fmax(um, isnan(v) ? INFINITY : v);
        }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) um = fmax(um, __shfl_down_sync(0xffffffffu, um, o));
    __syncthreads();
    if (lane == 0) s_dwarp[0][warp] = um;
    __syncthreads();
    if (tid == 0) {
        for (int w = 1; w < kW; w++) um = fmax(um, s_dwarp[0][w]);
        if (!aborted) *cl.map_shared_rank(&s_um[rank], 0) = um;
    }
    barrier();  // (also: no CTA leaves while a neighbour may read its shared memory)
    if (a.withhold >= 0 && tid == 0) a.stat[rank].status = aborted ? AMR_ETIMEOUT : status;
    else if (rank == 0 && tid == 0) {
        if (aborted) status = AMR_ETIMEOUT;
        else
            for (int r = 0; r < C; r++) um = fmax(um, s_um[r]);
        AmrPartStat s;
        s.iters = iters;
        s.refreshes = refreshes;
        s.status = status;
        s.pad = 0;
        s.rel_residual = bnorm2 > 0.0 ? sqrt(rr_true / bnorm2) : 0.0;
        s.umax = um;
        a.stat[part] = s;
    }
    if (a.t1 && tid == 0) atomicMax(a.t1, global_ns());
}

// for tests: a warp per case, the quotient of the sums of a and b, each cases x n, n <= 512; exact: by integers in any case
__global__ void __launch_bounds__(32) k_sum_quotient(int n, const float *a, const float *b, bool exact, float *out) {
    __shared__ float s[2][kMaxGroups];
    const int64_t at = (int64_t)blockIdx.x * n;
    for (int i = threadIdx.x; i < n; i += 32) {
        s[0][i] = a[at + i];
        s[1][i] = b[at + i];
    }
    __syncwarp();
    Pair p[2];
    float scale = 1.0f;
#pragma unroll
    for (int k = 1; k >= 0; k--) {
        if (k == 1) {
            const Pair t = pair_sum(n, [&](int i) { return i < n ? s[1][i] : 0.0f; });
            scale = scale_of((double)t.h);
        }
        p[k] = pair_sum(n, [&](int i) { return i < n ? s[k][i] * scale : 0.0f; });
    }
    bool sure;
    float v = pair_div(p[0], p[1], sure);
    if (!sure || exact) v = quotient(exact_sum(s[0], n, false), exact_sum(s[1], n, false));
    if (threadIdx.x == 0) out[blockIdx.x] = v;
}

// the kernels' attributes, once per device and process (a launch that changed them would race with others); the
// largest cluster the device takes with the largest slice
int device_cluster() {
    static std::mutex mu;
    static int found[64] = {0};
    int dev = 0;
    AMR_CUDA(cudaGetDevice(&dev));
    if (dev < 0 || dev >= 64) return 0;
    std::lock_guard<std::mutex> lk(mu);
    if (found[dev]) return found[dev] < 0 ? 0 : found[dev];
    int best = -1;
    const void *kernels[4] = {(const void *)k_resident_pcg<2, false>, (const void *)k_resident_pcg<3, false>,
                              (const void *)k_resident_pcg<2, true>, (const void *)k_resident_pcg<3, true>};
    bool ok = true, wide = true;
    for (const void *k : kernels) {
        ok &= cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                   (int)(k == kernels[2] || k == kernels[3] ? kMaxDynExact : kMaxDyn)) == cudaSuccess;
        wide &= cudaFuncSetAttribute(k, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) == cudaSuccess;
    }
    if (ok)
        for (int c : {16, 8}) {
            if (c > 8 && !wide) continue;
            cudaLaunchConfig_t cfg{};
            cudaLaunchAttribute at[1];
            at[0].id = cudaLaunchAttributeClusterDimension;
            at[0].val.clusterDim.x = (unsigned)c;
            at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
            cfg.gridDim = dim3((unsigned)c);
            cfg.blockDim = dim3(kT);
            cfg.attrs = at;
            cfg.numAttrs = 1;
            bool fits = true;
            for (const void *k : kernels) {
                int n = 0;
                cfg.dynamicSmemBytes = k == kernels[2] || k == kernels[3] ? kMaxDynExact : kMaxDyn;
                fits &= cudaOccupancyMaxActiveClusters(&n, k, &cfg) == cudaSuccess && n > 0;
            }
            if (fits) {
                best = c;
                break;
            }
        }
    cudaGetLastError();
    found[dev] = best;
    return best < 0 ? 0 : best;
}

}  // namespace

static size_t resident_bytes(int B, const AmrResidentShape &s) {
    return B == 3 ? slice_bytes<3>(s.slots, s.rows, s.window) : slice_bytes<2>(s.slots, s.rows, s.window);
}

// The cluster size that solves nodes [P0, P1), and the largest slice: the smallest whose slices stay within `prefer`
// bytes of shared memory, else the largest the device takes if its slices fit at all; 0: none.
static AmrResidentShape shape_of(const int64_t *rp, const int32_t *col, int B, int64_t P0, int64_t P1, size_t prefer,
                                 bool exact, int most) {
    AmrResidentShape best;
    const int64_t len = P1 - P0;
    if (most == 0 || len <= 0 || len > (int64_t)most * 65535) return best;
    std::vector<int64_t> place;
    for (int C = 1; C <= most; C *= 2) {
        if (exact && (len - 1) / 64 < C - 1) break;  // fewer groups of 64 rows than CTAs
        AmrResidentShape s;
        s.ctas = C;
        s.bounds.resize(C + 1);
        for (int r = 0; r <= C; r++)
            s.bounds[r] = r == 0   ? P0
                          : r == C ? P1
                                   : std::lower_bound(rp + P0, rp + P1, rp[P0] + (rp[P1] - rp[P0]) * r / C) - rp;
        if (exact)
            // Whole groups of 64 rows, one at least: a CTA's part in a sum is the sums of its rows, so one without rows
            // sends nothing, no other CTA waits for it, and they could write the next sum over the one that it reads.
            for (int r = 1; r < C; r++)
                s.bounds[r] = std::min(std::max(P0 + (s.bounds[r] - P0 + 32) / 64 * 64, s.bounds[r - 1] + 64),
                                       P0 + ((len - 1) / 64 - (C - 1 - r)) * 64);
        s.exact = exact;
        s.perm.resize(len);
        // a row's blocks, or with `exact` its runs of four blocks from a multiple of four
        auto width = [&](int64_t n) {
            const int64_t l = rp[n + 1] - rp[n];
            return exact && l > 0 ? ((rp[n] & 3) + l + 3) / 4 : l;
        };
        // what needs no order first: rows with blocks, and the least that the slices take
        int64_t most_rows = 0;
        AmrResidentShape least;
        for (int r = 0; r < C; r++) {
            const int64_t n0 = s.bounds[r], n1 = s.bounds[r + 1];
            int64_t used = 0;
            for (int64_t n = n0; n < n1; n++) used += rp[n + 1] > rp[n];
            most_rows = std::max(most_rows, used);
            s.rows = std::max(s.rows, n1 - n0);
            least.slots = std::max(least.slots, rp[n1] - rp[n0]);
        }
        if (s.rows > (exact ? kT * kRowsPerThread : 65535) || most_rows > kT * kRowsPerThread) continue;
        least.rows = s.rows;
        least.exact = exact;
        if (resident_bytes(B, least) > (exact ? kMaxDynExact : kMaxDyn)) continue;
        for (int r = 0; r < C; r++) {  // each slice's rows by falling width, equal ones in their order
            const int64_t n0 = s.bounds[r], n1 = s.bounds[r + 1];
            uint16_t *pm = s.perm.data() + (n0 - P0);
            place.assign(1, 0);
            for (int64_t n = n0; n < n1; n++) {
                const size_t w = (size_t)width(n);
                if (w >= place.size()) place.resize(w + 1, 0);
                place[w]++;
            }
            int64_t at = 0;  // counted, not sorted: a batch of 200 parts is laid out in 11 ms, with a sort per slice 81
            for (size_t w = place.size(); w-- > 0;) {
                const int64_t count = place[w];
                place[w] = at;
                at += count;
            }
            for (int64_t n = n0; n < n1; n++) pm[place[(size_t)width(n)]++] = (uint16_t)(n - n0);
        }
        const int S = threads_per_row(most_rows);
        bool fits = true;
        for (int r = 0; r < C && fits; r++) {
            const int64_t n0 = s.bounds[r], n1 = s.bounds[r + 1];
            const uint16_t *pm = s.perm.data() + (n0 - P0);
            int64_t lo = n0, hi = n1, slots = 0;
            for (int64_t n = n0; n < n1; n++)
                if (rp[n + 1] > rp[n]) {  // a row's columns ascend
                    lo = std::min<int64_t>(lo, col[rp[n]]);
                    hi = std::max<int64_t>(hi, col[rp[n + 1] - 1] + 1);
                }
            for (int64_t i = 0; i < n1 - n0; i += 32 / S) {  // the rows of a warp: the first is the longest
                slots += 32 * (exact ? 4 : 1) * ((width(n0 + pm[i]) + S - 1) / S);
            }
            s.slots = std::max(s.slots, slots);
            s.window = std::max(s.window, hi - lo);
            fits = s.window < 65536;
        }
        if (!fits) continue;
        s.bytes = resident_bytes(B, s);
        if (s.bytes > (exact ? kMaxDynExact : kMaxDyn)) continue;
        best = s;
        if (s.bytes <= prefer) break;
    }
    return best;
}

AmrResidentShape amr_resident_shape(const amr_model *m, int64_t P0, int64_t P1, size_t prefer, bool exact) {
    return shape_of(m->h_brow_ptr.data(), m->h_bcol.data(), m->B, P0, P1, prefer, exact, device_cluster());
}

int amr_test_resident_shape(int32_t ndim, int64_t nnodes, const int64_t *row_ptr, const int32_t *col, int64_t prefer,
                            int32_t exact, int32_t most, int64_t *bounds, int64_t *bytes) {
    const AmrResidentShape s = shape_of(row_ptr, col, ndim == 3 ? 3 : 2, 0, nnodes, (size_t)prefer, exact != 0, most);
    std::copy(s.bounds.begin(), s.bounds.end(), bounds);
    *bytes = (int64_t)s.bytes;
    return s.ctas;
}

size_t amr_resident_bytes(const amr_model *m, const AmrResidentShape &s) { return resident_bytes(m->B, s); }
size_t amr_resident_max_bytes() { return kMaxDyn; }

static void launch(int B, const AmrResidentShape &shape, int64_t nparts, const Args &a, cudaStream_t stream) {
    cudaLaunchConfig_t cfg{};
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = (unsigned)shape.ctas;
    at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
    cfg.gridDim = dim3((unsigned)(shape.ctas * nparts));
    cfg.blockDim = dim3(kT);
    cfg.dynamicSmemBytes = shape.bytes;
    cfg.stream = stream;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    auto kernel = B == 3 ? (shape.exact ? k_resident_pcg<3, true> : k_resident_pcg<3, false>)
                         : (shape.exact ? k_resident_pcg<2, true> : k_resident_pcg<2, false>);
    AMR_CUDA(cudaLaunchKernelEx(&cfg, kernel, a));
    AMR_COUNT(1);
}

static Args args_of(const amr_model *m, const AmrResidentShape &shape, const int64_t *slices, const uint16_t *perm,
                    const double *b, double *x, double *reac, double *rows64, AmrPartStat *stat) {
    Args a{};
    a.slices = slices; a.perm = perm;
    a.nb = m->bstride; a.rp = m->brow_ptr; a.cj = m->bcol; a.K32 = m->K32; a.K64 = m->K64; a.Minv = m->Minv32;
    a.fm = m->free_mask; a.b = b; a.x = x; a.reac = reac; a.rows64 = rows64; a.nnodes = m->nnodes; a.stat = stat;
    a.kcap = (int)shape.slots; a.wcap = (int)shape.window;
    a.wait_ns = kWaitNs;
    a.withhold = -1;
    return a;
}

void amr_resident_launch(amr_model *m, const AmrResidentShape &shape, int64_t nparts, const int64_t *slices,
                         const int64_t *first, const uint16_t *perm, const int64_t *list, const uint8_t *active,
                         const double *b, double *x, double *reac, double *rows64, AmrPartStat *stat,
                         unsigned long long *t0, unsigned long long *t1, double tol2, int max_iters, int force_every, cudaStream_t stream) {
    if (nparts <= 0) return;
    Args a = args_of(m, shape, slices, perm, b, x, reac, rows64, stat);
    a.first = first; a.list = list; a.active = active; a.t0 = t0; a.t1 = t1;
    a.tol2 = tol2; a.max_iters = max_iters; a.force_every = force_every;
    launch(m->B, shape, nparts, a, stream);
}

// A cluster whose rank `rank` withholds its part of p.q, with waits of limit_ns at most: every CTA's status.
static void withheld_sum(amr_model *m, bool exact, int rank, unsigned long long limit_ns, std::vector<int32_t> &status) {
    const AmrResidentShape shape = amr_resident_shape(m, 0, m->nnodes, exact ? kAmrSliceSingle : kMaxDyn, exact);
    if (!m->K_valid || !shape.ctas || rank < 0 || rank >= shape.ctas)
        throw AmrError(AMR_EINVAL, "no such CTA in the one-launch solve of this model");
    const int64_t n = m->nnodes * m->B;
    struct Scratch {
        int64_t *slices = nullptr;
        uint16_t *perm = nullptr;
        double *rows64 = nullptr, *b = nullptr, *x = nullptr, *reac = nullptr;
        AmrPartStat *stat = nullptr;
        ~Scratch() {
            amr_free(slices); amr_free(perm); amr_free(rows64); amr_free(b); amr_free(x); amr_free(reac); amr_free(stat);
        }
    } w;
    amr_alloc(&w.slices, shape.bounds.size());
    amr_alloc(&w.perm, shape.perm.size());
    amr_alloc(&w.rows64, 2 * m->nnodes);
    amr_alloc(&w.b, n);
    amr_alloc(&w.x, n);
    amr_alloc(&w.reac, n);
    amr_alloc(&w.stat, shape.ctas);
    const std::vector<double> ones(n, 1.0);
    amr_h2d(m, w.slices, shape.bounds.data(), shape.bounds.size() * sizeof(int64_t));
    amr_h2d(m, w.perm, shape.perm.data(), shape.perm.size() * sizeof(uint16_t));
    amr_h2d(m, w.b, ones.data(), n * sizeof(double));
    AMR_CUDA(cudaMemsetAsync(w.x, 0, n * sizeof(double), m->stream));
    AMR_CUDA(cudaMemsetAsync(w.stat, 0, shape.ctas * sizeof(AmrPartStat), m->stream));
    Args a = args_of(m, shape, w.slices, w.perm, w.b, w.x, w.reac, w.rows64, w.stat);
    a.tol2 = 1e-20; a.max_iters = 1000; a.force_every = 512; a.wait_ns = limit_ns; a.withhold = rank;
    launch(m->B, shape, 1, a, m->stream);
    std::vector<AmrPartStat> st(shape.ctas);
    amr_d2h(m, st.data(), w.stat, st.size() * sizeof(AmrPartStat));
    status.clear();
    for (const AmrPartStat &s : st) status.push_back(s.status);
}

int amr_test_sum_quotient(int64_t cases, int32_t n, const float *a, const float *b, int32_t exact, float *out) {
    if (cases < 1 || cases > INT32_MAX || n < 1 || n > kMaxGroups) return AMR_EINVAL;
    const size_t bytes = (size_t)cases * n * sizeof(float);
    float *d = nullptr;
    if (cudaMalloc(&d, 2 * bytes + cases * sizeof(float)) != cudaSuccess) return AMR_ENOMEM;
    float *db = d + cases * n, *dout = db + cases * n;
    cudaError_t e = cudaMemcpy(d, a, bytes, cudaMemcpyHostToDevice);
    if (e == cudaSuccess) e = cudaMemcpy(db, b, bytes, cudaMemcpyHostToDevice);
    if (e == cudaSuccess) {
        k_sum_quotient<<<(unsigned)cases, 32>>>(n, d, db, exact != 0, dout);
        e = cudaGetLastError();
    }
    if (e == cudaSuccess) e = cudaMemcpy(out, dout, cases * sizeof(float), cudaMemcpyDeviceToHost);
    cudaFree(d);
    return e == cudaSuccess ? AMR_OK : AMR_ECUDA;
}

int amr_test_resident_wait(amr_model *m, int32_t exact, int32_t rank, double limit_ms, int32_t *status, int32_t *ctas) {
    try {
        AmrStreamScope scope(m->stream);
        std::vector<int32_t> st;
        withheld_sum(m, exact != 0, rank, (unsigned long long)(limit_ms * 1e6), st);
        std::copy(st.begin(), st.end(), status);
        *ctas = (int32_t)st.size();
        return AMR_OK;
    } catch (const AmrError &e) {
        m->err = e.msg;
        return e.code;
    } catch (const std::exception &e) {
        m->err = e.what();
        return AMR_EINVAL;
    }
}
