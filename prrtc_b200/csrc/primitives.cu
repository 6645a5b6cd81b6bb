// primitives.cu -- standalone kernels: batched nearest neighbour, extend, the
// batched FK + collision checker, FK and Halton sampling.  sm_100a.
#include <cuda_runtime.h>
#include <float.h>
#include <limits.h>
#include <math.h>

#include <algorithm>
#include <mutex>

#include "kernels.h"
#include "prrtc_cull.cuh"
#include "prrtc_device.cuh"

namespace prrtc {

// ============================================================================ nearest neighbour

// Every CTA holds up to kNnQueries queries and strides over the tree, a column of
// 4 nodes per thread, so the tree is read once per 64 queries.  The dimensions go
// in blocks of 4: after a block, a warp whose 128 partial sums all exceed the
// query's best distance so far leaves the query (a sum of squares only grows, also
// in rounded arithmetic), which in 7 dimensions is nearly always after the first
// block.  The best distances are shared: each
// improvement goes to the CTA's and the global key at once, and every CTA
// rereads the global keys per column.  Keys order like (squared distance,
// index), so the result is the nearest node, the lowest index on a tie; NaN and
// infinite distances never pass.  Per (node, query) x - q (as x + -q, two nodes
// per instruction), then fma(d, d, sum) from +0 in dimension order, bit-identical
// to the reference's `dsq += diff*diff` (prrtc_nearest_neighbor.cu).
//
// One query is bound by HBM (33.5 M nodes x 7, 90% live: 131 us, 6.45 TB/s, 98%
// of the measured copy; a CTA per slice with its own minimum took 145 us), 64 by
// issue: 16 packed instructions, a vote and the loop per query and 128 nodes (4.19
// M nodes x 7: 505 -> 143 us against 8 queries per pass over the tree and all
// dimensions; rows that are not 16-byte aligned 3039 -> 148 us, since one load
// form serves both).  Loops of 1 or 4 queries measured the same.
constexpr int kNnQueries = 64;
constexpr unsigned long long kNnNone = 0x7f7fffffffffffffull;  // no node yet: FLT_MAX, above every index

__device__ __forceinline__ float2 add2(float2 a, float2 b) {
    unsigned long long x, y, r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(x) : "f"(a.x), "f"(a.y));
    asm("mov.b64 %0, {%1, %2};" : "=l"(y) : "f"(b.x), "f"(b.y));
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(x), "l"(y));
    asm("mov.b64 {%0, %1}, %2;" : "=f"(a.x), "=f"(a.y) : "l"(r));
    return a;
}
__device__ __forceinline__ float2 square_add2(float2 d, float2 acc) {
    unsigned long long x, y, r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(x) : "f"(d.x), "f"(d.y));
    asm("mov.b64 %0, {%1, %2};" : "=l"(y) : "f"(acc.x), "f"(acc.y));
    asm("fma.rn.f32x2 %0, %1, %1, %2;" : "=l"(r) : "l"(x), "l"(y));
    asm("mov.b64 {%0, %1}, %2;" : "=f"(acc.x), "=f"(acc.y) : "l"(r));
    return acc;
}

// DB blocks of 4 dimensions; VEC: rows start 16-byte aligned and a thread's 4
// nodes are neighbours (one 16-byte load per dimension), else they are T apart.
template <int DB, bool VEC>
__global__ void __launch_bounds__(256, DB <= 2 ? 3 : 2) nn_scan_kernel(const float* __restrict__ tree, int dim, int N,
                                                                      const int32_t* tree_size, int size,
                                                                      int limit, const float* __restrict__ q, int batch,
                                                                      int per_cta, unsigned long long* keys) {
    __shared__ __align__(16) float2 nq[kNnQueries][DB * 4];  // (-q, -q)
    __shared__ unsigned long long s_key[kNnQueries];
    constexpr int T = 256;
    const int tid = threadIdx.x, lane = tid & 31;
    const int q0 = blockIdx.y * per_cta, nqs = min(per_cta, batch - q0);
    for (int i = tid; i < nqs * DB * 4; i += T) {
        const int k = i / (DB * 4), d = i - k * DB * 4;
        const float x = d < dim ? -q[(size_t)(q0 + k) * dim + d] : 0.0f;
        nq[k][d] = make_float2(x, x);
    }
    if (tid < kNnQueries) s_key[tid] = kNnNone;
    __syncthreads();
    int n = tree_size ? tree_size[0] : size;
    n = min(max(1, min(n, N)), limit);
    volatile const unsigned* bound = reinterpret_cast<volatile const unsigned*>(s_key);  // high words: odd
    for (long long base = (long long)blockIdx.x * T * 4; base < n; base += (long long)gridDim.x * T * 4) {
        const int i0 = (int)base + (VEC ? 4 * tid : tid);
        constexpr int step = VEC ? 1 : T;
        unsigned long long seen = ~0ull;
        if (tid < nqs) seen = __ldcg(&keys[q0 + tid]);
        // nodes past the end read as far away (never NaN-free near ones)
        float2 v[DB * 4][2];
#pragma unroll
        for (int d = 0; d < DB * 4; ++d) {
            float4 x = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
            if (d < dim) {
                const float* row = tree + (size_t)d * N;
                if (VEC) {
                    if (i0 < n) x = __ldg(reinterpret_cast<const float4*>(row + i0));  // N % 4 == 0: inside the row
                } else {
                    if (i0 < n) x.x = __ldg(row + i0);
                    if (i0 + T < n) x.y = __ldg(row + i0 + T);
                    if (i0 + 2 * T < n) x.z = __ldg(row + i0 + 2 * T);
                    if (i0 + 3 * T < n) x.w = __ldg(row + i0 + 3 * T);
                }
            }
            v[d][0] = make_float2(x.x, x.y);
            v[d][1] = make_float2(x.z, x.w);
        }
        // a node past the end starts from infinity, so that its sum never passes
        const float2 s0 = make_float2(i0 < n ? 0.0f : INFINITY, i0 + step < n ? 0.0f : INFINITY);
        const float2 s1 = make_float2(i0 + 2 * step < n ? 0.0f : INFINITY, i0 + 3 * step < n ? 0.0f : INFINITY);
#pragma unroll 2
        for (int k = 0; k < nqs; ++k) {
            const float best = __uint_as_float(bound[2 * k + 1]);
            float2 a = s0, b = s1;
            bool in = true;
#pragma unroll
            for (int blk = 0; blk < DB; ++blk) {
                if (!in) break;
#pragma unroll
                for (int d = 4 * blk; d < 4 * blk + 4; ++d) {
                    const float2 m = nq[k][d];
                    a = square_add2(add2(v[d][0], m), a);
                    b = square_add2(add2(v[d][1], m), b);
                }
                in = __any_sync(0xffffffffu, fminf(fminf(a.x, a.y), fminf(b.x, b.y)) <= best);
            }
            if (!in) continue;
            // some node of the warp is as near as the best so far
            float lo = INFINITY;
            int li = 0x7fffffff;
            if (a.x < lo) { lo = a.x; li = i0; }
            if (a.y < lo) { lo = a.y; li = i0 + step; }
            if (b.x < lo) { lo = b.x; li = i0 + 2 * step; }
            if (b.y < lo) { lo = b.y; li = i0 + 3 * step; }
            const unsigned bits = __float_as_uint(lo), wmin = __reduce_min_sync(0xffffffffu, bits);
            const unsigned idx = __reduce_min_sync(0xffffffffu, bits == wmin ? (unsigned)li : 0x7fffffffu);
            const unsigned long long key = (unsigned long long)wmin << 32 | idx;
            if (lane == 0 && key < s_key[k] && atomicMin(&s_key[k], key) > key) atomicMin(&keys[q0 + k], key);
        }
        if (seen < kNnNone && seen < s_key[tid < nqs ? tid : 0] && tid < nqs) atomicMin(&s_key[tid], seen);
    }
}

// Batches on large trees: the tensor cores rule nodes out, the rest is computed as
// above.  A dot product in tf32 gives (1 - c)|x|^2 - 2 x.q for 16 nodes and 8
// queries per instruction (the norm from the squares against 1 - c); above
// best (1 + 2^-16) - (1 - c)|q|^2, the node is farther than the best so far.
// Rounding both factors to tf32 moves 2 x.q by at most 2^-10 (|x|^2 + |q|^2) and the
// norm by 2^-11 |x|^2; sums in float32 (of at most 17 terms, in any order and
// rounding) add 2^-17 (|x|^2 + |q|^2) + 2^-18 best; c = 2^-9 covers them, and 2^-16 the
// rounding of the exact sum.  Squares from 1e37 on, infinities and NaN count as
// near.  So every node that could be nearest is computed exactly, and the result
// is that of nn_scan_kernel bit for bit.
//
// A warp takes 32 nodes at a time, 4 neighbours per lane (one 16-byte load per
// dimension and 128 bytes in a row per warp): the fragments' rows may be nodes in
// any order.  The best distances start from a scan of the first kNnFirst nodes,
// and are shared as above.
//
// Bound by the latency of its own chain (16 warps per SM issue half the time; the
// tensor pipe is 35% busy, and the tree's 117 MB would take 18 us): 64 queries, 4.19
// M nodes x 7: 146 -> 58 us for the call's kernels, 14 dimensions 244 -> 98. A step
// of 32 nodes per warp took 65 us, the norm as one more dimension summed by
// shuffles 65 us, sums started from the best distance 73 us.
constexpr int kNnFirst = 8192;
// The filter from 16 queries and 2^23 pairs on: 64 queries x 131,072 nodes 18.4
// against 19.6 us by scan, 16 x 1 M 21.3 against 27.2, but 16 x 262,144 17.4 against
// 15.4 (the first scan and one more launch), and below 16 queries the scan waits
// for memory as the filter does.
constexpr int kNnFilterBatch = 16;
constexpr long long kNnFilterPairs = 1ll << 23;
constexpr int kNnGroups = 2;  // groups of 32 nodes per warp and step, up to 8 dimensions
constexpr float kNnSlack = 1.0f / 512;

__device__ __forceinline__ float min_nan(float a, float b, float c) {
    float r;
    asm("min.NaN.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
    return r;
}
__device__ __forceinline__ uint32_t to_tf32(float x) {
    uint32_t r;
    asm("cvt.rna.tf32.f32 %0, %1;" : "=r"(r) : "f"(x));
    return r;
}
// d = c + a (16 nodes x 8 KS) times b (8 KS x 8 queries).  volatile: the rare second
// pass must compute its products again, not keep the first pass's in registers
template <int KS>
__device__ __forceinline__ void mma_tf32(float (&d)[4], const uint32_t (&a)[KS][4], const uint32_t (&b)[KS][2],
                                         const float (&c)[4]) {
#pragma unroll
    for (int k = 0; k < KS; ++k) {
        const float* from = k ? d : c;
        asm volatile("mma.sync.aligned.m16n8k8.row.col.f32.tf32.tf32.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, "
                     "{%10, %11, %12, %13};"
                     : "=f"(d[0]), "=f"(d[1]), "=f"(d[2]), "=f"(d[3])
                     : "r"(a[k][0]), "r"(a[k][1]), "r"(a[k][2]), "r"(a[k][3]), "r"(b[k][0]), "r"(b[k][1]), "f"(from[0]),
                       "f"(from[1]), "f"(from[2]), "f"(from[3]));
    }
}

struct NnShared {
    float q[kNnQueries][17];            // the queries
    float start[kNnQueries];            // (1 - c)|q|^2 - best (1 + 2^-16) - 1e-36
    float qn[kNnQueries];               // (1 - c)|q|^2
    unsigned long long key[kNnQueries]; // best so far
};

// The pairs of `bits` (4 i + 2 e + r: query + r, node + 32 (i / 2) + 2 (i % 2) + e) that
// are not ruled out, exactly.
static __device__ __noinline__ void nn_exact(NnShared& s, unsigned bits, const float* __restrict__ tree, int dim, int N, int n,
                                             int node, int query, int nqs, unsigned long long* keys) {
    for (; bits; bits &= bits - 1u) {
        const int i = __ffs(bits) - 1, k = query + (i & 1), x = node + 32 * (i >> 3) + ((i >> 1) & 3);
        if (k >= nqs || x >= n) continue;
        float d2 = 0.0f;
        for (int d0 = 0; d0 < dim; d0 += 8) {  // eight loads on their way together
            float r[8];
#pragma unroll
            for (int d = 0; d < 8; ++d) r[d] = __ldg(tree + (size_t)min(d0 + d, dim - 1) * N + x);
#pragma unroll
            for (int d = 0; d < 8; ++d) {
                const float d1 = __fadd_rn(r[d], -s.q[k][min(d0 + d, dim - 1)]);
                if (d0 + d < dim) d2 = __fmaf_rn(d1, d1, d2);
            }
        }
        const unsigned long long key = (unsigned long long)__float_as_uint(d2) << 32 | (unsigned)x;
        if (d2 <= FLT_MAX && key < s.key[k] && atomicMin(&s.key[k], key) > key) {
            atomicMin(&keys[k], key);
            s.start[k] = s.qn[k] - __fmaf_ru(d2, 1.0f + 1.0f / 65536, 1e-36f);  // an older, larger best only rules out less
        }
    }
}

// KS steps of 8 dimensions, NT tiles of 8 queries, G groups of 32 nodes per warp and step.
template <int KS, int NT, int G, bool VEC>
__global__ void __launch_bounds__(256, 2) nn_filter_kernel(const float* __restrict__ tree, int dim, int N,
                                                           const int32_t* tree_size, int size, const float* __restrict__ q,
                                                           int batch, unsigned long long* keys) {
    __shared__ __align__(16) NnShared s;
    constexpr int T = 256, kCta = NT * 8;
    const int tid = threadIdx.x, lane = tid & 31, c = lane & 3, g = lane >> 2;
    const int q0 = blockIdx.y * kCta, nqs = min(kCta, batch - q0);
    keys += q0;
    if (tid < kCta) {
        float norm = 0.0f;
        for (int d = 0; d < dim; ++d) {
            const float x = tid < nqs ? q[(size_t)(q0 + tid) * dim + d] : 0.0f;
            s.q[tid][d] = x;
            norm = fmaf(x, x, norm);
        }
        s.qn[tid] = tid >= nqs ? INFINITY : (norm < 1e37f ? (1.0f - kNnSlack) * norm : NAN);
        s.key[tid] = tid < nqs ? min(kNnNone, __ldcg(&keys[tid])) : 0ull;
        s.start[tid] = s.qn[tid] - __fmaf_ru(__uint_as_float((unsigned)(s.key[tid] >> 32)), 1.0f + 1.0f / 65536, 1e-36f);
    }
    __syncthreads();
    uint32_t b[NT][KS][2];
#pragma unroll
    for (int j = 0; j < NT; ++j)
#pragma unroll
        for (int ks = 0; ks < KS; ++ks)
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const int slot = 8 * ks + 4 * h + c;
                b[j][ks][h] = to_tf32(slot < dim ? -2.0f * s.q[8 * j + g][slot] : 0.0f);
            }
    int n = tree_size ? tree_size[0] : size;
    n = max(1, min(n, N));
    uint32_t ones[KS][2];  // the norm: the squares against 1 - c, for every query
#pragma unroll
    for (int ks = 0; ks < KS; ++ks) ones[ks][0] = ones[ks][1] = to_tf32(1.0f - kNnSlack);
    const long long stride = (long long)gridDim.x * T * G;
    long long base = kNnFirst + ((long long)blockIdx.x * T + (tid & ~31)) * G;
    float4 v[G][KS][2];
    auto fetch = [&](long long from) {
#pragma unroll
        for (int f = 0; f < G; ++f)
#pragma unroll
            for (int ks = 0; ks < KS; ++ks)
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    const int d = 8 * ks + 4 * h + c;
                    const long long i = from + 32 * f + 4 * g;
                    float4 x = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
                    if (d < dim) {
                        const float* row = tree + (size_t)d * N;
                        if (VEC) {
                            if (i < n) x = __ldg(reinterpret_cast<const float4*>(row + i));  // N % 4 == 0: inside the row
                        } else {
                            if (i < n) x.x = __ldg(row + i);
                            if (i + 1 < n) x.y = __ldg(row + i + 1);
                            if (i + 2 < n) x.z = __ldg(row + i + 2);
                            if (i + 3 < n) x.w = __ldg(row + i + 3);
                        }
                    }
                    v[f][ks][h] = x;
                }
    };
    auto start = [&](int j) { return *reinterpret_cast<const volatile unsigned long long*>(&s.start[8 * j + 2 * c]); };
    fetch(base);
    for (; base < n; base += stride) {
        unsigned long long seen = ~0ull;
        if (tid < nqs) seen = __ldcg(&keys[tid]);
        // tile 2 f + t: nodes 2 t, 2 t + 1 of each lane's four in group f
        uint32_t a[2 * G][KS][4];
        float norm[2 * G][4], top = 0.0f;
#pragma unroll
        for (int f = 0; f < G; ++f)
#pragma unroll
            for (int t = 0; t < 2; ++t) {
                uint32_t sq[KS][4];
#pragma unroll
                for (int ks = 0; ks < KS; ++ks) {
                    const float4 lo = v[f][ks][0], hi = v[f][ks][1];
                    const float x[4] = {t ? lo.z : lo.x, t ? lo.w : lo.y, t ? hi.z : hi.x, t ? hi.w : hi.y};
#pragma unroll
                    for (int r = 0; r < 4; ++r) {
                        const float x2 = x[r] * x[r];
                        top = fmaxf(top, x2);
                        a[2 * f + t][ks][r] = to_tf32(x[r]);
                        sq[ks][r] = to_tf32(x2);
                    }
                }
                const float zero[4] = {0.0f, 0.0f, 0.0f, 0.0f};
                mma_tf32<KS>(norm[2 * f + t], sq, ones, zero);
            }
        fetch(base + stride);
        float m = top < 1e37f ? INFINITY : NAN;
#pragma unroll
        for (int j = 0; j < NT; ++j) {
            const unsigned long long w = start(j);
            float lo0 = INFINITY, lo1 = INFINITY;
#pragma unroll
            for (int i = 0; i < 2 * G; ++i) {
                float d[4];
                mma_tf32<KS>(d, a[i], b[j], norm[i]);
                lo0 = min_nan(lo0, d[0], d[2]);
                lo1 = min_nan(lo1, d[1], d[3]);
            }
            const float2 x = add2(make_float2(lo0, lo1), make_float2(__uint_as_float((unsigned)w), __uint_as_float((unsigned)(w >> 32))));
            m = min_nan(m, x.x, x.y);
        }
        if (__any_sync(0xffffffffu, !(m > 0.0f))) {
            const bool wide = __any_sync(0xffffffffu, !(top < 1e37f));
#pragma unroll 1
            for (int j = 0; j < NT; ++j) {
                uint32_t bj[KS][2];
#pragma unroll
                for (int ks = 0; ks < KS; ++ks)
#pragma unroll
                    for (int h = 0; h < 2; ++h) {
                        const int slot = 8 * ks + 4 * h + c;
                        bj[ks][h] = to_tf32(slot < dim ? -2.0f * s.q[8 * j + g][slot] : 0.0f);
                    }
                const unsigned long long w = start(j);
                const float s0 = __uint_as_float((unsigned)w), s1 = __uint_as_float((unsigned)(w >> 32));
                unsigned bits = 0u;
#pragma unroll
                for (int i = 0; i < 2 * G; ++i) {
                    float d[4];
                    mma_tf32<KS>(d, a[i], bj, norm[i]);
#pragma unroll
                    for (int r = 0; r < 4; ++r)
                        bits |= (unsigned)(wide || !(d[r] + (r & 1 ? s1 : s0) > 0.0f)) << (4 * i + r);
                }
                if (bits) nn_exact(s, bits, tree, dim, N, n, (int)base + 4 * g, 8 * j + 2 * c, nqs, keys);
                __syncwarp();
            }
        }
        if (tid < nqs && seen < s.key[tid]) {  // what other CTAs found
            atomicMin(&s.key[tid], seen);
            s.start[tid] = s.qn[tid] - __fmaf_ru(__uint_as_float((unsigned)(seen >> 32)), 1.0f + 1.0f / 65536, 1e-36f);
        }
        __syncwarp();
    }
}

__global__ void nn_decode_kernel(const unsigned long long* keys, int batch, int32_t* idx, float* dist) {
    const int b = blockIdx.x * blockDim.x + threadIdx.x;
    if (b >= batch) return;
    const unsigned long long k = keys[b];
    if (k == ~0ull) {
        idx[b] = 0;
        dist[b] = INFINITY;
        return;
    }
    idx[b] = (int32_t)(k & 0xffffffffull);
    dist[b] = __fsqrt_rn(__uint_as_float((unsigned)(k >> 32)));
}

cudaError_t launch_nearest(const float* tree, int dim, int N, const int32_t* tree_size, int size, const float* q, int batch,
                           int32_t* idx, float* dist, unsigned long long* keys, cudaStream_t st) {
    if (batch <= 0) return cudaSuccess;
    cudaError_t e = cudaMemsetAsync(keys, 0xFF, (size_t)batch * sizeof(unsigned long long), st);
    if (e != cudaSuccess) return e;
    const int sms = device_sm_count();
    const bool vec = (N & 3) == 0 && (reinterpret_cast<uintptr_t>(tree) & 15) == 0;
    // columns of 1024 nodes; a small tree is spread by giving each CTA fewer queries
    const int columns = (int)(((long long)N + 1023) / 1024);
    const int per_cta = (int)std::min<long long>(kNnQueries, std::max<long long>(4, (long long)batch * columns / (3 * sms)));
    const int tiles = (batch + per_cta - 1) / per_cta;
    const int db = (dim + 3) / 4;
    if (tiles > 65535) return cudaErrorInvalidConfiguration;
    const bool filter = batch >= kNnFilterBatch && (long long)batch * N >= kNnFilterPairs;
    const int limit = filter ? kNnFirst : INT_MAX;
    dim3 grid((unsigned)std::max(1, std::min(columns, (3 * sms + tiles - 1) / tiles)), (unsigned)tiles);
    int share = per_cta;
    if (filter) {  // the first nodes only: a CTA per column and few queries
        const int first = kNnFirst / 1024;
        share = std::max(4, (int)((long long)batch * first / (2 * sms)));
        share = std::min(share, kNnQueries);
        if ((batch + share - 1) / share > 65535) return cudaErrorInvalidConfiguration;
        grid = dim3((unsigned)first, (unsigned)((batch + share - 1) / share));
    }
#define PRRTC_NN_SCAN(DB)                                                                                              \
    if (vec) nn_scan_kernel<DB, true><<<grid, 256, 0, st>>>(tree, dim, N, tree_size, size, limit, q, batch, share, keys); \
    else nn_scan_kernel<DB, false><<<grid, 256, 0, st>>>(tree, dim, N, tree_size, size, limit, q, batch, share, keys)
    if (db <= 1) { PRRTC_NN_SCAN(1); }
    else if (db == 2) { PRRTC_NN_SCAN(2); }
    else if (db == 3) { PRRTC_NN_SCAN(3); }
    else { PRRTC_NN_SCAN(4); }
#undef PRRTC_NN_SCAN
    if (filter) {
        if ((e = cudaGetLastError()) != cudaSuccess) return e;
        const int nt = batch <= 32 ? 4 : 8, y = (batch + 8 * nt - 1) / (8 * nt);
        const int step = 256 * (dim <= 8 ? kNnGroups : 1), cols = (N - kNnFirst + step - 1) / step;
        const dim3 fgrid((unsigned)std::max(1, std::min(cols, (2 * sms + y - 1) / y)), (unsigned)y);
#define PRRTC_NN_FILTER(KS, NT, G)                                                                                    \
    if (vec) nn_filter_kernel<KS, NT, G, true><<<fgrid, 256, 0, st>>>(tree, dim, N, tree_size, size, q, batch, keys); \
    else nn_filter_kernel<KS, NT, G, false><<<fgrid, 256, 0, st>>>(tree, dim, N, tree_size, size, q, batch, keys)
        if (dim <= 8 && nt == 4) { PRRTC_NN_FILTER(1, 4, kNnGroups); }
        else if (dim <= 8) { PRRTC_NN_FILTER(1, 8, kNnGroups); }
        else if (nt == 4) { PRRTC_NN_FILTER(2, 4, 1); }
        else { PRRTC_NN_FILTER(2, 8, 1); }
#undef PRRTC_NN_FILTER
    }
    if ((e = cudaGetLastError()) != cudaSuccess) return e;
    nn_decode_kernel<<<(batch + 255) / 256, 256, 0, st>>>(keys, batch, idx, dist);
    return cudaGetLastError();
}

// ============================================================================ extend

// prrtc_extend.cu:14-73: new = near + (sample - near) * min(1, step / |sample - near|).
__global__ void extend_kernel(const float* tree, int dim, int N, const int32_t* nearest, const float* samples,
                              int batch, const float* step, float* out, int32_t* parents, int32_t* valid) {
    const int b = blockIdx.x * blockDim.x + threadIdx.x;
    if (b >= batch) return;
    const int ni = nearest[b];
    const float s = step[0];
    float dsq = 0.0f;
    float nv[kDimMax], sv[kDimMax];
    for (int d = 0; d < dim; ++d) {
        nv[d] = tree[(size_t)d * N + ni];
        sv[d] = samples[(size_t)b * dim + d];
        const float df = __fsub_rn(sv[d], nv[d]);
        dsq = d == 0 ? __fmul_rn(df, df) : __fmaf_rn(df, df, dsq);
    }
    const float scale = fminf(1.0f, __fdiv_rn(s, __fsqrt_rn(dsq)));
    for (int d = 0; d < dim; ++d) out[(size_t)b * dim + d] = __fmaf_rn(__fsub_rn(sv[d], nv[d]), scale, nv[d]);
    parents[b] = ni;
    valid[b] = 1;
}

cudaError_t launch_extend(const float* tree, int dim, int N, const int32_t* nearest, const float* samples,
                          int batch, const float* step, float* out, int32_t* parents, int32_t* valid,
                          cudaStream_t st) {
    if (batch <= 0) return cudaSuccess;
    extend_kernel<<<(batch + 127) / 128, 128, 0, st>>>(tree, dim, N, nearest, samples, batch, step, out, parents,
                                                       valid);
    return cudaGetLastError();
}

// ============================================================================ legacy iteration

// prrtc_iteration.cu:21-167 (the "prrtc_iteration" target): every call first
// resets the state to one node per tree, then each sample extends the smaller
// tree (equal sizes: tree = sample & 1) from its nearest node among the
// `completed` ones and appends the step-limited candidate.  The reference reads
// the live sizes and appends with atomics, so its tree choice and slot order
// depend on scheduling; here every sample sees the sizes after the reset and
// the samples of a tree take its slots in sample order -- the schedule in which
// every block reads before any block inserts.  One warp per sample.
__global__ void iteration_kernel(float* ta, float* tb, int32_t* pa, int32_t* pb, int dim, int N,
                                 const float* __restrict__ samples, int batch, int32_t* sizes, int32_t* completed,
                                 const float* step_ptr, int32_t* new_cfg, int32_t* new_par, int32_t* valid,
                                 int32_t* solved) {
    // state after the reset (prrtc_iteration.cu:28-45): sizes = completed = {1, 1}
    const int n0 = (batch + 1) >> 1, n1 = batch >> 1;  // samples per tree under the tie rule
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        const int room = max(0, N - 1);
        sizes[0] = completed[0] = 1 + min(n0, room);
        sizes[1] = completed[1] = 1 + min(n1, room);
        solved[0] = 0;
    }
    const int b = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
    if (b >= batch) return;
    const int t = b & 1;
    float* tree = t == 0 ? ta : tb;
    int32_t* par = t == 0 ? pa : pb;
    const float* q = samples + (size_t)b * dim;
    // nearest among the completed nodes [0, 1): the root
    const int nn = 0;
    float dsq = 0.0f;
    for (int d = 0; d < dim; ++d) {
        const float df = __fsub_rn(tree[(size_t)d * N + nn], q[d]);
        dsq = d == 0 ? __fmul_rn(df, df) : __fmaf_rn(df, df, dsq);
    }
    const float nd = __fsqrt_rn(dsq);
    const float step = step_ptr[0];
    const float scale = nd > 1e-8f ? fminf(1.0f, __fdiv_rn(step, nd)) : 1.0f;
    const int idx = 1 + (b >> 1);  // this sample's slot in tree t
    const bool ok = idx < N;
    for (int d = lane; d < dim; d += 32) {
        const float nv = tree[(size_t)d * N + nn];
        const float c = __fmaf_rn(__fsub_rn(q[d], nv), scale, nv);
        new_cfg[(size_t)b * dim + d] = __float_as_int(c);
        if (ok) tree[(size_t)d * N + idx] = c;
    }
    if (lane == 0) {
        new_par[b] = nn;
        valid[b] = ok ? 1 : 0;
        if (ok) par[idx] = nn;
    }
}

cudaError_t launch_iteration(float* ta, float* tb, int32_t* pa, int32_t* pb, int dim, int N, const float* samples,
                             int batch, int32_t* sizes, int32_t* completed, const float* step, int32_t* new_cfg,
                             int32_t* new_par, int32_t* valid, int32_t* solved, cudaStream_t st) {
    const int blocks = std::max(1, (batch * 32 + 127) / 128);
    iteration_kernel<<<blocks, 128, 0, st>>>(ta, tb, pa, pb, dim, N, samples, batch, sizes, completed, step, new_cfg,
                                             new_par, valid, solved);
    return cudaGetLastError();
}

// ============================================================================ batched collision check

// Persistent over chunks of CW configurations; the scene is bulk-copied into
// shared memory once per CTA.  The wait is bounded: when it runs out, the CTA
// sets bit kBlobStagingTimeout of the blob header's `error` word (global
// memory), lets the copy land (second bounded wait) and reads the scene from
// global memory instead -- the verdicts are the same either way.
#ifndef PRRTC_CHECK_CW
#define PRRTC_CHECK_CW 32       // configurations per CTA pass of the batched checker
#endif
#ifndef PRRTC_CHECK_MINBLOCKS
#define PRRTC_CHECK_MINBLOCKS 4 // resident CTAs per SM the register allocation must allow (shared memory allows 4 at CW 32)
#endif

template <int CW, bool FULL>
__global__ void __launch_bounds__(128, PRRTC_CHECK_MINBLOCKS) check_kernel(const unsigned char* __restrict__ gblob, int blob_cap,
                                                    const int32_t* pairs, int J, int S, int K, int Q, int dim,
                                                    const float* __restrict__ configs, int n, int32_t* verdicts,
                                                    PcView pc) {
    extern __shared__ __align__(128) unsigned char dsm[];
    __shared__ __align__(8) uint64_t mbar;
    const int tid = threadIdx.x;
    const bool staged = blob_cap > 0;
    const CcBufs B = cc_bufs(dsm + (staged ? blob_cap : 0), J, S, K, Q, CW);
    Scene sc;
    if (staged) {
        const int bytes = min(reinterpret_cast<const BlobHeader*>(gblob)->used_bytes, blob_cap);
        if (tid == 0) mbar_init(&mbar);
        __syncthreads();
        uint32_t phase = 0;
        int* err = reinterpret_cast<int*>(const_cast<unsigned char*>(gblob) + offsetof(BlobHeader, error));
        const bool ok = stage_blob(dsm, gblob, bytes, &mbar, phase, err, kBlobStagingTimeout, kWaitLimit);
        sc = scene_view(ok ? dsm : gblob);
    } else {
        sc = scene_view(gblob);
    }
    sc.pairs = reinterpret_cast<const int2*>(pairs);
    sc.pc = pc;
    if (tid == 0) B.hit[0] = B.hit[1] = 0u;
    int par = 0;
    __syncthreads();
    for (int c0 = blockIdx.x * CW; c0 < n; c0 += gridDim.x * CW) {
        const int nw = min(CW, n - c0);
        for (int i = tid; i < nw * dim; i += blockDim.x) {
            const int w = i / dim, d = i - w * dim;
            B.q[w * kDimMax + d] = configs[(size_t)(c0 + w) * dim + d];
        }
        __syncthreads();
        const uint32_t hit = cc_chunk<FULL>(CtaGroup{}, sc, B, nw, false, par);
        for (int w = tid; w < nw; w += blockDim.x) verdicts[c0 + w] = (hit >> w) & 1u;
    }
}

// One candidate pass size of the batched checker: its kernel, dynamic shared
// memory (the scene staged when it fits), and resident CTAs per SM.
struct CheckLaunch {
    int cw = 0, blob_cap = 0, per_sm = 0;
    size_t dyn = 0;
};

static std::mutex g_check_attr_mutex;

cudaError_t raise_dyn_limit(const void* kern, DynLimit (&limits)[kDynLimitDevices], size_t dyn) {
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    const unsigned long long ctx = current_context_key();
    std::lock_guard<std::mutex> lock(g_check_attr_mutex);
    DynLimit dflt;
    DynLimit& c = (dev >= 0 && dev < kDynLimitDevices) ? limits[dev] : dflt;
    if (!ctx || c.ctx != ctx) {
        c = DynLimit{};
        c.ctx = ctx;
    }
    if ((int)dyn > c.max_dyn) {
        if ((e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)dyn)) != cudaSuccess)
            return e;
        c.max_dyn = (int)dyn;
    }
    return cudaSuccess;
}

static DynLimit g_check_limit[6][kDynLimitDevices];  // 2 * (pass size: CW, CW/2, CW/4) + full

template <int CW>
static cudaError_t check_option(int full_sweep, int J, int S, int K, int Q, int blob_cap, CheckLaunch& o) {
    const size_t cc = (size_t)cc_smem_bytes(J, S, K, Q, CW);
    size_t dyn = cc + (size_t)blob_cap;
    if (dyn + kStaticSmem > device_max_smem()) {
        blob_cap = 0;
        dyn = cc;
    }
    auto kern = full_sweep ? check_kernel<CW, true> : check_kernel<CW, false>;
    constexpr int size_idx = CW == PRRTC_CHECK_CW ? 0 : (2 * CW == PRRTC_CHECK_CW ? 1 : 2);
    cudaError_t e = raise_dyn_limit(reinterpret_cast<const void*>(kern), g_check_limit[2 * size_idx + (full_sweep ? 1 : 0)], dyn);
    if (e != cudaSuccess) return e;
    int per_sm = 0;
    if ((e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, 128, dyn)) != cudaSuccess) return e;
    o.cw = CW;
    o.blob_cap = blob_cap;
    o.per_sm = per_sm;
    o.dyn = dyn;
    return cudaSuccess;
}

template <int CW>
static void check_go(const CheckLaunch& o, int full_sweep, const unsigned char* blob, const int32_t* pairs, int J,
                     int S, int K, int Q, int dim, const float* configs, int n, int32_t* verdicts, cudaStream_t st,
                     const PcView& cloud) {
    const long long chunks = (n + CW - 1) / CW;
    const long long grid = std::min<long long>(chunks, (long long)std::max(o.per_sm, 1) * device_sm_count());
    auto kern = full_sweep ? check_kernel<CW, true> : check_kernel<CW, false>;
    kern<<<(unsigned)grid, 128, o.dyn, st>>>(blob, o.blob_cap, pairs, J, S, K, Q, dim, configs, n, verdicts, cloud);
}

// The culled checker: warps of their own, CW configurations at a time
// (warp_check), the scene staged per CTA.
//
// Bound by instruction issue (75% of the issue slots, 22 warps per SM),
// not by memory: of the time of 2^20 random tabletop configurations (79% in
// collision) link frames take a quarter, self items a third, the links'
// primitives the rest.  80 registers per thread and 24 warps per SM measured 15%
// faster than 128 and 16; world links before self items 6% faster here but 20%
// slower on uneven scenes.  Against the general checker: 2^20 tabletop
// configurations 2112 -> 773 us (gated 2321 -> 830), uneven scene 2052 -> 805 us
// (gated 1301 -> 825), 60,000 dual-arm configurations 976 -> 253 us (gated 1333).
//
// A scene that is not culled (BlobHeader::cull: groups that do not cover the
// spheres, ...) takes the general checker in the same shared memory, by the whole
// CTA: up to CW configurations at a time, as many as the launch found room for, and
// fewer where there are CTAs to share them; FULL as the general launch would sweep.
template <bool FULL>
static __device__ __noinline__ void check_general(const unsigned char* blob, const int2* pairs, const PcView* pc,
                                                  unsigned char* smem, int CW, const float* configs, int n, int dim,
                                                  int32_t* verdicts) {
    Scene sc = scene_view(blob);
    sc.pairs = pairs;
    sc.pc = *pc;
    CW = min(CW, max(1, (int)((n + (long long)gridDim.x - 1) / gridDim.x)));
    const CcBufs B = cc_bufs(smem, sc.h->J, sc.h->S, sc.h->K, sc.h->Q, CW);
    if (threadIdx.x == 0) B.hit[0] = B.hit[1] = 0u;
    int par = 0;
    __syncthreads();
    for (long long c0 = (long long)blockIdx.x * CW; c0 < n; c0 += (long long)gridDim.x * CW) {
        const int nw = (int)min((long long)CW, n - c0);
        for (int i = threadIdx.x; i < nw * dim; i += blockDim.x) {
            const int w = i / dim, d = i - w * dim;
            B.q[w * kDimMax + d] = configs[(size_t)(c0 + w) * dim + d];
        }
        __syncthreads();
        const uint32_t hit = cc_chunk<FULL>(CtaGroup{}, sc, B, nw, false, par);
        for (int w = threadIdx.x; w < nw; w += blockDim.x) verdicts[c0 + w] = (hit >> w) & 1u;
    }
}

// Scenes of one launch: blockIdx.y of them, scene y's configurations being
// [offsets[y], offsets[y+1]) of n in all; offsets null: one scene.
struct CheckScenes {
    const int32_t* offsets;
    size_t blob_stride, pairs_stride;
};

// EDGES: the configurations are waypoints and `edges` their edges' flags (a form of
// its own: the tests of the flags cost bulk checks 1.6%).
template <bool EDGES>
__global__ void __launch_bounds__(256, 3) check_cull_kernel(const unsigned char* __restrict__ gblob, int blob_cap,
                                                            const int2* pairs, int J, int K, int dim, int CW,
                                                            const float* __restrict__ configs, int n,
                                                            int32_t* verdicts, PcView pc, CheckScenes scenes,
                                                            EdgeHits edges, int general_cw, int full_sweep) {
    extern __shared__ __align__(128) unsigned char dsm[];
    __shared__ __align__(8) uint64_t mbar;
    if (scenes.offsets) {
        const int lo = max(0, min(scenes.offsets[blockIdx.y], n)), hi = max(lo, min(scenes.offsets[blockIdx.y + 1], n));
        gblob += blockIdx.y * scenes.blob_stride;
        pairs += blockIdx.y * scenes.pairs_stride;
        configs += (size_t)lo * dim;
        verdicts += lo;
        n = hi - lo;
        if (n <= 0) return;
    }
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, n_warps = blockDim.x >> 5;
    const int bytes = min(reinterpret_cast<const BlobHeader*>(gblob)->used_bytes, blob_cap);
    if (tid == 0) mbar_init(&mbar);
    __syncthreads();
    uint32_t phase = 0;
    int* err = reinterpret_cast<int*>(const_cast<unsigned char*>(gblob) + offsetof(BlobHeader, error));
    if (!stage_blob(dsm, gblob, bytes, &mbar, phase, err, kBlobStagingTimeout, kWaitLimit)) {
        // the bulk copy did not arrive in time: copy the scene with plain loads
        for (int i = tid; i < bytes / 16; i += blockDim.x)
            reinterpret_cast<uint4*>(dsm)[i] = reinterpret_cast<const uint4*>(gblob)[i];
        __syncthreads();
    }
    Scene sc = scene_view(dsm);
    if (!sc.h->cull) {
        if (sc.h->enabled) {
            if (full_sweep) check_general<true>(dsm, pairs, &pc, dsm + blob_cap, general_cw, configs, n, dim, verdicts);
            else check_general<false>(dsm, pairs, &pc, dsm + blob_cap, general_cw, configs, n, dim, verdicts);
        } else {
            for (long long i = (long long)blockIdx.x * blockDim.x + tid; i < n; i += (long long)gridDim.x * blockDim.x)
                verdicts[i] = 0;
        }
        return;
    }
    sc.pairs = pairs;
    sc.pc = pc;
    const WarpBufs B = warp_bufs(dsm + blob_cap + warp * warp_check_bytes(J, K, CW), J, K, CW);
    // chunk index: warps of one CTA take neighbouring chunks
    for (long long c0 = ((long long)blockIdx.x * n_warps + warp) * CW; c0 < n; c0 += (long long)gridDim.x * n_warps * CW) {
        const int nw = (int)min((long long)CW, n - c0);
        if constexpr (EDGES) {
            if (__all_sync(0xffffffffu, lane >= nw || __ldcg(&edges.hit[(c0 + lane) / edges.G]) != 0)) {
                if (lane < nw) verdicts[c0 + lane] = 1;  // another waypoint has answered for the edge
                continue;
            }
        }
        for (int i = lane; i < nw * dim; i += 32) {
            const int w = i / dim, d = i - w * dim;
            B.q[w * kDimMax + d] = configs[c0 * dim + i];
        }
        __syncwarp();
        const unsigned hit = warp_check(sc, B, nw, CW);
        if (lane < nw) verdicts[c0 + lane] = (int)(hit >> lane & 1u);
        if constexpr (EDGES) {
            if (lane < nw && hit >> lane & 1u) edges.hit[(c0 + lane) / edges.G] = 1;
        }
        __syncwarp();
    }
}

// Limits of check_cull_kernel in one device's CUDA context: its largest dynamic
// shared memory so far and what decides residency, read once.
struct CullCheckAttrs {
    unsigned long long ctx = 0ull;
    int max_dyn = -1, regs = 0, sm_smem = 0, sms = 0;
};
static CullCheckAttrs g_cull_check_attr[2][kDynLimitDevices];

// Launches the culled checker, or returns cudaErrorInvalidConfiguration when
// its buffers do not fit (the caller then takes the general one).
static cudaError_t launch_check_cull(const unsigned char* blob, int blob_cap, const int32_t* pairs, int J, int S, int K,
                                     int Q, int dim, const float* configs, int n, int full_sweep, int32_t* verdicts,
                                     cudaStream_t st, const PcView& pc, const CheckScenes& scenes, int n_scenes,
                                     const EdgeHits& edges) {
    auto kern = edges.hit ? check_cull_kernel<true> : check_cull_kernel<false>;
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    const unsigned long long ctx = current_context_key();
    std::lock_guard<std::mutex> lock(g_check_attr_mutex);
    CullCheckAttrs dflt;
    CullCheckAttrs& a = dev >= 0 && dev < kDynLimitDevices ? g_cull_check_attr[edges.hit ? 1 : 0][dev] : dflt;
    if (!ctx || a.ctx != ctx) {
        a = CullCheckAttrs{};
        cudaFuncAttributes fa;
        if ((e = cudaFuncGetAttributes(&fa, kern)) != cudaSuccess ||
            (e = cudaDeviceGetAttribute(&a.sm_smem, cudaDevAttrMaxSharedMemoryPerMultiprocessor, dev)) != cudaSuccess)
            return e;
        a.regs = (fa.numRegs + 7) & ~7;
        a.sms = device_sm_count();
        a.ctx = ctx;
    }
    const int max_dyn = (int)(device_max_smem() - kStaticSmem);
    const int general = cc_smem_bytes(J, S, K, Q, 8);  // a scene that is not culled
    int best_cw = 0, best_wpc = 0, best_warps = 0, best_dyn = 0;
    const int least = pc.n > 0 ? 1 : 4;  // configurations per warp
    for (int cw = 32; cw >= least; cw /= 2) {
        for (int wpc = 4; wpc <= 8; wpc *= 2) {
            const int dyn = blob_cap + std::max(wpc * warp_check_bytes(J, K, cw), general);
            if (dyn > max_dyn) continue;
            const int per_sm = std::min(a.sm_smem / (dyn + 1024 + (int)kStaticSmem), 65536 / (a.regs * 32 * wpc));
            const int warps = std::min(per_sm * wpc, 24);
            if (warps > best_warps) { best_cw = cw; best_wpc = wpc; best_warps = warps; best_dyn = dyn; }
        }
    }
    if (best_warps == 0) return cudaErrorInvalidConfiguration;
    // With a cloud a configuration is 27 cells and their points per sphere until one
    // hits: one per warp, so that an edge's other waypoints find its flag set and
    // uneven configurations spread (3384 edges x 33 waypoints against 41,277 points:
    // 708 us; with 2 per warp 750, 4 1160, 16 2870, and 3070 without flags; 4000 x 8
    // against 1000 points: 283 us, with 8 per warp 530).
    int cw = pc.n > 0 ? 1 : best_cw, wpc = best_wpc;
    while (cw > least && (long long)cw * a.sms * best_warps > n) cw /= 2;  // fewer per warp before warps go idle
    const long long chunks = n / cw + n_scenes;  // of all scenes, about
    while (wpc > 1 && chunks < (long long)a.sms * wpc) wpc /= 2;
    int dyn = blob_cap + std::max(wpc * warp_check_bytes(J, K, cw), general);
    const int per_sm = std::max(1, std::min(a.sm_smem / (dyn + 1024 + (int)kStaticSmem), 65536 / (a.regs * 32 * wpc)));
    // the general checker's pass: as large as the shared memory of that many CTAs takes, but
    // not where a cloud is read through what is left of it as L1 (4000 configurations
    // against 200,000 points 683 us, 840 with the larger pass)
    int general_cw = 8;
    while (pc.n == 0 && general_cw < 32 &&
           blob_cap + cc_smem_bytes(J, S, K, Q, 2 * general_cw) <= std::min(max_dyn, a.sm_smem / per_sm - 1024 - (int)kStaticSmem))
        general_cw *= 2;
    dyn = std::max(dyn, blob_cap + cc_smem_bytes(J, S, K, Q, general_cw));
    if (std::max(dyn, best_dyn) > a.max_dyn) {
        if ((e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                      std::max(dyn, best_dyn))) != cudaSuccess)
            return e;
        a.max_dyn = std::max(dyn, best_dyn);
    }
    const long long resident = (long long)a.sms * per_sm;
    // the scenes' configurations may be spread unevenly: each gets the CTAs for
    // twice its even share, and a CTA strides over what is left
    const long long each = n_scenes == 1 ? (chunks + wpc - 1) / wpc : (2 * chunks / n_scenes + wpc - 1) / wpc;
    const long long grid = std::max(1ll, std::min(each, n_scenes == 1 ? resident : (2 * resident + n_scenes - 1) / n_scenes));
    kern<<<dim3((unsigned)grid, (unsigned)n_scenes), wpc * 32, dyn, st>>>(
        blob, blob_cap, reinterpret_cast<const int2*>(pairs), J, K, dim, cw, configs, n, verdicts, pc, scenes, edges,
        general_cw, full_sweep);
    return cudaGetLastError();
}

// Passes of PRRTC_CHECK_CW configurations, unless their buffers leave fewer
// than PRRTC_CHECK_MINBLOCKS CTAs per SM (large robots: the sphere centres and
// link frames of a pass grow with S and J); then half or a quarter as many
// configurations per pass, whichever keeps the most CTAs resident (the larger
// pass on a tie).  The dual arm with 120 spheres and 18 joints fits one CTA
// per SM at 32 configurations per pass, three at 16 and four at 8: 44.0 M
// checks/s at 32, 65.4 M at 8.
cudaError_t launch_check(const unsigned char* blob, int blob_cap, const int32_t* pairs, int J, int S, int K,
                         int Q, int dim, const float* configs, int n, int full_sweep, bool cull, int32_t* verdicts,
                         cudaStream_t st, const PcView* pc, const EdgeHits& edges) {
    if (n <= 0) return cudaSuccess;
    const PcView cloud = pc ? *pc : PcView{nullptr, nullptr, 0, 0, 0.0f, 0.0f};
    constexpr int CW = PRRTC_CHECK_CW;
    CheckLaunch best, o;
    if (cull) {
        const cudaError_t e = launch_check_cull(blob, blob_cap, pairs, J, S, K, Q, dim, configs, n, full_sweep, verdicts, st,
                                                 cloud, CheckScenes{nullptr, 0, 0}, 1, edges);
        if (e != cudaErrorInvalidConfiguration) return e;
    }
    cudaError_t e = check_option<CW>(full_sweep, J, S, K, Q, blob_cap, best);
    if (e != cudaSuccess) return e;
    if constexpr (CW / 2 >= 8) {
        if (best.per_sm < PRRTC_CHECK_MINBLOCKS) {
            if ((e = check_option<CW / 2>(full_sweep, J, S, K, Q, blob_cap, o)) != cudaSuccess) return e;
            if (o.per_sm > best.per_sm) best = o;
        }
    }
    if constexpr (CW / 4 >= 8) {
        if (best.per_sm < PRRTC_CHECK_MINBLOCKS) {
            if ((e = check_option<CW / 4>(full_sweep, J, S, K, Q, blob_cap, o)) != cudaSuccess) return e;
            if (o.per_sm > best.per_sm) best = o;
        }
    }
    if constexpr (CW / 2 >= 8) {
        if (best.cw == CW / 2) {
            check_go<CW / 2>(best, full_sweep, blob, pairs, J, S, K, Q, dim, configs, n, verdicts, st, cloud);
            return cudaGetLastError();
        }
    }
    if constexpr (CW / 4 >= 8) {
        if (best.cw == CW / 4) {
            check_go<CW / 4>(best, full_sweep, blob, pairs, J, S, K, Q, dim, configs, n, verdicts, st, cloud);
            return cudaGetLastError();
        }
    }
    check_go<CW>(best, full_sweep, blob, pairs, J, S, K, Q, dim, configs, n, verdicts, st, cloud);
    return cudaGetLastError();
}

cudaError_t launch_check_batch(const unsigned char* blobs, size_t blob_stride, const int32_t* pairs,
                               size_t pairs_stride, int n_scenes, int J, int S, int K, int Q, int dim,
                               const float* configs, const int32_t* offsets, int n, int full_sweep, int32_t* verdicts,
                               cudaStream_t st) {
    return launch_check_cull(blobs, (int)blob_stride, pairs, J, S, K, Q, dim, configs, n, full_sweep, verdicts, st,
                             PcView{nullptr, nullptr, 0, 0, 0.0f, 0.0f}, CheckScenes{offsets, blob_stride, pairs_stride},
                             n_scenes, EdgeHits{});
}

// ============================================================================ FK

// A tile of kFkTile configurations per CTA: the joint records once, the local
// transforms a (configuration, joint) per thread, then the chain in joint order,
// where row r of a frame needs row r of its parent only, so three lanes of a warp
// take a configuration, a row each, and write the frame over its local
// transform; the tile leaves in one coalesced copy, in output frame order (frame
// k = sorted joint topo_inv[k]).  Shared-memory rows are one 16-byte vector longer
// than J frames, which spreads a warp's configurations over the banks.
//
// Bound by shared-memory traffic and the chain of joints (48 B written per frame
// leave at 1.8 TB/s).  65,537 configurations x 18 joints (56.6 MB): 130 -> 31 us
// against a configuration per thread with its frames in local memory and 48 B
// stores 864 B apart; tiles of 20, or 256 threads, measured 33 and 37 us.
constexpr int kFkTile = 40, kFkThreads = 128;  // 10 configurations x 3 rows per warp

__host__ __device__ inline int fk_smem_bytes(int J) { return J * (int)sizeof(JointRec) + kFkTile * (J * 12 + 4) * 4 + J * 4; }

__global__ void __launch_bounds__(kFkThreads) fk_kernel(FkTables t, int dim, const float* __restrict__ configs, int n,
                                                        float* __restrict__ frames, bool vec) {
    extern __shared__ __align__(16) unsigned char fsm[];
    const int tid = threadIdx.x, J = t.J, row = J * 12 + 4;
    JointRec* jr = reinterpret_cast<JointRec*>(fsm);
    float* L = reinterpret_cast<float*>(jr + J);
    int* src = reinterpret_cast<int*>(L + kFkTile * row);  // joint of output frame k
    for (int j = tid; j < J; j += kFkThreads) {
        jr[j] = make_joint_rec(j, t.ptf, t.twists, t.parent, t.act, t.mmul, t.moff, t.mact, dim);
        const int s = t.topo_inv ? t.topo_inv[j] : j;
        src[j] = s < 0 || s >= J ? j : s;
    }
    __syncthreads();
    const float inv_j = 1.0f / (float)J, inv_v = 1.0f / (float)(3 * J);
    for (long long c0 = (long long)blockIdx.x * kFkTile; c0 < n; c0 += (long long)gridDim.x * kFkTile) {
        const int nc = (int)min((long long)kFkTile, n - c0);
        for (int i = tid; i < nc * J; i += kFkThreads) {
            const int c = (int)(((float)i + 0.5f) * inv_j), j = i - c * J;  // i / J (i is small)
            float X[12];
            joint_local(jr[j], joint_value(jr[j], configs + (c0 + c) * dim), X);
            float4* o = reinterpret_cast<float4*>(L + c * row + j * 12);
            o[0] = make_float4(X[0], X[1], X[2], X[3]);
            o[1] = make_float4(X[4], X[5], X[6], X[7]);
            o[2] = make_float4(X[8], X[9], X[10], X[11]);
        }
        __syncthreads();
        {
            const int lane = tid & 31, c = (tid >> 5) * 10 + lane / 3, r = lane - lane / 3 * 3;
            const bool on = lane < 30 && c < nc;
            float* base = L + (on ? c : 0) * row;
            float x = 0.0f, y = 0.0f, z = 0.0f, o = 0.0f;  // row r of frame `have`
            int have = -1;
            for (int j = 0; j < J; ++j) {
                const int p = jr[j].idx.x;
                if (p < 0 || p >= j) continue;  // a root's frame is its local transform
                float* l = base + j * 12;
                if (p != have) {
                    const float* a = base + p * 12;
                    x = a[3 * r]; y = a[3 * r + 1]; z = a[3 * r + 2]; o = a[9 + r];
                }
                const float4* v = reinterpret_cast<const float4*>(l);
                const float4 l0 = v[0], l1 = v[1], l2 = v[2];
                const float nx = fmaf(x, l0.x, fmaf(y, l0.w, z * l1.z)), ny = fmaf(x, l0.y, fmaf(y, l1.x, z * l1.w));
                const float nz = fmaf(x, l0.z, fmaf(y, l1.y, z * l2.x)), no = fmaf(x, l2.y, fmaf(y, l2.z, fmaf(z, l2.w, o)));
                __syncwarp();  // all three rows have read the local transform
                if (on) {
                    l[3 * r] = nx; l[3 * r + 1] = ny; l[3 * r + 2] = nz;
                    l[9 + r] = no;
                }
                x = nx; y = ny; z = nz; o = no;
                have = j;
            }
        }
        __syncthreads();
        float* out = frames + c0 * J * 12;
        for (int i = tid; i < nc * J * 3; i += kFkThreads) {  // a quarter frame each
            const int c = (int)(((float)i + 0.5f) * inv_v), e = i - c * J * 3, k = e / 3;
            const float4 w = reinterpret_cast<const float4*>(L + c * row + src[k] * 12)[e - 3 * k];
            if (vec) {
                reinterpret_cast<float4*>(out)[i] = w;
            } else {
                out[4 * i] = w.x; out[4 * i + 1] = w.y; out[4 * i + 2] = w.z; out[4 * i + 3] = w.w;
            }
        }
        __syncthreads();
    }
}

cudaError_t launch_fk(const FkTables& t, int dim, const float* configs, int n, float* frames, cudaStream_t st) {
    if (n <= 0 || t.J <= 0) return cudaSuccess;
    const int smem = fk_smem_bytes(t.J);
    cudaError_t e;
    static DynLimit limit[kDynLimitDevices];
    if (smem > 48 * 1024 &&
        (e = raise_dyn_limit(reinterpret_cast<const void*>(fk_kernel), limit, (size_t)smem)) != cudaSuccess)
        return e;
    const long long tiles = ((long long)n + kFkTile - 1) / kFkTile;
    fk_kernel<<<(unsigned)std::min<long long>(tiles, 8ll * device_sm_count()), kFkThreads, smem, st>>>(
        t, dim, configs, n, frames, (reinterpret_cast<uintptr_t>(frames) & 15) == 0);
    return cudaGetLastError();
}

// ============================================================================ Halton

__global__ void halton_kernel(int explorer, int n, int dim, const float* lo, const float* hi, float* out) {
    if (threadIdx.x != 0 || blockIdx.x != 0) return;
    int order[16], st[kDimMax];
    prime_order(explorer, order);
    for (int d = 0; d < kDimMax; ++d) st[d] = 1;
    float row[kDimMax];
    for (int i = 0; i < n; ++i) {
        halton_sample(order, st, dim, lo, hi, row);
        for (int d = 0; d < dim; ++d) out[(size_t)i * dim + d] = row[d];
    }
}

cudaError_t launch_halton(int explorer, int n, int dim, const float* lo, const float* hi, float* out,
                          cudaStream_t st) {
    if (n <= 0) return cudaSuccess;
    halton_kernel<<<1, 32, 0, st>>>(explorer, n, dim, lo, hi, out);
    return cudaGetLastError();
}

// ============================================================================ planner rules

// Tree-side choice of the planner (choose_tree) for n cases at once: explorer
// bid = blockIdx.x of nblocks = gridDim.x, case c with tree sizes sizes[2c],
// sizes[2c+1], the explorer's iteration count local_iter[c] and its mode-2 side
// vamp_in[c * nblocks + bid]; writes the chosen tree and the updated side.
__global__ void choose_tree_kernel(int mode, int n, const int32_t* sizes, const int32_t* local_iter,
                                   const int32_t* vamp_in, float tree_ratio, int32_t* tree_out, int32_t* vamp_out) {
    const int bid = blockIdx.x, nblocks = gridDim.x;
    for (int c = threadIdx.x; c < n; c += blockDim.x) {
        int vamp = vamp_in[(size_t)c * nblocks + bid];
        const int t = choose_tree(mode, local_iter[c], bid, nblocks, sizes[2 * c], sizes[2 * c + 1], tree_ratio, vamp);
        tree_out[(size_t)c * nblocks + bid] = t;
        vamp_out[(size_t)c * nblocks + bid] = vamp;
    }
}

cudaError_t launch_choose_tree(int mode, int n, const int32_t* sizes, const int32_t* local_iter,
                               const int32_t* vamp_in, int nblocks, float tree_ratio, int32_t* tree_out,
                               int32_t* vamp_out, cudaStream_t st) {
    if (n <= 0) return cudaSuccess;
    choose_tree_kernel<<<nblocks, 128, 0, st>>>(mode, n, sizes, local_iter, vamp_in, tree_ratio, tree_out, vamp_out);
    return cudaGetLastError();
}

// Dynamic-domain radius updates of the planner (radius_shrink / radius_grow):
// update i is op[i] (0 shrink, 1 grow) on radii[idx[i]].  Concurrent: one
// thread per update, so updates of one index contend on its CAS loop;
// sequential: one thread applies them in order.
__global__ void radius_update_kernel(float* radii, const int32_t* idx, const int32_t* op, int n, float alpha,
                                     float r0, float rmin, int sequential, int32_t* err) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (sequential) {
        if (i != 0) return;
        for (int k = 0; k < n; ++k) {
            if (op[k] == 0) radius_shrink(radii, idx[k], alpha, r0, rmin, err);
            else radius_grow(radii, idx[k], alpha, err);
        }
        return;
    }
    if (i >= n) return;
    if (op[i] == 0) radius_shrink(radii, idx[i], alpha, r0, rmin, err);
    else radius_grow(radii, idx[i], alpha, err);
}

cudaError_t launch_radius_update(float* radii, const int32_t* idx, const int32_t* op, int n, float alpha, float r0,
                                 float rmin, int sequential, int32_t* err, cudaStream_t st) {
    if (n <= 0) return cudaSuccess;
    radius_update_kernel<<<sequential ? 1 : (n + 127) / 128, sequential ? 32 : 128, 0, st>>>(
        radii, idx, op, n, alpha, r0, rmin, sequential, err);
    return cudaGetLastError();
}

// ============================================================================ FP32 probe

// 8 independent FFMA chains per thread: the FP32 pipe stays busy without
// dependency stalls.  2 * 8 * iters flops per thread.
__global__ void fp32_probe_kernel(int iters, float* sink) {
    float a0 = threadIdx.x * 1e-7f, a1 = a0 + 1e-7f, a2 = a0 + 2e-7f, a3 = a0 + 3e-7f;
    float a4 = a0 + 4e-7f, a5 = a0 + 5e-7f, a6 = a0 + 6e-7f, a7 = a0 + 7e-7f;
    const float m = 0.999999f, c = 1e-7f;
    for (int i = 0; i < iters; ++i) {
#pragma unroll
        for (int k = 0; k < 16; ++k) {
            a0 = fmaf(a0, m, c); a1 = fmaf(a1, m, c); a2 = fmaf(a2, m, c); a3 = fmaf(a3, m, c);
            a4 = fmaf(a4, m, c); a5 = fmaf(a5, m, c); a6 = fmaf(a6, m, c); a7 = fmaf(a7, m, c);
        }
    }
    const float r = a0 + a1 + a2 + a3 + a4 + a5 + a6 + a7;
    if (r == 12345.0f) sink[blockIdx.x] = r;  // never true; keeps the chains live
}

cudaError_t launch_fp32_probe(int blocks, int threads, int iters, float* sink, cudaStream_t st) {
    fp32_probe_kernel<<<blocks, threads, 0, st>>>(iters, sink);
    return cudaGetLastError();
}

// The same with packed FP32 (fma.rn.f32x2, sm_100): 8 independent chains of two
// lanes each per thread, 2 * 2 * 8 * 16 * iters flops per thread.  Measures
// whether one packed instruction delivers two FP32 FMAs per lane per issue
// slot, i.e. which FP32 peak a kernel built from packed FMAs runs against.
__device__ __forceinline__ unsigned long long pack2(float lo, float hi) {
    unsigned long long r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
    return r;
}

__global__ void fp32x2_probe_kernel(int iters, float* sink) {
    const float b = threadIdx.x * 1e-7f;
    unsigned long long a[8];
#pragma unroll
    for (int k = 0; k < 8; ++k) a[k] = pack2(b + (2 * k) * 1e-7f, b + (2 * k + 1) * 1e-7f);
    const unsigned long long m = pack2(0.999999f, 0.999999f), c = pack2(1e-7f, 1e-7f);
    for (int i = 0; i < iters; ++i) {
#pragma unroll
        for (int u = 0; u < 16; ++u) {
#pragma unroll
            for (int k = 0; k < 8; ++k) asm volatile("fma.rn.f32x2 %0, %0, %1, %2;" : "+l"(a[k]) : "l"(m), "l"(c));
        }
    }
    float r = 0.0f;
#pragma unroll
    for (int k = 0; k < 8; ++k) {
        float lo, hi;
        asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(a[k]));
        r += lo + hi;
    }
    if (r == 12345.0f) sink[blockIdx.x] = r;  // never true; keeps the chains live
}

cudaError_t launch_fp32x2_probe(int blocks, int threads, int iters, float* sink, cudaStream_t st) {
    fp32x2_probe_kernel<<<blocks, threads, 0, st>>>(iters, sink);
    return cudaGetLastError();
}

}  // namespace prrtc
