// planner.cu -- scene packing, the pRRTC explorer kernel (plain and persistent
// batched launch), output initialisation, device-clock timing and path
// extraction.  sm_100a.
//
// Algorithm: the reference's prrtc_planner_kernel (cuda-rrtc/CUDA/
// prrtc_planner.cu:675-1066).  Each explorer samples its Halton stream, picks a
// tree by balance mode, finds the nearest node, extends by step_size, checks the
// edge, inserts, then connects toward the other tree in ceil(d/step) checked
// sub-edges; the first explorer whose connect completes solves the problem.
//
// B200 design:
//  * an explorer is a CTA of 32-512 threads; nearest neighbour is a CTA scan of
//    the SoA tree with 128-bit L2-coherent loads and an argmin by integer minima
//    (ties to the lowest index);
//  * an edge's waypoints are checked by the whole CTA against the scene staged in
//    shared memory by one bulk TMA copy: link frames, a bound per link over the
//    pass, then only the links, waypoints and primitives that touch
//    (prrtc_cull.cuh); robots without a coarse model or of more than 32 joints
//    take the general check of every pair (prrtc_device.cuh);
//  * tree slots are pre-filled with NaN, so a reader scanning [0, tree_size)
//    never uses a half-written node (its squared distance is NaN and loses every
//    comparison); this replaces the reference's `completed` counter as the scan
//    bound, whose count-not-prefix semantics let a reader see an unwritten slot;
//  * the batched form is one persistent launch: CTAs pop (problem, explorer)
//    slots from a queue ordered by the caller (longest problems first).
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

#ifndef PRRTC_EXPLORE_MINBLOCKS
#define PRRTC_EXPLORE_MINBLOCKS 2  // resident 256-thread explorer CTAs per SM the register allocation must allow
#endif
constexpr int kWideThreads = 512;  // explorer size of the wide form (one CTA per SM)

// ============================================================================ pack

size_t blob_stride(const PackSrc& s) {
    const BlobLayout L = blob_layout(s.J, s.S, s.K, s.Q, s.sp_max, s.ws_max, s.wc_max, s.wb_max, s.wh_max);
    return ((size_t)L.bytes + 255) & ~(size_t)255;
}

__device__ __forceinline__ int clampi(int x, int lo, int hi) { return x < lo ? lo : (x > hi ? hi : x); }

constexpr float kCullStretchMax = 1e8f;  // box axes and normals of a length of up to 10,000 (squared) are culled
constexpr int kPackThreads = 512;

// Exclusive prefix of one value per thread over a CTA of kPackThreads, plus the
// CTA total.
__device__ __forceinline__ int pack_exclusive_scan(int v, int* warp_sums, int& total) {
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    int inc = v;
#pragma unroll
    for (int off = 1; off < 32; off <<= 1) {
        const int o = __shfl_up_sync(0xffffffffu, inc, off);
        if (lane >= off) inc += o;
    }
    if (lane == 31) warp_sums[warp] = inc;
    __syncthreads();
    int base = 0, sum = 0;
#pragma unroll
    for (int w = 0; w < kPackThreads / 32; ++w) {
        const int x = warp_sums[w];
        base += w < warp ? x : 0;
        sum += x;
    }
    __syncthreads();
    total = sum;
    return base + inc - v;
}

// One CTA per problem.  Converts the reference collision_context buffers into
// the packed blob (see prrtc_device.cuh).
//
// Bound by the latency of its dependent loads, not by bytes (a few KB per
// problem), so every table goes in one pass with one row per thread (rows of
// different tables on different warps, their loads in flight together), the
// dense-block test reads its pairs with a warp per coarse pair from operands
// already in shared memory, and the item lists are written at offsets from a
// scan.  One problem, cold caches: 25.5 -> 9.5 us (arm, tabletop scene) and
// 55.8 -> 15.6 us (dual arm, large scene) against the tables one after the
// other, one thread per coarse pair walking its 64 pairs and one thread writing
// the lists (16 warps: the dual arm's 131 coarse pairs take 9 rounds).  512
// problems at once: 23.3 -> 21.0 us.
__global__ void __launch_bounds__(kPackThreads) pack_kernel(PackSrc s, unsigned char* blobs, size_t stride, int cap) {
    __shared__ int warp_sums[kPackThreads / 32];
    __shared__ int4 t_blk[kPackThreads];   // (a0, na, b0, nb) of a tile of coarse pairs; na = 0: not a block
    __shared__ int t_r0[kPackThreads];
    __shared__ int t_dense[kPackThreads];
    __shared__ unsigned s_scale;  // bits of the largest coordinate size (L1) of a world primitive
    __shared__ int s_cull;
    const int b = blockIdx.x, tid = threadIdx.x, T = blockDim.x;
    unsigned char* blob = blobs + (size_t)b * stride;
    BlobHeader* h = reinterpret_cast<BlobHeader*>(blob);
    const int Ns = s.ws_cnt ? clampi(s.ws_cnt[b], 0, s.ws_max) : s.ws_max;
    const int Nc = s.wc_cnt ? clampi(s.wc_cnt[b], 0, s.wc_max) : s.wc_max;
    const int Nb = s.wb_cnt ? clampi(s.wb_cnt[b], 0, s.wb_max) : s.wb_max;
    const int Nh = s.wh_cnt ? clampi(s.wh_cnt[b], 0, s.wh_max) : s.wh_max;
    const int P = s.sp_cnt ? clampi(s.sp_cnt[b], 0, s.sp_max) : s.sp_max;
    // a table is batched [B, max, feat] exactly when its count pointer is set
    const float* ws = s.ws + (s.ws_cnt ? (size_t)b * s.ws_max * 4 : 0);
    const float* wc = s.wc + (s.wc_cnt ? (size_t)b * s.wc_max * 7 : 0);
    const float* wbx = s.wb + (s.wb_cnt ? (size_t)b * s.wb_max * 15 : 0);
    const float* wh = s.wh + (s.wh_cnt ? (size_t)b * s.wh_max * 6 : 0);
    const int* __restrict__ sp = s.sp + (s.sp_cnt ? (size_t)b * s.sp_max * 2 : 0);
    const int J = s.J, S = s.S, K = s.K, Q = s.Q;
    const BlobLayout L = blob_layout(J, S, K, Q, s.sp_max, s.ws_max, s.wc_max, s.wb_max, s.wh_max);

    // reference enable rules (prrtc_planner.cu:505-506, 1156-1157, 1173, 741-743)
    const bool enabled =
        J > 0 && J <= kMaxJoints && S > 0 && (Ns > 0 || Nc > 0 || Nb > 0 || Nh > 0 || P > 0 || s.has_cloud);
    const bool coarse_ok = K > 0 && K <= kMaxLinks && s.foff != nullptr;
    bool gated = enabled && coarse_ok && (s.mode == 2 || (s.mode == 3 && J <= 16));
    if (tid == 0) {
        s_scale = 0u;
        s_cull = enabled && coarse_ok && J <= 32 && !(s.mode == 1 && !(s.margin >= 0.0f)) && s.foff[0] == 0 && s.foff[K] == S;
    }
    __syncthreads();
    auto note_size = [&](float l1) { atomicMax(&s_scale, __float_as_uint(l1) & 0x7fffffffu); };  // NaN orders above all

    JointRec* jr = reinterpret_cast<JointRec*>(blob + L.o_joint);
    float4* sph = reinterpret_cast<float4*>(blob + L.o_sph);
    int* sfr = reinterpret_cast<int*>(blob + L.o_sfr);
    float4* grp = reinterpret_cast<float4*>(blob + L.o_grp);
    float4* o_ws = reinterpret_cast<float4*>(blob + L.o_ws);
    float4* o_wc = reinterpret_cast<float4*>(blob + L.o_wc);
    float4* o_wb = reinterpret_cast<float4*>(blob + L.o_wb);
    float4* o_wh = reinterpret_cast<float4*>(blob + L.o_wh);
    int2* cp = reinterpret_cast<int2*>(blob + L.o_cpair);
    // rows of every table in one index space, each table starting at a multiple
    // of 32 so that a warp holds rows of one table
    const int e0 = (J + 31) & ~31, e1 = e0 + ((S + 31) & ~31), e2 = e1 + ((K + 31) & ~31), e3 = e2 + ((Ns + 31) & ~31),
              e4 = e3 + ((Nc + 31) & ~31), e5 = e4 + ((Nb + 31) & ~31), e6 = e5 + ((Nh + 31) & ~31), e7 = e6 + Q;
    for (int r = tid; r < e7; r += T) {
        if (r < e0) {
            if (r < J) jr[r] = make_joint_rec(r, s.ptf, s.twists, s.parent, s.act, s.mmul, s.moff, s.mact, s.dim);
        } else if (r < e1) {
            const int i = r - e0;
            if (i < S) {
                sph[i] = make_float4(s.sloc[i * 3], s.sloc[i * 3 + 1], s.sloc[i * 3 + 2], s.srad[i]);
                const int li = s.sli[i];
                int f = (li >= 0 && li < J) ? (s.topo_inv ? s.topo_inv[li] : li) : -1;
                sfr[i] = (f >= 0 && f < J) ? f : -1;
            }
        } else if (r < e2) {
            const int k = r - e1;
            if (k < K) {
                grp[2 * k] = make_float4(s.cloc[k * 3], s.cloc[k * 3 + 1], s.cloc[k * 3 + 2], s.crad[k]);
                const int li = s.cli[k];
                int f = (li >= 0 && li < J) ? (s.topo_inv ? s.topo_inv[li] : li) : -1;
                if (f >= J) f = -1;
                const int s0 = s.foff ? clampi(s.foff[k], 0, S) : 0;
                const int s1 = s.foff ? clampi(s.foff[k + 1], 0, S) : 0;
                grp[2 * k + 1] = make_float4(__int_as_float(f), __int_as_float(s0), __int_as_float(s1), 0.0f);
            }
        } else if (r < e3) {  // world primitives, pre-conditioned for the FMA-form tests (prrtc_device.cuh)
            const int i = r - e2;
            if (i < Ns) {
                const float x = ws[i * 4], y = ws[i * 4 + 1], z = ws[i * 4 + 2], rad = ws[i * 4 + 3];
                note_size(fabsf(x) + fabsf(y) + fabsf(z) + fabsf(rad));
                o_ws[2 * i] = make_float4(-2.0f * x, -2.0f * y, -2.0f * z, -2.0f * rad);
                o_ws[2 * i + 1] = make_float4(x, y, z, fmaf(x, x, fmaf(y, y, fmaf(z, z, -rad * rad))));
            }
        } else if (r < e4) {
            const int i = r - e3;
            if (i < Nc) {
                const float* c = &wc[i * 7];
                const float dx = c[3] - c[0], dy = c[4] - c[1], dz = c[5] - c[2];
                note_size(fabsf(c[0]) + fabsf(c[1]) + fabsf(c[2]) + fabsf(dx) + fabsf(dy) + fabsf(dz) + fabsf(c[6]));
                const float l2 = dx * dx + dy * dy + dz * dz;
                const float il2 = l2 > 0.0f ? 1.0f / l2 : 0.0f;
                const float px = dx * il2, py = dy * il2, pz = dz * il2;
                o_wc[3 * i] = make_float4(c[0], c[1], c[2], c[6]);
                o_wc[3 * i + 1] = make_float4(px, py, pz, -(px * c[0] + py * c[1] + pz * c[2]));
                o_wc[3 * i + 2] = make_float4(dx, dy, dz, 0.0f);
            }
        } else if (r < e5) {
            const int i = r - e4;
            if (i < Nb) {
                const float* c = &wbx[i * 15];
#pragma unroll
                for (int k = 0; k < 3; ++k) {
                    const float ax = c[3 + 3 * k], ay = c[4 + 3 * k], az = c[5 + 3 * k];
                    const float off = -(ax * c[0] + ay * c[1] + az * c[2]);
                    o_wb[4 * i + k] = make_float4(ax * kBoxInv, ay * kBoxInv, az * kBoxInv, off * kBoxInv);
                }
                // how much longer than its argument a vector along the axes can be (their largest singular
                // value, bounded by the row sums of A A^T; sheared and long axes cull by a larger sphere)
                float rows[3] = {0.0f, 0.0f, 0.0f};
#pragma unroll
                for (int k = 0; k < 9; ++k) {
                    const float* u = c + 3 + 3 * (k / 3);
                    const float* v = c + 3 + 3 * (k % 3);
                    rows[k / 3] += fabsf(u[0] * v[0] + u[1] * v[1] + u[2] * v[2]);
                }
                const float stretch = fmaxf(1.0f, 1.00001f * sqrtf(fmaxf(rows[0], fmaxf(rows[1], rows[2]))));
                const bool ok = rows[0] <= kCullStretchMax && rows[1] <= kCullStretchMax && rows[2] <= kCullStretchMax;
                note_size(fabsf(c[0]) + fabsf(c[1]) + fabsf(c[2]) + fabsf(c[12]) + fabsf(c[13]) + fabsf(c[14]));
                if (!ok) atomicAnd(&s_cull, 0);
                o_wb[4 * i + 3] = make_float4(c[12] * kBoxInv, c[13] * kBoxInv, c[14] * kBoxInv, stretch);
            }
        } else if (r < e6) {
            const int i = r - e5;
            if (i < Nh) {
                const float* c = &wh[i * 6];
                o_wh[i] = make_float4(c[0], c[1], c[2], -(c[0] * c[3] + c[1] * c[4] + c[2] * c[5]));
                note_size(fabsf(c[3]) + fabsf(c[4]) + fabsf(c[5]));
                if (!(c[0] * c[0] + c[1] * c[1] + c[2] * c[2] <= kCullStretchMax)) atomicAnd(&s_cull, 0);
            }
        } else {
            const int q = r - e6;
            cp[q] = make_int2(s.cpairs[2 * q], s.cpairs[2 * q + 1]);
        }
    }
    // cull spheres (prrtc_cull.cuh): a link's reach about its coarse centre plus
    // the scene's share of the pad, 8 lanes per link; infinite when the reach is
    // not finite or too large for its squares, so that nothing is culled
    __syncthreads();  // s_scale
    if (coarse_ok) {
        const int k = tid >> 3, l8 = tid & 7;
        const bool mine = k < K;
        float reach = 0.0f;
        bool ok = true, own = true;
        if (mine) {
            const int f0 = s.foff[k], f1 = s.foff[k + 1];
            own = f0 >= 0 && f1 >= f0 && f1 <= S && s.cli[k] >= 0 && s.cli[k] < J;
            const float cx = s.cloc[3 * k], cy = s.cloc[3 * k + 1], cz = s.cloc[3 * k + 2];
            reach = fabsf(s.crad[k]);
            for (int i = clampi(f0, 0, S) + l8; i < clampi(f1, 0, S); i += 8) {
                const float dx = s.sloc[3 * i] - cx, dy = s.sloc[3 * i + 1] - cy, dz = s.sloc[3 * i + 2] - cz;
                const float x = sqrtf(dx * dx + dy * dy + dz * dz) + fabsf(s.srad[i]);  // no fine test passes beyond |r|
                ok = ok && x < 1e6f;
                own = own && s.sli[i] == s.cli[k];
                reach = fmaxf(reach, x);
            }
            if (s.topo_inv && own) own = s.topo_inv[s.cli[k]] >= 0 && s.topo_inv[s.cli[k]] < J;
        }
#pragma unroll
        for (int off = 4; off > 0; off >>= 1) reach = fmaxf(reach, __shfl_xor_sync(0xffffffffu, reach, off));
        const unsigned all_ok = __ballot_sync(0xffffffffu, ok) >> (tid & 24) & 0xffu;
        if (mine && l8 == 0) {
            const float local = fabsf(s.cloc[3 * k]) + fabsf(s.cloc[3 * k + 1]) + fabsf(s.cloc[3 * k + 2]);
            const float r = (1.0f + kCullPad) * reach + kCullScenePad * (local + __uint_as_float(s_scale));
            reinterpret_cast<float*>(grp + 2 * k + 1)[3] = all_ok == 0xffu && r < 1e6f ? r : INFINITY;
        }
        if (mine && !own) atomicAnd(&s_cull, 0);
    }
    // sphere chunks of at most kSphChunk: per group (gated; K <= kMaxLinks), else of the whole list
    int4* sch = reinterpret_cast<int4*>(blob + L.o_sch);
    int n_sch = 0;
    if (gated) {
        int s0 = 0, s1 = 0;
        if (tid < K) {
            s0 = clampi(s.foff[tid], 0, S);
            s1 = clampi(s.foff[tid + 1], 0, S);
        }
        int at = pack_exclusive_scan(s1 > s0 ? cdiv(s1 - s0, kSphChunk) : 0, warp_sums, n_sch);
        for (int a = s0; a < s1 && at < L.sch_cap; a += kSphChunk) sch[at++] = make_int4(a, min(kSphChunk, s1 - a), tid, 0);
        n_sch = min(n_sch, L.sch_cap);
    } else {
        n_sch = min(cdiv(S, kSphChunk), L.sch_cap);
        for (int i = tid; i < n_sch; i += T) sch[i] = make_int4(i * kSphChunk, min(kSphChunk, S - i * kSphChunk), -1, 0);
    }
    // self-pair items: the range decomposition of the coarse pairs, which a flat
    // checker reuses when the ranges tile [0, P)
    int4* item = reinterpret_cast<int4*>(blob + L.o_item);
    bool use_ranges = gated;
    if (!gated && coarse_ok && s.cranges && Q > 0) {
        int bad = 0;
        for (int q = tid; q < Q; q += T) bad |= s.cranges[2 * q] != (q > 0 ? s.cranges[2 * q - 1] : 0);
        use_ranges = __syncthreads_or(bad) == 0 && s.cranges[2 * Q - 1] == P;
    }
    int n_items = 0;
    bool overflow = false;
    if (use_ranges) {
        const int warp = tid >> 5, lane = tid & 31;
        for (int q0 = 0; q0 < Q && !overflow; q0 += T) {
            const int q = q0 + tid, nq = min(T, Q - q0);
            int r0 = 0, r1 = 0, a0 = 0, na = 0, b0 = 0, nb = 0;
            bool cand = false;
            if (q < Q) {
                const int x0 = s.cranges ? s.cranges[2 * q] : 0, x1 = s.cranges ? s.cranges[2 * q + 1] : 0;
                r0 = clampi(x0, 0, P);
                r1 = clampi(x1, 0, P);
                const int ci = s.cpairs[2 * q], cj = s.cpairs[2 * q + 1];
                if (coarse_ok && s.cranges && ci >= 0 && cj >= 0 && ci < K && cj < K && x0 >= 0 && x1 <= P && x0 <= x1) {
                    a0 = clampi(s.foff[ci], 0, S);
                    na = clampi(s.foff[ci + 1], 0, S) - a0;
                    b0 = clampi(s.foff[cj], 0, S);
                    nb = clampi(s.foff[cj + 1], 0, S) - b0;
                    cand = na > 0 && nb > 0 && nb <= 0xffff && x1 - x0 == na * nb;
                }
                t_blk[tid] = make_int4(a0, cand ? na : 0, b0, nb);
                t_r0[tid] = x0;
            }
            __syncthreads();
            // dense-block detection: the range is the row-major product of the pair's two groups
            // (two loads per lane cover a block of 8 x 8; unrolled, so that the loads of four pairs are in flight)
#pragma unroll 4
            for (int k = warp; k < nq; k += kPackThreads / 32) {
                const int4 blk = t_blk[k];
                const int* src = sp + 2 * (size_t)t_r0[k];
                const int total = blk.y * blk.w;
                bool ok = total > 0;
                if (lane < total) {
                    const int pi = __ldg(src + 2 * lane), pj = __ldg(src + 2 * lane + 1);
                    ok = pi == blk.x + lane / blk.w && pj == blk.z + lane % blk.w;
                }
                for (int m = lane + 32; m < total; m += 32) {
                    const int pi = __ldg(src + 2 * m), pj = __ldg(src + 2 * m + 1);
                    ok = ok && pi == blk.x + m / blk.w && pj == blk.z + m % blk.w;
                }
                ok = __all_sync(0xffffffffu, ok);
                if (lane == 0) t_dense[k] = ok ? 1 : 0;
            }
            __syncthreads();
            const bool dense = q < Q && t_dense[tid];
            const int n = q < Q ? (dense ? cdiv(na, kSphChunk) : cdiv(r1 > r0 ? r1 - r0 : 0, kPairChunk)) : 0;
            int tile_total;
            int at = n_items + pack_exclusive_scan(n, warp_sums, tile_total);
            n_items += tile_total;
            overflow = n_items > L.item_cap;  // uniform
            if (!overflow && q < Q) {
                // gate of a gated checker; a flat checker's block keeps its coarse pair as -2 - q
                const int gate = gated ? q : (dense ? -2 - q : -1);
                if (dense) {
                    for (int a = a0; a < a0 + na; a += kSphChunk)
                        item[at++] = make_int4(a, b0, (min(kSphChunk, a0 + na - a) << 16) | nb, gate);
                } else {
                    for (int p = r0; p < r1; p += kPairChunk) item[at++] = make_int4(p, -1, min(kPairChunk, r1 - p), gate);
                }
            }
        }
    }
    if (!use_ranges || overflow) {
        n_items = cdiv(P, kPairChunk);
        __syncthreads();  // an overflowing list's writes come first
        for (int i = tid; i < n_items; i += T)
            item[i] = make_int4(i * kPairChunk, -1, min(kPairChunk, P - i * kPairChunk), -1);
        if (overflow) gated = false;  // fall back to the flat sweep; verdicts are identical
    }
    __syncthreads();  // s_cull
    if (tid == 0) {
        BlobHeader hd;
        hd.J = J; hd.dim = s.dim; hd.S = S; hd.S_pad = odd_pad(S);
        hd.K = K; hd.Q = Q; hd.Ns = Ns; hd.Nc = Nc;
        hd.Nb = Nb; hd.Nh = Nh; hd.n_sch = n_sch; hd.n_items = n_items;
        hd.n_och = cdiv(Ns, kObsChunk) + cdiv(Nc, kObsChunk) + cdiv(Nb, kObsChunk) + cdiv(Nh, kObsChunk);
        hd.gated = gated ? 1 : 0;
        hd.enabled = enabled ? 1 : 0;
        hd.inflate_bits = __float_as_int(s.mode == 1 ? s.margin : 0.0f);
        hd.o_joint = L.o_joint; hd.o_sph = L.o_sph; hd.o_sfr = L.o_sfr; hd.o_grp = L.o_grp;
        hd.o_sch = L.o_sch; hd.o_ws = L.o_ws; hd.o_wc = L.o_wc; hd.o_wb = L.o_wb;
        hd.o_wh = L.o_wh; hd.o_item = L.o_item; hd.o_cpair = L.o_cpair; hd.used_bytes = L.bytes;
        hd.P = P; hd.cap_bytes = cap; hd.error = overflow ? kBlobItemOverflow : 0;
        hd.cull = s_cull && !overflow ? 1 : 0;
        *h = hd;
    }
}

cudaError_t launch_pack(const PackSrc& s, int batch, unsigned char* blobs, size_t stride, cudaStream_t st) {
    if (batch <= 0) return cudaSuccess;
    pack_kernel<<<batch, kPackThreads, 0, st>>>(s, blobs, stride, (int)stride);
    return cudaGetLastError();
}

// ============================================================================ nearest neighbour

// Argmin of the squared distance from q (shared memory) over nodes [0, n) of the
// SoA tree (row stride N), by the whole CTA.  dsq = d0*d0, then fma(dd, dd, dsq)
// in dimension order -- bit-identical to the reference's `dsq += diff*diff`
// (prrtc_planner.cu:845-849) under nvcc's default contraction (the chain starts
// from +0, which leaves d0*d0 as it is).  Valid in warp 0: the node (INT_MAX when
// there is none) in the low word, the bits of its squared distance in the high
// one; ties go to the lowest index, NaN slots never win.
//
// A scan of the usual small tree (hundreds of nodes) is one round trip to L2
// and a reduction, so the loads of 8 dimensions go out together, a warp reduces
// with two integer minima (a non-negative float orders like its bits) instead
// of ten shuffles, and warp 0 alone reduces over the warps, without a second
// barrier.  Out of line: the extend and the connect step share the code.
static __device__ __noinline__ unsigned long long group_nearest(const float* __restrict__ tree, int N, int dim, int n,
                                                                const float* q, unsigned* red_d, int* red_i) {
    const int tid = threadIdx.x, T = blockDim.x;
    float best = INFINITY;
    int bi = INT_MAX;
    if ((N & 3) == 0 && (reinterpret_cast<uintptr_t>(tree) & 15) == 0) {
        const int n4 = (n + 3) >> 2;
        const float4* t4 = reinterpret_cast<const float4*>(tree);
        const size_t row4 = (size_t)(N >> 2);
        for (int g = tid; g < n4; g += T) {
            float ax = 0.0f, ay = 0.0f, az = 0.0f, aw = 0.0f;
            for (int d0 = 0; d0 < dim; d0 += 8) {
                float4 v[8];
                float qr[8];
#pragma unroll
                for (int k = 0; k < 8; ++k) {
                    const int d = min(d0 + k, dim - 1);
                    v[k] = __ldcg(t4 + d * row4 + g);
                    qr[k] = q[d];
                }
#pragma unroll
                for (int k = 0; k < 8; ++k) {
                    if (d0 + k < dim) {
                        const float dx = __fsub_rn(v[k].x, qr[k]), dy = __fsub_rn(v[k].y, qr[k]);
                        const float dz = __fsub_rn(v[k].z, qr[k]), dw = __fsub_rn(v[k].w, qr[k]);
                        ax = __fmaf_rn(dx, dx, ax); ay = __fmaf_rn(dy, dy, ay);
                        az = __fmaf_rn(dz, dz, az); aw = __fmaf_rn(dw, dw, aw);
                    }
                }
            }
            const int i0 = g << 2;
            if (ax < best && i0 < n) { best = ax; bi = i0; }
            if (ay < best && i0 + 1 < n) { best = ay; bi = i0 + 1; }
            if (az < best && i0 + 2 < n) { best = az; bi = i0 + 2; }
            if (aw < best && i0 + 3 < n) { best = aw; bi = i0 + 3; }
        }
    } else {
        for (int i = tid; i < n; i += T) {
            float acc = 0.0f;
            for (int d = 0; d < dim; ++d) {
                const float dd = __fsub_rn(__ldcg(tree + (size_t)d * N + i), q[d]);
                acc = __fmaf_rn(dd, dd, acc);
            }
            if (acc < best) { best = acc; bi = i; }
        }
    }
    const int warp = tid >> 5, lane = tid & 31, nwarp = T >> 5;
    unsigned key = __float_as_uint(best);
    unsigned m = __reduce_min_sync(0xffffffffu, key);
    unsigned i = __reduce_min_sync(0xffffffffu, key == m ? (unsigned)bi : (unsigned)INT_MAX);
    if (lane == 0) { red_d[warp] = m; red_i[warp] = (int)i; }
    __syncthreads();
    if (warp == 0) {
        key = lane < nwarp ? red_d[lane] : 0x7f800000u;
        bi = lane < nwarp ? red_i[lane] : INT_MAX;
        m = __reduce_min_sync(0xffffffffu, key);
        i = __reduce_min_sync(0xffffffffu, key == m ? (unsigned)bi : (unsigned)INT_MAX);
    }
    return (unsigned long long)m << 32 | i;
}

// ============================================================================ explorer

struct Prob {
    int cap;  // this problem's tree capacity (<= the row stride N)
    float* tree[2];
    int* par[2];
    float* radii[2];
    int* sizes;
    int* completed;
    int* iter_count;
    int* conn;
    int* solved;
    unsigned long long* ts;
};

__device__ __forceinline__ Prob prob_ptrs(const PlanLaunch& L, int b) {
    Prob p;
    p.cap = L.caps ? max(1, min(L.caps[b], L.N)) : L.N;
    const size_t tn = (size_t)L.dim * L.N;
    p.tree[0] = L.tree_a + (size_t)b * tn;
    p.tree[1] = L.tree_b + (size_t)b * tn;
    p.par[0] = L.par_a + (size_t)b * L.N;
    p.par[1] = L.par_b + (size_t)b * L.N;
    p.radii[0] = L.radii + (size_t)b * 2 * L.N;
    p.radii[1] = p.radii[0] + L.N;
    p.sizes = L.sizes + 2 * b;
    p.completed = L.completed + 2 * b;
    p.iter_count = L.iter_count + b;
    p.conn = L.connection + 3 * b;
    p.solved = L.solved + b;
    p.ts = L.tstamp + 2 * b;
    return p;
}

struct ExplorerSmem {
    float sample[2][kDimMax];  // this iteration's and the next one's
    float base[kDimMax], cand[kDimMax], delta[kDimMax], curr[kDimMax], vec[kDimMax];
    unsigned red_d[32];
    int red_i[32];
    int order[16];
    int halton[kDimMax];
    int stop, t, n_t, n_o, nn, skip, new_idx, n_ext, ext_parent, ext_idx, G1, G2, vamp, cnn, abort_;
    int pre, pre_solved, pre_a, pre_b;  // solved flag and tree sizes read ahead for the next iteration
    int slot, problem, join_e;
};

// Tail join: once every explorer slot has been taken, a CTA that runs out of
// work picks a problem that is still running -- round-robin over the problems
// from a global ticket -- and runs an extra explorer on it (explorer index
// E + ticket: its own Halton sequence).  The hardest problems of a batch thus
// end with every idle CTA exploring them instead of E explorers and an idle
// GPU.  Returns the problem, or -1 when none is running.
__device__ int tail_join_pick(const PlanLaunch& L, int* e_out) {
    const int k = atomicAdd(&L.queue[2], 1);
    *e_out = L.E + k;
    for (int i = 0; i < L.B; ++i) {
        const int pi = (int)(((long long)k + i) % L.B);
        const int bb = L.order ? L.order[pi] : pi;
        if (ld_volatile(&L.solved[bb]) == 0) return bb;
    }
    return -1;
}

// Edge [base, base+delta] at waypoints t = (k+1)/G (prrtc_planner.cu:899-903).
// The G waypoints are visited in nchunk interleaved passes -- pass c checks
// waypoints c, c+nchunk, c+2*nchunk, ... -- so the first pass already samples
// the whole edge and a colliding edge usually stops after one pass.  The
// verdict (any waypoint in collision) does not depend on the order.
// The waypoints are computed inside the checker's FK step (no staging pass).
template <class Grp>
__device__ __forceinline__ bool group_edge_collides(const Grp& grp, const Scene& sc, const CcBufs& B, const float* base,
                                                    const float* delta, int G, int CW, int& par) {
    if (B.stats && grp.rank() == 0) atomicAdd(&B.stats[kStatEdges], 1ull);
    const int nchunk = (G + CW - 1) / CW;
    for (int c = 0; c < nchunk; ++c) {
        const int nw = (G - c + nchunk - 1) / nchunk;  // waypoints c, c+nchunk, ... below G
        const EdgeSrc e{base, delta, G, nchunk, c};
        if (cc_chunk<false>(grp, sc, B, nw, true, par, &e) != 0u) return true;
    }
    return false;
}

// Edge checker of the general form: any robot and coarse model.  The buffers and the
// scene are the kernel's own objects, the scene set in a branch for each place it
// may lie in: one view of a chosen pointer, whose accesses are then not known to be
// to shared memory, made plans 8-14% slower (kernel time of 310 tabletop problems, E =
// 1, arm without a coarse model: 2.72 ms, so 2.53).
struct GeneralEdges {
    const CcBufs& B;
    const Scene& sc;
    int CW;
    int par;
    __device__ __forceinline__ void reset() {
        if (threadIdx.x == 0) B.hit[0] = B.hit[1] = 0u;  // the checker's two result words
        par = 0;
    }
    template <class Grp>
    __device__ __forceinline__ bool collides(const Grp& grp, const float* base, const float* delta, int G) {
        return group_edge_collides(grp, sc, B, base, delta, G, CW, par);
    }
};

// A scene that the culled check does not take (BlobHeader::cull not set: groups
// that do not cover the spheres on their own frames, ...), in the culled
// kernel: the general checker in the same shared memory, CW waypoints at a
// time.  Out of line, so that its registers and code stay off the main path.
static __device__ __noinline__ bool general_edge_collides(const unsigned char* blob, const int2* pairs, const PcView* pc,
                                                   unsigned char* smem, unsigned long long* stats, const float* base,
                                                   const float* delta, int G, int CW) {
    Scene sc = scene_view(blob);
    sc.pairs = pairs;
    sc.pc = *pc;
    CcBufs B = cc_bufs(smem, sc.h->J, sc.h->S, sc.h->K, sc.h->Q, CW);
    B.stats = stats;
    __syncthreads();
    if (threadIdx.x == 0) B.hit[0] = B.hit[1] = 0u;
    __syncthreads();
    int par = 0;
    const bool r = group_edge_collides(CtaGroup{}, sc, B, base, delta, G, CW, par);
    __syncthreads();
    return r;
}

// Edge checker of the culled form (prrtc_cull.cuh).  One out-of-line copy
// serves the extend and the connect step: less code to fetch, and the
// explorer's own registers are saved around the call.  The buffers are
// addressed from the dynamic shared memory itself, so that their accesses stay
// shared-memory instructions.  Returns the answer in bit 0 and the next `par` in
// bit 1.
struct CulledEdges {  // in shared memory
    const int2* pairs;
    PcView pc;
    unsigned long long* stats;
    int blob_cap, J, K, n_obs, CW, CW_general;
};

static __device__ __noinline__ int culled_edge_collides(const CulledEdges* a, const float* base, const float* delta, int G,
                                                 int par) {
    extern __shared__ __align__(128) unsigned char dsm[];
    Scene sc = scene_view(dsm);
    if (!sc.h->cull) {
        if (!sc.h->enabled) {
            __syncthreads();  // as a check does: the caller rewrites what the last one read
            return par << 1;
        }
        return (general_edge_collides(dsm, a->pairs, &a->pc, dsm + a->blob_cap, a->stats, base, delta, G, a->CW_general)
                    ? 1 : 0) | par << 1;
    }
    CullBufs B = cull_bufs(dsm + a->blob_cap, a->J, a->K, a->n_obs, a->CW);
    B.stats = a->stats;
    sc.pairs = a->pairs;
    sc.pc = a->pc;
    if (B.stats && threadIdx.x == 0) atomicAdd(&B.stats[kStatEdges], 1ull);
    const int nchunk = (G + a->CW - 1) / a->CW;
    for (int c = 0; c < nchunk; ++c) {
        const int nw = (G - c + nchunk - 1) / nchunk;
        const EdgeSrc e{base, delta, G, nchunk, c};
        if (cull_check(CtaGroup{}, sc, B, nw, a->CW, par, e) != 0u) return 1 | par << 1;
    }
    return par << 1;
}

struct CulledEdgesRef {
    const CulledEdges* a;
    uint32_t* hit;
    int par;
    __device__ __forceinline__ void reset() {
        if (threadIdx.x < 6) hit[threadIdx.x] = 0u;
        par = 0;
    }
    template <class Grp>
    __device__ __forceinline__ bool collides(const Grp&, const float* base, const float* delta, int G) {
        const int r = culled_edge_collides(a, base, delta, G, par);
        par = r >> 1;
        return (r & 1) != 0;
    }
};

__device__ __forceinline__ void stamp_end(const Prob& P) {
    atomicCAS(&P.ts[1], 0ull, globaltimer());
}

// One explorer (problem P, index e of E) until the problem terminates or the
// explorer exits.  All threads of the group call it.
template <class Grp, class Edges>
__device__ __forceinline__ void run_explorer(const Grp& grp, const PlanLaunch& L, const Prob& P, Edges& edges,
                                             ExplorerSmem& X, int e) {
    const int tid = grp.rank();
    const int dim = L.dim, N = L.N;
    if (tid == 0) {
        prime_order(e, X.order);
        for (int d = 0; d < kDimMax; ++d) X.halton[d] = 1;
        X.vamp = 0;
        X.pre = 0;
    }
    edges.reset();
    grp.sync();
    // The next iteration's sample depends on the explorer alone, so another warp
    // than the one that waits for the problem's state draws it meanwhile.
    const int sampler = grp.size() > 32 ? 32 : 0;
    auto draw = [&](int lane, float* out) {  // halton_sample, one dimension per lane
        if (lane < dim) {
            const float val = halton_next(X.order[lane & 15], X.halton[lane]);
            out[lane] = __fmaf_rn(val, __fsub_rn(L.hi[lane], L.lo[lane]), L.lo[lane]);
        }
    };
    if (tid >= sampler && tid < sampler + 32) draw(tid - sampler, X.sample[1]);
    int local_iter = 0;
    // The per-iteration scalar work runs on warp 0 with one lane per dimension
    // (extend, connect vector); lane 0 does the rest.  Every lane repeats lane
    // 0's arithmetic for its own dimension, so results are the same bits as a
    // sequential loop.
    while (true) {
        ++local_iter;
        const float* sample = X.sample[local_iter & 1];
        if (tid == 0) {
            int sv, sa, sb;
            if (X.pre) {  // read with the last extension's node (one round trip for all)
                sv = X.pre_solved;
                sa = X.pre_a;
                sb = X.pre_b;
                X.pre = 0;  // for this iteration only: one without a nearest node reads none ahead
            } else {
                // the three loads go out together: one round trip, not three
                sv = ld_volatile(P.solved);
                sa = ld_volatile(&P.sizes[0]);
                sb = ld_volatile(&P.sizes[1]);
            }
            int stop = sv != 0;
            if (!stop && local_iter > L.max_iter) {
                if (atomicCAS(P.solved, 0, -1) == 0) stamp_end(P);
                atomicMax(P.iter_count, local_iter);
                stop = 1;
            }
            if (!stop) {
                const int t = choose_tree(L.balance_mode, local_iter, e % L.E, L.E, sa, sb, L.tree_ratio, X.vamp);
                X.t = t;
                X.n_t = min(t == 0 ? sa : sb, P.cap);
            }
            X.stop = stop;
        }
        if (tid >= sampler && tid < sampler + 32) draw(tid - sampler, X.sample[(local_iter + 1) & 1]);
        grp.sync();
        if (X.stop) break;
        const int t = X.t, o = 1 - t;
        unsigned long long nearest = group_nearest(P.tree[t], N, dim, X.n_t, sample, X.red_d, X.red_i);
        if (tid < 32) {
            const int lane = tid;
            const int nn = (int)(unsigned)nearest;
            int skip = nn == INT_MAX;
            if (!skip) {
                // radius and node loads issued together (one round trip), and
                // the state that the next iteration starts from if this one
                // inserts nothing
                const float rad = L.dd ? __ldcg(&P.radii[t][nn]) : 0.0f;
                const float bv = lane < dim ? __ldcg(&P.tree[t][(size_t)lane * N + nn]) : 0.0f;
                if (lane == 0) {
                    X.pre_solved = ld_volatile(P.solved);
                    X.pre_a = ld_volatile(&P.sizes[0]);
                    X.pre_b = ld_volatile(&P.sizes[1]);
                    X.pre = 1;
                }
                const float nd = __fsqrt_rn(__uint_as_float((unsigned)(nearest >> 32)));
                skip = L.dd && (rad < nd);
                if (!skip) {
                    const float scl = nd > 1e-8f ? fminf(1.0f, __fdiv_rn(L.step, nd)) : 1.0f;
                    if (lane < dim) {
                        X.base[lane] = bv;
                        const float c = __fmaf_rn(__fsub_rn(sample[lane], bv), scl, bv);
                        X.cand[lane] = c;
                        X.delta[lane] = __fsub_rn(c, bv);
                    }
                    __syncwarp();
                    if (lane == 0) X.G1 = edge_waypoints(X.delta, dim, L.granularity, L.edge_res);
                }
            }
            if (lane == 0) {
                if (L.stats) atomicAdd(&L.stats[kStatNnNodes], (unsigned long long)X.n_t);
                X.nn = nn;
                X.skip = skip;
            }
        }
        grp.sync();
        if (X.skip) continue;
        if (edges.collides(grp, X.base, X.delta, X.G1)) {
            if (tid == 0 && L.dd) radius_shrink(P.radii[t], X.nn, L.dd_alpha, L.dd_radius, L.dd_min_radius, &L.queue[1]);
            continue;
        }
        // insert (prrtc_planner.cu:925-947).  The other tree's size for the
        // connect scan is read together with the slot claim (one round trip
        // instead of two; any node published by then is scanned, as in the
        // reference's read after its insert).  The nearest node's radius grows
        // on another warp while the connect scan runs: nothing in this
        // iteration reads it.
        if (tid == 0) {
            const int so = ld_volatile(&P.sizes[o]);
            const int idx = atomicAdd(&P.sizes[t], 1);
            if (idx >= P.cap) {
                if (atomicCAS(P.solved, 0, -1) == 0) stamp_end(P);
                X.new_idx = -1;
            } else {
                P.par[t][idx] = X.nn;
                X.new_idx = idx;
            }
            X.n_o = min(so, P.cap);
            X.pre = 0;  // the sizes change: read again
        }
        grp.sync();
        if (X.new_idx < 0) break;
        if (tid < dim) __stcg(&P.tree[t][(size_t)tid * N + X.new_idx], X.cand[tid]);
        if (tid == 0) atomicAdd(&P.completed[t], 1);
        if (L.dd && tid == (grp.size() > 32 ? 32 : 0)) radius_grow(P.radii[t], X.nn, L.dd_alpha, &L.queue[1]);
        // connect (prrtc_planner.cu:949-1043)
        nearest = group_nearest(P.tree[o], N, dim, X.n_o, X.cand, X.red_d, X.red_i);
        if (tid < 32) {
            const int lane = tid;
            const int cnn = (int)(unsigned)nearest;
            int n_ext = 0;
            if (cnn != INT_MAX) {
                const float cd = __fsqrt_rn(__uint_as_float((unsigned)(nearest >> 32)));
                if (L.step > 1e-8f && cd > 1e-8f) n_ext = (int)ceilf(__fdiv_rn(cd, L.step));
                if (lane < dim) {
                    const float c = X.cand[lane];
                    X.curr[lane] = c;
                    X.vec[lane] = n_ext > 0 ? __fdiv_rn(__fsub_rn(__ldcg(&P.tree[o][(size_t)lane * N + cnn]), c),
                                                        (float)n_ext)
                                            : 0.0f;
                }
                __syncwarp();
                if (lane == 0) X.G2 = edge_waypoints(X.vec, dim, L.granularity, L.edge_res);
            } else {
                n_ext = -1;
            }
            if (lane == 0) {
                if (L.stats) atomicAdd(&L.stats[kStatNnNodes], (unsigned long long)X.n_o);
                X.cnn = cnn;
                X.n_ext = n_ext;
                X.ext_parent = X.new_idx;
                X.abort_ = 0;
            }
        }
        grp.sync();
        bool failed = X.n_ext < 0;
        const int n_ext = X.n_ext;
        for (int ext = 0; ext < n_ext && !failed; ++ext) {
            if (X.abort_) { failed = true; break; }
            if (edges.collides(grp, X.curr, X.vec, X.G2)) { failed = true; break; }
            if (tid < 32) {
                const int lane = tid;
                int eidx = 0;
                if (lane == 0) {
                    // whether another explorer solved the problem meanwhile, read with the claim
                    X.abort_ = ld_volatile(P.solved) != 0;
                    eidx = atomicAdd(&P.sizes[t], 1);
                }
                eidx = __shfl_sync(0xffffffffu, eidx, 0);
                if (eidx >= P.cap) {
                    if (lane == 0) {
                        if (atomicCAS(P.solved, 0, -1) == 0) stamp_end(P);
                        X.ext_idx = -1;
                    }
                } else {
                    if (lane < dim) X.curr[lane] = __fadd_rn(X.curr[lane], X.vec[lane]);
                    if (lane == 0) {
                        P.par[t][eidx] = X.ext_parent;
                        X.ext_parent = eidx;
                        X.ext_idx = eidx;
                    }
                }
            }
            grp.sync();
            if (X.ext_idx < 0) { failed = true; break; }
            if (tid < dim) __stcg(&P.tree[t][(size_t)tid * N + X.ext_idx], X.curr[tid]);
            if (tid == 0) atomicAdd(&P.completed[t], 1);
            // no barrier: the next sub-edge check only reads X.curr / X.vec, and
            // warp 0 next writes them after that check's barriers
        }
        if (!failed) {  // connection found (prrtc_planner.cu:1045-1062)
            if (tid == 0) {
                if (atomicCAS(P.solved, 0, 1) == 0) {
                    if (t == 0) { P.conn[0] = X.ext_parent; P.conn[1] = X.cnn; }
                    else { P.conn[0] = X.cnn; P.conn[1] = X.ext_parent; }
                    P.conn[2] = t;
                    stamp_end(P);
                }
                atomicMax(P.iter_count, local_iter);
            }
            break;
        }
    }
    grp.sync();
}

// Plain form: grid = E explorers of problem blockIdx.y.  Persistent form: CTAs
// pop (problem, explorer) slots until the queue is empty.  CULL: edges by the
// culled check, the scene always staged (launch_plan's rule).
//
// Bound by the latency of an explorer's chain (sample, nearest node, edge
// passes of link frames -> bounds -> touching primitives -> fine tests), not by
// arithmetic or memory: a lone CTA of 256 threads issues 0.18 instructions per
// cycle and scheduler, its warps waiting for fixed-latency results and shared
// memory.  So an explorer gets 128 registers per thread (80 and three CTAs per
// SM measured 8-12% slower per plan, no faster per batch), and more threads
// where SMs are idle (launch_plan).  Kernel times, medians of 20, against the general
// checker: 136 -> 82 us (16 spheres, 128 explorers), 2.38 -> 1.42 ms (512 uneven
// problems, E = 2), 4.71 ms -> 2.83 with 256 threads and 2.57 with 512 (200 tabletop
// problems, E = 1), 34.2 -> 6.78 and 5.59 ms (61 dual-arm problems, E = 1).
template <bool CULL, int THREADS, int MINBLOCKS>
__global__ void __launch_bounds__(THREADS, MINBLOCKS) explore_kernel(PlanLaunch L) {
    extern __shared__ __align__(128) unsigned char dsm[];
    __shared__ ExplorerSmem X;
    __shared__ CulledEdges C;
    __shared__ __align__(8) uint64_t mbar;
    const int tid = threadIdx.x;
    const bool staged = CULL || L.blob_cap > 0;
    unsigned char* blob_sm = dsm;
    unsigned char* bufs = dsm + (staged ? L.blob_cap : 0);
    if (tid == 0) mbar_init(&mbar);
    __syncthreads();
    uint32_t phase = 0;
    int cur = -1;
    const int total = L.persistent ? L.B * L.E : 1;
    for (int iter = 0;; ++iter) {
        int b, e;
        if (L.persistent) {
            if (tid == 0) {
                int slot = atomicAdd(&L.queue[0], 1);
                // skip the explorers of problems that already terminated
                while (slot < total) {
                    const int pi = slot / L.E;
                    const int bb = L.order ? L.order[pi] : pi;
                    if (ld_volatile(&L.solved[bb]) == 0) break;
                    slot = atomicAdd(&L.queue[0], 1);
                }
                X.slot = slot;
                X.problem = -1;
                if (slot >= total && L.tail_join) X.problem = tail_join_pick(L, &X.join_e);
            }
            __syncthreads();
            const int slot = X.slot;
            if (slot < total) {
                const int pi = slot / L.E;
                b = L.order ? L.order[pi] : pi;
                e = slot - pi * L.E;
            } else {
                if (X.problem < 0) break;
                b = X.problem;
                e = X.join_e;
            }
        } else {
            if (iter > 0) break;
            b = blockIdx.y;
            e = blockIdx.x;
        }
        const unsigned char* gblob = L.blobs + (size_t)b * L.blob_stride;
        if (b != cur) {
            if (staged) {
                const int bytes = reinterpret_cast<const BlobHeader*>(gblob)->used_bytes;
                if (!stage_blob(blob_sm, gblob, min(bytes, L.blob_cap), &mbar, phase, &L.queue[1], 1,
                                L.wait_polls == 0 ? kWaitLimit : max(L.wait_polls, 0)))
                    break;
            }
            cur = b;
        }
        const int2* pairs = reinterpret_cast<const int2*>(L.pairs) + (size_t)b * L.pairs_stride;
        const Prob P = prob_ptrs(L, b);
        if (L.persistent && tid == 0) atomicCAS(&P.ts[0], 0ull, globaltimer());
        if constexpr (CULL) {
            if (tid == 0) C = CulledEdges{pairs, L.pc, L.stats, L.blob_cap, L.J, L.K, L.n_obs, L.cw, L.cw_general};
            CulledEdgesRef edges;
            edges.a = &C;
            edges.hit = reinterpret_cast<uint32_t*>(bufs);  // first in the buffers
            run_explorer(CtaGroup{}, L, P, edges, X, e);
        } else {
            CcBufs B = cc_bufs(bufs, L.J, L.S, L.K, L.Q, L.cw);
            B.stats = L.stats;
            Scene sc;
            if (staged) sc = scene_view(blob_sm);
            else sc = scene_view(gblob);
            sc.pairs = pairs;
            sc.pc = L.pc;
            GeneralEdges edges{B, sc, L.cw, 0};
            run_explorer(CtaGroup{}, L, P, edges, X, e);
        }
    }
}

// Slot initialisation (the reference's memsets and FLT_MAX fill,
// prrtc_planner.cu:1192-1202, 85-95): slots [0, cap_b) of problem b's rows --
// two trees of dim rows, two parent rows, two radius rows -- become
// 0xFFFFFFFF in the trees and parents (a NaN tree slot, skipped by the
// nearest-neighbour scan until written; parent -1) and FLT_MAX in the radii
// (unset).  Only the problem's own
// capacity is written; words [cap_b, N) of its rows are never read by the
// planner and keep whatever they held.  A CTA writes 16 KB chunks of one row
// (uint4 stores when every row starts 16-byte aligned, N % 4 == 0); blockIdx.y
// strides over problems, blockIdx.x over a problem's (row, chunk) items.
constexpr int kFillChunk = 4096;  // 32-bit words per fill item

__device__ __forceinline__ uint32_t* fill_row(const PlanLaunch& L, int b, int r) {
    const size_t N = (size_t)L.N;
    if (r < L.dim) return reinterpret_cast<uint32_t*>(L.tree_a) + ((size_t)b * L.dim + r) * N;
    r -= L.dim;
    if (r < L.dim) return reinterpret_cast<uint32_t*>(L.tree_b) + ((size_t)b * L.dim + r) * N;
    r -= L.dim;
    if (r == 0) return reinterpret_cast<uint32_t*>(L.par_a) + (size_t)b * N;
    if (r == 1) return reinterpret_cast<uint32_t*>(L.par_b) + (size_t)b * N;
    return reinterpret_cast<uint32_t*>(L.radii) + ((size_t)b * 2 + (r - 2)) * N;
}

__global__ void __launch_bounds__(256) fill_kernel(PlanLaunch L) {
    const int rows = 2 * L.dim + 4;
    const bool vec = (L.N & 3) == 0;
    for (int b = blockIdx.y; b < L.B; b += gridDim.y) {
        const int cap = L.caps ? max(1, min(L.caps[b], L.N)) : L.N;
        const int chunks = (cap + kFillChunk - 1) / kFillChunk;
        for (int it = blockIdx.x; it < rows * chunks; it += gridDim.x) {
            const int r = it / chunks, c0 = (it - r * chunks) * kFillChunk;
            const int c1 = min(cap, c0 + kFillChunk);
            uint32_t* row = fill_row(L, b, r);
            const uint32_t w = r >= 2 * L.dim + 2 ? 0x7f7fffffu : ~0u;  // FLT_MAX radii, else all ones
            if (vec) {
                // c0 is a multiple of 4; the last vector may pass cap but stays
                // inside the row (N % 4 == 0), in words nobody reads
                uint4* v = reinterpret_cast<uint4*>(row + c0);
                const int n4 = (c1 - c0 + 3) >> 2;
                for (int k = threadIdx.x; k < n4; k += blockDim.x) v[k] = make_uint4(w, w, w, w);
            } else {
                for (int k = c0 + threadIdx.x; k < c1; k += blockDim.x) row[k] = w;
            }
        }
    }
}

// Roots and counters (prrtc_planner.cu:97-125, 1204-1237).  Tree slots,
// parents and radii of [0, cap_b) were set (NaN / -1 / FLT_MAX) by fill_kernel
// before.
__global__ void init_kernel(PlanLaunch L, int stamp_start) {
    const int b = blockIdx.x, tid = threadIdx.x;
    if (b >= L.B) return;
    const Prob P = prob_ptrs(L, b);
    int G = L.num_goals;
    if (L.goal_counts) G = max(1, min(L.goal_counts[b], L.num_goals));
    G = min(G, P.cap);
    const float* st = L.starts + (size_t)b * L.dim;
    const float* gl = L.goals + (size_t)b * L.num_goals * L.dim;
    for (int d = tid; d < L.dim; d += blockDim.x) P.tree[0][(size_t)d * L.N] = st[d];
    for (int i = tid; i < G * L.dim; i += blockDim.x) {
        const int g = i / L.dim, d = i - g * L.dim;
        P.tree[1][(size_t)d * L.N + g] = gl[g * L.dim + d];
    }
    for (int g = tid; g < G; g += blockDim.x) P.par[1][g] = g;
    if (tid == 0) {
        P.par[0][0] = 0;
        P.sizes[0] = 1; P.sizes[1] = G;
        P.completed[0] = 1; P.completed[1] = G;
        P.iter_count[0] = 0;
        P.conn[0] = -1; P.conn[1] = -1; P.conn[2] = -1;
        P.solved[0] = 0;
        P.ts[0] = stamp_start ? globaltimer() : 0ull;
        P.ts[1] = 0ull;
    }
    if (b == 0 && tid == 0) { L.queue[0] = 0; L.queue[1] = 0; L.queue[2] = 0; }
}

__global__ void finalize_kernel(PlanLaunch L) {
    const int b = blockIdx.x * blockDim.x + threadIdx.x;
    if (b >= L.B) return;
    const unsigned long long t0 = L.tstamp[2 * b], t1 = L.tstamp[2 * b + 1];
    L.ktime[b] = (t1 > t0 && t0 != 0ull) ? (float)((double)(t1 - t0) * 1e-6) : 0.0f;
    // a device wait ran out somewhere in the launch: problems left open are
    // reported as -2 instead of the "still running" 0
    if (L.queue[1] != 0 && L.solved[b] == 0) L.solved[b] = -2;
}

size_t plan_workspace_bytes(int B, int N, size_t blob_stride) {
    size_t b = 0;
    b += (size_t)B * blob_stride;
    b += ((size_t)B * 2 * N * sizeof(float) + 255) & ~(size_t)255;
    b += ((size_t)B * 2 * sizeof(unsigned long long) + 255) & ~(size_t)255;
    b += 256;
    return b;
}

void plan_carve_workspace(PlanLaunch& L, void* ws, size_t stride) {
    unsigned char* p = static_cast<unsigned char*>(ws);
    L.blobs = p;
    L.blob_stride = stride;
    p += (size_t)L.B * stride;
    L.radii = reinterpret_cast<float*>(p);
    p += ((size_t)L.B * 2 * L.N * sizeof(float) + 255) & ~(size_t)255;
    L.tstamp = reinterpret_cast<unsigned long long*>(p);
    p += ((size_t)L.B * 2 * sizeof(unsigned long long) + 255) & ~(size_t)255;
    L.queue = reinterpret_cast<int32_t*>(p);
}

int device_sm_count() {
    int dev = 0, n = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev);
    return n > 0 ? n : 1;
}

size_t device_max_smem() {
    int dev = 0, n = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&n, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
    return (size_t)n;
}

// explore_kernel's attributes as last set in one device's CUDA context.
struct ExploreAttrs {
    unsigned long long ctx = 0ull;  // context key (current_context_key)
    int max_dyn = -1;          // largest MaxDynamicSharedMemorySize set
    int carve = INT_MIN;       // carve-out preference set (-1 = none)
    bool have_smem = false;    // the three sizes below are known
    int sm_smem = 0, reserved = 0;
    size_t static_smem = 0;
};
constexpr int kMaxCachedDevices = 256;
static ExploreAttrs g_explore_attr[kMaxCachedDevices][3];  // [device][general, culled, culled wide]
static std::mutex g_explore_attr_mutex;

// An optional timing event on the stream; inside a stream capture it becomes an
// external event-record node, which records each time the graph runs.
static cudaError_t record_event(cudaEvent_t ev, cudaStream_t st) {
    if (!ev) return cudaSuccess;
    cudaStreamCaptureStatus cs = cudaStreamCaptureStatusNone;
    cudaError_t e = cudaStreamIsCapturing(st, &cs);
    if (e != cudaSuccess) return e;
    return cs == cudaStreamCaptureStatusActive ? cudaEventRecordWithFlags(ev, st, cudaEventRecordExternal)
                                               : cudaEventRecord(ev, st);
}

cudaError_t launch_plan(PlanLaunch& L, cudaStream_t st) {
    cudaError_t e;
    {
        // enough fill CTAs for about four per SM in total, at least 16 per problem
        const int gy = std::min(L.B, 65535);
        const int gx = std::max(16, (4 * device_sm_count() + gy - 1) / gy);
        fill_kernel<<<dim3(gx, gy), 256, 0, st>>>(L);
        if ((e = cudaGetLastError()) != cudaSuccess) return e;
    }
    init_kernel<<<L.B, 128, 0, st>>>(L, L.persistent ? 0 : 1);
    if ((e = cudaGetLastError()) != cudaSuccess) return e;

    const size_t max_smem = device_max_smem();
    const size_t static_smem = sizeof(ExplorerSmem) + sizeof(CulledEdges) + 64;
    size_t dyn = 0;
    // The culled form with 64 waypoints per pass, or as many (32, 16, 8) as
    // leave room for its CTAs: a pass costs mostly the latency of its phases,
    // so fewer passes win (batches of 300 tabletop problems, E = 2: 2.49 -> 2.20
    // ms against 16 per pass; 61 dual-arm problems, E = 1: 7.3 -> 5.2 ms).
    // Wide form, where the caller names no size: a batch of at most two explorers
    // per SM leaves most of the GPU idle at 256 threads, so each explorer gets 512,
    // one CTA per SM.  E = 1, a call in ms with 256 -> 512 threads: tabletop, 100
    // problems 2.15 -> 1.96, 200 3.89 -> 3.72, 296 3.99 -> 3.86; dual arm, 61 7.03 ->
    // 5.61, 149 9.92 -> 7.19, 296 11.04 -> 8.82; at E = 2 x 512 problems it loses,
    // 4.4 -> 4.7.  A plain launch of at most one explorer per SM gets 512 as well.
    const long long explorers = (long long)L.B * L.E;
    const bool wide = L.threads == 0 && explorers <= (L.persistent ? 2ll : 1ll) * device_sm_count();
    const bool one_per_sm = wide || explorers <= device_sm_count();
    bool cull = false;
    if (L.cull) {
        const size_t room = one_per_sm ? max_smem : max_smem / 2 - 1024;
        for (int cw = 64; cw >= 8 && !cull; cw /= 2) {
            // the buffers also hold the general checker's, for a scene that is not culled
            size_t need = (size_t)cull_smem_bytes(L.J, L.K, L.n_obs, cw);
            need = std::max(need, (size_t)cc_smem_bytes(L.J, L.S, L.K, L.Q, 8));
            if (need + (size_t)L.blob_cap + static_smem > (cw > 8 ? room : max_smem)) continue;
            cull = true;
            L.cw = cw;
            L.cw_general = 8;
            while (L.cw_general < cw && (size_t)cc_smem_bytes(L.J, L.S, L.K, L.Q, 2 * L.cw_general) <= need)
                L.cw_general *= 2;
            dyn = need + (size_t)L.blob_cap;
        }
    }
    if (!cull) {
        const size_t cc = (size_t)cc_smem_bytes(L.J, L.S, L.K, L.Q, L.cw);
        dyn = cc + (size_t)L.blob_cap;
        if (dyn + static_smem > max_smem) {  // scene too large to stage: read it from global memory
            L.blob_cap = 0;
            dyn = cc;
        }
    }
    if (cull && wide) L.threads = kWideThreads;
    else if (L.threads == 0) L.threads = cull ? 256 : 128;
    const int form = !cull ? 0 : (L.threads > 256 ? 2 : 1);
    void (*const kern)(PlanLaunch) = form == 0   ? explore_kernel<false, 256, PRRTC_EXPLORE_MINBLOCKS>
                                     : form == 1 ? explore_kernel<true, 256, PRRTC_EXPLORE_MINBLOCKS>
                                                 : explore_kernel<true, kWideThreads, 1>;
    // ctas_per_sm > 0: the smallest shared-memory carve-out that holds that many
    // CTAs, so the rest of the SM's unified L1 / shared memory is L1 (the
    // explorers read trees, radii and unstaged scene data through it); measured
    // faster than the largest carve-out's one more resident CTA per SM (-1: no
    // preference).  The kernel's attributes are set only when they change, from
    // a cache per device and CUDA context: querying or setting them while the
    // previous batch's planner still ran measured as a host-side wait for that
    // launch, which serialised back-to-back calls (e2e 134 K against 198 K
    // plans/s with a carve-out set on every call).
    {
        int dev = 0;
        if ((e = cudaGetDevice(&dev)) != cudaSuccess) return e;
        const unsigned long long ctx = current_context_key();
        std::lock_guard<std::mutex> lock(g_explore_attr_mutex);
        ExploreAttrs dflt;
        ExploreAttrs& c = (dev >= 0 && dev < kMaxCachedDevices) ? g_explore_attr[dev][form] : dflt;
        if (!ctx || c.ctx != ctx) {
            c = ExploreAttrs{};
            c.ctx = ctx;
        }
        if ((int)dyn > c.max_dyn) {
            if ((e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)dyn)) !=
                cudaSuccess)
                return e;
            c.max_dyn = (int)dyn;
        }
        int carve = -1;
        if (L.persistent && L.ctas_per_sm > 0) {
            if (!c.have_smem) {
                cudaFuncAttributes fa;
                if ((e = cudaDeviceGetAttribute(&c.sm_smem, cudaDevAttrMaxSharedMemoryPerMultiprocessor, dev)) !=
                        cudaSuccess ||
                    (e = cudaDeviceGetAttribute(&c.reserved, cudaDevAttrReservedSharedMemoryPerBlock, dev)) !=
                        cudaSuccess ||
                    (e = cudaFuncGetAttributes(&fa, kern)) != cudaSuccess)
                    return e;
                c.static_smem = fa.sharedSizeBytes;
                c.have_smem = true;
            }
            const size_t need = (size_t)L.ctas_per_sm * (dyn + c.static_smem + (size_t)c.reserved);
            carve = c.sm_smem > 0 ? (int)std::min<size_t>(100, (100 * need + c.sm_smem - 1) / (size_t)c.sm_smem) : -1;
        }
        if (carve != c.carve) {
            if ((e = cudaFuncSetAttribute(kern, cudaFuncAttributePreferredSharedMemoryCarveout, carve)) !=
                cudaSuccess)
                return e;
            c.carve = carve;
        }
    }
    if (L.persistent) {
        int per_sm = 0;
        if ((e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, L.threads, dyn)) !=
            cudaSuccess)
            return e;
        per_sm = std::max(per_sm, 1);
        if (L.ctas_per_sm > 0) per_sm = std::min(per_sm, L.ctas_per_sm);
        long long grid = (long long)per_sm * device_sm_count();
        if (L.resident > 0) grid = std::min<long long>(grid, L.resident);
        // no more CTAs than explorer slots: with several batches in flight (one per
        // capacity bucket) a full-GPU grid per launch measured slower, its CTAs
        // piling extra explorers onto a few problems
        grid = std::min<long long>(grid, (long long)L.B * L.E);
        if ((e = record_event(L.explore_events[0], st)) != cudaSuccess) return e;
        kern<<<(unsigned)std::max<long long>(grid, 1), L.threads, dyn, st>>>(L);
    } else {
        if ((e = record_event(L.explore_events[0], st)) != cudaSuccess) return e;
        kern<<<dim3(L.E, L.B), L.threads, dyn, st>>>(L);
    }
    if ((e = cudaGetLastError()) != cudaSuccess) return e;
    if ((e = record_event(L.explore_events[1], st)) != cudaSuccess) return e;
    finalize_kernel<<<(L.B + 127) / 128, 128, 0, st>>>(L);
    return cudaGetLastError();
}

// ============================================================================ path extraction

// One CTA (32 threads) per problem: lane 0 walks the parent chains
// (prrtc.py:603-640), all lanes copy configurations; cost = sum of segment norms.
__global__ void extract_paths_kernel(int B, int dim, int N, const float* ta, const float* tb, const int32_t* pa,
                                     const int32_t* pb, const int32_t* conn, const int32_t* solved, int max_len,
                                     float* paths, int32_t* lengths, float* costs) {
    const int b = blockIdx.x, lane = threadIdx.x;
    extern __shared__ int chain[];  // max_len entries: node index, negative = tree B (-1 - idx)
    __shared__ int s_len;
    const float* TA = ta + (size_t)b * dim * N;
    const float* TB = tb + (size_t)b * dim * N;
    const int32_t* PA = pa + (size_t)b * N;
    const int32_t* PB = pb + (size_t)b * N;
    if (lane == 0) {
        int len = 0;
        if (solved[b] == 1) {
            const int a = conn[3 * b], c = conn[3 * b + 1];
            if (a >= 0 && c >= 0 && a < N && c < N) {
                int na = 0, curr = a;
                for (int it = 0; it < N; ++it) {  // count tree-A chain
                    ++na;
                    const int p = PA[curr];
                    if (p == curr || p < 0 || p >= N) break;
                    curr = p;
                }
                if (na > max_len) len = -1;
                else {
                    curr = a;
                    for (int i = na - 1; i >= 0; --i) {
                        chain[i] = curr;
                        const int p = PA[curr];
                        if (p == curr || p < 0 || p >= N) break;
                        curr = p;
                    }
                    len = na;
                    curr = c;
                    for (int it = 0; it < N; ++it) {
                        if (len >= max_len) { len = -1; break; }
                        chain[len++] = -1 - curr;
                        const int p = PB[curr];
                        if (p == curr || p < 0 || p >= N) break;
                        curr = p;
                    }
                }
            }
        }
        s_len = len;
    }
    __syncthreads();
    const int len = s_len;
    float* out = paths + (size_t)b * max_len * dim;
    for (int i = lane; i < max(len, 0) * dim; i += blockDim.x) {
        const int k = i / dim, d = i - k * dim;
        const int node = chain[k];
        out[i] = node >= 0 ? TA[(size_t)d * N + node] : TB[(size_t)d * N + (-1 - node)];
    }
    __syncthreads();
    float c = 0.0f;
    for (int k = lane; k + 1 < len; k += blockDim.x) {
        float s2 = 0.0f;
        for (int d = 0; d < dim; ++d) {
            const float df = out[(k + 1) * dim + d] - out[k * dim + d];
            s2 = fmaf(df, df, s2);
        }
        c += sqrtf(s2);
    }
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) c += __shfl_xor_sync(0xffffffffu, c, off);
    if (lane == 0) {
        lengths[b] = len;
        costs[b] = len > 0 ? c : INFINITY;
    }
}

cudaError_t launch_extract_paths(int B, int dim, int N, const float* ta, const float* tb, const int32_t* pa,
                                 const int32_t* pb, const int32_t* conn, const int32_t* solved, int max_len,
                                 float* paths, int32_t* lengths, float* costs, cudaStream_t st) {
    const size_t smem = (size_t)max_len * sizeof(int);
    cudaError_t e;
    static DynLimit limit[kDynLimitDevices];
    if (smem > 48 * 1024 &&
        (e = raise_dyn_limit(reinterpret_cast<const void*>(extract_paths_kernel), limit, smem)) != cudaSuccess)
        return e;
    extract_paths_kernel<<<B, 32, smem, st>>>(B, dim, N, ta, tb, pa, pb, conn, solved, max_len, paths, lengths,
                                              costs);
    return cudaGetLastError();
}

// Result block: one [B,16] int32 row per problem (columns kBlk*), the scalars
// a caller reads back in one copy.  Column kBlkOffset is the exclusive prefix
// sum of the solved path lengths (one CTA, chunks of 1024 problems scanned
// with warp shuffles), or -1 for a problem whose path is not packed: unsolved,
// longer than the path buffer, or past packed_cap waypoints.
__global__ void result_block_kernel(int B, const ResultSrc R, int32_t* block, long long packed_cap) {
    __shared__ long long warp_sum[32];
    __shared__ long long s_carry;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    if (tid == 0) s_carry = 0;
    __syncthreads();
    for (int b0 = 0; b0 < B; b0 += blockDim.x) {
        const int b = b0 + tid;
        int len = 0;
        if (b < B) len = (R.solved[b] == 1 && R.lengths[b] > 0) ? R.lengths[b] : 0;
        long long x = len;  // inclusive scan within the warp
#pragma unroll
        for (int off = 1; off < 32; off <<= 1) {
            const long long y = __shfl_up_sync(0xffffffffu, x, off);
            if (lane >= off) x += y;
        }
        if (lane == 31) warp_sum[warp] = x;
        __syncthreads();
        if (warp == 0) {
            const int nwarps = blockDim.x >> 5;
            long long v = lane < nwarps ? warp_sum[lane] : 0;
#pragma unroll
            for (int off = 1; off < 32; off <<= 1) {
                const long long y = __shfl_up_sync(0xffffffffu, v, off);
                if (lane >= off) v += y;
            }
            if (lane < nwarps) warp_sum[lane] = v;  // inclusive over warps
        }
        __syncthreads();
        const long long carry = s_carry;
        const long long excl = carry + (warp > 0 ? warp_sum[warp - 1] : 0) + x - len;
        if (b < B) {
            int32_t* row = block + (size_t)b * 16;
            row[kBlkSizeA] = R.sizes[2 * b];
            row[kBlkSizeB] = R.sizes[2 * b + 1];
            row[kBlkCompletedA] = R.completed[2 * b];
            row[kBlkCompletedB] = R.completed[2 * b + 1];
            row[kBlkIterations] = R.iterations[b];
            row[kBlkConn + 0] = R.conn[3 * b];
            row[kBlkConn + 1] = R.conn[3 * b + 1];
            row[kBlkConn + 2] = R.conn[3 * b + 2];
            row[kBlkSolved] = R.solved[b];
            row[kBlkKernelMs] = __float_as_int(R.kernel_ms[b]);
            row[kBlkLength] = R.lengths[b];
            row[kBlkCost] = __float_as_int(R.costs[b]);
            row[kBlkOffset] = (len > 0 && excl + len <= packed_cap) ? (int32_t)excl : -1;
            row[13] = row[14] = row[15] = 0;
        }
        __syncthreads();
        if (tid == blockDim.x - 1) s_carry = carry + warp_sum[(blockDim.x >> 5) - 1];
        __syncthreads();
    }
}

// Solved paths copied back to back into packed (the offsets of the result
// block), so that a caller reads every path with one contiguous copy.
__global__ void pack_paths_kernel(int B, int dim, int max_len, const float* paths, const int32_t* block,
                                  float* packed) {
    const int b = blockIdx.x;
    const int32_t* row = block + (size_t)b * 16;
    const int off = row[kBlkOffset], len = row[kBlkLength];
    if (off < 0 || len <= 0) return;
    const float* src = paths + (size_t)b * max_len * dim;
    float* dst = packed + (size_t)off * dim;
    for (int i = threadIdx.x; i < len * dim; i += blockDim.x) dst[i] = src[i];
}

cudaError_t launch_result_block(int B, int dim, int max_len, const ResultSrc& R, int32_t* block,
                                const float* paths, float* packed, long long packed_cap, cudaStream_t st) {
    result_block_kernel<<<1, 1024, 0, st>>>(B, R, block, packed ? packed_cap : 0);
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess || !packed || packed_cap <= 0) return e;
    pack_paths_kernel<<<B, 64, 0, st>>>(B, dim, max_len, paths, block, packed);
    return cudaGetLastError();
}

}  // namespace prrtc
