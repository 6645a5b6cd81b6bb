// smooth.cu -- hand-written adjoint of the post-plan smoothing cost.  sm_100a.
//
// For a path of W waypoints q_w (dim each):
//   C = sum_w sum_pairs softplus_beta(margin - d_pair(q_w)) + w_len * sum_w |q_{w+1} - q_w|^2
// over every (robot sphere, world primitive) pair and every self pair, with
// softplus_beta(x) = log(1 + exp(beta x)) / beta.
//
// Backward pass per waypoint, nothing stored between the forward and backward
// sweeps except per-sphere centres (a warp per waypoint, or a lane per waypoint
// for paths of one scene):
//   1. recompute FK (joint-local transforms in parallel, then the chain in joint
//      order) and the sphere centres c_s;
//   2. g_s = dC/dc_s from every pair: -sigmoid(beta (m - d)) * dd/dc_s;
//   3. per frame f: G_f = sum g_s, M_f = sum c_s x g_s over its spheres, then
//      folded into parents in reverse topological order (subtree sums);
//   4. joint j with world pose (R_j, t_j) and twist (v, w):
//        dC/dv_j = (R_j w) . (M_j - t_j x G_j) + (R_j v) . G_j
//      (a point p below joint j moves with dp/dv_j = (R_j w) x (p - t_j) + R_j v);
//   5. dC/dq_a = sum over joints driven by a of dv_j/dq_a * dC/dv_j (1 for an
//      actuated joint, mimic_mul for a mimic joint) plus the length term.
#include <cuda_runtime.h>
#include <limits.h>
#include <math.h>

#include <algorithm>
#include <mutex>
#include <type_traits>

#include "kernels.h"
#include "prrtc_device.cuh"

namespace prrtc {

// softplus_beta(x) and sigmoid(beta x) from one exponential: with z = beta x
// and e = exp(-|z|), softplus_beta = (max(z, 0) + log1p(e)) / beta and
// sigmoid = 1/(1+e) for z >= 0, e/(1+e) otherwise.  Below z = kTailZ a pair
// adds less than exp(kTailZ)/beta (below 1e-15 for beta >= 1) to the cost and
// to every gradient entry; its sigmoid is reported as 0 so that callers can
// skip the gradient scatter.
constexpr float kTailZ = -34.0f;

// log1p(e) for e in [0, 1] without branches: log1p(e) = 2 atanh(s) with
// s = e / (2 + e) in [0, 1/3], and atanh(s) = s + s^3/3 + s^5/5 + ... summed
// to s^15 (the first omitted term is below 1.5e-9 of the sum for s <= 1/3).
__device__ __forceinline__ float log1p_unit(float e) {
    const float s = __fdividef(e, 2.0f + e);
    const float s2 = s * s;
    float p = 1.0f / 15.0f;
    p = fmaf(p, s2, 1.0f / 13.0f);
    p = fmaf(p, s2, 1.0f / 11.0f);
    p = fmaf(p, s2, 1.0f / 9.0f);
    p = fmaf(p, s2, 1.0f / 7.0f);
    p = fmaf(p, s2, 1.0f / 5.0f);
    p = fmaf(p, s2, 1.0f / 3.0f);
    p = fmaf(p, s2, 1.0f);
    return 2.0f * s * p;
}

struct SmoothArgs {
    const unsigned char* blob;
    const int2* pairs;
    size_t blob_stride;   // bytes between the scenes of consecutive paths (0: one scene for every path)
    size_t pairs_stride;  // int2 between the self-pair lists of consecutive paths (0: shared list)
    int J, S, dim;
    const float* wp;
    int P, W;
    float margin, beta, w_len;
    float* cost;
    float* grad;
};

constexpr int kStageRow = 36;  // a value per lane and a 16-byte step, for the banks
constexpr int kStage = 6 * kStageRow + 32;

// per-warp shared memory: pose J*12, ctr S*4, g S*4, acc J*8, stage, dv J, q dim (padded)
__host__ __device__ inline int smooth_warp_floats(int J, int S) {
    return (J * 12 + S * 4 + S * 4 + J * 8 + kStage + J + kDimMax + 3) & ~3;  // keep every warp slice 16-byte aligned
}

// Accumulate the cost term of a pair at distance d.  sig = sigmoid(beta
// (margin - d)) is the factor of -dd/dc in the gradient (0 for a skipped pair).
template <bool COST>
__device__ __forceinline__ void pair_term(float d, float margin, float beta, float inv_beta, float& cost,
                                          float& sig) {
    const float z = beta * (margin - d);
    const float e = __expf(-fabsf(z));
    if constexpr (COST) cost = fmaf(fmaxf(z, 0.0f) + log1p_unit(e), inv_beta, cost);
    const float r = __fdividef(1.0f, 1.0f + e);
    sig = z >= kTailZ ? (z >= 0.0f ? r : e * r) : 0.0f;
}

// |v| and 1/|v| (0 and 0 for v = 0) from one reciprocal square root
__device__ __forceinline__ void norm_rnorm(float d2, float& n, float& rn) {
    rn = d2 > 0.0f ? rsqrtf(d2) : 0.0f;
    n = d2 * rn;
}

// v of each lane of `on` added to the floats at base[key * stride + 0 .. N), lanes
// of one key in lane order, so the sums are the same bits in every run and launch.
// `heads` starts the runs of lanes of one key (lane 0 is one); `apart`: no two
// runs have the same key, so a lane per run and component may add its run's values,
// else the runs follow one another.  `stage`: N rows of kStageRow floats and a row
// of 32 masks.  A chain of some 8 cycles per value from shared memory; shared-memory
// float atomics take the same order, but by compare-and-swap rounds, and a search
// for equal keys by __match_any_sync costs a pass per key.
template <int N>
__device__ __forceinline__ void add_runs(unsigned on, unsigned heads, bool apart, int key, float* base, int stride,
                                         const float (&v)[N], float* stage) {
    constexpr unsigned kAll = 0xffffffffu;
    constexpr int kRuns = 32 / N;
    const int lane = threadIdx.x & 31, runs = __popc(heads), nth = lane / N, c = lane - nth * N;
    unsigned* masks = reinterpret_cast<unsigned*>(stage + N * kStageRow);
#pragma unroll
    for (int i = 0; i < N; ++i) stage[i * kStageRow + lane] = v[i];
    if (heads >> lane & 1u) {  // the lanes of the run that starts here
        const unsigned above = heads & (kAll - 1u << lane), next = above & (0u - above);
        masks[__popc(heads & ((1u << lane) - 1u))] = (next - 1u) & (kAll << lane) & on;
    }
    __syncwarp();
    const int step = apart ? kRuns : 1;
    for (int r0 = 0; r0 < runs; r0 += step) {
        const int r = r0 + nth;
        const unsigned mine = nth < step && r < runs ? masks[r] : 0u;
        float* b = base + __shfl_sync(kAll, key, mine ? __ffs(mine) - 1 : 0) * stride + c;
        if (mine) {
            const float* row = stage + c * kStageRow;
            int i = (__ffs(mine) - 1) & ~3;
            const int end = 32 - __clz(mine);
            float sum = *b;
            do {  // 8 lanes of the run at a time
                const float4 t = *reinterpret_cast<const float4*>(row + i), u = *reinterpret_cast<const float4*>(row + i + 4);
                const unsigned m = mine >> i;
                if (m & 1u) sum += t.x;
                if (m & 2u) sum += t.y;
                if (m & 4u) sum += t.z;
                if (m & 8u) sum += t.w;
                if (m & 16u) sum += u.x;
                if (m & 32u) sum += u.y;
                if (m & 64u) sum += u.z;
                if (m & 128u) sum += u.w;
                i += 8;
            } while (i < end);
            *b = sum;
        }
        __syncwarp();
    }
}

// A warp per waypoint, WARPS waypoints of one path per CTA, the scene staged in
// shared memory (STAGED) or read from global memory.  Every sum is taken in a
// fixed order, so a gradient is the same bits in every run and launch: a
// descent of normalised steps crosses the kinks of box distances, where sums in
// another order move single paths by 1e-3 within 50 steps.
//
// Bound by the latency of its dependent chains (a waypoint's 4,376 pairs in one
// warp; at 32 paths 3.5 warps per scheduler issue 55% of the time).  32 paths x 64
// waypoints in tabletop worlds of their own: 119 -> 57 us for the gradient alone,
// from ordered sums over runs of pairs in the place of shared-memory atomics, the
// next pairs fetched ahead of the sums, three lanes in the place of one for the
// frames' chain, and the scene in shared memory; the bits are those of the
// atomics.  Two spheres per lane for each primitive, in the place of two passes
// over them, measured the same at 32 paths and 4% slower at 128.
// COST false: the gradient alone, zero at a path's end points (a descent step).
template <int WARPS, bool STAGED, bool COST>
__global__ void __launch_bounds__(WARPS * 32) smooth_kernel(SmoothArgs a, int blob_cap, int per_path) {
    extern __shared__ __align__(128) unsigned char dsm[];
    __shared__ __align__(8) uint64_t mbar;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    // per_path CTAs for each path, or (one scene for all, per_path 0) all paths'
    // waypoints one after the other
    int p, w;
    bool mine;
    if (per_path > 0) {
        p = blockIdx.x / per_path;
        w = (blockIdx.x - p * per_path) * WARPS + warp;
        mine = w < a.W;
    } else {
        const long long c = (long long)blockIdx.x * WARPS + warp;
        p = (int)(c / a.W);
        w = (int)(c - (long long)p * a.W);
        mine = c < (long long)a.P * a.W;
    }
    const unsigned char* gblob = a.blob + (size_t)p * a.blob_stride;  // stride 0 where a CTA spans paths
    if constexpr (STAGED) {
        const int bytes = min(reinterpret_cast<const BlobHeader*>(gblob)->used_bytes, blob_cap);
        if (threadIdx.x == 0) mbar_init(&mbar);
        __syncthreads();
        uint32_t phase = 0;
        if (!stage_blob(dsm, gblob, bytes, &mbar, phase, nullptr, 0, kWaitLimit)) {
            // the bulk copy did not arrive in time: copy the scene with plain loads
            for (int i = threadIdx.x; i < bytes / 16; i += WARPS * 32)
                reinterpret_cast<uint4*>(dsm)[i] = reinterpret_cast<const uint4*>(gblob)[i];
            __syncthreads();
        }
    }
    if (!mine) return;
    if constexpr (!COST) {
        if (w == 0 || w == a.W - 1) {
            if (lane < a.dim) a.grad[((size_t)p * a.W + w) * a.dim + lane] = 0.0f;
            return;
        }
    }
    const Scene sc = scene_view(STAGED ? dsm : gblob);
    const int2* pairs = a.pairs + (size_t)p * a.pairs_stride;
    const BlobHeader& h = *sc.h;
    const int J = a.J, S = a.S, dim = a.dim;
    float* base = reinterpret_cast<float*>(dsm + (STAGED ? blob_cap : 0)) + (size_t)warp * smooth_warp_floats(J, S);
    float* pose = base;
    float4* ctr = reinterpret_cast<float4*>(pose + J * 12);
    float4* g = ctr + S;
    float* acc = reinterpret_cast<float*>(g + S);  // [J][8]: G xyz, M xyz
    float* stage = acc + J * 8;  // add_runs' rows
    float* dv = stage + kStage;
    float* q = dv + J;
    const float* qw = a.wp + ((size_t)p * a.W + w) * dim;
    if (lane < dim) q[lane] = qw[lane];
    __syncwarp();
    // 1. FK (recomputed) and centres
    for (int j = lane; j < J; j += 32) {
        const JointRec& jr = sc.joints[j];
        joint_local(jr, joint_value(jr, q), &pose[j * 12]);
    }
    __syncwarp();
    // the chain in joint order: row r of a frame needs row r of its parent's, so
    // three lanes take a row each (the operations of `compose`)
    for (int j = 0; j < J; ++j) {
        const int pj = sc.joints[j].idx.x;
        if (pj < 0 || pj >= j) continue;
        float o[4] = {0.0f, 0.0f, 0.0f, 0.0f};
        if (lane < 3) {
            const float* A = &pose[pj * 12];
            const float* L = &pose[j * 12];
            const float x = A[3 * lane], y = A[3 * lane + 1], z = A[3 * lane + 2];
#pragma unroll
            for (int c = 0; c < 3; ++c) o[c] = fmaf(x, L[c], fmaf(y, L[3 + c], z * L[6 + c]));
            o[3] = fmaf(x, L[9], fmaf(y, L[10], fmaf(z, L[11], A[9 + lane])));
        }
        __syncwarp();
        if (lane < 3) {
            float* T = &pose[j * 12];
#pragma unroll
            for (int c = 0; c < 3; ++c) T[3 * lane + c] = o[c];
            T[9 + lane] = o[3];
        }
        __syncwarp();
    }
    for (int s = lane; s < S; s += 32) {
        const int f = sc.sfr[s];
        const float4 l = sc.sph[s];
        ctr[s] = f >= 0 ? xform_point(&pose[f * 12], l) : make_float4(kFar, kFar, kFar, l.w);
        g[s] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    }
    for (int i = lane; i < J * 8; i += 32) acc[i] = 0.0f;
    __syncwarp();
    // 2a. world pairs: one sphere per lane
    float cost = 0.0f;
    const float inv_beta = 1.0f / a.beta;
    for (int s = lane; s < S; s += 32) {
        if (sc.sfr[s] < 0) continue;
        const float4 cs = ctr[s];
        const float r = cs.w;
        float gx = 0.0f, gy = 0.0f, gz = 0.0f;
        for (int o = 0; o < h.Ns; ++o) {
            const float4 o1 = sc.ws[2 * o + 1];
            const float4 ob = make_float4(o1.x, o1.y, o1.z, -0.5f * sc.ws[2 * o].w);
            const float dx = cs.x - ob.x, dy = cs.y - ob.y, dz = cs.z - ob.z;
            float n, rn, sig;
            norm_rnorm(fmaf(dx, dx, fmaf(dy, dy, dz * dz)), n, rn);
            pair_term<COST>(n - r - ob.w, a.margin, a.beta, inv_beta, cost, sig);
            const float k = -sig * rn;
            gx = fmaf(k, dx, gx); gy = fmaf(k, dy, gy); gz = fmaf(k, dz, gz);
        }
        for (int o = 0; o < h.Nc; ++o) {
            const float4 p1 = sc.wc[3 * o], dp = sc.wc[3 * o + 1], dl = sc.wc[3 * o + 2];
            const float wx = cs.x - p1.x, wy = cs.y - p1.y, wz = cs.z - p1.z;
            const float t = __saturatef(fmaf(dp.x, cs.x, fmaf(dp.y, cs.y, fmaf(dp.z, cs.z, dp.w))));
            const float ex = fmaf(-t, dl.x, wx), ey = fmaf(-t, dl.y, wy), ez = fmaf(-t, dl.z, wz);
            float n, rn, sig;
            norm_rnorm(fmaf(ex, ex, fmaf(ey, ey, ez * ez)), n, rn);
            pair_term<COST>(n - r - p1.w, a.margin, a.beta, inv_beta, cost, sig);
            const float k = -sig * rn;
            gx = fmaf(k, ex, gx); gy = fmaf(k, ey, gy); gz = fmaf(k, ez, gz);
        }
        for (int o = 0; o < h.Nb; ++o) {
            // records are stored scaled by 1/kBoxScale (a power of two): undo exactly
            float4 ax[3] = {sc.wb[4 * o], sc.wb[4 * o + 1], sc.wb[4 * o + 2]};
#pragma unroll
            for (int k = 0; k < 3; ++k)
                ax[k] = make_float4(ax[k].x * kBoxScale, ax[k].y * kBoxScale, ax[k].z * kBoxScale, ax[k].w * kBoxScale);
            float4 hl = sc.wb[4 * o + 3];
            hl = make_float4(hl.x * kBoxScale, hl.y * kBoxScale, hl.z * kBoxScale, 0.0f);
            const float hh[3] = {hl.x, hl.y, hl.z};
            // signed distance to the box without branches: outside, |max(q, 0)|
            // with gradient sum_k sign(l_k) max(q_k, 0)/n a_k; inside, the
            // largest q_k (first axis on ties) with gradient sign(l_k) a_k
            float l[3], qv[3];
#pragma unroll
            for (int k = 0; k < 3; ++k) {
                l[k] = fmaf(ax[k].x, cs.x, fmaf(ax[k].y, cs.y, fmaf(ax[k].z, cs.z, ax[k].w)));
                qv[k] = fabsf(l[k]) - hh[k];
            }
            const float p0 = fmaxf(qv[0], 0.0f), p1 = fmaxf(qv[1], 0.0f), p2 = fmaxf(qv[2], 0.0f);
            const float out2 = fmaf(p0, p0, fmaf(p1, p1, p2 * p2));
            float n, rn;
            norm_rnorm(out2, n, rn);
            const float qmax = fmaxf(qv[0], fmaxf(qv[1], qv[2]));
            const bool outside = out2 > 0.0f;
            const float d = (outside ? n : qmax) - r;
            const bool k0 = qv[0] == qmax, k1 = !k0 && qv[1] == qmax, k2 = !k0 && !k1;
            const float c0 = copysignf(outside ? p0 * rn : (k0 ? 1.0f : 0.0f), l[0]);
            const float c1 = copysignf(outside ? p1 * rn : (k1 ? 1.0f : 0.0f), l[1]);
            const float c2 = copysignf(outside ? p2 * rn : (k2 ? 1.0f : 0.0f), l[2]);
            const float ddx = fmaf(c0, ax[0].x, fmaf(c1, ax[1].x, c2 * ax[2].x));
            const float ddy = fmaf(c0, ax[0].y, fmaf(c1, ax[1].y, c2 * ax[2].y));
            const float ddz = fmaf(c0, ax[0].z, fmaf(c1, ax[1].z, c2 * ax[2].z));
            float sig;
            pair_term<COST>(d, a.margin, a.beta, inv_beta, cost, sig);
            gx = fmaf(-sig, ddx, gx); gy = fmaf(-sig, ddy, gy); gz = fmaf(-sig, ddz, gz);
        }
        for (int o = 0; o < h.Nh; ++o) {
            const float4 hs = sc.wh[o];
            const float d = fmaf(hs.x, cs.x, fmaf(hs.y, cs.y, fmaf(hs.z, cs.z, hs.w))) - r;
            float sig;
            pair_term<COST>(d, a.margin, a.beta, inv_beta, cost, sig);
            gx = fmaf(-sig, hs.x, gx); gy = fmaf(-sig, hs.y, gy); gz = fmaf(-sig, hs.z, gz);
        }
        g[s] = make_float4(gx, gy, gz, 0.0f);
    }
    __syncwarp();
    // 2b. self pairs (explicit list), 32 at a time, into both spheres; the terms of
    // two lots and the pairs of the next two are on their way while sums are taken
    auto pair_at = [&](int k) { return k < h.P ? __ldg(&pairs[k]) : make_int2(-1, -1); };
    auto self_term = [&](int2 pr, float (&v)[3]) {
        v[0] = v[1] = v[2] = 0.0f;
        if (!(pr.x >= 0 && pr.y >= 0 && pr.x < S && pr.y < S && sc.sfr[pr.x] >= 0 && sc.sfr[pr.y] >= 0)) return false;
        const float4 ci = ctr[pr.x], cj = ctr[pr.y];
        const float dx = ci.x - cj.x, dy = ci.y - cj.y, dz = ci.z - cj.z;
        float n, rn, sig;
        norm_rnorm(fmaf(dx, dx, fmaf(dy, dy, dz * dz)), n, rn);
        pair_term<COST>(n - ci.w - cj.w, a.margin, a.beta, inv_beta, cost, sig);
        const float kk = -sig * rn;
        v[0] = kk * dx; v[1] = kk * dy; v[2] = kk * dz;
        return sig != 0.0f;  // else nothing to add
    };
    auto self_sum = [&](int k, int2 pr, bool on, const float (&v)[3]) {
        const unsigned live = __ballot_sync(0xffffffffu, on);
        if (!live) return;
        // runs of pairs with one first sphere and rising second ones: in a run the
        // second spheres are all different
        const int px = __shfl_up_sync(0xffffffffu, pr.x, 1), py = __shfl_up_sync(0xffffffffu, pr.y, 1);
        const bool head = lane == 0 || pr.x != px || pr.y <= py;
        const unsigned heads = __ballot_sync(0xffffffffu, head);
        const bool apart = __all_sync(0xffffffffu, lane == 0 || !head || pr.x > px || k >= h.P);
        add_runs<3>(live, heads, apart, pr.x, reinterpret_cast<float*>(g), 4, v, stage);
        const int run = __popc(heads & (0xffffffffu >> (31 - lane)));
        for (int r = 1; r <= __popc(heads); ++r) {
            if (on && run == r) {
                float4* t = &g[pr.y];
                t->x -= v[0]; t->y -= v[1]; t->z -= v[2];
            }
            __syncwarp();
        }
    };
    int2 pr0 = pair_at(lane), pr1 = pair_at(32 + lane);
    for (int k0 = 0; k0 < h.P; k0 += 64) {
        const int2 next0 = pair_at(k0 + 64 + lane), next1 = pair_at(k0 + 96 + lane);
        float v0[3], v1[3];
        const bool on0 = self_term(pr0, v0), on1 = self_term(pr1, v1);
        self_sum(k0 + lane, pr0, on0, v0);
        self_sum(k0 + 32 + lane, pr1, on1, v1);
        pr0 = next0;
        pr1 = next1;
    }
    __syncwarp();
    // 3. frame sums
    for (int s0 = 0; s0 < S; s0 += 32) {
        const int s = min(s0 + lane, S - 1), f = sc.sfr[s];
        const float4 cs = ctr[s], gs = g[s];
        const float v[6] = {gs.x, gs.y, gs.z, cs.y * gs.z - cs.z * gs.y, cs.z * gs.x - cs.x * gs.z,
                            cs.x * gs.y - cs.y * gs.x};
        const int fp = __shfl_up_sync(0xffffffffu, f, 1);
        const bool head = lane == 0 || f != fp;
        add_runs<6>(__ballot_sync(0xffffffffu, s0 + lane < S && f >= 0), __ballot_sync(0xffffffffu, head),
                    __all_sync(0xffffffffu, !head || lane == 0 || f > fp), f, acc, 8, v, stage);
    }
    // 4. reverse sweep: subtree sums a component per lane, then a joint per lane
    if (lane < 6) {
        for (int j = J - 1; j >= 0; --j) {
            const int pj = sc.joints[j].idx.x;
            if (pj >= 0 && pj < j) acc[pj * 8 + lane] += acc[j * 8 + lane];
        }
    }
    __syncwarp();
    for (int j = lane; j < J; j += 32) {
        const JointRec& jr = sc.joints[j];
        const float* F = &pose[j * 12];
        const float* A = &acc[j * 8];
        const float wx = fmaf(F[0], jr.tw.x, fmaf(F[1], jr.tw.y, F[2] * jr.tw.z));
        const float wy = fmaf(F[3], jr.tw.x, fmaf(F[4], jr.tw.y, F[5] * jr.tw.z));
        const float wz = fmaf(F[6], jr.tw.x, fmaf(F[7], jr.tw.y, F[8] * jr.tw.z));
        const float vx = fmaf(F[0], jr.tv.x, fmaf(F[1], jr.tv.y, F[2] * jr.tv.z));
        const float vy = fmaf(F[3], jr.tv.x, fmaf(F[4], jr.tv.y, F[5] * jr.tv.z));
        const float vz = fmaf(F[6], jr.tv.x, fmaf(F[7], jr.tv.y, F[8] * jr.tv.z));
        const float tx = F[9], ty = F[10], tz = F[11];
        const float mx = A[3] - (ty * A[2] - tz * A[1]);
        const float my = A[4] - (tz * A[0] - tx * A[2]);
        const float mz = A[5] - (tx * A[1] - ty * A[0]);
        dv[j] = wx * mx + wy * my + wz * mz + vx * A[0] + vy * A[1] + vz * A[2];
    }
    __syncwarp();
    // 5. joint-space gradient + length term
    float lenc = 0.0f;
    if (lane < dim) {
        float gq = 0.0f;
        for (int j = 0; j < J; ++j) {
            const JointRec& jr = sc.joints[j];
            if (jr.idx.z >= 0) {
                if (jr.idx.z == lane) gq = fmaf(jr.tv.w, dv[j], gq);
            } else if (jr.idx.y == lane) {
                gq += dv[j];
            }
        }
        const float qc = q[lane];
        if (w + 1 < a.W) {
            const float dn = a.wp[((size_t)p * a.W + w + 1) * dim + lane] - qc;
            gq -= 2.0f * a.w_len * dn;
            lenc = a.w_len * dn * dn;
        }
        if (w > 0) {
            const float dp = qc - a.wp[((size_t)p * a.W + w - 1) * dim + lane];
            gq += 2.0f * a.w_len * dp;
        }
        if (a.grad) a.grad[((size_t)p * a.W + w) * dim + lane] = gq;
    }
    if constexpr (COST) {
        cost += lenc;
#pragma unroll
        for (int off = 16; off > 0; off >>= 1) cost += __shfl_xor_sync(0xffffffffu, cost, off);
        if (lane == 0) atomicAdd(&a.cost[p], cost);
    }
}

// One step of the descent for every path: x - lr g / max(|g|, 1e-12), held
// between the joint limits; norms [P] are the gradients' lengths.  The
// operations and their order are those of the tensor expression (multiply,
// divide, subtract, then the two bounds, NaN kept).
__global__ void smooth_update_kernel(float* __restrict__ x, const float* __restrict__ g, const float* __restrict__ norms,
                                     const float* __restrict__ lo, const float* __restrict__ hi, float lr, int per_path,
                                     int dim, long long n) {
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const float len = norms[i / per_path], gn = len != len ? len : fmaxf(len, 1e-12f);
    float v = __fsub_rn(x[i], __fdiv_rn(__fmul_rn(lr, g[i]), gn));
    const int d = (int)(i % dim);
    v = v != v || lo[d] != lo[d] ? v + lo[d] : fmaxf(v, lo[d]);
    v = v != v || hi[d] != hi[d] ? v + hi[d] : fminf(v, hi[d]);
    x[i] = v;
}

cudaError_t launch_smooth_update(float* x, const float* g, const float* norms, const float* lo, const float* hi,
                                 float lr, int P, int W, int dim, cudaStream_t st) {
    const long long n = (long long)P * W * dim;
    if (n <= 0) return cudaSuccess;
    smooth_update_kernel<<<(unsigned)((n + 255) / 256), 256, 0, st>>>(x, g, norms, lo, hi, lr, W * dim, dim, n);
    return cudaGetLastError();
}

// ----------------------------------------------------------------------------- a warp's lanes are waypoints

// The form for paths of one scene and robots of up to 32 joints, unless the
// caller wants the sums in smooth_kernel's order: a CTA takes 32 waypoints, one
// per lane.  All lanes of a warp then look at the same primitive, read from
// shared memory once for the warp, with neighbouring waypoints' distances, which
// are alike, so the warp as a whole takes the short series for pairs that are far
// apart (below) instead of the full softplus.
//
// The gradient is the same bits in every run of the same call: every one of its
// sums has one order.  The warps draw units from a counter, a unit being two
// spheres against every primitive or against every sphere that they make a self
// pair with.  A sphere's sums stay in registers and meet in shared memory as two
// terms, so their order does not matter, and frame sums go over the spheres in
// order.  A self pair is computed twice for that, once for each of its spheres:
// adding its terms to the other one by atomics has another order in every run (369 us
// a call for 512 paths x 64 waypoints in the tabletop scene, 344 with this), and terms
// left in shared memory for each sphere's warp to add after a barrier took 571 us.
// (The cost is added up by atomics.)
//
// Bound by instruction issue: 77% of the issue slots, 51 instructions per computed
// pair and warp (a reciprocal square root and an exponential each, two reciprocals
// more near contact: the special-function pipe is 31% busy).  Against a warp per
// waypoint with a sphere per lane (smooth_kernel), 4,376 pairs each: 512 paths x 64
// waypoints, tabletop scene, 858 -> 322 us of kernel time; 40 dual-arm paths x 96
// waypoints (44,360 pairs) 920 -> 346 us a call.  One sphere at a time instead of
// two was 7% slower, the library's exponential and reciprocal square root 45%.
struct SmoothBufs {
    float* pose;    // [32][J][12]
    float* ctr;     // [S][3][32] (the radius is the scene's)
    float* g;       // [S][3][32]; the joints' local transforms [32][J][12] before
    float* acc;     // [J][6][32] frame sums G, M
    float* q;       // [32][kDimMax], then dv [32][J]
    float* cost;    // [32]
    uint32_t* sub;  // [J] mask of the joint's subtree (itself included)
    uint32_t* adj;  // [S][words of S bits] the spheres that a sphere makes a self pair with
    int* next;      // unit counter, then whether the list repeats a pair
};

__host__ __device__ inline int smooth_g_bytes(int J, int S) { return S * 384 > J * 1536 ? S * 384 : J * 1536; }
__host__ __device__ inline int smooth_wide_bytes(int J, int S) {
    return 32 * J * 48 + S * 3 * 128 + smooth_g_bytes(J, S) + J * 6 * 128 + 32 * (kDimMax > J ? kDimMax : J) * 4 + 128 + 128 +
           align16(S * cdiv(S, 32) * 4) + 16;
}

__device__ __forceinline__ SmoothBufs smooth_bufs(unsigned char* p, int J, int S) {
    SmoothBufs b;
    b.pose = reinterpret_cast<float*>(p);   p += 32 * J * 48;
    b.ctr = reinterpret_cast<float*>(p);    p += S * 3 * 128;
    b.g = reinterpret_cast<float*>(p);      p += smooth_g_bytes(J, S);
    b.acc = reinterpret_cast<float*>(p);    p += J * 6 * 128;
    b.q = reinterpret_cast<float*>(p);      p += 32 * max(kDimMax, J) * 4;
    b.cost = reinterpret_cast<float*>(p);   p += 128;
    b.sub = reinterpret_cast<uint32_t*>(p); p += 128;
    b.adj = reinterpret_cast<uint32_t*>(p); p += align16(S * cdiv(S, 32) * 4);
    b.next = reinterpret_cast<int*>(p);
    return b;
}

// The hardware's exponential and reciprocal square root (2 ulp), without the
// code for denormal operands: t is finite and d2 at least 1e-36.
__device__ __forceinline__ float wide_ex2(float x) {
    float r;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r;
}
__device__ __forceinline__ float wide_rsqrt(float x) {
    float r;
    asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r;
}

// The larger operand, NaN where one is (fmaxf would give the other): a distance
// that is not a number stays one.
__device__ __forceinline__ float wide_max(float a, float b) {
    float r;
    asm("max.NaN.f32 %0, %1, %2;" : "=f"(r) : "f"(a), "f"(b));
    return r;
}

// Pair terms, all 32 lanes together.  z = beta (margin - d): cost collects
// softplus(z) in units of 1/beta, sig is the sigmoid, the factor of -dd/dc.
// With e = exp(-|z|):
//   some lane nearer than z = -5.6, or not a number: as pair_term;
//   all lanes below that (e < 2^-8): log1p(e) = e - e^2/2 + e^3/3 and e/(1+e) = e -
//     e^2 + e^3, both to e^3 (relative 6e-8, a float's rounding);
//   all lanes below the tail of pair_term (z = kTailZ): the cost only, as there
//     (false: no gradient).
// N terms at once, one vote for all (independent chains, half the branches).
template <int N>
__device__ __forceinline__ bool wide_terms(const float (&z)[N], float& cost, float (&sig)[N]) {
    float e[N], top = z[0];
#pragma unroll
    for (int k = 0; k < N; ++k) {
        e[k] = wide_ex2(-fabsf(z[k]) * 1.44269504089f);
        top = wide_max(top, z[k]);
    }
    if (__any_sync(0xffffffffu, !(top <= -5.6f))) {
#pragma unroll
        for (int k = 0; k < N; ++k) {
            const float r = __fdividef(1.0f, 1.0f + e[k]);
            cost += fmaxf(z[k], 0.0f) + log1p_unit(e[k]);
            sig[k] = z[k] >= 0.0f ? r : e[k] * r;
        }
        return true;
    }
    if (__any_sync(0xffffffffu, top > kTailZ)) {
#pragma unroll
        for (int k = 0; k < N; ++k) {
            cost = fmaf(e[k], fmaf(e[k], fmaf(e[k], 1.0f / 3.0f, -0.5f), 1.0f), cost);
            sig[k] = e[k] * fmaf(e[k], e[k] - 1.0f, 1.0f);
        }
        return true;
    }
#pragma unroll
    for (int k = 0; k < N; ++k) cost += e[k];
    return false;
}

// The CTAs of a cluster meet: writes before it, of every thread of them, are seen after it.
__device__ __forceinline__ void cluster_sync() {
    asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
    asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}
// The value at `p` (in this CTA's shared memory) in the cluster's CTA `rank`.
__device__ __forceinline__ float cluster_load(const float* p, int rank) {
    unsigned at;
    float v;
    asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(at) : "r"((unsigned)__cvta_generic_to_shared(p)), "r"(rank));
    asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(v) : "r"(at));
    return v;
}

template <int THREADS, int MINBLOCKS>
__global__ void __launch_bounds__(THREADS, MINBLOCKS)
    smooth_wide_kernel(SmoothArgs a, int blob_cap, int parts) {
    extern __shared__ __align__(128) unsigned char dsm[];
    __shared__ __align__(8) uint64_t mbar;
    constexpr unsigned kAll = 0xffffffffu;
    constexpr int T = THREADS, WARPS = THREADS / 32;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int J = a.J, S = a.S, dim = a.dim, W = a.W;
    // 32 of all paths' waypoints, one path after the other
    const long long n_all = (long long)a.P * W;
    const int group = blockIdx.x / parts, part = blockIdx.x - group * parts;
    const long long first = (long long)group * 32;
    const int nw = (int)min(32ll, n_all - first);
    const unsigned char* gblob = a.blob;
    const int2* pairs = a.pairs;
    const SmoothBufs B = smooth_bufs(dsm + blob_cap, J, S);
    if (tid == 0) {
        mbar_init(&mbar);
        B.next[0] = B.next[1] = 0;
    }
    const int adj_words = cdiv(S, 32);
    for (int i = tid; i < S * adj_words; i += T) B.adj[i] = 0u;
    for (int i = tid; i < 32 * dim; i += T) {
        const int w = i / dim, d = i - w * dim;
        B.q[w * kDimMax + d] = w < nw ? a.wp[first * dim + i] : 0.0f;
    }
    if (tid < 32) B.cost[tid] = 0.0f;
    __syncthreads();
    uint32_t phase = 0;
    const int bytes = min(reinterpret_cast<const BlobHeader*>(gblob)->used_bytes, blob_cap);
    if (!stage_blob(dsm, gblob, bytes, &mbar, phase, nullptr, 0, kWaitLimit)) {
        // the bulk copy did not arrive in time: copy the scene with plain loads
        for (int i = tid; i < bytes / 16; i += T) reinterpret_cast<uint4*>(dsm)[i] = reinterpret_cast<const uint4*>(gblob)[i];
        __syncthreads();
    }
    const Scene sc = scene_view(dsm);
    const BlobHeader& h = *sc.h;
    // 1. frames, subtree masks, sphere centres
    if (tid < J) {
        uint32_t m = 0u;
        for (int k = tid; k < J; ++k) {  // k is in tid's subtree iff tid is on k's way to the root
            int x = k;
            while (x > tid) {
                const int p = sc.joints[x].idx.x;
                x = p >= 0 && p < x ? p : -1;
            }
            m |= x == tid ? 1u << k : 0u;
        }
        B.sub[tid] = m;
    }
    // both directions of every self pair; a bit that was set already is a pair (or its reverse) that the list repeats
    // (four loads on their way together)
    for (int k0 = tid; k0 < h.P; k0 += 4 * T) {
        int2 pr[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) pr[i] = k0 + i * T < h.P ? __ldg(&pairs[k0 + i * T]) : make_int2(-1, -1);
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const int x = pr[i].x, y = pr[i].y;
            if (x < 0 || y < 0 || x >= S || y >= S || sc.sfr[x] < 0 || sc.sfr[y] < 0) continue;
            const uint32_t b0 = atomicOr(&B.adj[x * adj_words + (y >> 5)], 1u << (y & 31)) >> (y & 31);
            const uint32_t b1 = atomicOr(&B.adj[y * adj_words + (x >> 5)], 1u << (x & 31)) >> (x & 31);
            if ((b0 | b1) & 1u) B.next[1] = 1;
        }
    }
    // local transforms, a (waypoint, joint) per thread, then the chain: row r of a
    // frame needs row r of its parent's only, so a thread per (waypoint, row)
    // composes the joints in order, by the same operations as `compose`
    for (int i = tid; i < 32 * J; i += T) {
        const int w = i / J, j = i - w * J;
        const JointRec& jr = sc.joints[j];
        joint_local(jr, joint_value(jr, B.q + w * kDimMax), B.g + i * 12);
    }
    __syncthreads();
    if (tid < 96) {
        const int w = tid / 3, r = tid - w * 3;
        for (int j = 0; j < J; ++j) {
            const float* b = B.g + (w * J + j) * 12;
            float* o = B.pose + (w * J + j) * 12;
            const int p = sc.joints[j].idx.x;
            if (p >= 0 && p < j) {
                const float* a_ = B.pose + (w * J + p) * 12;
                const float x = a_[3 * r], y = a_[3 * r + 1], z = a_[3 * r + 2], t = a_[9 + r];
#pragma unroll
                for (int c = 0; c < 3; ++c) o[3 * r + c] = fmaf(x, b[c], fmaf(y, b[3 + c], z * b[6 + c]));
                o[9 + r] = fmaf(x, b[9], fmaf(y, b[10], fmaf(z, b[11], t)));
            } else {
#pragma unroll
                for (int c = 0; c < 3; ++c) o[3 * r + c] = b[3 * r + c];
                o[9 + r] = b[9 + r];
            }
        }
    }
    __syncthreads();
    for (int i = tid; i < S * 96; i += T) B.g[i] = 0.0f;
    for (int i = tid; i < S * 32; i += T) {
        const int s = i >> 5, w = i & 31, f = sc.sfr[s];
        float4 c = make_float4(kFar, kFar, kFar, 0.0f);
        if (f >= 0) {
            const float4* p = reinterpret_cast<const float4*>(B.pose + (w * J + f) * 12);
            const float4 p0 = p[0], p1 = p[1], p2 = p[2];
            const float F[12] = {p0.x, p0.y, p0.z, p0.w, p1.x, p1.y, p1.z, p1.w, p2.x, p2.y, p2.z, p2.w};
            c = xform_point(F, sc.sph[s]);
        }
        B.ctr[s * 96 + w] = c.x;
        B.ctr[s * 96 + 32 + w] = c.y;
        B.ctr[s * 96 + 64 + w] = c.z;
    }
    __syncthreads();
    auto centre = [&](int s, int w) {
        const float* x = B.ctr + s * 96 + w;
        return make_float4(x[0], x[32], x[64], sc.sph[s].w);
    };
    float total = 0.0f;
    // 2. units
    const int n_world = (S + 1) >> 1, n_units = 2 * n_world;
    const bool repeats = B.next[1] != 0;
    // how often the list has the pair of spheres i and j (both ways; twice for a sphere with itself), once unless it repeats pairs
    auto times = [&](int i, int j) {
        int n = 0;
        for (int k0 = 0; k0 < h.P; k0 += 32) {
            const int2 pr = k0 + lane < h.P ? __ldg(&pairs[k0 + lane]) : make_int2(-1, -1);
            n += __popc(__ballot_sync(kAll, pr.x == i && pr.y == j)) + __popc(__ballot_sync(kAll, pr.x == j && pr.y == i));
        }
        return n;
    };
    while (true) {
        int u = 0;
        if (lane == 0) u = atomicAdd(B.next, 1);
        u = part + parts * __shfl_sync(kAll, u, 0);
        if (u >= n_units) break;
        // spheres 2u and 2u + 1 against every primitive, or against their self-pair partners; an absent one's terms
        // vanish (its radius is far below 0)
        const bool world = u < n_world;
        if (!world) u -= n_world;
        const int Ns = world ? h.Ns : 0, Nc = world ? h.Nc : 0, Nb = world ? h.Nb : 0, Nh = world ? h.Nh : 0;
        const int words = world ? 0 : adj_words;
        float cost = 0.0f;  // of this unit (short sums lose less)
        float4 c[2];
        float gx[2], gy[2], gz[2];
        bool on[2];
#pragma unroll
        for (int k = 0; k < 2; ++k) {
            const int s = 2 * u + k;
            on[k] = s < S && sc.sfr[min(s, S - 1)] >= 0;
            c[k] = centre(min(s, S - 1), lane);
            if (!on[k]) c[k].w = -1e30f;
            gx[k] = gy[k] = gz[k] = 0.0f;
        }
        for (int o = 0; o < Ns; ++o) {
            const float4 ob = sc.ws[2 * o + 1];
            const float ro = -0.5f * sc.ws[2 * o].w;
            float dx[2], dy[2], dz[2], rn[2], z[2], sig[2];
#pragma unroll
            for (int k = 0; k < 2; ++k) {
                dx[k] = c[k].x - ob.x; dy[k] = c[k].y - ob.y; dz[k] = c[k].z - ob.z;
                const float d2 = wide_max(fmaf(dx[k], dx[k], fmaf(dy[k], dy[k], dz[k] * dz[k])), 1e-36f);
                rn[k] = wide_rsqrt(d2);
                z[k] = a.beta * (a.margin - (d2 * rn[k] - c[k].w - ro));
            }
            if (wide_terms<2>(z, cost, sig)) {
#pragma unroll
                for (int k = 0; k < 2; ++k) {
                    const float m = -sig[k] * rn[k];
                    gx[k] = fmaf(m, dx[k], gx[k]); gy[k] = fmaf(m, dy[k], gy[k]); gz[k] = fmaf(m, dz[k], gz[k]);
                }
            }
        }
        for (int o = 0; o < Nc; ++o) {
            const float4 p1 = sc.wc[3 * o], dp = sc.wc[3 * o + 1], dl = sc.wc[3 * o + 2];
            float ex[2], ey[2], ez[2], rn[2], z[2], sig[2];
#pragma unroll
            for (int k = 0; k < 2; ++k) {
                const float u_ = __saturatef(fmaf(dp.x, c[k].x, fmaf(dp.y, c[k].y, fmaf(dp.z, c[k].z, dp.w))));
                ex[k] = fmaf(-u_, dl.x, c[k].x - p1.x);
                ey[k] = fmaf(-u_, dl.y, c[k].y - p1.y);
                ez[k] = fmaf(-u_, dl.z, c[k].z - p1.z);
                const float d2 = wide_max(fmaf(ex[k], ex[k], fmaf(ey[k], ey[k], ez[k] * ez[k])), 1e-36f);
                rn[k] = wide_rsqrt(d2);
                z[k] = a.beta * (a.margin - (d2 * rn[k] - c[k].w - p1.w));
            }
            if (wide_terms<2>(z, cost, sig)) {
#pragma unroll
                for (int k = 0; k < 2; ++k) {
                    const float m = -sig[k] * rn[k];
                    gx[k] = fmaf(m, ex[k], gx[k]); gy[k] = fmaf(m, ey[k], gy[k]); gz[k] = fmaf(m, ez[k], gz[k]);
                }
            }
        }
        for (int o = 0; o < Nb; ++o) {
            // signed distance as in smooth_kernel, in units of kBoxScale metres (records are stored scaled)
            const float4 a0 = sc.wb[4 * o], a1 = sc.wb[4 * o + 1], a2 = sc.wb[4 * o + 2], hl = sc.wb[4 * o + 3];
            float l0[2], l1[2], l2[2], rn[2], z[2], sig[2];
            bool outside[2];
#pragma unroll
            for (int k = 0; k < 2; ++k) {
                l0[k] = fmaf(a0.x, c[k].x, fmaf(a0.y, c[k].y, fmaf(a0.z, c[k].z, a0.w)));
                l1[k] = fmaf(a1.x, c[k].x, fmaf(a1.y, c[k].y, fmaf(a1.z, c[k].z, a1.w)));
                l2[k] = fmaf(a2.x, c[k].x, fmaf(a2.y, c[k].y, fmaf(a2.z, c[k].z, a2.w)));
                const float q0 = fabsf(l0[k]) - hl.x, q1 = fabsf(l1[k]) - hl.y, q2 = fabsf(l2[k]) - hl.z;
                const float p0 = fmaxf(q0, 0.0f), p1 = fmaxf(q1, 0.0f), p2 = fmaxf(q2, 0.0f);
                const float out2 = fmaf(p0, p0, fmaf(p1, p1, p2 * p2));
                outside[k] = out2 > 0.0f;
                rn[k] = outside[k] ? rsqrtf(out2) : 0.0f;
                const float d = kBoxScale * (outside[k] ? out2 * rn[k] : fmaxf(q0, fmaxf(q1, q2))) - c[k].w;
                z[k] = a.beta * (a.margin - d);
            }
            if (wide_terms<2>(z, cost, sig)) {
#pragma unroll
                for (int k = 0; k < 2; ++k) {
                    const float q0 = fabsf(l0[k]) - hl.x, q1 = fabsf(l1[k]) - hl.y, q2 = fabsf(l2[k]) - hl.z;
                    const float qmax = fmaxf(q0, fmaxf(q1, q2)), m = -kBoxScale * sig[k];  // the axes are stored times kBoxInv
                    const bool k0 = q0 == qmax, k1 = !k0 && q1 == qmax, k2 = !k0 && !k1;
                    const float c0 = copysignf(outside[k] ? fmaxf(q0, 0.0f) * rn[k] : (k0 ? 1.0f : 0.0f), l0[k]);
                    const float c1 = copysignf(outside[k] ? fmaxf(q1, 0.0f) * rn[k] : (k1 ? 1.0f : 0.0f), l1[k]);
                    const float c2 = copysignf(outside[k] ? fmaxf(q2, 0.0f) * rn[k] : (k2 ? 1.0f : 0.0f), l2[k]);
                    gx[k] = fmaf(m, fmaf(c0, a0.x, fmaf(c1, a1.x, c2 * a2.x)), gx[k]);
                    gy[k] = fmaf(m, fmaf(c0, a0.y, fmaf(c1, a1.y, c2 * a2.y)), gy[k]);
                    gz[k] = fmaf(m, fmaf(c0, a0.z, fmaf(c1, a1.z, c2 * a2.z)), gz[k]);
                }
            }
        }
        for (int o = 0; o < Nh; ++o) {
            const float4 hs = sc.wh[o];
            float z[2], sig[2];
#pragma unroll
            for (int k = 0; k < 2; ++k)
                z[k] = a.beta * (a.margin - (fmaf(hs.x, c[k].x, fmaf(hs.y, c[k].y, fmaf(hs.z, c[k].z, hs.w))) - c[k].w));
            if (wide_terms<2>(z, cost, sig)) {
#pragma unroll
                for (int k = 0; k < 2; ++k) {
                    gx[k] = fmaf(-sig[k], hs.x, gx[k]); gy[k] = fmaf(-sig[k], hs.y, gy[k]); gz[k] = fmaf(-sig[k], hs.z, gz[k]);
                }
            }
        }
        const bool odd = 2 * u + 1 < S;
        for (int word = 0; word < words; ++word) {
            const uint32_t w0 = B.adj[2 * u * adj_words + word], w1 = odd ? B.adj[(2 * u + 1) * adj_words + word] : 0u;
            for (uint32_t rest = w0 | w1; rest; rest &= rest - 1u) {
                const int bit = __ffs(rest) - 1, j = 32 * word + bit;
                int n[2] = {(int)(w0 >> bit & 1u), (int)(w1 >> bit & 1u)};
                if (repeats) {
                    n[0] = n[0] ? times(2 * u, j) : 0;
                    n[1] = n[1] ? times(2 * u + 1, j) : 0;
                }
                const float4 cj = centre(j, lane);
                float dx[2], dy[2], dz[2], rn[2], z[2], sig[2];
#pragma unroll
                for (int k = 0; k < 2; ++k) {
                    dx[k] = c[k].x - cj.x; dy[k] = c[k].y - cj.y; dz[k] = c[k].z - cj.z;
                    const float d2 = wide_max(fmaf(dx[k], dx[k], fmaf(dy[k], dy[k], dz[k] * dz[k])), 1e-36f);
                    rn[k] = wide_rsqrt(d2);
                    z[k] = a.beta * (a.margin - (d2 * rn[k] - c[k].w - cj.w));
                }
                for (; n[0] > 0 || n[1] > 0; --n[0], --n[1]) {
                    if (n[0] <= 0) z[0] = -1e30f;  // not a pair: no term
                    if (n[1] <= 0) z[1] = -1e30f;
                    if (wide_terms<2>(z, cost, sig)) {
#pragma unroll
                        for (int k = 0; k < 2; ++k) {
                            if (n[k] <= 0) continue;
                            const float m = -sig[k] * rn[k];
                            gx[k] = fmaf(m, dx[k], gx[k]); gy[k] = fmaf(m, dy[k], gy[k]); gz[k] = fmaf(m, dz[k], gz[k]);
                        }
                    }
                }
            }
        }
        // the two units of a sphere add to zero: of two terms the order does not matter
#pragma unroll
        for (int k = 0; k < 2; ++k) {
            if (!on[k]) continue;
            float* G = B.g + (2 * u + k) * 96 + lane;
            atomicAdd(G, gx[k]); atomicAdd(G + 32, gy[k]); atomicAdd(G + 64, gz[k]);
        }
        total = fmaf(world ? 1.0f : 0.5f, cost, total);  // a self pair is in the units of both its spheres
    }
    atomicAdd(&B.cost[lane], total);
    __syncthreads();
    // 3. frame sums, a joint per warp over the spheres in order
    for (int j = warp; j < J; j += WARPS) {
        float A[6] = {0.0f, 0.0f, 0.0f, 0.0f, 0.0f, 0.0f};
        for (int s0 = 0; s0 < S; s0 += 32) {
            for (unsigned on = __ballot_sync(kAll, s0 + lane < S && sc.sfr[min(s0 + lane, S - 1)] == j); on; on &= on - 1u) {
                const int s = s0 + __ffs(on) - 1;
                const float4 c = centre(s, lane);
                const float x = B.g[s * 96 + lane], y = B.g[s * 96 + 32 + lane], z = B.g[s * 96 + 64 + lane];
                A[0] += x; A[1] += y; A[2] += z;
                A[3] += c.y * z - c.z * y;
                A[4] += c.z * x - c.x * z;
                A[5] += c.x * y - c.y * x;
            }
        }
#pragma unroll
        for (int k = 0; k < 6; ++k) B.acc[j * 192 + 32 * k + lane] = A[k];
    }
    __syncthreads();
    // 4. dC/dv of every joint from its subtree's sums (dv in the place of q)
    float* dv = B.q;
    for (int i = tid; i < J * 32; i += T) {
        const int j = i >> 5, w = i & 31;
        float A[6] = {0.0f, 0.0f, 0.0f, 0.0f, 0.0f, 0.0f};
        for (uint32_t m = B.sub[j]; m; m &= m - 1u) {
            const float* x = B.acc + (__ffs(m) - 1) * 192 + w;
#pragma unroll
            for (int k = 0; k < 6; ++k) A[k] += x[32 * k];
        }
        const JointRec& jr = sc.joints[j];
        const float* F = B.pose + (w * J + j) * 12;
        const float wx = fmaf(F[0], jr.tw.x, fmaf(F[1], jr.tw.y, F[2] * jr.tw.z));
        const float wy = fmaf(F[3], jr.tw.x, fmaf(F[4], jr.tw.y, F[5] * jr.tw.z));
        const float wz = fmaf(F[6], jr.tw.x, fmaf(F[7], jr.tw.y, F[8] * jr.tw.z));
        const float vx = fmaf(F[0], jr.tv.x, fmaf(F[1], jr.tv.y, F[2] * jr.tv.z));
        const float vy = fmaf(F[3], jr.tv.x, fmaf(F[4], jr.tv.y, F[5] * jr.tv.z));
        const float vz = fmaf(F[6], jr.tv.x, fmaf(F[7], jr.tv.y, F[8] * jr.tv.z));
        const float tx = F[9], ty = F[10], tz = F[11];
        const float mx = A[3] - (ty * A[2] - tz * A[1]);
        const float my = A[4] - (tz * A[0] - tx * A[2]);
        const float mz = A[5] - (tx * A[1] - ty * A[0]);
        dv[w * J + j] = wx * mx + wy * my + wz * mz + vx * A[0] + vy * A[1] + vz * A[2];
    }
    __syncthreads();
    // 5. joint-space gradient + length term, coalesced over (waypoint, dimension)
    const float inv_beta = 1.0f / a.beta;
    float* share = B.g;  // [nw][dim], in the place of the sphere gradients
    for (int i = tid; i < nw * dim; i += T) {
        const int w = i / dim, d = i - w * dim;
        float gq = 0.0f;
        for (int j = 0; j < J; ++j) {
            const JointRec& jr = sc.joints[j];
            if (jr.idx.z >= 0) {
                if (jr.idx.z == d) gq = fmaf(jr.tv.w, dv[w * J + j], gq);
            } else if (jr.idx.y == d) {
                gq += dv[w * J + j];
            }
        }
        const long long at = first * dim + i;
        const int in_path = (int)((first + w) % W);
        if (part == 0) {
            const float qc = a.wp[at];
            if (in_path + 1 < W) {
                const float dn = a.wp[at + dim] - qc;
                gq -= 2.0f * a.w_len * dn;
                atomicAdd(&B.cost[w], a.beta * a.w_len * dn * dn);  // in units of 1/beta, as the pair terms
            }
            if (in_path > 0) gq += 2.0f * a.w_len * (qc - a.wp[at - dim]);
        }
        if (a.grad) {
            if (parts == 1) a.grad[at] = gq;
            else if (parts == 2) atomicAdd(&a.grad[at], gq);  // zero before the launch; of two terms the order does not matter
            else share[i] = gq;
        }
    }
    if (parts > 2 && a.grad) {  // the parts are the CTAs of a cluster: their shares are added in their order
        cluster_sync();
        for (int i = part * T + tid; i < nw * dim; i += parts * T) {
            float sum = 0.0f;
            for (int k = 0; k < parts; ++k) sum += cluster_load(share + i, k);
            a.grad[first * dim + i] = sum;
        }
        cluster_sync();  // the shares are read before a CTA ends
    }
    __syncthreads();
    // 6. cost per path: one atomic per CTA when its waypoints are of one path
    if (warp == 0) {
        float v = lane < nw ? B.cost[lane] * inv_beta : 0.0f;
        const long long p0 = first / W, p1 = (first + nw - 1) / W;
        if (p0 == p1) {
#pragma unroll
            for (int off = 16; off > 0; off >>= 1) v += __shfl_xor_sync(kAll, v, off);
            if (lane == 0) atomicAdd(&a.cost[p0], v);
        } else if (lane < nw) {
            atomicAdd(&a.cost[(first + lane) / W], v);
        }
    }
}

// Launch of `parts` CTAs per cluster (up to 2: none).
static cudaLaunchConfig_t cluster_config(cudaLaunchAttribute& cluster, int threads, size_t smem, int parts) {
    cluster.id = cudaLaunchAttributeClusterDimension;
    cluster.val.clusterDim = {(unsigned)parts, 1u, 1u};
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)parts);
    cfg.blockDim = dim3(threads);
    cfg.dynamicSmemBytes = smem;
    cfg.attrs = &cluster;
    cfg.numAttrs = parts > 2 ? 1 : 0;
    return cfg;
}

// How many clusters of 3 to 8 CTAs the device holds at once, 0 if none, for a kernel
// of which `per_sm` CTAs (up to 3) fit an SM: asked once per device and CUDA context.
static int cluster_room(void (*kern)(SmoothArgs, int, int), int per_sm, int threads, size_t smem, int parts) {
    struct Room {
        unsigned long long ctx = 0ull;
        int n = 0;
    };
    static Room rooms[4][9][kDynLimitDevices];
    static std::mutex mutex;
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess) return 0;
    const unsigned long long ctx = current_context_key();
    std::lock_guard<std::mutex> lock(mutex);
    Room none;
    Room& r = dev >= 0 && dev < kDynLimitDevices ? rooms[per_sm][parts][dev] : none;
    if (!ctx || r.ctx != ctx) {
        cudaLaunchAttribute cluster;
        const cudaLaunchConfig_t cfg = cluster_config(cluster, threads, smem, parts);
        r = Room{ctx, 0};
        if (cudaOccupancyMaxActiveClusters(&r.n, kern, &cfg) != cudaSuccess) {
            cudaGetLastError();
            r.n = 0;
        }
    }
    return r.n;
}

cudaError_t launch_smooth(const unsigned char* blob, size_t blob_stride, int blob_cap, const int32_t* pairs,
                          size_t pairs_stride,
                          int J, int S, int dim, const float* wp, int P, int W, float margin, float beta, float w_len,
                          float* cost, float* grad, bool ordered, cudaStream_t st) {
    if (P <= 0 || W <= 0) return cudaSuccess;
    cudaError_t e;
    if (cost && (e = cudaMemsetAsync(cost, 0, (size_t)P * sizeof(float), st)) != cudaSuccess) return e;
    SmoothArgs a{blob, reinterpret_cast<const int2*>(pairs), blob_stride, pairs_stride, J, S, dim, wp, P, W,
                 margin, beta, w_len, cost, grad};
    const bool shared = blob_stride == 0 && pairs_stride == 0;
    if (shared && !ordered && cost && J <= 32) {
        // 256 threads and up to three CTAs per SM (registers), or 512 where
        // shared memory allows only one (large robots)
        const size_t wide = (size_t)blob_cap + smooth_wide_bytes(J, S);
        const int by_smem = (int)((device_max_smem() + 1024) / (wide + 1024 + kStaticSmem));
        const bool big = by_smem < 2;
        const long long ctas = ((long long)P * W + 31) / 32;
        if (wide + kStaticSmem <= device_max_smem() && ctas * 8 <= INT32_MAX) {
            void (*const kern)(SmoothArgs, int, int) = big ? smooth_wide_kernel<512, 1> : smooth_wide_kernel<256, 3>;
            // Several CTAs may share 32 waypoints, each with a share of the pairs,
            // and add up their gradients (which are linear in the pairs' terms):
            // as many as make the last wave of the launch full, a twelfth of a
            // CTA's time being its frames and closing sums.  Two add into zeroed
            // memory; more are a cluster, which adds in their order.
            // A cluster lies within one GPC, so fewer of them fit than the SMs would
            // hold CTAs (8 dual-arm paths of 64 waypoints: 16 clusters of 8 took two
            // waves, 171 us a call; as clusters of 7 they take one, 111).
            // How many is the same for every scene of as many CTAs per SM, so that a call's
            // gradient does not depend on the calls before it.
            const int per_sm = big ? 1 : std::min(by_smem, 3);
            const size_t most = (device_max_smem() + 1024) / per_sm - 1024 - kStaticSmem;  // what so many CTAs have each, at least `wide`
            static DynLimit limit[2][kDynLimitDevices];
            if ((e = raise_dyn_limit(reinterpret_cast<const void*>(kern), limit[big ? 1 : 0], most)) != cudaSuccess)
                return e;
            const long long room = (long long)device_sm_count() * per_sm;
            const int threads = big ? 512 : 256;
            int parts = 1;
            double best = 1e30;
            for (int p = 1; p <= 8; ++p) {
                const long long fit = p > 2 ? cluster_room(kern, per_sm, threads, most, p) : room / p;
                if (fit < 1) continue;
                const double c = (double)((ctas + fit - 1) / fit) * (1.0 / p + 1.0 / 12);
                if (c < 0.97 * best) { best = c; parts = p; }
            }
            if (parts == 2 && grad &&
                (e = cudaMemsetAsync(grad, 0, (size_t)P * W * dim * sizeof(float), st)) != cudaSuccess)
                return e;
            cudaLaunchAttribute cluster;
            cudaLaunchConfig_t cfg = cluster_config(cluster, threads, wide, parts);
            cfg.gridDim = dim3((unsigned)(ctas * parts));
            cfg.stream = st;
            if ((e = cudaLaunchKernelEx(&cfg, kern, a, blob_cap, parts)) != cudaSuccess) return e;
            return cudaGetLastError();
        }
    }
    constexpr int WARPS = 8;
    size_t smem = (size_t)WARPS * smooth_warp_floats(J, S) * sizeof(float);
    auto per_path = [&](int warps) { return shared ? 0 : (W + warps - 1) / warps; };
    auto blocks = [&](int warps) {
        return (unsigned)(shared ? ((long long)P * W + warps - 1) / warps : (long long)P * per_path(warps));
    };
    if (smem + blob_cap + kStaticSmem <= device_max_smem()) {
        smem += blob_cap;
        auto kern = cost ? smooth_kernel<WARPS, true, true> : smooth_kernel<WARPS, true, false>;
        static DynLimit limit[2][kDynLimitDevices];
        if ((e = raise_dyn_limit(reinterpret_cast<const void*>(kern), limit[cost ? 1 : 0], smem)) != cudaSuccess) return e;
        kern<<<blocks(WARPS), WARPS * 32, smem, st>>>(a, blob_cap, per_path(WARPS));
        return cudaGetLastError();
    }
    // scene or robot too large to stage: fewer waypoints per CTA, the scene in
    // global memory (four take robots of about 1,760 spheres, two twice that)
    auto few = [&](auto count) {
        constexpr int FEW = decltype(count)::value;
        const size_t bytes = (size_t)FEW * smooth_warp_floats(J, S) * sizeof(float);
        auto kern = cost ? smooth_kernel<FEW, false, true> : smooth_kernel<FEW, false, false>;
        static DynLimit limit[2][kDynLimitDevices];
        if (bytes > 48 * 1024 &&
            (e = raise_dyn_limit(reinterpret_cast<const void*>(kern), limit[cost ? 1 : 0], bytes)) != cudaSuccess)
            return e;
        kern<<<blocks(FEW), FEW * 32, bytes, st>>>(a, 0, per_path(FEW));
        return cudaGetLastError();
    };
    if ((size_t)4 * smooth_warp_floats(J, S) * sizeof(float) + 64 <= device_max_smem()) return few(std::integral_constant<int, 4>());
    return few(std::integral_constant<int, 2>());
}

}  // namespace prrtc
