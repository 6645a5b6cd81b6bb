// prrtc_cull.cuh -- the culled collision check: the verdicts of cc_chunk
// (prrtc_device.cuh), bit for bit, from a small part of its pair tests.
//
// Every link has a cull sphere (pack kernel): the centre of its coarse sphere
// and a radius that encloses its fine spheres and the coarse sphere with a pad.
// A primitive whose distance from the cull sphere is positive cannot pass any
// fine test of that link, so only the links, waypoints and primitives that
// touch are tested, with the same arithmetic as cc_chunk's.
//
// The pad covers rounding.  The expanded sphere test, |c|^2 - r^2 + |o|^2 - r_o^2 -
// 2 (c.o + r r_o), is off by at most e M^2, e = 1.1e-6, M = |c| + |o| + radii, on a fine
// sphere and on the cull sphere.  With m = |c| + R (R without the pad, c the cull
// sphere's centre; a link's fine spheres lie within m of the origin) and a gap of g
// between the unpadded sphere and the primitive, M <= 2 (m + r_o) + g, so a fine test
// can only pass for g^2 + 2 g r_o < e M^2, hence only for e M^2 < B = 4.5e-6 (m + r_o)^2.
// A pad of d = 3.2e-3 m + 4.6e-6 r_o keeps it from that: a cull sphere found apart has
// g^2 + 2 g (R + r_o) > d^2 + 2 d (R + r_o) - B, which gives g > 2.2e-3 m + 2.3e-6 r_o, and
// then g^2 + 2 g r_o > B.  So the pad grows with the robot's own coordinates and
// hardly with the primitives' (a floor of 500 m pads by 1 cm).  The other tests are
// first order in the distance and need 1e-6 (m + size of the primitive).  Comparisons
// are written so that NaN and infinities count as touching.
//
// For the waypoints of an edge a first level bounds each link's cull spheres
// over the whole pass by one sphere (centre of the middle waypoint) and lists
// the primitives that it touches; the waypoints then test that list only.
//
// Fine work is a shared-memory list of (link, waypoint, mask of primitives) and
// one of (self item, waypoint); 8 lanes take an entry, a sphere per lane, and
// place their sphere centres from the link frames as they need them (no pass
// over all spheres, no centre buffer).
#pragma once

#include "prrtc_device.cuh"

namespace prrtc {

constexpr int kCullLinkList = 256;  // primitives listed per link of an edge; more: all of them are tested

// Shared-memory buffers of a culled edge pass of CW waypoints.
struct CullBufs {
    float* pose;       // [CW][J][12]
    float4* cctr;      // [K][CW] coarse sphere centres, .w = radius + inflation (gated) or the cull radius (flat)
    float4* swept;     // [K] bound of the link's cull spheres over the pass
    uint32_t* dirty;   // [CW][2] links whose coarse sphere touches the world (gated)
    int2* wlist;       // [wcap] (group of 32 << 12 | link << 6 | waypoint, mask of primitives in the group)
    int* slist;        // [scap] self item << 6 | waypoint
    int4* ncand;       // [K] primitives listed for a link: ends of the spheres, capsules, boxes, all; .w -1: too many
    uint16_t* cand;    // [K][ccap]
    uint32_t* hit;     // [6]: result words, world and self list lengths, alternating between calls
    int wcap, scap, ccap;
    unsigned long long* stats;
};

__host__ __device__ inline int cull_link_list(int n_obs) { return n_obs < kCullLinkList ? (n_obs + 7) & ~7 : kCullLinkList; }
// List capacities: room for every second link of every waypoint; a pass that
// needs more goes over all (link, waypoint) pairs.
__host__ __device__ inline int cull_wcap(int K, int CW) { return (K * CW / 2 + 63) & ~31; }
__host__ __device__ inline int cull_scap(int CW) { return 12 * CW; }

__host__ __device__ inline int cull_smem_bytes(int J, int K, int n_obs, int CW) {
    int b = CW * J * 48 + K * CW * 16 + K * 32 + CW * 8;
    b += cull_wcap(K, CW) * 8 + cull_scap(CW) * 4 + 32;
    return b + align16(K * cull_link_list(n_obs) * 2);
}

__device__ __forceinline__ CullBufs cull_bufs(unsigned char* p, int J, int K, int n_obs, int CW) {
    CullBufs b;
    b.wcap = cull_wcap(K, CW);
    b.scap = cull_scap(CW);
    b.ccap = cull_link_list(n_obs);
    b.hit = reinterpret_cast<uint32_t*>(p);    p += 32;
    b.pose = reinterpret_cast<float*>(p);      p += CW * J * 48;
    b.cctr = reinterpret_cast<float4*>(p);     p += K * CW * 16;
    b.swept = reinterpret_cast<float4*>(p);    p += K * 16;
    b.ncand = reinterpret_cast<int4*>(p);      p += K * 16;
    b.dirty = reinterpret_cast<uint32_t*>(p);  p += CW * 8;
    b.wlist = reinterpret_cast<int2*>(p);      p += b.wcap * 8;
    b.slist = reinterpret_cast<int*>(p);       p += b.scap * 4;
    b.cand = reinterpret_cast<uint16_t*>(p);
    b.stats = nullptr;
    return b;
}

// Whether a launch can use the culled check at all (the scene's own flag,
// BlobHeader::cull, decides per problem).
inline bool cull_shape_ok(int J, int K, int n_obs, float inflate) {
    return J >= 1 && J <= 32 && K >= 1 && K <= kMaxLinks && n_obs < 65536 && inflate >= 0.0f;
}

// True when a sphere at distance sqrt(d2) with radius sum b certainly does not
// touch (false for NaN, and for a distance so large that it may be an overflow).
__device__ __forceinline__ bool cull_far(float d2, float b) { return d2 > b * b && d2 < 1e30f; }

// A cull sphere: centre and padded radius, and -(|c|^2 - R^2), the sphere
// test's threshold.
struct CullBall {
    float4 c;
    float thr;
};

__device__ __forceinline__ CullBall cull_ball(float4 c, float R) {
    const float4 b = make_float4(c.x, c.y, c.z, R);
    return CullBall{b, -sphere_A(b)};
}

// Whether one primitive of each type may touch the ball: the fine tests' own
// forms on the cull sphere (four FMAs and a comparison for a sphere; the sign of
// a radius is dropped, since the fine test squares the sum).
__device__ __forceinline__ bool cull_sphere(const Scene& sc, int o, const CullBall& b) {
    const float4 O = sc.ws[2 * o];
    const float h = fmaf(b.c.x, O.x, fmaf(b.c.y, O.y, fmaf(b.c.z, O.z, fmaf(b.c.w, -fabsf(O.w), sc.ws[2 * o + 1].w))));
    return !(h > b.thr);
}
__device__ __forceinline__ bool cull_capsule(const Scene& sc, int o, const CullBall& b) {
    const float4 p1 = sc.wc[3 * o], dp = sc.wc[3 * o + 1], d = sc.wc[3 * o + 2];
    const float4 c = b.c;
    const float t = __saturatef(fmaf(dp.x, c.x, fmaf(dp.y, c.y, fmaf(dp.z, c.z, dp.w))));
    const float ex = fmaf(-t, d.x, c.x - p1.x), ey = fmaf(-t, d.y, c.y - p1.y), ez = fmaf(-t, d.z, c.z - p1.z);
    return !cull_far(fmaf(ex, ex, fmaf(ey, ey, ez * ez)), c.w + fabsf(p1.w));
}
__device__ __forceinline__ bool cull_box(const Scene& sc, int o, const CullBall& b) {
    const float4 cc[1] = {b.c};
    const float4 hl = sc.wb[4 * o + 3];
    float v[1];
    h_box<1>(v, cc, sc.wb[4 * o], sc.wb[4 * o + 1], sc.wb[4 * o + 2], hl);
    const float r = b.c.w * hl.w * kBoxInv;  // hl.w: the axes' stretch, at least 1
    return !(v[0] > r * r);
}
__device__ __forceinline__ bool cull_halfspace(const Scene& sc, int o, const CullBall& b) {
    const float4 cc[1] = {b.c};
    const float4 n = sc.wh[o];
    float v[1];
    h_halfspace<1>(v, cc, n);
    const float n2 = fmaxf(1.0f, fmaf(n.x, n.x, fmaf(n.y, n.y, n.z * n.z)));  // the normal's length may exceed 1
    return !(v[0] > 0.0f && v[0] * v[0] > b.c.w * b.c.w * (1.000001f * n2));
}

// The exact test of primitive o (combined index) against one sphere: the
// arithmetic of obstacles_vs_spheres.
__device__ __forceinline__ bool prim_hits(const Scene& sc, const BlobHeader& h, int o, float4 c) {
    const float4 cc[1] = {c};
    float v[1];
    if (o < h.Ns) {
        h_sphere<1>(v, cc, sc.ws[2 * o], sc.ws[2 * o + 1].w);
        return v[0] <= -sphere_A(c);
    }
    o -= h.Ns;
    if (o < h.Nc) {
        h_capsule<1>(v, cc, sc.wc[3 * o], sc.wc[3 * o + 1], sc.wc[3 * o + 2]);
        return v[0] <= 0.0f;
    }
    o -= h.Nc;
    if (o < h.Nb) {
        h_box<1>(v, cc, sc.wb[4 * o], sc.wb[4 * o + 1], sc.wb[4 * o + 2], sc.wb[4 * o + 3]);
        return v[0] <= (c.w * kBoxInv) * (c.w * kBoxInv);
    }
    h_halfspace<1>(v, cc, sc.wh[o - h.Nb]);
    return v[0] <= c.w;
}

__device__ __forceinline__ int prim_flops(const BlobHeader& h, int o) {
    return o < h.Ns ? kFlopSphere : (o < h.Ns + h.Nc ? kFlopCapsule : (o < h.Ns + h.Nc + h.Nb ? kFlopBox : kFlopHalfspace));
}

// One point in the frame of joint f at waypoint w (three 16-byte loads).
__device__ __forceinline__ float4 pose_point(const float* pose, int J, int w, int f, float4 l) {
    const float4* p = reinterpret_cast<const float4*>(pose + (w * J + f) * 12);
    const float4 p0 = p[0], p1 = p[1], p2 = p[2];
    const float F[12] = {p0.x, p0.y, p0.z, p0.w, p1.x, p1.y, p1.z, p1.w, p2.x, p2.y, p2.z, p2.w};
    return xform_point(F, l);
}

// Centre of fine sphere s at waypoint w (the arithmetic of cc_centres).
__device__ __forceinline__ float4 fine_centre(const Scene& sc, const float* pose, int J, int w, int s, float inflate) {
    const int f = sc.sfr[s];
    if (f < 0) return absent_sphere();
    float4 l = sc.sph[s];
    l.w += inflate;
    return pose_point(pose, J, w, f, l);
}

// Padded cull radius of a link whose coarse centre is c (grp record .w: the padded
// reach of its spheres and the scene's share of the pad).
__device__ __forceinline__ float cull_radius(float reach, float inflate, float4 c) {
    return reach + (1.0f + kCullPad) * inflate + kCullPad * (fabsf(c.x) + fabsf(c.y) + fabsf(c.z));
}

// Coarse centre of link k at waypoint w with the radius that its checker works
// with: the coarse sphere's own for a gated one, else the cull radius.
__device__ __forceinline__ float4 link_centre(const Scene& sc, const float* pose, int J, int w, int k, float inflate,
                                              bool gated) {
    float4 l = sc.grp[2 * k];
    const float4 g = sc.grp[2 * k + 1];
    l.w += inflate;
    float4 c = pose_point(pose, J, w, __float_as_int(g.x), l);
    if (!gated) c.w = cull_radius(g.w, inflate, c);
    return c;
}

// The cull radius that belongs to a stored link centre.
__device__ __forceinline__ float link_radius(const Scene& sc, int k, float inflate, bool gated, float4 c) {
    return gated ? cull_radius(sc.grp[2 * k + 1].w, inflate, c) : c.w;
}

// Whether self item ii needs its fine test at waypoint w: the gate of a gated
// checker (as cc_chunk), or whether the cull spheres of its block's links touch.
// Items of no coarse pair always do.
__device__ __forceinline__ bool cull_self_touch(const Scene& sc, const CullBufs& B, int CW, int4 item, int w, float inflate) {
    const int q = item.w >= 0 ? item.w : -2 - item.w;
    if (q < 0) return true;
    const int2 cp = sc.cpair[q];
    if (cp.x < 0 || cp.y < 0 || cp.x >= sc.h->K || cp.y >= sc.h->K) return false;
    const float4 a = B.cctr[cp.x * CW + w], b = B.cctr[cp.y * CW + w];
    const float dx = a.x - b.x, dy = a.y - b.y, dz = a.z - b.z;
    const float d2 = fmaf(dx, dx, fmaf(dy, dy, dz * dz));
    if (item.w >= 0) {
        const float t = a.w + b.w - inflate;
        return d2 <= t * t;
    }
    return !cull_far(d2, a.w + b.w);  // a flat checker's block: .w is the cull radius
}

// Fine test of self item ii at waypoint w by 8 consecutive lanes (l8 = 0..7 of
// `mask`) together: a sphere of the first group per lane.
__device__ __forceinline__ bool cull_self_item(const Scene& sc, const CullBufs& B, int CW, int ii, int w, int l8,
                                               unsigned mask, float inflate, unsigned& flops) {
    const BlobHeader& h = *sc.h;
    const int J = h.J, S = h.S;
    const int4 item = sc.item[ii];
    bool hit = false;
    if (item.y >= 0) {  // block: spheres [a0, a0+na) x [b0, b0+nb)
        const int na = item.z >> 16, nb = item.z & 0xffff;
        const float half = 0.5f * inflate;
        float4 a[1] = {l8 < na ? fine_centre(sc, B.pose, J, w, item.x + l8, inflate) : absent_sphere()};
        a[0].w -= half;
        const float thr = -sphere_A(a[0]);
        for (int b0 = 0; b0 < nb; b0 += 8) {
            float4 b = b0 + l8 < nb ? fine_centre(sc, B.pose, J, w, item.y + b0 + l8, inflate) : absent_sphere();
            b.w -= half;
            const float4 O = make_float4(-2.0f * b.x, -2.0f * b.y, -2.0f * b.z, -2.0f * b.w);
            const float A = sphere_A(b);
#pragma unroll
            for (int m = 0; m < 8; ++m) {
                const float4 Om = make_float4(__shfl_sync(mask, O.x, m, 8), __shfl_sync(mask, O.y, m, 8),
                                              __shfl_sync(mask, O.z, m, 8), __shfl_sync(mask, O.w, m, 8));
                float v[1];
                h_sphere<1>(v, a, Om, __shfl_sync(mask, A, m, 8));
                hit |= v[0] <= thr;
            }
        }
        flops += l8 < na ? nb * kFlopPair + 2 * kFlopXform : 0;
    } else {  // explicit pairs [p0, p0+count) of the pair list (global memory)
        const int p1 = min(item.x + item.z, h.P);
        for (int p = item.x + l8; p < p1; p += 8) {
            const int2 pr = __ldg(&sc.pairs[p]);
            if (pr.x < 0 || pr.y < 0 || pr.x >= S || pr.y >= S) continue;
            const float4 a = fine_centre(sc, B.pose, J, w, pr.x, inflate), b = fine_centre(sc, B.pose, J, w, pr.y, inflate);
            const float dx = a.x - b.x, dy = a.y - b.y, dz = a.z - b.z;
            const float t = a.w + b.w - inflate;
            hit |= fmaf(dx, dx, fmaf(dy, dy, dz * dz)) <= t * t;
            flops += kFlopPairExplicit + 2 * kFlopXform;
        }
    }
    return hit;
}

// Fine test of link k at waypoint w in a pass whose world list ran over, by 8
// consecutive lanes (l8 = 0..7 of `mask`): they find the touching primitives again,
// four of 32 each, and test them with a sphere per lane.  c: the link's centre;
// list: its `listed` primitives, or every one for listed < 0.  Out of line: the code
// is rarely needed.  It takes values, not the buffers: with their address taken
// every access to them is through local memory, 8% of a plan (explore_kernel of 16
// spheres, 128 explorers: 82 -> 89 us).
static __device__ __noinline__ bool cull_link_again(const unsigned char* blob, const float* pose, int k, int w, int l8,
                                                    unsigned mask, const uint16_t* list, int listed, float4 c) {
    const Scene sc = scene_view(blob);
    const BlobHeader& h = *sc.h;
    const float inflate = __int_as_float(h.inflate_bits);
    const int e0 = h.Ns, e1 = e0 + h.Nc, e2 = e1 + h.Nb, n = listed >= 0 ? listed : e2 + h.Nh;
    if (listed < 0) list = nullptr;
    const float4 gr = sc.grp[2 * k + 1];
    const CullBall ball = cull_ball(c, link_radius(sc, k, inflate, h.gated != 0, c));
    const int s1 = __float_as_int(gr.z);
    bool hit = false;
    for (int i0 = 0; i0 < n; i0 += 32) {
        unsigned bits = 0u;
        for (int i = i0 + l8; i < min(n, i0 + 32); i += 8) {
            const int o = list ? (int)list[i] : i;
            const bool t = o < e0 ? cull_sphere(sc, o, ball)
                           : o < e1 ? cull_capsule(sc, o - e0, ball)
                           : o < e2 ? cull_box(sc, o - e1, ball) : cull_halfspace(sc, o - e2, ball);
            bits |= (unsigned)t << (i - i0);
        }
        bits = __reduce_or_sync(mask, bits);
        for (int s = __float_as_int(gr.y) + l8; s < s1 && bits; s += 8) {
            const float4 f = fine_centre(sc, pose, h.J, w, s, inflate);
#pragma unroll 1
            for (unsigned rest = bits; rest; rest &= rest - 1u) {
                const int i = i0 + __ffs(rest) - 1;
                hit |= prim_hits(sc, h, list ? (int)list[i] : i, f);
            }
        }
    }
    return hit;
}

// Up to 32 spheres against the point cloud, one per lane (the whole warp calls
// it): lane's sphere c (radius + inflation in .w) belongs to configuration w,
// and `alive` (the same in every lane) says which configurations still matter.
// Returns the configurations hit, as a mask, the same in every lane.  The
// verdicts are pc_sphere_hits': every cell of a sphere's bounding box, a box of
// more than kPcMaxCells cells is a hit.
//
// A sphere spans 8 to 27 cells, most of them empty, and an occupied one holds
// some 20 points.  A lane that walked its own sphere's cells and points made the
// warp wait for its longest chain of dependent loads, so the cells of all 32
// spheres are dealt out over the lanes, and the points of an occupied cell over
// 8 of them: 128 edges of 16 waypoints against 20,000 points take 80 us a call
// instead of 464, 4000 edges of 33 against 500 points 567 us instead of 684.
__device__ __forceinline__ unsigned cloud_batch(const PcView& pc, float4 c, bool valid, int w, unsigned alive,
                                                unsigned& flops) {
    constexpr unsigned kAll = 0xffffffffu;
    const int lane = threadIdx.x & 31, l8 = lane & 7, sub = lane >> 3;
    const float R = c.w + pc.r_env;
    valid = valid && (alive >> w & 1u) && fabsf(c.x) < kPcExtent && fabsf(c.y) < kPcExtent && fabsf(c.z) < kPcExtent && R >= 0.0f;
    bool hit = valid && !(R < 1.0e3f);
    int x0 = 0, y0 = 0, z0 = 0, nx = 0, ny = 0, n = 0;
    if (valid && !hit) {
        x0 = (int)floorf((c.x - R) * pc.inv_cell);
        y0 = (int)floorf((c.y - R) * pc.inv_cell);
        z0 = (int)floorf((c.z - R) * pc.inv_cell);
        const int x1 = (int)floorf((c.x + R) * pc.inv_cell), y1 = (int)floorf((c.y + R) * pc.inv_cell);
        const int z1 = (int)floorf((c.z + R) * pc.inv_cell);
        const long long cells = ((long long)x1 - x0 + 1) * ((long long)y1 - y0 + 1) * ((long long)z1 - z0 + 1);
        hit = cells > kPcMaxCells;
        if (!hit) {
            nx = x1 - x0 + 1;
            ny = y1 - y0 + 1;
            n = (int)cells;
        }
    }
    unsigned hits = __reduce_or_sync(kAll, hit ? 1u << w : 0u);
    alive &= ~hits;
    if (!(alive >> w & 1u)) n = 0;
    int incl = n;  // cells of lanes 0..lane
#pragma unroll
    for (int off = 1; off < 32; off <<= 1) {
        const int v = __shfl_up_sync(kAll, incl, off);
        if (lane >= off) incl += v;
    }
    const int total = __shfl_sync(kAll, incl, 31);
    const float R2 = R * R;
    for (int base = 0; base < total && alive; base += 32) {
        const int idx = base + lane;
        int own = 0;  // the first lane whose count passes idx
#pragma unroll
        for (int step = 16; step > 0; step >>= 1) own += __shfl_sync(kAll, incl, own + step - 1) <= idx ? step : 0;
        own = min(own, 31);
        const int r = idx - __shfl_sync(kAll, incl, own) + __shfl_sync(kAll, n, own);
        const int onx = max(1, __shfl_sync(kAll, nx, own)), ony = max(1, __shfl_sync(kAll, ny, own));
        const int ow = __shfl_sync(kAll, w, own);
        const int ryz = r / onx, rx = r - ryz * onx, rz = ryz / ony, ry = ryz - rz * ony;
        const unsigned b = pc_hash(__shfl_sync(kAll, x0, own) + rx, __shfl_sync(kAll, y0, own) + ry,
                                   __shfl_sync(kAll, z0, own) + rz, pc.mask);
        int p0 = 0, p1 = 0;
        if (idx < total && (alive >> ow & 1u)) {
            p0 = __ldg(&pc.start[b]);
            p1 = __ldg(&pc.start[b + 1]);
        }
        for (unsigned todo = __ballot_sync(kAll, p1 > p0); todo;) {
            unsigned t = todo;  // the next four occupied cells, one per group of 8 lanes
            int src = -1;
#pragma unroll
            for (int g = 0; g < 4; ++g) {
                if (g == sub && t) src = __ffs(t) - 1;
                t &= t - 1u;
            }
            todo = t;
            const int from = max(src, 0);
            const int e = __shfl_sync(kAll, own, from), ew = __shfl_sync(kAll, ow, from);
            const int e0 = __shfl_sync(kAll, p0, from), e1 = __shfl_sync(kAll, p1, from);
            const float cx = __shfl_sync(kAll, c.x, e), cy = __shfl_sync(kAll, c.y, e), cz = __shfl_sync(kAll, c.z, e);
            const float cr = __shfl_sync(kAll, R2, e);
            hit = false;
            if (src >= 0 && (alive >> ew & 1u)) {
#pragma unroll 2
                for (int p = e0 + l8; p < e1; p += 8) {
                    const float4 q = __ldg(&pc.pts[p]);
                    const float dx = cx - q.x, dy = cy - q.y, dz = cz - q.z;
                    hit |= fmaf(dx, dx, fmaf(dy, dy, dz * dz)) <= cr;
                    flops += kFlopPoint;
                }
            }
            const unsigned h = __reduce_or_sync(kAll, hit ? 1u << ew : 0u);
            hits |= h;
            alive &= ~h;
        }
    }
    return hits;
}

// One type's primitives of a link's bound (a warp, a primitive per lane):
// appends those that touch to the link's list and returns its new length.
template <class Touch>
__device__ __forceinline__ int cull_append(int count, int base, int n, int cap, uint16_t* list, int lane, Touch touch) {
#pragma unroll 1
    for (int o0 = 0; o0 < count; o0 += 32) {
        const int o = o0 + lane;
        const bool t = o < count && touch(o);
        const unsigned b = __ballot_sync(0xffffffffu, t);
        const int at = n + __popc(b & ((1u << lane) - 1u));
        if (t && at < cap) list[at] = (uint16_t)(base + o);
        n += __popc(b);
    }
    return n;
}

// Whether any of nw (<= CW <= 64) waypoints of `edge` collides (non-zero).
// Called by every thread of the CTA with the same `par`, which the call flips: the
// result words and list lengths alternate between calls, so that a call clears the
// next call's after its first barrier.  All must be zero and `par` 0 before the
// first call.  The scene must have BlobHeader::cull set.
template <class G>
__device__ __forceinline__ uint32_t cull_check(const G& g, const Scene& sc, const CullBufs& B, int nw, int CW, int& par,
                                               const EdgeSrc& edge) {
    const BlobHeader& h = *sc.h;
    const int tid = g.rank(), T = g.size(), lane = tid & 31, warp = tid >> 5, n_warps = T >> 5;
    const int J = h.J, S = h.S, K = h.K;
    const int Ns = h.Ns, Nc = h.Nc, Nb = h.Nb, Nh = h.Nh;
    const bool gated = h.gated != 0;
    const float inflate = __int_as_float(h.inflate_bits);
    uint32_t* hw = B.hit + par;
    volatile uint32_t* vhit = hw;
    int* nwl = reinterpret_cast<int*>(B.hit + 2 + par);
    int* nsl = reinterpret_cast<int*>(B.hit + 4 + par);
    par ^= 1;
    unsigned flops = 0;

    // 1. link frames (as cc_chunk) and coarse centres
    if (gated)
        for (int i = tid; i < 2 * nw; i += T) B.dirty[i] = 0u;
    fk_segments(sc, nullptr, B.pose, &edge, nw, J, tid, T, [&](int w, int j, int SEG) {
        for (int k = j; k < K; k += SEG) {
            B.cctr[k * CW + w] = link_centre(sc, B.pose, J, w, k, inflate, gated);
        }
    });
    g.sync();
    if (tid == 0) {  // the next call's words (every thread has read them by now)
        B.hit[par] = 0u;
        B.hit[2 + par] = B.hit[4 + par] = 0u;
    }
    // 2. one bound per link over the pass, and the primitives it touches (a warp per link)
    for (int k = warp; k < K; k += n_warps) {
        const float4 m = B.cctr[k * CW + (nw >> 1)];
        unsigned far2 = 0u;  // bits of the largest squared distance (NaN orders above infinity)
        for (int w = lane; w < nw; w += 32) {
            const float4 c = B.cctr[k * CW + w];
            const float dx = c.x - m.x, dy = c.y - m.y, dz = c.z - m.z;
            far2 = max(far2, __float_as_uint(fmaf(dx, dx, fmaf(dy, dy, dz * dz))) & 0x7fffffffu);
        }
        const float d = __fsqrt_ru(__uint_as_float(__reduce_max_sync(0xffffffffu, far2)));
        const float R = cull_radius(sc.grp[2 * k + 1].w, inflate, m) + (1.0f + 2.0f * kCullPad) * d;
        uint16_t* list = B.cand + k * B.ccap;
        const CullBall ball = cull_ball(m, R);
        int4 n;
        n.x = cull_append(Ns, 0, 0, B.ccap, list, lane, [&](int o) { return cull_sphere(sc, o, ball); });
        n.y = cull_append(Nc, Ns, n.x, B.ccap, list, lane, [&](int o) { return cull_capsule(sc, o, ball); });
        n.z = cull_append(Nb, Ns + Nc, n.y, B.ccap, list, lane, [&](int o) { return cull_box(sc, o, ball); });
        n.w = cull_append(Nh, Ns + Nc + Nb, n.z, B.ccap, list, lane, [&](int o) { return cull_halfspace(sc, o, ball); });
        if (lane == 0) {
            B.swept[k] = make_float4(m.x, m.y, m.z, R);
            B.ncand[k] = n.w <= B.ccap ? n : make_int4(0, 0, 0, -1);
            if (B.stats) flops += Ns * kFlopSphere + Nc * kFlopCapsule + Nb * kFlopBox + Nh * kFlopHalfspace;
        }
    }
    g.sync();
    // 3. touching (link, waypoint) primitives and self items: a warp per link or item, a waypoint per lane
    const int wide = (nw + 31) >> 5;
    for (int u = warp; u < K * wide + h.n_items; u += n_warps) {
        if (u < K * wide) {
            const int k = wide == 1 ? u : u >> 1, w = (wide == 1 ? 0 : (u & 1) << 5) + lane;
            int4 n = make_int4(Ns, Ns + Nc, Ns + Nc + Nb, Ns + Nc + Nb + Nh);
            const uint16_t* list = nullptr;  // the link's list, or every primitive
            const int4 m = B.ncand[k];
            if (m.w >= 0) {
                n = m;
                list = B.cand + k * B.ccap;
            }
            auto at_index = [&](int i) { return list ? (int)list[i] : i; };
            if (w >= nw) continue;
            const float4 c = B.cctr[k * CW + w];
            const CullBall ball = cull_ball(c, link_radius(sc, k, inflate, gated, c));
            bool dirty = false;
            for (int i0 = 0; i0 < n.w; i0 += 32) {
                const int i1 = min(n.w, i0 + 32);
                unsigned bits = 0u;
                int i = i0;
#pragma unroll 1
                for (; i < min(n.x, i1); ++i) bits |= (unsigned)cull_sphere(sc, at_index(i), ball) << (i - i0);
#pragma unroll 1
                for (; i < min(n.y, i1); ++i) bits |= (unsigned)cull_capsule(sc, at_index(i) - Ns, ball) << (i - i0);
#pragma unroll 1
                for (; i < min(n.z, i1); ++i) bits |= (unsigned)cull_box(sc, at_index(i) - Ns - Nc, ball) << (i - i0);
#pragma unroll 1
                for (; i < i1; ++i) bits |= (unsigned)cull_halfspace(sc, at_index(i) - Ns - Nc - Nb, ball) << (i - i0);
                if (!bits) continue;
                if (gated)
                    for (unsigned rest = bits; rest && !dirty; rest &= rest - 1u)
                        dirty = prim_hits(sc, h, at_index(i0 + __ffs(rest) - 1), c);
                const int at = atomicAdd(nwl, 1);
                if (at < B.wcap) B.wlist[at] = make_int2((i0 >> 5) << 12 | k << 6 | w, (int)bits);
            }
            if (dirty) atomicOr(&B.dirty[2 * w + (k >> 5)], 1u << (k & 31));
            if (B.stats)
                flops += n.x * kFlopSphere + (n.y - n.x) * kFlopCapsule + (n.z - n.y) * kFlopBox + (n.w - n.z) * kFlopHalfspace;
        } else {
            const int ii = u - K * wide;
            const int4 item = sc.item[ii];
            const int q = item.w >= 0 ? item.w : -2 - item.w;
            if (q >= 0) {  // links whose bounds are apart: no waypoint touches
                const int2 cp = sc.cpair[q];
                if (cp.x < 0 || cp.y < 0 || cp.x >= K || cp.y >= K) continue;
                const float4 a = B.swept[cp.x], b = B.swept[cp.y];
                const float dx = a.x - b.x, dy = a.y - b.y, dz = a.z - b.z;
                if (cull_far(fmaf(dx, dx, fmaf(dy, dy, dz * dz)), a.w + b.w)) continue;
            }
            for (int w = lane; w < nw; w += 32) {
                flops += kFlopPairExplicit;
                if (!cull_self_touch(sc, B, CW, item, w, inflate)) continue;
                const int at = atomicAdd(nsl, 1);
                if (at < B.scap) B.slist[at] = ii << 6 | w;
            }
        }
    }
    g.sync();
    // 4. fine tests, 8 lanes per entry.  A list that ran over is not used: every
    // (link, waypoint), or every (item, waypoint), is an entry then.  Nothing here
    // may depend on *vhit without a vote of the 8 lanes: it changes under other
    // warps, and lanes that disagreed would wait for one another.
    const bool wfull = *nwl > B.wcap, sfull = *nsl > B.scap;
    const int Lw = wfull ? K * nw : *nwl, Ls = sfull ? h.n_items * nw : *nsl;
    const bool cloud = sc.pc.n > 0;
    if (Lw + Ls > 0 || cloud) {
        const int l8 = tid & 7;
        const unsigned mask = 0xffu << (lane & 24);
        for (int it = tid >> 3; it < Lw + Ls; it += T >> 3) {
            bool hit = false;
            int w;
            const uint32_t seen = __shfl_sync(mask, (uint32_t)*vhit, 0, 8);
            if (it < Lw) {
                int2 e = make_int2(0, 0);
                int k;
                if (wfull) {
                    k = it / nw;
                    w = it - k * nw;
                } else {
                    e = B.wlist[it];
                    k = (e.x >> 6) & 63;
                    w = e.x & 63;
                }
                if (seen) continue;
                if (gated && !(B.dirty[2 * w + (k >> 5)] & (1u << (k & 31)))) continue;
                if (wfull) {
                    if (cull_link_again(reinterpret_cast<const unsigned char*>(sc.h), B.pose, k, w, l8, mask, B.cand + k * B.ccap,
                                        B.ncand[k].w, B.cctr[k * CW + w]))
                        atomicOr(hw, 1u);
                    continue;
                }
                const float4 gr = sc.grp[2 * k + 1];
                const int i0 = (e.x >> 12) << 5;
                const uint16_t* list = B.ncand[k].w >= 0 ? B.cand + k * B.ccap + i0 : nullptr;
                const int s1 = __float_as_int(gr.z);
#pragma unroll 1
                for (int s = __float_as_int(gr.y) + l8; s < s1; s += 8) {
                    const float4 c = fine_centre(sc, B.pose, J, w, s, inflate);
#pragma unroll 1
                    for (unsigned rest = (unsigned)e.y; rest; rest &= rest - 1u) {
                        const int i = __ffs(rest) - 1;
                        const int o = list ? (int)list[i] : i0 + i;
                        hit |= prim_hits(sc, h, o, c);
                        if (B.stats) flops += prim_flops(h, o);
                    }
                    flops += kFlopXform;
                }
            } else {
                int ii;
                if (sfull) {
                    ii = (it - Lw) / nw;
                    w = (it - Lw) - ii * nw;
                } else {
                    const int e = B.slist[it - Lw];
                    ii = e >> 6;
                    w = e & 63;
                }
                if (seen) continue;
                if (sfull && !cull_self_touch(sc, B, CW, sc.item[ii], w, inflate)) continue;
                hit = cull_self_item(sc, B, CW, ii, w, l8, mask, inflate, flops);
            }
            if (hit) atomicOr(hw, 1u);
        }
        if (cloud) {
            // every sphere of every waypoint, a batch of 32 per warp (the hit
            // word is read by one lane for all)
            for (int it0 = warp << 5; it0 < S * nw; it0 += n_warps << 5) {
                const uint32_t seen = __shfl_sync(0xffffffffu, (uint32_t)*vhit, 0);
                if (seen) break;
                const int it = it0 + lane, s = min(it, S * nw - 1) / nw, w = min(it, S * nw - 1) - s * nw;
                const float4 c = fine_centre(sc, B.pose, J, w, s, inflate);
                if (cloud_batch(sc.pc, c, it < S * nw, 0, 1u, flops) && lane == 0) atomicOr(hw, 1u);
            }
        }
    }
    if (B.stats) {
        if (tid == 0) {
            flops += (unsigned)(nw * (J * (kFlopJointLocal + kFlopJointChain) + K * kFlopXform));
            atomicAdd(&B.stats[kStatConfigs], (unsigned long long)nw);
        }
        if (flops) atomicAdd(&B.stats[kStatFlops], (unsigned long long)flops);
    }
    if (Lw + Ls == 0 && !cloud) return *vhit;  // no entry, so no write of the word: no barrier
    g.sync();
    return *vhit;
}

// ----------------------------------------------------------------------------- configurations

// Culled check of up to 32 unrelated configurations by one warp, no CTA barrier:
// link frames, self items, then the links from the tip to the base, a
// (configuration, link) per lane.  Each lane marks the primitives that its link's cull sphere touches,
// and the warp tests the marked links right away, 8 lanes per link.  A
// configuration leaves at its first hit, and the links still to do are dealt
// out over the configurations that are left, so the lanes stay full while most
// configurations of a cluttered scene end after two or three links.
struct WarpBufs {
    float* q;        // [CW][kDimMax]; masks of touched primitives after the frames are done
    float* pose;     // [CW][J][12]
    float4* cctr;    // [K][CW] as CullBufs
    int* list;       // [32] configurations left
};

__host__ __device__ inline int warp_check_bytes(int J, int K, int CW) {
    return (CW * kDimMax * 4 > 1024 ? CW * kDimMax * 4 : 1024) + CW * J * 48 + K * CW * 16 + 128;
}

__device__ __forceinline__ WarpBufs warp_bufs(unsigned char* p, int J, int K, int CW) {
    WarpBufs b;
    b.list = reinterpret_cast<int*>(p);     p += 128;
    b.pose = reinterpret_cast<float*>(p);   p += CW * J * 48;
    b.cctr = reinterpret_cast<float4*>(p);  p += K * CW * 16;
    b.q = reinterpret_cast<float*>(p);
    return b;
}

// Primitives [i0, i0 + 32) that may touch the ball, as a mask.
__device__ __forceinline__ unsigned cull_mask(const Scene& sc, int Ns, int Nc, int Nb, int Nh, int i0, const CullBall& b) {
    const int e0 = Ns, e1 = Ns + Nc, e2 = e1 + Nb, e3 = e2 + Nh, i1 = min(e3, i0 + 32);
    unsigned bits = 0u;
    int i = i0;
#pragma unroll 4
    for (; i < min(e0, i1); ++i) bits |= (unsigned)cull_sphere(sc, i, b) << (i - i0);
#pragma unroll 1
    for (; i < min(e1, i1); ++i) bits |= (unsigned)cull_capsule(sc, i - e0, b) << (i - i0);
#pragma unroll 2
    for (; i < min(e2, i1); ++i) bits |= (unsigned)cull_box(sc, i - e1, b) << (i - i0);
#pragma unroll 1
    for (; i < i1; ++i) bits |= (unsigned)cull_halfspace(sc, i - e2, b) << (i - i0);
    return bits;
}

// nw configurations (B.q); returns the mask of those in collision.  The scene
// must have BlobHeader::cull set.
__device__ __forceinline__ unsigned warp_check(const Scene& sc, const WarpBufs& B, int nw, int CW) {
    constexpr unsigned kAll = 0xffffffffu;
    const BlobHeader& h = *sc.h;
    const int lane = threadIdx.x & 31, l8 = lane & 7, sub = lane >> 3;
    const unsigned mask = 0xffu << (lane & 24);
    const int J = h.J, S = h.S, K = h.K;
    const int Ns = h.Ns, Nc = h.Nc, Nb = h.Nb, Nh = h.Nh, n_obs = Ns + Nc + Nb + Nh;
    const bool gated = h.gated != 0;
    const float inflate = __int_as_float(h.inflate_bits);
    fk_segments(sc, B.q, B.pose, nullptr, nw, J, lane, 32, [&](int w, int j, int SEG) {
        for (int k = j; k < K; k += SEG) {
            B.cctr[k * CW + w] = link_centre(sc, B.pose, J, w, k, inflate, gated);
        }
    });
    __syncwarp();
    unsigned alive = nw >= 32 ? kAll : (1u << nw) - 1u;  // the same in every lane
    // self items, an (item, configuration) per lane
    if (h.n_items > 0) {
        const int n = nw;
        CullBufs cb;
        cb.pose = B.pose;
        cb.cctr = B.cctr;
        unsigned flops = 0;
        for (int it0 = 0; it0 < n * h.n_items; it0 += 32) {
            const int it = it0 + lane, ii = it / n;
            bool touch = false;
            int w = 0;
            if (it < n * h.n_items) {
                w = it - ii * n;
                touch = (alive >> w & 1u) && cull_self_touch(sc, cb, CW, sc.item[ii], w, inflate);
            }
            for (unsigned todo = __ballot_sync(kAll, touch); todo;) {
                unsigned t = todo;
                int src = -1;
#pragma unroll
                for (int g = 0; g < 4; ++g) {
                    if (g == sub && t) src = __ffs(t) - 1;
                    t &= t - 1u;
                }
                todo = t;
                const int from = max(src, 0);
                const int ew = __shfl_sync(kAll, w, from), ei = __shfl_sync(kAll, ii, from);
                bool hit = false;
                if (src >= 0 && (alive >> ew & 1u)) hit = cull_self_item(sc, cb, CW, ei, ew, l8, mask, inflate, flops);
                alive &= ~__reduce_or_sync(kAll, hit ? 1u << ew : 0u);
            }
        }
    }
    uint32_t* marks = reinterpret_cast<uint32_t*>(B.q);  // [8][32] masks of a gated round
    int k1 = K;  // links [0, k1) are left
    while (k1 > 0 && alive) {
        const int n = __popc(alive), per = min(k1, 32 / n);  // `per` links of n configurations at once
        if (alive >> lane & 1u) B.list[__popc(alive & ((1u << lane) - 1u))] = lane;
        __syncwarp();
        const int kk = lane / n;
        const bool act = kk < per;
        const int k = act ? k1 - 1 - kk : 0, w = act ? B.list[lane - kk * n] : 0;
        k1 -= per;
        __syncwarp();
        const float4 c = B.cctr[k * CW + w];
        const CullBall ball = cull_ball(c, link_radius(sc, k, inflate, gated, c));
        // Tests the links marked in `bits` (primitives i0 + bit) of the lanes.
        auto fine = [&](unsigned bits, int i0) {
            for (unsigned todo = __ballot_sync(kAll, bits != 0u && (alive >> w & 1u)); todo;) {
                // the next four marked lanes, one per group of 8
                unsigned t = todo;
                int src = -1;
#pragma unroll
                for (int g = 0; g < 4; ++g) {
                    if (g == sub && t) src = __ffs(t) - 1;
                    t &= t - 1u;
                }
                todo = t;
                const int from = max(src, 0);
                const int ew = __shfl_sync(kAll, w, from), ek = __shfl_sync(kAll, k, from);
                unsigned rest = __shfl_sync(kAll, bits, from);
                bool hit = false;
                if (src >= 0 && (alive >> ew & 1u)) {
                    const float4 gr = sc.grp[2 * ek + 1];
                    const int s1 = __float_as_int(gr.z);
                    for (int s0 = __float_as_int(gr.y); s0 < s1; s0 += 8) {
                        const float4 f = s0 + l8 < s1 ? fine_centre(sc, B.pose, J, ew, s0 + l8, inflate) : absent_sphere();
                        for (unsigned m = rest; m; m &= m - 1u) {
                            hit = prim_hits(sc, h, i0 + __ffs(m) - 1, f);
                            hit = __any_sync(mask, hit);
                            if (hit) break;
                        }
                        if (hit) break;
                    }
                }
                alive &= ~__reduce_or_sync(kAll, hit ? 1u << ew : 0u);
            }
        };
        if (!gated) {
            for (int i0 = 0; i0 < n_obs; i0 += 32) {
                const unsigned bits = act && (alive >> w & 1u) ? cull_mask(sc, Ns, Nc, Nb, Nh, i0, ball) : 0u;
                fine(bits, i0);
            }
        } else {
            // the gate first: does the coarse sphere touch any primitive?
            bool dirty = false;
            for (int i0 = 0; i0 < n_obs; i0 += 32) {
                const unsigned bits = act ? cull_mask(sc, Ns, Nc, Nb, Nh, i0, ball) : 0u;
                for (unsigned m = bits; m && !dirty; m &= m - 1u) dirty = prim_hits(sc, h, i0 + __ffs(m) - 1, c);
                if (i0 < 256) marks[(i0 >> 5) * 32 + lane] = bits;
            }
            if (__any_sync(kAll, dirty)) {
                for (int i0 = 0; i0 < n_obs; i0 += 32) {
                    unsigned bits = 0u;
                    if (dirty && (alive >> w & 1u))
                        bits = i0 < 256 ? marks[(i0 >> 5) * 32 + lane] : cull_mask(sc, Ns, Nc, Nb, Nh, i0, ball);
                    fine(bits, i0);
                }
            }
        }
    }
    // the point cloud: a (sphere, configuration) per lane
    if (sc.pc.n > 0 && alive) {
        const int m = __popc(alive);
        __syncwarp();
        if (alive >> lane & 1u) B.list[__popc(alive & ((1u << lane) - 1u))] = lane;
        __syncwarp();
        unsigned flops = 0;
        for (int it0 = 0; it0 < m * S && alive; it0 += 32) {
            const int it = min(it0 + lane, m * S - 1), s = it / m, w = B.list[it - s * m];
            const float4 c = fine_centre(sc, B.pose, J, w, s, inflate);
            alive &= ~cloud_batch(sc.pc, c, it0 + lane < m * S, w, alive, flops);
        }
    }
    return (nw >= 32 ? kAll : (1u << nw) - 1u) & ~alive;
}

}  // namespace prrtc
