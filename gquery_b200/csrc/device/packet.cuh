// Warp-coherent ("packet") closest-point traversal, shared by the single-scene kernel
// (packet.cu) and the multi-scene batch kernel (batch.cu).
//
// The lanes of a warp that hold queries on the same scene walk its tree once: every
// lane tests the same node against its own query, a child is entered when at least one
// lane's search ball reaches it, and each lane keeps its own squared radius, winner and
// per-entry stack keys (a lane skips a popped entry whose key exceeds its radius).
// Morton-adjacent queries share most of the nodes they need, so the warp runs with its
// lanes in step instead of diverging per query.
//
// Answers equal those of the binary reference traversal except at FP32 distance ties:
// box tests are conservative (squared distances, 2^-18 slack, outward-rounded quantised
// boxes), leaf tests use the reference's closest-point formulas, and the caller
// recomputes the winner's record exactly.
#pragma once

#include <cuda_fp16.h>

#include "prim.cuh"
#include "queries.cuh"

namespace gqd {
namespace pkt {

constexpr int kNone = 0x7fffffff;
// Largest sort key of a hit child of a wide node: unused and missed child slots sort as
// +inf, and a hit whose key overflowed to +inf (a query with an infinite or huge
// coordinate) is clamped so that the hits stay ahead of them in the sorted order.
constexpr float kMaxHitKey = 3.40282347e38f;
constexpr float kSlack = 1.0000038f;  // 1 + 2^-18
constexpr int kPStack = 96;

__device__ __forceinline__ float exp_scale(uint32_t meta, int ax) {
    return __int_as_float((int)((meta >> (8 * ax)) & 0xffu) << 23);
}
__device__ __forceinline__ float qf(uint32_t lo4, uint32_t hi4, int k) {
    return __int_as_float((int)__byte_perm((k < 4) ? lo4 : hi4, 0x4B000000u, 0x7540u + (unsigned)(k & 3)));
}
// minimum of a non-negative float (or +inf) over the warp
__device__ __forceinline__ float warp_min(float x) {
    return __uint_as_float(__reduce_min_sync(0xffffffffu, __float_as_uint(x)));
}
__device__ __forceinline__ void pcas(float &ka, int &ra, float &kb, int &rb) {
    const bool sw = kb < ka;
    const float k0 = sw ? kb : ka, k1 = sw ? ka : kb;
    const int r0 = sw ? rb : ra, r1 = sw ? ra : rb;
    ka = k0; kb = k1; ra = r0; rb = r1;
}
__device__ __forceinline__ void psort8(float (&k)[8], int (&r)[8]) {  // Batcher odd-even merge sort
    pcas(k[0], r[0], k[1], r[1]); pcas(k[2], r[2], k[3], r[3]); pcas(k[4], r[4], k[5], r[5]); pcas(k[6], r[6], k[7], r[7]);
    pcas(k[0], r[0], k[2], r[2]); pcas(k[1], r[1], k[3], r[3]); pcas(k[4], r[4], k[6], r[6]); pcas(k[5], r[5], k[7], r[7]);
    pcas(k[1], r[1], k[2], r[2]); pcas(k[5], r[5], k[6], r[6]);
    pcas(k[0], r[0], k[4], r[4]); pcas(k[1], r[1], k[5], r[5]); pcas(k[2], r[2], k[6], r[6]); pcas(k[3], r[3], k[7], r[7]);
    pcas(k[2], r[2], k[4], r[4]); pcas(k[3], r[3], k[5], r[5]);
    pcas(k[1], r[1], k[2], r[2]); pcas(k[3], r[3], k[4], r[4]); pcas(k[5], r[5], k[6], r[6]);
}

// The walk's stack of (node, this lane's key) entries.
// Plain: each lane keeps both words of every entry in its local memory.
// Compact: the node of each entry is kept once per warp in shared memory (every lane
// writes the same word and reads back its own write, so no lane depends on another's
// store), and the lane's key is rounded down to FP16 in its local memory: 10 bytes per
// entry and warp instead of 256.  A key rounded down admits every entry the exact key
// admits, and at worst a few more, which cost a visit and change no answer.
template <bool COMPACT>
struct PStack;
template <>
struct PStack<false> {
    int2 *e;
    __device__ __forceinline__ PStack(int2 *p) : e(p) {}
    __device__ __forceinline__ void put(int i, int ref, float key) { e[i] = make_int2(ref, fbits(key)); }
    __device__ __forceinline__ void get(int i, int &ref, float &key) const {
        const int2 x = e[i];
        ref = x.x;
        key = __int_as_float(x.y);
    }
};
template <>
struct PStack<true> {
    int *refs;     // this warp's row (shared memory)
    __half *keys;  // this lane's keys (local memory)
    __device__ __forceinline__ void put(int i, int ref, float key) {
        refs[i] = ref;
        keys[i] = __float2half_rd(key);
    }
    __device__ __forceinline__ void get(int i, int &ref, float &key) const {
        ref = refs[i];
        key = __half2float(keys[i]);
    }
};

// square root within an ulp or two (one instruction)
__device__ __forceinline__ float sqrt_approx(float x) {
    float y;
    asm("sqrt.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}

// Ends the asynchronous copies that the walks started to bring nodes into L1: shared memory
// may go to another block, or be used for something else, only after this.
__device__ __forceinline__ void copies_done() { asm volatile("cp.async.wait_all;" ::: "memory"); }

// squared distances from p to the nearest / farthest point of a box
template <int D>
__device__ __forceinline__ void box_sq(const float *lo, const float *hi, const float *p, float &a2, float &b2) {
    a2 = 0.f;
    b2 = 0.f;
#pragma unroll
    for (int c = 0; c < D; ++c) {
        const float u = lo[c] - p[c], v = p[c] - hi[c];
        const float a = fmaxf(fmaxf(u, v), 0.f), b = fminf(u, v);
        a2 = __fmaf_rn(a, a, a2);
        b2 = __fmaf_rn(b, b, b2);
    }
}

// Squared distance below which x may have a point of the cylinder's set (gq_cyl_t).
__device__ __forceinline__ float cyl_bound(const float4 &c, const float4 &n, float px, float py, float pz) {
    const float ex = px - c.x, ey = py - c.y, ez = pz - c.z;
    const float h = __fmaf_rn(ez, n.z, __fmaf_rn(ey, n.y, ex * n.x));
    const float gx = __fmaf_rn(-h, n.x, ex), gy = __fmaf_rn(-h, n.y, ey), gz = __fmaf_rn(-h, n.z, ez);
    const float t = sqrt_approx(__fmaf_rn(gz, gz, __fmaf_rn(gy, gy, gx * gx)));
    const float a = fmaxf(fabsf(h) - n.w, 0.f), b = fmaxf(t - c.w, 0.f);
    return __fmaf_rn(a, a, b * b);
}

// The bound a cylinder has to exceed for its triangles to be left untested: (sqrt(r) + eps)^2
// for the squared radius r, and the smallest normal number on top, below which the root is
// taken of zero and squares lose their digits.  eps (2^-19 of the coordinates' size) is ten
// times the rounding of cyl_bound and of the closest point that the triangle test forms
// together, so a triangle that is left out would have had a key of at least r.  (The triangle
// test's barycentric coordinates lose digits with the square of the distance over the
// triangle's size, but the point they give stays in the triangle up to the margin.)
__device__ __forceinline__ float cyl_limit(float r, float eps) {
    const float s = sqrt_approx(r) + eps;
    return __fmaf_rn(s, s, 1.17549435e-38f);
}

// Squared distance from p to the closest point of triangle abc: the arithmetic of
// tri_closest (prim.cuh), rounding for rounding, with its seven regions chosen by selects
// around one division instead of branches, for lanes that hold unrelated triangles.  The
// closest point is base + e v + ac w: (a, ab) for a, the edges ab and ac and the inside,
// (b, cb) for b and the edge bc, c alone; terms of zero weight add exactly nothing.
__device__ __forceinline__ float tri_key(float px, float py, float pz, float ax, float ay, float az, float bx, float by,
                                         float bz, float cx, float cy, float cz) {
    const float abx = bx - ax, aby = by - ay, abz = bz - az;
    const float acx = cx - ax, acy = cy - ay, acz = cz - az;
    const float apx = px - ax, apy = py - ay, apz = pz - az;
    const float d1 = gq_dot3(abx, aby, abz, apx, apy, apz);
    const float d2 = gq_dot3(acx, acy, acz, apx, apy, apz);
    const float bpx = px - bx, bpy = py - by, bpz = pz - bz;
    const float d3 = gq_dot3(abx, aby, abz, bpx, bpy, bpz);
    const float d4 = gq_dot3(acx, acy, acz, bpx, bpy, bpz);
    const float cpx = px - cx, cpy = py - cy, cpz = pz - cz;
    const float d5 = gq_dot3(abx, aby, abz, cpx, cpy, cpz);
    const float d6 = gq_dot3(acx, acy, acz, cpx, cpy, cpz);
    const float vc = d1 * d4 - d3 * d2, vb = d5 * d2 - d1 * d6, va = d3 * d6 - d5 * d4;
    const float s43 = d4 - d3, s56 = d5 - d6;
    const bool in_a = (d1 <= 0.f) & (d2 <= 0.f);
    const bool in_b = !in_a & (d3 >= 0.f) & (d4 <= d3);
    const bool in_c = !in_a & !in_b & (d6 >= 0.f) & (d5 <= d6);
    const bool vertex = in_a | in_b | in_c;
    const bool on_ab = !vertex & (vc <= 0.f) & (d1 >= 0.f) & (d3 <= 0.f);
    const bool on_ac = !vertex & !on_ab & (vb <= 0.f) & (d2 >= 0.f) & (d6 <= 0.f);
    const bool on_bc = !vertex & !on_ab & !on_ac & (va <= 0.f) & (s43 >= 0.f) & (s56 >= 0.f);
    float num = 1.f, den = va + vb + vc;
    if (on_bc) num = s43, den = s43 + s56;
    if (on_ac) num = d2, den = d2 - d6;
    if (on_ab) num = d1, den = d1 - d3;
    if (vertex) den = 1.f;
    const float x = gq_div(num, den);
    float v = vb * x, w = vc * x;
    if (on_ab | on_bc) v = x, w = 0.f;
    if (on_ac) v = 0.f, w = x;
    if (vertex) v = 0.f, w = 0.f;
    const bool from_b = in_b | on_bc;
    const float ox = from_b ? bx : in_c ? cx : ax, oy = from_b ? by : in_c ? cy : ay, oz = from_b ? bz : in_c ? cz : az;
    const float ux = on_bc ? cx - bx : abx, uy = on_bc ? cy - by : aby, uz = on_bc ? cz - bz : abz;
    const float ex = px - ((ox + ux * v) + acx * w), ey = py - ((oy + uy * v) + acy * w),
                ez = pz - ((oz + uz * v) + acz * w);
    return gq_dot3(ex, ey, ez, ex, ey, ez);
}

// Pairs of a triangle and a lane that are tested side by side: two rounds of the warp (32 / 64 /
// 96: 250,007 points near a 327,680-triangle surface 786 / 743 / 724 us, 8,388,608 uniform points
// on 1,310,720 triangles 22.4 / 22.7 / 23.9 ms).
constexpr int kRunPairs = 64;
// Shared memory of one warp for the (triangle of a run, lane) pairs of leaf().
struct LeafBuf {
    float key[kRunPairs];
    uint8_t pair[kRunPairs];  // triangle << 5 | lane
    uint32_t sink[32];
};
static_assert(GQ_COLLAPSE_MAX <= 8, "a pair of leaf() fits a byte");

// Triangle j for the lanes with `act`; whether it is its leaf's last.
__device__ __forceinline__ bool tri_test(const DevScene &s, int j, bool act, const float *p, float &r, int &idx) {
    const float4 t0 = ldg4(s.prims, 3 * (int64_t)j), t1 = ldg4(s.prims, 3 * (int64_t)j + 1),
                 t2 = ldg4(s.prims, 3 * (int64_t)j + 2);
    if (act) {
        float pt[3], u, v;
        tri_closest<true>(p[0], p[1], p[2], t0.x, t0.y, t0.z, t0.w, t1.x, t1.y, t1.z, t1.w, t2.x, pt, &u, &v);
        const float ex = p[0] - pt[0], ey = p[1] - pt[1], ez = p[2] - pt[2];
        const float key = gq_dot3(ex, ey, ez, ex, ey, ez);
        if (key < r) {
            r = key;
            idx = j;
        }
    }
    return (fbits(t2.z) & GQ_ITEM_LAST) != 0;
}

// A run of at most GQ_COLLAPSE_MAX triangles from `first`, for the lanes in cmask.
//
// A triangle test costs about 100 instructions and nearly none improves a lane: of 584 per
// tile of 32 queries (8,388,608 uniform points on 1,310,720 triangles; counts of a model of
// the walk) 32 do.  So the run's cylinder (about 20 instructions) comes first: it leaves out 72
// of the tile's 126 runs, and most lanes of the others.
//
// FORM > 0: at most kRunPairs pairs of a triangle and a lane that is left (few lanes need a run
// where queries are sparse: 8 of 32 near a surface, 4 for 2,003 points) are listed in shared
// memory, every lane of the warp tests one, and each query's lane then takes its keys in the
// triangles' order.  Otherwise the lanes test the triangles one by one.  FORM 2, bound by
// latency, asks the cylinder only where there are more pairs (cylinder first / pairs first:
// 16,384 points on 327,680 curved triangles 2.16 / 2.31 ms, on 318,402 coplanar ones 455 / 426 us).
//
// FORM 1, without / with the cylinder before the pairs: 2,097,157 points near 327,680 triangles 7.7 /
// 6.6 ms, 8,388,608 uniform on 1,310,720 20.4 / 17.5; on a tube of 320,000 slivers, which bound nothing,
// 21.9 / 22.0 and 43.1 / 39.4.  A disc per triangle before its test, in place of the pairs: 8.9, 18.2,
// 30.6 and 47.6 ms.
//
// A test that is left out would have left every lane's radius and winner as they are
// (cyl_limit), and the pairs are taken in the order of the plain loop, so the walk
// and its answers are those of testing every triangle, ties included.
// RUNCYL: the run is a pair record's (run_cyl holds its cylinder).
template <bool RUNCYL, int FORM>
__device__ __forceinline__ void run3(const DevScene &s, int first, int count, unsigned cmask, const float *p, float eps,
                                     float &r, int &idx, LeafBuf *buf) {
    const unsigned lane = threadIdx.x & 31u;
    unsigned need = cmask;
    if (RUNCYL && !(FORM == 2 && __popc(cmask) * count <= kRunPairs)) {
        const float4 c = ldg4(s.run_cyl, 2 * (int64_t)first), n = ldg4(s.run_cyl, 2 * (int64_t)first + 1);
        if (c.w < kInf) {
            need = __ballot_sync(0xffffffffu, ((cmask >> lane) & 1u) &&
                                                  !(cyl_bound(c, n, p[0], p[1], p[2]) > cyl_limit(r, eps)));
            if (!need) return;
        }
    }
    const bool act = (need >> lane) & 1u;
    const int lanes = __popc(need), total = lanes * count;
    if (FORM && total <= kRunPairs) {
        const int rank = __popc(need & ((1u << lane) - 1u));
        if (act)
            for (int t = 0; t < count; ++t) buf->pair[t * lanes + rank] = (uint8_t)(t << 5 | lane);
        __syncwarp();
        for (int k0 = 0; k0 < total; k0 += 32) {
            const int k = k0 + (int)lane;
            const unsigned e = k < total ? buf->pair[k] : 0u;
            const float x = __shfl_sync(0xffffffffu, p[0], e & 31u), y = __shfl_sync(0xffffffffu, p[1], e & 31u),
                        z = __shfl_sync(0xffffffffu, p[2], e & 31u);
            if (k < total) {
                const int64_t j = 3 * (int64_t)(first + (int)(e >> 5));
                const float4 t0 = ldg4(s.prims, j), t1 = ldg4(s.prims, j + 1), t2 = ldg4(s.prims, j + 2);
                buf->key[k] = tri_key(x, y, z, t0.x, t0.y, t0.z, t0.w, t1.x, t1.y, t1.z, t1.w, t2.x);
            }
        }
        __syncwarp();
        if (act)
            for (int t = 0; t < count; ++t) {
                const float key = buf->key[t * lanes + rank];
                if (key < r) {
                    r = key;
                    idx = first + t;
                }
            }
        __syncwarp();  // the buffer is free again
        return;
    }
    for (int j = first; j < first + count; ++j) tri_test(s, j, act, p, r, idx);
}

// Leaf: every lane that needs it (cmask) tests the leaf's items against its query.
template <int D, bool RUNCYL, int FORM>
__device__ __forceinline__ void leaf(const DevScene &s, int ref, unsigned cmask, const float *p, float eps, float &r,
                                     int &idx, LeafBuf *buf) {
    const bool act = (cmask >> (threadIdx.x & 31u)) & 1u;
    // a run of a collapsed subtree (bit 30 clear): first in bits 0-23, count in 24-29;
    // an ordinary leaf ~first (first < 2^30, so bit 30 set) runs to its last item
    const bool run = (ref & 0x40000000) == 0;
    int j = run ? (ref & 0xffffff) : ~ref;
    const int end = run ? j + ((ref >> 24) & 0x3f) : 0;
    if (run && end == j) return;  // an empty run (INT32_MIN, an unused wide slot): nothing to test
    if (D == 3 && run) {
        run3<RUNCYL, FORM>(s, j, end - j, cmask, p, eps, r, idx, buf);
        return;
    }
    for (;;) {
        bool last;
        if (D == 3) {
            last = tri_test(s, j, act, p, r, idx);  // a leaf of more than GQ_COLLAPSE_MAX triangles, or a device-built tree's
        } else {
            const float4 a = ldg4(s.prims, 2 * (int64_t)j);
            const int4 f = __ldg(reinterpret_cast<const int4 *>(s.prims) + 2 * (int64_t)j + 1);
            last = run ? j + 1 == end : (f.y & GQ_ITEM_LAST) != 0;
            if (act) {
                const float ux = a.z - a.x, uy = a.w - a.y, vx = p[0] - a.x, vy = p[D - 1] - a.y;
                const float t = gq_clamp(gq_div(gq_dot2(vx, vy, ux, uy), gq_dot2(ux, uy, ux, uy)), 0.f, 1.f);
                const float qx = gq_lerp(a.x, a.z, t) - p[0], qy = gq_lerp(a.y, a.w, t) - p[D - 1];
                const float key = gq_dot2(qx, qy, qx, qy);
                if (key < r) {
                    r = key;
                    idx = j;
                }
            }
        }
        if (last) break;
        ++j;
    }
}

// One traversal for the lanes in `mask` (warp-uniform).  All 32 lanes must call it.
// r: this lane's squared search radius (+inf to start; lanes outside `mask` are
// ignored), idx: its best item slot (-1: none).  LAYOUT 0: binary pairs,
// 1: quantised 8-wide nodes (3D only).  STK: entries of the caller's stack `stk`; the
// warp stops with `ovf` set rather than overflow it.
// COMPACT: the stack of PStack<true> (FP16 keys, one node word per warp).
// FORM (LAYOUT 0): 1 run3's pairs (3D); 2 those and the children brought into L1 ahead, for calls
// whose time is the latency of a few walks rather than their number.  buf: this warp's
// LeafBuf in shared memory.
template <int D, int LAYOUT, bool MINFIRST, int STK = kPStack, bool COMPACT = false, int FORM = 0>
__device__ __forceinline__ void closest_point(const DevScene &s, unsigned mask, const float *p, float &r, int &idx,
                                              bool &ovf, PStack<COMPACT> stk, LeafBuf *buf = nullptr) {
    const unsigned lane = threadIdx.x & 31u;
    const bool mine = (mask >> lane) & 1u;
    if (!mine) r = 0.f;  // never needs a node
    float eps = 0.f;
    if (D == 3) eps = (fmaxf(fmaxf(fabsf(p[0]), fabsf(p[1])), fabsf(p[D - 1])) + s.coord_bound) * 1.9073486e-06f;  // 2^-19
    const unsigned sink = FORM == 2 ? (unsigned)__cvta_generic_to_shared(&buf->sink[lane]) : 0u;
    int cur = LAYOUT ? s.wroot_ref : s.root_ref;
    unsigned cmask = mask;
    int sp = -1;
    for (;;) {
        if (cur == kNone) {
            bool found = false;
            while (sp >= 0) {
                int eref;
                float ekey;
                stk.get(sp--, eref, ekey);
                const unsigned m = __ballot_sync(0xffffffffu, ekey <= r * kSlack);
                if (m) {
                    cur = eref;
                    cmask = m;
                    found = true;
                    break;
                }
            }
            if (!found) break;
        }
        const bool act = (cmask >> lane) & 1u;
        if (cur < 0) {
            leaf<D, LAYOUT == 0, FORM>(s, cur, cmask, p, eps, r, idx, buf);
            cur = kNone;
            continue;
        }
        if (LAYOUT == 0) {
            float lo[2][D], hi[2][D];
            int rl, rr;
            if (D == 3) {
                const float4 a = ldg4(s.pairs, 4 * (int64_t)cur), b = ldg4(s.pairs, 4 * (int64_t)cur + 1),
                             c = ldg4(s.pairs, 4 * (int64_t)cur + 2);
                const int4 rf = __ldg(reinterpret_cast<const int4 *>(s.pairs) + 4 * (int64_t)cur + 3);
                lo[0][0] = a.x; lo[0][1] = a.y; lo[0][D - 1] = a.z; hi[0][0] = a.w; hi[0][1] = b.x; hi[0][D - 1] = b.y;
                lo[1][0] = b.z; lo[1][1] = b.w; lo[1][D - 1] = c.x; hi[1][0] = c.y; hi[1][1] = c.z; hi[1][D - 1] = c.w;
                // a small subtree is tested as one run (sub_l / sub_r of the pair record)
                rl = rf.z ? (int)(0x80000000u | (unsigned)rf.z) : rf.x;
                rr = rf.w ? (int)(0x80000000u | (unsigned)rf.w) : rf.y;
            } else {
                const float4 a = ldg4(s.pairs, 3 * (int64_t)cur), b = ldg4(s.pairs, 3 * (int64_t)cur + 1);
                const int4 rf = __ldg(reinterpret_cast<const int4 *>(s.pairs) + 3 * (int64_t)cur + 2);
                lo[0][0] = a.x; lo[0][D - 1] = a.y; hi[0][0] = a.z; hi[0][D - 1] = a.w;
                lo[1][0] = b.x; lo[1][D - 1] = b.y; hi[1][0] = b.z; hi[1][D - 1] = b.w;
                rl = rf.z ? (int)(0x80000000u | (unsigned)rf.z) : rf.x;
                rr = rf.w ? (int)(0x80000000u | (unsigned)rf.w) : rf.y;
            }
            if (FORM == 2) {
                // Bring what a visit of either child reads first into L1 while the boxes are
                // tested: half a warp per child, 4 bytes a lane to a place nobody reads.  An
                // asynchronous copy needs no destination register, which a load would have to
                // wait for at the next node.
                const int cref = lane < 16 ? rl : rr;
                const unsigned w = lane & 15u;
                constexpr unsigned kPair = D == 3 ? 64 : 48, kItem = D == 3 ? 48 : 32;
                const char *from = (const char *)s.pairs + ((int64_t)(cref >= 0 ? cref : cur) * kPair + min(4 * w, kPair - 4));
                if (cref < 0 && (cref & 0x40000000) == 0)  // a run: its items, at most 288 B
                    from = (const char *)s.prims +
                           ((int64_t)(cref & 0xffffff) * kItem + min(16 * w, kItem * ((cref >> 24) & 0x3fu) - 4));
                asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(sink), "l"(from));
            }
            float a2l = kInf, b2l = kInf, a2r = kInf, b2r = kInf;
            if (act) {
                box_sq<D>(lo[0], hi[0], p, a2l, b2l);
                box_sq<D>(lo[1], hi[1], p, a2r, b2r);
                r = fminf(r, fminf(b2l, b2r) * kSlack);
            }
            const float lim = r * kSlack;
            const bool hl = act && a2l <= lim, hr = act && a2r <= lim;
            const unsigned ml = __ballot_sync(0xffffffffu, hl), mr = __ballot_sync(0xffffffffu, hr);
            if (ml && mr) {
                const float kl = warp_min(hl ? a2l : kInf), kr = warp_min(hr ? a2r : kInf);
                const bool right_first = kr < kl;
                if (sp + 1 >= min(STK, s.stack_cap)) {
                    ovf = true;
                    break;
                }
                ++sp;
                stk.put(sp, right_first ? rl : rr, right_first ? (hl ? a2l : kInf) : (hr ? a2r : kInf));
                cur = right_first ? rr : rl;
                cmask = right_first ? mr : ml;
            } else if (ml) {
                cur = rl;
                cmask = ml;
            } else if (mr) {
                cur = rr;
                cmask = mr;
            } else {
                cur = kNone;
            }
        } else {
            const int64_t nb = 6 * (int64_t)cur;
            const float4 h = ldg4(s.wnodes, nb);
            const int4 r0 = __ldg(reinterpret_cast<const int4 *>(s.wnodes) + nb + 1);
            const int4 r1 = __ldg(reinterpret_cast<const int4 *>(s.wnodes) + nb + 2);
            const uint4 q0 = __ldg(reinterpret_cast<const uint4 *>(s.wnodes) + nb + 3);
            const uint4 q1 = __ldg(reinterpret_cast<const uint4 *>(s.wnodes) + nb + 4);
            const uint4 q2 = __ldg(reinterpret_cast<const uint4 *>(s.wnodes) + nb + 5);
            const uint32_t meta = (uint32_t)fbits(h.w);
            const int nc = (int)(meta >> 24);
            const float sx = exp_scale(meta, 0), sy = exp_scale(meta, 1), sz = exp_scale(meta, 2);
            float key[8];
            int ref[8] = {r0.x, r0.y, r0.z, r0.w, r1.x, r1.y, r1.z, r1.w};
            float shrink = kInf;
#pragma unroll
            for (int k = 0; k < 8; ++k) {
                // NaN for inactive lanes and unused slots: it fails every `<= lim`, also while
                // lim is +inf (an unused slot holds no node)
                float a2 = __int_as_float(0x7fc00000), b2 = kInf;
                if (act && k < nc) {
                    const float lo3[3] = {__fmaf_rn(qf(q0.x, q0.y, k), sx, h.x), __fmaf_rn(qf(q0.z, q0.w, k), sy, h.y),
                                          __fmaf_rn(qf(q1.x, q1.y, k), sz, h.z)};
                    const float hi3[3] = {__fmaf_rn(qf(q1.z, q1.w, k), sx, h.x), __fmaf_rn(qf(q2.x, q2.y, k), sy, h.y),
                                          __fmaf_rn(qf(q2.z, q2.w, k), sz, h.z)};
                    box_sq<3>(lo3, hi3, p, a2, b2);
                }
                key[k] = a2;
                shrink = fminf(shrink, b2);
            }
            if (act) r = fminf(r, shrink * kSlack);
            const float lim = r * kSlack;
            float wkey[8];
            unsigned wmask[8];
            int cnt = 0;
#pragma unroll
            for (int k = 0; k < 8; ++k) {
                const bool hit = key[k] <= lim;
                key[k] = hit ? key[k] : kInf;
                wmask[k] = __ballot_sync(0xffffffffu, hit);
                // hits clamped below the others' +inf: they sort first, and the nearest-first
                // choice is a hit, so that it pushes at most cnt - 1 entries
                wkey[k] = wmask[k] ? fminf(warp_min(key[k]), kMaxHitKey) : kInf;
                cnt += wmask[k] ? 1 : 0;
            }
            if (cnt == 0) {
                cur = kNone;
                continue;
            }
            if (sp + cnt > min(STK, s.stack_cap)) {
                ovf = true;
                break;
            }
            if (MINFIRST) {
                float bk = wkey[0];
                int best = 0;
#pragma unroll
                for (int k = 1; k < 8; ++k) {
                    const bool lt = wkey[k] < bk;
                    bk = lt ? wkey[k] : bk;
                    best = lt ? k : best;
                }
                int c0 = ref[0];
                unsigned m0 = wmask[0];
#pragma unroll
                for (int k = 7; k >= 0; --k) {
                    if (k == best) {
                        c0 = ref[k];
                        m0 = wmask[k];
                    } else if (wmask[k]) {
                        stk.put(++sp, ref[k], key[k]);
                    }
                }
                cur = c0;
                cmask = m0;
                continue;
            }
            // children in the order of the nearest lane's distance; lane keys travel with the refs
            int slot[8] = {0, 1, 2, 3, 4, 5, 6, 7};
            float wk[8];
#pragma unroll
            for (int k = 0; k < 8; ++k) wk[k] = wkey[k];
            psort8(wk, slot);
#pragma unroll
            for (int k = 7; k >= 1; --k) {
                if (k < cnt) {
                    int sref = ref[0];
                    float skey = key[0];
#pragma unroll
                    for (int m = 1; m < 8; ++m) {
                        sref = (slot[k] == m) ? ref[m] : sref;
                        skey = (slot[k] == m) ? key[m] : skey;
                    }
                    stk.put(++sp, sref, skey);
                }
            }
            int c0 = ref[0];
            unsigned m0 = wmask[0];
#pragma unroll
            for (int m = 1; m < 8; ++m) {
                c0 = (slot[0] == m) ? ref[m] : c0;
                m0 = (slot[0] == m) ? wmask[m] : m0;
            }
            cur = c0;
            cmask = m0;
        }
    }
}

}  // namespace pkt
}  // namespace gqd
