// Ray walk over the quantised 8-wide BVH, one ray per lane (the 8-wide variant's default).
//
// The other per-lane walk (traverse.cuh) spends about 430 instructions on a node with 7 of
// 32 lanes active: every child's planes are decoded, shifted and scaled one by one, the hits are
// sorted with their references, and a lane tests the items of its leaf while the others
// wait.  Here
//   * a plane's t is one byte permute and one fma (the node's grid is brought into the
//     ray's parameter once, and near and far rows are chosen by the direction's sign), and the
//     sort moves one word per child, about 240 instructions in all;
//   * the leaf items of all waiting lanes are tested together, one per lane (leaves());
//   * a warp holds as many rays as its share of the call (ray_walk.cu).
// Binary pairs instead of 8-wide nodes (50 instructions a node, three times the nodes) were slower:
// 6.9 against 6.0 ms on 8,388,608 sorted rays, as a step waits for its node's read either way.
//
// Boxes are tested conservatively: each plane's t is moved outward by eps / |direction|, eps
// = 2^-20 of the coordinates' size, sixteen times the rounding of the fma form, so every
// box that holds a triangle or segment the leaf test can hit is entered.  The leaf tests are
// the reference's.  The nearest hit does not depend on the order of the visits unless two
// items are hit at exactly the same t; such a ray (2 of 8,388,608 on the benchmark) is
// walked again by the other walk, whose order picks the winner: the answers are that
// walk's bit for bit.  So is a ray whose products could leave the range in which the margins
// hold (init()).
#pragma once

#include "prim.cuh"
#include "queries.cuh"
#include "records.cuh"
#include "traverse.cuh"

namespace gqd {
namespace rayw {

constexpr int kNone = 0x7fffffff;
using Stack = int2[GQ_STACK_WIDE];

template <int D>
struct Lane {
    float p[D], v[D];
    float iv[D], on[D], of[D];  // 1 / direction; -p iv moved down / up by eps |iv|
    float r;                    // r_max, then the nearest hit
    int idx, cur, sp;
    bool again, ovf;            // again: the other walk answers this ray
};

// Both planes of one axis: the near one into tn, the far one into tf.
template <int D>
__device__ __forceinline__ void slab(const Lane<D> &L, const float *lo, const float *hi, float &tn, float &tf) {
    tn = 0.f;
    tf = L.r;
#pragma unroll
    for (int k = 0; k < D; ++k) {
        const bool neg = L.iv[k] < 0.f;
        tn = fmaxf(tn, __fmaf_rn(neg ? hi[k] : lo[k], L.iv[k], L.on[k]));
        tf = fminf(tf, __fmaf_rn(neg ? lo[k] : hi[k], L.iv[k], L.of[k]));
    }
}

// The ray of query qi; cur = kNone when it cannot hit.
template <int D>
__device__ __forceinline__ void init(const DevScene &s, Lane<D> &L, const gq_vecs &a, const gq_vecs &b,
                                     const float *rmax_in, int64_t qi) {
    float pmax = 0.f, vmax = 0.f;
#pragma unroll
    for (int k = 0; k < D; ++k) {
        L.p[k] = trav::qget(a, qi, k);
        L.v[k] = trav::qget(b, qi, k);
        pmax = fmaxf(pmax, fabsf(L.p[k]));
        vmax = fmaxf(vmax, fabsf(L.v[k]));
    }
    const float size = pmax + s.coord_bound, eps = size * 9.5367432e-07f;  // 2^-20
    bool tame = true;
#pragma unroll
    for (int k = 0; k < D; ++k) {
        // a component below 1e-12 of the largest moves the ray by less than eps over any
        // distance that matters, and would overflow the products
        L.iv[k] = gq_div(1.f, copysignf(fmaxf(fabsf(L.v[k]), vmax * 1e-12f), L.v[k]));
        // Parameters t are at most some 2^9 times size / |direction| (a node's origin lies 2^15
        // of its steps low), the margin is 2^-20 of it.  From 2^-110 to 2^110 neither
        // overflows, and the margin is above 2^5 times what subnormal products lose.  Outside,
        // and where a component is infinite (iv = 0, and with it every t), boxes could be lost or
        // none left out.
        const float t = size * fabsf(L.iv[k]);
        tame = tame && t >= 7.7037198e-34f && t <= 1.2980742e33f;
        const float o = -(L.p[k] * L.iv[k]), e = eps * fabsf(L.iv[k]);
        L.on[k] = o - e;
        L.of[k] = o + e;
    }
    L.r = rmax_in ? rmax_in[qi] : kInf;
    L.idx = -1;
    L.sp = -1;
    L.again = !tame && vmax > 0.f;
    L.ovf = false;
    float tn, tf;
    slab<D>(L, s.root_lo, s.root_hi, tn, tf);
    bool enter = tame && tn <= tf;  // a ray without a direction hits nothing
    if (enter) {
        // the reference's own test of the root box (bvh.py:209-216), which decides
        float t_root;
        bool hit;
        if (D == 3)
            hit = box_ray3(s.root_lo[0], s.root_lo[1], s.root_lo[2], s.root_hi[0], s.root_hi[1], s.root_hi[2], L.p[0],
                           L.p[1], L.p[D - 1], L.v[0], L.v[1], L.v[D - 1], L.r, t_root);
        else
            hit = box_ray2(s.root_lo[0], s.root_lo[1], s.root_hi[0], s.root_hi[1], L.p[0], L.p[D - 1], L.v[0],
                           L.v[D - 1], L.r, t_root);
        enter = hit && t_root <= L.r;
    }
    L.cur = enter ? s.wroot_ref : kNone;
}

template <int D>
__device__ __forceinline__ void pop(Lane<D> &L, const int2 *stk) {
    L.cur = kNone;
    while (L.sp >= 0) {
        const int2 e = stk[L.sp--];
        if (__int_as_float(e.y) <= L.r) {
            L.cur = e.x;
            break;
        }
    }
}

// 2^15 + byte k of the 8-byte row (lo4, hi4), built with one byte permute.
__device__ __forceinline__ float q15(uint32_t lo4, uint32_t hi4, int k) {
    return __int_as_float((int)__byte_perm((k < 4) ? lo4 : hi4, 0x47000000u, 0x7404u | (unsigned)(k & 3) << 4));
}
__device__ __forceinline__ void order2(uint32_t &a, uint32_t &b) {
    const uint32_t lo = min(a, b), hi = max(a, b);
    a = lo;
    b = hi;
}

// Node cur: the nearest hit child next, the others on the stack, the farthest deepest.
// The planes of child k are org + (2^15 + q) 2^e; with A = 2^e iv and B = org iv + on (of)
// each plane's t is one fma of q.  The keys carry the child's slot in their last three
// bits, so the sort moves one word per child.
template <int D>
__device__ __forceinline__ void node(const void *wnodes, Lane<D> &L, int2 *stk) {
    constexpr int F4 = (D == 3) ? 6 : 5;  // 16-byte words per node
    const int64_t at = F4 * (int64_t)L.cur;
    const float4 h = ldg4(wnodes, at);
    const uint4 q0 = __ldg(reinterpret_cast<const uint4 *>(wnodes) + at + 3);
    const uint4 q1 = __ldg(reinterpret_cast<const uint4 *>(wnodes) + at + 4);
    uint4 q2 = make_uint4(0, 0, 0, 0);
    if (D == 3) q2 = __ldg(reinterpret_cast<const uint4 *>(wnodes) + at + 5);
    const uint32_t meta = (uint32_t)fbits(D == 3 ? h.w : h.z);
    const int nc = (int)(meta >> 24);
    float A[D], Bn[D], Bf[D];
    uint32_t nl[D], nh[D], fl[D], fh[D];  // near and far rows, children 0-3 and 4-7
    {
        const uint32_t rl[3][2] = {{q0.x, q0.y}, {q0.z, q0.w}, {q1.x, q1.y}};
        const uint32_t rh[3][2] = {{D == 3 ? q1.z : q1.x, D == 3 ? q1.w : q1.y},
                                   {D == 3 ? q2.x : q1.z, D == 3 ? q2.y : q1.w}, {q2.z, q2.w}};
        const float org[3] = {h.x, h.y, h.z};
#pragma unroll
        for (int k = 0; k < D; ++k) {
            const float sc = trav::exp_scale(meta, k);
            const float o = __fmaf_rn(8355840.f, sc, org[k]);  // stored 2^23 steps low: now 2^15
            A[k] = sc * L.iv[k];
            // a hundredth of a step outward: the rounding of B is below 2^-8 of a step
            Bn[k] = __fmaf_rn(o, L.iv[k], __fmaf_rn(fabsf(A[k]), -0.01f, L.on[k]));
            Bf[k] = __fmaf_rn(o, L.iv[k], __fmaf_rn(fabsf(A[k]), 0.01f, L.of[k]));
            const bool neg = L.iv[k] < 0.f;
            nl[k] = neg ? rh[k][0] : rl[k][0];
            nh[k] = neg ? rh[k][1] : rl[k][1];
            fl[k] = neg ? rl[k][0] : rh[k][0];
            fh[k] = neg ? rl[k][1] : rh[k][1];
        }
    }
    uint32_t key[8];
    int cnt = 0;
#pragma unroll
    for (int k = 0; k < 8; ++k) {
        float tn = 0.f, tf = L.r;
#pragma unroll
        for (int c = 0; c < D; ++c) {
            tn = fmaxf(tn, __fmaf_rn(q15(nl[c], nh[c], k), A[c], Bn[c]));
            tf = fminf(tf, __fmaf_rn(q15(fl[c], fh[c], k), A[c], Bf[c]));
        }
        const bool hit = (k < nc) && tn <= tf;
        key[k] = hit ? ((uint32_t)fbits(tn) & ~7u) | (uint32_t)k : 0xffffffffu;
        cnt += hit ? 1 : 0;
    }
    if (cnt == 0) {
        pop<D>(L, stk);
        return;
    }
    if (L.sp + cnt > GQ_STACK_WIDE) {
        L.ovf = true;
        L.sp = -1;
        L.cur = kNone;
        return;
    }
    if (cnt > 1) {
        order2(key[0], key[1]); order2(key[2], key[3]); order2(key[4], key[5]); order2(key[6], key[7]);
        order2(key[0], key[2]); order2(key[1], key[3]); order2(key[4], key[6]); order2(key[5], key[7]);
        order2(key[1], key[2]); order2(key[5], key[6]);
        order2(key[0], key[4]); order2(key[1], key[5]); order2(key[2], key[6]); order2(key[3], key[7]);
        order2(key[2], key[4]); order2(key[3], key[5]);
        order2(key[1], key[2]); order2(key[3], key[4]); order2(key[5], key[6]);
    } else {
#pragma unroll
        for (int k = 1; k < 8; ++k) key[0] = min(key[0], key[k]);
    }
    const int *refs = reinterpret_cast<const int *>(wnodes) + 4 * (at + 1);
#pragma unroll
    for (int k = 7; k >= 1; --k)
        if (k < cnt) stk[++L.sp] = make_int2(__ldg(refs + (key[k] & 7u)), (int)(key[k] & ~7u));
    L.cur = __ldg(refs + (key[0] & 7u));
}

template <int D>
__device__ __forceinline__ float item_ray(const void *prims, int j, const float *p, const float *v, bool &last) {
    if (D == 3) {
        const float4 t0 = ldg4(prims, 3 * (int64_t)j), t1 = ldg4(prims, 3 * (int64_t)j + 1),
                     t2 = ldg4(prims, 3 * (int64_t)j + 2);
        last = (fbits(t2.z) & GQ_ITEM_LAST) != 0;
        return tri_ray(p[0], p[1], p[D - 1], v[0], v[1], v[D - 1], t0.x, t0.y, t0.z, t0.w, t1.x, t1.y, t1.z, t1.w, t2.x,
                       kInf);
    }
    const float4 a = ldg4(prims, 2 * (int64_t)j);
    last = (__ldg(reinterpret_cast<const int4 *>(prims) + 2 * (int64_t)j + 1).y & GQ_ITEM_LAST) != 0;
    return seg_ray(p[0], p[D - 1], v[0], v[D - 1], a.x, a.y, a.z, a.w);
}

// The nearest item (j at t = key) of a leaf or run.  Both walks test its items in order and keep
// the first of equals; only an equal item of another leaf (L.idx) leaves the order open.
template <int D>
__device__ __forceinline__ void take(Lane<D> &L, float key, int j) {
    if (key < L.r) {
        L.r = key;
        L.idx = j;
        L.again = false;
    } else if (key == L.r && L.idx >= 0) {
        L.again = true;
    }
}

// Shared memory of one warp for leaves().
struct LeafBuf {
    float key[32 * GQ_COLLAPSE_MAX];
    uint8_t pair[32 * GQ_COLLAPSE_MAX];  // item << 5 | lane
};

// The leaves of all lanes with cur < 0, and each of those lanes' next node.  All 32 lanes call.
//
// A run holds up to six items and the rays that skim a surface meet hundreds of them
// one after another, which is what a call of few rays waits for; so the pairs (item, lane) of all
// waiting lanes are listed in shared memory and every lane of the warp tests one.
// Each ray's lane then takes the first of its smallest keys.
// MANY: the rays may be of different scenes (each lane passes its scene's items).
template <int D, bool MANY>
__device__ __forceinline__ void leaves(const void *prims, Lane<D> &L, const int2 *stk, LeafBuf &buf) {
    const unsigned lane = threadIdx.x & 31u, below = (1u << lane) - 1u;
    const bool here = L.cur < 0;
    // a run child (bit 30 clear) holds its count, an ordinary leaf ends at its last item
    const bool run = here && (L.cur & 0x40000000) == 0;
    const int first = run ? (L.cur & 0xffffff) : ~L.cur, count = run ? (L.cur >> 24) & 0x3f : 0;
    unsigned m[GQ_COLLAPSE_MAX];
    int total = 0;
#pragma unroll
    for (int t = 0; t < GQ_COLLAPSE_MAX; ++t) {
        m[t] = __ballot_sync(0xffffffffu, t < count);
        if (t < count) buf.pair[total + __popc(m[t] & below)] = (uint8_t)(t << 5 | lane);
        total += __popc(m[t]);
    }
    __syncwarp();
    for (int k0 = 0; k0 < total; k0 += 32) {
        const int k = k0 + (int)lane;
        const unsigned e = k < total ? buf.pair[k] : 0u;
        const int j = __shfl_sync(0xffffffffu, first, e & 31u) + (int)(e >> 5);
        float p[D], v[D];
#pragma unroll
        for (int c = 0; c < D; ++c) {
            p[c] = __shfl_sync(0xffffffffu, L.p[c], e & 31u);
            v[c] = __shfl_sync(0xffffffffu, L.v[c], e & 31u);
        }
        const void *items = prims;
        if (MANY) {
            const unsigned long long at = (unsigned long long)prims;
            items = (const void *)__shfl_sync(0xffffffffu, at, e & 31u);
        }
        bool last;
        if (k < total) buf.key[k] = item_ray<D>(items, j, p, v, last);
    }
    __syncwarp();
    float key = kInf;  // nearest of the leaf
    int at = first, base = 0;
#pragma unroll
    for (int t = 0; t < GQ_COLLAPSE_MAX; ++t) {
        if (t < count) {
            const float k = buf.key[base + __popc(m[t] & below)];
            if (k < key) {
                key = k;
                at = first + t;
            }
        }
        base += __popc(m[t]);
    }
    __syncwarp();  // the buffer is free again
    if (here) {
        if (!run)
            for (int j = first;; ++j) {
                bool last;
                const float k = item_ray<D>(prims, j, L.p, L.v, last);
                if (k < key) {
                    key = k;
                    at = j;
                }
                if (last) break;
            }
        take<D>(L, key, at);
        pop<D>(L, stk);
    }
}

// A ray with an exact tie or outside this walk's range: the other walk over the 8-wide nodes.
// Returns its primitive and the bits of its t, -2 after a stack overflow.
template <int D>
__device__ __noinline__ int2 other_walk(const DevScene &s, const gq_vecs &a, const gq_vecs &b, const float *rmax_in,
                                        int64_t qi) {
    trav::Stack<true> stk;
    trav::Lane<D, true, true> W;
    trav::lane_init(s, W, a, b, rmax_in, qi);
    while (!trav::lane_run<D, true, true, 0>(s, W, stk, 1 << 30)) {
    }
    return make_int2(W.ovf ? -2 : W.idx, fbits(W.r));
}

template <int D>
__device__ __forceinline__ void finish(const DevScene &s, Lane<D> &L, const gq_vecs &a, const gq_vecs &b,
                                       const float *rmax_in, int64_t qi, int64_t n, const gq_ray_out &o) {
    if (L.again) {
        const int2 w = other_walk<D>(s, a, b, rmax_in, qi);
        L.idx = w.x;
        L.r = __int_as_float(w.y);
        L.ovf = w.x == -2;
    }
    if (L.ovf && s.err) atomicOr(s.err, GQ_DEVERR_STACK);
    const bool found = L.idx >= 0 && !L.ovf;
    if (D == 3)
        ray3_record(s.prims, L.idx, found, L.p[0], L.p[1], L.p[D - 1], L.v[0], L.v[1], L.v[D - 1], L.r, o, n, qi);
    else
        ray2_record(s.prims, L.idx, found, L.p[0], L.p[D - 1], L.v[0], L.v[D - 1], L.r, o, n, qi);
}

}  // namespace rayw
}  // namespace gqd
