// Closest points of a handful of queries (fewer than a warp-coherent tile holds): one
// query per warp, up to 32 nodes of its tree at a time, with the answers of the per-lane
// walk in the reference's order (traverse.cuh) bit for bit.
//
// A lone lane reads some 300 nodes one after another; here the warp expands its stack's top 32 entries per step, a few
// tens of steps in all.  The reference keeps the first of several primitives at the same
// distance, in its depth-first order, nearer child first.  That order is a property of the
// query and the tree: two leaves are visited in the order of the children they lie under at
// their lowest common ancestor, whichever boxes are pruned elsewhere.  So every entry
// carries its path (one bit per level, 0 = the child visited first), and among equal
// distances the smallest path wins.
//
// Pruning keeps every box within eps (2^-19 of the coordinates' size) of the radius, so all
// candidates for the minimum are met.  Where the reference's own pruning could have
// decided otherwise by a rounding (a box's farthest point within eps of the answer, or a
// leaf box farther than its primitive), the query is walked again in the plain order.  A
// query so far away that eps spans the scene, or without a finite distance, ends up there
// as soon as that shows: no answer is nearer than the root box (16 points a million radii from
// 327,680 triangles 15.9 -> 0.62 ms).
#include <algorithm>

#include "prim.cuh"
#include "queries.cuh"
#include "records.cuh"
#include "traverse.cuh"

namespace gqd {

namespace {

constexpr int kStackF = 512;                       // entries per warp
constexpr int kReserveF = 2 * GQ_STACK_EXACT + 2;  // room for a depth-first descent (sil_warp.cuh)

struct Entry {
    int ref;
    float key;
    unsigned long long path;  // the levels' bits from the top, then a one, then zeros (depth at most 63)
};

template <int D>
__device__ __forceinline__ float item_dist(const DevScene &s, int j, const float *p, bool &last) {
    if (D == 3) {
        const float4 t0 = ldg4(s.prims, 3 * (int64_t)j), t1 = ldg4(s.prims, 3 * (int64_t)j + 1),
                     t2 = ldg4(s.prims, 3 * (int64_t)j + 2);
        last = (fbits(t2.z) & GQ_ITEM_LAST) != 0;
        return tri_closest<false>(p[0], p[1], p[D - 1], t0.x, t0.y, t0.z, t0.w, t1.x, t1.y, t1.z, t1.w, t2.x);
    }
    const float4 a = ldg4(s.prims, 2 * (int64_t)j);
    last = (__ldg(reinterpret_cast<const int4 *>(s.prims) + 2 * (int64_t)j + 1).y & GQ_ITEM_LAST) != 0;
    return seg_dist(p[0], p[D - 1], a.x, a.y, a.z, a.w);
}

template <int D>
__device__ __noinline__ void plain_walk(const DevScene &s, const gq_vecs &q, int64_t qi, int64_t n, const gq_cp_out &o) {
    trav::Stack<false> stk;
    trav::Lane<D, false, false> L;
    trav::lane_init(s, L, q, q, nullptr, qi);
    while (!trav::lane_run<D, false, false, 0>(s, L, stk, 1 << 30)) {
    }
    trav::lane_write(s, L, qi, n, o, gq_ray_out{});
}

template <int D>
__global__ void __launch_bounds__(32) k_cp_few(DevScene s, gq_vecs q, int64_t n, gq_cp_out o) {
    __shared__ Entry stk[kStackF];
    const unsigned lane = threadIdx.x;
    const unsigned above = ~((2u << lane) - 1u);  // lanes with a higher index
    const int64_t qi = blockIdx.x;
    float p[D], pmax = 0.f;
#pragma unroll
    for (int k = 0; k < D; ++k) {
        p[k] = trav::qget(q, qi, k);
        pmax = fmaxf(pmax, fabsf(p[k]));
    }
    const float eps = (pmax + s.coord_bound) * 1.9073486e-06f;  // 2^-19
    float best = kInf;             // smallest distance this lane has seen,
    int idx = -1;                  // its primitive
    unsigned long long path = ~0ull;  // and that one's place in the reference's order
    bool odd = false;              // a leaf box farther than that primitive
    float far = kInf;              // smallest farthest-point distance of any box
    float sure;                    // an answer may stand only while that is above this
    {
        float dmin, dmax, sum = 0.f;
        if (D == 3)
            box_dist3(s.root_lo[0], s.root_lo[1], s.root_lo[2], s.root_hi[0], s.root_hi[1], s.root_hi[2], p[0], p[1],
                      p[D - 1], dmin, dmax);
        else
            box_dist2(s.root_lo[0], s.root_lo[1], s.root_hi[0], s.root_hi[1], p[0], p[D - 1], dmin, dmax);
#pragma unroll
        for (int k = 0; k < D; ++k) sum += p[k];
        sure = sum == sum ? dmin + eps : kInf;  // a NaN is ignored by the box tests
    }
    float R = kInf;                // the warp's radius
    int sp = 1;
    if (lane == 0) stk[0] = Entry{s.root_ref, 0.f, 1ull << 63};
    __syncwarp();
    bool full = false;  // left to the plain walk
    while (sp > 0) {
        if (__any_sync(0xffffffffu, !(far > sure))) {
            full = true;
            break;
        }
        const int take = (sp + 32 <= kStackF - kReserveF) ? min(sp, 32) : 1;
        const bool mine = (int)lane < take;
        Entry e{0, 0.f, 0ull};
        if (mine) e = stk[sp - 1 - (int)lane];
        __syncwarp();
        sp -= take;
        Entry e0{0, 0.f, 0ull}, e1{0, 0.f, 0ull};  // pushed by this lane, e1 on top
        int np = 0;
        float r = R;
        if (mine && !(e.key > R + eps)) {
            if (e.ref < 0) {
                for (int j = ~e.ref;; ++j) {
                    bool last;
                    const float key = item_dist<D>(s, j, p, last);
                    if (key < best || (key == best && e.path < path)) {
                        odd = (key == best && odd) | (e.key > key);
                        best = key;
                        idx = j;
                        path = e.path;
                    } else if (key == best) {
                        odd |= e.key > key;
                    }
                    r = fminf(r, key);
                    if (last) break;
                }
            } else {
                float lo[2][D], hi[2][D];
                int rl, rr;
                if (D == 3) {
                    const float4 a = ldg4(s.pairs, 4 * (int64_t)e.ref), b = ldg4(s.pairs, 4 * (int64_t)e.ref + 1),
                                 c = ldg4(s.pairs, 4 * (int64_t)e.ref + 2);
                    const int4 rf = __ldg(reinterpret_cast<const int4 *>(s.pairs) + 4 * (int64_t)e.ref + 3);
                    lo[0][0] = a.x; lo[0][1] = a.y; lo[0][D - 1] = a.z;
                    hi[0][0] = a.w; hi[0][1] = b.x; hi[0][D - 1] = b.y;
                    lo[1][0] = b.z; lo[1][1] = b.w; lo[1][D - 1] = c.x;
                    hi[1][0] = c.y; hi[1][1] = c.z; hi[1][D - 1] = c.w;
                    rl = rf.x;
                    rr = rf.y;
                } else {
                    const float4 a = ldg4(s.pairs, 3 * (int64_t)e.ref), b = ldg4(s.pairs, 3 * (int64_t)e.ref + 1);
                    const int4 rf = __ldg(reinterpret_cast<const int4 *>(s.pairs) + 3 * (int64_t)e.ref + 2);
                    lo[0][0] = a.x; lo[0][D - 1] = a.y; hi[0][0] = a.z; hi[0][D - 1] = a.w;
                    lo[1][0] = b.x; lo[1][D - 1] = b.y; hi[1][0] = b.z; hi[1][D - 1] = b.w;
                    rl = rf.x;
                    rr = rf.y;
                }
                bool h0, h1;
                float k0, k1, f = kInf;  // f: the smaller farthest-point distance
                trav::child_cp<D, 0>(lo[0], hi[0], p, f, h0, k0);
                trav::child_cp<D, 0>(lo[1], hi[1], p, f, h1, k1);
                far = fminf(far, f);
                r = fminf(r, f);
                h0 = !(k0 > r + eps);
                h1 = !(k1 > r + eps);
                // the reference visits the left child first unless the right one is nearer
                const bool sw = k1 < k0;
                const unsigned long long mark = e.path & (0ull - e.path);
                const Entry first{sw ? rr : rl, sw ? k1 : k0, (e.path ^ mark) | mark >> 1};
                const Entry second{sw ? rl : rr, sw ? k0 : k1, e.path | mark >> 1};
                const bool hf = sw ? h1 : h0, hs = sw ? h0 : h1;
                np = (int)hf + (int)hs;
                e0 = hs ? second : first;
                e1 = first;
            }
        }
        R = __uint_as_float(__reduce_min_sync(0xffffffffu, __float_as_uint(r)));
        const unsigned has1 = __ballot_sync(0xffffffffu, np >= 1), has2 = __ballot_sync(0xffffffffu, np >= 2);
        const int before = __popc(has1 & above) + __popc(has2 & above), total = __popc(has1) + __popc(has2);
        if (sp + total > kStackF) {
            full = true;
            break;
        }
        if (np >= 1) stk[sp + before] = e0;
        if (np >= 2) stk[sp + before + 1] = e1;
        __syncwarp();
        sp += total;
    }
    // the smallest distance, and among its holders the smallest path
    const float m = __uint_as_float(__reduce_min_sync(0xffffffffu, __float_as_uint(best)));
    const bool at = best == m;
    const unsigned hi32 = at ? (unsigned)(path >> 32) : ~0u;
    const unsigned mh = __reduce_min_sync(0xffffffffu, hi32);
    const unsigned lo32 = at && hi32 == mh ? (unsigned)path : ~0u;
    const unsigned ml = __reduce_min_sync(0xffffffffu, lo32);
    const unsigned who = __ballot_sync(0xffffffffu, at && hi32 == mh && (unsigned)path == ml);
    const float fm = __uint_as_float(__reduce_min_sync(0xffffffffu, __float_as_uint(far)));
    const bool unsure = __any_sync(0xffffffffu, at && odd) || full || !(m < kInf) || !(fm > m + eps);
    if (unsure) {
        if (lane == 0) plain_walk<D>(s, q, qi, n, o);
    } else if (lane == (unsigned)(__ffs(who) - 1)) {
        if (D == 3)
            cp3_record(s.prims, idx, true, p[0], p[1], p[D - 1], o, n, qi);
        else
            cp2_record(s.prims, idx, true, p[0], p[D - 1], o, n, qi);
    }
}

}  // namespace

cudaError_t launch_cp_few(const DevScene &s, gq_vecs q, int64_t n, const gq_cp_out &o, cudaStream_t st) {
    if (n <= 0) return cudaSuccess;
    if (s.dim == 3)
        k_cp_few<3><<<dim3((unsigned)n), 32, 0, st>>>(s, q, n, o);
    else
        k_cp_few<2><<<dim3((unsigned)n), 32, 0, st>>>(s, q, n, o);
    return cudaGetLastError();
}

}  // namespace gqd
