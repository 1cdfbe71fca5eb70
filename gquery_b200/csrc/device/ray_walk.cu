// Persistent launch of the ray walk over the 8-wide nodes (ray_walk.cuh).
#include <algorithm>

#include "ray_walk.cuh"

namespace gqd {

namespace {

constexpr int kBlockR = 128;

// `lanes` rays at a time per warp (lanes 0 .. lanes - 1).  Rays need between one and some
// hundred steps, so lanes go their own way: a warp takes new rays when at least `refill` of its
// lanes are done (their records are written together then), and tests leaves when at
// least `leaves` lanes wait at one or no lane is at a node.  Bound by the latency of the
// node reads and of the instructions between them (one SM runs 24 warps at 80 registers: 5 /
// 6 / 8 blocks an SM 2.58 / 2.38 / 2.58 ms for 8,388,608 rays); a quarter, a half or an eighth of the lanes for
// `refill` and `leaves` are within 2%.
template <int D>
__global__ void __launch_bounds__(kBlockR, 6) k_ray_walk(DevScene s, gq_vecs a, gq_vecs b, const float *rmax_in, int64_t n,
                                                      const int32_t *perm, gq_ray_out o, unsigned long long *counter,
                                                      int lanes, int refill, int leaves) {
    const unsigned lane = threadIdx.x & 31u, below = (1u << lane) - 1u;
    const bool mine = (int)lane < lanes;
    __shared__ rayw::LeafBuf leaf_buf[kBlockR / 32];
    rayw::Stack stk;
    rayw::Lane<D> L;
    L.cur = rayw::kNone;
    int64_t qi = -1;  // the query whose record is still to be written
    bool drained = false;
    for (;;) {
        const unsigned idle = __ballot_sync(0xffffffffu, mine && L.cur == rayw::kNone);
        const int n_idle = __popc(idle);
        if (n_idle == lanes || (!drained && n_idle >= refill)) {
            if (L.cur == rayw::kNone && qi >= 0) {
                rayw::finish<D>(s, L, a, b, rmax_in, qi, n, o);
                qi = -1;
            }
            if (drained) break;  // every lane was idle
            unsigned long long base = 0;
            if (lane == 0) base = atomicAdd(counter, (unsigned long long)n_idle);
            base = __shfl_sync(0xffffffffu, base, 0);
            drained = base + n_idle >= (unsigned long long)n;
            if ((idle >> lane) & 1u) {
                const unsigned long long i = base + __popc(idle & below);
                if (i < (unsigned long long)n) {
                    qi = perm ? (int64_t)__ldg(perm + i) : (int64_t)i;
                    rayw::init<D>(s, L, a, b, rmax_in, qi);
                }
            }
            continue;
        }
        if ((unsigned)L.cur < (unsigned)rayw::kNone) rayw::node<D>(s.wnodes, L, stk);
        const unsigned at_leaf = __ballot_sync(0xffffffffu, L.cur < 0);
        if (at_leaf) {
            const unsigned at_node = __ballot_sync(0xffffffffu, (unsigned)L.cur < (unsigned)rayw::kNone);
            if (at_node == 0 || __popc(at_leaf) >= leaves) rayw::leaves<D, false>(s.prims, L, stk, leaf_buf[threadIdx.x >> 5]);
        }
    }
}

template <int D>
cudaError_t launch(const DevScene &s, gq_vecs x, gq_vecs v, const float *r_max, int64_t n, const int32_t *perm,
                   const gq_ray_out &o, unsigned long long *counter, cudaStream_t st) {
    static std::atomic<int> known{0};
    const int64_t blocks = resident_blocks(known, (const void *)k_ray_walk<D>, kBlockR, 0), warps = blocks * (kBlockR / 32);
    // fewer rays than lanes on the GPU: fewer per warp, so that they do not wait for one another
    const int lanes = (int)std::min<int64_t>(32, std::max<int64_t>(1, (n + warps - 1) / warps));
    const int refill = std::max(1, lanes / 4), leaves = std::max(1, lanes / 4);
    const int64_t want = std::min<int64_t>(blocks, ((n + lanes - 1) / lanes * 32 + kBlockR - 1) / kBlockR);
    cudaError_t e = cudaMemsetAsync(counter, 0, sizeof(unsigned long long), st);
    if (e != cudaSuccess) return e;
    k_ray_walk<D><<<dim3((unsigned)want), kBlockR, 0, st>>>(s, x, v, r_max, n, perm, o, counter, lanes, refill, leaves);
    return cudaGetLastError();
}

}  // namespace

cudaError_t launch_ray_walk(const DevScene &s, gq_vecs x, gq_vecs v, const float *r_max, int64_t n, const int32_t *perm,
                            const gq_ray_out &o, unsigned long long *counter, cudaStream_t st) {
    if (n <= 0) return cudaSuccess;
    // a tree that is one leaf has no nodes: its root is the leaf
    if ((!s.wnodes && s.wroot_ref >= 0) || !counter) return cudaErrorInvalidValue;
    return s.dim == 3 ? launch<3>(s, x, v, r_max, n, perm, o, counter, st)
                      : launch<2>(s, x, v, r_max, n, perm, o, counter, st);
}

}  // namespace gqd
