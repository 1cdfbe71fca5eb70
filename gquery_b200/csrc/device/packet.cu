// Single-scene warp-coherent closest point (see packet.cuh): persistent warps take 32
// consecutive queries of the Morton order at a time.
#include <algorithm>

#include "packet.cuh"
#include "records.cuh"

namespace gqd {

namespace {

constexpr int kMaxBlock = 256;

__device__ __forceinline__ float qget(const gq_vecs &v, int64_t i, int k) {
    return v.ptr[(int64_t)k * v.comp_stride + i * v.elem_stride];
}

// Registers: 56 keep 36 warps on an SM; the form that fetches ahead is bound by latency and takes 65
// (at most 64 / 72: 2,003 points on 327,680 triangles 2.13 / 2.10 ms, 1,048,576 on 20,480 0.94 / 0.90,
// 1,048,576 on 161,920 2.75 / 2.65).
template <int D, int LAYOUT, bool MINFIRST, int STK, bool COMPACT, int FORM>
__global__ void __maxnreg__(FORM == 2 ? 72 : 56) k_cp_packet(DevScene s, gq_vecs q, int64_t n, const int32_t *perm, const int32_t *tiles,
                                                         gq_cp_out o, unsigned long long *counter) {
    const unsigned lane = threadIdx.x & 31u;
    // (ref, this lane's key) per entry; refs are the same in every lane
    int2 plain[COMPACT ? 1 : STK];
    __shared__ int refs[COMPACT ? kMaxBlock / 32 : 1][COMPACT ? STK : 1];
    __half keys[COMPACT ? STK : 1];
    pkt::PStack<COMPACT> stk = [&]() {
        if constexpr (COMPACT)
            return pkt::PStack<true>{refs[threadIdx.x >> 5], keys};
        else
            return pkt::PStack<false>(plain);
    }();
    extern __shared__ pkt::LeafBuf leaf_buf[];
    pkt::LeafBuf *buf = FORM ? leaf_buf + (threadIdx.x >> 5) : nullptr;
    for (;;) {
        unsigned long long base = 0;
        if (lane == 0) base = atomicAdd(counter, 32ull);
        base = __shfl_sync(0xffffffffu, base, 0);
        if (base >= (unsigned long long)n) break;
        const int64_t i = (tiles ? 32 * (int64_t)__ldg(tiles + base / 32) : (int64_t)base) + lane;
        const bool alive = i < n;
        const int64_t qi = alive ? (perm ? (int64_t)__ldg(perm + i) : i) : 0;
        float p[D];
#pragma unroll
        for (int k = 0; k < D; ++k) p[k] = alive ? qget(q, qi, k) : 0.f;
        float r = kInf;
        int idx = -1;
        bool ovf = false;
        pkt::closest_point<D, LAYOUT, MINFIRST, STK, COMPACT, FORM>(s, __ballot_sync(0xffffffffu, alive), p, r, idx, ovf,
                                                             stk, buf);
        if (ovf && lane == 0 && s.err) atomicOr(s.err, GQ_DEVERR_STACK);
        if (alive) {
            if (D == 3)
                cp3_record(s.prims, idx, (idx >= 0) && !ovf, p[0], p[1], p[D - 1], o, n, qi);
            else
                cp2_record(s.prims, idx, (idx >= 0) && !ovf, p[0], p[D - 1], o, n, qi);
        }
    }
    if (FORM == 2) pkt::copies_done();
}

template <int D, int LAYOUT, bool MINFIRST, int STK, bool COMPACT = false, int FORM = 0>
cudaError_t launch(const DevScene &s, const Tune &t, gq_vecs q, int64_t n, const int32_t *perm, const gq_cp_out &o,
                   unsigned long long *counter, cudaStream_t st) {
    int block = t.block, slot = block_slot(block);
    if (slot < 0) slot = 1, block = 128;
    const size_t smem = FORM ? (size_t)(block / 32) * sizeof(pkt::LeafBuf) : 0;
    static std::atomic<int> known[3] = {};
    const int64_t blocks = resident_blocks(known[slot], (const void *)k_cp_packet<D, LAYOUT, MINFIRST, STK, COMPACT, FORM>,
                                           block, smem);
    const int64_t warps = (n + 31) / 32;
    const int64_t want = std::min<int64_t>(blocks, (warps * 32 + block - 1) / block);
    cudaError_t e = cudaMemsetAsync(counter, 0, sizeof(unsigned long long), st);
    if (e != cudaSuccess) return e;
    k_cp_packet<D, LAYOUT, MINFIRST, STK, COMPACT, FORM><<<dim3((unsigned)want), block, smem, st>>>(s, q, n, perm, t.tiles, o,
                                                                                                   counter);
    return cudaGetLastError();
}

// Calls of fewer queries bring children into L1 ahead (packet.cuh): their time is the latency of
// the heaviest tiles; from here on the GPU has some fifteen tiles per resident warp and the
// form with more warps wins where it matters.  Without / with, uniform points on 1,310,720 curved
// and 200,000 scattered triangles and on a tube of 320,000 slivers: 1,048,576 8.6 / 7.6, 0.69 / 0.68 and 16.6 / 15.7
// ms, 2,097,157 9.8 / 10.2, 1.05 / 1.09 and 21.6 / 20.1, 3,000,000 11.2 / 13.3, 1.49 / 1.52 and 25.0 / 23.9,
// 4,000,000 12.3 / 14.3, 2.05 / 2.08 and 29.6 / 28.1.
// Device-built trees, one triangle per leaf, leave it out earlier: 327,680 curved and 200,000
// scattered triangles, 262,144 points 7.3 / 6.7 and 0.55 / 0.55 ms, 1,048,576 8.4 / 8.0 and 0.69 / 0.80.
// All forms give the same answers bit for bit.
// 2D (no pairs), without / with, us: 65,536 points on 4,096 / 16,384 / 65,536 segments 164 / 144, 311 / 236 and
// 905 / 624, 1,048,576 points 260 / 271, 404 / 393 and 856 / 768 (8,192 segments 305 / 313: a tree that stays in
// L1 anyway), 4,194,304 on 65,536 1,890 / 1,913.
constexpr int64_t kAheadBelow3D = 1 << 21, kAheadNoRuns = 1 << 19;
constexpr int64_t kAheadBelow2D = 1 << 21, kSmallCall2D = 1 << 16, kLargeLine = 1 << 14;

template <int D, int LAYOUT, bool MINFIRST>
cudaError_t launch_stk(const DevScene &s, const Tune &t, gq_vecs q, int64_t n, const int32_t *perm,
                       const gq_cp_out &o, unsigned long long *counter, cudaStream_t st) {
    constexpr int kForm = D == 3 ? 1 : 0;  // triangles as pairs
    if (t.packet == 2) {  // the compact stack (FP16 keys, one node word per warp)
        if (t.stack == 32) return launch<D, LAYOUT, MINFIRST, 32, true, kForm>(s, t, q, n, perm, o, counter, st);
        return launch<D, LAYOUT, MINFIRST, pkt::kPStack, true, kForm>(s, t, q, n, perm, o, counter, st);
    }
    if constexpr (LAYOUT == 0) {
        const bool ahead = D == 3 ? n < (s.has_runs ? kAheadBelow3D : kAheadNoRuns)
                                  : n < (s.n_prims >= kLargeLine ? kAheadBelow2D : kSmallCall2D);
        if (ahead)
            return t.stack == 32 ? launch<D, LAYOUT, MINFIRST, 32, false, 2>(s, t, q, n, perm, o, counter, st)
                                 : launch<D, LAYOUT, MINFIRST, pkt::kPStack, false, 2>(s, t, q, n, perm, o, counter, st);
    }
    if (t.stack == 32) return launch<D, LAYOUT, MINFIRST, 32, false, kForm>(s, t, q, n, perm, o, counter, st);
    return launch<D, LAYOUT, MINFIRST, pkt::kPStack, false, kForm>(s, t, q, n, perm, o, counter, st);
}

// Bounding cylinder of triangles [first, first + count) (gq_cyl_t), in double, rounded
// outward.  The axis is the sum of the triangles' area normals.
__device__ void cylinder_of(const gq_tri_t *prims, int64_t first, int count, gq_cyl_t &out) {
    double n[3] = {0, 0, 0}, lo[3] = {INFINITY, INFINITY, INFINITY}, hi[3] = {-INFINITY, -INFINITY, -INFINITY};
    bool ok = true;
    for (int j = 0; j < count; ++j) {
        const gq_tri_t &t = prims[first + j];
        const double v[3][3] = {{t.ax, t.ay, t.az}, {t.bx, t.by, t.bz}, {t.cx, t.cy, t.cz}};
        double e[3][3], l2[3];
        for (int k = 0; k < 3; ++k) {
            l2[k] = 0;
            for (int c = 0; c < 3; ++c) {
                e[k][c] = v[(k + 1) % 3][c] - v[k][c];
                l2[k] += e[k][c] * e[k][c];
                lo[c] = fmin(lo[c], v[k][c]);
                hi[c] = fmax(hi[c], v[k][c]);
            }
        }
        const double m[3] = {e[0][1] * e[1][2] - e[0][2] * e[1][1], e[0][2] * e[1][0] - e[0][0] * e[1][2],
                             e[0][0] * e[1][1] - e[0][1] * e[1][0]};
        const double area = sqrt(m[0] * m[0] + m[1] * m[1] + m[2] * m[2]);
        // height over the longest edge at least 1/64 of that edge
        ok = ok && area * 64.0 >= fmax(l2[0], fmax(l2[1], l2[2])) && area > 1e-36;
        for (int c = 0; c < 3; ++c) n[c] += m[c];
    }
    const double nl = sqrt(n[0] * n[0] + n[1] * n[1] + n[2] * n[2]);
    ok = ok && nl > 0.0 && nl < INFINITY;
    const float a[3] = {(float)(n[0] / nl), (float)(n[1] / nl), (float)(n[2] / nl)};
    double c0[3] = {0.5 * (lo[0] + hi[0]), 0.5 * (lo[1] + hi[1]), 0.5 * (lo[2] + hi[2])};
    double half = 0, radius = 0;
    float cf[3] = {0.f, 0.f, 0.f};
    for (int pass = 0; pass < 2; ++pass) {  // the second with the centre at mid height
        for (int c = 0; c < 3; ++c) cf[c] = (float)c0[c];
        double h0 = INFINITY, h1 = -INFINITY;
        radius = 0;
        for (int j = 0; j < count; ++j) {
            const gq_tri_t &t = prims[first + j];
            const double v[3][3] = {{t.ax, t.ay, t.az}, {t.bx, t.by, t.bz}, {t.cx, t.cy, t.cz}};
            for (int k = 0; k < 3; ++k) {
                const double e[3] = {v[k][0] - cf[0], v[k][1] - cf[1], v[k][2] - cf[2]};
                const double h = e[0] * a[0] + e[1] * a[1] + e[2] * a[2];
                double g2 = 0;
                for (int c = 0; c < 3; ++c) {
                    const double g = e[c] - h * a[c];
                    g2 += g * g;
                }
                h0 = fmin(h0, h);
                h1 = fmax(h1, h);
                radius = fmax(radius, sqrt(g2));
            }
        }
        for (int c = 0; c < 3; ++c) c0[c] = cf[c] + 0.5 * (h0 + h1) * a[c];
        half = fmax(fabs(h0), fabs(h1));
    }
    // 2^-20 of the cylinder's own size covers the rounding of the axis
    const double slack = (radius + half) * 9.5367431640625e-07;
    out.cx = cf[0];
    out.cy = cf[1];
    out.cz = cf[2];
    out.radius = ok ? __double2float_ru(radius + slack) : kInf;
    out.nx = ok ? a[0] : 0.f;
    out.ny = ok ? a[1] : 0.f;
    out.nz = ok ? a[2] : 0.f;
    out.half = ok ? __double2float_ru(half + slack) : kInf;
}

__global__ void __launch_bounds__(128) k_no_cyl(gq_cyl_t *out, int64_t n) {
    const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (i < n) out[i] = gq_cyl_t{0.f, 0.f, 0.f, kInf, 0.f, 0.f, 0.f, kInf};
}

// The walk meets the largest runs only: the two runs of a pair that is itself inside a run
// are left out (they may start at the same triangle as the run around them).
__global__ void __launch_bounds__(128) k_run_cyl(const gq_pair3_t *pairs, int64_t n, int32_t root, const gq_tri_t *prims,
                                                 int64_t n_prims, gq_cyl_t *out) {
    const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (i >= 2 * n) return;
    const uint32_t l = (uint32_t)pairs[i >> 1].sub_l, r = (uint32_t)pairs[i >> 1].sub_r;
    if (l && r && (l >> 24) + (r >> 24) <= GQ_COLLAPSE_MAX && (i >> 1) != root) return;
    const uint32_t sub = (i & 1) ? r : l;
    const int64_t first = sub & 0xffffffu, count = sub >> 24;
    if (count < 1 || first + count > n_prims) return;
    cylinder_of(prims, first, (int)count, out[first]);
}

}  // namespace

cudaError_t build_cylinders(const DevScene &s, int64_t n_pairs, gq_cyl_t *run_cyl) {
    // whatever runs the records of a file name, a place without a cylinder bounds nothing
    k_no_cyl<<<dim3((unsigned)((s.n_prims + 127) / 128)), 128>>>(run_cyl, s.n_prims);
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return e;
    if (n_pairs > 0)
        k_run_cyl<<<dim3((unsigned)((2 * n_pairs + 127) / 128)), 128>>>(
            static_cast<const gq_pair3_t *>(s.pairs), n_pairs, s.root_ref, static_cast<const gq_tri_t *>(s.prims),
            s.n_prims, run_cyl);
    return cudaGetLastError();
}

cudaError_t launch_cp_packet(const DevScene &s, int layout, const Tune &t, gq_vecs q, int64_t n,
                             const int32_t *perm, const gq_cp_out &o, unsigned long long *counter, cudaStream_t st) {
    if (n <= 0) return cudaSuccess;
    // layout: 0 binary pairs, 1 quantised 8-wide (children sorted), 2 quantised 8-wide (nearest first)
    if (s.dim == 2) return launch_stk<2, 0, false>(s, t, q, n, perm, o, counter, st);
    if (layout == 2) return launch_stk<3, 1, true>(s, t, q, n, perm, o, counter, st);
    if (layout == 1) return launch_stk<3, 1, false>(s, t, q, n, perm, o, counter, st);
    return launch_stk<3, 0, false>(s, t, q, n, perm, o, counter, st);
}

}  // namespace gqd
