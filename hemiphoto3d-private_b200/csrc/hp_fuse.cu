// Depth-map fusion into a dense point cloud (hp_fuse_depth_maps).
//
// The reference declares the stage's consumer, fuseDepthMaps(depth_maps,
// poses, images) -> DensePointCloud (src/dense_recon/point_cloud.h:7), and
// leaves it a stub (src/dense_recon/point_cloud.cu:4-8).  The rule fused here
// is stated in include/hpmvs.h: a pixel's back-projected point is checked in
// each neighbour view for depth, reprojection and normal agreement, the mean
// of the agreeing points is emitted once, by the lowest-index view that sees
// it.
//
// The maps stay where the solve left them and neighbours are gathered straight
// from them.  The output is compacted in (view, row, column) order without
// atomics: a counting pass decides every pixel and leaves ballots and per-CTA
// numbers, one CTA scans the numbers, and a writing pass fuses the emitted
// pixels, listed so that its warps are full, at their CTA's offset.  Every
// operation is an explicitly rounded intrinsic (no contraction into FMAs the
// source does not spell out), so the CPU oracle's plain-C restatement gives the
// same bits.
//
// Both passes are bound by the latency of their dependent gathers, so the
// counting pass makes as few as decide: the lower-index neighbours first (most
// pixels are emitted by one of them, and the first that agrees settles it), the
// higher ones only until min_views agree.  Only emitted pixels are fused, and
// against the higher-index neighbours alone.  Cameras come in 16-byte loads, each
// where it is used, so 40 registers (48 warps an SM) serve with few spills.
// 8 views of 1920 x 1080, 6 neighbours, whole call: 3.30 ms with both passes
// fusing every pixel, 1.93 with these passes at 64 registers and the pixel's
// camera held, 1.85 / 1.71 / 1.67 ms with it reloaded and 4 / 5 / 6 CTAs per SM;
// 1.06 ms since the caller keeps the workspace, for repeated calls on one context
// (a context's first call allocates it: with 7 neighbours 1.38 ms, then 1.02).
#include "hp_internal.h"

namespace hp {

namespace {

struct Fused {
    float px, py, pz, nx, ny, nz, c;
};

__device__ __forceinline__ int fuse_view_of(const FuseArgs& a, int block) {
    int lo = 0, hi = a.n_views - 1;
    while (lo < hi) {  // last view whose first CTA is at or before `block`
        const int mid = (lo + hi + 1) >> 1;
        if (a.view_block[mid] <= block) lo = mid; else hi = mid - 1;
    }
    return lo;
}

// R^T (x, y, z): a camera-frame direction in the world frame.
__device__ __forceinline__ float3 rot_to_world(const float* R, float x, float y, float z) {
    return make_float3(__fmaf_rn(R[0], x, __fmaf_rn(R[3], y, __fmul_rn(R[6], z))),
                       __fmaf_rn(R[1], x, __fmaf_rn(R[4], y, __fmul_rn(R[7], z))),
                       __fmaf_rn(R[2], x, __fmaf_rn(R[5], y, __fmul_rn(R[8], z))));
}

// Pixel (fx, fy) of view v at depth d, in the world frame: R^T (d K^-1 [x y 1] - t).
__device__ __forceinline__ float3 to_world(const FuseCamera& v, float fx, float fy, float d) {
    const float* k = v.kinv;
    const float cx = __fmul_rn(d, __fmaf_rn(k[0], fx, __fmaf_rn(k[1], fy, k[2])));
    const float cy = __fmul_rn(d, __fmaf_rn(k[3], fx, __fmaf_rn(k[4], fy, k[5])));
    const float cz = __fmul_rn(d, __fmaf_rn(k[6], fx, __fmaf_rn(k[7], fy, k[8])));
    return rot_to_world(v.R, __fsub_rn(cx, v.t[0]), __fsub_rn(cy, v.t[1]), __fsub_rn(cz, v.t[2]));
}

// World point in view v's camera frame: R X + t.
__device__ __forceinline__ float3 to_camera(const FuseCamera& v, float3 X) {
    const float* R = v.R;
    return make_float3(__fmaf_rn(R[0], X.x, __fmaf_rn(R[1], X.y, __fmaf_rn(R[2], X.z, v.t[0]))),
                       __fmaf_rn(R[3], X.x, __fmaf_rn(R[4], X.y, __fmaf_rn(R[5], X.z, v.t[1]))),
                       __fmaf_rn(R[6], X.x, __fmaf_rn(R[7], X.y, __fmaf_rn(R[8], X.z, v.t[2]))));
}

// Homogeneous pixel K p of a camera-frame point.
__device__ __forceinline__ float3 to_pixel(const float* K, float3 p) {
    return make_float3(__fmaf_rn(K[0], p.x, __fmaf_rn(K[1], p.y, __fmul_rn(K[2], p.z))),
                       __fmaf_rn(K[3], p.x, __fmaf_rn(K[4], p.y, __fmul_rn(K[5], p.z))),
                       __fmaf_rn(K[6], p.x, __fmaf_rn(K[7], p.y, __fmul_rn(K[8], p.z))));
}

__device__ __forceinline__ FuseCamera load_camera(const FuseView& v) {
    static_assert(sizeof(FuseCamera) == 8 * sizeof(float4), "camera words");
    const float4* p = reinterpret_cast<const float4*>(&v.cam);
    float4 q[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) q[i] = __ldg(p + i);
    FuseCamera c;
    memcpy(&c, q, sizeof c);
    return c;
}

// A pixel's point and normal in the world frame.
struct Seen {
    float fx, fy;
    float3 X, n;
};

// Whether pixel (x, y) of view v is valid; then its point and normal.
__device__ __forceinline__ bool see(const FuseArgs& a, const FuseView& v, int x, int y, Seen* s) {
    const FuseCamera vc = load_camera(v);
    const size_t idx = static_cast<size_t>(y) * v.W + x;
    const float d = v.depth[idx];
    if (!(d > 0.0f)) return false;
    if (v.conf && !(v.conf[idx] >= a.min_conf)) return false;
    s->fx = static_cast<float>(x);
    s->fy = static_cast<float>(y);
    s->X = to_world(vc, s->fx, s->fy, d);
    s->n = rot_to_world(vc.R, v.normal[3 * idx], v.normal[3 * idx + 1], v.normal[3 * idx + 2]);
    return true;
}

// Whether neighbour w agrees with the pixel s of view v; then its own point Y
// and normal m there, and its pixel q.  v's camera is loaded again where it is
// needed rather than held in 30 registers.
__device__ __forceinline__ bool agrees(const FuseArgs& a, const FuseView& v, const Seen& s, const FuseView& w,
                                       float3* Y, float3* m, size_t* q) {
    const FuseCamera wc = load_camera(w);
    const float3 p = to_camera(wc, s.X);
    if (!(p.z > 0.0f)) return false;
    const float3 h = to_pixel(wc.K, p);
    if (!(h.z > 0.0f)) return false;
    const float u = __fdiv_rn(h.x, h.z), vv = __fdiv_rn(h.y, h.z);
    // The loose range keeps the conversion below in range (and rejects NaN).
    if (!(u >= -0.5f && u <= static_cast<float>(w.W) && vv >= -0.5f && vv <= static_cast<float>(w.H))) return false;
    const int qx = __float2int_rn(u), qy = __float2int_rn(vv);
    if (qx < 0 || qx >= w.W || qy < 0 || qy >= w.H) return false;
    *q = static_cast<size_t>(qy) * w.W + qx;
    const float dj = w.depth[*q];
    if (!(dj > 0.0f)) return false;
    if (w.conf && !(w.conf[*q] >= a.min_conf)) return false;
    if (!(fabsf(__fsub_rn(p.z, dj)) <= __fmul_rn(a.max_depth_rel, dj))) return false;
    *Y = to_world(wc, static_cast<float>(qx), static_cast<float>(qy), dj);
    const FuseCamera vc = load_camera(v);
    const float3 r = to_camera(vc, *Y);
    if (!(r.z > 0.0f)) return false;
    const float3 g = to_pixel(vc.K, r);
    if (!(g.z > 0.0f)) return false;
    const float du = __fsub_rn(__fdiv_rn(g.x, g.z), s.fx), dv = __fsub_rn(__fdiv_rn(g.y, g.z), s.fy);
    if (!(__fmaf_rn(du, du, __fmul_rn(dv, dv)) <= a.max_reproj_sq)) return false;
    *m = rot_to_world(wc.R, w.normal[3 * *q], w.normal[3 * *q + 1], w.normal[3 * *q + 2]);
    return __fmaf_rn(s.n.x, m->x, __fmaf_rn(s.n.y, m->y, __fmul_rn(s.n.z, m->z))) >= a.min_normal_cos;
}

// Whether pixel (x, y) of view i emits a point: valid, no agreeing neighbour of
// lower index (that one emits this surface point), min_views views agree.
__device__ __forceinline__ bool emits(const FuseArgs& a, int i, int x, int y) {
    const FuseView& v = a.views[i];
    Seen s;
    if (!see(a, v, x, y, &s)) return false;
    const int* nb = a.neighbors + v.nb_begin;
    const int n = v.nb_count;
    float3 Y, m;
    size_t q;
    for (int k = 0; k < n; ++k)
        if (nb[k] < i && agrees(a, v, s, a.views[nb[k]], &Y, &m, &q)) return false;
    int count = 1;
    for (int k = 0; k < n && count < a.min_views; ++k)
        if (nb[k] > i && agrees(a, v, s, a.views[nb[k]], &Y, &m, &q)) ++count;
    return count >= a.min_views;
}

// The point of an emitting pixel: means over it and its agreeing neighbours
// (all of higher index), in list order.
__device__ __forceinline__ Fused fuse_pixel(const FuseArgs& a, int i, int x, int y) {
    const FuseView& v = a.views[i];
    Seen s{};
    see(a, v, x, y, &s);
    float sx = s.X.x, sy = s.X.y, sz = s.X.z, snx = s.n.x, sny = s.n.y, snz = s.n.z;
    float sc = v.gray ? v.gray[static_cast<size_t>(y) * v.W + x] : 0.0f;
    int count = 1;
    for (int k = 0; k < v.nb_count; ++k) {
        const int j = a.neighbors[v.nb_begin + k];
        if (j < i) continue;
        const FuseView& w = a.views[j];
        float3 Y, m;
        size_t q;
        if (!agrees(a, v, s, w, &Y, &m, &q)) continue;
        sx = __fadd_rn(sx, Y.x);
        sy = __fadd_rn(sy, Y.y);
        sz = __fadd_rn(sz, Y.z);
        snx = __fadd_rn(snx, m.x);
        sny = __fadd_rn(sny, m.y);
        snz = __fadd_rn(snz, m.z);
        sc = __fadd_rn(sc, w.gray ? w.gray[q] : 0.0f);
        ++count;
    }
    Fused f;
    const float c = static_cast<float>(count);
    f.px = __fdiv_rn(sx, c);
    f.py = __fdiv_rn(sy, c);
    f.pz = __fdiv_rn(sz, c);
    const float len = __fsqrt_rn(__fmaf_rn(snx, snx, __fmaf_rn(sny, sny, __fmul_rn(snz, snz))));
    const bool unit = len > 0.0f;
    f.nx = unit ? __fdiv_rn(snx, len) : 0.0f;
    f.ny = unit ? __fdiv_rn(sny, len) : 0.0f;
    f.nz = unit ? __fdiv_rn(snz, len) : 0.0f;
    f.c = __fdiv_rn(sc, c);
    return f;
}

constexpr int STEP_WORDS = FUSE_THREADS / 32;  // ballot words per step

__global__ void __launch_bounds__(FUSE_THREADS, FUSE_BLOCKS) fuse_count_kernel(FuseArgs a, unsigned* ballots,
                                                                               int* block_counts) {
    const int i = fuse_view_of(a, blockIdx.x);
    const int W = a.views[i].W;
    const long long px = static_cast<long long>(W) * a.views[i].H;
    const long long first = static_cast<long long>(blockIdx.x - a.view_block[i]) * a.steps * FUSE_THREADS +
                            threadIdx.x;
    int n = 0;
#pragma unroll 1
    for (int step = 0; step < a.steps; ++step) {
        const long long p = first + step * FUSE_THREADS;
        bool emit = false;
        if (p < px) {
            const int y = static_cast<int>(p / W);
            emit = emits(a, i, static_cast<int>(p - static_cast<long long>(y) * W), y);
        }
        const unsigned votes = __ballot_sync(0xffffffffu, emit);
        if ((threadIdx.x & 31) == 0)
            ballots[(static_cast<size_t>(blockIdx.x) * a.steps + step) * STEP_WORDS + (threadIdx.x >> 5)] = votes;
        n += emit;
    }
    __shared__ int total;
    if (threadIdx.x == 0) total = 0;
    __syncthreads();
    n = __reduce_add_sync(0xffffffffu, n);
    if ((threadIdx.x & 31) == 0) atomicAdd(&total, n);
    __syncthreads();
    if (threadIdx.x == 0) block_counts[blockIdx.x] = total;
}

// One CTA: exclusive prefix of the per-CTA counts, and their total.
// Tiles of SCAN_TILE counts: coalesced loads kept in flight together, then a
// scan of each tile in turn.
constexpr int SCAN_THREADS = 1024, SCAN_PER = 8, SCAN_TILE = SCAN_THREADS * SCAN_PER;
__global__ void __launch_bounds__(SCAN_THREADS) fuse_scan_kernel(const int* counts, int n, long long* offsets,
                                                                 long long* total) {
    __shared__ long long warp_sum[SCAN_PER][SCAN_THREADS / 32];
    const int t = threadIdx.x, lane = t & 31, w = t >> 5;
    long long run = 0;
    for (int base = 0; base < n; base += SCAN_TILE) {
        int own[SCAN_PER];
        long long incl[SCAN_PER];
#pragma unroll
        for (int r = 0; r < SCAN_PER; ++r) {
            const int k = base + r * SCAN_THREADS + t;
            own[r] = k < n ? counts[k] : 0;
        }
#pragma unroll
        for (int r = 0; r < SCAN_PER; ++r) {
            long long s = own[r];
            for (int o = 1; o < 32; o <<= 1) {
                const long long add = __shfl_up_sync(0xffffffffu, s, o);
                if (lane >= o) s += add;
            }
            incl[r] = s;
            if (lane == 31) warp_sum[r][w] = s;
        }
        __syncthreads();
        if (w < SCAN_PER) {  // warp r: inclusive scan of row r's warp sums
            long long s = warp_sum[w][lane];
            for (int o = 1; o < 32; o <<= 1) {
                const long long add = __shfl_up_sync(0xffffffffu, s, o);
                if (lane >= o) s += add;
            }
            warp_sum[w][lane] = s;
        }
        __syncthreads();
#pragma unroll
        for (int r = 0; r < SCAN_PER; ++r) {
            const int k = base + r * SCAN_THREADS + t;
            if (k < n) offsets[k] = run + (w > 0 ? warp_sum[r][w - 1] : 0) + incl[r] - own[r];
            run += warp_sum[r][SCAN_THREADS / 32 - 1];
        }
        __syncthreads();
    }
    if (t == 0) *total = run;
}

__global__ void __launch_bounds__(FUSE_THREADS, FUSE_BLOCKS) fuse_write_kernel(
    FuseArgs a, const unsigned* ballots, const long long* offsets, float* positions, float* normals, float* colors,
    long long capacity) {
    __shared__ unsigned short list[FUSE_STEPS * FUSE_THREADS];  // the CTA's emitted pixels in order
    __shared__ int listed;
    const long long base = offsets[blockIdx.x];
    if (threadIdx.x < 32) {  // one ballot word a lane
        static_assert(FUSE_STEPS * STEP_WORDS == 32, "one word a lane");
        const int words = a.steps * STEP_WORDS;
        unsigned word =
            threadIdx.x < words ? ballots[static_cast<size_t>(blockIdx.x) * words + threadIdx.x] : 0u;
        int at = __popc(word);
        for (int o = 1; o < 32; o <<= 1) {
            const int add = __shfl_up_sync(0xffffffffu, at, o);
            if (threadIdx.x >= o) at += add;
        }
        if (threadIdx.x == 31) listed = at;
        at -= __popc(word);
        for (; word; word &= word - 1) list[at++] = static_cast<unsigned short>(threadIdx.x * 32 + __ffs(word) - 1);
    }
    __syncthreads();
    const int i = fuse_view_of(a, blockIdx.x);
    const int W = a.views[i].W;
    const long long first = static_cast<long long>(blockIdx.x - a.view_block[i]) * a.steps * FUSE_THREADS;
    for (int k = threadIdx.x; k < listed; k += FUSE_THREADS) {
        const long long o = base + k;
        if (o >= capacity) break;
        const long long p = first + list[k];
        const int y = static_cast<int>(p / W);
        const Fused f = fuse_pixel(a, i, static_cast<int>(p - static_cast<long long>(y) * W), y);
        if (positions) {
            positions[3 * o] = f.px;
            positions[3 * o + 1] = f.py;
            positions[3 * o + 2] = f.pz;
        }
        if (normals) {
            normals[3 * o] = f.nx;
            normals[3 * o + 1] = f.ny;
            normals[3 * o + 2] = f.nz;
        }
        if (colors) {
            colors[3 * o] = f.c;
            colors[3 * o + 1] = f.c;
            colors[3 * o + 2] = f.c;
        }
    }
}

}  // namespace

cudaError_t launch_fuse_count(const FuseArgs& a, int blocks, unsigned* ballots, int* block_counts, cudaStream_t st) {
    if (blocks <= 0) return cudaSuccess;
    fuse_count_kernel<<<blocks, FUSE_THREADS, 0, st>>>(a, ballots, block_counts);
    return cudaGetLastError();
}

cudaError_t launch_fuse_scan(const int* block_counts, int blocks, long long* block_offsets, long long* total,
                             cudaStream_t st) {
    fuse_scan_kernel<<<1, SCAN_THREADS, 0, st>>>(block_counts, blocks, block_offsets, total);
    return cudaGetLastError();
}

cudaError_t launch_fuse_write(const FuseArgs& a, int blocks, const unsigned* ballots,
                              const long long* block_offsets, float* positions, float* normals, float* colors,
                              long long capacity, cudaStream_t st) {
    if (blocks <= 0) return cudaSuccess;
    fuse_write_kernel<<<blocks, FUSE_THREADS, 0, st>>>(a, ballots, block_offsets, positions, normals, colors, capacity);
    return cudaGetLastError();
}

}  // namespace hp
