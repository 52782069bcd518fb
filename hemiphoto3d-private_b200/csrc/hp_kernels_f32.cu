// Plain FP32 PatchMatch kernels for sm_100a: hypothesis initialisation, full-map
// NCC cost, and the fused red-black propagate + refine pass.
//
// Parity contract.  The reference's cost (computePixelCost,
// src/dense_recon/patchmatch_mvs.cu:222-343) samples sources through the
// texture unit's linear filter, whose weights carry only 8 fractional bits; a
// warped coordinate that moves by one ulp can flip a weight by 1/256 and the
// cost by ~1e-5.  To hold the 1e-5 bound this file reproduces the reference's
// per-tap rounding exactly - the operation sequence its --use_fast_math build
// executes, pinned with explicitly rounded intrinsics (see cost_f32) - and
// samples sources with tex2D on the same filter configuration; the per-pixel
// plane setup and the NCC finalisation keep the reference's expressions in a
// translation unit built with the same flags.  The result is bit-identical to
// the reference's compute_ncc_cost_kernel.  Everything around the arithmetic
// is this engine's own: packed float4 hypotheses, a shared-memory reference
// tile, red-black compaction (every thread owns a pixel of the active color),
// row-batched texture fetches, duplicate-candidate elimination, batched
// multi-view launches and counter-based RNG.  Engine-defined arithmetic
// outside the taps (initialisation, refinement) uses explicitly rounded
// intrinsics so the CPU restatement reproduces it bit for bit.
#include "hp_internal.h"
#include "hp_rng.cuh"
#include "hp_filter.cuh"
#include "hp_pass.cuh"
#include "hp_tile.cuh"

namespace hp {

#ifdef HP_COUNT_TAPS
// Instrumented builds only (make count): taps sampled.
__device__ unsigned long long g_taps32;
unsigned long long f32_taps() {
    unsigned long long v = 0, z = 0;
    cudaDeviceSynchronize();
    cudaMemcpyFromSymbol(&v, g_taps32, sizeof v);
    cudaMemcpyToSymbol(g_taps32, &z, sizeof z);
    return v;
}
#endif

namespace {

// Resident CTAs per SM the half-pass is register-budgeted for.  A window row's
// fetches are in flight together, so up to 8 taps a row 64 registers hold them
// (2 x 1920 x 1080, r 7, s 2: 97.9 ms, against 99.9 with 3 CTAs and 108.8 with
// 2); longer rows want 80 (5 x 640 x 480, r 5, s 1: 45.9 ms with 3 or 4, 48.3
// with 2; one 320 x 240 view 1247, 1276 and 1262 us with 3, 4 and 2).
// Launches with at most three CTAs for an SM have nothing to gain from a fourth
// (253 x 175, r 3 s 1, 3 sources, 6 iterations 664 -> 639 us; r 1 s 1, 1 source 260
// -> 254), and whole items (PassForm::WHOLE) spill at 64 registers (573 x 303, r 1
// s 1, 1 source 353 -> 342 us).
template <int R, int ST, PassForm F>
constexpr int pass_blocks() {
    return F == PassForm::ROOMY || F == PassForm::WHOLE || (2 * R) / ST + 1 > 8 ? 3 : 4;
}
// Persistent launches of few tiles take two CTAs an SM: beyond the tiles that can run at
// a time, CTAs wait on dependencies where others would run, and a CTA that runs has the
// registers.  With many tiles all of pass_blocks() pay, from 4 tiles an SM (of all views
// together) for rows of up to 8 taps, from 8 for longer ones.  2 CTAs -> pass_blocks():
//  r 7 s 2, 6 sources, 5 iterations: 3 x 320 x 240 (3.0 tiles an SM) 2860 -> 3428 us, 3 x
//   457 x 279 (5.7) 4928 -> 4475, 4 x 1920 x 1080 (109) 116.3 -> 103.7 ms;
//  r 5 s 1, 4 sources: 5.7 tiles an SM 5446 -> 5468 us, 8.9 8784 -> 8611, 109 133.4 -> 128.0 ms;
//  r 3 s 2, 3 sources (items whole): 1.0 486 -> 705 us, 3.0 660 -> 595, 109 25.3 -> 20.3 ms.
template <int R, int ST>
constexpr int many_tiles() { return (2 * R) / ST + 1 <= 8 ? 4 : 8; }
template <int R, int ST, PassForm F, bool MANY>
constexpr int persistent_blocks() { return MANY ? pass_blocks<R, ST, F>() : 2; }
constexpr int COST_BLOCKS = 3;  // full-map cost, 1920 x 1080, r 5, s 1: 1486 us, 1574 with 2, 1506 with 4

// Locate the view and tile of this CTA in a batch launch.
__device__ __forceinline__ const ViewDesc* locate_tile(const BatchList& bl, int t, int* tx, int* ty) {
    int lo = 0, hi = bl.n_active - 1;
    while (lo < hi) {  // last k with tile_prefix[k] <= t
        int mid = (lo + hi + 1) >> 1;
        if (bl.tile_prefix[mid] <= t) lo = mid; else hi = mid - 1;
    }
    const ViewDesc* v = &bl.views[bl.active[lo]];
    int local = t - bl.tile_prefix[lo];
    *tx = local % v->tiles_x;
    *ty = local / v->tiles_x;
    return v;
}

// Reference window source: rows [y0-r, y0+TILE_H+r), cols [x0-r, x0+TILE_W+r),
// clamped to the image edge like the reference's clamp-addressed texel fetches
// (patchmatch_mvs.cu:275-276, :371-380).
__device__ __forceinline__ void load_ref_tile(float* s_ref, int tw, int th, const ViewDesc* v, int x0, int y0,
                                              int r) {
    const int W = v->W, H = v->H;
    for (int i = threadIdx.x; i < tw * th; i += CTA_THREADS) {
        int ty = i / tw, tx = i - ty * tw;
        int gx = min(max(x0 - r + tx, 0), W - 1);
        int gy = min(max(y0 - r + ty, 0), H - 1);
        s_ref[i] = __ldg(v->ref + static_cast<size_t>(gy) * v->ref_pitch + gx);
    }
}

// Approximate reciprocal (PTX rcp.approx.ftz.f32): the instruction the
// reference's fast-math build uses for 1.0f / w_z.
__device__ __forceinline__ float rcp_approx(float x) {
    float r;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r;
}

// Cost of hypothesis (d, n) at pixel (x, y): per-source NCC over the window,
// top_k lowest of (1 - NCC) averaged (computePixelCost, :222-343).  plane_f32
// prepares the hypothesis once; cost_f32 is one source's 1 - NCC.
//
// Per tap the warp arithmetic is pinned with explicitly rounded intrinsics to
// the operation sequence the reference compiles to (found by a bit-exact
// search against its kernels on B200):
//   q = fma(a0, x, a1*y) + a2,  f = s * inv(n.P),  w_z = fma(b2, f, q_z),
//   u = fma(b0, f, q_x) * rcp(w_z),  sums accumulated with fma in tap order.
// Because nothing is left to the compiler's reassociation, the taps can be
// restructured for throughput: each window row issues all its texture
// fetches before consuming any (SIDE fetches in flight per thread), the
// row-invariant products a1*y are computed once per row (the same rounded
// value), and samples are accumulated in tap order, skipping invalid taps
// exactly as the reference's `continue`s do.
// Sums of the reference window and of its squares in tap order: what the taps
// of any source add up to when all of them are valid.
template <int R, int ST>
__device__ __forceinline__ float2 window_sums(const float* __restrict__ s_ref, int tw, int lx, int ly) {
    constexpr int SIDE = (2 * R) / ST + 1;
    float sum = 0.0f, sum2 = 0.0f;
#pragma unroll 1
    for (int i = 0; i < SIDE; ++i)
#pragma unroll
        for (int j = 0; j < SIDE; ++j) {
            const float rv = s_ref[(ly + i * ST) * tw + lx + j * ST];
            sum = __fadd_rn(sum, rv);
            sum2 = __fmaf_rn(rv, rv, sum2);
        }
    return make_float2(sum, sum2);
}

struct PlaneF32 {
    float nK0, nK1, nK2;  // K^-T n
    float inv_n_dot_P;
    bool ok;              // false: |n.P| < 1e-8, every cost is 2
};

// Plane through P = d K^-1 [x y 1] with normal n.
__device__ __forceinline__ PlaneF32 plane_f32(const ViewDesc* __restrict__ v, int x, int y, float4 h) {
    const float d = h.x, cnx = h.y, cny = h.z, cnz = h.w;
    const float ki0 = v->kinv[0], ki1 = v->kinv[1], ki2 = v->kinv[2];
    const float ki3 = v->kinv[3], ki4 = v->kinv[4], ki5 = v->kinv[5];
    const float ki6 = v->kinv[6], ki7 = v->kinv[7], ki8 = v->kinv[8];
    const float fx = static_cast<float>(x);
    const float fy = static_cast<float>(y);
    PlaneF32 p{0.f, 0.f, 0.f, 0.f, false};
    const float Px = d * (ki0 * fx + ki1 * fy + ki2);
    const float Py = d * (ki3 * fx + ki4 * fy + ki5);
    const float Pz = d * (ki6 * fx + ki7 * fy + ki8);
    const float n_dot_P = cnx * Px + cny * Py + cnz * Pz;
    if (fabsf(n_dot_P) < 1e-8f) return p;
    p.inv_n_dot_P = 1.0f / n_dot_P;
    p.nK0 = ki0 * cnx + ki3 * cny + ki6 * cnz;
    p.nK1 = ki1 * cnx + ki4 * cny + ki7 * cnz;
    p.nK2 = ki2 * cnx + ki5 * cny + ki8 * cnz;
    p.ok = true;
    return p;
}

// Cost of source s under the plane p at pixel (x, y), tile position (lx, ly).
template <int R, int ST>
__device__ __forceinline__ float cost_f32(const float* __restrict__ s_ref, int tw, int lx, int ly, int x, int y,
                                          const PlaneF32& p, float2 ref_sums, const ViewDesc* __restrict__ v,
                                          int s) {
    constexpr unsigned WARP = 0xffffffffu;
    constexpr int SIDE = (2 * R) / ST + 1;
    constexpr int min_count = (SIDE * SIDE) / 2;
    const float nK0 = p.nK0, nK1 = p.nK1, nK2 = p.nK2, inv_n_dot_P = p.ok ? p.inv_n_dot_P : 0.0f;
    const float fx = static_cast<float>(x);
    const float fy = static_cast<float>(y);
    const float fw1 = static_cast<float>(v->W) - 1.0f;
    const float fh1 = static_cast<float>(v->H) - 1.0f;
    const float* A = v->ab[s];
    const float a0 = A[0], a1 = A[1], a2 = A[2], a3 = A[3], a4 = A[4], a5 = A[5];
    const float a6 = A[6], a7 = A[7], a8 = A[8], b0 = A[9], b1 = A[10], b2 = A[11];
    const cudaTextureObject_t tex = v->src_tex[s];
    float sum_ref = 0.0f, sum_src = 0.0f, sum_ref2 = 0.0f, sum_src2 = 0.0f, sum_rs = 0.0f;
    int count = 0;
    // Two decisions from the window's corners under the plane-induced
    // homography H = A + b (K^-T n)^T / (n.P); in front of the camera
    // (w_z > 1e-6) the warped window is the convex quad of its corners.
    // Wholly beyond one edge of the source by 0.25 px: no valid tap, so the
    // reference's count rule gives 2 and no tap is sampled.  Wholly inside by
    // 0.25 px: every tap is valid, and needs no test of its own.  The margin
    // covers the rounding differences between this and the per-tap arithmetic
    // below for the second decision while 16 roundings of the largest partial
    // sums of either (Mx = |A| and |b| |m| terms over the window, likewise My,
    // Mz), at most (Mx + |u| Mz) 2^-20 / w_z, stay under 0.2 px; |u| and |v|
    // are below the image's sides there.
    bool inside, sampled = p.ok;
    {
        const float m0 = nK0 * inv_n_dot_P, m1 = nK1 * inv_n_dot_P, m2 = nK2 * inv_n_dot_P;
        const float hz0 = fmaf(b2, m0, a6), hz1 = fmaf(b2, m1, a7), hz2 = fmaf(b2, m2, a8);
        const float hx0 = fmaf(b0, m0, a0), hx1 = fmaf(b0, m1, a1), hx2 = fmaf(b0, m2, a2);
        const float hy0 = fmaf(b1, m0, a3), hy1 = fmaf(b1, m1, a4), hy2 = fmaf(b1, m2, a5);
        bool left = true, right = true, top_ = true, bottom = true;
        float in = 1e30f, zmin = 1e30f;
#pragma unroll
        for (int c = 0; c < 4; ++c) {
            const float px = fx + static_cast<float>((c & 1) ? (SIDE - 1) * ST - R : -R);
            const float py = fy + static_cast<float>((c & 2) ? (SIDE - 1) * ST - R : -R);
            const float wz = fmaf(hz0, px, fmaf(hz1, py, hz2));
            const float wx = fmaf(hx0, px, fmaf(hx1, py, hx2));
            const float wy = fmaf(hy0, px, fmaf(hy1, py, hy2));
            zmin = fminf(zmin, wz);
            left = left && wx < -0.25f * wz;
            right = right && wx >= (fw1 + 0.25f) * wz;
            top_ = top_ && wy < -0.25f * wz;
            bottom = bottom && wy >= (fh1 + 0.25f) * wz;
            in = fminf(in, fminf(fminf(fmaf(-0.25f, wz, wx), fmaf(fw1 - 0.25f, wz, -wx)),
                                 fminf(fmaf(-0.25f, wz, wy), fmaf(fh1 - 0.25f, wz, -wy))));
        }
        const bool front = zmin > 1e-6f;
        if (front && (left || right || top_ || bottom)) sampled = false;
        const float X = fabsf(fx) + static_cast<float>(SIDE * ST), Y = fabsf(fy) + static_cast<float>(SIDE * ST);
        const float Ms = fmaf(fabsf(m0), X, fmaf(fabsf(m1), Y, fabsf(m2)));
        const float Mx = fmaf(fabsf(b0), Ms, fmaf(fabsf(a0), X, fmaf(fabsf(a1), Y, fabsf(a2))));
        const float My = fmaf(fabsf(b1), Ms, fmaf(fabsf(a3), X, fmaf(fabsf(a4), Y, fabsf(a5))));
        const float Mz = fmaf(fabsf(b2), Ms, fmaf(fabsf(a6), X, fmaf(fabsf(a7), Y, fabsf(a8))));
        // Not-a-numbers fail: `in` ignores them, the bound does not.
        inside = front && in > 0.0f && fmaf(fw1, Mz, Mx) <= 2e5f * zmin && fmaf(fh1, Mz, My) <= 2e5f * zmin;
    }
    // The vote is the last step that needs the whole warp.  A lane without a
    // window to sample (wholly outside, no plane, past the last item or the
    // image) leaves here: while it ran along until the warp's last sampling lane
    // was done, its fetches took the texture unit's time (1921 x 1081, 6 sources,
    // cost of random planes: r 5 s 1 4166 -> 3991 us, r 7 s 2 2234 -> 2147; solve
    // of 2 x 1920 x 1080, r 7, s 2: 93.9 -> 90.8 ms).
    const bool all_inside = __all_sync(WARP, inside || !sampled);
    if (!sampled) return 2.0f;
#ifdef HP_COUNT_TAPS
    atomicAdd(&g_taps32, static_cast<unsigned long long>(SIDE * SIDE));
#endif
    if (all_inside) {
        // Every tap of every sampled lane is valid: no tests, and the reference
        // sums are the window's own.  The same operations on the same values
        // as below, so the same bits.
        sum_ref = ref_sums.x;
        sum_ref2 = ref_sums.y;
        count = SIDE * SIDE;
#pragma unroll 1
        for (int i = 0; i < SIDE; ++i) {
            const float wpy = fy + static_cast<float>(i * ST - R);
            const float tqx = __fmul_rn(a1, wpy), tqy = __fmul_rn(a4, wpy), tqz = __fmul_rn(a7, wpy);
            const float tsv = __fmul_rn(nK1, wpy);
            float smp[SIDE];
#pragma unroll
            for (int j = 0; j < SIDE; ++j) {
                const float wpx = fx + static_cast<float>(j * ST - R);
                const float qx = __fadd_rn(__fmaf_rn(a0, wpx, tqx), a2);
                const float qy = __fadd_rn(__fmaf_rn(a3, wpx, tqy), a5);
                const float qz = __fadd_rn(__fmaf_rn(a6, wpx, tqz), a8);
                const float sval = __fadd_rn(__fmaf_rn(nK0, wpx, tsv), nK2);
                const float factor = __fmul_rn(sval, inv_n_dot_P);
                const float wz = __fmaf_rn(b2, factor, qz);
                const float iw = rcp_approx(wz);
                const float u = __fmul_rn(__fmaf_rn(b0, factor, qx), iw);
                const float vv = __fmul_rn(__fmaf_rn(b1, factor, qy), iw);
                smp[j] = tex2D<float>(tex, __fadd_rn(u, 0.5f), __fadd_rn(vv, 0.5f));
            }
            const float* rrow = s_ref + (ly + i * ST) * tw + lx;
#pragma unroll
            for (int j = 0; j < SIDE; ++j) {
                const float rv = rrow[j * ST], sv = smp[j];
                sum_src = __fadd_rn(sum_src, sv);
                sum_src2 = __fmaf_rn(sv, sv, sum_src2);
                sum_rs = __fmaf_rn(rv, sv, sum_rs);
            }
        }
    } else {
#pragma unroll 1
        for (int i = 0; i < SIDE; ++i) {
            const float wpy = fy + static_cast<float>(i * ST - R);
            const float tqx = __fmul_rn(a1, wpy), tqy = __fmul_rn(a4, wpy), tqz = __fmul_rn(a7, wpy);
            const float tsv = __fmul_rn(nK1, wpy);
            float smp[SIDE];
            unsigned ok = 0;
#pragma unroll
            for (int j = 0; j < SIDE; ++j) {
                const float wpx = fx + static_cast<float>(j * ST - R);
                const float qx = __fadd_rn(__fmaf_rn(a0, wpx, tqx), a2);
                const float qy = __fadd_rn(__fmaf_rn(a3, wpx, tqy), a5);
                const float qz = __fadd_rn(__fmaf_rn(a6, wpx, tqz), a8);
                const float sval = __fadd_rn(__fmaf_rn(nK0, wpx, tsv), nK2);
                const float factor = __fmul_rn(sval, inv_n_dot_P);
                const float wz = __fmaf_rn(b2, factor, qz);
                const float iw = rcp_approx(wz);
                const float u = __fmul_rn(__fmaf_rn(b0, factor, qx), iw);
                const float vv = __fmul_rn(__fmaf_rn(b1, factor, qy), iw);
                const bool skip = fabsf(wz) < 1e-8f || u < 0.0f || u >= fw1 || vv < 0.0f || vv >= fh1;
                ok |= static_cast<unsigned>(!skip) << j;
                smp[j] = tex2D<float>(tex, __fadd_rn(u, 0.5f), __fadd_rn(vv, 0.5f));
            }
            const float* rrow = s_ref + (ly + i * ST) * tw + lx;
#pragma unroll
            for (int j = 0; j < SIDE; ++j) {
                if (ok & (1u << j)) {
                    const float rv = rrow[j * ST];
                    const float sv = smp[j];
                    sum_ref = __fadd_rn(sum_ref, rv);
                    sum_src = __fadd_rn(sum_src, sv);
                    sum_ref2 = __fmaf_rn(rv, rv, sum_ref2);
                    sum_src2 = __fmaf_rn(sv, sv, sum_src2);
                    sum_rs = __fmaf_rn(rv, sv, sum_rs);
                    count++;
                }
            }
        }
    }
    float c;
    if (count < min_count) {
        c = 2.0f;
    } else {
        // Opaque: one copy of the expressions below for both branches above, so one choice of fused products.
        asm volatile("" : "+r"(count));
        const float fc = static_cast<float>(count);
        const float num = fc * sum_rs - sum_ref * sum_src;
        const float den_r = fc * sum_ref2 - sum_ref * sum_ref;
        const float den_s = fc * sum_src2 - sum_src * sum_src;
        if (den_r < 1e-6f || den_s < 1e-6f) {
            c = 2.0f;
        } else {
            float ncc = num / (sqrtf(den_r) * sqrtf(den_s));
            ncc = fmaxf(-1.0f, fminf(1.0f, ncc));
            c = 1.0f - ncc;
        }
    }
    return c;
}

__global__ void __launch_bounds__(256) init_kernel(BatchList bl) {
    int tile_x, tile_y;
    const ViewDesc* v = locate_tile(bl, blockIdx.x, &tile_x, &tile_y);
    tile_init(v, tile_x, tile_y);
}

// The reference's mean of the k lowest (a fast-math division: a multiplication
// by an approximate reciprocal, monotone in the sum).
__device__ __forceinline__ float mean_f32(float sum, int k) { return sum / static_cast<float>(k); }

// Full-map cost of the current hypotheses of one tile (compute_ncc_cost_kernel,
// patchmatch_mvs.cu:349-513).  Each thread owns two pixels of its row.
template <int R, int ST, int TH>
__device__ __forceinline__ void tile_cost(const ViewDesc* v, int x0, int y0, const SolveConsts& sc, float* s_ref) {
    constexpr int tw = TILE_W + 2 * R, th = TH + 2 * R;
    load_ref_tile(s_ref, tw, th, v, x0, y0, R);
    __syncthreads();
    // Lanes own consecutive pixels (a warp 32 of a tile row): its taps of one
    // window position then lie next to each other.
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    constexpr int WARPS_A_ROW = CTA_THREADS / 32 / TH;  // 1, each taking both halves of its row, or 2
    const int ly = warp / WARPS_A_ROW, y = y0 + ly;
    if (y >= v->H) return;
    for (int j = 0; j < 2 / WARPS_A_ROW; ++j) {
        // Whole warps vote; lanes past the image name its last column and neither sample nor store.
        const int left = 32 * (j + warp % WARPS_A_ROW), lx = min(left + lane, v->W - 1 - x0), x = x0 + lx;
        if (lx < left) break;
        const size_t idx = static_cast<size_t>(y) * v->W + x;
        PlaneF32 p = plane_f32(v, x, y, v->hyp[idx]);
        const bool live = left + lane == lx;
        p.ok = p.ok && live;
        const float2 sums = window_sums<R, ST>(s_ref, tw, lx, ly);
        Lowest low;
        for (int s = 0; s < v->S; ++s) low.insert(cost_f32<R, ST>(s_ref, tw, lx, ly, x, y, p, sums, v, s));
        if (live) v->cost[idx] = mean_f32(low.sum(min(sc.top_k, v->S)), min(sc.top_k, v->S));
    }
}

// SPLIT: two CTAs of 64 x 4 pixels to a tile (split_cost).
template <int R, int ST, bool SPLIT>
__global__ void __launch_bounds__(CTA_THREADS, COST_BLOCKS) cost_kernel(BatchList bl, SolveConsts sc) {
    constexpr int TH = SPLIT ? TILE_H / 2 : TILE_H;
    __shared__ float s_ref[(TILE_W + 2 * R) * (TH + 2 * R)];
    int tile_x, tile_y;
    const ViewDesc* v = locate_tile(bl, SPLIT ? blockIdx.x >> 1 : blockIdx.x, &tile_x, &tile_y);
    tile_cost<R, ST, TH>(v, tile_x * TILE_W, tile_y * TILE_H + (SPLIT ? (blockIdx.x & 1) * TH : 0), sc, s_ref);
}

// Shared memory of a half-pass beyond the reference tile.
template <int PX, PassForm F>
struct Shared32 {
    static constexpr bool WHOLE = F == PassForm::WHOLE;
    float4 plane[WHOLE ? 1 : CTA_THREADS];  // nK and 1 / (n.P) of the chunk's items
    float unit[WHOLE ? 1 : HP_MAX_SOURCES * CTA_THREADS];
    unsigned char ok[WHOLE ? 1 : CTA_THREADS];
    float2 sums[PX];            // window_sums of each pixel
    PassShared<CTA_THREADS, PX> pass;
};

// Scorer of the half-pass (red_black_pass).
template <int R, int ST, int PX, PassForm F>
struct Scorer32 {
    static constexpr bool BLOCKS = true, BY_PLANE = true, WHOLE_WARPS = true, EAGER = true;
    static constexpr PassForm FORM = F;
    using Plane = PlaneF32;
    const ViewDesc* v;
    const float* s_ref;
    Shared32<PX, F>& sm;
    int x0, y0;
    __device__ __forceinline__ void begin(int lx, int ly) {
        sm.sums[threadIdx.x] = window_sums<R, ST>(s_ref, TILE_W + 2 * R, lx, ly);
    }
    __device__ __forceinline__ void publish() {}
    __device__ __forceinline__ PlaneF32 plane(int x, int y, float4 h, bool ok) const {
        PlaneF32 p = plane_f32(v, x, y, h);
        p.ok = p.ok && ok;
        return p;
    }
    __device__ __forceinline__ bool has(const PlaneF32&) const { return true; }  // score's vote wants every lane
    __device__ __forceinline__ void store(int k, const PlaneF32& p) {
        sm.plane[k] = make_float4(p.nK0, p.nK1, p.nK2, p.inv_n_dot_P);
        sm.ok[k] = p.ok;
    }
    __device__ __forceinline__ PlaneF32 load(int k) const {
        const float4 q = sm.plane[k];
        return PlaneF32{q.x, q.y, q.z, q.w, sm.ok[k] != 0};
    }
    __device__ __forceinline__ float score(int s, PlaneF32 p, int o, int lx, int ly, bool live) const {
        p.ok = p.ok && live;
        return cost_f32<R, ST>(s_ref, TILE_W + 2 * R, lx, ly, x0 + lx, y0 + ly, p, sm.sums[o], v, s);
    }
    __device__ __forceinline__ float mean(float sum, int k) const { return mean_f32(sum, k); }
};

template <int R, int ST, int TH, PassForm F>
__device__ __forceinline__ void tile_propagate(const ViewDesc* v, int x0, int y0, const SolveConsts& sc,
                                               int iteration, int color, float* s_ref,
                                               Shared32<TILE_W * TH / 2, F>& sm) {
    constexpr int PX = TILE_W * TH / 2;
    load_ref_tile(s_ref, TILE_W + 2 * R, TH + 2 * R, v, x0, y0, R);
    __syncthreads();
    Scorer32<R, ST, PX, F> scorer{v, s_ref, sm, x0, y0};
    red_black_pass<CTA_THREADS, PX>(v, x0, y0, sc, iteration, color, scorer, sm.unit, sm.pass);
}

template <int R, int ST, PassForm F>
__global__ void __launch_bounds__(CTA_THREADS, pass_blocks<R, ST, F>())
    propagate_kernel(BatchList bl, SolveConsts sc, int iteration, int color) {
    constexpr bool HALVES = F == PassForm::ROOMY || F == PassForm::SPLIT;
    constexpr int TH = HALVES ? TILE_H / 2 : TILE_H;
    __shared__ float s_ref[(TILE_W + 2 * R) * (TH + 2 * R)];
    __shared__ Shared32<TILE_W * TH / 2, F> sm;
    int tile_x, tile_y;
    const ViewDesc* v = locate_tile(bl, HALVES ? blockIdx.x >> 1 : blockIdx.x, &tile_x, &tile_y);
    const int y0 = tile_y * TILE_H + (HALVES ? (blockIdx.x & 1) * TH : 0);
    tile_propagate<R, ST, TH, F>(v, tile_x * TILE_W, y0, sc, iteration, color, s_ref, sm);
}

// Persistent form: one launch runs every stage of every view of a solve
// (see Schedule), each CTA taking tiles until the tickets run out.  The stage
// bodies are the functions the per-stage kernels above run, so the results
// are bit-identical to the per-stage launch sequence.
template <int R, int ST, PassForm F, bool MANY>
__global__ void __launch_bounds__(CTA_THREADS, persistent_blocks<R, ST, F, MANY>()) persistent_kernel(Schedule s) {
    __shared__ float s_ref[(TILE_W + 2 * R) * (TILE_H + 2 * R)];
    __shared__ Shared32<CTA_THREADS, F> sm;
    // The claimed tile lives in shared memory: warp 0 decodes it once and
    // thread 0 publishes it after the stage, so no thread carries it through the body.
    __shared__ SchedTile s_tile;
    __shared__ int s_ok;
    for (;;) {
        if (threadIdx.x < 32) {
            const bool ok = sched_claim(s, &s_tile);
            if (threadIdx.x == 0) s_ok = ok;
        }
        __syncthreads();
        if (!s_ok) break;
        // Rebuilt from the kernel parameter rather than read back from shared
        // memory, so the compiler knows it addresses global memory (a pointer
        // loaded from shared memory is generic: the FP32 kernel ran 22% slower).
        const ViewDesc* v = &s.views[s_tile.view];
        const int stage = s_tile.stage, tx = s_tile.tx, ty = s_tile.ty;
        if (stage == 0) {
            tile_init(v, tx, ty);
            __syncthreads();
            tile_cost<R, ST, TILE_H>(v, tx * TILE_W, ty * TILE_H, s.sc, s_ref);
        } else if (stage <= 2 * v->iterations) {
            const int k = stage - 1;
            tile_propagate<R, ST, TILE_H, F>(v, tx * TILE_W, ty * TILE_H, s.sc, k >> 1, k & 1, s_ref, sm);
        } else if (is_filter_stage(v, stage)) {
            tile_filter(s.views, v, tx, ty, true);  // geometric check, then the maps
        } else {
            tile_unpack(v, tx, ty);
        }
        __syncthreads();
        if (threadIdx.x == 0) sched_publish(s, s_tile);
    }
}

template <int R, int ST>
cudaError_t launch_rs(const BatchList& bl, const SolveConsts& sc, int iteration, int color, bool full,
                      cudaStream_t st) {
    constexpr int N = window_taps(R, ST);
    const int tiles = bl.total_tiles, sms = device_sms();
    if (full) {
        if (split_cost(tiles, sms))  // whole tiles -> halves, 701 x 439 (605 tiles), r 3 s 2, 6 sources: 152 -> 130 us
            cost_kernel<R, ST, true><<<2 * tiles, CTA_THREADS, 0, st>>>(bl, sc);
        else
            cost_kernel<R, ST, false><<<tiles, CTA_THREADS, 0, st>>>(bl, sc);
        return cudaGetLastError();
    }
    switch (pass_form(PASS_RULE_F32, N, bl.max_sources, tiles, sms)) {
        case PassForm::ROOMY: {
            SolveConsts k = sc;
            k.roomy = 1;
            propagate_kernel<R, ST, PassForm::ROOMY><<<2 * tiles, CTA_THREADS, 0, st>>>(bl, k, iteration, color);
            break;
        }
        case PassForm::SPLIT:
            propagate_kernel<R, ST, PassForm::SPLIT><<<2 * tiles, CTA_THREADS, 0, st>>>(bl, sc, iteration, color);
            break;
        case PassForm::WHOLE:
            if constexpr (N <= PASS_RULE_F32.whole)
                propagate_kernel<R, ST, PassForm::WHOLE><<<tiles, CTA_THREADS, 0, st>>>(bl, sc, iteration, color);
            break;
        case PassForm::UNITS:
            propagate_kernel<R, ST, PassForm::UNITS><<<tiles, CTA_THREADS, 0, st>>>(bl, sc, iteration, color);
            break;
    }
    return cudaGetLastError();
}

cudaError_t dispatch_f32(const BatchList& bl, const SolveConsts& sc, int iteration, int color, bool full,
                         cudaStream_t st) {
    if (bl.total_tiles <= 0) return cudaSuccess;
    if (sc.stride != 1 && sc.stride != 2) return cudaErrorInvalidValue;
#define HP_CASE(RR)                                                                  \
    case RR:                                                                         \
        return sc.stride == 1 ? launch_rs<RR, 1>(bl, sc, iteration, color, full, st) \
                              : launch_rs<RR, 2>(bl, sc, iteration, color, full, st);
    switch (sc.radius) {
        HP_CASE(1)
        HP_CASE(2)
        HP_CASE(3)
        HP_CASE(4)
        HP_CASE(5)
        HP_CASE(6)
        HP_CASE(7)
        default: return cudaErrorInvalidValue;
    }
#undef HP_CASE
}

template <int R, int ST, PassForm F>
cudaError_t persistent_rsf(const Schedule& s, int grid, cudaStream_t st, int* occ) {
    const bool many = s.tiles > many_tiles<R, ST>() * device_sms();
    const auto kernel = many ? persistent_kernel<R, ST, F, true> : persistent_kernel<R, ST, F, false>;
    if (occ) return cudaOccupancyMaxActiveBlocksPerMultiprocessor(occ, kernel, CTA_THREADS, 0);
    kernel<<<grid, CTA_THREADS, 0, st>>>(s);
    return cudaGetLastError();
}

template <int R, int ST>
cudaError_t persistent_rs(const Schedule& s, int grid, cudaStream_t st, int* occ) {
    constexpr int N = window_taps(R, ST);
    if constexpr (N <= PASS_RULE_F32.whole_persistent)
        if (persistent_whole(PASS_RULE_F32, N, s.max_sources, s.tiles, device_sms()))
            return persistent_rsf<R, ST, PassForm::WHOLE>(s, grid, st, occ);
    return persistent_rsf<R, ST, PassForm::UNITS>(s, grid, st, occ);
}

cudaError_t persistent_dispatch(int radius, int stride, const Schedule& s, int grid, cudaStream_t st, int* occ) {
    if (stride != 1 && stride != 2) return cudaErrorInvalidValue;
#define HP_CASE(RR) \
    case RR:        \
        return stride == 1 ? persistent_rs<RR, 1>(s, grid, st, occ) : persistent_rs<RR, 2>(s, grid, st, occ);
    switch (radius) {
        HP_CASE(1)
        HP_CASE(2)
        HP_CASE(3)
        HP_CASE(4)
        HP_CASE(5)
        HP_CASE(6)
        HP_CASE(7)
        default: return cudaErrorInvalidValue;
    }
#undef HP_CASE
}

}  // namespace

cudaError_t launch_persistent_f32(const Schedule& s, int grid, cudaStream_t st) {
    if (s.total <= 0 || grid <= 0) return cudaSuccess;
    Schedule k = s;
    if (!k.abort) k.abort = k.status + 1;
    return persistent_dispatch(k.sc.radius, k.sc.stride, k, grid, st, nullptr);
}

cudaError_t persistent_occupancy_f32(const SolveConsts& sc, int tiles, int max_sources, int* blocks_per_sm) {
    Schedule s{};
    s.tiles = tiles;
    s.max_sources = max_sources;
    return persistent_dispatch(sc.radius, sc.stride, s, 0, nullptr, blocks_per_sm);
}

cudaError_t launch_init(const BatchList& bl, int tile_h, cudaStream_t st) {
    if (bl.total_tiles <= 0) return cudaSuccess;
    init_kernel<<<bl.total_tiles, 32 * tile_h, 0, st>>>(bl);
    return cudaGetLastError();
}

cudaError_t launch_cost_f32(const BatchList& bl, const SolveConsts& sc, cudaStream_t st) {
    return dispatch_f32(bl, sc, 0, 0, true, st);
}

cudaError_t launch_propagate_f32(const BatchList& bl, const SolveConsts& sc, int iteration, int color,
                                 cudaStream_t st) {
    return dispatch_f32(bl, sc, iteration, color, false, st);
}

}  // namespace hp
