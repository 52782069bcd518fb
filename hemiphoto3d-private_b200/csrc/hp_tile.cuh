// Tile-level stages shared by the FP32 and FP16 kernels (hypothesis
// initialisation, output unpacking) and the device side of the persistent
// schedule (ticket decoding, bounded dependency waits, completion flags).
#pragma once

#include "hp_check.cuh"
#include "hp_internal.h"
#include "hp_rng.cuh"

namespace hp {

// Initial hypotheses of one tile: depth uniform in [dmin, dmax]; normal from
// theta in [0, 2pi) and cos(phi) in (0, 1), flipped to face the camera,
// normalised (init_depth_normal_kernel, src/dense_recon/patchmatch_mvs.cu:164-216).
// Pixels the view's SfM seed map covers take their seed's plane instead.
// Every operation is explicitly rounded, so the result does not depend on the
// including translation unit's flags (no intermediate is ever subnormal:
// depths lie in [dmin, dmax] and normal components are at least ~1e-10).
__device__ __forceinline__ void tile_init(const ViewDesc* v, int tile_x, int tile_y) {
    const int ly = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int y = tile_y * v->tile_h + ly;
    if (y >= v->H) return;
    for (int j = 0; j < 2; ++j) {
        const int x = tile_x * TILE_W + j * 32 + lane;
        if (x >= v->W) continue;
        const uint32_t idx = static_cast<uint32_t>(y * v->W + x);
        if (v->seed_map) {  // SfM seed (runPatchMatchMVS, patchmatch_mvs.cu:1111-1177)
            const int k = v->seed_map[idx];
            if (k >= 0) {
                const hp_seed sd = v->seeds[k];
                v->hyp[idx] = make_float4(sd.depth, sd.normal[0], sd.normal[1], sd.normal[2]);
                continue;
            }
        }
        const uint4 r = philox4x32_10(make_uint4(idx, v->view_id, 0u, 0u), v->seed_lo, v->seed_hi);
        const float depth = __fmaf_rn(u01(r.x), __fsub_rn(v->dmax, v->dmin), v->dmin);
        const float3 ray = view_ray(v->kinv, x, y);
        float st, ct;
        sincos_2pi(u01(r.y), &st, &ct);
        const float cp = u01(r.z);
        const float sp = __fsqrt_rn(fmaxf(0.0f, __fmaf_rn(-cp, cp, 1.0f)));
        float3 n = make_float3(__fmul_rn(sp, ct), __fmul_rn(sp, st), cp);
        if (dot3_rn(n, ray) > 0.0f) n = make_float3(-n.x, -n.y, -n.z);
        n = normalize3_rn(n.x, n.y, n.z);
        v->hyp[idx] = make_float4(depth, n.x, n.y, n.z);
    }
}

// Stored costs carry one bit of history.  A cost is never negative, so the sign
// bit of v->cost marks a pixel whose last half-pass left its plane as it was
// ("settled"); readers of the cost itself drop it with cost_value.
__device__ __forceinline__ float cost_value(float c) { return fabsf(c); }
__device__ __forceinline__ bool cost_settled(float c) { return (__float_as_uint(c) >> 31) != 0u; }

__device__ __forceinline__ bool same_plane(float4 a, float4 b) {
    return __float_as_uint(a.x) == __float_as_uint(b.x) && __float_as_uint(a.y) == __float_as_uint(b.y) &&
           __float_as_uint(a.z) == __float_as_uint(b.z) && __float_as_uint(a.w) == __float_as_uint(b.w);
}

// The neighbour planes (bit 0..3: left, right, up, down) that pixel (x, y) must
// score in this half-pass.  Left out, because none of them can win:
//  - a plane outside the depth range (the reference's rule);
//  - a plane bit-identical to the pixel's own or to an earlier listed one:
//    same pixel, same plane, same arithmetic, same cost;
//  - with `memo`, the plane of a settled neighbour, and any plane identical to
//    one.  The neighbour is of the other color, so exactly one half-pass of its
//    own lies between two visits of this pixel: a settled neighbour holds the
//    plane it held at this pixel's previous visit, which scored it then (or a
//    bit-identical one).  The pixel's cost has been at most that score ever
//    since, and a candidate must be strictly lower.  `memo` is false where no
//    previous visit by the same solve exists: in iteration 0, and in a single
//    half-pass on caller maps.
// On 1920 x 1080, r 7, s 2, 6 sources, 12 iterations this leaves 1.54 of the
// 1.78 planes per visit the identity rule alone leaves (3000 x 2000 with noise,
// 8 sources: 1.53 of 1.94).
//
// Settled neighbours' planes are read for those identity tests only, so a pixel
// could read the costs first and then, mostly, no plane at all.  That is two round
// trips in a row, which small launches and small windows pay in full: EAGER fetches
// all planes and costs at once, then decides (planes after costs -> at once: FP32
// 253 x 175, r 1 s 1, 1 source, 6 iterations 253 -> 228 us; 1920 x 1080, 12
// iterations, r 1 s 1, 1 source FP32 4.87 -> 4.18 ms, FP16-acc r 5 s 2, 4 sources
// 17.25 -> 16.58; FP16-acc plans of 4 x 1920 x 1080, r 7 s 2, 6 sources 135.6 ->
// 133.1).  Per-pass FP16-acc launches in units with wide rows in shared memory have
// little L1 left for the planes and read them late (1920 x 1080, 6 sources, r 7 s 2
// 34.4 ms, at once 35.3; r 3 s 1 27.3 and 28.1).
template <bool EAGER>
__device__ __forceinline__ unsigned neighbour_needs(const ViewDesc* v, int x, int y, float4 own, bool memo) {
    const int W = v->W, H = v->H;
    const float dmin = v->dmin, dmax = v->dmax;
    unsigned need = 0, settled = 0;
    auto at = [&](int cand) {
        return static_cast<size_t>(y + (cand == 2 ? -1 : (cand == 3 ? 1 : 0))) * W + x +
               (cand == 0 ? -1 : (cand == 1 ? 1 : 0));
    };
    float4 h[4];
    float c[4];
#pragma unroll
    for (int cand = 0; cand < 4; ++cand) {
        h[cand] = make_float4(0.f, 0.f, 0.f, 0.f);
        c[cand] = 0.f;
        const bool inside = cand == 0 ? x > 0 : (cand == 1 ? x + 1 < W : (cand == 2 ? y > 0 : y + 1 < H));
        if (inside) {
            need |= 1u << cand;
            if (memo) c[cand] = v->cost[at(cand)];
            if constexpr (EAGER) h[cand] = v->hyp[at(cand)];
        }
    }
#pragma unroll
    for (int cand = 0; cand < 4; ++cand)
        if (cost_settled(c[cand])) settled |= 1u << cand;
    need &= ~settled;
    auto plane = [&](int cand) {
        if constexpr (EAGER) return h[cand];
        return v->hyp[at(cand)];
    };
#pragma unroll
    for (int cand = 0; cand < 4; ++cand) {
        if (!(need & (1u << cand))) continue;
        const float4 p = plane(cand);
        bool drop = p.x < dmin || p.x > dmax || same_plane(p, own);
#pragma unroll
        for (int j = 0; j < 4; ++j)
            if (!drop && j != cand && (((j < cand ? need : 0u) | settled) & (1u << j))) drop = same_plane(p, plane(j));
        if (drop) need &= ~(1u << cand);
    }
    return need;
}

// Final stage of a view in a persistent launch: its tile's packed state into
// the output maps (depth, camera-frame AoS normal, cost, and confidence
// 1 - cost / 2 when wanted).
__device__ __forceinline__ void tile_unpack(const ViewDesc* v, int tile_x, int tile_y) {
    const int ly = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int y = tile_y * v->tile_h + ly;
    if (y >= v->H) return;
    if (!HP_CHECK(v->out_depth && v->out_normal && v->out_cost, HP_CHECK_OUTPUT, v->W, v->H, tile_x, tile_y, 0, 0,
                  0.f, 0.f, 0.f, 0.f))
        return;
    for (int j = 0; j < 2; ++j) {
        const int x = tile_x * TILE_W + j * 32 + lane;
        if (x >= v->W) continue;
        const size_t i = static_cast<size_t>(y) * v->W + x;
        const float4 h = __ldcg(v->hyp + i);
        v->out_depth[i] = h.x;
        v->out_normal[3 * i] = h.y;
        v->out_normal[3 * i + 1] = h.z;
        v->out_normal[3 * i + 2] = h.w;
        const float c = cost_value(__ldcg(v->cost + i));
        v->out_cost[i] = c;
        if (v->out_conf) v->out_conf[i] = __fsub_rn(1.0f, __fmul_rn(c, 0.5f));
    }
}

__device__ __forceinline__ int ld_acquire_gpu(const int* p) {
    int v;
    asm volatile("ld.acquire.gpu.global.s32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}

__device__ __forceinline__ void st_release_gpu(int* p, int v) {
    asm volatile("st.release.gpu.global.s32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}

__device__ __forceinline__ int ld_relaxed_gpu(const int* p) {
    int v;
    asm volatile("ld.relaxed.gpu.global.s32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}

__device__ __forceinline__ unsigned long long global_ns() {
    unsigned long long t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}

struct SchedTile {
    const ViewDesc* v;
    int view, stage;
    int tile, tx, ty;
    int ticket;
};

// Whether stage `stage` of view v is its geometric-consistency stage (which
// follows its last half-pass when the view has one).
__device__ __forceinline__ bool is_filter_stage(const ViewDesc* v, int stage) {
    return v->filter != nullptr && stage == 2 * v->iterations + 1;
}

__device__ __forceinline__ unsigned ld_acquire_gpu_u32(const unsigned* p) {
    unsigned v;
    asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}

// Claiming is the work of warp 0, all its lanes together: between a CTA's stages
// its other warps wait for it, so its chain of memory accesses is kept short.
// The ticket's entry is found 32 probes at a time and the dependencies' flags
// are polled by a lane each, where one thread took a binary search and up to
// five polls in a row (5 uneven views, FP16-acc: 33.75 -> 33.38 ms; 6 uneven
// requests through the server 83.2 -> 82.5 ms).
__device__ __forceinline__ SchedTile decode_ticket(const Schedule& s, int t) {
    const int lane = threadIdx.x & 31;
    int lo = 0, n = s.n_entries;
    while (n > 1) {  // the entry is among [lo, lo + n): the last starting at or before t
        const int step = (n + 31) >> 5;
        const bool le = lane * step < n && s.entry_ticket[lo + lane * step] <= t;
        const int seg = 31 - __clz(__ballot_sync(0xffffffffu, le));
        lo += seg * step;
        n = min(step, n - seg * step);
    }
    const int2 info = s.entry_info[lo];
    SchedTile r;
    r.v = &s.views[info.x];
    r.view = info.x;
    r.stage = info.y;
    r.tile = t - s.entry_ticket[lo];
    r.tx = r.tile % r.v->tiles_x;
    r.ty = r.tile / r.v->tiles_x;
    r.ticket = t;
    return r;
}

// A wait of `ticket` ran out: record SCHED_TIMEOUT and the ticket (the first
// recorded wins) and raise the abort flag.
__device__ __forceinline__ void sched_abort(const Schedule& s, int ticket) {
    if (atomicCAS(s.status, SCHED_OK, SCHED_TIMEOUT) == SCHED_OK) atomicExch(s.status + 2, ticket);
    atomicExch(s.abort, 1);
}

// The abort flag is up.  When another launch raised it (a shared flag), this
// launch records SCHED_ABORTED: it stops with work left undone.
__device__ __forceinline__ bool sched_aborted(const Schedule& s) {
    if (!ld_relaxed_gpu(s.abort)) return false;
    atomicCAS(s.status, SCHED_OK, SCHED_ABORTED);
    return true;
}

// Bounded poll of warp 0 for `ticket`: spins while ready() is false on any
// lane.  Bounded by the schedule's time limit and by a poll count (in case the
// global timer stands still); false when this or another CTA gave up.  The
// time limit counts only after kMinPolls sleeping polls, so a step of the
// global timer during a short wait cannot end it.
struct WaitBudget {
    unsigned long long start = 0;
    unsigned polls = 0;
};

template <class Ready>
__device__ __forceinline__ bool sched_poll(const Schedule& s, int ticket, WaitBudget& b, Ready ready) {
    constexpr unsigned kMinPolls = 4096, kMaxPolls = 1u << 26;
    while (!__all_sync(0xffffffffu, ready())) {
        bool stop = false;
        if ((threadIdx.x & 31) == 0) {
            if (sched_aborted(s)) {
                stop = true;
            } else if (++b.polls > 16) {
                const unsigned long long now = global_ns();
                if (b.start == 0) b.start = now;
                if ((now - b.start > s.wait_limit_ns && b.polls > kMinPolls) || b.polls > kMaxPolls) {
                    sched_abort(s, ticket);
                    stop = true;
                } else {
                    __nanosleep(256);
                }
            }
        }
        if (__shfl_sync(0xffffffffu, stop, 0)) return false;
    }
    return true;
}

// Warp 0 of a CTA: wait until the tile and its 4-neighbour tiles have finished
// stage - 1 (lanes 0 to 4 poll one each).  A filter stage also waits until
// every ticket of the solve proper has finished and the previous filtered
// view's stage has finished on all its tiles (both counts only grow, and every
// ticket they count precedes this one, so each is held by a running CTA).
__device__ __forceinline__ bool sched_wait(const Schedule& s, const SchedTile& t) {
    if (t.stage == 0) return true;
    const int need = t.stage - 1;
    const int lane = threadIdx.x & 31, tx = t.v->tiles_x;
    const int* flag = nullptr;
    if (lane == 0) flag = t.v->done + t.tile;
    if (lane == 1 && t.tx > 0) flag = t.v->done + t.tile - 1;
    if (lane == 2 && t.tx + 1 < tx) flag = t.v->done + t.tile + 1;
    if (lane == 3 && t.ty > 0) flag = t.v->done + t.tile - tx;
    if (lane == 4 && t.ty + 1 < t.v->tiles_y) flag = t.v->done + t.tile + tx;
    WaitBudget b;
    if (!sched_poll(s, t.ticket, b, [&] { return !flag || ld_acquire_gpu(flag) >= need; })) return false;
    if (s.main_done && is_filter_stage(t.v, t.stage)) {
        const unsigned main_total = static_cast<unsigned>(s.main_total);
        if (!sched_poll(s, t.ticket, b, [&] { return lane > 0 || ld_acquire_gpu_u32(s.main_done) >= main_total; }))
            return false;
        const int prev = t.v->filter->prev;
        if (prev >= 0) {
            const ViewDesc* pv = &s.views[prev];
            const int* cnt = pv->filter->tiles_done;
            const int want = pv->tiles_x * pv->tiles_y;
            if (!sched_poll(s, t.ticket, b, [&] { return lane > 0 || ld_acquire_gpu(cnt) >= want; })) return false;
        }
    }
    return true;
}

// Thread 0, after the CTA's barrier at the end of a stage: publish it.
__device__ __forceinline__ void sched_publish(const Schedule& s, const SchedTile& t) {
    if (t.view == s.stall_view && t.tile == s.stall_tile) return;
    // The barrier before this orders the CTA's stores ahead of the release (cumulative at gpu scope).
    st_release_gpu(t.v->done + t.tile, t.stage);
    if (s.main_done) {
        __threadfence();  // the counts below are relaxed atomics
        if (t.ticket < s.main_total)
            atomicAdd(s.main_done, 1u);
        else if (is_filter_stage(t.v, t.stage))
            atomicAdd(t.v->filter->tiles_done, 1);
    }
}

// Warp 0: claims the CTA's next ticket and decodes it into *out (written by
// lane 0); false when the schedule is exhausted or aborted (including a
// dependency wait of this ticket that ran out).
__device__ __forceinline__ bool sched_claim(const Schedule& s, SchedTile* out) {
    int t = -1;
    if ((threadIdx.x & 31) == 0 && !sched_aborted(s)) t = static_cast<int>(atomicAdd(s.counter, 1u));
    t = __shfl_sync(0xffffffffu, t, 0);
    if (t < 0 || t >= s.total) return false;
    const SchedTile d = decode_ticket(s, t);
    if (!sched_wait(s, d)) return false;
    if ((threadIdx.x & 31) == 0) *out = d;
    return true;
}

}  // namespace hp
