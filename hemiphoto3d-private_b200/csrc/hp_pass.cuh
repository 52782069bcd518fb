// The red-black half-pass of one tile (propagate_and_refine_kernel,
// src/dense_recon/patchmatch_mvs.cu:519-655), shared by the FP32 and FP16
// kernels: which planes are scored, by which lanes, and how a pixel adopts one.
// A scorer supplies the arithmetic of a cost.
//
// Scoring is split into units of (item, source): an item is a pixel with a
// plane to score, and the CTA's threads take the units of up to NT items in
// order (unit u: item u % n, source u / n).  Every warp then has full lanes
// whatever the number of items, where one lane per item, all sources in a row,
// left the last warps of a list of ~390 items idle for six sources at a time.
// Rounds: the neighbour planes of all pixels of the tile (L, R, U, D; every
// lane lists the ones its pixel must score, the lists concatenated), then one
// round per refinement step with one perturbed plane per pixel.  Owners fold
// their costs in L, R, U, D order with a strict less, exactly as if they had
// scored them one after the other, so results depend neither on which lane
// scored what nor on the tile's shape.
//
// A refinement trial is rarely better than the plane it perturbs, and usually
// much worse: on 1920 x 1080, r 7, s 2, 6 sources, 80-95% of the trials of
// iterations 1 to 7 are beaten by the bound below after 4 of 6 sources, 35%
// still in iteration 11.  So its sources are sampled in two parts, longest
// baseline first (there a wrong plane shows most): all trials on the leading
// S - k + 1 sources, k = min(top_k, S), and on the others only the trials that
// can still win.  Neighbour planes mostly win or come close, so theirs are
// sampled in one part.  Measured with the settled-neighbour rule
// (neighbour_needs), before -> after: FP16-acc 4 x 1920 x 1080, r 7, s 2, 6
// sources, 12 iterations 143.3 -> 126.9 ms; 3000 x 2000, 8 sources 132.9 ->
// 117.2 ms; r 5, s 1 on 1920 x 1080 65.9 -> 56.1 ms.
//
// With few window samples a pixel (few taps, few sources) what a unit costs beside
// them - its plane, statistics and source's coefficients read again, its cost stored,
// a barrier for every part - outweighs the bound.  There a thread scores its item
// whole, all sources in a row, and its own trials with no barrier between them
// (PassForm::WHOLE; the lines are at PassRule).  The loops over neighbours and trials
// are then two, each with its own copy of the scoring code: one loop for both kept the
// state of both alive and spilled (FP16-acc 1921 x 1081, r 1 s 1, 6 sources 9713 us
// with one, 7965 with two).
#pragma once

#include "hp_check.cuh"
#include "hp_internal.h"
#include "hp_rng.cuh"
#include "hp_tile.cuh"

namespace hp {

// The three lowest source costs, inserted one by one.  A cost of 2 (the worst)
// changes nothing, so sources without a valid window need not be inserted.
struct Lowest {
    float top0 = 2.0f, top1 = 2.0f, top2 = 2.0f;
    __device__ __forceinline__ void insert(float c) {
        if (c < top2) {
            top2 = c;
            if (top2 < top1) {
                float t = top1; top1 = top2; top2 = t;
                if (top1 < top0) { t = top0; top0 = top1; top1 = t; }
            }
        }
    }
    __device__ __forceinline__ float sum(int k) const {
        float s = top0;
        if (k > 1) s = __fadd_rn(s, top1);
        if (k > 2) s = __fadd_rn(s, top2);
        return s;
    }
};

// Shared memory of a half-pass with NT threads on PX active pixels, beyond the
// scorer's own and the source costs (HP_MAX_SOURCES rows of NT floats: cost of
// item k at the q-th source of the view's order at q * NT + k).
template <int NT, int PX>
struct PassShared {
    float cost[PX * 4];            // neighbour costs, slot (thread << 2 | cand)
    unsigned short items[PX * 4];  // neighbour items (thread << 2 | cand), then the surviving trials
    unsigned char need[PX];        // neighbour planes each thread's pixel scores (bit per cand)
    int warp_total[NT / 32];
    int survivors;
};

// Tile position of thread t's pixel (the active pixels of a TILE_W x NT / 32
// tile), by rows or by blocks.
// Blocks: a warp covers 32 x 2 pixels, four lanes a 4 x 2 block of them.  The
// texture unit takes a fetch by fours, and their footprints then share a few
// texels, where four pixels two apart in one row spread over a 7 x 1 run (FP32,
// 2 x 1920 x 1080, r 7, s 2: 106.9 -> 100.0 ms; 16 x 4 and 8 x 8 warps measure
// the same there).
// Rows: a warp covers 64 pixels of one row.  The software sampler's quads lie in
// rows, and a warp in one row touches the fewest L1 lines (FP16-acc, r 7, s 2,
// rows / 32 x 2 / 16 x 4 / 8 x 8: 4 x 1920 x 1080 128.0 / 129.2 / 132.1 / 133.8
// ms; 5 and 6 uneven views in persistent launches 32.6 and 80.3 ms against 33.7
// and 83.7).  Its windows beyond shared memory (r 5, s 1) also read the reference
// tile, and take blocks: 56.3 / 55.1 / 56.7 / 58.7 ms.
template <bool BLOCKS>
__device__ __forceinline__ int2 pass_pixel(int t, int y0, int color) {
    const int ly = BLOCKS ? ((t >> 6) << 1) | ((t >> 1) & 1) : t >> 5;
    const int lx = BLOCKS ? (t & 32) + 4 * ((t & 31) >> 2) + 2 * (t & 1) : 2 * (t & 31);
    return make_int2(lx + ((y0 + ly + color) & 1), ly);
}

// The thread that owns the active pixel at tile position (lx, ly).
template <bool BLOCKS>
__device__ __forceinline__ int pass_thread(int lx, int ly) {
    return BLOCKS ? ((ly >> 1) << 6) | (lx & 32) | (((lx & 31) >> 2) << 2) | ((ly & 1) << 1) | ((lx >> 1) & 1)
                  : ly << 5 | lx >> 1;
}

// One half-pass of the tile at (x0, y0), TILE_W x PX / 32 pixels: threads below
// PX own an active pixel each, where the reference idles half its grid.  The
// others, in launches of half tiles (PassForm), only score.
// The scorer K, per thread:
//   begin(lx, ly)               prepares the window of the thread's own pixel (active pixels only)
//   publish()                   makes it readable by the other threads (after the next barrier)
//   plane(x, y, h, ok)          plane h at pixel (x, y) prepared for scoring, ok false: no plane
//   has(p)                      false: every cost is 2, score need not be called
//   store(k, p), load(k)        the prepared plane of item k in shared memory (units only)
//   score(source, p, o, lx, ly, live)  cost of a source under plane p at tile position (lx, ly), thread o's pixel; lanes
//                               that are not live take part for their warp's sake
//   mean(sum, k)                sum / k, monotone in sum
//   BLOCKS                      pass_pixel's layout
//   EAGER                       neighbour_needs' order of reads
//   BY_PLANE                    neighbour items are listed by the plane they score, not by pixel
//   FORM                        the launch's PassForm
//   WHOLE_WARPS                 score starts with a vote of all 32 lanes of a warp
template <int NT, int PX, class K>
__device__ __forceinline__ void red_black_pass(const ViewDesc* v, int x0, int y0, const SolveConsts& sc,
                                               int iteration, int color, K& scorer, float* unit,
                                               PassShared<NT, PX>& sm) {
    const int W = v->W, H = v->H, S = v->S;
    const int tid = threadIdx.x, lane = tid & 31;
    const int2 own = pass_pixel<K::BLOCKS>(tid, y0, color);
    const int lx = own.x, ly = own.y, x = x0 + lx, y = y0 + ly;
    // Read through a broadcast: the compiler then knows that it is the same for a warp's lanes.
    const int warp = __shfl_sync(0xffffffffu, tid >> 5, 0);
    const bool active = (NT == PX || tid < PX) && y < H && x < W;  // every thread takes part in the barriers
    const size_t idx = static_cast<size_t>(y) * W + x;
    float4 best = make_float4(0.f, 0.f, 0.f, 0.f);
    float best_cost = 0.f;
    unsigned need = 0;
    bool settled = true;
    if (active) {
        scorer.begin(lx, ly);
        best = v->hyp[idx];
        best_cost = sc.memo ? cost_value(v->cost[idx]) : v->cost[idx];  // a caller's cost as it is
        need = neighbour_needs<K::EAGER>(v, x, y, best, sc.memo && iteration > 0);
    }
    scorer.publish();
    // Neighbour items are listed by pixel (bit 4 + c of `list`: the own pixel's neighbour c), or by plane: thread t
    // lists the tile's pixels around the inactive pixel of its own 2-pixel cell (bit c: the pixel whose neighbour c that
    // one is), then its own pixel's planes from outside the tile.  The up to four items of a plane are then adjacent
    // lanes, whose windows nearly coincide in every source.  That suits the texture unit (2 x 1920 x 1080, r 7, s 2:
    // 97.9 -> 90.7 ms, 5 x 640 x 480, r 5, s 1: 45.7 -> 42.1 ms), while the software sampler is better off with the
    // planes of one pixel, whose windows keep to its rows of quads (4 x 1920 x 1080: 129.2 ms, by plane 136.6).
    unsigned list = need << 4;
    const int nx = lx ^ 1, ny = ly;  // tiles start at even columns: the cell is columns lx, lx ^ 1
    auto owner = [&](int c) {
        return pass_thread<K::BLOCKS>(nx + (c == 0 ? 1 : (c == 1 ? -1 : 0)), ny + (c == 2 ? 1 : (c == 3 ? -1 : 0)));
    };
    if constexpr (K::BY_PLANE) {
        if (NT == PX || tid < PX) sm.need[tid] = static_cast<unsigned char>(need);
        __syncthreads();
        list = 0;
        constexpr int TH = PX / 32;
#pragma unroll
        for (int c = 0; c < 4; ++c) {
            const bool in = (NT == PX || tid < PX) &&
                            (c == 0 ? nx + 1 < TILE_W : (c == 1 ? nx > 0 : (c == 2 ? ny + 1 < TH : ny > 0)));
            if (in && ((sm.need[owner(c)] >> c) & 1u)) list |= 1u << c;
            const bool outside = c == 0 ? lx == 0 : (c == 1 ? lx + 1 == TILE_W : (c == 2 ? ly == 0 : ly + 1 == TH));
            if (outside && ((need >> c) & 1u)) list |= 16u << c;
        }
    }
    // Exclusive scan of the item counts over the warp, then over the CTA's warps.
    const int cnt = __popc(list);
    int incl = cnt;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int t = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += t;
    }
    if (lane == 31) sm.warp_total[warp] = incl;
    __syncthreads();
    int total = 0;
    {
        int k = incl - cnt;
#pragma unroll
        for (int w = 0; w < NT / 32; ++w) {
            const int t = sm.warp_total[w];
            k += w < warp ? t : 0;
            total += t;
        }
        for (int c = 0; K::BY_PLANE && c < 4; ++c)
            if (list & (1u << c)) sm.items[k++] = static_cast<unsigned short>((owner(c) << 2) | c);
        for (int c = 0; c < 4; ++c)
            if (list & (16u << c)) sm.items[k++] = static_cast<unsigned short>((tid << 2) | c);
    }
    __syncthreads();  // the item list is complete
    // Values that steer the loops below, read through a broadcast: the compiler then knows that a warp stays together
    // in them, and a texture handle stays in a uniform register (with a scorer's votes inside it is otherwise fetched
    // lane by lane: FP32, 2 x 1920 x 1080, 149.7 ms against 115.1).
    total = __shfl_sync(0xffffffffu, total, 0);
    const int kk = min(sc.top_k, S);
    // With warps idle, two parts of few sources would take two turns where one takes one.  A half-pass on caller maps
    // (memo off) scores every trial whole.
    const int lead = !sc.memo || (sc.roomy && S <= 3) ? S : S - kk + 1;
    float drange = __fmul_rn(__fsub_rn(v->dmax, v->dmin), 0.5f);
    float nrange = 1.0f;
    for (int i = 0; i < iteration; ++i) {
        drange = __fmul_rn(drange, sc.iter_decay);
        nrange = __fmul_rn(nrange, sc.iter_decay);
    }
    // The prepared plane of a neighbour item, and its pixel's place in the tile.
    auto neighbour = [&](int item, int2* at) {
        *at = pass_pixel<K::BLOCKS>(item >> 2, y0, color);
        const int cand = item & 3, ox = x0 + at->x, oy = y0 + at->y;
        const int nxp = ox + (cand == 0 ? -1 : (cand == 1 ? 1 : 0));
        const int nyp = oy + (cand == 2 ? -1 : (cand == 3 ? 1 : 0));
        float4 h = make_float4(0.f, 0.f, 0.f, 0.f);
        const bool ok = HP_CHECK(nxp >= 0 && nxp < W && nyp >= 0 && nyp < H, HP_CHECK_NEIGHBOUR, ox, oy, nxp, nyp, W,
                                 H, 0.f, 0.f, 0.f, 0.f);
        if (ok) h = v->hyp[static_cast<size_t>(nyp) * W + nxp];
        return scorer.plane(ox, oy, h, ok);
    };
    // Random refinement around the running best (:583-648): the trial of refinement step `step` (active pixels only).
    auto perturbed = [&](int step) {
        const uint4 rr =
            philox4x32_10(make_uint4(static_cast<uint32_t>(idx), v->view_id, 1u + static_cast<uint32_t>(iteration),
                                     static_cast<uint32_t>(step)),
                          v->seed_lo, v->seed_hi);
        const float cd = __fmaf_rn(__fmaf_rn(u01(rr.x), 2.0f, -1.0f), drange, best.x);
        const float cx = __fmaf_rn(__fmaf_rn(u01(rr.y), 2.0f, -1.0f), nrange, best.y);
        const float cy = __fmaf_rn(__fmaf_rn(u01(rr.z), 2.0f, -1.0f), nrange, best.z);
        const float cz = __fmaf_rn(__fmaf_rn(u01(rr.w), 2.0f, -1.0f), nrange, best.w);
        float3 cn = normalize3_rn(cx, cy, cz);
        if (dot3_rn(cn, view_ray(v->kinv, x, y)) > 0.0f) cn = make_float3(-cn.x, -cn.y, -cn.z);
        return make_float4(fmaxf(v->dmin, fminf(v->dmax, cd)), cn.x, cn.y, cn.z);
    };
    auto narrow = [&] {  // the next step's ranges
        drange = __fmul_rn(drange, sc.step_decay);
        nrange = __fmul_rn(nrange, sc.step_decay);
    };
    // The neighbours' costs, L, R, U, D, each adopted when strictly lower.
    auto fold = [&] {
#pragma unroll
        for (int cand = 0; cand < 4; ++cand) {
            if (need & (1u << cand)) {
                const float nc = sm.cost[(tid << 2) | cand];
                if (nc < best_cost) {
                    const int nxp = x + (cand == 0 ? -1 : (cand == 1 ? 1 : 0));
                    const int nyp = y + (cand == 2 ? -1 : (cand == 3 ? 1 : 0));
                    best_cost = nc;
                    settled = false;
                    best = v->hyp[static_cast<size_t>(nyp) * W + nxp];
                }
            }
        }
    };
    if constexpr (K::FORM == PassForm::WHOLE) {
        auto cost = [&](const typename K::Plane& p, int o, int2 at, bool live) {
            Lowest low;
            if (scorer.has(p))
#pragma unroll 1
                for (int s = 0; s < S; ++s) low.insert(scorer.score(s, p, o, at.x, at.y, live));
            return scorer.mean(low.sum(kk), kk);
        };
#pragma unroll 1
        for (int k0 = warp * 32; k0 < total; k0 += NT) {
            const bool live = k0 + lane < total;
            if (!K::WHOLE_WARPS && !live) continue;
            const int item = sm.items[min(k0 + lane, total - 1)];
            int2 at;
            const typename K::Plane p = neighbour(item, &at);
            const float c = cost(p, item >> 2, at, live);
            if (live) sm.cost[item] = c;
        }
        __syncthreads();  // every neighbour cost is in its owner's slot; no barrier follows
        if (K::WHOLE_WARPS ? !__any_sync(0xffffffffu, active) : !active) return;
        fold();
#pragma unroll 1
        for (int step = 0; step < sc.refine_steps; ++step) {
            const float4 trial = active ? perturbed(step) : make_float4(0.f, 0.f, 0.f, 0.f);
            const float c = cost(scorer.plane(x, y, trial, active), tid, own, active);
            if (active && c < best_cost) {
                best_cost = c;
                settled = false;
                best = trial;
            }
            narrow();
        }
    } else {
#pragma unroll 1
        for (int round = 0; round <= sc.refine_steps; ++round) {
            float4 trial = make_float4(0.f, 0.f, 0.f, 0.f);
            if (round > 0) {
                if (active) trial = perturbed(round - 1);
                narrow();
            }
            const int count = round == 0 ? total : PX;
            float c = 2.0f;
            bool keep = true;
#pragma unroll 1
            for (int c0 = 0; c0 < count; c0 += NT) {
                const int n = min(NT, count - c0);
                int item = tid << 2;
                if (round > 0) {
                    scorer.store(tid, scorer.plane(x, y, trial, active));
                } else if (tid < n) {
                    int2 at;
                    item = sm.items[c0 + tid];
                    scorer.store(tid, neighbour(item, &at));
                }
                if (tid == 0) sm.survivors = 0;
                __syncthreads();  // the chunk's planes are complete
                // Sources first .. last - 1 of the view's order, for the chunk's items (second part: the listed ones).
                int units = n, first = 0, last = round == 0 ? S : lead;
#pragma unroll 1
                for (;;) {
#pragma unroll 1
                    for (int q = first; q < last; ++q) {
                        const int source = v->order[q];
                        // The first warp to take a batch of this source follows the one that took the previous source's
                        // last.
                        const int turn = (q - first) * ((units + 31) >> 5);
#pragma unroll 1
                        for (int u0 = ((warp - turn) & (NT / 32 - 1)) * 32; u0 < units; u0 += NT) {
                            // A scorer that votes wants whole warps: lanes past the last item name it too and are
                            // not live.
                            const int u = K::WHOLE_WARPS ? min(u0 + lane, units - 1) : u0 + lane;
                            const bool live = u0 + lane < units;
                            if (!K::WHOLE_WARPS && !live) continue;
                            const int k = first > 0 ? sm.items[u] : u;
                            const int o = round == 0 ? sm.items[c0 + k] >> 2 : k;
                            const int2 at = pass_pixel<K::BLOCKS>(o, y0, color);
                            const typename K::Plane p = scorer.load(k);
                            const float cost = scorer.has(p) ? scorer.score(source, p, o, at.x, at.y, live) : 2.0f;
                            if (live) unit[q * NT + k] = cost;
                        }
                    }
                    __syncthreads();  // the part's source costs are complete
                    if (last == S) break;
                    // The k-th lowest of all source costs is at least the lowest of the leading S - k + 1, so the mean is
                    // at least that over k (rounded addition and mean() are monotone): a trial whose bound reaches the
                    // pixel's cost cannot win.
                    float low = 2.0f;
                    for (int q = 0; q < lead; ++q) low = fminf(low, unit[q * NT + tid]);
                    keep = active && scorer.mean(low, kk) < best_cost;
                    const unsigned votes = __ballot_sync(0xffffffffu, keep);
                    int at = 0;
                    if (lane == 0 && votes) at = atomicAdd(&sm.survivors, __popc(votes));
                    at = __shfl_sync(0xffffffffu, at, 0);
                    if (keep) sm.items[at + __popc(votes & ((1u << lane) - 1u))] = static_cast<unsigned short>(tid);
                    __syncthreads();  // the survivors' list is complete
                    units = __shfl_sync(0xffffffffu, sm.survivors, 0);
                    first = lead;
                    last = S;
                }
                if (tid < n && keep) {
                    Lowest low;
                    for (int q = 0; q < S; ++q) low.insert(unit[q * NT + tid]);
                    c = scorer.mean(low.sum(kk), kk);
                    if (round == 0) sm.cost[item] = c;
                }
            }
            if (round == 0) {
                __syncthreads();  // every neighbour cost is in its owner's slot
                fold();
            } else if (active && keep && c < best_cost) {
                best_cost = c;
                settled = false;
                best = trial;
            }
        }
    }
    if (!active) return;
    v->hyp[idx] = best;
    v->cost[idx] = sc.memo && settled ? -best_cost : best_cost;
}

}  // namespace hp
