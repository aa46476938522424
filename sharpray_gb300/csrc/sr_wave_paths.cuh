// sr_wave_paths.cuh — the render of a small image, and what a bounce loop leaves of a large one, as one
// persistent kernel.  sr_wave_paths.cu and sr_wave_paths_384.cu instantiate it at two block sizes.
//
// The bounce loop of sr_wavefront.cu runs every path one segment per bounce, and a bounce lasts as
// long as its longest traversal plus six dependent launches: 170 us for 65,536 pixels, most of it
// latency on a nearly idle GPU (10 warps per SM in the traversal, which starts with a cold L1 every
// time).  A frame of a million paths fills those kernels; a small image does not.  Here one block per
// SM owns the paths of some pixels for the whole render and runs them in rounds of its own: all its
// slots that are ready for a step take it (surface events, fog, miss, finished samples: the wavefront
// kernels' own per-path functions on up to 32 slots of one kind per warp), then its warps trace the
// rays that came out of that.  A round waits for the block's rays only, and not even for all of them:
// when one in kKeepDiv is left, the round ends and those lanes go on with them in the next one.
// Every path's operations and their order are those of the wavefront, so images are identical.
//
// The phases are a matter of the instruction cache: the code of all steps is 170-340 KB, more than
// an SM holds.  With warps that took any work at any time (queues of each kind in shared memory, no
// barriers) an instruction waited 13 of 20 cycles for its fetch, and 256x256 pixels took 12.6 ms;
// in phases, where the SM's warps run the same code, 5.3 ms.  One block of 512 threads and 128
// registers: 256 x 2 blocks 5.6 ms, 384 x 2 6.7, 768 x 1 6.4, 128 x 6 9.3 (fewer slots per block mean
// less coherent batches and several phases at once on an SM; fewer registers mean spills).  With few
// slots 384 threads of 168 registers do as much: 256x256 4.81 instead of 5.00 ms, 48x40 1.15 / 1.23,
// 320x320 2.88 / 2.91, 384x384 3.56 / 3.48, 512x512 5.10 / 4.86 (8 spp).
// Measured, bounce loop -> this kernel: 48x40 with glass 4.5 -> 1.9 ms, 256x256 8.6 -> 5.3, 192x192
// in fog with its adjoint 15.8 -> 7.2 per view, 512x512 4.8 -> 4.1 (8 spp).
//
// A bounce loop's last paths come here too: a thread per path ran each to its end in a warp of 32
// different ones, 4.2 ms for the last 1/16 of a 1080p fog frame, whose bounces by then took as long
// as full ones.
#pragma once

#include <cuda_runtime.h>

#include "sr_wave_kernels.cuh"

namespace sr {

constexpr uint32_t kPathSlots = 2048;  // slots of a block (1024: 512x512 24.7 instead of 18 ms)
// Ready slots are stepped while they are at least one in kReadyDiv of the live ones; rays are traced
// until one in kKeepDiv is left (192x192 views: none left 35.3 ms, 1/16 28.8, 1/8 29.4, 1/4 33.4, 1/2
// 44.4).  Against 1/8 and 1/16, 1/4 and 1/24 take a 48x40 tile from 1.80 to 1.73 ms, 256x256 from 4.83
// to 4.75, a 512x512 render and replay from 16.9 to 16.7, the views ±0 (steps from 1/16 on: 1.88 and
// 4.92 ms; rays until 1/8: 1.85 and 4.84, until 1/32: 1.76 and 4.82).
constexpr uint32_t kReadyDiv = 4, kKeepDiv = 24;
// Node visits of a burst, which ends early once three quarters of the busy lanes wait for a leaf action
// (256x256: 8 visits or 16 and half of the lanes waiting, at most 16: 5.18 and 5.16 ms; 16 and three
// quarters 5.00; 4 visits 5.25).
constexpr int kBurst = 16;

// What a slot waits for; the first three are the events (EV_FOG, EV_MISS, EV_SURF).
enum : int { K_FIN = 3, kKinds = 4 };

struct BlockQueues {
    // slots whose next step needs no ray (ping-pong); two kinds share a list, filled from its two ends
    uint16_t ready[2][kKinds / 2][kPathSlots];
    uint16_t ray[kPathSlots], shadow[kPathSlots];
    uint32_t n_ready[2][kKinds], n_ray, n_shadow;
    uint32_t fetch;
    uint32_t active;           // rays taken or to be taken this round and not answered yet
    uint32_t slot[kPathSlots];  // the block's slots: the global slot of each
    uint32_t word[kPathSlots];  // per slot: what follows its rays (event or K_FIN) << 8 | rays in flight
    uint32_t live;             // slots with a pixel
    bool finished;             // a sample was finished since this was last looked at
    bool publisher;            // this block publishes the render's progress
    uint64_t idle;             // rounds since a sample was last seen to be finished
};
constexpr uint32_t kLookRounds = 16;  // rounds between looks at these three

// Place of item i of kind k in its list.
__device__ __forceinline__ uint32_t place(int k, uint32_t i) { return k & 1 ? kPathSlots - 1u - i : i; }

// The calling lanes' items appended to a list where `pred` holds (one atomic per warp).
__device__ __forceinline__ void append(uint16_t* list, uint32_t* count, uint32_t item, bool pred, int k = 0) {
    const unsigned m = __ballot_sync(0xffffffffu, pred);
    if (!m) return;
    const int lane = threadIdx.x & 31;
    uint32_t base = 0;
    if (lane == 0) base = atomicAdd(count, (uint32_t)__popc(m));
    base = __shfl_sync(0xffffffffu, base, 0);
    if (pred) list[place(k, base + (uint32_t)__popc(m & ((1u << lane) - 1u)))] = (uint16_t)item;
}

// Slot l of the calling block as an index over all blocks: granules of 2^grain_log2 slots (at most an 8x4
// pixel tile) are dealt out to the blocks in turn, so that every block gets pixels from all over the image.
__device__ __forceinline__ uint32_t dealt(uint32_t l, uint32_t grain_log2) {
    return (((l >> grain_log2) * gridDim.x + blockIdx.x) << grain_log2) + (l & ((1u << grain_log2) - 1u));
}

// A live path of the bounce loop, as its queues of parity `cur` hold it.
struct LivePath {
    uint32_t slot;
    int then;     // what follows its rays: an event or K_FIN (0 with `ray`: the ray tells)
    bool ray;     // its path ray is to be traced
    bool traced;  // its shadow ray has been traced (a query that the last traversal kernel set aside)
};
static __device__ bool live_path(const WaveGroups& G, int cur, uint32_t k, LivePath& p) {
    for (int g = 0; g < G.groups; ++g) {
        const WaveState& W = G.W[g];
        const uint32_t nt = W.counts[kCountTrace + cur];
        if (k < nt) {
            p = {(uint32_t)__float_as_int(W.q_trace[cur][k].a.w), 0, true, false};
            return true;
        }
        k -= nt;
        for (int e = 0; e < 3; ++e) {
            const uint32_t ne = W.counts[kCountEvent + 3 * cur + e];
            if (k < ne) {
                p = {W.q_event[cur][(size_t)e * W.slots + k], e, false, false};
                return true;
            }
            k -= ne;
        }
        const uint32_t nl = W.counts[kCountLate + cur];
        if (k < nl) {
            p = {W.q_late[cur][k], K_FIN, false, false};
            return true;
        }
        k -= nl;
        const uint32_t nd = wave_deferred(W.counts, W.defer_cap, cur);
        if (k < nd) {
            p = {*reinterpret_cast<const uint32_t*>(W.defer[cur] + (size_t)k * kDeferF4), 0, true, true};
            return true;
        }
        k -= nd;
    }
    return false;
}

// cur_queues < 0: the whole render, its first camera rays made by k_paths_init; else what the bounce loop
// left, the live paths of parity cur_queues.  With more than `most` of those the loop did not hand over: its
// cap ended it, the render is an error, and nothing is run.
template <int THREADS, bool GENERAL, int ADJ>
__global__ void __launch_bounds__(THREADS, 1)
    k_wave_paths(const __grid_constant__ WaveGroups G, DevScene S, DevView V, DevParams P, DevAovs out, int cur_queues,
                 uint32_t most, uint32_t grain_log2, uint32_t* err, uint32_t* progress, const AdjPass* A) {
    __shared__ BlockQueues q;
    const WaveState& W = G.W[0];  // (groups differ in their queues only)
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    if (cur_queues >= 0) {  // (this kernel leaves these counts alone: every block reads the same)
        uint32_t handed = 0;
        for (int g = 0; g < G.groups; ++g) handed += wave_live(G.W[g].counts, cur_queues, G.W[g].defer_cap);
        if (handed > most) return;
    }
    if (tid < 2 * kKinds) (&q.n_ready[0][0])[tid] = 0;
    if (tid == 0) q.n_ray = q.n_shadow = q.live = q.active = 0, q.idle = 0, q.finished = q.publisher = false;
    __syncthreads();

    Ctr c;
    [[maybe_unused]] double g_density = 0.0;  // adjoint replay: this thread's d loss / d fog density
    const bool loop_shadows = GENERAL && S.has_transparent;

    // ---- the block's paths ----
    for (uint32_t base = 0; base < kPathSlots; base += THREADS) {
        const uint32_t l = base + tid, k = dealt(l, grain_log2);
        LivePath p{k, 0, true, true};
        // (kPathSlots is no multiple of 384 threads)
        const bool valid = l < kPathSlots && (cur_queues < 0 ? k < W.slots && W.ev_mark[k] : live_path(G, cur_queues, k, p));
        bool shadow = false;
        if (valid) {
            q.slot[l] = p.slot;
            shadow = !p.traced && (ibits(ld_rec(&W.rec[rix(W, p.slot, R_PATH)]).b.w) & PF_NEE);
            q.word[l] = ((uint32_t)p.then << 8) | ((p.ray ? 1u : 0u) + (shadow ? 1u : 0u));
        }
        append(q.ray, &q.n_ray, l, valid && p.ray);
        append(q.shadow, &q.n_shadow, l, shadow);
#pragma unroll
        for (int e = 0; e < kKinds; ++e)
            append(q.ready[0][e >> 1], &q.n_ready[0][e], l, valid && !p.ray && !shadow && p.then == e, e);
        const unsigned m = __ballot_sync(0xffffffffu, valid);
        if (lane == 0 && m) atomicAdd(&q.live, (uint32_t)__popc(m));
    }
    // this lane's traversal carried from one round to the next: its stack, and its state between rounds
    StackEntry entries[kSceneStack];
    uint32_t carried[SceneQuery<false, GENERAL, true>::kQueryWords];
    bool busy = false, shadow = false;
    [[maybe_unused]] ShadowChain chain;
    uint32_t l = 0;  // ... and its slot
    int cur = 0;
    // A round steps a slot or answers a ray, so until a sample is finished there are at most as many rounds
    // as the slots' samples have steps and rays: a step, a path ray and a shadow ray for each of bounces + 2
    // segments, and the sample's end.  Samples are bounded by the pixels' max_samples.
    const uint64_t most_idle = (uint64_t)kPathSlots * (3ull * ((uint64_t)P.bounces + 2u) + 1u) + 2u * kLookRounds;
    uint32_t round = 0;
    for (;;) {
        __syncthreads();
        const uint32_t live = q.live;
        if (live == 0) break;
        uint32_t n[kKinds];
        uint32_t ready = 0;
#pragma unroll
        for (int k = 0; k < kKinds; ++k) ready += n[k] = q.n_ready[cur][k];
        const uint32_t nray = q.n_ray, nshadow = q.n_shadow, kept = q.active;
        __syncthreads();  // every thread has read the counts, and takes the same branch
        bool stuck = !ready && !nray && !nshadow && !kept;  // cannot happen: a live slot waits for something
        if ((round++ & (kLookRounds - 1u)) == 0) {
            if (tid == 0) {
                q.idle = q.finished ? 0 : q.idle + kLookRounds;
                q.finished = false;
                stuck = stuck || q.idle > most_idle;
                // finished pixels, published by one block at a time so that they only grow; one that is done
                // leaves it to the first that asks
                if (progress) {
                    if (!q.publisher) q.publisher = atomicCAS(&W.counts[kCountPublisher], 0u, 1u) == 0u;
                    if (q.publisher) *(volatile uint32_t*)progress = *(volatile uint32_t*)(W.counts + kCountDone);
                }
            }
            stuck = __syncthreads_or(stuck);
        }
        if (stuck) {
            if (tid == 0) atomicOr(err, SR_DEVERR_LOOP);
            break;
        }
        if (ready && (ready * kReadyDiv >= live || nray + nshadow + kept == 0)) {
            // ---- one step of every ready slot: surface events first, then fog, miss, finished samples ----
            const int nxt = cur ^ 1;
            const uint32_t c_surf = (n[EV_SURF] + 31u) >> 5, c_fog = (n[EV_FOG] + 31u) >> 5,
                           c_miss = (n[EV_MISS] + 31u) >> 5, c_fin = (n[K_FIN] + 31u) >> 5;
            const uint32_t chunks = c_surf + c_fog + c_miss + c_fin;
            for (uint32_t ch = warp; ch < chunks; ch += (THREADS / 32)) {
                int kind = EV_SURF;
                uint32_t i = ch;
                if (i >= c_surf) {
                    i -= c_surf, kind = EV_FOG;
                    if (i >= c_fog) {
                        i -= c_fog, kind = EV_MISS;
                        if (i >= c_miss) i -= c_miss, kind = K_FIN;
                    }
                }
                i = 32u * i + lane;
                const bool valid = i < q.n_ready[cur][kind];
                const uint32_t l = valid ? q.ready[cur][kind >> 1][place(kind, i)] : 0u;  // (hides the carried traversal's slot)
                const uint32_t s = q.slot[l];
                SegOut o;
                if (kind == K_FIN) {
                    float g = 0.0f;
                    if (valid) o = finalize_sample<false, GENERAL, ADJ>(W, S, V, P, out, s, c, A, &g);
                    if constexpr (ADJ == kAdjReplay) g_density += (double)g;
                    const unsigned dead = __ballot_sync(0xffffffffu, valid && !o.live);
                    if (lane == 0 && dead) atomicSub(&q.live, (uint32_t)__popc(dead));
                    if (lane == 0) q.finished = true;
                } else if (valid) {
                    if (kind == EV_SURF)
                        o = shade_segment<false, GENERAL, ADJ, false>(W, S, P, s, EV_SURF, c, A);
                    else
                        o = shade_segment<false, GENERAL, ADJ, true>(W, S, P, s, kind, c, A);
                }
                __syncwarp();
                const bool on = valid && (o.live || kind != K_FIN);
                const bool ray = on && o.live && o.next < 0, shadow = on && o.shadow;
                const int then = !o.live ? (int)K_FIN : (o.next >= 0 ? o.next : 0);
                if (ray || shadow) q.word[l] = ((uint32_t)then << 8) | ((ray ? 1u : 0u) + (shadow ? 1u : 0u));
                append(q.ray, &q.n_ray, l, ray);
                append(q.shadow, &q.n_shadow, l, shadow);
                const bool now = on && !ray && !shadow;
#pragma unroll
                for (int k = 0; k < kKinds; ++k) append(q.ready[nxt][k >> 1], &q.n_ready[nxt][k], l, now && then == k, k);
            }
            __syncthreads();
            if (tid < kKinds) q.n_ready[cur][tid] = 0;
            cur = nxt;
            continue;
        }

        // ---- the rays: the persistent loop of persistent_queries over the block's lists ----
        const uint32_t total = nray + nshadow;
        const uint32_t keep = (total + kept) / kKeepDiv;
        if (tid == 0) {
            q.fetch = q.n_ray = q.n_shadow = 0;
            q.active = total + kept;
        }
        __syncthreads();
        // one of slot l's rays is answered (ev: its segment's event, or 0 for a shadow ray): its next
        // step's kind, or -1 while the other ray is in flight
        auto answered = [&](uint32_t l, uint32_t ev) {
            const uint32_t old = atomicAdd(&q.word[l], (ev << 8) - 1u);
            return (old & 0xffu) == 1u ? (int)((old >> 8) + ev) : -1;
        };
        {
            const LaneShare use(total + kept, (THREADS / 32));
            LocalStack stack{entries};
            SceneQuery<false, GENERAL, true> sq;
            if (busy) sq.load(carried);
            bool pending = false, exhausted = total == 0;
            for (;;) {
                unsigned idle = __ballot_sync(0xffffffffu, !busy) & use.lanes;
                int nidle = __popc(idle);
                if (exhausted ? __any_sync(0xffffffffu, pending) : nidle >= use.refill) {
                    int next = -1;
                    bool done = false;
                    if (pending) {
                        const uint32_t s = q.slot[l];
                        uint32_t ev = 0;
                        bool on = false;  // a shadow ray behind a transparent object
                        if (!(loop_shadows ? shadow : sq.any_hit)) {
                            ev = (uint32_t)extend_answer(W, s, sq.best, W.rec[rix(W, s, R_RAY)].b.w);
                        } else if (loop_shadows) {
                            on = !chain.template step<false>(W, S, s, sq.best, sq.wr, c, err);
                            if (on) sq.init(S, Ray(sq.wr), false);
                        } else {
                            float tr = 0.0f;
                            if (sq.best.obj < 0) {
                                tr = 1.0f;
                                if (S.has_fog) tr = 1.0f * fog_transmittance_inf(S, sq.wr);
                            }
                            st4(&W.rec[rix(W, s, R_SH0)].a, make_float4(tr, tr, tr, 0.f));
                        }
                        if (!on) next = answered(l, ev);
                        done = !on;
                        busy = on;
                        pending = false;
                    }
                    const unsigned gone = __ballot_sync(0xffffffffu, done);
                    if (gone && lane == 0) atomicSub(&q.active, (uint32_t)__popc(gone));
                    if constexpr (GENERAL) {
                        idle = __ballot_sync(0xffffffffu, !busy) & use.lanes;
                        nidle = __popc(idle);
                    }
#pragma unroll
                    for (int k = 0; k < kKinds; ++k) append(q.ready[cur][k >> 1], &q.n_ready[cur][k], l, next == k, k);
                    if (!exhausted) {
                        uint32_t base = 0;
                        if (lane == 0) base = atomicAdd(&q.fetch, (uint32_t)nidle);
                        base = __shfl_sync(0xffffffffu, base, 0);
                        if (base + (uint32_t)nidle >= total) exhausted = true;
                        const uint32_t idx = base + (uint32_t)__popc(idle & ((1u << lane) - 1u));
                        if (((idle >> lane) & 1u) && idx < total) {  // shadow rays first
                            const bool any = idx < nshadow;
                            l = any ? q.shadow[idx] : q.ray[idx - nshadow];
                            const uint32_t s = q.slot[l];
                            const Rec r = ld_rec(&W.rec[rix(W, s, any ? R_SH0 : R_RAY)]);
                            sq.init(S, make_ray(V3{r.a.x, r.a.y, r.a.z}, V3{r.b.x, r.b.y, r.b.z}),
                                    any && !loop_shadows);
                            if (loop_shadows && any) chain.begin();
                            shadow = any;
                            busy = true;
                        }
                        __syncwarp();
                    }
                }
                const unsigned busy_mask = __ballot_sync(0xffffffffu, busy);
                if (!busy_mask) {
                    if (exhausted) break;
                    continue;
                }
                if (exhausted && __shfl_sync(0xffffffffu, *(volatile uint32_t*)&q.active, 0) <= keep) break;
                unsigned wait = __ballot_sync(0xffffffffu, busy && sq.state != QS_NODE);
                const int leaf_wait = (3 * __popc(busy_mask) + 3) >> 2;
#pragma unroll 1
                for (int k = 0; k < kBurst; ++k) {
                    if (!(busy_mask & ~wait)) break;
                    if (busy && sq.state == QS_NODE) sq.template node_action<false>(S, stack, c, err);
                    wait = __ballot_sync(0xffffffffu, busy && sq.state != QS_NODE);
                    if (__popc(wait) >= leaf_wait) break;
                }
                if (busy && sq.state != QS_NODE && sq.state != QS_DONE) sq.template leaf_action<false>(S, stack, c, err);
                if (busy && sq.state == QS_DONE) {
                    busy = false;
                    pending = true;
                }
            }
            if (busy) sq.save(carried);
        }
    }
    if (tid == 0 && q.publisher) {
        __threadfence_system();
        atomicExch(&W.counts[kCountPublisher], 0u);
    }
    if constexpr (ADJ == kAdjReplay) {
        __shared__ double part[THREADS / 32];
        for (int d = 16; d > 0; d >>= 1) g_density += __shfl_xor_sync(0xffffffffu, g_density, d);
        if (lane == 0) part[warp] = g_density;
        __syncthreads();
        if (tid == 0 && A->grad_f) {
            for (int w = 1; w < THREADS / 32; ++w) g_density += part[w];
            if (g_density != 0.0) atomicAdd(A->density, g_density);
        }
    }
}

// The kernel's launches at one block size.
template <int THREADS, bool GENERAL, int ADJ>
static void launch_paths(const WaveLaunch& L, const WaveGroups& G, int cur, uint32_t grid, uint32_t grain,
                         cudaStream_t st) {
    k_wave_paths<THREADS, GENERAL, ADJ><<<grid, THREADS, 0, st>>>(G, L.S, L.V, L.P, L.out, cur, L.tail_paths, grain,
                                                              L.err, L.progress, L.adj);
}

template <int THREADS>
static void launch_paths_at(const WaveLaunch& L, const WaveGroups& G, int cur, uint32_t grid, uint32_t grain,
                            cudaStream_t st) {
    if (L.general)
        L.adj_mode == kAdjReplay   ? launch_paths<THREADS, true, kAdjReplay>(L, G, cur, grid, grain, st)
        : L.adj_mode == kAdjRecord ? launch_paths<THREADS, true, kAdjRecord>(L, G, cur, grid, grain, st)
                                   : launch_paths<THREADS, true, kAdjNone>(L, G, cur, grid, grain, st);
    else
        L.adj_mode == kAdjReplay   ? launch_paths<THREADS, false, kAdjReplay>(L, G, cur, grid, grain, st)
        : L.adj_mode == kAdjRecord ? launch_paths<THREADS, false, kAdjRecord>(L, G, cur, grid, grain, st)
                                   : launch_paths<THREADS, false, kAdjNone>(L, G, cur, grid, grain, st);
}

// 384 threads (sr_wave_paths_384.cu).
void launch_paths_384(const WaveLaunch& L, const WaveGroups& G, int cur, uint32_t grid, uint32_t grain, cudaStream_t st);

}  // namespace sr
