// The wavefront pipeline of the drop-in: camera generation, extend (nearest hit), shade
// (surface, emission, next-event estimation setup, BSDF sampling, roulette), shadow (any hit)
// and accumulate, over persistent grid-stride queues. One wave is a set of path slots; a slot
// is (pixel, sample index) and keeps its own radiance, so the film adds each pixel's samples in
// sample order (integrator/mod.rs:1140-1891, render.rs:388-497, image.rs:82-93).
#include <cuda_runtime.h>

#include <algorithm>

#include "rtg_image.cuh"
#include "rtg_kernels.h"
#include "rtg_shade.cuh"

namespace rtg {

__constant__ SobolTable c_sobol;

// Figures at a choice compare builds that differ in that one thing, at the time it was made; the 1080p
// product frame (1 M triangles, 64 spp, depth 12) takes 157 ms now, the instanced frame (10 M triangles,
// 4 spp) 36 ms.

// Threads per block of the traversal kernels (the stride of their shared stacks).
constexpr int TRACE_THREADS = 128;
// RTG_REFILL_MIN (build setting): idle lanes a k_trace warp waits for before it takes new rays
// (1: every step with an idle lane). A refill costs the whole warp a ballot, an atomic, a shuffle
// and two dependent loads, so taking rays for eight lanes at a time beats taking them one by one as
// rays end: at 4, 8, 12 and 16 the 1080p product frame took 197.6, 192.7, 193.8 and 196.2 ms.
#ifndef RTG_REFILL_MIN
#define RTG_REFILL_MIN 8
#endif
// Blocks per SM the traversal kernels are compiled for (56 registers at 9, 64 at 8; of the kernels in
// use 12 bytes are spilled in EXTEND and in the two that walk): more warps hide the node fetches until
// registers spill. All kernels at 7, 8, 9 and 10 blocks: 1080p product frame 154.4, 148.8, 145.8 and
// 150.6 ms, instanced frame 32.6, 31.7, 31.2 and 33.0 ms, adaptive frame (thin rounds) 70.2 at 8, 71.8 at
// 9, 73.3 ms at 10. (With each leaf's box held against its hits, at 8 and 9: 158.6 and 156.9, 37.6 and
// 36.8 ms.) So the kernel of the smaller waves, which
// traces both kinds of rays, takes 8 and the others 9. RTG_TRACE_MIN_BLOCKS (build setting): both.
#ifdef RTG_TRACE_MIN_BLOCKS
#define RTG_TRACE_BLOCKS(together) RTG_TRACE_MIN_BLOCKS
#else
#define RTG_TRACE_BLOCKS(together) ((together) ? 8 : 9)
#endif
// Blocks of 128 threads per SM that the shade kernels are compiled for (their register cap:
// 65536 / (128 x this)); a build may set it (RTG_SHADE_MIN_BLOCKS) to compare occupancies.
#ifndef RTG_SHADE_MIN_BLOCKS
#define RTG_SHADE_MIN_BLOCKS 8
#endif

// Flags of a path slot.
constexpr uint32_t PF_HAS_PDF = 1, PF_PRIMARY = 2, PF_MEDIUM = 4;
// A panoramic camera's sample that sees nothing (scene/mod.rs:227): its ray has an empty interval
// (no hit, no floor) and its radiance is multiplied by its black weight when it reaches the film.
constexpr uint32_t PF_NOTHING = 8;
// The path's flags also hold the cut-outs it passed (bits 8-14, at most MAX_CUTOUTS) and its vertex
// count (bits 16-26): a cut-out pass is no vertex, so a path's bounce can fall behind the round.
constexpr uint32_t PF_CUT_SHIFT = 8, PF_CUT_MASK = 0x7fu << 8, PF_BOUNCE_SHIFT = 16, PF_BOUNCE_MASK = 0x7ffu << 16;
constexpr uint32_t MAX_CUTOUTS = 64;
// sampler.rs:127-135: the hashed dimension deciding whether vertex `bounce`'s ray passes its
// `crossing`-th cut-out.
RTG_D uint32_t cutout_dim(uint32_t bounce, uint32_t crossing) { return (1u << 20) + bounce * 64u + (crossing < 63u ? crossing : 63u); }

__device__ __forceinline__ void wave_slot(const WaveDesc& w, uint32_t slot, uint32_t& x, uint32_t& y, uint32_t& index) {
    if (w.epix) {
        const uint32_t r = w.by_ek.of(slot), j = slot - r * w.ek, s = w.by_ne.of(r), e = r - s * w.ne;
        const uint32_t packed = w.epix[e];
        x = packed & 0xffffu;
        y = packed >> 16;
        index = ((w.ebase ? __ldg(&w.ebase[e]) : 0u) + w.first + s) * w.ek + j;  // render.rs:376 sub_sample (wrapping)
        return;
    }
    if (w.xys) {
        x = w.xys[3 * slot];
        y = w.xys[3 * slot + 1];
        index = w.xys[3 * slot + 2];
        return;
    }
    const uint32_t s = w.by_pixels.of(slot), rem = slot - s * (w.w * w.h), row = w.by_width.of(rem);
    y = w.y0 + row;
    x = w.x0 + (rem - row * w.w);
    index = w.first + s;
}

// The segment of a batched wave that holds `slot`: the last with slot_begin <= slot.
__device__ __forceinline__ uint32_t seg_of_slot(const WaveDesc& w, uint32_t slot) {
    uint32_t lo = 0, hi = w.nseg;
    while (hi - lo > 1) {
        uint32_t mid = (lo + hi) >> 1;
        if (__ldg(&w.segs[mid].slot_begin) <= slot) lo = mid;
        else hi = mid;
    }
    return lo;
}

// Job, pixel and sample index of a slot of a batched wave.
__device__ __forceinline__ void batch_slot(const WaveDesc& w, uint32_t slot, uint32_t& job, uint32_t& x, uint32_t& y, uint32_t& index) {
    const SegDev& g = w.segs[seg_of_slot(w, slot)];
    const uint32_t local = slot - g.slot_begin;
    const uint32_t s = g.by_pixels.of(local), rem = local - s * (g.w * g.h), row = g.by_width.of(rem);
    job = g.job;
    y = g.y0 + row;
    x = rem - row * g.w;
    index = g.first + s;
}

__device__ __forceinline__ void add_clamped(float4& sum, Rgb c, bool indirect, float clamp) {  // integrator/mod.rs:855
    if (!(finitef(c.r) && finitef(c.g) && finitef(c.b))) return;
    float p = rmax(rmax(c.r, c.g), c.b);
    if (indirect && clamp > 0.0f && p > clamp) c = c * (clamp / p);
    sum.x = sum.x + c.r;
    sum.y = sum.y + c.g;
    sum.z = sum.z + c.b;
}

// The counts of a wave's rounds and the key bins at its start: n paths in round 0.
__device__ __forceinline__ void start_rounds(const PathBuffers& P, uint32_t rounds, uint32_t n) {
    if (blockIdx.x) return;
    for (uint32_t k = threadIdx.x; k < 4 * (rounds + 1); k += blockDim.x) P.counters[ROUND_COUNTERS + k] = k == COUNT_PATHS ? n : 0;
    for (uint32_t k = threadIdx.x; k < 2 * KEY_BINS; k += blockDim.x) P.bins[k] = 0;
}
// The paths a round's kernels work on: none where the tail kernel takes the round (its queue holds
// at most `tail` paths) or an earlier one, which leaves it empty.
__device__ __forceinline__ uint32_t round_paths(const PathBuffers& P, uint32_t round, uint32_t tail) {
    const uint32_t n = *(volatile uint32_t*)&P.counters[round_counter(round, COUNT_PATHS)];
    return round >= TAIL_FIRST_ROUND && n <= tail ? 0 : n;
}
// Lanes of each warp that n units of work fill when every resident warp takes its share: a thin
// round is as long as its slowest ray, and a ray in a warp of its own does not wait for the leaves
// and nodes of 31 others.
__device__ __forceinline__ uint32_t lanes_for(uint32_t n) {
    const uint32_t warps = gridDim.x * (blockDim.x >> 5);
    return min(32u, (n + warps - 1) / warps);
}

// Two neighbouring fields of a path's records (o and d, thr and sum, hit and sel): one 32-byte sector,
// one access.
__device__ __forceinline__ void load_sector(const void* p, uint64_t v[4]) {
    asm volatile("ld.global.v4.b64 {%0, %1, %2, %3}, [%4];" : "=l"(v[0]), "=l"(v[1]), "=l"(v[2]), "=l"(v[3]) : "l"(p) : "memory");
}
__device__ __forceinline__ void load_pair(const PathField& f, uint32_t slot, float4& a, float4& b) {
    uint64_t v[4];
    load_sector(&f[slot], v);
    a = make_float4(__uint_as_float((uint32_t)v[0]), __uint_as_float((uint32_t)(v[0] >> 32)), __uint_as_float((uint32_t)v[1]), __uint_as_float((uint32_t)(v[1] >> 32)));
    b = make_float4(__uint_as_float((uint32_t)v[2]), __uint_as_float((uint32_t)(v[2] >> 32)), __uint_as_float((uint32_t)v[3]), __uint_as_float((uint32_t)(v[3] >> 32)));
}
__device__ __forceinline__ void load_vertex(const PathBuffers& P, uint32_t slot, uint4& hit, float4& sel) {
    uint64_t v[4];
    load_sector(&P.hit[slot], v);
    hit = make_uint4((uint32_t)v[0], (uint32_t)(v[0] >> 32), (uint32_t)v[1], (uint32_t)(v[1] >> 32));
    sel = make_float4(__uint_as_float((uint32_t)v[2]), __uint_as_float((uint32_t)(v[2] >> 32)), __uint_as_float((uint32_t)v[3]), __uint_as_float((uint32_t)(v[3] >> 32)));
}
__device__ __forceinline__ uint64_t pack2(float x, float y) { return ((uint64_t)__float_as_uint(y) << 32) | __float_as_uint(x); }
__device__ __forceinline__ void store_pair(const PathField& f, uint32_t slot, float4 a, float4 b) {
    asm volatile("st.global.v4.b64 [%0], {%1, %2, %3, %4};" ::"l"(&f[slot]), "l"(pack2(a.x, a.y)), "l"(pack2(a.z, a.w)), "l"(pack2(b.x, b.y)), "l"(pack2(b.z, b.w)) : "memory");
}

// ---- camera generation ---------------------------------------------------------------------------
// BATCH: the slots belong to the jobs of a batched wave, each with its own camera.
template <bool BATCH>
__global__ void k_camera(const __grid_constant__ SceneDev S, WaveDesc w, PathBuffers P, uint32_t rounds) {
    for (uint32_t slot = blockIdx.x * blockDim.x + threadIdx.x; slot < w.n; slot += gridDim.x * blockDim.x) {
        uint32_t x, y, index;
        V3 o, d;
        bool sees;
        if constexpr (BATCH) {
            uint32_t job;
            batch_slot(w, slot, job, x, y, index);
            sees = camera_ray(w.jobs[job].S, c_sobol, x, y, index, o, d);
        } else {
            wave_slot(w, slot, x, y, index);
            sees = camera_ray(S, c_sobol, x, y, index, o, d);
        }
        store_pair(P.o, slot, make_float4(o.x, o.y, o.z, __uint_as_float(PF_PRIMARY | (sees ? 0u : PF_NOTHING))), make_float4(d.x, d.y, d.z, 0.0f));
        store_pair(P.thr, slot, make_float4(1.0f, 1.0f, 1.0f, 1.0f), make_float4(0.0f, 0.0f, 0.0f, 0.0f));
        P.queue[0][slot] = slot;
    }
    start_rounds(P, rounds, w.n);
}

// Material key of a path's next vertex, for the material-sorted shade.
__device__ __forceinline__ uint32_t material_key(const SceneDev& S, bool got, uint32_t inst) {
    uint32_t k = got ? __ldg(&S.instances[inst].material) : S.n_materials;
    return k < 255u ? k : 255u;
}

// Adds one to bins[key] for every active lane, one atomic per distinct key of the warp.
__device__ __forceinline__ void warp_count(uint32_t* bins, uint32_t key) {
    uint32_t mask = __match_any_sync(__activemask(), key);
    if ((threadIdx.x & 31) == (uint32_t)(__ffs((int)mask) - 1)) atomicAdd(&bins[key], (uint32_t)__popc(mask));
}

// ---- ray order (RaySort): coherence keys, their prefix and the scatter ---------------------------------
// Cell of coordinate v on a grid of n cells from lo with `scale` cells per unit (NaN and below: 0).
__device__ __forceinline__ uint32_t sort_cell(float v, float lo, float scale, uint32_t n) {
    const float f = (v - lo) * scale;
    return f > 0.0f ? (uint32_t)fminf(f, (float)(n - 1u)) : 0u;
}
// The coherence key of a ray: the octant of d (3 bits) over the Morton code of o's cell.
__device__ __forceinline__ uint32_t ray_key(const RaySort& R, V3 o, V3 d) {
    const uint32_t n = 1u << R.ray_bits;
    const uint32_t cx = sort_cell(o.x, R.lo[0], R.scale[0], n), cy = sort_cell(o.y, R.lo[1], R.scale[1], n),
                   cz = sort_cell(o.z, R.lo[2], R.scale[2], n);
    uint32_t m = 0;
#pragma unroll
    for (uint32_t b = 0; b < RAY_SORT_MAX_BITS; ++b)
        m |= (((cx >> b) & 1u) << (3u * b)) | (((cy >> b) & 1u) << (3u * b + 1u)) | (((cz >> b) & 1u) << (3u * b + 2u));
    const uint32_t oct = (d.x < 0.0f ? 1u : 0u) | (d.y < 0.0f ? 2u : 0u) | (d.z < 0.0f ? 4u : 0u);
    return (oct << (3u * R.ray_bits)) | m;
}

// bins[nk, 2 nk) = exclusive prefix of the histogram bins[0, nk), which is cleared. One block of
// 1024 threads: each warp sums a contiguous chunk, the chunk sums are scanned, then each warp
// scans its chunk row by row (coalesced).
__global__ void __launch_bounds__(1024) k_key_scan(uint32_t* bins, uint32_t nk) {
    __shared__ uint32_t chunk[32];
    const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31u;
    const uint32_t per = ((nk + 31u) / 32u + 31u) & ~31u;
    const uint32_t b0 = min(warp * per, nk), b1 = min(b0 + per, nk);
    uint32_t s = 0;
    for (uint32_t e = b0 + lane; e < b1; e += 32u) s += bins[e];
    s = __reduce_add_sync(0xffffffffu, s);
    if (lane == 0) chunk[warp] = s;
    __syncthreads();
    if (warp == 0) {
        const uint32_t v = chunk[lane];
        uint32_t x = v;
#pragma unroll
        for (uint32_t o = 1; o < 32u; o <<= 1) {
            const uint32_t y = __shfl_up_sync(0xffffffffu, x, o);
            if (lane >= o) x += y;
        }
        chunk[lane] = x - v;
    }
    __syncthreads();
    uint32_t off = chunk[warp];
    for (uint32_t r = b0; r < b1; r += 32u) {
        const uint32_t e = r + lane;
        const uint32_t v = e < b1 ? bins[e] : 0u;
        uint32_t x = v;
#pragma unroll
        for (uint32_t o = 1; o < 32u; o <<= 1) {
            const uint32_t y = __shfl_up_sync(0xffffffffu, x, o);
            if (lane >= o) x += y;
        }
        if (e < b1) {
            bins[nk + e] = off + x - v;
            bins[e] = 0u;
        }
        off += __shfl_sync(0xffffffffu, x, 31);
    }
}

// out = the *count items of `list` (null: 0, 1, 2, ...) ordered by keys[item] (any order within a
// key: every ray's result depends on its own item only).
__global__ void k_key_scatter(const uint32_t* __restrict__ list, const uint32_t* __restrict__ keys, uint32_t* cursors,
                              const uint32_t* count, uint32_t* out) {
    const uint32_t n = *(volatile const uint32_t*)count;
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const uint32_t item = list ? list[i] : i;
        out[atomicAdd(&cursors[keys[item]], 1u)] = item;
    }
}

// ---- trace: the nearest hit of every active path, the any hit of every shadow ray --------------------
// An unblocked shadow ray adds its light to its path.
__device__ __forceinline__ void shadow_unblocked(const PathBuffers& P, uint32_t i) {
    const float4 c = P.sh_c[i];
    const uint32_t slot = __float_as_uint(c.w);
    float4 s = P.sum[slot];
    s.x = s.x + c.x; s.y = s.y + c.y; s.z = s.z + c.z;
    P.sum[slot] = s;
}
// A shadow ray on its way through cut-outs and thin walls (integrator/mod.rs:629-690): nearest hits
// along the ray; a passable surface multiplies what arrives by its straight transmittance (a thin
// wall's) times its opacity plus 1 - opacity, and the ray goes on from just behind it, up to 32
// crossings (MAX_SHADOW_CROSSINGS); any other surface blocks it.
struct ShadowWalk {
    V3 o;  // where its present part starts
    float travelled;
    Rgb keep;
    uint32_t crossings;
};
enum : int { WALK_BLOCKED, WALK_ARRIVES, WALK_GOES_ON };
// The walk's surface at (inst, tri, t): blocked, at the light, or on from behind it for up to `next`.
__device__ __noinline__ int shadow_crossing(const SceneDev& S, ShadowWalk& walk, V3 d, float t_max, uint32_t inst, uint32_t tri, float t, float& next) {
    if (inst >= S.n_instances || !S.instances[inst].passable) return WALK_BLOCKED;
    HitInfo h;
    const DevInstance* I = nullptr;
    if (!hit_details(S, walk.o, d, 1.0e-3f, f_inf(), inst, tri, t, h, I)) return WALK_BLOCKED;
    const uint32_t m = I->material;
    const float opacity = rclamp(S.materials[m].opacity, 0.0f, 1.0f);
    walk.keep = walk.keep * (straight_transmittance(S.bsdfs[2 * m], dot(h.geometric, d)) * opacity + splat(1.0f - opacity));
    if (rmax(rmax(walk.keep.r, walk.keep.g), walk.keep.b) <= 0.0f) return WALK_BLOCKED;
    const V3 origin = offset_origin(h.point, -h.geometric);
    walk.travelled += dot(origin - walk.o, d);
    next = t_max - walk.travelled;
    if (next != next || next <= 1.0e-3f) return WALK_ARRIVES;
    walk.o = origin;
    return ++walk.crossings < 32u ? WALK_GOES_ON : WALK_BLOCKED;
}
// A walked shadow ray that arrives adds its light, less what it crossed, to its path.
__device__ __forceinline__ void shadow_arrived(const SceneDev& S, const PathBuffers& P, float4 c4, bool indirect, Rgb keep) {
    if (!(peak(keep) > 0.0f)) return;
    const uint32_t slot = __float_as_uint(c4.w);
    Rgb c = rgb(c4.x, c4.y, c4.z) * keep;
    if (indirect && S.clamp_indirect > 0.0f) {
        const float p = rmax(rmax(c.r, c.g), c.b);
        if (p > S.clamp_indirect) c = c * (S.clamp_indirect / p);
    }
    float4 s4 = P.sum[slot];
    s4.x = s4.x + c.r; s4.y = s4.y + c.g; s4.z = s4.z + c.b;
    P.sum[slot] = s4;
}
// Persistent warps over the extension queue of round `round` (EXTEND, SHADOW_TOO) and the shadow rays
// of the round before it (SHADOW_TOO) or of `round` itself (SHADOW): a lane whose ray has finished
// takes the next one (one atomic per warp on the round's position) while the rest of the warp keeps
// traversing, so no lane idles until the slowest ray of its warp is done. In a thin round only
// lanes_for lanes take rays. A round's shadow rays and the next round's extension rays depend on
// nothing of each other (a path's radiance waits for its shadow ray only at the next vertex), so one
// launch traces both: its end, where the slowest rays keep a few warps busy, comes once.
// WALK and WALK_TOO: as SHADOW and SHADOW_TOO where surfaces are passable; a lane walks its shadow ray
// on from crossing to crossing (against a launch a round with a thread per ray, whose warps wait for
// their longest walk: studio frame 800x600 of glass and cut-outs 16.0 to 15.1 ms; 6 blocks an SM
// 15.4).
// `order`: the active queue in the order to trace it (the round's queue, or its ray-sorted copy);
// `perm` (may be null): the shadow queue in the order to trace it.
enum TraceRays { EXTEND, SHADOW, SHADOW_TOO, WALK, WALK_TOO };
template <TraceRays RAYS>
__global__ void __launch_bounds__(TRACE_THREADS, RTG_TRACE_BLOCKS(RAYS != EXTEND && RAYS != SHADOW)) k_trace(const __grid_constant__ SceneDev S, PathBuffers P, uint32_t round, const uint32_t* __restrict__ order,
                                         const uint32_t* __restrict__ perm, uint32_t tail) {
    __shared__ uint64_t s_stack[SHORT_STACK * TRACE_THREADS];
    uint64_t deep[STACK_CAP - SHORT_STACK];
    SplitStack stack{s_stack + threadIdx.x, deep, TRACE_THREADS};
    constexpr bool WALKS = RAYS == WALK || RAYS == WALK_TOO, TOO = RAYS == SHADOW_TOO || RAYS == WALK_TOO, ALONE = RAYS == SHADOW || RAYS == WALK;
    constexpr TraceMode MODE = RAYS == EXTEND || WALKS ? TRACE_NEAREST : (RAYS == SHADOW ? TRACE_ANY : TRACE_EITHER);
    const uint32_t paths = ALONE ? 0 : round_paths(P, round, tail);
    const uint32_t shadows = RAYS == EXTEND ? 0 : *(volatile uint32_t*)&P.counters[round_counter(ALONE ? round : round - 1, COUNT_SHADOW)];
    const uint32_t n = paths + shadows;
    if (n == 0) return;
    uint32_t* position = &P.counters[round_counter(round, ALONE ? NEXT_SHADOW : NEXT_PATH)];
    uint32_t* bins = P.bins + KEY_BINS * (round & 1);
    const uint32_t lane = threadIdx.x & 31u, lanes = lanes_for(n), enough = min(lanes, (uint32_t)RTG_REFILL_MIN);
    uint32_t err = 0, ray = 0;  // the path's slot or the shadow ray
    bool busy = false, drained = false;
    Trav T;
    ShadowWalk walk;
    for (;;) {
        bool done = false, hit = false;
        if (!drained) {
            const uint32_t idle = __ballot_sync(0xffffffffu, !busy && lane < lanes);
            if ((uint32_t)__popc(idle) >= enough) {
                const int leader = __ffs((int)idle) - 1;
                uint32_t base = 0;
                if ((int)lane == leader) base = atomicAdd(position, (uint32_t)__popc(idle));
                base = __shfl_sync(0xffffffffu, base, leader);
                if (base + (uint32_t)__popc(idle) >= n) drained = true;
                const uint32_t i = base + (uint32_t)__popc(idle & ((1u << lane) - 1u));
                if (!busy && lane < lanes && i < n) {
                    float4 o, d;
                    bool camera = false, sees = true;
                    float tmax = f_inf();
                    if (RAYS == EXTEND || (TOO && i < paths)) {
                        ray = order[i];
                        load_pair(P.o, ray, o, d);
                        const uint32_t pf = __float_as_uint(o.w);
                        camera = (pf & PF_PRIMARY) != 0;
                        sees = !(pf & PF_NOTHING);
                        T.any = false;
                    } else {
                        ray = perm ? perm[i - paths] : i - paths;
                        o = P.sh_o[ray];
                        d = P.sh_d[ray];
                        tmax = o.w;
                        T.any = true;
                        if (WALKS) walk = {v3(o.x, o.y, o.z), 0.0f, splat(1.0f), 0u};
                    }
                    busy = sees && trav_init(S, T, v3(o.x, o.y, o.z), v3(d.x, d.y, d.z), 1.0e-3f, tmax, camera);
                    done = !busy;
                }
            }
        }
        const auto src = [&](V3& ro, V3& rd) {
            const bool any = RAYS != EXTEND && (ALONE || T.any);
            const float4 o = any ? P.sh_o[ray] : P.o[ray], d = any ? P.sh_d[ray] : P.d[ray];
            ro = WALKS && any ? walk.o : v3(o.x, o.y, o.z);
            rd = v3(d.x, d.y, d.z);
        };
        if (busy && !trav_at_leaf(T)) done = trav_node<MODE, true>(S, T, 1.0e-3f, stack, &err, hit, src);
        busy = busy && !done;
        if (busy && trav_at_leaf(T)) done = trav_leaf<MODE, true>(S, T, 1.0e-3f, stack, &err, hit, src);
        busy = busy && !done;
        if (WALKS && done && (ALONE || T.any)) {
            float next = 0.0f;
            const float4 d4 = P.sh_d[ray];
            const int crossed = hit ? shadow_crossing(S, walk, v3(d4.x, d4.y, d4.z), P.sh_o[ray].w, T.best_i, T.best_k, T.best_t, next) : WALK_ARRIVES;
            busy = crossed == WALK_GOES_ON && trav_init(S, T, walk.o, v3(d4.x, d4.y, d4.z), 1.0e-3f, next, false);
            if (!busy && crossed != WALK_BLOCKED) shadow_arrived(S, P, P.sh_c[ray], d4.w != 0.0f, walk.keep);
        } else if (done) {
            if (RAYS == SHADOW || (RAYS == SHADOW_TOO && T.any)) {
                if (!hit) shadow_unblocked(P, ray);
            } else {
                P.hit[ray] = hit ? make_uint4(T.best_i, T.best_k, __float_as_uint(T.best_t), 1u)
                                 : make_uint4(0xffffffffu, 0xffffffffu, 0u, 0u);
                const uint32_t key = material_key(S, hit, T.best_i);
                P.key[ray] = key;
                warp_count(bins, key);
            }
        }
        if (drained && !__any_sync(0xffffffffu, busy)) break;
    }
    if (err) atomicOr(&P.counters[3], err);
}

// ---- the order of shading ------------------------------------------------------------------------
// `out` = the round's n paths of `in` ordered by material key (the order inside a key does not
// matter: every path's result depends on its own slot only). Each block orders the next SORT_CHUNK
// of them in shared memory, takes its part of every key's run with one atomic, and writes the runs
// coalesced; the runs' starts it sums itself from the histogram k_trace left. Sorting only within
// the chunks a shade block reads would save the pass but not pay: with all blocks in the same few
// materials at a time the kernel's instructions stay in the caches (1080p frame, chunks of 512, 1024
// and 2048: 254, 231 and 213 ms; whole queue 193 ms). Against a pass with an atomic per warp and key
// after a one-thread prefix: 11.1 to 1.8 ms of the 1080p frame's 13 rounds.
constexpr uint32_t SORT_THREADS = 256, SORT_PER = 8, SORT_CHUNK = SORT_THREADS * SORT_PER;
static_assert(SORT_THREADS == MATERIAL_KEYS, "a thread per key");
__device__ __forceinline__ uint32_t block_prefix(uint32_t v, uint32_t* s_warp) {  // exclusive, over SORT_THREADS
    const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
    uint32_t x = v;
#pragma unroll
    for (uint32_t o = 1; o < 32u; o <<= 1) {
        const uint32_t y = __shfl_up_sync(0xffffffffu, x, o);
        if (lane >= o) x += y;
    }
    if (lane == 31u) s_warp[warp] = x;
    __syncthreads();
    uint32_t before = x - v;
    for (uint32_t w = 0; w < warp; ++w) before += s_warp[w];
    __syncthreads();
    return before;
}
__global__ void __launch_bounds__(SORT_THREADS) k_material_sort(PathBuffers P, uint32_t round, const uint32_t* __restrict__ in, uint32_t* __restrict__ out,
                                                                 uint32_t tail) {
    __shared__ uint32_t s_slot[SORT_CHUNK], s_to[SORT_CHUNK], s_count[MATERIAL_KEYS], s_run[MATERIAL_KEYS], s_warp[SORT_THREADS / 32];
    const uint32_t n = round_paths(P, round, tail), tid = threadIdx.x;
    uint32_t* bins = P.bins + KEY_BINS * (round & 1);
    uint32_t* cursors = bins + MATERIAL_KEYS;
    if (blockIdx.x * SORT_CHUNK >= n) return;
    const uint32_t run = block_prefix(bins[tid], s_warp);  // where this thread's key starts in `out`
    for (uint32_t base = blockIdx.x * SORT_CHUNK; base < n; base += gridDim.x * SORT_CHUNK) {
        const uint32_t m = min(SORT_CHUNK, n - base);
        s_count[tid] = 0;
        __syncthreads();
        uint32_t slot[SORT_PER], at[SORT_PER];  // at: the key, and above it the place among the chunk's
#pragma unroll
        for (uint32_t j = 0; j < SORT_PER; ++j) {
            const uint32_t e = j * SORT_THREADS + tid;
            if (e < m) slot[j] = in[base + e];
        }
#pragma unroll
        for (uint32_t j = 0; j < SORT_PER; ++j)
            if (j * SORT_THREADS + tid < m) at[j] = P.key[slot[j]];
#pragma unroll
        for (uint32_t j = 0; j < SORT_PER; ++j)
            if (j * SORT_THREADS + tid < m) at[j] |= atomicAdd(&s_count[at[j]], 1u) << 8;
        __syncthreads();
        const uint32_t count = s_count[tid];
        const uint32_t local = block_prefix(count, s_warp);
        s_count[tid] = local;
        if (count) s_run[tid] = run + atomicAdd(&cursors[tid], count) - local;
        __syncthreads();
#pragma unroll
        for (uint32_t j = 0; j < SORT_PER; ++j)
            if (j * SORT_THREADS + tid < m) {
                const uint32_t key = at[j] & 255u, e = s_count[key] + (at[j] >> 8);
                s_slot[e] = slot[j];
                s_to[e] = s_run[key];
            }
        __syncthreads();
        for (uint32_t e = tid; e < m; e += SORT_THREADS) out[s_to[e] + e] = s_slot[e];
        __syncthreads();
    }
}
// Calls f(slot) for the n paths of `order`, a path per lane (of whole warps also in thin rounds:
// the paths of one material share their code). The round's key bins, read for the last time before,
// are cleared for the next round but one.
template <class F>
__device__ __forceinline__ void for_each_path(const PathBuffers& P, const uint32_t* __restrict__ order, uint32_t n, uint32_t round, F f) {
    if (blockIdx.x == 0)
        for (uint32_t k = threadIdx.x; k < KEY_BINS; k += blockDim.x) P.bins[KEY_BINS * (round & 1) + k] = 0;
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) f(order[i]);
}

// ---- shade: one vertex of every active path ----------------------------------------------------------
// One vertex of the path in `slot` with the scene constants S and lights L; xyi(x, y, index) gives
// the path's pixel and sample index (the sampler's key).
// With P.rbins set, each surviving path's next ray gets its coherence key (in P.key) and is counted
// in the histogram; with P.sbins set, each shadow ray likewise (in P.sh_key).
// PLAIN: the scene is plain (SceneDev::plain); what it cannot hold falls away from the code.
// With `tail` (the tail kernel), the shadow ray goes to *tail instead of the shadow queue and the
// surviving path to no queue. Returns whether the path goes on.
struct TailShadow {
    bool on;
    float4 o, d, c;
};
template <bool PLAIN, class XYI>
__device__ __forceinline__ bool shade_slot(const SceneDev& S, const LightsDev& L, const PathBuffers& P, const RaySort& R, uint32_t slot, uint32_t round,
                                           XYI xyi, uint32_t& rays_local, uint32_t& shadow_local, TailShadow* tail = nullptr) {
    float4 o4, d4, thr4, sum;
    load_pair(P.o, slot, o4, d4);
    load_pair(P.thr, slot, thr4, sum);
    uint4 hit;
    float4 sel4;
    load_vertex(P, slot, hit, sel4);
    uint32_t flags = __float_as_uint(o4.w);
    const uint32_t bounce = (flags & PF_BOUNCE_MASK) >> PF_BOUNCE_SHIFT;
    V3 ro = v3(o4.x, o4.y, o4.z), rd = v3(d4.x, d4.y, d4.z);
    float offset = sum.w, pdf = d4.w;
    bool has_pdf = (flags & PF_HAS_PDF) != 0, primary = (flags & PF_PRIMARY) != 0;
    Rgb thr = rgb(thr4.x, thr4.y, thr4.z);
    float alpha = thr4.w;
    rays_local += 1;
    float t_geometry = hit.w ? __uint_as_float(hit.z) : f_inf();
    // floor_t (integrator/mod.rs:493)
    float t_floor = f_inf();
    if (!PLAIN && S.floor_mode == 1 && rd.z != 0.0f && !(flags & PF_NOTHING)) {
        float t = (S.floor_z - ro.z) / rd.z;
        if (t > 1.0e-3f && t < f_inf()) t_floor = t;
    }
    float t_nearest = rmin(t_geometry, t_floor);
    if (!PLAIN && (flags & PF_MEDIUM) && finitef(t_nearest)) {
        const DevMaterial& mm = S.materials[P.medium[slot]];
        thr = thr * rgb(fexp(-mm.sigma[0] * t_nearest), fexp(-mm.sigma[1] * t_nearest), fexp(-mm.sigma[2] * t_nearest));
    }
    Sel from;
    from.p = v3(sel4.x, sel4.y, sel4.z);
    from.by_flux = !(L.per_point && L.n_entries > 0);
    from.total = sel4.w;
    Rgb crossed = crossed_from<PLAIN>(L, ro, rd, 1.0e-3f, t_nearest, has_pdf, pdf, from, offset);
    add_clamped(sum, thr * crossed, bounce >= 2, S.clamp_indirect);
    bool alive = false;
    do {
        if (t_nearest == f_inf()) {
            if (primary && S.background == 0) {
                Rgb seen = escaped<PLAIN>(L, rd, false, 0.0f, from);
                Rgb c = thr * (S.exterior == 1.0f ? seen : seen * S.exterior);
                sum.x = sum.x + c.r; sum.y = sum.y + c.g; sum.z = sum.z + c.b;
            } else if (primary && (S.background == 1 || (!PLAIN && S.background == 3))) {
                uint32_t x, y, index;
                xyi(x, y, index);
                float su, sv;
                screen_of(S, c_sobol, x, y, index, su, sv);
                Rgb c = thr * backdrop(S, su, sv);
                sum.x = sum.x + c.r; sum.y = sum.y + c.g; sum.z = sum.z + c.b;
            } else if (primary && S.background == 2) {
                alpha = peak(crossed) > 0.0f ? 1.0f : 0.0f;
            } else {
                add_clamped(sum, thr * escaped<PLAIN>(L, rd, has_pdf, pdf, from), bounce >= 2, S.clamp_indirect);
            }
            break;
        }
        V3 s_point, s_hit, s_normal, s_geom;
        bool s_inst = false, s_outside = true;
        uint32_t inst = 0;
        const DevInstance* I = nullptr;
        const DevMaterial* mat = nullptr;
        if (!PLAIN && t_floor < t_geometry) {
            V3 pp = ro + rd * t_floor;
            V3 point = v3(pp.x, pp.y, S.floor_z);
            V3 nn = v3(0.0f, 0.0f, rd.z < 0.0f ? 1.0f : -1.0f);
            s_point = point; s_hit = point; s_normal = nn; s_geom = nn;
        } else {
            HitInfo h;
            if (!hit_details<PLAIN>(S, ro, rd, 1.0e-3f, f_inf(), hit.x, hit.y, __uint_as_float(hit.z), h, I)) break;
            // bevel.rs:232 shading_point without a bevel
            V3 ng = h.geometric, nrm = h.normal;
            if (dot(nrm, ng) < 0.0f) nrm = -nrm;
            if (dot(nrm, rd) >= -1.0e-4f) nrm = ng;
            s_point = terminator_point(S, I, h);
            s_hit = h.point;
            s_normal = nrm;
            s_geom = ng;
            s_inst = true;
            inst = hit.x;
            s_outside = h.outside;
            mat = S.materials + I->material;
            if (!PLAIN && mat->kind == MATERIAL_EMISSIVE) {
                // A BSDF-sampled ray that finds a mesh light weighs it against the light's own
                // sample (integrator/mod.rs:1556); other emitters and camera rays weigh 1.
                if (h.front || !(I->flags & 1u)) {
                    const float wgt = has_pdf ? emitter_weight(L, I->emitter, pdf, from, offset + t_geometry, dot(ng, rd)) : 1.0f;
                    add_clamped(sum, thr * rgb(mat->emission[0], mat->emission[1], mat->emission[2]) * wgt, bounce >= 2, S.clamp_indirect);
                }
                break;
            }
            // A cut-out lets the ray through with probability 1 - opacity: no vertex, the same
            // direction, density and selection; the path goes back to the extension queue
            // (integrator/mod.rs:1571).
            const uint32_t cut = (flags & PF_CUT_MASK) >> PF_CUT_SHIFT;
            if (!PLAIN && S.any_cutout && mat->opacity < 1.0f && cut < MAX_CUTOUTS) {
                uint32_t x, y, index;
                xyi(x, y, index);
                const float u = sample_at(S, c_sobol, sample_key(S, x, y, index), index, cutout_dim(bounce, cut));
                flags = (flags & ~PF_CUT_MASK) | ((cut + 1u) << PF_CUT_SHIFT);
                if (u >= rmax(mat->opacity, 0.0f)) {
                    const V3 o2 = offset_origin(h.point, -ng);
                    offset += dot(o2 - ro, rd);
                    P.o[slot] = make_float4(o2.x, o2.y, o2.z, __uint_as_float(flags));
                    alive = true;
                    break;
                }
            }
        }
        if (bounce >= S.max_depth) break;
        const Bsdf& b = S.bsdfs[PLAIN || mat ? 2 * I->material + (s_outside ? 0 : 1) : 2 * S.n_materials];
        // Prepared::frame (integrator/mod.rs:833)
        Frame fr = frame_from_normal(s_normal);
        if (!PLAIN && s_inst && I->tangent_on) {
            V3 cands[2] = {cross(ld3(I->tan_axis), s_point - ld3(I->tan_centre)), ld3(I->tan_x)};
            for (int k = 0; k < 2; ++k) {
                V3 t = cands[k] - s_normal * dot(s_normal, cands[k]);
                if (len2(t) > 1.0e-12f) {
                    V3 xx = normalize(t);
                    fr.x = xx; fr.y = cross(s_normal, xx); fr.z = s_normal;
                    break;
                }
            }
        }
        V3 wo = to_local(fr, -rd);
        if (wo.z <= 0.0f) break;  // below the surface the BSDF is zero and has no samples
        V3 ng = s_geom;
        V3 origin = offset_origin(s_point, ng);
        uint32_t dims = bounce_dim(bounce);
        uint32_t x, y, index;
        xyi(x, y, index);
        uint64_t key = sample_key(S, x, y, index);
        // Next-event estimation: one light; the shadow ray goes to the shadow queue.
        const BsdfWo bo = bsdf_wo<PLAIN>(S.energy, b, wo);
        const LobeWeights lobes = lobe_weights<PLAIN>(b, bo, wo);
        float weights[SEL_KEPT];
        Sel selection = select_at<PLAIN>(L, s_point, weights);
        LightSample ls;
        if (sample_light<PLAIN>(L, selection, weights, sample_at(S, c_sobol, key, index, dims + OFF_LIGHT_SELECT), sample_at(S, c_sobol, key, index, dims + OFF_LIGHT),
                         sample_at(S, c_sobol, key, index, dims + OFF_LIGHT + 1), ls)) {
            V3 wi = to_local(fr, ls.wi);
            const bool mis = ls.glossy && !ls.delta;
            Rgb f;
            float bsdf_density = 0.0f;
            bsdf_eval_pdf<PLAIN>(S.energy, b, bo, &lobes, wo, wi, ls.glossy ? LOBES_ALL : LOBES_DIFFUSE, f, mis ? &bsdf_density : nullptr);
            if (peak(f) > 0.0f) {
                V3 from_p = wi.z < 0.0f ? offset_origin(s_hit, -ng) : origin;
                float weight = mis ? power_heuristic(ls.pdf, bsdf_density) : 1.0f;
                Rgb c = thr * f * ls.radiance * (absf(wi.z) * weight / ls.pdf);
                bool finite_c = finitef(c.r) && finitef(c.g) && finitef(c.b);
                // The clamp applies to what arrives: after the shadow walk when it may attenuate.
                const bool walk = !PLAIN && ls.shadow && S.any_passable;
                if (finite_c && bounce >= 1 && S.clamp_indirect > 0.0f && !walk) {
                    float p = rmax(rmax(c.r, c.g), c.b);
                    if (p > S.clamp_indirect) c = c * (S.clamp_indirect / p);
                }
                if (!ls.shadow) {
                    if (finite_c) { sum.x = sum.x + c.r; sum.y = sum.y + c.g; sum.z = sum.z + c.b; }
                } else {
                    shadow_local += 1;
                    float tmax = finitef(ls.distance) ? ls.distance * (1.0f - 1.0e-4f) : f_inf();
                    bool floor_blocks = false;
                    if (!PLAIN && S.floor_mode == 1 && ls.wi.z != 0.0f) {
                        float t = (S.floor_z - from_p.z) / ls.wi.z;
                        floor_blocks = t > 1.0e-3f && t < tmax;
                    }
                    if (finite_c && !floor_blocks) {
                        const float4 so = make_float4(from_p.x, from_p.y, from_p.z, tmax);
                        const float4 sd = make_float4(ls.wi.x, ls.wi.y, ls.wi.z, bounce >= 1 ? 1.0f : 0.0f);  // w: indirect
                        const float4 sc = make_float4(c.r, c.g, c.b, __uint_as_float(slot));
                        if (tail) {
                            tail->on = true;
                            tail->o = so;
                            tail->d = sd;
                            tail->c = sc;
                        } else {
                            uint32_t k = atomicAdd(&P.counters[round_counter(round, COUNT_SHADOW)], 1u);
                            P.sh_o[k] = so;
                            P.sh_d[k] = sd;
                            P.sh_c[k] = sc;
                            if (P.sbins) {
                                const uint32_t sk = ray_key(R, from_p, ls.wi);
                                P.sh_key[k] = sk;
                                atomicAdd(&P.sbins[sk], 1u);
                            }
                        }
                    }
                }
            }
        }
        // The next direction.
        BsdfSample bs;
        if (!bsdf_sample<PLAIN>(S.energy, b, bo, lobes, wo, sample_at(S, c_sobol, key, index, dims + OFF_BSDF), sample_at(S, c_sobol, key, index, dims + OFF_BSDF + 1), bs))
            break;
        bool transmitted = bs.wi.z < 0.0f;
        V3 wi = !PLAIN && bs.straight ? rd : normalize(to_world(fr, bs.wi));
        if (transmitted) {
            if (dot(wi, ng) >= 0.0f) break;
        } else if (dot(wi, ng) <= 0.0f) {
            break;
        }
        thr = thr * bs.weight;
        if (bounce >= 2) {
            float survive = rclamp(peak(thr), 0.05f, 1.0f);
            if (sample_at(S, c_sobol, key, index, dims + OFF_ROULETTE) >= survive) break;
            thr = thr / survive;
        }
        float pk = peak(thr);
        if (!(pk > 0.0f && finitef(pk))) break;
        V3 next_origin = transmitted ? offset_origin(s_hit, -ng) : origin;
        if (!PLAIN && bs.straight) {
            offset += dot(next_origin - ro, rd);
        } else {
            flags |= PF_HAS_PDF;
            flags &= ~PF_PRIMARY;
            pdf = bs.pdf;
            P.sel[slot] = make_float4(s_point.x, s_point.y, s_point.z, selection.total);
            offset = 0.0f;
            if (!PLAIN && transmitted) {
                if (s_outside && mat && mat->has_medium) {
                    flags |= PF_MEDIUM;
                    P.medium[slot] = I->material;
                } else {
                    flags &= ~PF_MEDIUM;
                }
            }
        }
        flags = (flags & ~PF_BOUNCE_MASK) | ((bounce + 1u) << PF_BOUNCE_SHIFT);
        store_pair(P.o, slot, make_float4(next_origin.x, next_origin.y, next_origin.z, __uint_as_float(flags)), make_float4(wi.x, wi.y, wi.z, pdf));
        alive = true;
    } while (false);
    sum.w = offset;
    store_pair(P.thr, slot, make_float4(thr.r, thr.g, thr.b, alpha), sum);
    if (alive && !tail) {
        uint32_t k = atomicAdd(&P.counters[round_counter(round + 1, COUNT_PATHS)], 1u);
        P.queue[(round + 1) & 1][k] = slot;
        if (P.rbins) {
            const float4 no = P.o[slot], nd = P.d[slot];
            const uint32_t rk = ray_key(R, v3(no.x, no.y, no.z), v3(nd.x, nd.y, nd.z));
            P.key[slot] = rk;
            atomicAdd(&P.rbins[rk], 1u);
        }
    }
    return alive;
}

// BATCH: the slots belong to the jobs of a batched wave, each with its own constants and lights.
// Eight blocks per SM (64 registers, with some spills) beat the 128 registers the compiler would
// use on its own: the kernel waits on scattered hit-detail loads, and more warps hide them.
// Instruction fetch and issue weigh as much as the loads (4,200 instructions a vertex before), so a
// vertex computes nothing twice: the BSDF's terms of wo and the half vector's are shared by value,
// density and sampling, the light weights by sum and pick, the selection's sum is kept for the next
// vertex's MIS weights, sampler columns and table cells come summed and packed from tables, and
// slots are divided by multiplication. 1080p frame 229.0 -> 210.8 ms, studio still 32.1 -> 23.9 ms,
// 512^2 fit iteration 47.3 -> 39.3 ms (the last two with the shorter node steps), films bit-equal.
// PLAIN: the variant for plain scenes (SceneDev::plain). A vertex of one still went past the code of
// every light, environment and material, and the kernel's size is what its instruction fetch stalls
// on (3.4-7.4 of some 18 stall cycles an issue): 1080p frame 210.8 -> 192.6 ms, 512^2 fit iteration
// 39.3 -> 32.8 ms. Other scenes take the general kernel, as before. At 4, 5, 6, 7, 8 and 10 blocks an
// SM the frame takes 195.4, 198.4, 199.7, 197.7, 192.7 and 202.2 ms.
// `order`: the active queue in the order to shade it (material-sorted, or as traced).
template <bool BATCH, bool PLAIN>
__global__ void __launch_bounds__(128, RTG_SHADE_MIN_BLOCKS) k_shade(const __grid_constant__ SceneDev S, const LightsDev* __restrict__ Lg, PathBuffers P, uint32_t round, WaveDesc w,
                                                  const uint32_t* __restrict__ order, RaySort R) {
    const uint32_t n = round_paths(P, round, R.tail_paths);
    uint32_t rays_local = 0, shadow_local = 0;
    for_each_path(P, order, n, round, [&](uint32_t slot) {
        if constexpr (BATCH) {
            uint32_t job, x, y, index;
            batch_slot(w, slot, job, x, y, index);
            const JobDev& J = w.jobs[job];
            shade_slot<PLAIN>(J.S, *J.lights, P, R, slot, round, [&](uint32_t& xx, uint32_t& yy, uint32_t& ii) { xx = x; yy = y; ii = index; },
                       rays_local, shadow_local);
        } else {
            shade_slot<PLAIN>(S, *Lg, P, R, slot, round, [&](uint32_t& xx, uint32_t& yy, uint32_t& ii) { wave_slot(w, slot, xx, yy, ii); },
                       rays_local, shadow_local);
        }
    });
    // Ray counts: camera + extension rays in rays[0], shadow rays in rays[1]; one atomic per warp.
    uint32_t total = __reduce_add_sync(0xffffffffu, rays_local);
    uint32_t shadows = __reduce_add_sync(0xffffffffu, shadow_local);
    if ((threadIdx.x & 31) == 0 && total) atomicAdd(P.rays, (unsigned long long)total);
    if ((threadIdx.x & 31) == 0 && shadows) atomicAdd(P.rays + 1, (unsigned long long)shadows);
}

// ---- the section view: k_trace through the section's queries (geometry/section.rs) --------------------
// One ray per thread: a query may be several traversals (the kept part, the cap's probe beyond the
// plane, the studio on the removed side), so the lane refill of k_trace does not apply. Launched
// instead of it for a scene with a section; they write the same records (a cap is a hit with
// triangle CAP_TRIANGLE).
__global__ void __launch_bounds__(TRACE_THREADS) k_extend_section(const __grid_constant__ SceneDev S, PathBuffers P, uint32_t round, const uint32_t* __restrict__ order, uint32_t tail) {
    __shared__ uint64_t s_stack[SHORT_STACK * TRACE_THREADS];
    uint64_t deep[STACK_CAP - SHORT_STACK];
    SplitStack stack{s_stack + threadIdx.x, deep, TRACE_THREADS};
    const uint32_t n = round_paths(P, round, tail);
    uint32_t err = 0;
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const uint32_t slot = order[i];
        const float4 o = P.o[slot], d = P.d[slot];
        const uint32_t pf = __float_as_uint(o.w);
        TraceResult res;
        const bool got = !(pf & PF_NOTHING) &&
                         trace_q<false>(S, v3(o.x, o.y, o.z), v3(d.x, d.y, d.z), 1.0e-3f, f_inf(), (pf & PF_PRIMARY) != 0, res, &err, stack);
        P.hit[slot] = got ? make_uint4(res.inst, res.tri, __float_as_uint(res.t), 1u) : make_uint4(0xffffffffu, 0xffffffffu, 0u, 0u);
        const uint32_t key = material_key(S, got, got ? res.inst : 0u);
        P.key[slot] = key;
        warp_count(P.bins + KEY_BINS * (round & 1), key);
    }
    if (err) atomicOr(&P.counters[3], err);
}

__global__ void __launch_bounds__(TRACE_THREADS) k_shadow_section(const __grid_constant__ SceneDev S, PathBuffers P, uint32_t round, const uint32_t* __restrict__ perm) {
    __shared__ uint64_t s_stack[SHORT_STACK * TRACE_THREADS];
    uint64_t deep[STACK_CAP - SHORT_STACK];
    SplitStack stack{s_stack + threadIdx.x, deep, TRACE_THREADS};
    const uint32_t n = *(volatile uint32_t*)&P.counters[round_counter(round, COUNT_SHADOW)];
    uint32_t err = 0;
    for (uint32_t j = blockIdx.x * blockDim.x + threadIdx.x; j < n; j += gridDim.x * blockDim.x) {
        const uint32_t ray = perm ? perm[j] : j;
        const float4 o = P.sh_o[ray], d = P.sh_d[ray];
        TraceResult unused;
        if (!trace_q<true>(S, v3(o.x, o.y, o.z), v3(d.x, d.y, d.z), 1.0e-3f, o.w, false, unused, &err, stack)) shadow_unblocked(P, ray);
    }
    if (err) atomicOr(&P.counters[3], err);
}

// ---- shadow walks of sections and batched waves ------------------------------------------------------
// Shadow rays through cut-outs and thin walls where k_trace's walk cannot take them: each part of a
// section's walk is several queries, and in a batched wave (BATCH) each ray's job gives its
// materials. One thread per ray.
template <bool BATCH>
__global__ void __launch_bounds__(TRACE_THREADS) k_shadow_walk(const __grid_constant__ SceneDev S, PathBuffers P, uint32_t round, WaveDesc w, const uint32_t* __restrict__ perm) {
    __shared__ uint64_t s_stack[SHORT_STACK * TRACE_THREADS];
    uint64_t deep[STACK_CAP - SHORT_STACK];
    SplitStack stack{s_stack + threadIdx.x, deep, TRACE_THREADS};
    const uint32_t n = *(volatile uint32_t*)&P.counters[round_counter(round, COUNT_SHADOW)];
    uint32_t err = 0;
    for (uint32_t j = blockIdx.x * blockDim.x + threadIdx.x; j < n; j += gridDim.x * blockDim.x) {
        const uint32_t i = perm ? perm[j] : j;
        const float4 o4 = P.sh_o[i], d4 = P.sh_d[i], c4 = P.sh_c[i];
        const uint32_t slot = __float_as_uint(c4.w);
        const SceneDev* Sp = &S;
        if constexpr (BATCH) {
            uint32_t job, x, y, index;
            batch_slot(w, slot, job, x, y, index);
            Sp = &w.jobs[job].S;
        }
        const SceneDev& J = *Sp;
        const V3 d = v3(d4.x, d4.y, d4.z);
        const float t_max = o4.w;
        ShadowWalk walk = {v3(o4.x, o4.y, o4.z), 0.0f, splat(1.0f), 0u};
        float tmax = t_max;
        int crossed = WALK_GOES_ON;
        while (crossed == WALK_GOES_ON) {
            TraceResult res;
            crossed = trace_q<false>(J, walk.o, d, 1.0e-3f, tmax, false, res, &err, stack)
                          ? shadow_crossing(J, walk, d, t_max, res.inst, res.tri, res.t, tmax) : WALK_ARRIVES;
        }
        if (crossed == WALK_ARRIVES) shadow_arrived(J, P, c4, d4.w != 0.0f, walk.keep);
    }
    if (err) atomicOr(&P.counters[3], err);
}

// ---- tail: the last rounds of a wave, a path per lane -------------------------------------------------
// The wave's last launch. From the first round whose extension queue holds at most `limit` paths on,
// the other kernels do nothing, and here each lane carries its share of those paths through the
// wave's remaining rounds alone: the nearest hit (as k_trace), the vertex (shade_slot), the next
// ray; each path's arithmetic in the order the wavefront gives it, so its sum has the same bits.
// What bounds it is the chain of one path's rays and vertices, so warps work in pairs: lane for lane,
// the second warp traces the vertices' shadow rays and adds their light while the first traces the
// paths' next rays; they meet twice a vertex. Against one lane for both rays in turn: 720p viewport
// 4.60 to 4.20 ms, 617x351 crop 3.46 to 3.25, small fit 2.13 to 2.05, adaptive frame 70.3 to 68.7;
// with the shadow rays in the upper half of the same warp, whose vertices then come from twice the
// warps, the viewport gained half of that and a 256x256 frame lost 2 %. A wave whose last rounds hold few
// paths then pays one launch as long as its slowest path instead of a chain of launches, each as
// long as its slowest ray. Scenes with passable surfaces (shadow walks) and batched waves keep the
// wavefront.
template <bool PLAIN>
__global__ void __launch_bounds__(TRACE_THREADS) k_tail(const __grid_constant__ SceneDev S, const LightsDev* __restrict__ Lg, PathBuffers P, WaveDesc w, uint32_t rounds,
                                        uint32_t limit) {
    uint32_t round = TAIL_FIRST_ROUND;
    while (round < rounds && P.counters[round_counter(round, COUNT_PATHS)] > limit) ++round;
    const uint32_t n = round < rounds ? P.counters[round_counter(round, COUNT_PATHS)] : 0;
    if (n == 0) return;
    // Up to eight paths a pair run spread over all pairs; more run in full warps, which meet each
    // other's code less often (with a warp for both kinds of rays, spread against full: a 64 x 64 tile
    // 0.51 and 0.56 ms, a 720p viewport, whose tail holds up to 16,384 paths, 4.74 and 4.39 ms; up to
    // 2, 4 and 8 a pair: adaptive frame 68.7, 69.0 and 68.7 ms, tile 0.52, 0.51 and 0.51 ms).
    const uint32_t pairs = gridDim.x * (TRACE_THREADS / 64), spread = (n + pairs - 1) / pairs;
    const uint32_t rounds_left = rounds - round, lanes = spread <= 8u ? spread : 32u;
    __shared__ uint64_t s_stack[SHORT_STACK * TRACE_THREADS];
    __shared__ TailShadow s_shadow[TRACE_THREADS / 2];
    __shared__ bool s_more[TRACE_THREADS / 64];
    uint64_t deep[STACK_CAP - SHORT_STACK];
    SplitStack stack{s_stack + threadIdx.x, deep, TRACE_THREADS};
    const uint32_t* __restrict__ queue = P.queue[round & 1];
    const RaySort R;  // no coherence keys
    uint32_t err = 0, rays_local = 0, shadow_local = 0;
    const uint32_t pair = threadIdx.x >> 6, lane = threadIdx.x & 31u, first = blockIdx.x * (TRACE_THREADS / 64) + pair;
    TailShadow& sh = s_shadow[pair * 32 + lane];
    const auto meet = [&] {
        if (pair) asm volatile("bar.sync 2, 64;" ::: "memory");
        else asm volatile("bar.sync 1, 64;" ::: "memory");
    };
    static_assert(TRACE_THREADS == 128, "two pairs of warps a block");
    if (!(threadIdx.x & 32u)) {
        uint32_t i = lane < lanes ? first * lanes + lane : n, slot = 0, r = 0;
        for (bool more = true; more;) {
            if (i < n && r == 0) slot = queue[i];
            TraceResult res;
            bool got = false;
            if (i < n) {
                float4 o, d;
                load_pair(P.o, slot, o, d);
                const uint32_t pf = __float_as_uint(o.w);
                got = !(pf & PF_NOTHING) &&
                      traverse<false, true>(S, v3(o.x, o.y, o.z), v3(d.x, d.y, d.z), 1.0e-3f, f_inf(), (pf & PF_PRIMARY) != 0, res, &err, stack);
                P.hit[slot] = got ? make_uint4(res.inst, res.tri, __float_as_uint(res.t), 1u) : make_uint4(0xffffffffu, 0xffffffffu, 0u, 0u);
            }
            __syncwarp();
            meet();  // the last vertices' shadow rays have added their light
            TailShadow next;
            next.on = false;
            if (i < n) {
                const bool alive = shade_slot<PLAIN>(S, *Lg, P, R, slot, round, [&](uint32_t& xx, uint32_t& yy, uint32_t& ii) { wave_slot(w, slot, xx, yy, ii); },
                                                     rays_local, shadow_local, &next);
                if (alive && r + 1 < rounds_left) {
                    ++r;
                } else {
                    r = 0;
                    i += pairs * lanes;
                }
            }
            if (next.on) sh = next;
            else sh.on = false;
            more = __any_sync(0xffffffffu, i < n || next.on);
            if (lane == 0) s_more[pair] = more;
            __syncwarp();
            meet();
        }
    } else {
        TailShadow ray;
        ray.on = false;
        for (bool more = true; more;) {
            if (ray.on) {
                TraceResult unused;
                if (!traverse<true, true>(S, v3(ray.o.x, ray.o.y, ray.o.z), v3(ray.d.x, ray.d.y, ray.d.z), 1.0e-3f, ray.o.w, false, unused, &err, stack)) {
                    float4* const to = &P.sum[__float_as_uint(ray.c.w)];  // shadow_unblocked's addition
                    float4 sum = *to;
                    sum.x = sum.x + ray.c.x;
                    sum.y = sum.y + ray.c.y;
                    sum.z = sum.z + ray.c.z;
                    *to = sum;
                }
            }
            __syncwarp();
            meet();
            meet();  // the vertices' next shadow rays are there
            ray = sh;
            more = s_more[pair];
        }
    }
    __syncwarp();
    uint32_t total = __reduce_add_sync(0xffffffffu, rays_local);
    uint32_t shadows = __reduce_add_sync(0xffffffffu, shadow_local);
    if ((threadIdx.x & 31) == 0 && total) atomicAdd(P.rays, (unsigned long long)total);
    if ((threadIdx.x & 31) == 0 && shadows) atomicAdd(P.rays + 1, (unsigned long long)shadows);
    if (err) atomicOr(&P.counters[3], err);
}

// ---- accumulate: film += each pixel's samples in sample-index order (image.rs:82) -------------------------
// A sample's radiance times its camera weight (render.rs:465): white, or black for a panoramic
// camera's (`dark`) sample that sees nothing.
__device__ __forceinline__ float4 sample_sum(const PathBuffers& P, uint32_t slot, bool dark) {
    const float4 c = P.sum[slot];
    if (!dark || !(__float_as_uint(P.o[slot].w) & PF_NOTHING)) return c;
    return make_float4(c.x * 0.0f, c.y * 0.0f, c.z * 0.0f, c.w);
}
// Film pixel (x, y) += the ns samples in slots slot0, slot0 + stride, ..., in that order
// (Film::splat_alpha, image.rs:82).
__device__ __forceinline__ void accumulate_pixel(const FilmDev& F, uint32_t x, uint32_t y, const PathBuffers& P, uint32_t slot0, uint32_t stride,
                                                 uint32_t ns, bool dark) {
    if (x < F.ox || y < F.oy || x - F.ox >= F.w || y - F.oy >= F.h) return;
    size_t fi = (size_t)(y - F.oy) * F.w + (x - F.ox);
    float r = F.rgb[3 * fi], g = F.rgb[3 * fi + 1], b = F.rgb[3 * fi + 2];
    float wt = F.weight[fi], al = F.alpha[fi], l2 = F.lum2[fi];
    for (uint32_t s = 0; s < ns; ++s) {
        uint32_t slot = slot0 + s * stride;
        float4 c = sample_sum(P, slot, dark);
        r = r + c.x; g = g + c.y; b = b + c.z;
        wt = wt + 1.0f;
        al = al + P.thr[slot].w;
        float l = luminance(rgb(c.x, c.y, c.z));
        l2 = l2 + l * l;
    }
    F.rgb[3 * fi] = r; F.rgb[3 * fi + 1] = g; F.rgb[3 * fi + 2] = b;
    F.weight[fi] = wt; F.alpha[fi] = al; F.lum2[fi] = l2;
}

__global__ void k_accumulate(WaveDesc w, PathBuffers P, FilmDev F) {
    uint32_t npix = w.w * w.h;
    uint32_t ns = w.n / npix;
    for (uint32_t p = blockIdx.x * blockDim.x + threadIdx.x; p < npix; p += gridDim.x * blockDim.x) {
        const uint32_t x = w.x0 + p % w.w, y = w.y0 + p / w.w;
        if (w.edge && w.edge[(size_t)y * w.edge_stride + x]) continue;  // splatted by the edge waves
        accumulate_pixel(F, x, y, P, p, npix, ns, w.dark);
    }
}

// An edge wave: per edge pixel and sample index, the mean of its k samples (summed in order,
// times 1 / k), splatted once (render.rs:477-488), sample indices in order.
__global__ void k_accumulate_edges(WaveDesc w, PathBuffers P, FilmDev F) {
    const uint32_t k = w.ek, ns = w.n / (w.ne * k);
    const float inv = 1.0f / (float)k;
    for (uint32_t e = blockIdx.x * blockDim.x + threadIdx.x; e < w.ne; e += gridDim.x * blockDim.x) {
        const uint32_t x = w.epix[e] & 0xffffu, y = w.epix[e] >> 16;
        if (x < F.ox || y < F.oy || x - F.ox >= F.w || y - F.oy >= F.h) continue;
        const size_t fi = (size_t)(y - F.oy) * F.w + (x - F.ox);
        float r = F.rgb[3 * fi], g = F.rgb[3 * fi + 1], b = F.rgb[3 * fi + 2];
        float wt = F.weight[fi], al = F.alpha[fi], l2 = F.lum2[fi];
        for (uint32_t s = 0; s < ns; ++s) {
            float sr = 0.0f, sg = 0.0f, sb = 0.0f, cov = 0.0f;
            for (uint32_t j = 0; j < k; ++j) {
                const uint32_t slot = (s * w.ne + e) * k + j;
                const float4 c = sample_sum(P, slot, w.dark);
                sr = sr + c.x; sg = sg + c.y; sb = sb + c.z;
                cov = cov + P.thr[slot].w;
            }
            const Rgb m = rgb(sr * inv, sg * inv, sb * inv);
            r = r + m.r; g = g + m.g; b = b + m.b;
            wt = wt + 1.0f;
            al = al + cov * inv;
            const float l = luminance(m);
            l2 = l2 + l * l;
        }
        F.rgb[3 * fi] = r; F.rgb[3 * fi + 1] = g; F.rgb[3 * fi + 2] = b;
        F.weight[fi] = wt; F.alpha[fi] = al; F.lum2[fi] = l2;
    }
}

// ---- edge mask (pixel_filter.rs:149-268) -------------------------------------------------------------
// What the centre ray of a pixel meets first (render.rs:503 centre_ray, integrator/mod.rs:911
// first_hit, passes.rs:168 Exact::of): x = part (instance + 1, 0xffffffff the floor, 0 the
// background), y = material (+ 1, the same codes), z = depth along the view axis (bits).
__global__ void __launch_bounds__(TRACE_THREADS) k_edge_exact(const __grid_constant__ SceneDev S, const LightsDev* __restrict__ Lg, uint4* exact) {
    __shared__ uint64_t s_stack[SHORT_STACK * TRACE_THREADS];
    uint64_t deep[STACK_CAP - SHORT_STACK];
    SplitStack stack{s_stack + threadIdx.x, deep, TRACE_THREADS};
    const LightsDev& L = *Lg;
    const uint32_t n = S.width * S.height;
    uint32_t err = 0;
    for (uint32_t p = blockIdx.x * blockDim.x + threadIdx.x; p < n; p += gridDim.x * blockDim.x) {
        const uint32_t x = p % S.width, y = p / S.width;
        V3 o, d;
        const bool sees = camera_ray_at(S, ((float)x + 0.5f) / (float)S.width, ((float)y + 0.5f) / (float)S.height, 0.0f, 0.0f, o, d);
        TraceResult res;
        const bool got = sees && trace_q<false>(S, o, d, 1.0e-3f, f_inf(), true, res, &err, stack);
        const float t_geometry = got ? res.t : f_inf();
        float t_floor = f_inf();
        if (S.floor_mode == 1 && d.z != 0.0f && sees) {
            const float t = (S.floor_z - o.z) / d.z;
            if (t > 1.0e-3f && t < f_inf()) t_floor = t;
        }
        const float t_nearest = rmin(t_geometry, t_floor);
        uint4 e = make_uint4(0u, 0u, __float_as_uint(f_inf()), 0u);
        if (!(t_nearest == f_inf() || camera_sees_panel(L, o, d, t_nearest))) {
            float t = t_floor;
            bool ok = true;
            if (t_floor < t_geometry) {
                e.x = e.y = 0xffffffffu;
            } else {
                HitInfo h;
                const DevInstance* I = nullptr;
                ok = hit_details(S, o, d, 1.0e-3f, f_inf(), res.inst, res.tri, res.t, h, I) && I != nullptr;
                if (ok) {
                    e.x = res.inst + 1u;
                    e.y = I->material < S.n_materials ? I->material + 1u : 0u;
                }
                t = res.t;
            }
            if (ok) {
                const V3 fwd = ld3(S.cam_fwd);
                e.z = __float_as_uint(S.projection ? t * len(d) : t * dot(d, fwd) + dot(o - ld3(S.cam_pos), fwd));
            } else {
                e = make_uint4(0u, 0u, __float_as_uint(f_inf()), 0u);
            }
        }
        exact[p] = e;
    }
    (void)err;
}
// ---- guide passes (passes.rs:141-229, render.rs:515-640) --------------------------------------------
// What a camera ray (o, d) meets first (integrator/mod.rs:911 first_hit): `e` = part, material
// and depth bits as k_edge_exact writes them, the normal facing the ray (the floor's +-z), and the
// albedo (passes.rs:209: the material's base colour, the default material's for an index out of
// range, the floor's colour, black for the background).
// `sees`: false for a panoramic camera's ray that sees nothing (an empty interval: the background).
static __device__ __noinline__ void first_hit_passes(const SceneDev& S, const LightsDev& L, V3 o, V3 d, bool sees, SplitStack& stack, uint32_t* err, uint4& e,
                                 V3& normal, Rgb& albedo) {
    TraceResult res;
    const bool got = sees && trace_q<false>(S, o, d, 1.0e-3f, f_inf(), true, res, err, stack);
    const float t_geometry = got ? res.t : f_inf();
    float t_floor = f_inf();
    if (S.floor_mode == 1 && d.z != 0.0f && sees) {
        const float t = (S.floor_z - o.z) / d.z;
        if (t > 1.0e-3f && t < f_inf()) t_floor = t;
    }
    const float t_nearest = rmin(t_geometry, t_floor);
    e = make_uint4(0u, 0u, __float_as_uint(f_inf()), 0u);
    normal = v3(0.0f, 0.0f, 0.0f);
    albedo = rgb(0.0f, 0.0f, 0.0f);
    if (t_nearest == f_inf() || camera_sees_panel(L, o, d, t_nearest)) return;
    float t = t_floor;
    if (t_floor < t_geometry) {
        e.x = e.y = 0xffffffffu;
        normal = v3(0.0f, 0.0f, d.z < 0.0f ? 1.0f : -1.0f);
        albedo = rgb(S.floor_color[0], S.floor_color[1], S.floor_color[2]);
    } else {
        HitInfo h;
        const DevInstance* I = nullptr;
        if (!(hit_details(S, o, d, 1.0e-3f, f_inf(), res.inst, res.tri, res.t, h, I) && I != nullptr)) return;
        e.x = res.inst + 1u;
        const bool known = I->material < S.n_materials;
        e.y = known ? I->material + 1u : 0u;
        normal = h.normal;
        albedo = known ? rgb(S.materials[I->material].base[0], S.materials[I->material].base[1], S.materials[I->material].base[2])
                       : rgb(0.8f, 0.8f, 0.8f);
        t = res.t;
    }
    const V3 fwd = ld3(S.cam_fwd);
    e.z = __float_as_uint(S.projection ? t * len(d) : t * dot(d, fwd) + dot(o - ld3(S.cam_pos), fwd));  // passes.rs:191
}

// passes.rs:221 coverage_of: whether first_hit_passes met a surface of an instance (its part id is
// the instance + 1; the floor's is all ones, the background's and a light panel's 0).
__device__ __forceinline__ bool first_hit_covers(uint4 e) { return e.x != 0u && e.x != 0xffffffffu; }

// The exact passes of the centre rays of a rectangle (render.rs:529), background outside the image.
__global__ void __launch_bounds__(TRACE_THREADS) k_exact_passes(const __grid_constant__ SceneDev S, const LightsDev* __restrict__ Lg, uint32_t x0, uint32_t y0,
                                                                 uint32_t w, uint32_t h, float* normal, float* depth, uint32_t* part,
                                                                 uint32_t* material) {
    __shared__ uint64_t s_stack[SHORT_STACK * TRACE_THREADS];
    uint64_t deep[STACK_CAP - SHORT_STACK];
    SplitStack stack{s_stack + threadIdx.x, deep, TRACE_THREADS};
    uint32_t err = 0;
    const uint32_t n = w * h;
    for (uint32_t p = blockIdx.x * blockDim.x + threadIdx.x; p < n; p += gridDim.x * blockDim.x) {
        const uint32_t x = x0 + p % w, y = y0 + p / w;
        uint4 e = make_uint4(0u, 0u, __float_as_uint(f_inf()), 0u);
        V3 nn = v3(0.0f, 0.0f, 0.0f);
        Rgb a;
        if (x < S.width && y < S.height) {
            V3 o, d;
            const bool sees = camera_ray_at(S, ((float)x + 0.5f) / (float)S.width, ((float)y + 0.5f) / (float)S.height, 0.0f, 0.0f, o, d);
            first_hit_passes(S, *Lg, o, d, sees, stack, &err, e, nn, a);
        }
        normal[3 * p] = nn.x;
        normal[3 * p + 1] = nn.y;
        normal[3 * p + 2] = nn.z;
        depth[p] = __uint_as_float(e.z);
        part[p] = e.x;
        material[p] = e.y;
    }
    (void)err;
}

// The albedo of samples [first, first + count) of a rectangle's pixels inside the image, added in
// sample order to `sum` (3 a pixel) with `weight` += 1 each (render.rs:590 render_tile_albedo_traced):
// an edge pixel (`edge`, the image's mask, may be null) adds the mean of its k sub-samples. With
// `alpha` (may be null) the coverage of the same first hits is added likewise (passes.rs:221
// coverage_of: 1 for a surface of an instance, 0 for the floor, a light panel or the background).
__global__ void __launch_bounds__(TRACE_THREADS) k_albedo_pass(const __grid_constant__ SceneDev S, const LightsDev* __restrict__ Lg, const uint8_t* __restrict__ edge,
                                                                uint32_t x0, uint32_t y0, uint32_t w, uint32_t h, uint32_t first,
                                                                uint32_t count, float* sum, float* weight, float* alpha) {
    __shared__ uint64_t s_stack[SHORT_STACK * TRACE_THREADS];
    uint64_t deep[STACK_CAP - SHORT_STACK];
    SplitStack stack{s_stack + threadIdx.x, deep, TRACE_THREADS};
    uint32_t err = 0;
    const uint32_t n = w * h;
    for (uint32_t p = blockIdx.x * blockDim.x + threadIdx.x; p < n; p += gridDim.x * blockDim.x) {
        const uint32_t x = x0 + p % w, y = y0 + p / w;
        if (x >= S.width || y >= S.height) continue;
        const uint32_t k = (edge && S.edge_k > 1 && edge[(size_t)y * S.width + x]) ? S.edge_k : 1u;
        float r = sum[3 * p], g = sum[3 * p + 1], b = sum[3 * p + 2], wt = weight[p], cv = alpha ? alpha[p] : 0.0f;
        for (uint32_t s = 0; s < count; ++s) {
            uint4 e;
            V3 nn, o, d;
            Rgb a;
            float c;
            if (k <= 1) {
                const bool sees = camera_ray(S, c_sobol, x, y, first + s, o, d);
                first_hit_passes(S, *Lg, o, d, sees, stack, &err, e, nn, a);
                c = first_hit_covers(e) ? 1.0f : 0.0f;
            } else {
                Rgb acc = rgb(0.0f, 0.0f, 0.0f);
                float covered = 0.0f;
                for (uint32_t j = 0; j < k; ++j) {
                    const bool sees = camera_ray(S, c_sobol, x, y, (first + s) * k + j, o, d);  // render.rs:376 sub_sample
                    first_hit_passes(S, *Lg, o, d, sees, stack, &err, e, nn, a);
                    acc = rgb(acc.r + a.r, acc.g + a.g, acc.b + a.b);
                    covered = covered + (first_hit_covers(e) ? 1.0f : 0.0f);
                }
                const float inv = 1.0f / (float)k;
                a = rgb(acc.r * inv, acc.g * inv, acc.b * inv);
                c = covered * inv;
            }
            r = r + a.r;
            g = g + a.g;
            b = b + a.b;
            wt = wt + 1.0f;
            cv = cv + c;
        }
        sum[3 * p] = r;
        sum[3 * p + 1] = g;
        sum[3 * p + 2] = b;
        weight[p] = wt;
        if (alpha) alpha[p] = cv;
    }
    (void)err;
}

// The albedo of each camera ray's first hit from the wave's first extend (the ray in P.o / P.d,
// the hit in P.hit): first_hit_passes without its traversal, which the extend has done with the
// same ray, class and interval.
__global__ void k_albedo_hits(const __grid_constant__ SceneDev S, const LightsDev* __restrict__ Lg, WaveDesc w, PathBuffers P) {
    const LightsDev& L = *Lg;
    for (uint32_t slot = blockIdx.x * blockDim.x + threadIdx.x; slot < w.n; slot += gridDim.x * blockDim.x) {
        const float4 of = P.o[slot], df = P.d[slot];
        const V3 o = v3(of.x, of.y, of.z), d = v3(df.x, df.y, df.z);
        const uint4 hit = P.hit[slot];
        const bool got = hit.w != 0u;
        const float t_geometry = got ? __uint_as_float(hit.z) : f_inf();
        float t_floor = f_inf();
        if (S.floor_mode == 1 && d.z != 0.0f && !(__float_as_uint(of.w) & PF_NOTHING)) {
            const float t = (S.floor_z - o.z) / d.z;
            if (t > 1.0e-3f && t < f_inf()) t_floor = t;
        }
        const float t_nearest = rmin(t_geometry, t_floor);
        float4 a = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        if (!(t_nearest == f_inf() || camera_sees_panel(L, o, d, t_nearest))) {
            if (t_floor < t_geometry) {
                a = make_float4(S.floor_color[0], S.floor_color[1], S.floor_color[2], 0.0f);
            } else {
                HitInfo h;
                const DevInstance* I = nullptr;
                if (hit_details(S, o, d, 1.0e-3f, f_inf(), hit.x, hit.y, __uint_as_float(hit.z), h, I) && I != nullptr) {
                    if (I->material < S.n_materials) {
                        const float* b = S.materials[I->material].base;
                        a = make_float4(b[0], b[1], b[2], 0.0f);
                    } else {
                        a = make_float4(0.8f, 0.8f, 0.8f, 0.0f);
                    }
                }
            }
        }
        w.alb[slot] = a;
    }
}

// The wave's albedo into the film's guide sums, each pixel's samples in index order (the edge
// pixels of a list wave the mean of their k sub-samples, render.rs:590).
__global__ void k_accumulate_albedo(WaveDesc w, FilmDev F) {
    const bool list = w.epix != nullptr;
    const uint32_t k = list ? w.ek : 1u;
    const uint32_t units = list ? w.ne : w.w * w.h;
    const uint32_t ns = w.n / (units * k);
    const float inv = 1.0f / (float)k;
    for (uint32_t e = blockIdx.x * blockDim.x + threadIdx.x; e < units; e += gridDim.x * blockDim.x) {
        uint32_t x, y;
        if (list) {
            x = w.epix[e] & 0xffffu;
            y = w.epix[e] >> 16;
        } else {
            x = w.x0 + e % w.w;
            y = w.y0 + e / w.w;
            if (w.edge && w.edge[(size_t)y * w.edge_stride + x]) continue;  // from the edge waves
        }
        if (x < F.ox || y < F.oy || x - F.ox >= F.w || y - F.oy >= F.h) continue;
        const size_t fi = (size_t)(y - F.oy) * F.w + (x - F.ox);
        float r = w.guide_sum[3 * fi], g = w.guide_sum[3 * fi + 1], b = w.guide_sum[3 * fi + 2], wt = w.guide_weight[fi];
        for (uint32_t s = 0; s < ns; ++s) {
            float ar, ag, ab;
            if (k > 1) {
                ar = ag = ab = 0.0f;
                for (uint32_t j = 0; j < k; ++j) {
                    const float4 c = w.alb[(s * units + e) * k + j];
                    ar = ar + c.x;
                    ag = ag + c.y;
                    ab = ab + c.z;
                }
                ar = ar * inv;
                ag = ag * inv;
                ab = ab * inv;
            } else {
                const float4 c = w.alb[s * units + e];
                ar = c.x;
                ag = c.y;
                ab = c.z;
            }
            r = r + ar;
            g = g + ag;
            b = b + ab;
            wt = wt + 1.0f;
        }
        w.guide_sum[3 * fi] = r;
        w.guide_sum[3 * fi + 1] = g;
        w.guide_sum[3 * fi + 2] = b;
        w.guide_weight[fi] = wt;
    }
}

// A pixel is an edge when a neighbour inside the image sees another part, another material, or
// a depth more than 2 % away (two background pixels never differ).
__global__ void k_edge_mask(const __grid_constant__ SceneDev S, const uint4* __restrict__ exact, uint8_t* mask) {
    const uint32_t w = S.width, h = S.height, n = w * h;
    for (uint32_t p = blockIdx.x * blockDim.x + threadIdx.x; p < n; p += gridDim.x * blockDim.x) {
        const uint32_t x = p % w, y = p / w;
        const uint4 c = exact[p];
        const float cd = __uint_as_float(c.z);
        bool edge = false;
        for (uint32_t ny = y ? y - 1 : 0; ny < min(y + 2, h); ++ny)
            for (uint32_t nx = x ? x - 1 : 0; nx < min(x + 2, w); ++nx) {
                const uint4 o = exact[ny * w + nx];
                const float od = __uint_as_float(o.z);
                edge |= c.x != o.x || c.y != o.y || absf(cd - od) > 0.02f * rmin(cd, od);
            }
        mask[p] = edge ? 1 : 0;
    }
}
__global__ void k_edge_list(const uint8_t* __restrict__ mask, uint32_t stride, uint32_t x0, uint32_t y0, uint32_t w, uint32_t h,
                            uint32_t* list, uint32_t* count) {
    const uint32_t n = w * h;
    for (uint32_t p = blockIdx.x * blockDim.x + threadIdx.x; p < n; p += gridDim.x * blockDim.x) {
        const uint32_t x = x0 + p % w, y = y0 + p / w;
        if (mask[(size_t)y * stride + x]) list[atomicAdd(count, 1u)] = x | (y << 16);
    }
}

// A batched wave: every pixel of every segment into its job's film. A job has at most one segment
// per wave, so no pixel is added twice here, and waves run in sample order.
__global__ void k_accumulate_jobs(WaveDesc w, PathBuffers P) {
    for (uint32_t p = blockIdx.x * blockDim.x + threadIdx.x; p < w.npix; p += gridDim.x * blockDim.x) {
        uint32_t lo = 0, hi = w.nseg;
        while (hi - lo > 1) {
            uint32_t mid = (lo + hi) >> 1;
            if (__ldg(&w.segs[mid].pix_begin) <= p) lo = mid;
            else hi = mid;
        }
        const SegDev& g = w.segs[lo];
        uint32_t local = p - g.pix_begin, npix = g.w * g.h;
        accumulate_pixel(w.jobs[g.job].film, local % g.w, g.y0 + local / g.w, P, g.slot_begin + local, npix, g.ns, w.jobs[g.job].S.projection != 0);
    }
}

// ---- film output (image.rs:186-221): resolve, exposure, then either the tone curve and sRGB at 8 or 16
// bits, or (bits 32) the exposed linear light as floats with no curve and no clamp (to_linear_exposed) ----
__global__ void k_film_encode(FilmDev F, float gain, uint32_t kind, AgxMatrices agx, uint32_t bits, void* out) {
    const uint32_t n = F.w * F.h;
    for (uint32_t p = blockIdx.x * blockDim.x + threadIdx.x; p < n; p += gridDim.x * blockDim.x) {
        float w = F.weight[p];
        Rgb px = rgb(0.0f, 0.0f, 0.0f);
        if (w > 0.0f) {
            float inv = 1.0f / w;
            px = rgb(F.rgb[3 * p] * inv, F.rgb[3 * p + 1] * inv, F.rgb[3 * p + 2] * inv);
        }
        if (bits == 32) {
            float* o = static_cast<float*>(out) + 3 * p;
            o[0] = px.r * gain;
            o[1] = px.g * gain;
            o[2] = px.b * gain;
            continue;
        }
        Rgb m = tonemap_apply(kind, px * gain, agx);
        float v[3] = {srgb_encode(m.r), srgb_encode(m.g), srgb_encode(m.b)};
        for (int c = 0; c < 3; ++c) {
            if (bits == 8) static_cast<uint8_t*>(out)[3 * p + c] = (uint8_t)saturate_cast(v[c] * 255.0f + 0.5f, 255.0f);
            else static_cast<uint16_t*>(out)[3 * p + c] = (uint16_t)saturate_cast(v[c] * 65535.0f + 0.5f, 65535.0f);
        }
    }
}

// ---- ray batches for the traversal parity harness ---------------------------------------------------
__global__ void __launch_bounds__(TRACE_THREADS) k_trace_batch(const __grid_constant__ SceneDev S, const float* __restrict__ rays, uint32_t n, uint32_t mode, uint32_t* out,
                                                     uint32_t* counters) {
    __shared__ uint64_t s_stack[SHORT_STACK * TRACE_THREADS];
    uint64_t deep[STACK_CAP - SHORT_STACK];
    SplitStack stack{s_stack + threadIdx.x, deep, TRACE_THREADS};
    uint32_t err = 0;
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const float* r = rays + 8 * i;
        TraceResult res;
        V3 o = v3(r[0], r[1], r[2]), d = v3(r[3], r[4], r[5]);
        if (mode & 2u) {
            out[i] = trace_q<true>(S, o, d, r[6], r[7], (mode & 1u) != 0, res, &err, stack) ? 1u : 0u;
        } else {
            bool got = trace_q<false>(S, o, d, r[6], r[7], (mode & 1u) != 0, res, &err, stack);
            out[3 * i] = got ? res.inst : 0xffffffffu;
            out[3 * i + 1] = got && res.tri != CAP_TRIANGLE ? __ldg(&S.tris[res.tri].tri) : 0xffffffffu;
            out[3 * i + 2] = got ? __float_as_uint(res.t) : 0u;
        }
    }
    if (err) atomicOr(&counters[3], err);
}

}  // namespace rtg

#include "rtg_adjoint.cuh"

namespace rtg {

// ---- launchers ---------------------------------------------------------------------------------------
void set_sobol(const SobolTable& t, cudaStream_t s) { cudaMemcpyToSymbolAsync(c_sobol, &t, sizeof(t), 0, cudaMemcpyHostToDevice, s); }

// Blocks of the persistent traversal kernels that fit on the device at once (their grid: more
// blocks would only start after the queue has drained).
static int resident_blocks(const void* kernel, int threads) {
    int dev = 0, sms = 0, per_sm = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess ||
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, threads, 0) != cudaSuccess || per_sm < 1)
        return 0;
    return sms * per_sm;
}

// A traversal kernel's launch; with order.l2_persist, with an L2 access-policy window over the
// scene's traversal data (persisting for its hit ratio, the rest streaming).
template <class... KArgs, class... Args>
static void launch_traversal(const RaySort& order, int grid, cudaStream_t st, void (*kernel)(KArgs...), Args... args) {
    if (!(order.l2_persist && order.l2_base && order.l2_bytes)) {
        kernel<<<grid, TRACE_THREADS, 0, st>>>(args...);
        return;
    }
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(grid);
    cfg.blockDim = dim3(TRACE_THREADS);
    cfg.stream = st;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeAccessPolicyWindow;
    attr[0].val.accessPolicyWindow.base_ptr = const_cast<void*>(order.l2_base);
    attr[0].val.accessPolicyWindow.num_bytes = order.l2_bytes;
    attr[0].val.accessPolicyWindow.hitRatio = order.l2_hit_ratio;
    attr[0].val.accessPolicyWindow.hitProp = cudaAccessPropertyPersisting;
    attr[0].val.accessPolicyWindow.missProp = cudaAccessPropertyStreaming;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    cudaLaunchKernelEx(&cfg, kernel, args...);
}

// Whether a wave's last rounds run in k_tail: a limit set, no shadow walks, not batched.
// The tail traces with the plain traversal: scenes with passable surfaces or a section keep the wavefront.
static bool tail_on(const SceneDev& S, const RaySort& order, bool batch) {
    return order.tail_paths > 0 && !S.any_passable && !S.section_on && !batch;
}
// Blocks of the persistent kernels for a wave of n paths: all that are resident, unless the wave
// has fewer paths than these have warps.
static int blocks_of(int resident, uint32_t n, int fallback) {
    return resident > 0 ? (int)std::min<uint32_t>((uint32_t)resident, (n + TRACE_THREADS / 32 - 1) / (TRACE_THREADS / 32)) : fallback;
}

// Shadow rays through passable surfaces are walked inside k_trace, except a section's and a batch's.
static bool walks_on(const SceneDev& S, bool batch) { return S.any_passable && !S.section_on && !batch; }
// Whether a wave of n paths traces each round's shadow rays with the next round's extension rays.
// Timed waves trace them apart, so that the events are around extension rays only. So do waves of
// more than 2^25 paths: their launches' ends weigh little, and shadow rays visit children in slot
// order there, which needs no sort. 1080p product frame apart and together, ms: 8 Mi paths 14.6 and 13.6,
// 16 Mi 24.6 and 23.6, 32 Mi 43.4 and 43.0, 47 Mi 62.9 and 62.7, 63 Mi 80.6 and 81.6, 127 Mi 154.6 and 159.0.
static bool together_on(const SceneDev& S, uint32_t n, bool batch, bool timed) {
    return !S.section_on && (!S.any_passable || walks_on(S, batch)) && !timed && n <= (1u << 25);
}
uint32_t wave_launches(const SceneDev& S, const RaySort& order, const PathBuffers& P, uint32_t n, bool batch, bool timed) {
    const uint32_t rounds = wave_rounds(S);
    const bool rsort = order.ray_bits > 0 && P.rbins, ssort = rsort && order.shadow_sort && P.sbins;
    const bool tail = tail_on(S, order, batch) && rounds > TAIL_FIRST_ROUND;
    const uint32_t shadows = !together_on(S, n, batch, timed) ? rounds : (walks_on(S, batch) ? 1u : 0u);
    return 2 + rounds * (2 + (order.material_sort ? 1u : 0u) + (ssort ? 2u : 0u)) + shadows + (rsort ? 2u * (rounds - 1u) : 0u) + (tail ? 1u : 0u);
}

void launch_wave(const SceneDev& S, const LightsDev* L, const WaveDesc& wave, const PathBuffers& P, const FilmDev* film, cudaStream_t st,
                 int grid, WaveTiming* timing, const RaySort& tuning) {
    static const int ext_resident = resident_blocks((const void*)k_trace<EXTEND>, TRACE_THREADS);
    static const int both_resident = resident_blocks((const void*)k_trace<SHADOW_TOO>, TRACE_THREADS);
    static const int tail_resident = resident_blocks((const void*)k_tail<false>, TRACE_THREADS);
    static const int shade_resident = resident_blocks((const void*)k_shade<false, false>, 128);
    static const int sort_resident = resident_blocks((const void*)k_material_sort, SORT_THREADS);
    WaveDesc w = with_divisors(wave);
    w.dark = S.projection != 0;
    const int g = grid;
    const int g_trace = blocks_of(ext_resident, w.n, g), g_both = blocks_of(both_resident, w.n, g), g_shade = blocks_of(shade_resident, w.n, g);
    const int g_sort = std::min<int>(sort_resident > 0 ? sort_resident : g, (int)((w.n + SORT_CHUNK - 1) / SORT_CHUNK));
    const bool batch = w.segs != nullptr;
    const uint32_t rounds = wave_rounds(S);
    RaySort order = tuning;
    if (!tail_on(S, order, batch) || rounds <= TAIL_FIRST_ROUND) order.tail_paths = 0;
    const bool rsort = order.ray_bits > 0 && order.ray_bits <= RAY_SORT_MAX_BITS && P.rbins;
    const bool ssort = rsort && order.shadow_sort && P.sbins;
    const uint32_t nk = ray_sort_keys(order.ray_bits);
    if (batch) k_camera<true><<<g, 256, 0, st>>>(S, w, P, rounds);
    else k_camera<false><<<g, 256, 0, st>>>(S, w, P, rounds);
    // Traced with the next round's extension rays, the last round's shadow rays need a launch of their
    // own where there are any: its vertices are at the greatest depth, unless cut-outs shift that.
    const bool walks = walks_on(S, batch), together = together_on(S, w.n, batch, timing != nullptr);
    const uint32_t* perm = nullptr;  // the last round's shadow rays in the order to trace them (null: as queued)
    for (uint32_t round = 0; round < rounds; ++round) {
        uint32_t* const queue = P.queue[round & 1];
        // The camera rays are traced in pixel order; later rounds' rays in coherence order.
        const uint32_t* traced = queue;
        if (rsort && round > 0) {
            k_key_scan<<<1, 1024, 0, st>>>(P.rbins, nk);
            k_key_scatter<<<g, 256, 0, st>>>(queue, P.key, P.rbins + nk, &P.counters[round_counter(round, COUNT_PATHS)], P.sorted);
            traced = P.sorted;
        }
        const bool timed = timing && timing->ev_count + 2 <= WaveTiming::MAX_EVENTS;
        if (timed) cudaEventRecord(timing->ev[timing->ev_count++], st);
        if (S.section_on) launch_traversal(order, g_trace, st, k_extend_section, S, P, round, traced, order.tail_paths);
        else if (together && round > 0) launch_traversal(order, g_both, st, walks ? k_trace<WALK_TOO> : k_trace<SHADOW_TOO>, S, P, round, traced, perm, order.tail_paths);
        else launch_traversal(order, g_trace, st, k_trace<EXTEND>, S, P, round, traced, perm, order.tail_paths);
        if (timed) cudaEventRecord(timing->ev[timing->ev_count++], st);
        if (round == 0 && w.alb && film && !batch) k_albedo_hits<<<g, 256, 0, st>>>(S, L, w, P);
        // The material-sorted copy goes to whichever list the traversal did not read.
        const uint32_t* shaded = traced;
        if (order.material_sort) {
            uint32_t* sorted = traced == P.sorted ? queue : P.sorted;
            k_material_sort<<<g_sort, SORT_THREADS, 0, st>>>(P, round, traced, sorted, order.tail_paths);
            shaded = sorted;
        }
        // Keys for the next round's rays (none after the last round) and for this round's shadow rays.
        PathBuffers Q = P;
        Q.rbins = rsort && round + 1 < rounds ? P.rbins : nullptr;
        Q.sbins = ssort ? P.sbins : nullptr;
        (batch ? (S.plain ? k_shade<true, true> : k_shade<true, false>) : (S.plain ? k_shade<false, true> : k_shade<false, false>))
            <<<g_shade, 128, 0, st>>>(S, L, Q, round, w, shaded, order);
        // The round's queue is free once shade has read it: it holds the shadow rays' order.
        perm = nullptr;
        if (ssort) {
            k_key_scan<<<1, 1024, 0, st>>>(P.sbins, nk);
            k_key_scatter<<<g, 256, 0, st>>>(nullptr, P.sh_key, P.sbins + nk, &P.counters[round_counter(round, COUNT_SHADOW)], queue);
            perm = queue;
        }
        if (together && !(walks && round + 1 == rounds)) continue;
        if (walks) launch_traversal(order, g_both, st, k_trace<WALK>, S, P, round, traced, perm, 0u);
        else if (S.any_passable) (batch ? k_shadow_walk<true> : k_shadow_walk<false>)<<<g, TRACE_THREADS, 0, st>>>(S, P, round, w, perm);
        else if (S.section_on) launch_traversal(order, g_trace, st, k_shadow_section, S, P, round, perm);
        else launch_traversal(order, g_trace, st, k_trace<SHADOW>, S, P, round, traced, perm, 0u);
    }
    if (order.tail_paths)
        (S.plain ? k_tail<true> : k_tail<false>)<<<blocks_of(tail_resident, w.n, g), TRACE_THREADS, 0, st>>>(S, L, P, w, rounds, order.tail_paths);
    if (batch) k_accumulate_jobs<<<g, 256, 0, st>>>(w, P);
    else if (film && w.epix) k_accumulate_edges<<<g, 256, 0, st>>>(w, P, *film);
    else if (film) k_accumulate<<<g, 256, 0, st>>>(w, P, *film);
    if (w.alb && film && !batch) k_accumulate_albedo<<<g, 256, 0, st>>>(w, *film);
}

cudaError_t launch_edge_mask(const SceneDev& S, const LightsDev* L, uint4* exact, uint8_t* mask, cudaStream_t st, int grid) {
    k_edge_exact<<<grid, TRACE_THREADS, 0, st>>>(S, L, exact);
    k_edge_mask<<<grid, 256, 0, st>>>(S, exact, mask);
    return cudaGetLastError();
}
cudaError_t launch_exact_passes(const SceneDev& S, const LightsDev* L, uint32_t x0, uint32_t y0, uint32_t w, uint32_t h, float* normal,
                                float* depth, uint32_t* part, uint32_t* material, cudaStream_t st, int grid) {
    k_exact_passes<<<grid, TRACE_THREADS, 0, st>>>(S, L, x0, y0, w, h, normal, depth, part, material);
    return cudaGetLastError();
}
cudaError_t launch_albedo_pass(const SceneDev& S, const LightsDev* L, const uint8_t* edge, uint32_t x0, uint32_t y0, uint32_t w, uint32_t h,
                               uint32_t first, uint32_t count, float* sum, float* weight, float* alpha, cudaStream_t st, int grid) {
    k_albedo_pass<<<grid, TRACE_THREADS, 0, st>>>(S, L, edge, x0, y0, w, h, first, count, sum, weight, alpha);
    return cudaGetLastError();
}
cudaError_t launch_edge_list(const uint8_t* mask, uint32_t stride, uint32_t x0, uint32_t y0, uint32_t w, uint32_t h, uint32_t* list,
                             uint32_t* count, cudaStream_t st, int grid) {
    cudaMemsetAsync(count, 0, 4, st);
    k_edge_list<<<grid, 256, 0, st>>>(mask, stride, x0, y0, w, h, list, count);
    return cudaGetLastError();
}

void launch_adjoint_delta(const FilmDev& F, const float* target, float4* dpath, double* loss, const PathBuffers& P, uint32_t count, cudaStream_t st,
                          int grid) {
    k_adjoint_delta<<<grid, 256, 0, st>>>(F, target, dpath, loss, P, count);
}
void launch_adjoint_wave(const SceneDev& S, const LightsDev* L, const WaveDesc& wave, const PathBuffers& P, const AdjointDev& A, cudaStream_t st,
                         int grid) {
    static const int ext_resident = resident_blocks((const void*)k_trace<EXTEND>, TRACE_THREADS);
    static const int sh_resident = resident_blocks((const void*)k_shadow_adjoint, TRACE_THREADS);
    static const int shade_resident = resident_blocks((const void*)k_shade_adjoint<false>, 128);
    static const int sort_resident = resident_blocks((const void*)k_material_sort, SORT_THREADS);
    const WaveDesc w = with_divisors(wave);
    const int g = grid;
    const int g_ext = blocks_of(ext_resident, w.n, g), g_sh = blocks_of(sh_resident, w.n, g), g_shade = blocks_of(shade_resident, w.n, g);
    const int g_sort = std::min<int>(sort_resident > 0 ? sort_resident : g, (int)((w.n + SORT_CHUNK - 1) / SORT_CHUNK));
    const uint32_t rounds = S.max_depth + 1;
    k_adjoint_camera<<<g, 256, 0, st>>>(S, w, P, A, rounds);
    for (uint32_t bounce = 0; bounce < rounds; ++bounce) {
        k_trace<EXTEND><<<g_ext, TRACE_THREADS, 0, st>>>(S, P, bounce, P.queue[bounce & 1], nullptr, 0);
        k_material_sort<<<g_sort, SORT_THREADS, 0, st>>>(P, bounce, P.queue[bounce & 1], P.sorted, 0);
        (S.plain ? k_shade_adjoint<true> : k_shade_adjoint<false>)<<<g_shade, 128, 0, st>>>(S, L, P, bounce, w, A);
        k_shadow_adjoint<<<g_sh, TRACE_THREADS, 0, st>>>(S, P, bounce, w, A);
    }
    k_adjoint_residual<<<g, 256, 0, st>>>(w, P, A);
}
void launch_film_encode(const FilmDev& F, float ev, uint32_t tonemap, uint32_t bits, void* out, cudaStream_t st, int grid) {
    k_film_encode<<<grid, 256, 0, st>>>(F, fexp2(ev), tonemap, agx_matrices(), bits, out);
}
void launch_trace_batch(const SceneDev& S, const float* rays, uint32_t n, uint32_t mode, uint32_t* out, uint32_t* counters,
                        cudaStream_t st, int grid) {
    k_trace_batch<<<grid, TRACE_THREADS, 0, st>>>(S, rays, n, mode, out, counters);
}

}  // namespace rtg
