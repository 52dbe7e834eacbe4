// ff_trace.cu — persistent closest-hit / any-hit trace kernel behind ff_trace.
//
// Replaces wf_extend / wf_shadow (CUDA-RayTracer/kernel.cu:488-543), which
// launch one thread per queued ray over a binary BVH with a 64-entry local
// stack.  Here every warp is persistent: idle lanes take new rays from a
// global counter with one warp-aggregated atomic, so lanes whose rays finish
// early are refilled instead of idling until the slowest ray of the warp ends
// (Aila & Laine 2009, "Understanding the efficiency of ray traversal on GPUs").
#include <algorithm>

#include "ff_internal.h"
#include "ff_trace.cuh"

static_assert(kMaxStack == kMaxStackDepth, "stack size must match the build-time depth check");

namespace {

constexpr int kTraceBlock = 128;
// Refill when at least this many lanes of the warp are idle.
constexpr int kRefillIdle = 8;

constexpr uint32_t kPool = 64;

// Output: hits[ray] for every ray, or, with tags (the wavefront's queues),
// per the ray's tag: a closest hit goes to hits[tag] (tag = the path slot, so
// the next stage reads its hit in slot order without the queue index), an
// any-hit answer to occ[tag] (1 occluded, 0 clear; tag = 4 * slot + shadow
// ray index, so the next stage reads one 4-byte word of answers per slot).
//
// TWO (closest hit only): rays whose tmin carries the sign bit are traced
// two-sided (ff_test_tri_closest); a back-face hit reports prim = -2 - index.
template <bool ANY, bool TAGGED, bool TWO = false>
__global__ void __launch_bounds__(kTraceBlock, 8)
    k_trace(FFBvhView bvh, const ff_ray* __restrict__ rays, ff_hit* __restrict__ hits, uint64_t n,
            unsigned long long* __restrict__ counter, unsigned int* __restrict__ err,
            const uint32_t* __restrict__ n_dev, const uint32_t* __restrict__ tags, uint8_t* __restrict__ occ)
{
    // Queue-driven launches (the wavefront) read the ray count written by the
    // producing stage; n is then the queue capacity.
    if (n_dev) n = min(n, (uint64_t)*n_dev);
    // A ray visits every node at most once; more steps than nodes means a
    // malformed BVH.  The ray is then ended and counted in err[0] instead of
    // looping.
    const uint32_t max_steps = bvh.num_nodes + 2u;
    __shared__ uint2 s_stack[kShortStack * kTraceBlock];
    FFStack st;
    st.sm = s_stack + threadIdx.x;
    st.stride = kTraceBlock;
    st.sp = 0;
    const uint32_t lane = threadIdx.x & 31u;
    const uint32_t lt_mask = (1u << lane) - 1u;

    FFRayState r;
    uint2 cur = make_uint2(0u, 0u);
    uint64_t ray_id = 0;
    uint32_t tag = 0;
    uint32_t steps = 0;
    bool active = false;
    bool exhausted = false;
    // the warp's share of the rays: pool_left of them from pool_next.  A
    // caller's rays are taken kPool at a time (all warps' atomics go to one
    // address, one after the other), near the end only as many as needed, so
    // that the last ones spread over all warps: 16.8M incoherent closest hits
    // 1419 -> 1381 us, 3M any hits 231 -> 226 us.  The wavefront's queues are
    // short, and their tails weigh more (256 x 256 x 16 render 2.06 -> 2.09
    // ms): there a warp takes what its idle lanes need.
    uint64_t pool_next = 0;
    uint32_t pool_left = 0;

    while (true) {
        // Refill idle lanes with new rays.
        const uint32_t want = __ballot_sync(0xffffffffu, !active && !exhausted);
        if (want) {
            const uint32_t need = __popc(want), rank = __popc(want & lt_mask);
            uint64_t mine = pool_next + rank;
            if (pool_left < need) {
                const uint32_t more = need - pool_left;
                const uint32_t take = !TAGGED && pool_next + (uint64_t)gridDim.x * (2u * kTraceBlock) < n ? kPool : more;
                unsigned long long base = 0;
                if (lane == 0) base = atomicAdd(counter, (unsigned long long)take);
                base = __shfl_sync(0xffffffffu, base, 0);
                if (rank >= pool_left) mine = base + (rank - pool_left);
                pool_next = base + more;
                pool_left = take - more;
            } else {
                pool_next += need;
                pool_left -= need;
            }
            if (!active && !exhausted) {
                ray_id = mine;
                if (ray_id < n) {
                    float4 r0, r1;
                    if (TAGGED) {   // (a queue's rays sit on 32-byte boundaries, a caller's on 16)
                        const ff_ray q = ld_sector(rays + ray_id);
                        r0 = make_float4(q.ox, q.oy, q.oz, q.tmin);
                        r1 = make_float4(q.dx, q.dy, q.dz, q.tmax);
                        tag = __ldg(tags + ray_id);
                    } else {
                        r0 = __ldg(reinterpret_cast<const float4*>(rays + ray_id));
                        r1 = __ldg(reinterpret_cast<const float4*>(rays + ray_id) + 1);
                    }
                    // untagged two-sided launches (ff_trace with FF_TRACE_TWO_SIDED) mark every ray;
                    // tagged ones (the wavefront) carry the mark in each ray's tmin
                    const float tmin = (TWO && !TAGGED) ? -(r0.w > 0.f ? r0.w : 0.f) : r0.w;
                    ff_ray_setup(r, make_float3(r0.x, r0.y, r0.z), make_float3(r1.x, r1.y, r1.z), tmin, r1.w, ANY);
                    cur = ff_root_group(r);
                    st.reset();
                    steps = 0;
                    active = bvh.num_nodes > 0;
                    if (!active) {
                        if (!TAGGED) hits[ray_id] = ff_hit{r.tmax, 0.f, 0.f, -1};
                        else if (ANY) occ[tag] = 0;
                        else hits[tag] = ff_hit{r.tmax, 0.f, 0.f, -1};
                    }
                } else {
                    exhausted = true;
                }
            }
        }
        if (!__any_sync(0xffffffffu, active)) {
            if (__all_sync(0xffffffffu, exhausted)) break;
            continue;
        }
        // Traverse until enough lanes are idle to make a refill worthwhile.
        while (true) {
            if (active) {
                const bool done = ff_traverse_step<ANY, TWO>(bvh, r, cur, st);
                if (st.overflow || ++steps > max_steps) atomicAdd(err, 1u);
                if (done || steps > max_steps) {
                    const int32_t prim = TWO ? ff_hit_of(r).prim : (r.prim == 0xffffffffu ? -1 : (int32_t)r.prim);
                    const float4 out = make_float4(r.tmax, r.u, r.v, __int_as_float(prim));
                    if (!TAGGED) *reinterpret_cast<float4*>(hits + ray_id) = out;
                    else if (ANY) occ[tag] = prim >= 0 ? 1 : 0;
                    else *reinterpret_cast<float4*>(hits + tag) = out;
                    active = false;
                }
            }
            const uint32_t idle = __ballot_sync(0xffffffffu, !active && !exhausted);
            const uint32_t busy = __ballot_sync(0xffffffffu, active);
            if (busy == 0u || __popc(idle) >= kRefillIdle) break;
        }
    }
}

// Lanes that trace one ray together in k_trace_group, and rays per block.
constexpr uint32_t kGroup = 8;
constexpr uint32_t kGroupRays = kTraceBlock / kGroup;

// k_trace for few rays: eight lanes per ray.  A launch with fewer rays than
// the GPU has threads ends with its longest ray (22 nodes where the average
// ray of the small room takes 2.6), and a lone ray in k_trace pays for every
// child and every triangle one after the other, about 2 us a step.  Here each
// lane tests one child of the node, then one of the node's (at most 24)
// triangles a round, so that a step is a node load, one box test, a ballot,
// and one to three triangle rounds.  The whole warp does per ray about twice
// the instructions of k_trace, whose lanes share them, so this pays while
// rays are few (kFewRays).  Loading the next node before the triangles of the
// last one are tested made it 8% slower: the step is a chain of dependent
// instructions more than of loads.
//
// Lane `sub` of a group takes slot sub ^ oct_inv, so the ballot over the hit
// internal children is the traversal-ordered hit mask itself.  Every box and
// triangle test is k_trace's (the same operations on the same values), nodes
// are visited in the same order, a closest hit is the minimum of (t, original
// index) and an any-hit ray reports the first occluder in triangle order, so
// the answers are bit for bit k_trace's.
template <bool ANY, bool TAGGED, bool TWO = false>
__global__ void __launch_bounds__(kTraceBlock, 8)
    k_trace_group(FFBvhView bvh, const ff_ray* __restrict__ rays, ff_hit* __restrict__ hits, uint64_t n,
                  unsigned long long* __restrict__ counter, unsigned int* __restrict__ err,
                  const uint32_t* __restrict__ n_dev, const uint32_t* __restrict__ tags, uint8_t* __restrict__ occ)
{
    if (n_dev) n = min(n, (uint64_t)*n_dev);
    const uint32_t max_steps = bvh.num_nodes + 2u;
    __shared__ uint2 s_stack[kGroupRays][kMaxStack];
    const uint32_t lane = threadIdx.x & 31u, sub = lane % kGroup, first = lane - sub;
    uint2* stack = s_stack[threadIdx.x / kGroup];
    FFRayState r;   // the same in all lanes of the group
    uint2 cur = make_uint2(0u, 0u);
    uint64_t ray_id = 0;
    uint32_t tag = 0, steps = 0;
    int sp = 0;
    bool active = false, exhausted = false;
    while (true) {
        if (!active && !exhausted) {
            unsigned long long base = 0;
            if (sub == 0) base = atomicAdd(counter, 1ull);
            ray_id = __shfl_sync(0xffu << first, base, (int)first);
            if (ray_id < n) {
                const float4 r0 = __ldg(reinterpret_cast<const float4*>(rays + ray_id));
                const float4 r1 = __ldg(reinterpret_cast<const float4*>(rays + ray_id) + 1);
                if (TAGGED) tag = __ldg(tags + ray_id);
                const float tmin = (TWO && !TAGGED) ? -(r0.w > 0.f ? r0.w : 0.f) : r0.w;
                ff_ray_setup(r, make_float3(r0.x, r0.y, r0.z), make_float3(r1.x, r1.y, r1.z), tmin, r1.w, ANY);
                cur = ff_root_group(r);
                sp = 0;
                steps = 0;
                active = true;
            } else {
                exhausted = true;
            }
        }
        __syncwarp();
        if (!__any_sync(0xffffffffu, active)) break;   // (every group is exhausted)
        // the next node's children, one a lane
        uint32_t tmask = 0, tri_base = 0;
        bool inner = false, bad = false;
        uint32_t imask = 0, child_base = 0;
        if (active && bvh.num_nodes) {
            const uint32_t bit = 31u - __clz(cur.y & 0xff000000u);
            cur.y &= ~(1u << bit);
            const uint32_t slot = (bit - 24u) ^ r.oct_inv;
            const uint32_t child = cur.x + __popc(cur.y & 0xffu & ((1u << slot) - 1u));
            if (cur.y & 0xff000000u) {
                bad = sp >= kMaxStack;
                if (!bad && sub == 0) stack[sp] = cur;
                if (!bad) ++sp;
            }
            bad |= child >= bvh.num_nodes;
            cur.y = 0;
            if (!bad) {
                const uint32_t s = sub ^ r.oct_inv;
                const FFNode8* nd = bvh.nodes + child;
                const uint4 n0 = __ldg(reinterpret_cast<const uint4*>(nd));
                const uint2 n1 = __ldg(reinterpret_cast<const uint2*>(nd) + 2);
                const uint8_t* q = reinterpret_cast<const uint8_t*>(nd) + 24 + s;
                const uint32_t meta = __ldg(q);
                q += 8;   // plane bytes of this slot: lo x, y, z, hi x, y, z, 8 bytes apart
                const uint32_t px = r.inv.x >= 0.f ? 0u : 24u, py = r.inv.y >= 0.f ? 8u : 32u,
                               pz = r.inv.z >= 0.f ? 16u : 40u;
                auto plane = [&](uint32_t at) { return __uint_as_float(0x4B000000u | __ldg(q + at)) - 8388608.0f; };
                const float nx = plane(px), fx = plane(24u - px), ny = plane(py), fy = plane(40u - py), nz = plane(pz),
                            fz = plane(56u - pz);
                const float ax = __uint_as_float((n0.w & 0xffu) << 23) * r.inv.x,
                            ay = __uint_as_float(((n0.w >> 8) & 0xffu) << 23) * r.inv.y,
                            az = __uint_as_float(((n0.w >> 16) & 0xffu) << 23) * r.inv.z;
                const float bx = (__uint_as_float(n0.x) - r.o.x) * r.inv.x, by = (__uint_as_float(n0.y) - r.o.y) * r.inv.y,
                            bz = (__uint_as_float(n0.z) - r.o.z) * r.inv.z;
                const float tb = __fmaf_rn(fabsf(r.tmax), FF_BOX_WIDEN, r.tmax);
                float tn = fmax3f(__fmaf_rn(nx, ax, bx), __fmaf_rn(ny, ay, by), __fmaf_rn(nz, az, bz));
                float tf = fmin3f(__fmaf_rn(fx, ax, bx), __fmaf_rn(fy, ay, by), __fmaf_rn(fz, az, bz));
                tn = __fmaf_rn(-fabsf(tn), FF_BOX_WIDEN, tn);
                tf = __fmaf_rn(fabsf(tf), FF_BOX_WIDEN, tf);
                imask = n0.w >> 24;
                child_base = n1.x;
                tri_base = n1.y;
                if (fmaxf(tn, r.tmin) <= fminf(tf, tb)) {
                    inner = (imask >> s) & 1u;
                    if (!inner) tmask = (meta >> 5) << (meta & 31u);
                }
            }
        }
        __syncwarp();   // (votes order no memory: lane 0's push before the group's pop below)
        const uint32_t kids = (__ballot_sync(0xffffffffu, inner) >> first) & 0xffu;
#pragma unroll
        for (uint32_t k = 1; k < kGroup; k <<= 1) tmask |= __shfl_xor_sync(0xffffffffu, tmask, k);
        // the triangles, one a lane and round
        bool done = bad;
#pragma unroll 1
        for (uint32_t round = 0; round < 3u; ++round) {
            if (!__any_sync(0xffffffffu, !done && (tmask >> (kGroup * round)) != 0u)) break;
            const uint32_t i = kGroup * round + sub;
            bool hit = !done && ((tmask >> i) & 1u);
            if (hit && tri_base + i >= bvh.num_tris) {   // never on a validated BVH
                atomicAdd(err, 1u);
                hit = false;
            }
            if (ANY) {
                float t = 0.f;
                uint32_t id = 0;
                if (hit) hit = ff_occluder(bvh.tris, tri_base + i, r, t, id);
                const uint32_t who = (__ballot_sync(0xffffffffu, hit) >> first) & 0xffu;
                if (who) {
                    const int from = (int)first + __ffs(who) - 1;
                    r.tmax = __shfl_sync(0xffu << first, t, from);
                    r.prim = __shfl_sync(0xffu << first, id, from);
                    done = true;
                }
            } else {
                FFCandidate h;
                h.back = false;
                if (hit) hit = ff_candidate<TWO>(bvh.tris, tri_base + i, r, h) && ff_better<TWO>(r, h.t, h.id);
                const uint32_t who = (__ballot_sync(0xffffffffu, hit) >> first) & 0xffu;
                if (who) {
                    // the group's best: smallest t (-0 and 0 alike), then smallest index
                    unsigned long long key =
                        hit ? (unsigned long long)__float_as_uint(h.t + 0.f) << 32 | h.id : ~0ull, best = key;
#pragma unroll
                    for (uint32_t k = 1; k < kGroup; k <<= 1) {
                        const unsigned long long other = __shfl_xor_sync(0xffu << first, best, (int)k);
                        best = other < best ? other : best;
                    }
                    float u = 0.f, v = 0.f;
                    const bool mine = hit && key == best;
                    if (mine) {
                        u = h.u();
                        v = h.v();
                        h.id |= (TWO && h.back) ? kBackFace : 0u;
                    }
                    const int from = (int)first + __ffs((__ballot_sync(0xffu << first, mine) >> first) & 0xffu) - 1;
                    r.tmax = __shfl_sync(0xffu << first, h.t, from);
                    r.prim = __shfl_sync(0xffu << first, h.id, from);
                    r.u = __shfl_sync(0xffu << first, u, from);
                    r.v = __shfl_sync(0xffu << first, v, from);
                }
            }
        }
        if (active) {
            cur = make_uint2(child_base, kids << 24 | imask);
            if (!done && !kids) {
                if (sp == 0) done = true;
                else cur = stack[--sp];
            }
            ++steps;
            if ((bad || steps > max_steps) && sub == 0) atomicAdd(err, 1u);
            if (done || bad || steps > max_steps) {
                if (sub == 0) {
                    const int32_t prim = TWO ? ff_hit_of(r).prim : (r.prim == 0xffffffffu ? -1 : (int32_t)r.prim);
                    const float4 out = make_float4(r.tmax, r.u, r.v, __int_as_float(prim));
                    if (!TAGGED) *reinterpret_cast<float4*>(hits + ray_id) = out;
                    else if (ANY) occ[tag] = prim >= 0 ? 1 : 0;
                    else *reinterpret_cast<float4*>(hits + tag) = out;
                }
                active = false;
            }
        }
        __syncwarp();
    }
}

// Rays up to which a launch goes to k_trace_group.  us per launch, k_trace and
// k_trace_group, incoherent closest hits in the small room (on the 82k-triangle
// mesh): 100 rays 24.1 and 17.0 (23.2, 17.2), 4,000 33.0 and 24.7 (43.3,
// 33.8), 32,000 36.9 and 33.6 (55.8, 49.6), 65,536 38.2 and 42.9 (59.3, 58.1);
// any hits cross at the same place.
constexpr uint64_t kFewRays = 40960;

// Traversal work of n rays (ff_trace_count): one thread per ray over the same
// traversal step as k_trace, so each ray visits the same nodes and tests the
// same triangles; out[0] += node records fetched, out[1] += triangles tested.
// QUEUE: a wavefront queue whose length is in n_dev (n its capacity), whose
// rays carry their own two-sided mark (as k_trace<*, tagged> reads them).
template <bool ANY, bool TWO = false, bool QUEUE = false>
__global__ void __launch_bounds__(kTraceBlock) k_trace_count(FFBvhView bvh, const ff_ray* __restrict__ rays,
                                                             uint64_t n, unsigned long long* __restrict__ out,
                                                             unsigned int* __restrict__ err,
                                                             const uint32_t* __restrict__ n_dev = nullptr)
{
    if (QUEUE) n = min(n, (uint64_t)*n_dev);
    __shared__ uint2 s_stack[kShortStack * kTraceBlock];
    FFStack st;
    st.sm = s_stack + threadIdx.x;
    st.stride = kTraceBlock;
    st.sp = 0;
    FFCount count;
    const uint32_t max_steps = bvh.num_nodes + 2u;
    for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < n; i += (uint64_t)gridDim.x * blockDim.x) {
        if (!bvh.num_nodes) break;
        const float4 r0 = __ldg(reinterpret_cast<const float4*>(rays + i));
        const float4 r1 = __ldg(reinterpret_cast<const float4*>(rays + i) + 1);
        FFRayState r;
        const float tmin = (TWO && !QUEUE) ? -(r0.w > 0.f ? r0.w : 0.f) : r0.w;
        ff_ray_setup(r, make_float3(r0.x, r0.y, r0.z), make_float3(r1.x, r1.y, r1.z), tmin, r1.w, ANY);
        uint2 cur = ff_root_group(r);
        st.reset();
        uint32_t steps = 0;
        while (!ff_traverse_step<ANY, FFCount, TWO>(bvh, r, cur, st, count)) {
            if (st.overflow || ++steps > max_steps) {
                atomicAdd(err, 1u);
                break;
            }
        }
    }
    unsigned long long a = count.nodes, b = count.tris;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        a += __shfl_down_sync(0xffffffffu, a, o);
        b += __shfl_down_sync(0xffffffffu, b, o);
    }
    if ((threadIdx.x & 31u) == 0) {
        atomicAdd(out, a);
        atomicAdd(out + 1, b);
    }
}

}  // namespace

void ff_launch_trace_count(ff_context* ctx, const ff_scene* s, const ff_ray* d_rays, uint64_t n, bool any_hit,
                           unsigned long long* d_out, unsigned int* err, bool two_sided)
{
    if (n == 0) return;
    uint64_t grid = (uint64_t)ctx->num_sms * 8;
    const uint64_t need = (n + kTraceBlock - 1) / kTraceBlock;
    if (grid > need) grid = need;
    if (any_hit)
        k_trace_count<true><<<(unsigned)grid, kTraceBlock, 0, ctx->stream>>>(s->view(), d_rays, n, d_out, err);
    else if (two_sided)
        k_trace_count<false, true><<<(unsigned)grid, kTraceBlock, 0, ctx->stream>>>(s->view(), d_rays, n, d_out, err);
    else
        k_trace_count<false><<<(unsigned)grid, kTraceBlock, 0, ctx->stream>>>(s->view(), d_rays, n, d_out, err);
    FF_CUDA_CHECK(cudaGetLastError());
}

void ff_launch_trace_count_queue(ff_context* ctx, const FFBvhView& bvh, const ff_ray* d_rays, const uint32_t* n_dev,
                                 uint64_t cap, bool any_hit, bool two_sided, unsigned long long* d_out,
                                 unsigned int* err, cudaStream_t stream)
{
    if (cap == 0) return;
    uint64_t grid = (uint64_t)ctx->num_sms * 8;
    const uint64_t need = (cap + kTraceBlock - 1) / kTraceBlock;
    if (grid > need) grid = need;
    const dim3 g((unsigned)grid), b(kTraceBlock);
    if (any_hit)
        k_trace_count<true, false, true><<<g, b, 0, stream>>>(bvh, d_rays, cap, d_out, err, n_dev);
    else if (two_sided)
        k_trace_count<false, true, true><<<g, b, 0, stream>>>(bvh, d_rays, cap, d_out, err, n_dev);
    else
        k_trace_count<false, false, true><<<g, b, 0, stream>>>(bvh, d_rays, cap, d_out, err, n_dev);
    FF_CUDA_CHECK(cudaGetLastError());
}

namespace {

using TraceKernel = void (*)(FFBvhView, const ff_ray*, ff_hit*, uint64_t, unsigned long long*, unsigned int*,
                             const uint32_t*, const uint32_t*, uint8_t*);

// Launches the kernel for at most n rays (n_dev: their number on the device).
// Up to kFewRays rays go to k_trace_group, eight lanes a ray, more to
// k_trace.  max_blocks_per_sm limits k_trace's persistent grid (0: as many
// as fit).
void launch_trace(ff_context* ctx, const FFBvhView& bvh, const ff_ray* d_rays, uint64_t n, ff_hit* d_hits, bool any_hit,
                  bool two, unsigned long long* counter, unsigned int* err, const uint32_t* n_dev,
                  const uint32_t* tags, uint8_t* occ, cudaStream_t st, int max_blocks_per_sm)
{
    two = two && !any_hit;
    const bool few = n <= kFewRays;
    static const TraceKernel kernels[2][2][3] = {
        {{k_trace<false, false>, k_trace<true, false>, k_trace<false, false, true>},
         {k_trace<false, true>, k_trace<true, true>, k_trace<false, true, true>}},
        {{k_trace_group<false, false>, k_trace_group<true, false>, k_trace_group<false, false, true>},
         {k_trace_group<false, true>, k_trace_group<true, true>, k_trace_group<false, true, true>}}};
    const TraceKernel fn = kernels[few][tags != nullptr][any_hit ? 1 : (two ? 2 : 0)];
    // occupancy of the variant launched, on the context's device; calls on
    // one context are externally synchronised, so the per-context cache
    // needs no lock
    int& blocks_per_sm = ctx->trace_bps[(any_hit ? 1 : 0) | (tags ? 2 : 0) | (two ? 4 : 0) | (few ? 8 : 0)];
    if (blocks_per_sm == 0) {
        int b = 0;
        FF_CUDA_CHECK(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&b, fn, kTraceBlock, 0));
        blocks_per_sm = b < 1 ? 1 : b;
    }
    const int bps = !few && max_blocks_per_sm > 0 ? std::min(max_blocks_per_sm, blocks_per_sm) : blocks_per_sm;
    const uint64_t per_block = few ? kGroupRays : kTraceBlock;
    const uint64_t grid = std::min((uint64_t)ctx->num_sms * bps, (n + per_block - 1) / per_block);
    fn<<<dim3((unsigned)grid), dim3(kTraceBlock), 0, st>>>(bvh, d_rays, d_hits, n, counter, err, n_dev, tags, occ);
    FF_CUDA_CHECK(cudaGetLastError());
}

}  // namespace

void ff_launch_trace(ff_context* ctx, const ff_scene* s, const ff_ray* d_rays, uint64_t n, ff_hit* d_hits,
                     bool any_hit, bool two_sided)
{
    if (n == 0) return;
    unsigned long long* counter = reinterpret_cast<unsigned long long*>(ctx->counters());
    unsigned int* err = ctx->trace_err();
    FF_CUDA_CHECK(cudaMemsetAsync(counter, 0, sizeof(unsigned long long), ctx->stream));
    launch_trace(ctx, s->view(), d_rays, n, d_hits, any_hit, two_sided, counter, err, nullptr, nullptr, nullptr,
                 ctx->stream, 0);
}

// Same launch as ff_launch_trace, with the work counter and the error counter
// supplied by the caller instead of taken from the context's allocation.
void ff_launch_trace_scratch(ff_context* ctx, const ff_scene* s, const ff_ray* d_rays, uint64_t n, ff_hit* d_hits,
                             bool any_hit, unsigned long long* counter, unsigned int* err, bool two_sided)
{
    if (n == 0) return;
    launch_trace(ctx, s->view(), d_rays, n, d_hits, any_hit, two_sided, counter, err, nullptr, nullptr, nullptr, ctx->stream,
                 0);
}

// Trace a device-resident queue whose length the previous stage wrote to
// n_dev (at most cap rays), on the context's stream.  counter must be zeroed
// by the caller before the launch.  two_sided (closest hit only): the
// kernel honours the per-ray two-sided mark (the sign bit of tmin).
void ff_launch_trace_queue(ff_context* ctx, const FFBvhView& bvh, const ff_ray* d_rays, const uint32_t* n_dev,
                           uint64_t cap, ff_hit* d_hits, bool any_hit, unsigned long long* counter, unsigned int* err,
                           const uint32_t* tags, uint8_t* occ, cudaStream_t stream, bool two_sided, int max_blocks_per_sm)
{
    if (cap == 0) return;
    launch_trace(ctx, bvh, d_rays, cap, d_hits, any_hit, two_sided, counter, err, n_dev, tags, occ,
                 stream ? stream : ctx->stream, max_blocks_per_sm);
}
