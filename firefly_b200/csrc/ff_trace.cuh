// ff_trace.cuh — ray traversal of the 8-wide quantised BVH and the
// reference-exact ray/triangle tests.  Used by the standalone trace kernel
// (ff_trace.cu) and by the wavefront stages.
#pragma once

#include "ff_common.cuh"

// Per-ray traversal state kept in registers.
//
// Two-sided closest hits (rays inside a refracting object, and ff_trace with
// FF_TRACE_TWO_SIDED) ride on the sign bit of tmin in the traversal kernels
// instantiated with TWO = true: a ray whose tmin has its sign bit set (-0.0
// for tmin 0) also accepts back faces, and such a ray's interval starts at
// |tmin|.  A back-face hit keeps bit 31 of prim set.  Kernels with TWO =
// false never look at the sign and cull back faces as the reference does.
struct FFRayState {
    float3 o, d, inv;
    float tmin, tmax;   // closest-hit: tmax is the current best t (starts at min(tmax, K_HUGE))
    float u, v;
    uint32_t prim;      // original triangle index, 0xffffffff = none; bit 31: back face (TWO kernels)
    uint32_t oct_inv;   // 7 ^ octant of d (bit a set = d_a < 0)
};

// A closest hit as the C ABI reports it: prim = the original index for a
// front face, -2 - index for a back face of a two-sided ray, -1 for none.
FF_D ff_hit ff_hit_of(const FFRayState& r)
{
    int32_t prim = -1;
    if (r.prim != 0xffffffffu) {
        const int32_t id = (int32_t)(r.prim & ~kBackFace);
        prim = (r.prim & kBackFace) ? -2 - id : id;
    }
    return ff_hit{r.tmax, r.u, r.v, prim};
}

FF_D float safe_inv(float x)
{
    const float tiny = 1e-20f;
    return 1.0f / (fabsf(x) > tiny ? x : copysignf(tiny, x));
}

FF_D void ff_ray_setup(FFRayState& r, float3 o, float3 d, float tmin, float tmax, bool any)
{
    r.o = o;
    r.d = d;
    r.inv = make_float3(safe_inv(d.x), safe_inv(d.y), safe_inv(d.z));
    r.tmin = tmin;
    r.tmax = any ? tmax : fminf(tmax, FF_K_HUGE);
    r.u = r.v = 0.f;
    r.prim = 0xffffffffu;
    r.oct_inv = (d.x < 0.f ? 0u : 1u) | (d.y < 0.f ? 0u : 2u) | (d.z < 0.f ? 0u : 4u);
}

// Byte s of (lo4, hi4) as the float 2^23 + byte, without an integer-to-float
// conversion: one byte permute puts the byte in the low mantissa bits under
// the exponent byte 0x4B; the node test subtracts 2^23 from two such values
// with one packed add (exact for 0..255).
FF_D float byte_plus_2p23(uint32_t lo4, uint32_t hi4, int s)
{
    return __uint_as_float(__byte_perm(s < 4 ? lo4 : hi4, 0x4B000000u, 0x7440u | (uint32_t)(s & 3)));
}

// Three-input min / max of sm_100 (one instruction instead of two; exact,
// and NaN-ignoring like fminf / fmaxf).
FF_D float fmin3f(float a, float b, float c)
{
    float r;
    asm("min.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
    return r;
}
FF_D float fmax3f(float a, float b, float c)
{
    float r;
    asm("max.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
    return r;
}

// Intersect the ray with the 8 child boxes of node idx.  Returns the new node
// group (x = child_base, y = hit bits 24..31 in traversal order | imask) and
// the triangle group (x = tri_base, y = 24-bit mask of triangles to test).
FF_D void ff_intersect_node(const FFNode8* __restrict__ nodes, uint32_t idx, const FFRayState& r,
                            uint2& node_group, uint2& tri_group)
{
    const uint4* p = reinterpret_cast<const uint4*>(nodes + idx);
    const uint4 n0 = __ldg(p + 0);
    const uint4 n1 = __ldg(p + 1);
    const uint4 n2 = __ldg(p + 2);
    const uint4 n3 = __ldg(p + 3);
    const uint4 n4 = __ldg(p + 4);
    const float px = __uint_as_float(n0.x), py = __uint_as_float(n0.y), pz = __uint_as_float(n0.z);
    const uint32_t ex = n0.w & 0xffu, ey = (n0.w >> 8) & 0xffu, ez = (n0.w >> 16) & 0xffu;
    const uint32_t imask = n0.w >> 24;
    const float sx = __uint_as_float(ex << 23), sy = __uint_as_float(ey << 23), sz = __uint_as_float(ez << 23);
    const float ax = sx * r.inv.x, ay = sy * r.inv.y, az = sz * r.inv.z;
    const float bx = (px - r.o.x) * r.inv.x, by = (py - r.o.y) * r.inv.y, bz = (pz - r.o.z) * r.inv.z;
    // near/far plane words per axis, chosen by the sign of the direction
    const uint32_t nx0 = r.inv.x >= 0.f ? n2.x : n3.z, nx1 = r.inv.x >= 0.f ? n2.y : n3.w;
    const uint32_t fx0 = r.inv.x >= 0.f ? n3.z : n2.x, fx1 = r.inv.x >= 0.f ? n3.w : n2.y;
    const uint32_t ny0 = r.inv.y >= 0.f ? n2.z : n4.x, ny1 = r.inv.y >= 0.f ? n2.w : n4.y;
    const uint32_t fy0 = r.inv.y >= 0.f ? n4.x : n2.z, fy1 = r.inv.y >= 0.f ? n4.y : n2.w;
    const uint32_t nz0 = r.inv.z >= 0.f ? n3.x : n4.z, nz1 = r.inv.z >= 0.f ? n3.y : n4.w;
    const uint32_t fz0 = r.inv.z >= 0.f ? n4.z : n3.x, fz1 = r.inv.z >= 0.f ? n4.w : n3.y;
    // the widening as explicit fused multiply-adds: the same result in every
    // translation unit, whatever its contraction setting (-fmad)
    const float tb = __fmaf_rn(fabsf(r.tmax), FF_BOX_WIDEN, r.tmax);
    // packed FP32: one add removes 2^23 from two plane bytes and one fma gives
    // two slab distances (the same IEEE operations per lane as fmaf, so the
    // same values): x and y of the near planes, of the far planes, and the
    // near and far z
    const float2 axy = make_float2(ax, ay), bxy = make_float2(bx, by), azz = make_float2(az, az),
                 bzz = make_float2(bz, bz);
    const float2 m23 = make_float2(-8388608.0f, -8388608.0f);
    // meta bytes, four at a time (after Ylitie et al. 2017, "Efficient incoherent
    // ray traversal on GPUs through compressed wide BVHs"): where an internal child (offset bits 24..31,
    // both upper bits set, which no leaf's offset has) or a leaf's triangles
    // go in the 32-bit answer, and the bits that go there (one bit for an
    // internal child, the unary count of a leaf, none for an empty slot, so
    // that its degenerate box needs no test).  With the masks formed per child
    // the 64-spp step took 245.1 ms, so 240.4; 16.8M incoherent closest hits
    // 1461 and 1413 us.
    const uint32_t oct4 = r.oct_inv * 0x01010101u;
    uint32_t shift4[2], bits4[2];
#pragma unroll
    for (int k = 0; k < 2; ++k) {
        const uint32_t meta4 = k == 0 ? n1.z : n1.w;
        const uint32_t inner4 = ((meta4 & (meta4 << 1) & 0x10101010u) >> 4) * 0xffu;
        shift4[k] = (meta4 ^ (oct4 & inner4)) & 0x1f1f1f1fu;
        bits4[k] = (meta4 >> 5) & 0x07070707u;
    }
    uint32_t hits = 0;
#pragma unroll
    for (int s = 0; s < 8; ++s) {
        const float2 qn = __fadd2_rn(make_float2(byte_plus_2p23(nx0, nx1, s), byte_plus_2p23(ny0, ny1, s)), m23);
        const float2 qf = __fadd2_rn(make_float2(byte_plus_2p23(fx0, fx1, s), byte_plus_2p23(fy0, fy1, s)), m23);
        const float2 qz = __fadd2_rn(make_float2(byte_plus_2p23(nz0, nz1, s), byte_plus_2p23(fz0, fz1, s)), m23);
        const float2 tnxy = __ffma2_rn(qn, axy, bxy);
        const float2 tfxy = __ffma2_rn(qf, axy, bxy);
        const float2 tz = __ffma2_rn(qz, azz, bzz);
        float tn = fmax3f(tnxy.x, tnxy.y, tz.x);
        float tf = fmin3f(tfxy.x, tfxy.y, tz.y);
        tn = __fmaf_rn(-fabsf(tn), FF_BOX_WIDEN, tn);
        tf = __fmaf_rn(fabsf(tf), FF_BOX_WIDEN, tf);
        if (fmaxf(tn, r.tmin) <= fminf(tf, tb))
            hits |= __byte_perm(bits4[s >> 2], 0u, 0x4440u | (uint32_t)(s & 3))
                    << __byte_perm(shift4[s >> 2], 0u, 0x4440u | (uint32_t)(s & 3));
    }
    node_group = make_uint2(n1.x, (hits & 0xff000000u) | imask);
    tri_group = make_uint2(n1.y, hits & 0x00ffffffu);
}

// dTriangle::intersect with TEST_CULL (CUDA-RayTracer/dTriangle.cu:34-61),
// then dTriangle::hit's t < 0 rejection (:99) and intersect()'s strict
// t < tmin acceptance (:170), with ties to the lowest original index.  The
// edge tests compare float values, so they run in FP32 exactly as the
// reference's float-vs-double comparisons; the FP64 reciprocal and products
// run only for candidates that pass them.
//
// TWO: a ray with the sign bit of tmin set also takes back faces (no
// reference counterpart: the reference only culls).  A back face is a
// determinant at or below -K_EPSILON; the test then runs on the negated
// determinant and numerators (negation is exact), i.e. the mirror image of
// the front-face test, and the hit keeps kBackFace in prim.  Front faces go
// through exactly the arithmetic above.
//
// Both tests run straight through to one branch: in a warp of diverged rays
// some lane nearly always reaches the last FP32 comparison, so leaving at
// each one only adds branches (3M any-hit rays on the 1.3M-triangle mesh 241
// -> 230 us, its 64-spp step 240.4 -> 234.8 ms).
struct FFCandidate {
    float t, uf, vf;   // uf, vf: numerators of u and v over det
    double inv_det;
    uint32_t id;       // original index
    bool back;         // a back face (TWO)
    FF_D float u() const { return __double2float_rn(__dmul_rn((double)uf, inv_det)); }
    FF_D float v() const { return __double2float_rn(__dmul_rn((double)vf, inv_det)); }
};
// The test but for the comparison with the best hit so far.
template <bool TWO>
FF_D bool ff_candidate(const FFTri* __restrict__ tris, uint32_t k, const FFRayState& r, FFCandidate& h)
{
    const float4 a = __ldg(&tris[k].a);
    const float4 b = __ldg(&tris[k].b);
    const float4 c = __ldg(&tris[k].c);
    const float3 v0 = make_float3(a.x, a.y, a.z);
    const float3 e1 = make_float3(b.x, b.y, b.z);
    const float3 e2 = make_float3(c.x, c.y, c.z);
    const float3 pvec = rn_cross(r.d, e2);
    float det = rn_dot(e1, pvec);
    bool out = det < FF_K_EPSILON;
    float sg = 1.f;
    if (TWO) {
        h.back = signbit(r.tmin) && det <= -FF_K_EPSILON;
        sg = h.back ? -1.f : 1.f;
        det = h.back ? -det : det;
        out = out && !h.back;
    }
    const float3 tvec = rn_sub(r.o, v0);
    h.uf = TWO ? sg * rn_dot(tvec, pvec) : rn_dot(tvec, pvec);
    out |= (h.uf < 0.f) | (h.uf > det);
    const float3 qvec = rn_cross(tvec, e1);
    h.vf = TWO ? sg * rn_dot(r.d, qvec) : rn_dot(r.d, qvec);
    out |= (h.vf < 0.f) | (__fadd_rn(h.uf, h.vf) > det);
    const float tf = TWO ? sg * rn_dot(e2, qvec) : rn_dot(e2, qvec);
    if (out) return false;
    h.inv_det = __drcp_rn((double)det);
    h.t = __double2float_rn(__dmul_rn((double)tf, h.inv_det));
    h.id = (uint32_t)__float_as_int(a.w);
    return !(h.t < 0.f) && h.t >= (TWO ? fabsf(r.tmin) : r.tmin);
}
// Whether a candidate replaces the best hit so far.
template <bool TWO>
FF_D bool ff_better(const FFRayState& r, float t, uint32_t id)
{
    const uint32_t best = TWO ? (r.prim & ~kBackFace) : r.prim;
    return t < r.tmax || (t == r.tmax && r.prim != 0xffffffffu && id < best);
}

template <bool TWO = false>
FF_D void ff_test_tri_closest(const FFTri* __restrict__ tris, uint32_t k, FFRayState& r)
{
    FFCandidate h;
    if (ff_candidate<TWO>(tris, k, r, h) && ff_better<TWO>(r, h.t, h.id)) {
        r.tmax = h.t;
        r.prim = (TWO && h.back) ? (h.id | kBackFace) : h.id;
        r.u = h.u();
        r.v = h.v();
    }
}

// dTriangle::shadow_hit (CUDA-RayTracer/dTriangle.cu:110-138) and the
// t < tmin test of intersect_shadows (:233).  Returns true on an occluder,
// with its t and original index.  An FP32 pre-test rejects candidates that
// the FP64 test would certainly reject (sign of u, v and u + v > 1 with
// margin); the FP64 test decides the rest.
FF_D bool ff_occluder(const FFTri* __restrict__ tris, uint32_t k, const FFRayState& r, float& t, uint32_t& id)
{
    const float4 a = __ldg(&tris[k].a);
    const float4 b = __ldg(&tris[k].b);
    const float4 c = __ldg(&tris[k].c);
    const float3 v0 = make_float3(a.x, a.y, a.z);
    const float3 e1 = make_float3(b.x, b.y, b.z);
    const float3 e2 = make_float3(c.x, c.y, c.z);
    const float3 pvec = rn_cross(r.d, e2);
    const float det = rn_dot(e1, pvec);
    bool out = (det > -FF_K_EPSILON) & (det < FF_K_EPSILON);
    const float3 tvec = rn_sub(r.o, v0);
    const float uf = rn_dot(tvec, pvec);
    const bool neg = det < 0.f;
    out |= (uf != 0.f) & ((uf < 0.f) != neg);  // u < 0
    const float3 qvec = rn_cross(tvec, e1);
    const float vf = rn_dot(r.d, qvec);
    out |= (vf != 0.f) & ((vf < 0.f) != neg);  // v < 0
    out |= fabsf(uf) + fabsf(vf) > fabsf(det) * 1.000001f;  // u + v > 1
    if (out) return false;
    const double inv_det = __drcp_rn((double)det);
    const double u = __dmul_rn((double)uf, inv_det);
    if (u < 0.0 || u > 1.0) return false;
    const double v = __dmul_rn((double)vf, inv_det);
    if (v < 0.0 || __dadd_rn(u, v) > 1.0) return false;
    const float tf = rn_dot(e2, qvec);
    t = __double2float_rn(__dmul_rn((double)tf, inv_det));
    id = (uint32_t)__float_as_int(a.w);
    return !(t < 0.f) && t >= r.tmin && t < r.tmax;
}

FF_D bool ff_test_tri_any(const FFTri* __restrict__ tris, uint32_t k, FFRayState& r)
{
    float t;
    uint32_t id;
    if (!ff_occluder(tris, k, r, t, id)) return false;
    r.prim = id;
    r.tmax = t;  // the traversal ends here; tmax now reports the occluder's t
    return true;
}

// Traversal stack: kShortStack entries per thread in shared memory (strided
// by the block size so a warp's pushes hit distinct banks), deeper entries in
// a local array.  Every push happens at most once per BVH level, so the depth
// needed is bounded by the BVH depth, which the host checks against
// kShortStack + kLocalStack at build time.
constexpr int kShortStack = 8;
constexpr int kLocalStack = 56;
constexpr int kMaxStack = kShortStack + kLocalStack;

struct FFStack {
    uint2* sm;     // this thread's column in shared memory
    int stride;    // block size
    int sp;
    bool overflow; // set instead of writing past the end (never expected: depth is checked at build)
    uint2 local[kLocalStack];
    FF_D void reset()
    {
        sp = 0;
        overflow = false;
    }
    FF_D void push(uint2 v)
    {
        if (sp >= kMaxStack) {
            overflow = true;
            return;
        }
        if (sp < kShortStack) sm[sp * stride] = v;
        else local[sp - kShortStack] = v;
        ++sp;
    }
    FF_D uint2 pop()
    {
        --sp;
        return sp < kShortStack ? sm[sp * stride] : local[sp - kShortStack];
    }
};

// Work counters for ff_traverse_step: FFNoCount compiles to nothing (the
// product kernels); FFCount tallies the node records fetched and the
// triangles tested (ff_trace_count).
struct FFNoCount {
    FF_D void node() {}
    FF_D void tri() {}
};
struct FFCount {
    unsigned long long nodes = 0, tris = 0;
    FF_D void node() { ++nodes; }
    FF_D void tri() { ++tris; }
};

// One traversal step: take the next child node of the current group, test
// its children, then test the triangles it exposed.  Returns true when the
// ray is finished.
template <bool ANY, class C, bool TWO = false>
FF_D bool ff_traverse_step(const FFBvhView& bvh, FFRayState& r, uint2& cur, FFStack& st, C& count)
{
    uint2 tri_group = make_uint2(0u, 0u);
    if (cur.y & 0xff000000u) {
        const uint32_t bit = 31u - __clz(cur.y & 0xff000000u);
        cur.y &= ~(1u << bit);
        const uint32_t slot = (bit - 24u) ^ r.oct_inv;
        const uint32_t child = cur.x + __popc(cur.y & 0xffu & ((1u << slot) - 1u));
        if (cur.y & 0xff000000u) st.push(cur);
        if (child >= bvh.num_nodes) {  // never taken on a validated BVH
            st.overflow = true;
            return true;
        }
        count.node();
        ff_intersect_node(bvh.nodes, child, r, cur, tri_group);
    }
    while (tri_group.y) {
        const uint32_t i = __ffs(tri_group.y) - 1;
        tri_group.y &= tri_group.y - 1;
        if (tri_group.x + i >= bvh.num_tris) {
            st.overflow = true;
            return true;
        }
        count.tri();
        if (ANY) {
            if (ff_test_tri_any(bvh.tris, tri_group.x + i, r)) return true;
        } else {
            ff_test_tri_closest<TWO>(bvh.tris, tri_group.x + i, r);
        }
    }
    if (!(cur.y & 0xff000000u)) {
        if (st.sp == 0) return true;
        cur = st.pop();
    }
    return st.overflow;
}
template <bool ANY, bool TWO = false>
FF_D bool ff_traverse_step(const FFBvhView& bvh, FFRayState& r, uint2& cur, FFStack& st)
{
    FFNoCount none;
    return ff_traverse_step<ANY, FFNoCount, TWO>(bvh, r, cur, st, none);
}

// Root group: a fake parent whose only internal child (node 0) sits in the
// slot the ray visits first.
FF_D uint2 ff_root_group(const FFRayState& r)
{
    return make_uint2(0u, (1u << 31) | (1u << (7u ^ r.oct_inv)));
}

// One whole traversal per thread (megakernel paths): closest hit of the ray
// (o, d, [0, inf)), two-sided when `two` (h.prim = -2 - index for a back
// face), or any hit of `ray`; a traversal that exceeds its step bound or
// overflows the stack counts in *err and reports what it found.  Returns
// whether anything was hit.
FF_D bool ff_closest_hit(const FFBvhView& bvh, float3 o, float3 d, FFStack& st, unsigned int* err, ff_hit& h,
                         bool two = false)
{
    FFRayState r;
    ff_ray_setup(r, o, d, two ? -0.f : 0.f, __int_as_float(0x7f800000), false);
    if (bvh.num_nodes) {
        uint2 cur = ff_root_group(r);
        st.reset();
        uint32_t steps = 0;
        while (!ff_traverse_step<false, true>(bvh, r, cur, st)) {
            if (++steps > bvh.num_nodes + 2 || st.overflow) {
                atomicAdd(err, 1u);
                break;
            }
        }
    }
    h = ff_hit_of(r);
    return h.prim != -1;
}

FF_D bool ff_occluded(const FFBvhView& bvh, const ff_ray& ray, FFStack& st, unsigned int* err)
{
    if (!bvh.num_nodes) return false;
    FFRayState r;
    ff_ray_setup(r, make_float3(ray.ox, ray.oy, ray.oz), make_float3(ray.dx, ray.dy, ray.dz), ray.tmin, ray.tmax, true);
    uint2 cur = ff_root_group(r);
    st.reset();
    uint32_t steps = 0;
    while (!ff_traverse_step<true>(bvh, r, cur, st)) {
        if (++steps > bvh.num_nodes + 2 || st.overflow) {
            atomicAdd(err, 1u);
            break;
        }
    }
    return r.prim != 0xffffffffu;
}
