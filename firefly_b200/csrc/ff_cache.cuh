// ff_cache.cuh — inputs of the learned radiance cache: the multiresolution
// hash-grid encoding of the position (16 levels x 2 features, 2^19 entries
// per level), degree-4 real spherical harmonics (16 coefficients) of the
// outgoing direction, the shading normal and the roughness, assembled into
// the 64 inputs of the MLP:
//   0..31  hash features, level l at 2l, 2l+1
//   32..47 SH(wo)
//   48..50 normal, 51 roughness, 52 constant 1 (the first layer's bias)
//   53..63 zero
#pragma once

#include <cuda_fp16.h>

#include "ff_common.cuh"

namespace ffc {

constexpr int kLevels = 16;
constexpr int kInputs = 64;
constexpr int kWidth = 64;
constexpr int kLayers = 5;          // 4 hidden layers of 64 (W0..W3) and the output layer W4
constexpr int kOutputs = 3;
constexpr int kTile = 128;          // records per tensor-core tile (M)

struct Grid {
    const __half2* table_h;         // [kLevels << log2_T] features used by the MLP
    float2* grad;                   // [kLevels << log2_T] gradient accumulator (training)
    uint32_t log2_T;
    float3 lo, inv_ext;             // position normalisation (scene box)
    float scale[kLevels];           // cells per unit cube side at each level
    uint32_t dense_side[kLevels];   // side+1 of a densely indexed level, 0 for hashed levels
    // The first cell_levels levels (dense ones of at most kCellMax cells) once
    // more, by cells: the 8 corner entries of a cell in one 32-byte sector, the
    // cells of level l from cell_off[l], x fastest.
    const uint4* cells;
    uint32_t cell_levels;
    uint32_t cell_off[kLevels];
};
constexpr uint32_t kCellMax = 1u << 18;   // cells of a level kept by cells (8 MB a level; the default levels have 10 in all)

// One record: a vertex (position, roughness, outgoing direction, normal)
// and a value (training: target radiance; render queries: path throughput).
struct alignas(16) Record {
    float px, py, pz, rough;
    float wx, wy, wz, v0;
    float nx, ny, nz, v1;
    uint32_t pixel;
    float v2, pad0, pad1;
};
static_assert(sizeof(Record) == 64, "record layout");

// A record in two 32-byte accesses; the loads only where the array sits on a
// 32-byte boundary (a caller's may not).
struct __align__(32) RecordHalf {
    float f[8];
};
__device__ __forceinline__ void store_record(Record* p, const Record& r)
{
    const RecordHalf* h = reinterpret_cast<const RecordHalf*>(&r);
    RecordHalf* q = reinterpret_cast<RecordHalf*>(p);
    st_sector(q, h[0]);
    st_sector(q + 1, h[1]);
}
__device__ __forceinline__ Record load_record(const Record* p)
{
    if (reinterpret_cast<uintptr_t>(p) & 31u) return *p;
    union {
        RecordHalf h[2];
        Record r;
    } u;
    u.h[0] = ld_sector(reinterpret_cast<const RecordHalf*>(p));
    u.h[1] = ld_sector(reinterpret_cast<const RecordHalf*>(p) + 1);
    return u.r;
}

__device__ __forceinline__ Record make_record(float3 pos, float rough, float3 wo, float3 n, float3 v, uint32_t pixel)
{
    Record r;
    r.px = pos.x;
    r.py = pos.y;
    r.pz = pos.z;
    r.rough = rough;
    r.wx = wo.x;
    r.wy = wo.y;
    r.wz = wo.z;
    r.v0 = v.x;
    r.nx = n.x;
    r.ny = n.y;
    r.nz = n.z;
    r.v1 = v.y;
    r.pixel = pixel;
    r.v2 = v.z;
    r.pad0 = r.pad1 = 0.f;
    return r;
}

__device__ __forceinline__ float3 normalised_pos(const Grid& g, float px, float py, float pz)
{
    float3 p = make_float3((px - g.lo.x) * g.inv_ext.x, (py - g.lo.y) * g.inv_ext.y, (pz - g.lo.z) * g.inv_ext.z);
    p.x = fminf(fmaxf(p.x, 0.f), 1.f);
    p.y = fminf(fmaxf(p.y, 0.f), 1.f);
    p.z = fminf(fmaxf(p.z, 0.f), 1.f);
    return p;
}

// The level-l cell holding p and p's place in it.
struct Cell {
    uint32_t x, y, z;
    float tx, ty, tz;
};
__device__ __forceinline__ Cell level_cell(const Grid& g, int l, float3 p)
{
    const float s = g.scale[l];
    const float fx = p.x * s, fy = p.y * s, fz = p.z * s;
    const int cells = (int)s;
    int ix = min((int)floorf(fx), cells - 1), iy = min((int)floorf(fy), cells - 1), iz = min((int)floorf(fz), cells - 1);
    ix = max(ix, 0);
    iy = max(iy, 0);
    iz = max(iz, 0);
    Cell c;
    c.x = (uint32_t)ix, c.y = (uint32_t)iy, c.z = (uint32_t)iz;
    c.tx = fminf(fmaxf(fx - (float)ix, 0.f), 1.f);
    c.ty = fminf(fmaxf(fy - (float)iy, 0.f), 1.f);
    c.tz = fminf(fmaxf(fz - (float)iz, 0.f), 1.f);
    return c;
}
// Trilinear weight and table index of corner k (bit 0 = +x, bit 1 = +y, bit 2 = +z).
__device__ __forceinline__ float corner_weight(const Cell& c, int k)
{
    return ((k & 1) ? c.tx : 1.f - c.tx) * (((k >> 1) & 1) ? c.ty : 1.f - c.ty) * ((k >> 2) ? c.tz : 1.f - c.tz);
}
__device__ __forceinline__ uint32_t corner_index(const Grid& g, int l, const Cell& c, int k)
{
    const uint32_t x = c.x + (k & 1), y = c.y + ((k >> 1) & 1), z = c.z + (k >> 2);
    const uint32_t side = g.dense_side[l];
    const uint32_t i = side ? x + side * (y + side * z) : (x * 1u) ^ (y * 2654435761u) ^ (z * 805459861u);
    return ((uint32_t)l << g.log2_T) + (i & ((1u << g.log2_T) - 1u));
}

// Entry j (0..3) of four packed half2 entries.
__device__ __forceinline__ uint32_t pick4(uint4 q, uint32_t j)
{
    return j == 0u ? q.x : (j == 1u ? q.y : (j == 2u ? q.z : q.w));
}
__device__ __forceinline__ float2 half2_bits(uint32_t u)
{
    __half2 h;
    *reinterpret_cast<uint32_t*>(&h) = u;
    return __half22float2(h);
}

// The table entries of one level's 8 corners, loaded without branches, so that
// the loads of several levels are in flight together.
//
// By cells, one 32-byte load.  Else corners k (x) and k + 1 (x + 1) share y
// and z, so their entries usually sit in one aligned group of four: on a
// dense level they are neighbours, and on a hashed level x enters the hash by
// XOR, so the two indices differ in the bits of x ^ (x + 1), which stay below
// 4 three times in four.  The group is one 16-byte load (one sector per lane
// instead of two); an entry outside it is read alone, by a predicated load.
// With a branch around that load every level's four pairs waited for one
// another: 16 levels took 100,000 cycles in a launch of one tile per SM.
struct CornerEntries {
    uint32_t e[8];
};
__device__ __forceinline__ CornerEntries cell_entries(const Grid& g, int l, const Cell& c)
{
    const uint32_t n = (uint32_t)g.scale[l];
    const uint4* p = g.cells + 2 * (size_t)(g.cell_off[l] + c.x + n * (c.y + n * c.z));
    CornerEntries r;
    asm("ld.global.v8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
        : "=r"(r.e[0]), "=r"(r.e[1]), "=r"(r.e[2]), "=r"(r.e[3]), "=r"(r.e[4]), "=r"(r.e[5]), "=r"(r.e[6]), "=r"(r.e[7])
        : "l"(p));
    return r;
}
struct PairLoads {
    uint4 q[4];
    uint32_t alone[4], i0[4], i1[4];
};
__device__ __forceinline__ PairLoads load_pairs(const Grid& g, int l, const Cell& c)
{
    PairLoads r;
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        r.i0[k] = corner_index(g, l, c, 2 * k);
        r.i1[k] = corner_index(g, l, c, 2 * k + 1);
        r.q[k] = __ldg(reinterpret_cast<const uint4*>(g.table_h + (r.i0[k] & ~3u)));
        asm("{\n\t.reg .pred p;\n\t"
            "setp.ge.u32 p, %2, 4;\n\t"
            "mov.b32 %0, 0;\n\t"
            "@p ld.global.nc.b32 %0, [%1];\n\t}"
            : "=r"(r.alone[k])
            : "l"(g.table_h + r.i1[k]), "r"(r.i0[k] ^ r.i1[k]));
    }
    return r;
}
__device__ __forceinline__ CornerEntries pair_entries(const PairLoads& a)
{
    CornerEntries r;
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        r.e[2 * k] = pick4(a.q[k], a.i0[k] & 3u);
        r.e[2 * k + 1] = (a.i0[k] ^ a.i1[k]) < 4u ? pick4(a.q[k], a.i1[k] & 3u) : a.alone[k];
    }
    return r;
}
// Trilinear feature: the sum over the corners in order.
__device__ __forceinline__ float2 blend(const Cell& c, const CornerEntries& e)
{
    float2 f = make_float2(0.f, 0.f);
#pragma unroll
    for (int k = 0; k < 8; ++k) {
        const float w = corner_weight(c, k);
        const float2 v = half2_bits(e.e[k]);
        f.x += w * v.x;
        f.y += w * v.y;
    }
    return f;
}
// The features of levels l and l + 1 at p.
__device__ __forceinline__ void two_features(const Grid& g, int l, float3 p, float2& fa, float2& fb)
{
    const Cell ca = level_cell(g, l, p), cb = level_cell(g, l + 1, p);
    if (l + 1 < (int)g.cell_levels) {
        const CornerEntries a = cell_entries(g, l, ca), b = cell_entries(g, l + 1, cb);
        fa = blend(ca, a);
        fb = blend(cb, b);
    } else if (l < (int)g.cell_levels) {
        const CornerEntries a = cell_entries(g, l, ca);
        const PairLoads b = load_pairs(g, l + 1, cb);
        fa = blend(ca, a);
        fb = blend(cb, pair_entries(b));
    } else {
        fa = blend(ca, pair_entries(load_pairs(g, l, ca)));
        fb = blend(cb, pair_entries(load_pairs(g, l + 1, cb)));
    }
}

// Real spherical harmonics of degree 0..3 (16 functions) of the unit
// direction (x, y, z), in the order (l, m) = (0,0), (1,-1), (1,0), (1,1),
// (2,-2) .. (2,2), (3,-3) .. (3,3); normalisation constants from
// sqrt((2l+1)/(4 pi) * (l-|m|)!/(l+|m|)!), with the Condon-Shortley phase.
__device__ __forceinline__ void sh16(float x, float y, float z, float* o)
{
    const float c00 = (float)(0.5 / 1.7724538509055160273);                 // 1/(2 sqrt(pi))
    const float c1 = (float)(0.48860251190291992159);                       // sqrt(3/(4 pi))
    const float c2a = (float)(1.0925484305920790705);                       // sqrt(15/pi)/2
    const float c2b = (float)(0.31539156525252000603);                      // sqrt(5/pi)/4
    const float c2c = (float)(0.54627421529603953527);                      // sqrt(15/pi)/4
    const float c3a = (float)(0.59004358992664351035);                      // sqrt(35/(2 pi))/4
    const float c3b = (float)(2.8906114426405540554);                       // sqrt(105/pi)/2
    const float c3c = (float)(0.45704579946446573616);                      // sqrt(21/(2 pi))/4
    const float c3d = (float)(0.37317633259011539141);                      // sqrt(7/pi)/4
    const float c3e = (float)(1.4453057213202770277);                       // sqrt(105/pi)/4
    const float xx = x * x, yy = y * y, zz = z * z;
    o[0] = c00;
    o[1] = -c1 * y;
    o[2] = c1 * z;
    o[3] = -c1 * x;
    o[4] = c2a * x * y;
    o[5] = -c2a * y * z;
    o[6] = c2b * (3.f * zz - 1.f);
    o[7] = -c2a * x * z;
    o[8] = c2c * (xx - yy);
    o[9] = -c3a * y * (3.f * xx - yy);
    o[10] = c3b * x * y * z;
    o[11] = -c3c * y * (5.f * zz - 1.f);
    o[12] = c3d * z * (5.f * zz - 3.f);
    o[13] = -c3c * x * (5.f * zz - 1.f);
    o[14] = c3e * z * (xx - yy);
    o[15] = -c3a * x * (xx - 3.f * yy);
}

}  // namespace ffc
