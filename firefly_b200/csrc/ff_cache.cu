// ff_cache.cu — learned radiance cache: a multiresolution hash grid and a
// 64-wide MLP (4 hidden ReLU layers, 3 outputs, no biases except through the
// constant input) evaluated and trained on the fifth-generation tensor cores.
//
// Both kernels work on tiles of 128 records; thread (warp w, lane) owns row
// r = 32 (w % 4) + lane of a tile, which is exactly the part of a 128-lane
// TMEM accumulator its warp may read (subpartition w % 4).
//   k_cache_infer  encode -> X (smem) -> 5 MMAs chains (K = 64 in four K=16
//                  steps) with a ReLU/bf16 epilogue TMEM -> smem between
//                  layers; activations overwrite the input tile.  Its CTA
//                  runs kGroups independent tile pipelines of 4 warps (one
//                  thread per row, all 64 columns) over one copy of the
//                  weights: while one group waits on its MMAs the others
//                  gather hash-grid features, so the encoder's L2 gathers
//                  overlap the tensor-core chains of the other tiles.  The
//                  gathers bound it: about 54 sectors a query from L2 (2M
//                  queries 732 us with 80 sectors and a branch around every
//                  fifth load, 621 us so).  With at most one tile a CTA the
//                  groups share its encoding (4,096 records 61 -> 38 us).
//   k_cache_train  the same forward keeping every layer's activations, the
//                  relative-L2 loss gradient, then per layer (top down) the
//                  weight gradient act^T * delta (M = 64, both operands
//                  MN-major, accumulated in TMEM over all tiles of the CTA)
//                  and the input gradient delta * W (W read MN-major from
//                  the forward image); the input gradient of the hash
//                  features is scattered to the grid's FP32 gradient.
//                  Four threads per row (quarter h = w / 4 of the columns):
//                  a batch of 16,384 is one tile per SM, so what counts is
//                  the chain within a tile.  Clocks of a tile, before and
//                  after: encoding 35,000 and 14,000 (branch-free loads,
//                  levels dealt out evenly, twice the threads), the forward
//                  layers with the wait for the slowest warp 19,000 and
//                  11,000, scatter 38,000 and 31,000 (pairs of entries in one
//                  atomic; bound by the atomics in L2).
// Weights live in FP32 (master), their bf16 images pre-swizzled for shared
// memory; Adam updates both.  The grid keeps FP32 features with an FP16
// copy that the encoder reads (16 x 2^19 x 4 B = 32 MB, L2-resident), the
// coarse levels of it by cells (10 MB).
#include <cuda_bf16.h>
#include <cuda_fp16.h>

#include <atomic>
#include <cmath>
#include <new>

#include "ff_cache.cuh"
#include "ff_internal.h"
#include "ff_umma.cuh"

using namespace ffc;
using namespace ffu;

namespace {

constexpr int kThreads = 512;                             // training: four threads per row
constexpr uint32_t kTileBytes = 128u * 128u;             // 128 rows x 64 bf16
constexpr uint32_t kWBytes = 64u * 128u;                  // one 64 x 64 bf16 weight image
constexpr uint32_t kImgBytes = kLayers * kWBytes;         // 40 KB
constexpr uint32_t kParams = kLayers * kWidth * kWidth;   // FP32 master weights (W4 rows >= 3 stay zero)
constexpr uint32_t kWaitPolls = 1u << 22;
constexpr int kGroups = 3;                                // inference: tile pipelines per CTA
constexpr int kInferThreads = 128 * kGroups;
constexpr uint32_t kInferSmem = kImgBytes + kGroups * kTileBytes + 1024 + 64;
constexpr uint32_t kTrainSmem = kImgBytes + 6 * kTileBytes + 1024 + 64;
constexpr uint32_t kTrainTmemCols = 512;                  // D (64) + 5 weight-gradient accumulators (5 x 64)
constexpr uint32_t kInferTmemCols = 256;                 // 64 per group, allocated as a power of two

constexpr uint32_t ID_FWD = idesc_bf16(128, 64, false, false);
constexpr uint32_t ID_OUT = idesc_bf16(128, 16, false, false);
constexpr uint32_t ID_DGRAD = idesc_bf16(128, 64, false, true);
constexpr uint32_t ID_WGRAD = idesc_bf16(64, 64, true, true);

__device__ __forceinline__ uint32_t pack_bf16(float a, float b)
{
    __nv_bfloat162 v = __floats2bfloat162_rn(a, b);
    return *reinterpret_cast<uint32_t*>(&v);
}
__device__ __forceinline__ float2 unpack_bf16(uint32_t u)
{
    __nv_bfloat162 v = *reinterpret_cast<__nv_bfloat162*>(&u);
    return __bfloat1622float2(v);
}

// 8 values -> chunk c of row r of a swizzled tile
__device__ __forceinline__ void store_chunk(uint8_t* tile, uint32_t r, uint32_t c, const float* v)
{
    uint4 q = make_uint4(pack_bf16(v[0], v[1]), pack_bf16(v[2], v[3]), pack_bf16(v[4], v[5]), pack_bf16(v[6], v[7]));
    *reinterpret_cast<uint4*>(tile + r * 128u + (((c ^ (r & 7u)) & 7u) << 4)) = q;
}
__device__ __forceinline__ uint4 load_chunk(const uint8_t* tile, uint32_t r, uint32_t c)
{
    return *reinterpret_cast<const uint4*>(tile + r * 128u + (((c ^ (r & 7u)) & 7u) << 4));
}

// The hash features of row r, level pairs first, first + step, ... of 8 (two
// levels: half a 16-byte chunk).  The first levels cost one load by cells, the
// later ones five, so threads that share a row take pairs in turn.
__device__ __forceinline__ void encode_levels(const Grid& g, const Record& rec, bool valid, uint32_t r, uint8_t* tile,
                                              uint32_t first, uint32_t step)
{
    const float3 p = valid ? normalised_pos(g, rec.px, rec.py, rec.pz) : make_float3(0.f, 0.f, 0.f);
#pragma unroll 1
    for (uint32_t l = 2u * first; l < (uint32_t)kLevels; l += 2u * step) {
        float2 a, b;
        two_features(g, (int)l, p, a, b);
        uint2 q = make_uint2(pack_bf16(a.x, a.y), pack_bf16(b.x, b.y));
        if (!valid) q = make_uint2(0u, 0u);
        *reinterpret_cast<uint2*>(tile + r * 128u + ((((l >> 2) ^ (r & 7u)) & 7u) << 4) + ((l & 2u) << 2)) = q;
    }
}

// The other 32 inputs of row r, chunk by chunk: 4 and 5 the spherical
// harmonics, 6 normal, roughness and the constant, 7 zero.
__device__ __forceinline__ void encode_chunk(const Record& rec, bool valid, uint32_t r, uint8_t* tile, uint32_t chunk)
{
    float f[16];
#pragma unroll
    for (int k = 0; k < 16; ++k) f[k] = 0.f;
    if (valid && chunk < 6) {
        sh16(rec.wx, rec.wy, rec.wz, f);
        if (chunk == 5) {
#pragma unroll
            for (int k = 0; k < 8; ++k) f[k] = f[8 + k];
        }
    } else if (valid && chunk == 6) {
        f[0] = rec.nx;
        f[1] = rec.ny;
        f[2] = rec.nz;
        f[3] = rec.rough;
        f[4] = 1.f;
    }
    store_chunk(tile, r, chunk, f);
}

// ReLU epilogue: TMEM columns [32h, 32h+32) of row r -> chunks 4h..4h+3 of
// dst, and [16h, 16h+16) -> chunks 2h, 2h + 1.
__device__ __forceinline__ void relu_epilogue(uint32_t taddr_row, uint32_t h, uint32_t r, uint8_t* dst)
{
    float v[32];
    tmem_ld32(taddr_row + 32u * h, v);
#pragma unroll
    for (int k = 0; k < 32; ++k) v[k] = fmaxf(v[k], 0.f);
#pragma unroll
    for (int c = 0; c < 4; ++c) store_chunk(dst, r, 4 * h + c, v + 8 * c);
}
__device__ __forceinline__ void relu_epilogue16(uint32_t taddr_row, uint32_t h, uint32_t r, uint8_t* dst)
{
    float v[16];
    tmem_ld16(taddr_row + 16u * h, v);
#pragma unroll
    for (int k = 0; k < 16; ++k) v[k] = fmaxf(v[k], 0.f);
#pragma unroll
    for (int c = 0; c < 2; ++c) store_chunk(dst, r, 2 * h + c, v + 8 * c);
}

// Copy the weight images to shared memory.
__device__ __forceinline__ void load_weights(const uint4* __restrict__ img, uint8_t* w_s)
{
    uint4* d = reinterpret_cast<uint4*>(w_s);
    for (uint32_t i = threadIdx.x; i < kImgBytes / 16; i += blockDim.x) d[i] = img[i];
}

__device__ __forceinline__ void issue_forward(uint32_t d, uint32_t a_s, uint32_t w_s, uint32_t idesc)
{
#pragma unroll
    for (uint32_t k = 0; k < 4; ++k) mma_bf16(d, sw128_desc(a_s + 32u * k), sw128_desc(w_s + 32u * k), idesc, k > 0);
}

struct CacheArgs {
    Grid grid;
    const uint4* w_img;
    const Record* recs;
    const uint32_t* n_dev;      // record count on the device (or null: n)
    uint32_t offset;            // with n_dev: records before recs that are not this launch's
    uint32_t n;                 // records at most
    float* out_rgb;             // infer: n * 3 (or null)
    float4* frame;              // infer: += throughput * max(y, 0) at the record's pixel (or null)
    float* grad_w;              // train: [5][64][64]
    float* loss;                // train: sum of the per-record losses
    float inv_n;                // train: 1 / records in the batch
    unsigned int* err;
    uint32_t wait_polls;        // bound of each MMA wait (the drain after a failure keeps kWaitPolls)
};

__device__ __forceinline__ uint32_t count_of(const CacheArgs& a)
{
    if (!a.n_dev) return a.n;
    const uint32_t c = *a.n_dev;
    return c > a.offset ? min(c - a.offset, a.n) : 0u;
}

// Align the dynamic shared memory to the 1024-byte swizzle atom.
__device__ __forceinline__ uint8_t* aligned_smem(uint8_t* raw)
{
    const uint32_t s = smem_addr(raw);
    return raw + (((s + 1023u) & ~1023u) - s);
}

// Barrier of one group's 128 threads (ids 1..kGroups; 0 is __syncthreads).
__device__ __forceinline__ void group_sync(uint32_t id)
{
    asm volatile("bar.sync %0, 128;" ::"r"(id) : "memory");
}
// The same barrier, returning whether any of the group's threads passed p.
__device__ __forceinline__ bool group_sync_or(uint32_t id, bool p)
{
    uint32_t any;
    asm volatile(
        "{\n\t.reg .pred p, q;\n\t"
        "setp.ne.u32 p, %1, 0;\n\t"
        "bar.red.or.pred q, %2, 128, p;\n\t"
        "selp.u32 %0, 1, 0, q;\n\t}\n"
        : "=r"(any)
        : "r"((uint32_t)p), "r"(id)
        : "memory");
    return any != 0;
}

__global__ void __launch_bounds__(kInferThreads, 2) k_cache_infer(CacheArgs a)
{
    extern __shared__ uint8_t smem_raw[];
    uint8_t* base = aligned_smem(smem_raw);
    uint8_t* w_s = base;
    uint64_t* mbars = reinterpret_cast<uint64_t*>(base + kImgBytes + kGroups * kTileBytes);
    uint32_t* tslot = reinterpret_cast<uint32_t*>(mbars + kGroups);
    const uint32_t tid = threadIdx.x, warp = tid >> 5, lane = tid & 31u;
    // group g = warps 4g..4g+3; warp 4g+q reads TMEM lanes 32q.. (its subpartition)
    const uint32_t g = warp >> 2, q = warp & 3u, r = 32u * q + lane;
    uint8_t* act = base + kImgBytes + g * kTileBytes;
    const uint32_t mbar = smem_addr(mbars + g), bar = 1u + g;
    const bool leader = (tid & 127u) == 0;
    const uint32_t n = count_of(a);
    const uint32_t tiles = (n + kTile - 1) / kTile;
    if (blockIdx.x >= tiles) return;  // block-uniform, before any TMEM is held

    load_weights(a.w_img, w_s);
    if (tid < kGroups) mbar_init(smem_addr(mbars + tid), 1);
    __syncwarp();
    if (warp == 0) tmem_alloc(smem_addr(tslot), kInferTmemCols);
    fence_smem_async();
    fence_before_sync();
    __syncthreads();
    fence_after_sync();
    const uint32_t tmem_all = *tslot;
    const uint32_t tmem = tmem_all + 64u * g;   // this group's accumulator columns
    const uint32_t trow = tmem_addr(tmem, 32u * q, 0);
    const uint32_t w0 = smem_addr(w_s), x0 = smem_addr(act);
    uint32_t phase = 0;
    bool failed = false;

    // tiles go to the CTAs' first groups, then to their second: few tiles
    // spread over as many SMs (each SM's L1 serves the gathers of its own)
    // with at most one tile a CTA, all groups encode it, a third of the levels
    // each, before the first one runs the layers
    const bool solo = tiles <= gridDim.x;
    if (solo) {
        const uint32_t i = blockIdx.x * kTile + r;
        const bool valid = i < n;
        Record rec;
        if (valid) rec = load_record(a.recs + i);
        uint8_t* x = base + kImgBytes;   // the first group's tile
        encode_levels(a.grid, rec, valid, r, x, g, kGroups);
        for (uint32_t c = 4 + g; c < 8; c += kGroups) encode_chunk(rec, valid, r, x, c);
        fence_smem_async();
        __syncthreads();
    }
    for (uint32_t t = blockIdx.x + gridDim.x * g; t < tiles && !failed; t += gridDim.x * kGroups) {
        const uint32_t i = t * kTile + r;
        const bool valid = i < n;
        Record rec;
        if (valid) rec = load_record(a.recs + i);
        if (!solo) {
            encode_levels(a.grid, rec, valid, r, act, 0, 1);
#pragma unroll
            for (uint32_t c = 4; c < 8; ++c) encode_chunk(rec, valid, r, act, c);
        }
        fence_smem_async();
        fence_before_sync();
        group_sync(bar);
        for (int l = 0; l < kLayers; ++l) {
            if (leader) {
                fence_after_sync();
                issue_forward(tmem, x0, w0 + (uint32_t)l * kWBytes, l + 1 < kLayers ? ID_FWD : ID_OUT);
                mma_commit(mbar);
            }
            const bool ok = mbar_wait(mbar, phase, a.wait_polls);
            phase ^= 1u;
            if (group_sync_or(bar, !ok)) {
                failed = true;
                break;
            }
            fence_after_sync();
            if (l + 1 < kLayers) {
                relu_epilogue(trow, 0, r, act);
                relu_epilogue(trow, 1, r, act);
            } else {
                float y[16];
                tmem_ld16(trow, y);
                if (valid) {
                    if (a.out_rgb) {
                        a.out_rgb[3 * (size_t)i + 0] = y[0];
                        a.out_rgb[3 * (size_t)i + 1] = y[1];
                        a.out_rgb[3 * (size_t)i + 2] = y[2];
                    }
                    if (a.frame) {
                        float4* f = a.frame + rec.pixel;
                        float4 c = *f;
                        c.x += rec.v0 * fmaxf(y[0], 0.f);
                        c.y += rec.v1 * fmaxf(y[1], 0.f);
                        c.z += rec.v2 * fmaxf(y[2], 0.f);
                        *f = c;
                    }
                }
            }
            fence_smem_async();
            fence_before_sync();
            group_sync(bar);
        }
    }
    if (failed && leader) {
        atomicAdd(a.err, 1u);
        mbar_wait(mbar, phase ^ 1u, kWaitPolls);   // the commit that did not arrive, once more
    }
    fence_before_sync();
    __syncthreads();
    if (warp == 0) {
        fence_after_sync();
        tmem_dealloc(tmem_all, kInferTmemCols);
    }
}

__global__ void __launch_bounds__(kThreads, 1) k_cache_train(CacheArgs a)
{
    extern __shared__ uint8_t smem_raw[];
    uint8_t* base = aligned_smem(smem_raw);
    uint8_t* w_s = base;
    uint8_t* act[5];                             // X, H1..H4
    for (int l = 0; l < 5; ++l) act[l] = base + kImgBytes + (uint32_t)l * kTileBytes;
    uint8_t* dlt = base + kImgBytes + 5 * kTileBytes;
    uint64_t* mbar_p = reinterpret_cast<uint64_t*>(dlt + kTileBytes);
    uint32_t* tslot = reinterpret_cast<uint32_t*>(dlt + kTileBytes + 16);
    const uint32_t tid = threadIdx.x, warp = tid >> 5, lane = tid & 31u;
    const uint32_t q = warp & 3u, h = warp >> 2, r = 32u * q + lane;   // quarter h of row r's columns
    const uint32_t mbar = smem_addr(mbar_p);
    const uint32_t n = count_of(a);
    const uint32_t tiles = (n + kTile - 1) / kTile;
    if (blockIdx.x >= tiles) return;

    load_weights(a.w_img, w_s);
    if (tid == 0) mbar_init(mbar, 1);
    __syncwarp();
    if (warp == 0) tmem_alloc(smem_addr(tslot), kTrainTmemCols);
    fence_smem_async();
    fence_before_sync();
    __syncthreads();
    fence_after_sync();
    const uint32_t tmem = *tslot;
    const uint32_t trow = tmem_addr(tmem, 32u * q, 0);
    const uint32_t w0 = smem_addr(w_s), d0 = smem_addr(dlt);
    uint32_t a_s[5];
    for (int l = 0; l < 5; ++l) a_s[l] = smem_addr(act[l]);
    uint32_t phase = 0;
    bool failed = false, accumulating = false;
    float loss = 0.f;
    const float inv_n = a.n_dev ? 1.f / (float)n : a.inv_n;

    auto step = [&]() -> bool {         // commit, wait, agree
        if (tid == 0) mma_commit(mbar);
        const bool ok = mbar_wait(mbar, phase, a.wait_polls);
        phase ^= 1u;
        const bool bad = __syncthreads_or(!ok);
        fence_after_sync();
        return !bad;
    };
    auto sync_out = [&]() {             // smem writes and TMEM reads done before the next issue
        fence_smem_async();
        fence_before_sync();
        __syncthreads();
    };

    for (uint32_t t = blockIdx.x; t < tiles && !failed; t += gridDim.x) {
        const uint32_t i = t * kTile + r;
        const bool valid = i < n;
        Record rec;
        if (valid) rec = load_record(a.recs + i);
        encode_levels(a.grid, rec, valid, r, act[0], h, 4);
        encode_chunk(rec, valid, r, act[0], 4 + h);
        sync_out();
        // forward, keeping the activations
        for (int l = 0; l < 4 && !failed; ++l) {
            if (tid == 0) {
                fence_after_sync();
                issue_forward(tmem, a_s[l], w0 + (uint32_t)l * kWBytes, ID_FWD);
            }
            if (!step()) { failed = true; break; }
            relu_epilogue16(trow, h, r, act[l + 1]);
            sync_out();
        }
        if (failed) break;
        if (tid == 0) {
            fence_after_sync();
            issue_forward(tmem, a_s[4], w0 + 4u * kWBytes, ID_OUT);
        }
        if (!step()) { failed = true; break; }
        // relative L2 loss, sum_c (y - t)^2 / (y^2 + 0.01), its gradient
        // with the denominator held constant; delta of the output layer
        const float zero[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
        if (h == 0) {
            float y[16];
            tmem_ld16(trow, y);
            float dy[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
            if (valid) {
                const float tg[3] = {rec.v0, rec.v1, rec.v2};
#pragma unroll
                for (int c = 0; c < 3; ++c) {
                    const float den = y[c] * y[c] + 0.01f;
                    const float e = y[c] - tg[c];
                    loss += e * e / den;
                    dy[c] = 2.f * e / den * inv_n;
                }
            }
            store_chunk(dlt, r, 0, dy);
        } else {
            store_chunk(dlt, r, 2 * h, zero);
        }
        store_chunk(dlt, r, 2 * h + 1, zero);
        sync_out();
        // backward: layer l maps act[l] to the pre-activation whose gradient is in dlt
        for (int l = 4; l >= 0; --l) {
            if (tid == 0) {
                fence_after_sync();
                const uint32_t g = tmem + 64u + 64u * (uint32_t)l;
#pragma unroll
                for (uint32_t k = 0; k < 8; ++k)
                    mma_bf16(g, sw128_desc(a_s[l] + 2048u * k), sw128_desc(d0 + 2048u * k), ID_WGRAD,
                             (accumulating || k > 0) ? 1u : 0u);
#pragma unroll
                for (uint32_t k = 0; k < 4; ++k)
                    mma_bf16(tmem, sw128_desc(d0 + 32u * k), sw128_desc(w0 + (uint32_t)l * kWBytes + 2048u * k),
                             ID_DGRAD, k > 0);
            }
            if (!step()) { failed = true; break; }
            if (l > 0) {
                // delta of layer l: (delta W_l) * relu'(act[l])
                float v[16];
                tmem_ld16(trow + 16u * h, v);
#pragma unroll
                for (int c = 0; c < 2; ++c) {
                    const uint4 m = load_chunk(act[l], r, 2 * h + c);
                    const uint32_t mw[4] = {m.x, m.y, m.z, m.w};
#pragma unroll
                    for (int j = 0; j < 4; ++j) {
                        const float2 av = unpack_bf16(mw[j]);
                        if (!(av.x > 0.f)) v[8 * c + 2 * j] = 0.f;
                        if (!(av.y > 0.f)) v[8 * c + 2 * j + 1] = 0.f;
                    }
                    store_chunk(dlt, r, 2 * h + c, v + 8 * c);
                }
            } else {
                // input gradient of the hash features: columns 8h..8h+7 are levels 4h..4h+3
                float v[8];
                tmem_ld8(trow + 8u * h, v);
                if (valid) {
                    const float3 p = normalised_pos(a.grid, rec.px, rec.py, rec.pz);
#pragma unroll
                    for (int j = 0; j < 4; ++j) {
                        const int l = 4 * (int)h + j;
                        const Cell c = level_cell(a.grid, l, p);
                        const float gx = v[2 * j], gy = v[2 * j + 1];
#pragma unroll
                        for (int k = 0; k < 8; k += 2) {
                            // corners x and x + 1: where their entries are the two halves of
                            // 16 bytes (every other x), one atomic for both
                            const uint32_t i0 = corner_index(a.grid, l, c, k), i1 = corner_index(a.grid, l, c, k + 1);
                            const float w0 = corner_weight(c, k), w1 = corner_weight(c, k + 1);
                            const float2 v0 = make_float2(w0 * gx, w0 * gy), v1 = make_float2(w1 * gx, w1 * gy);
                            if ((i0 ^ i1) == 1u) {
                                const bool swap = i0 & 1u;
                                const float2 lo = swap ? v1 : v0, hi = swap ? v0 : v1;
                                atomicAdd(reinterpret_cast<float4*>(a.grid.grad + (i0 & ~1u)),
                                          make_float4(lo.x, lo.y, hi.x, hi.y));
                            } else {
                                atomicAdd(a.grid.grad + i0, v0);
                                atomicAdd(a.grid.grad + i1, v1);
                            }
                        }
                    }
                }
            }
            sync_out();
        }
        accumulating = true;
    }
    if (!failed && accumulating) {
        // weight gradients: accumulator l holds act[l]^T delta, rows m = input
        // unit (M = 64: TMEM lanes 0-15 of each subpartition), columns n
        for (int l = 0; l < kLayers; ++l) {
            float v[16];
            tmem_ld16(trow + 64u + 64u * (uint32_t)l + 16u * h, v);
            if (lane < 16) {
                const uint32_t m = 16u * q + lane;
                float* gw = a.grad_w + (size_t)l * kWidth * kWidth;
                for (int j = 0; j < 16; ++j) {
                    const uint32_t nn = 16u * h + (uint32_t)j;
                    if (l == kLayers - 1 && nn >= (uint32_t)kOutputs) break;
                    atomicAdd(gw + nn * kWidth + m, v[j]);
                }
            }
        }
    }
    for (int off = 16; off; off >>= 1) loss += __shfl_down_sync(0xffffffffu, loss, off);
    if (lane == 0 && loss != 0.f) atomicAdd(a.loss, loss);
    if (failed && tid == 0) {
        atomicAdd(a.err, 1u);
        mbar_wait(mbar, phase ^ 1u, kWaitPolls);   // the commit that did not arrive, once more
    }
    fence_before_sync();
    __syncthreads();
    if (warp == 0) {
        fence_after_sync();
        tmem_dealloc(tmem, kTrainTmemCols);
    }
}

// ---------------------------------------------------------------- parameters
__device__ __forceinline__ float hash01(uint32_t seed, uint32_t i)
{
    return (float)(ff_wang_hash(ff_wang_hash(seed) ^ (i * 0x9E3779B9u + 0x7F4A7C15u)) >> 8) * (1.f / 16777216.f);
}

__global__ void k_init_grid(float2* __restrict__ table, __half2* __restrict__ table_h, uint32_t n, uint32_t seed)
{
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const float2 v = make_float2((hash01(seed, 2 * i) * 2.f - 1.f) * 1e-4f, (hash01(seed, 2 * i + 1) * 2.f - 1.f) * 1e-4f);
    table[i] = v;
    table_h[i] = __floats2half2_rn(v.x, v.y);
}

// Xavier-uniform weights; rows 3..63 of the output layer are zero.
__global__ void k_init_mlp(float* __restrict__ w, uint32_t seed)
{
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= kParams) return;
    const uint32_t l = i / (kWidth * kWidth), row = (i / kWidth) % kWidth;
    const float fan_out = l == kLayers - 1 ? (float)kOutputs : (float)kWidth;
    const float lim = sqrtf(6.f / ((float)kWidth + fan_out));
    w[i] = (l == kLayers - 1 && row >= (uint32_t)kOutputs) ? 0.f : (hash01(seed ^ 0xA5A5A5A5u, i) * 2.f - 1.f) * lim;
}

__device__ __forceinline__ void put_image(uint8_t* img, uint32_t i, float w)
{
    const uint32_t l = i / (kWidth * kWidth), row = (i / kWidth) % kWidth, col = i % kWidth;
    *reinterpret_cast<__nv_bfloat16*>(img + l * kWBytes + sw128_offset(row, col)) = __float2bfloat16_rn(w);
}

__global__ void k_pack_mlp(const float* __restrict__ w, uint8_t* __restrict__ img)
{
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < kParams) put_image(img, i, w[i]);
}

struct AdamHP {
    float lr, b1, b2, eps, c1, c2;      // c1 = 1 - b1^t, c2 = 1 - b2^t
};

__global__ void k_adam_mlp(float* __restrict__ w, float* __restrict__ g, float* __restrict__ m, float* __restrict__ v,
                           uint8_t* __restrict__ img, AdamHP hp)
{
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= kParams) return;
    const float gi = g[i];
    g[i] = 0.f;
    const uint32_t l = i / (kWidth * kWidth), row = (i / kWidth) % kWidth;
    if (l == kLayers - 1 && row >= (uint32_t)kOutputs) return;
    const float mi = hp.b1 * m[i] + (1.f - hp.b1) * gi;
    const float vi = hp.b2 * v[i] + (1.f - hp.b2) * gi * gi;
    m[i] = mi;
    v[i] = vi;
    const float wi = w[i] - hp.lr * (mi / hp.c1) / (sqrtf(vi / hp.c2) + hp.eps);
    w[i] = wi;
    put_image(img, i, wi);
}

// Writes entry i (half precision) to the cells around it, where its level is
// also kept by cells (Grid::cells): each of up to 8 cells has it as another corner.
__device__ __forceinline__ void put_cells(const Grid& g, uint32_t* __restrict__ cells, uint32_t i, __half2 value)
{
    const uint32_t l = i >> g.log2_T;
    if (l >= g.cell_levels) return;
    const uint32_t side = g.dense_side[l], n = side - 1u;
    const uint32_t j = i & ((1u << g.log2_T) - 1u);
    const uint32_t x = j % side, y = (j / side) % side, z = j / (side * side);
    if (z > n) return;   // past the level's last entry
#pragma unroll
    for (uint32_t k = 0; k < 8; ++k) {
        const uint32_t cx = x - (k & 1u), cy = y - ((k >> 1) & 1u), cz = z - (k >> 2);   // (wraps below 0)
        if (cx < n && cy < n && cz < n)
            cells[8 * (size_t)(g.cell_off[l] + cx + n * (cy + n * cz)) + k] = *reinterpret_cast<uint32_t*>(&value);
    }
}

__global__ void k_cells(Grid g, uint32_t* __restrict__ cells, const __half2* __restrict__ table_h)
{
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < g.cell_levels << g.log2_T) put_cells(g, cells, i, table_h[i]);
}

// Sparse Adam over the grid: entries no record touched keep their state.
// One thread per four entries, a 32-byte sector of each array: the scan of
// the gradients is the bulk of the traffic, and what a touched entry costs is
// the sectors it is in, not its bytes.  16 levels of 2^19 entries after 16,384
// records: 66 us an entry per thread, 59 so (54% of the DRAM peak).
struct __align__(32) Sector {
    float2 e[4];
};
__global__ void k_adam_grid(Sector* __restrict__ table, uint4* __restrict__ table_h, Sector* __restrict__ g,
                            Sector* __restrict__ m, Sector* __restrict__ v, uint32_t n, AdamHP hp, Grid grid,
                            uint32_t* __restrict__ cells)
{
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const Sector gi = ld_sector(g + i);
    bool any = false;
#pragma unroll
    for (int k = 0; k < 4; ++k) any |= gi.e[k].x != 0.f || gi.e[k].y != 0.f;
    if (!any) return;
    Sector mi = ld_sector(m + i), vi = ld_sector(v + i), p = ld_sector(table + i);
    uint4 h = table_h[i];
    uint32_t* hw = &h.x;
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        const float2 d = gi.e[k];
        if (d.x == 0.f && d.y == 0.f) continue;
        float2 &mk = mi.e[k], &vk = vi.e[k], &pk = p.e[k];
        mk.x = hp.b1 * mk.x + (1.f - hp.b1) * d.x;
        mk.y = hp.b1 * mk.y + (1.f - hp.b1) * d.y;
        vk.x = hp.b2 * vk.x + (1.f - hp.b2) * d.x * d.x;
        vk.y = hp.b2 * vk.y + (1.f - hp.b2) * d.y * d.y;
        pk.x -= hp.lr * (mk.x / hp.c1) / (sqrtf(vk.x / hp.c2) + hp.eps);
        pk.y -= hp.lr * (mk.y / hp.c1) / (sqrtf(vk.y / hp.c2) + hp.eps);
        const __half2 half = __floats2half2_rn(pk.x, pk.y);
        hw[k] = *reinterpret_cast<const uint32_t*>(&half);
        put_cells(grid, cells, 4u * i + (uint32_t)k, half);
    }
    Sector zero;
#pragma unroll
    for (int k = 0; k < 4; ++k) zero.e[k] = make_float2(0.f, 0.f);
    st_sector(g + i, zero);
    st_sector(m + i, mi);
    st_sector(v + i, vi);
    st_sector(table + i, p);
    table_h[i] = h;
}

__global__ void k_half_of(const float2* __restrict__ table, __half2* __restrict__ table_h, uint32_t n)
{
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) table_h[i] = __floats2half2_rn(table[i].x, table[i].y);
}

unsigned grid_for(size_t n, unsigned block) { return (unsigned)((n + block - 1) / block); }

}  // namespace

// ---------------------------------------------------------------- host side
void ff_cache_setup_grid(ff_cache* c)
{
    Grid& g = c->grid;
    g.table_h = c->table_h.as<__half2>();
    g.grad = c->grid_grad.as<float2>();
    g.log2_T = c->prm.log2_table_size;
    const float3 lo = c->lo, hi = c->hi;
    const float3 ext = make_float3(fmaxf(hi.x - lo.x, 1e-6f), fmaxf(hi.y - lo.y, 1e-6f), fmaxf(hi.z - lo.z, 1e-6f));
    g.lo = lo;
    g.inv_ext = make_float3(1.f / ext.x, 1.f / ext.y, 1.f / ext.z);
    const double b = std::exp((std::log((double)c->prm.max_resolution) - std::log((double)c->prm.base_resolution)) /
                              (kLevels - 1));
    const uint64_t T = 1ull << g.log2_T;
    for (int l = 0; l < kLevels; ++l) {
        const uint32_t cells = (uint32_t)std::floor((double)c->prm.base_resolution * std::pow(b, l) + 1e-9);
        g.scale[l] = (float)cells;
        const uint64_t side = (uint64_t)cells + 1;
        g.dense_side[l] = side * side * side <= T ? (uint32_t)side : 0u;
    }
    // the leading dense levels also by cells (their resolutions never fall)
    uint64_t total = 0;
    g.cell_levels = 0;
    for (int l = 0; l < kLevels; ++l) {
        const uint64_t cells = (uint64_t)g.scale[l], n = cells * cells * cells;
        if (!g.dense_side[l] || n > kCellMax) break;
        g.cell_off[l] = (uint32_t)total;
        total += n;
        g.cell_levels = (uint32_t)l + 1u;
    }
    // (a copy: a device without the room for it gets the same answers from the table)
    try {
        c->cells.alloc(32 * total);
    } catch (const FFError& e) {
        if (e.status != FF_ERR_OOM) throw;
        g.cell_levels = 0;
    }
    g.cells = c->cells.as<uint4>();
}

// The cells' copy of the half-precision table, from scratch.
static void fill_cells(ff_cache* c, cudaStream_t st)
{
    const Grid& g = c->grid;
    if (!g.cell_levels) return;
    k_cells<<<grid_for((size_t)g.cell_levels << g.log2_T, 256), 256, 0, st>>>(g, c->cells.as<uint32_t>(),
                                                                              c->table_h.as<__half2>());
}

void ff_cache_init_params(ff_cache* c)
{
    cudaStream_t st = c->ctx->stream;
    const uint32_t n = kLevels << c->prm.log2_table_size;
    k_init_grid<<<grid_for(n, 256), 256, 0, st>>>(c->table.as<float2>(), c->table_h.as<__half2>(), n, c->prm.seed);
    fill_cells(c, st);
    k_init_mlp<<<grid_for(kParams, 256), 256, 0, st>>>(c->mlp.as<float>(), c->prm.seed);
    k_pack_mlp<<<grid_for(kParams, 256), 256, 0, st>>>(c->mlp.as<float>(), c->mlp_img.as<uint8_t>());
    FF_CUDA_CHECK(cudaMemsetAsync(c->grid_grad.ptr, 0, sizeof(float2) * n, st));
    FF_CUDA_CHECK(cudaMemsetAsync(c->grid_m.ptr, 0, sizeof(float2) * n, st));
    FF_CUDA_CHECK(cudaMemsetAsync(c->grid_v.ptr, 0, sizeof(float2) * n, st));
    FF_CUDA_CHECK(cudaMemsetAsync(c->mlp_grad.ptr, 0, sizeof(float) * kParams, st));
    FF_CUDA_CHECK(cudaMemsetAsync(c->mlp_m.ptr, 0, sizeof(float) * kParams, st));
    FF_CUDA_CHECK(cudaMemsetAsync(c->mlp_v.ptr, 0, sizeof(float) * kParams, st));
    FF_CUDA_CHECK(cudaGetLastError());
    c->step = 0;
}

// The dynamic shared memory above 48 KB is an attribute of the kernel on each
// device: set once per (kernel, device).
static void allow_smem(ff_cache* c, const void* fn, uint32_t bytes, int which)
{
    static std::atomic<uint64_t> done[2];
    const uint64_t bit = 1ull << (c->ctx->device & 63);
    if (done[which].load() & bit) return;
    FF_CUDA_CHECK(cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes));
    done[which].fetch_or(bit);
}

static CacheArgs make_args(ff_cache* c, const Record* recs, uint32_t n, const uint32_t* n_dev)
{
    CacheArgs a{};
    a.grid = c->grid;
    a.w_img = c->mlp_img.as<uint4>();
    a.recs = recs;
    a.n_dev = n_dev;
    a.n = n;
    a.grad_w = c->mlp_grad.as<float>();
    a.loss = c->loss.as<float>();
    a.err = c->err.as<unsigned int>();
    a.wait_polls = c->wait_polls == FF_DEBUG_WAIT_DEFAULT ? kWaitPolls : c->wait_polls;
    return a;
}

void ff_cache_launch_infer(ff_cache* c, const void* recs, uint32_t n_max, const uint32_t* n_dev, float* out_rgb,
                           float4* frame)
{
    allow_smem(c, reinterpret_cast<const void*>(k_cache_infer), kInferSmem, 0);
    if (n_max == 0) return;
    CacheArgs a = make_args(c, static_cast<const Record*>(recs), n_max, n_dev);
    a.out_rgb = out_rgb;
    a.frame = frame;
    const uint32_t tiles = (n_max + kTile - 1) / kTile;
    const uint32_t grid = std::min<uint32_t>(tiles, (uint32_t)c->ctx->num_sms * 2u);
    k_cache_infer<<<grid, kInferThreads, kInferSmem, c->ctx->stream>>>(a);
    FF_CUDA_CHECK(cudaGetLastError());
}

// Gradients of the batch (added to the accumulators) and, unless
// gradients_only, one Adam step of the MLP and the grid.  With n_dev the
// batch is records [offset, offset + n_max) of a list whose length is on the
// device, and the loss is normalised by the records actually present.
static void launch_train(ff_cache* c, const Record* recs, uint32_t offset, uint32_t n_max, const uint32_t* n_dev,
                         uint32_t n_norm, bool gradients_only, cudaStream_t st)
{
    allow_smem(c, reinterpret_cast<const void*>(k_cache_train), kTrainSmem, 1);
    if (n_max == 0) return;
    CacheArgs a = make_args(c, recs + offset, n_max, n_dev);
    a.offset = offset;
    a.inv_n = 1.f / (float)std::max<uint32_t>(n_norm, 1u);
    const uint32_t tiles = (n_max + kTile - 1) / kTile;
    const uint32_t grid = std::min<uint32_t>(tiles, (uint32_t)c->ctx->num_sms);
    k_cache_train<<<grid, kThreads, kTrainSmem, st>>>(a);
    FF_CUDA_CHECK(cudaGetLastError());
    if (gradients_only) return;
    c->step += 1;
    AdamHP hp;
    hp.lr = c->prm.lr;
    hp.b1 = c->prm.beta1;
    hp.b2 = c->prm.beta2;
    hp.eps = c->prm.eps;
    hp.c1 = 1.f - (float)std::pow((double)hp.b1, (double)c->step);
    hp.c2 = 1.f - (float)std::pow((double)hp.b2, (double)c->step);
    k_adam_mlp<<<grid_for(kParams, 256), 256, 0, st>>>(c->mlp.as<float>(), c->mlp_grad.as<float>(), c->mlp_m.as<float>(),
                                                      c->mlp_v.as<float>(), c->mlp_img.as<uint8_t>(), hp);
    const uint32_t ng = kLevels << c->prm.log2_table_size;
    k_adam_grid<<<grid_for(ng / 4, 256), 256, 0, st>>>(c->table.as<Sector>(), c->table_h.as<uint4>(),
                                                      c->grid_grad.as<Sector>(), c->grid_m.as<Sector>(),
                                                      c->grid_v.as<Sector>(), ng / 4, hp, c->grid, c->cells.as<uint32_t>());
    FF_CUDA_CHECK(cudaGetLastError());
}

void ff_cache_launch_train(ff_cache* c, const void* recs, uint32_t n, bool gradients_only)
{
    launch_train(c, static_cast<const Record*>(recs), 0, n, nullptr, n, gradients_only, c->ctx->stream);
}

void ff_cache_launch_train_slice(ff_cache* c, const void* recs, uint32_t offset, uint32_t n_max, const uint32_t* n_dev,
                                 cudaStream_t st)
{
    launch_train(c, static_cast<const Record*>(recs), offset, n_max, n_dev, n_max, false, st);
}

void ff_cache_refresh_copies(ff_cache* c)
{
    cudaStream_t st = c->ctx->stream;
    const uint32_t n = kLevels << c->prm.log2_table_size;
    k_half_of<<<grid_for(n, 256), 256, 0, st>>>(c->table.as<float2>(), c->table_h.as<__half2>(), n);
    fill_cells(c, st);
    k_pack_mlp<<<grid_for(kParams, 256), 256, 0, st>>>(c->mlp.as<float>(), c->mlp_img.as<uint8_t>());
    FF_CUDA_CHECK(cudaGetLastError());
}

uint32_t ff_cache_num_params() { return kParams; }
