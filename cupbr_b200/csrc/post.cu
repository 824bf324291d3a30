// Bloom and tone mapping (PostProcessor::bloom, ToneMapper::toneMap).
//
// The reference builds a 6-level pyramid with 12 launches and 2 device
// copies (PostProcessor.cpp:125-142, PyramidConstructor.cu:9-169), but its
// upscale step reads pyramid_down[d + 1] (PyramidConstructor.cu:84), so the
// output only depends on levels 0 and 1:
//     out = hdr + T(hdr) + tent3x3(box2x2(T(hdr))) / 16
// with T the soft-knee threshold.  Here that is one pass (k_bloom): a block
// builds the level-1 pixels of its tile and their border in shared memory
// from the HDR image and forms the tile's output from them, optionally
// tone-mapped.  The float operations and their order are the reference's, so
// results match it exactly.  Bloom in place (the entry point that allocates
// nothing takes output buffers over its input) keeps two passes,
// k_bloom_down and k_bloom_up, with level 1 in global memory.
#include "post.hpp"

#include <mutex>

#include "dev_common.cuh"

namespace cupbr_b200 {

namespace {


// thresholding_kernel, PyramidConstructor.cu:9-30
__device__ __forceinline__ float threshold_scale(f3 c, float4 th) {
    float br = c.x > c.y ? c.x : c.y;
    br = c.z > br ? c.z : br;
    float rq = clampf(br - th.y, 0.0f, th.z);
    rq = th.w * rq * rq;
    return fmaxf(rq, br - th.x) / fmaxf(br, 1e-5f);
}
__device__ __forceinline__ f3 threshold(f3 c, float4 th) {
    const float s = threshold_scale(c, th);
    return mk(c.x * s, c.y * s, c.z * s);
}

__device__ __forceinline__ f3 ld3(const float* p) { return mk(p[0], p[1], p[2]); }

// ToneMapper.cu:17-41 (REINHARD) and :43-69 (GAMMA), channel k of one pixel
__device__ __forceinline__ uint32_t tone_direct(float x, int type, float exposure, int k) {
    float m;
    if (type == 0) {
        const float e = (k == 2) ? (float)(1.0f / 2.2) : 1.0f / 2.2f;
        m = powf((float)(1.0 - (double)expf(-x * exposure)), e);
    } else {
        m = x <= 0.0031308f ? 12.92f * x : 1.055f * powf(x, 1.0f / 2.4f) - 0.055f;
    }
    return (uint32_t)(clampf(m, 0.0f, 1.0f) * 255.0f);
}

// ---- tone-map levels from tables
//
// A channel's 8-bit level is a step function of u = x * exposure (REINHARD:
// tone_direct evaluates expf(-x * exposure), and (-x) * e == -(x * e)) or of
// u = x (GAMMA).  For u in [2^-20, 2^5) a table holds one 32-bit word per
// bucket of 2^16 consecutive float bit patterns (128 buckets per octave):
// (level at the bucket's first float) << 17, plus 2^17 minus the offset of
// the one level step inside the bucket (2^16 when there is none), so adding
// the low 16 bits of u carries into the level from the step on.
// k_tone_levels_build makes the tables by evaluating tone_direct at every
// float of that range on the device, so a looked-up level is tone_direct's
// level.  Any other u has the level of the end of the range it is clamped to:
// below 2^-20 every formula gives level 0 (REINHARD: (2^-20)^(1/2.2) * 255 <
// 0.5; GAMMA: 12.92 * 2^-20 * 255 < 0.01), as it does for NaN and for negative
// inputs above -TONE_NEGATIVE (below it REINHARD's expf can overflow and its
// level jump to 255: those take the formulas); from 2^5 up (+inf included) level 255 (REINHARD: 1 - e^-32 rounds to 1;
// GAMMA: the power term exceeds 4).  cupbr_tonemap_verify_levels compares
// both for every 32-bit input.  A build that meets a bucket it cannot
// describe (a decrease or more than one step inside) leaves the tables
// unpublished and the kernels with the formulas.  Tables: 0 REINHARD red /
// green, 1 REINHARD blue (its exponent rounds differently), 2 GAMMA; 12.8 KB
// each, small enough to keep in shared memory, where lanes with unrelated
// values cost a few bank conflicts instead of one L1 line each.
constexpr uint32_t TONE_LO_BITS = 0x35800000u;  // 2^-20
constexpr uint32_t TONE_HI_BITS = 0x42000000u;  // 2^5
constexpr uint32_t TONE_SHIFT = 16;
constexpr uint32_t TONE_BUCKETS = (TONE_HI_BITS - TONE_LO_BITS) >> TONE_SHIFT;  // 3200
constexpr uint32_t TONE_NO_STEP = 1u << TONE_SHIFT;
constexpr uint32_t TONE_FLAG = 0xffffffffu;  // this bucket needs the formulas
constexpr float TONE_NEGATIVE = 88.0f;  // expf(88) is finite
constexpr int TONE_TABLES = 3;
static __device__ __align__(16) uint32_t g_tone_levels[TONE_TABLES][TONE_BUCKETS];
// 1 once g_tone_levels is complete; until then (and after a device reset
// reloads the module) the kernels use the formulas.
static __device__ uint32_t g_tone_ready;

__device__ __forceinline__ bool tone_tables_ready() {
    uint32_t v;
    asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(&g_tone_ready) : "memory");
    return v != 0;
}

// The two tables a tone-map type reads: REINHARD red / green and blue, or
// GAMMA for every channel.
struct ToneTables {
    const uint32_t* rg;
    const uint32_t* b;
};
__device__ __forceinline__ ToneTables tone_tables_global(int type) {
    return type == 0 ? ToneTables{g_tone_levels[0], g_tone_levels[1]} : ToneTables{g_tone_levels[2], g_tone_levels[2]};
}
// Bytes of shared memory stage_tone_tables fills for a type.
__host__ __device__ constexpr uint32_t tone_smem_bytes(int type) {
    return (type == 0 ? 2u : 1u) * TONE_BUCKETS * (uint32_t)sizeof(uint32_t);
}
// Copies the type's tables into s (tone_smem_bytes(type) bytes) when the
// tables are complete; block-uniform, with __syncthreads inside.  Returns
// false (tables not yet built) to every thread of the block otherwise.
__device__ __forceinline__ bool stage_tone_tables(uint32_t* s, int type, ToneTables& tt) {
    __shared__ uint32_t s_ready;
    if (threadIdx.x == 0) s_ready = tone_tables_ready() ? 1u : 0u;
    __syncthreads();
    if (!s_ready) return false;
    const uint4* src = reinterpret_cast<const uint4*>(type == 0 ? g_tone_levels[0] : g_tone_levels[2]);
    uint4* dst = reinterpret_cast<uint4*>(s);
    const uint32_t n16 = tone_smem_bytes(type) / 16;  // the two REINHARD tables are adjacent
    for (uint32_t i = threadIdx.x; i < n16; i += blockDim.x) dst[i] = src[i];
    __syncthreads();
    tt = type == 0 ? ToneTables{s, s + TONE_BUCKETS} : ToneTables{s, s};
    return true;
}

__device__ __forceinline__ uint32_t tone_lookup(float u, const uint32_t* tbl) {
    // fmaxf takes the bound for NaN
    const float c = fminf(fmaxf(u, __uint_as_float(TONE_LO_BITS)), __uint_as_float(TONE_HI_BITS - 1));
    const uint32_t b = __float_as_uint(c) - TONE_LO_BITS;
    return (tbl[b >> TONE_SHIFT] + (b & (TONE_NO_STEP - 1))) >> (TONE_SHIFT + 1);
}

// The formulas, out of line: they run before the tables are built, and their
// code would crowd the instruction cache at every call site.
__device__ __noinline__ uint32_t tonemap_px_direct(f3 c, int type, float exposure) {
    return tone_direct(c.x, type, exposure, 0) | tone_direct(c.y, type, exposure, 1) << 8 |
           tone_direct(c.z, type, exposure, 2) << 16 | 0xff000000u;
}
// One pixel's RGBA8 as a little-endian word.
__device__ __forceinline__ uint32_t tonemap_px(f3 c, int type, float exposure, bool tables, const ToneTables& tt) {
    const float e = type == 0 ? exposure : 1.0f;  // x * 1 == x
    const f3 u = c * e;
    if (!tables || fminf(fminf(u.x, u.y), u.z) < -TONE_NEGATIVE) return tonemap_px_direct(c, type, exposure);
    return tone_lookup(u.x, tt.rg) | tone_lookup(u.y, tt.rg) << 8 | tone_lookup(u.z, tt.b) << 16 | 0xff000000u;
}

// One block per (bucket, table): 256 threads evaluate tone_direct at 256
// consecutive floats each and report the bucket's steps.
__global__ void __launch_bounds__(256) k_tone_levels_build() {
    const uint32_t q = blockIdx.x, t = blockIdx.y;
    const uint32_t first = TONE_LO_BITS + (q << TONE_SHIFT);
    constexpr uint32_t per = (1u << TONE_SHIFT) / 256;
    const uint32_t b0 = first + threadIdx.x * per;
    const int type = t == 2 ? 1 : 0, k = t == 1 ? 2 : 0;
    constexpr uint32_t nowhere = 0xffffffffu;
    uint32_t prev = tone_direct(__uint_as_float(threadIdx.x == 0 ? b0 : b0 - 1), type, 1.0f, k);
    uint32_t steps = 0, bad = 0, pos = nowhere;
    for (uint32_t i = 0; i < per; ++i) {
        const uint32_t cur = tone_direct(__uint_as_float(b0 + i), type, 1.0f, k);
        if (cur < prev) bad = 1;
        if (cur > prev) {
            steps += cur - prev;
            if (pos == nowhere) pos = b0 + i;
        }
        prev = cur;
    }
    __shared__ uint32_t s_steps, s_bad, s_pos;
    if (threadIdx.x == 0) {
        s_steps = 0;
        s_bad = 0;
        s_pos = nowhere;
    }
    __syncthreads();
    if (steps) {
        atomicAdd(&s_steps, steps);
        atomicMin(&s_pos, pos);
    }
    if (bad) atomicOr(&s_bad, 1u);
    __syncthreads();
    if (threadIdx.x == 0) {
        const uint32_t base = tone_direct(__uint_as_float(first), type, 1.0f, k);
        const bool ok = s_bad == 0 && s_steps <= 1;
        const uint32_t off = s_steps ? s_pos - first : TONE_NO_STEP;  // 1 .. 2^16
        g_tone_levels[t][q] = ok ? (base << (TONE_SHIFT + 1)) + (2 * TONE_NO_STEP - off) : TONE_FLAG;
    }
}

// One block, after the build: publishes the tables if every bucket has a word.
__global__ void k_tone_levels_publish() {
    int flagged = 0;
    const uint32_t* w = &g_tone_levels[0][0];
    for (uint32_t i = threadIdx.x; i < TONE_TABLES * TONE_BUCKETS; i += blockDim.x) flagged |= w[i] == TONE_FLAG;
    if (__syncthreads_or(flagged) || threadIdx.x != 0) return;
    asm volatile("st.release.gpu.global.u32 [%0], %1;" ::"l"(&g_tone_ready), "r"(1u) : "memory");
}

// Every 32-bit input of every table: the looked-up level against the
// formula's (inputs spread over the grid's threads, counts per table).
__global__ void k_tone_levels_verify(unsigned long long* __restrict__ mismatches) {
    const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
    unsigned long long miss[TONE_TABLES] = {0, 0, 0};
    for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < (1ull << 32); i += stride) {
        const float x = __uint_as_float((uint32_t)i);
#pragma unroll
        for (int t = 0; t < TONE_TABLES; ++t) {
            const int type = t == 2 ? 1 : 0, k = t == 1 ? 2 : 0;
            if (x < -TONE_NEGATIVE) continue;  // the kernels take the formulas
            miss[t] += tone_lookup(x, g_tone_levels[t]) != tone_direct(x, type, 1.0f, k);
        }
    }
#pragma unroll
    for (int t = 0; t < TONE_TABLES; ++t)
        if (miss[t]) atomicAdd(&mismatches[t], miss[t]);
}

__global__ void k_tonemap(const float* __restrict__ hdr, uint32_t n, int type, float exposure, uint32_t* __restrict__ out) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    out[i] = tonemap_px(ld3(hdr + 3 * (size_t)i), type, exposure, tone_tables_ready(), tone_tables_global(type));
}

// downsample_kernel (PyramidConstructor.cu:32-65) of the thresholded level 0
__global__ void k_bloom_down(const float* __restrict__ hdr, uint32_t w, uint32_t h, float4 th, float* __restrict__ d1,
                             uint32_t w2, uint32_t h2) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= w2 * h2) return;
    const uint32_t y = i / w2, x = i - w2 * y;
    f3 r = splat(0.0f);
    const uint32_t ox[4] = {0, 0, 1, 1}, oy[4] = {0, 1, 0, 1};
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        uint32_t sx = 2 * x + ox[k], sy = 2 * y + oy[k];
        if (sx >= w) sx = w - 1;
        if (sy >= h) sy = h - 1;
        r += threshold(ld3(hdr + 3 * ((size_t)sx + (size_t)sy * w)), th);
    }
    float* o = d1 + 3 * (size_t)i;
    o[0] = r.x / 4.0f; o[1] = r.y / 4.0f; o[2] = r.z / 4.0f;
}

// upscale_and_combine_kernel at level 0 (PyramidConstructor.cu:67-112)
// followed by combine_kernel (:114-125).
__global__ void k_bloom_up(const float* hdr, uint32_t w, uint32_t h, float4 th, const float* __restrict__ d1,
                           uint32_t w2, uint32_t h2, float* out) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= w * h) return;
    const int32_t y = (int32_t)(i / w), x = (int32_t)(i - w * (uint32_t)y);
    const int32_t dx = x / 2, dy = y / 2;
    const float kern[3][3] = {{1.0f, 2.0f, 1.0f}, {2.0f, 4.0f, 2.0f}, {1.0f, 2.0f, 1.0f}};
    f3 r = splat(0.0f);
#pragma unroll
    for (int32_t u = -1; u < 2; ++u)
#pragma unroll
        for (int32_t v = -1; v < 2; ++v) {
            int32_t sx = dx + u, sy = dy + v;
            if (sx < 0) sx = 0;
            if (sx >= (int32_t)w2) sx = (int32_t)w2 - 1;
            if (sy < 0) sy = 0;
            if (sy >= (int32_t)h2) sy = (int32_t)h2 - 1;
            r += ld3(d1 + 3 * ((size_t)sx + (size_t)sy * w2)) * kern[u + 1][v + 1];
        }
    const f3 c = ld3(hdr + 3 * (size_t)i);
    const f3 up = r / 16.0f + threshold(c, th);
    const f3 res = c + up;
    float* o = out + 3 * (size_t)i;
    o[0] = res.x; o[1] = res.y; o[2] = res.z;
}

__device__ __forceinline__ void ld12(const float* __restrict__ p, f3 v[4]) {
    const float4* q = reinterpret_cast<const float4*>(p);
    const float4 a = __ldg(q), b = __ldg(q + 1), c = __ldg(q + 2);
    v[0] = mk(a.x, a.y, a.z);
    v[1] = mk(a.w, b.x, b.y);
    v[2] = mk(b.z, b.w, c.x);
    v[3] = mk(c.y, c.z, c.w);
}
// One quad of pixels per thread.
__device__ __forceinline__ void tonemap_quad(const float* __restrict__ hdr, uint32_t i4, uint32_t n, int type,
                                             float exposure, bool tables, const ToneTables& tt,
                                             uint32_t* __restrict__ out) {
    if (4 * i4 + 3 < n) {  // pixels 4 i4 .. 4 i4 + 3
        f3 v[4];
        ld12(hdr + 12 * (size_t)i4, v);
        uint32_t o[4];
#pragma unroll
        for (int k = 0; k < 4; ++k) o[k] = tonemap_px(v[k], type, exposure, tables, tt);
        reinterpret_cast<uint4*>(out)[i4] = make_uint4(o[0], o[1], o[2], o[3]);
    } else {
        for (uint32_t i = 4 * i4; i < n; ++i) out[i] = tonemap_px(ld3(hdr + 3 * (size_t)i), type, exposure, tables, tt);
    }
}
// The level tables read through L1, where lanes with unrelated values touch a
// line each: for images too small to pay for copying the tables.
__global__ void k_tonemap4(const float* __restrict__ hdr, uint32_t n, int type, float exposure,
                           uint32_t* __restrict__ out) {
    tonemap_quad(hdr, blockIdx.x * blockDim.x + threadIdx.x, n, type, exposure, tone_tables_ready(),
                 tone_tables_global(type), out);
}
// The level tables in shared memory, one copy (12.8 or 25.6 KB) per SM: one
// block of 1024 threads per SM strides over the image, which leaves the L1 of
// the SMs it shares with a renderer's traversal kernels (pipelined render())
// nearly as it is.
constexpr uint32_t TONEMAP_THREADS = 1024;
// From here on copying the tables pays: 1024 x 512 8.3 -> 6.2 us, 1920 x 1080
// 19 -> 9.5, 7680 x 4320 (noise) 236 -> 92, where 16 B per pixel take 81 us; 640 x
// 360 has no time to save over the launch.
constexpr uint32_t TONEMAP_SMEM_PIXELS = 1u << 19;
__global__ void __launch_bounds__(TONEMAP_THREADS) k_tonemap4_smem(const float* __restrict__ hdr, uint32_t n, int type,
                                                                   float exposure, uint32_t* __restrict__ out) {
    extern __shared__ __align__(16) uint32_t s_tone[];
    ToneTables tt{};
    const bool tables = stage_tone_tables(s_tone, type, tt);
    for (uint32_t i4 = blockIdx.x * TONEMAP_THREADS + threadIdx.x; i4 < (n + 3) / 4; i4 += gridDim.x * TONEMAP_THREADS)
        tonemap_quad(hdr, i4, n, type, exposure, tables, tt, out);
}

// N floats (a multiple of VEC) from p, VEC at a time (p aligned to them).
template <int VEC, int N>
__device__ __forceinline__ void ld_floats(const float* __restrict__ p, float* v) {
#pragma unroll
    for (int k = 0; k < N; k += VEC) {
        if (VEC == 4) {
            const float4 q = __ldg(reinterpret_cast<const float4*>(p + k));
            v[k] = q.x; v[k + 1] = q.y; v[k + 2] = q.z; v[k + 3] = q.w;
        } else if (VEC == 2) {
            const float2 q = __ldg(reinterpret_cast<const float2*>(p + k));
            v[k] = q.x; v[k + 1] = q.y;
        } else {
            v[k] = __ldg(p + k);
        }
    }
}
template <int VEC, int N>
__device__ __forceinline__ void st_words(uint32_t* p, const uint32_t* v) {
#pragma unroll
    for (int k = 0; k < N; k += VEC) {
        if (VEC == 4) *reinterpret_cast<uint4*>(p + k) = make_uint4(v[k], v[k + 1], v[k + 2], v[k + 3]);
        else if (VEC == 2) *reinterpret_cast<uint2*>(p + k) = make_uint2(v[k], v[k + 1]);
        else p[k] = v[k];
    }
}

// downsample_kernel (PyramidConstructor.cu:32-65) of the thresholded level 0
// at level-1 pixel (x, y), x < w / 2, y < h / 2 (no tap needs an edge clamp):
// the taps in the order (2x, 2y), (2x, 2y + 1), (2x + 1, 2y), (2x + 1, 2y + 1).
__device__ __forceinline__ f3 level1_at(const float* __restrict__ hdr, uint32_t w, float4 th, uint32_t x, uint32_t y) {
    const float* a = hdr + 3 * ((size_t)(2 * y) * w + 2 * x);
    const float* b = a + 3 * (size_t)w;
    f3 t = splat(0.0f);
    t += threshold(ld3(a), th);
    t += threshold(ld3(b), th);
    t += threshold(ld3(a + 3), th);
    t += threshold(ld3(b + 3), th);
    return mk(t.x / 4.0f, t.y / 4.0f, t.z / 4.0f);
}

// level1_at out of line, for the tiles at the image's right and bottom edges.
__device__ __noinline__ f3 level1_edge(const float* __restrict__ hdr, uint32_t w, float4 th, uint32_t x, uint32_t y) {
    return level1_at(hdr, w, th, x, y);
}

// Bloom of an image in one pass, tile by tile: 64 x 32 pixels per block of
// 256 threads, 4 x 2 pixels (two level-1 pixels) per thread.  The thread
// keeps its pixels and their threshold factors in registers from the level-1
// stage to the output, so the image is read once; the 100 level-1 pixels
// around the tile are computed from the neighbours' pixels (L1 / L2).  VEC:
// floats per load and words per store, by the alignment of the image's rows
// (their width and the buffers' addresses).  TONEMAP: out8 receives
// ToneMapper::toneMap of the result and nothing goes to out; a grid of one
// wave strides over the tiles and keeps the level tables in shared memory
// (smem_tables) once a block has tiles enough to pay for copying them.
//
// 16 B of DRAM traffic per pixel (28 with HDR output), 118 instructions; bound
// by issue (57 % busy) and the loads at the head of each tile.  B200, two passes
// with level 1 in global memory -> this: 7680 x 4320 with Reinhard 294 -> 191 us,
// to HDR 241 -> 187; rows off 16 bytes (scalar kernels before) 7679 x 4319 1035
// -> 214 and 364 -> 238; 1366 x 768 42 -> 12 and 18.5 -> 12.3; 1920 x 1080 25 ->
// 17.5 and 18.6 -> 14.7.  Asking L2 for the next tile while one is worked on:
// 191 -> 201.  5 blocks per SM instead of 4 (48 registers): HDR 8K 187 -> 179,
// 1080p 14.7 -> 16.4.
constexpr uint32_t BLOOM_TW = 64, BLOOM_TH = 32, BLOOM_THREADS = 256;
constexpr uint32_t BLOOM_LW = BLOOM_TW / 2 + 2, BLOOM_LH = BLOOM_TH / 2 + 2;  // level-1 tile with its border
template <bool TONEMAP, int VEC>
__global__ void __launch_bounds__(BLOOM_THREADS, 4) k_bloom(const float* __restrict__ hdr, uint32_t w, uint32_t h,
                                                            float4 th, float* __restrict__ out,
                                                            uint32_t* __restrict__ out8, int type, float exposure,
                                                            uint32_t tiles_x, uint32_t tiles, bool smem_tables) {
    extern __shared__ __align__(16) uint32_t s_dyn[];  // level tables, or the tile's output
    __shared__ __align__(8) float s_l1[3][BLOOM_LH][BLOOM_LW + 2];
    ToneTables tt{};
    bool tables = false;
    if (TONEMAP) {
        if (smem_tables) {
            tables = stage_tone_tables(s_dyn, type, tt);
        } else {
            tables = tone_tables_ready();
            tt = tone_tables_global(type);
        }
    }
    const uint32_t tx = threadIdx.x & 15u, ty = threadIdx.x >> 4;
    const uint32_t w2 = w / 2, h2 = h / 2;
    for (uint32_t tile = blockIdx.x; tile < tiles; tile += gridDim.x) {
        const uint32_t by = tile / tiles_x, bx = tile - by * tiles_x;
        const uint32_t x = bx * BLOOM_TW + 4 * tx, y = by * BLOOM_TH + 2 * ty;
        f3 c[2][4];
        float sc[2][4];
#pragma unroll
        for (int r = 0; r < 2; ++r) {
            float v[12];
            const float* p = hdr + 3 * ((size_t)(y + r) * w + x);
            if (y + r < h && x + 3 < w) {
                ld_floats<VEC, 12>(p, v);
            } else {
#pragma unroll
                for (uint32_t k = 0; k < 12; ++k) v[k] = y + r < h && x + k / 3 < w ? __ldg(p + k) : 0.0f;
            }
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                c[r][k] = mk(v[3 * k], v[3 * k + 1], v[3 * k + 2]);
                sc[r][k] = threshold_scale(c[r][k], th);
            }
        }
        const uint32_t lx = x / 2, ly = y / 2;
#pragma unroll
        for (uint32_t k = 0; k < 2; ++k) {
            f3 t = splat(0.0f);
            if (lx + k < w2 && ly < h2) {
                t += c[0][2 * k] * sc[0][2 * k];
                t += c[1][2 * k] * sc[1][2 * k];
                t += c[0][2 * k + 1] * sc[0][2 * k + 1];
                t += c[1][2 * k + 1] * sc[1][2 * k + 1];
                t = mk(t.x / 4.0f, t.y / 4.0f, t.z / 4.0f);
            } else if (lx + k <= w2 + 1 && ly <= h2 + 1) {
                // the level-1 edge, which the tent filter clamps to
                t = level1_edge(hdr, w, th, min(lx + k, w2 - 1), min(ly, h2 - 1));
            }
            s_l1[0][ty + 1][2 * tx + 1 + k] = t.x;
            s_l1[1][ty + 1][2 * tx + 1 + k] = t.y;
            s_l1[2][ty + 1][2 * tx + 1 + k] = t.z;
        }
        // the border: its top and bottom rows, then its left and right columns
        if (threadIdx.x < 2 * BLOOM_LW + 2 * (BLOOM_LH - 2)) {
            uint32_t i = threadIdx.x, hx, hy;
            if (i < 2 * BLOOM_LW) {
                hy = i < BLOOM_LW ? 0 : BLOOM_LH - 1;
                hx = i < BLOOM_LW ? i : i - BLOOM_LW;
            } else {
                i -= 2 * BLOOM_LW;
                hx = i < BLOOM_LH - 2 ? 0 : BLOOM_LW - 1;
                hy = 1 + (i < BLOOM_LH - 2 ? i : i - (BLOOM_LH - 2));
            }
            const int32_t gx = (int32_t)(bx * (BLOOM_TW / 2) + hx) - 1, gy = (int32_t)(by * (BLOOM_TH / 2) + hy) - 1;
            const f3 t = level1_at(hdr, w, th, (uint32_t)min(max(gx, 0), (int32_t)w2 - 1),
                                   (uint32_t)min(max(gy, 0), (int32_t)h2 - 1));
            s_l1[0][hy][hx] = t.x;
            s_l1[1][hy][hx] = t.y;
            s_l1[2][hy][hx] = t.z;
        }
        __syncthreads();
        // upscale_and_combine_kernel (PyramidConstructor.cu:67-112): all eight
        // pixels take their tent filter from level-1 row ly, the quad's centres
        // are columns lx and lx + 1, so one 4 x 3 neighbourhood and two filtered
        // values serve them all
        const float kern[3][3] = {{1.0f, 2.0f, 1.0f}, {2.0f, 4.0f, 2.0f}, {1.0f, 2.0f, 1.0f}};
        float rr[3][2];
#pragma unroll
        for (int ch = 0; ch < 3; ++ch) {
            float nb[4][3];  // columns lx - 1 .. lx + 2, rows ly - 1 .. ly + 1
#pragma unroll
            for (int v = 0; v < 3; ++v) {
                const float2 a = *reinterpret_cast<const float2*>(&s_l1[ch][ty + v][2 * tx]);
                const float2 b = *reinterpret_cast<const float2*>(&s_l1[ch][ty + v][2 * tx + 2]);
                nb[0][v] = a.x; nb[1][v] = a.y; nb[2][v] = b.x; nb[3][v] = b.y;
            }
            // r += nb * kern, the product exact (a weight of 1, 2 or 4), so one
            // fused multiply-add rounds exactly as the reference's multiply then add
#pragma unroll
            for (int base = 0; base < 2; ++base) {
                float r = 0.0f;
#pragma unroll
                for (int u = 0; u < 3; ++u)
#pragma unroll
                    for (int v = 0; v < 3; ++v) r = __fmaf_rn(nb[base + u][v], kern[u][v], r);
                rr[ch][base] = r / 16.0f;
            }
        }
#pragma unroll
        for (int r = 0; r < 2; ++r) {
            if (y + r >= h || x >= w) continue;
            f3 res[4];
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                const f3 up = mk(rr[0][k / 2], rr[1][k / 2], rr[2][k / 2]) + c[r][k] * sc[r][k];
                res[k] = c[r][k] + up;
            }
            const size_t p0 = (size_t)(y + r) * w + x;
            if (TONEMAP) {
                uint32_t o[4];
#pragma unroll
                for (int k = 0; k < 4; ++k) o[k] = tonemap_px(res[k], type, exposure, tables, tt);
                if (x + 3 < w) {
                    st_words<VEC, 4>(out8 + p0, o);
                } else {
#pragma unroll
                    for (uint32_t k = 0; k < 4; ++k)
                        if (x + k < w) out8[p0 + k] = o[k];
                }
            } else {
                uint32_t o[12];
#pragma unroll
                for (int k = 0; k < 4; ++k) {
                    o[3 * k] = __float_as_uint(res[k].x);
                    o[3 * k + 1] = __float_as_uint(res[k].y);
                    o[3 * k + 2] = __float_as_uint(res[k].z);
                }
                if (VEC == 4) {
                    st_words<4, 12>(reinterpret_cast<uint32_t*>(out) + 3 * p0, o);  // w is a multiple of 4
                } else {
                    // rows that start off 16 bytes: through shared memory, so that a
                    // warp stores consecutive words
                    st_words<4, 12>(&s_dyn[(2 * ty + r) * 3 * BLOOM_TW + 12 * tx], o);
                }
            }
        }
        if (!TONEMAP && VEC != 4) {
            __syncthreads();
            const uint32_t x0 = bx * BLOOM_TW, y0 = by * BLOOM_TH;
            const uint32_t n = 3 * min(BLOOM_TW, w - x0), rows = min(BLOOM_TH, h - y0);
            constexpr uint32_t LANES = 3 * BLOOM_TW / VEC;  // stores of a row
            for (uint32_t i = threadIdx.x; i < LANES * BLOOM_TH; i += BLOOM_THREADS) {
                const uint32_t r = i / LANES, k = (i - r * LANES) * VEC;
                if (r < rows && k < n)  // VEC == 2: w and so n are even
                    st_words<VEC, VEC>(reinterpret_cast<uint32_t*>(out) + 3 * ((size_t)(y0 + r) * w + x0) + k,
                                       &s_dyn[r * 3 * BLOOM_TW + k]);
            }
        }
        __syncthreads();  // s_l1 of the block's next tile
    }
}

// Level-1 scratch for the bloom entry point that allocates nothing
// (bloom_static_scratch below).  It lives in the module's global memory:
// every GPU that loads the library holds these 12 MiB until the process
// exits.  Host code must not pass this symbol to a kernel directly: on the
// host it names a host-side stand-in, not the device address.
static __device__ __align__(256) float g_bloom_scratch[3 * BLOOM_NOALLOC_MAX_HALF_PIXELS];

std::mutex g_scratch_mutex;
float* g_scratch_ptr[BLOOM_NOALLOC_MAX_DEVICES] = {};

std::mutex g_tone_mutex;
bool g_tone_enqueued[BLOOM_NOALLOC_MAX_DEVICES] = {};

}  // namespace

cudaError_t ensure_tone_levels(cudaStream_t st) {
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    if (dev < 0 || dev >= BLOOM_NOALLOC_MAX_DEVICES) return cudaSuccess;  // the kernels use the formulas
    std::lock_guard<std::mutex> lock(g_tone_mutex);
    if (g_tone_enqueued[dev]) return cudaSuccess;
    // ~0.6 G formula evaluations, once per device (about a millisecond);
    // kernels on other streams use the formulas until the publish runs.
    k_tone_levels_build<<<dim3(TONE_BUCKETS, TONE_TABLES), 256, 0, st>>>();
    k_tone_levels_publish<<<1, 256, 0, st>>>();
    e = cudaGetLastError();
    if (e == cudaSuccess) g_tone_enqueued[dev] = true;
    return e;
}

cudaError_t verify_tone_levels(unsigned long long mismatches[3], uint32_t flagged[3], cudaStream_t st) {
    cudaError_t e = ensure_tone_levels(st);
    if (e != cudaSuccess) return e;
    unsigned long long* d = nullptr;
    if ((e = cudaMalloc(&d, 3 * sizeof(unsigned long long))) != cudaSuccess) return e;
    static uint32_t host_tbl[TONE_TABLES][TONE_BUCKETS];
    static std::mutex host_mutex;
    std::lock_guard<std::mutex> lock(host_mutex);
    if ((e = cudaMemsetAsync(d, 0, 3 * sizeof(unsigned long long), st)) == cudaSuccess) {
        k_tone_levels_verify<<<148 * 16, 256, 0, st>>>(d);
        if ((e = cudaGetLastError()) == cudaSuccess &&
            (e = cudaMemcpyAsync(mismatches, d, 3 * sizeof(unsigned long long), cudaMemcpyDeviceToHost, st)) ==
                cudaSuccess &&
            (e = cudaMemcpyFromSymbolAsync(host_tbl, g_tone_levels, sizeof(host_tbl), 0, cudaMemcpyDeviceToHost,
                                           st)) == cudaSuccess)
            e = cudaStreamSynchronize(st);
    }
    cudaFree(d);
    if (e != cudaSuccess) return e;
    for (int t = 0; t < TONE_TABLES; ++t) {
        flagged[t] = 0;
        for (uint32_t q = 0; q < TONE_BUCKETS; ++q) flagged[t] += host_tbl[t][q] == TONE_FLAG;
    }
    return cudaSuccess;
}

// Bloom of an image whose output lies over its input.
static cudaError_t bloom_in_place(const float* hdr, uint32_t w, uint32_t h, const float th[4], float* out,
                                  cudaStream_t st) {
    // Set-up, once per device: ask the runtime for the device address of
    // the scratch array with the caller's device current.
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    if (dev < 0 || dev >= BLOOM_NOALLOC_MAX_DEVICES) return cudaErrorInvalidDevice;
    float* scratch = nullptr;
    {
        std::lock_guard<std::mutex> lock(g_scratch_mutex);
        if (!g_scratch_ptr[dev]) {
            void* p = nullptr;
            e = cudaGetSymbolAddress(&p, g_bloom_scratch);
            if (e != cudaSuccess) return e;
            g_scratch_ptr[dev] = static_cast<float*>(p);
        }
        scratch = g_scratch_ptr[dev];
    }
    // k_bloom_down writes every scratch element that k_bloom_up reads, so
    // nothing left over from an earlier call needs clearing.
    const uint32_t w2 = w / 2, h2 = h / 2;
    const float4 t4 = make_float4(th[0], th[1], th[2], th[3]);
    k_bloom_down<<<(w2 * h2 + 255) / 256, 256, 0, st>>>(hdr, w, h, t4, scratch, w2, h2);
    k_bloom_up<<<(w * h + 255) / 256, 256, 0, st>>>(hdr, w, h, t4, scratch, w2, h2, out);
    return cudaGetLastError();
}

// 16-byte alignment of the vectorised kernels' rows (cudaMalloc'd images
// are 256-byte aligned; caller buffers may not be).
static bool aligned16(const void* p) { return ((uintptr_t)p & 15u) == 0; }

// SMs of the current device, and resident blocks of 256 threads over all of
// them for a kernel with `smem` bytes of dynamic shared memory: the grid of the
// bloom kernel with staged tables (one wave, each block copying the tables
// once).  Cached per device and slot (kernel, type).
static uint32_t device_sms() {
    static std::mutex m;
    static uint32_t cache[BLOOM_NOALLOC_MAX_DEVICES] = {};
    int dev = 0, sms = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= BLOOM_NOALLOC_MAX_DEVICES) return 148;
    std::lock_guard<std::mutex> lock(m);
    if (!cache[dev]) {
        if (cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || sms <= 0) {
            (void)cudaGetLastError();
            return 148;
        }
        cache[dev] = (uint32_t)sms;
    }
    return cache[dev];
}
template <typename K>
static uint32_t wave_blocks(K kernel, uint32_t smem, int slot) {
    static std::mutex m;
    static uint32_t cache[BLOOM_NOALLOC_MAX_DEVICES][6] = {};
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= BLOOM_NOALLOC_MAX_DEVICES) return 148 * 4;
    std::lock_guard<std::mutex> lock(m);
    if (!cache[dev][slot]) {
        int per = 0;
        if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, kernel, 256, smem) != cudaSuccess || per <= 0) {
            (void)cudaGetLastError();
            return 148 * 4;
        }
        cache[dev][slot] = device_sms() * (uint32_t)per;
    }
    return cache[dev][slot];
}

cudaError_t launch_tonemap(const float* hdr, uint32_t npix, int type, float exposure, uint8_t* rgba, cudaStream_t st) {
    if (npix == 0) return cudaSuccess;
    cudaError_t e = ensure_tone_levels(st);
    if (e != cudaSuccess) return e;
    if (aligned16(hdr) && aligned16(rgba)) {
        const uint32_t n4 = (npix + 3) / 4, sms = device_sms();
        if (npix >= TONEMAP_SMEM_PIXELS)
            k_tonemap4_smem<<<sms, TONEMAP_THREADS, tone_smem_bytes(type), st>>>(hdr, npix, type, exposure,
                                                                                reinterpret_cast<uint32_t*>(rgba));
        else
            k_tonemap4<<<(n4 + 255) / 256, 256, 0, st>>>(hdr, npix, type, exposure, reinterpret_cast<uint32_t*>(rgba));
    } else {
        k_tonemap<<<(npix + 255) / 256, 256, 0, st>>>(hdr, npix, type, exposure, reinterpret_cast<uint32_t*>(rgba));
    }
    return cudaGetLastError();
}

// Floats per access that the rows of a w-pixel image at p (and of its output
// at q) allow: rows start on 16 bytes when w is a multiple of 4, on 8 when it
// is even.
static int bloom_vec(uint32_t w, const void* p, const void* q) {
    const uintptr_t a = (uintptr_t)p | (uintptr_t)q;
    return w % 4 == 0 && (a & 15u) == 0 ? 4 : w % 2 == 0 && (a & 7u) == 0 ? 2 : 1;
}

template <int VEC>
static cudaError_t launch_bloom_vec(const float* hdr, uint32_t w, uint32_t h, float4 th, float* out, uint8_t* rgba,
                                    int type, float exposure, cudaStream_t st) {
    const uint32_t tiles_x = (w + BLOOM_TW - 1) / BLOOM_TW, tiles = tiles_x * ((h + BLOOM_TH - 1) / BLOOM_TH);
    if (rgba) {
        const uint32_t wave = wave_blocks(k_bloom<true, VEC>, tone_smem_bytes(type),
                                          (type == 0 ? 0 : 1) + (VEC == 4 ? 0 : VEC == 2 ? 2 : 4));
        // copying the tables costs a block about as much as two tiles' reads
        const bool staged = tiles >= 2 * wave;
        k_bloom<true, VEC><<<staged ? wave : tiles, BLOOM_THREADS, staged ? tone_smem_bytes(type) : 0, st>>>(
            hdr, w, h, th, nullptr, reinterpret_cast<uint32_t*>(rgba), type, exposure, tiles_x, tiles, staged);
    } else {
        constexpr uint32_t smem = VEC == 4 ? 0u : 12u * BLOOM_TW * BLOOM_TH;
        k_bloom<false, VEC><<<tiles, BLOOM_THREADS, smem, st>>>(hdr, w, h, th, out, nullptr, 0, 0.0f, tiles_x, tiles,
                                                               false);
    }
    return cudaGetLastError();
}

cudaError_t launch_bloom(const float* hdr, uint32_t w, uint32_t h, const float th[4], float* out, uint8_t* rgba,
                         int type, float exposure, cudaStream_t st) {
    const float4 t4 = make_float4(th[0], th[1], th[2], th[3]);
    if (rgba) {
        cudaError_t e = ensure_tone_levels(st);
        if (e != cudaSuccess) return e;
    }
    switch (bloom_vec(w, hdr, rgba ? (const void*)rgba : (const void*)out)) {
        case 4: return launch_bloom_vec<4>(hdr, w, h, t4, out, rgba, type, exposure, st);
        case 2: return launch_bloom_vec<2>(hdr, w, h, t4, out, rgba, type, exposure, st);
        default: return launch_bloom_vec<1>(hdr, w, h, t4, out, rgba, type, exposure, st);
    }
}

cudaError_t bloom_static_scratch(const float* hdr, uint32_t w, uint32_t h, const float th[4], float* out,
                                 cudaStream_t st) {
    const uintptr_t a = (uintptr_t)hdr, b = (uintptr_t)out, bytes = sizeof(float) * 3 * (uintptr_t)w * h;
    if (a + bytes <= b || b + bytes <= a) return launch_bloom(hdr, w, h, th, out, nullptr, 0, 0.0f, st);
    return bloom_in_place(hdr, w, h, th, out, st);
}

}  // namespace cupbr_b200
