// Dequantize-fused GEMM on the sm_100a tensor cores for any number of rows, any K and N:
//     C[m,n] = A[m,k] (f32 or bf16) . dequant(W)[k,n] (+ addend),   f32 results at f32 accuracy.
//
// Stands in for the MatMul / FusedMatMulAdd dispatch with a quantized weight_format
// (src/compile.rs:1408-1419, 1511-1522 of meganeura; kernel src/shaders/matmul.wgsl with
// dequant_q4 / dequant_q8 as the B-tile load).
//
// Operands are sums of f16 values, whose products the tensor cores form exactly:
//   activations  x = (hi + lo * 2^-12) * 2^e, e per row and 128 k (split_rows_kernel): 22 bits of an f32 at least, down to
//                2^-29 of the row's largest value in these 128 k (the products with lo come first and the accumulator is scaled
//                by 2^-12 before the others are added); a bf16 value fits hi alone down to 2^-31, so that case has one plane and
//                two products instead of three.  Rows with more than 16 values below 2^-29 (bf16: 2^-27) are summed in plain f32.
//   weights      Q8: code * d has at most 19 bits, hi = rn16(code * d), lo = fma16(code, d, -hi), both exact, two
//                instructions for two weights.  Q4: hi = fma16(code, d, m), lo = rn16(code * d + m - hi), the difference
//                in f32: 2^-23 of the weight at most is left.  Both are multiples of 2^-24 as d and m are, so nothing is
//                lost for small scales.  The minimum is part of the weight: d * sum(code x) + m * sum(x) would cancel where
//                a large activation meets a weight near zero (2.2e-5 off for a value of 1000 in every 128, m = -7 d).
// The tensor core truncates when it adds to its f32 accumulator, which over a long K would cost more than f32 sums do
// (9e-6 for bf16 activations and K = 4096 in one accumulator).  So one accumulator takes a chunk of 128 k only, the small
// products first; then it is added to a register sum in f32, times 2^e: 2.2e-7 off the exact product at K = 4096 and 2.0e-7 at
// K = 512, where f32 sums in order of k are 1.1e-6 and 3.9e-7 off.  With bf16 activations and K from 2048 on two chunks share an
// accumulator and a scale: 5e-7, and half the drains (149 -> 143 us for 512 x 4096 x 14336 in a long run).
//
// Up to 16 f32 rows on Q8 weights that no streaming GEMV takes would otherwise be summed in short f32 trees, 1.2e-7 off.  For them an
// accumulator takes 32 k and its sums are added with what they round away: 1.0e-7 (2.0e-7 with 128 k).  16 x 12320 x 4099: 66 us
// (45 with 128 k, 3312 with that GEMV).
//
// Weights are the left operand, straight from TMEM: a tile is 128 weight columns (TMEM lanes) by up to 128
// tokens (any multiple of 16), so that few tokens cost few products and no shared-memory pass for weights.
// Tiles are cut along K into chunks and the chunks of all tiles are shared out evenly over the CTAs (1 per SM); where a
// tile is spread over several CTAs, each leaves its partial sums in the workspace and the one that finishes last adds
// them up in order: results do not depend on timing.
//   warp 0        token planes, 64 k of one plane per copy (cp.async.bulk of a block that split_rows_kernel has laid
//                 out in the 128-byte swizzle), ring of 8; scales of a chunk, ring of 8.
//   warp 1        MMA issue: tcgen05.mma.kind::f16, M=128 (weight columns), N=tokens, K=16, A in TMEM.
//   warps 4-11    drain: 32 weight columns by half of the tokens per warp, sums in registers; results.
//   warps 12-19   weights: two groups of four, chunks in turn; cp.async of a warp's 32 columns two chunks
//                 of its own ahead, conversion, tcgen05.st.
// TMEM: two accumulators of 128 columns, two weight stages of 64 (hi) + 64 (lo) columns.
// Sums that are not finite (non-finite inputs, a weight beyond the f16 range) are noted in the workspace and computed again
// element by element on the CUDA cores once the CTA's pipeline has ended, so that no bounded wait depends on how many they are;
// a row with a NaN is known after one look at it.
//
// What bounds it: of the 2650 cycles that a chunk of 128 x 128 takes with f32 activations the tensor core needs 1536 (2100 and 1024
// for bf16), the rest is the hand-over of a weight stage: products of chunk i - 2 done, conversion (1500 cycles, four warps),
// products of chunk i; 52 % of the issue slots are taken (62 % with Q4, whose weights take three times the instructions of Q8's).
// Measured and dropped: weight stages of 64 k (147 instead of 112 us for bf16, twice the waits), two issuing warps, both groups on
// every chunk, two token tiles per converted weight (no change).
// In a long run (the power cap adds a tenth) 512 x 4096 x 12288 Q4 f32 takes 155 us against 1993 on the CUDA cores, 512 x 4096 x 14336 Q8
// bf16 142 against 147 us of a kernel with one 112-column strip of bf16 weight pairs per CTA and 512 tokens, whose sums were
// 9.4e-6 off.
//
// Every mbarrier wait is bounded; when one runs out the device-wide error word is raised (mgq_device_status reports
// MGQ_ERR_TIMEOUT), the roles run to their ends without waiting and the CTA frees its TMEM.
#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <mutex>
#include <utility>
#include <vector>

#include "mgq_launch.cuh"
#include "mgq_tcgen05.cuh"

namespace mgq {
namespace {

constexpr uint32_t kChunk = 128;                   // k per accumulator
constexpr uint32_t kCols = 128;                    // weight columns of a tile
constexpr uint32_t kMaxTok = 128;                  // tokens of a tile
// Chunks that share an accumulator and a scale.  Below 2048 k the f32 sums of the tiled kernel would be as exact as pairs are.
__host__ __device__ constexpr uint32_t group_of(uint32_t planes, uint32_t k) { return planes == 1 && k >= 2048 ? 2 : 1; }
constexpr uint32_t kSlots = 8;                     // ring of token sub-tiles (64 k of one plane)
constexpr uint32_t kScaleSlots = 8;
constexpr uint32_t kRaw = 4;                       // chunks of packed weights in flight, two per group
constexpr uint32_t kSplitThreads = 640;
constexpr uint32_t kPassElems = 1u << 25;          // activations per launch: bounds the workspace (128 MB of planes)

__device__ unsigned int g_split_error = 0;

struct SplitParams {
    const uint8_t *w;
    const void *a;
    const float *addend;
    float *c;
    const uint8_t *planes;          // [m tile][chunk][slot][tokens * 128 B]
    const float *scales;            // [m tile][chunk][tokens]
    float *partial;                 // [CTA][2][128 tokens][128 columns]
    unsigned int *counters;         // one per tile
    unsigned int *odd_by;           // [tile][drain warp]: 1 + the CTA whose warp has left masks, or 0
    unsigned long long *odd;        // [tile][drain thread]: its tokens whose sums are not finite
    unsigned long long num_blocks;
    uint32_t m, k, n, bpc;
    uint32_t tok, m_tiles, tiles;   // tokens of a tile, tiles
    uint32_t chunks;                // per tile
    uint32_t units;                 // tiles * chunks
    uint32_t wide;                  // packed weights can be copied 16 bytes at a time
};

struct __align__(16) SplitShared {
    unsigned long long slot_full[kSlots], slot_empty[kSlots / 2];      // empty: a chunk's sub-tiles together
    unsigned long long sc_full[kScaleSlots], sc_empty[kScaleSlots];
    unsigned long long w_full[2], w_empty[2], d_empty[2], d_full[2], flushed;
    uint32_t tmem_base;
    volatile int failed;
    uint32_t last;
};

__host__ __device__ constexpr uint32_t raw_bytes(int fmt) { return fmt == MGQ_FMT_Q8 ? 144u : 80u; }      // of a column and chunk: Q4 = 16 header bytes | 64 nibble bytes

// CTA that owns unit u, and first unit of CTA g, when `units` are shared out over `ctas`.
__host__ __device__ inline uint32_t unit_owner(uint32_t u, uint32_t units, uint32_t ctas)
{
    return (uint32_t)((((unsigned long long)u + 1) * ctas - 1) / units);
}
__host__ __device__ inline uint32_t unit_start(uint32_t g, uint32_t units, uint32_t ctas)
{
    return (uint32_t)((unsigned long long)g * units / ctas);
}

// ------------------------------------------------------------------------------------ activations

__device__ __forceinline__ float load_act(const void *a, size_t i, bool bf16)
{
    return bf16 ? __bfloat162float(static_cast<const __nv_bfloat16 *>(a)[i]) : static_cast<const float *>(a)[i];
}

// Powers of two: values up to `top` come out below 2^15 when multiplied by `down`.
__device__ __forceinline__ void pick_scale(float top, float &down, float &up)
{
    const int e = (int)((__float_as_uint(top) >> 23) & 0xFFu) - 127;      // 128: infinity or NaN
    const int s = max(min(14 - e, 126), -126);
    down = __uint_as_float((uint32_t)(127 + s) << 23);
    up = __uint_as_float((uint32_t)(127 - s) << 23);
}

constexpr uint32_t kLowShift = 12;                 // the low plane is stored 2^12 times as large: |lo| <= 2^3, beside |hi| <= 2^15

// Four consecutive places of one row: f16 parts of v * down into the planes' swizzled sub-tiles.  pos: place within the chunk.
__device__ __forceinline__ void store4(uint8_t *block, uint32_t sub, uint32_t planes, uint32_t t, uint32_t pos, const float (&v)[4], float down)
{
    __align__(8) __half hi[4], lo[4];
#pragma unroll
    for (int i = 0; i < 4; i++) {
        const float s = v[i] * down;
        hi[i] = __float2half_rn(s);
        lo[i] = __float2half_rn((s - __half2float(hi[i])) * (float)(1u << kLowShift));
    }
    const uint32_t half = pos >> 6, byte = (pos & 63u) * 2u;
    uint8_t *h = block + (size_t)((planes == 2 ? 2u : 0u) + half) * sub + t * 128u, *l = block + (size_t)half * sub + t * 128u;      // lo, lo, hi, hi
    const uint32_t at = (((byte >> 4) ^ (t & 7u)) << 4) | (byte & 15u);
    *reinterpret_cast<uint2 *>(h + at) = *reinterpret_cast<const uint2 *>(hi);
    if (planes == 2) *reinterpret_cast<uint2 *>(l + at) = *reinterpret_cast<const uint2 *>(lo);
}

// A warp per row and group of chunks.  Bound by the read of the activations (8 MB for 512 x 4096 f32) and as many bytes written,
// all of which stay in L2 for the GEMM behind it.
__global__ void __launch_bounds__(256) split_rows_kernel(const void *a, bool bf16, bool vec, uint8_t *planes_out, float *scales_out, unsigned int *counters, uint32_t words,
                                                         uint32_t m, uint32_t k, uint32_t tok, uint32_t chunks, uint32_t planes, bool q4)
{
    pdl_launch_dependents();
    const uint32_t lane = threadIdx.x & 31u, gid = blockIdx.x * 8 + (threadIdx.x >> 5);
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < words; i += gridDim.x * blockDim.x) counters[i] = 0;      // the GEMM's counters and marks
    const uint32_t span = group_of(planes, k), groups = (chunks + span - 1) / span;
    const uint32_t row = gid / groups, first_chunk = gid % groups * span;
    if (row >= m) return;
    const uint32_t mt = row / tok, t = row % tok, sub = tok * 128u;
    float v[2][4] = {};
    uint32_t top = 0;                                           // largest magnitude by its bits: NaN stays the largest
#pragma unroll
    for (uint32_t c = 0; c < 2; c++) {
        const uint32_t kk = (first_chunk + c) * kChunk + lane * 4;
        if (c < span && kk < k) {
            const size_t at = (size_t)row * k + kk;
            if (vec && !bf16) {
                const float4 q = *reinterpret_cast<const float4 *>(static_cast<const float *>(a) + at);
                v[c][0] = q.x; v[c][1] = q.y; v[c][2] = q.z; v[c][3] = q.w;
            } else if (vec) {
                const uint2 q = *reinterpret_cast<const uint2 *>(static_cast<const __nv_bfloat16 *>(a) + at);
                v[c][0] = __uint_as_float(q.x << 16); v[c][1] = __uint_as_float(q.x & 0xFFFF0000u);
                v[c][2] = __uint_as_float(q.y << 16); v[c][3] = __uint_as_float(q.y & 0xFFFF0000u);
            } else {
#pragma unroll
                for (int i = 0; i < 4; i++) v[c][i] = load_act(a, at + i, bf16);
            }
        }
    }
#pragma unroll
    for (uint32_t c = 0; c < 2; c++)
#pragma unroll
        for (int i = 0; i < 4; i++) top = max(top, __float_as_uint(v[c][i]) & 0x7FFFFFFFu);
    top = __reduce_max_sync(0xffffffffu, top);
    float down, up;
    pick_scale(__uint_as_float(top), down, up);
    // below it f16 parts of that scale hold less than 22 bits of a value; a lone part holds 8 down to 2^-31, but 256 k with
    // one value of 10^8 at weights of 0 were 1.1e-5 off (with bf16 operands in their own range 7.5e-6)
    const float least = __uint_as_float(top) * (planes == 2 ? 0x1p-29f : 0x1p-27f);
    uint32_t small = 0;
#pragma unroll
    for (uint32_t c = 0; c < 2; c++)
#pragma unroll
        for (int i = 0; i < 4; i++) small += fabsf(v[c][i]) < least && v[c][i] != 0.f ? 1u : 0u;
    const bool wide = __reduce_add_sync(0xffffffffu, small) > kChunk / 8;
#pragma unroll
    for (uint32_t c = 0; c < 2; c++) {
        if (c >= span || first_chunk + c >= chunks) break;      // uniform over the warp
        const size_t block = (size_t)mt * chunks + first_chunk + c;
        // too many small values, not finite, or so large (from 2^120 on) that f32 sums overflow on their way: a NaN scale makes the row's sums NaN, which the
        // GEMM computes again in plain f32
        if (lane == 0) scales_out[block * tok + t] = wide || top >= (127u + 120u) << 23 ? __uint_as_float(0x7FC00000u) : up;
        if (q4) {
            // Q4 weights unpack as pairs (k, k + 4) of eight: order 0 4 1 5 2 6 3 7
            const bool odd = lane & 1u;
            const float r0 = __shfl_xor_sync(0xffffffffu, odd ? v[c][0] : v[c][2], 1), r1 = __shfl_xor_sync(0xffffffffu, odd ? v[c][1] : v[c][3], 1);
            if (odd) { v[c][0] = r0; v[c][1] = v[c][2]; v[c][2] = r1; }
            else     { v[c][3] = r1; v[c][2] = v[c][1]; v[c][1] = r0; }
        }
        store4(planes_out + block * 2 * planes * sub, sub, planes, t, lane * 4, v[c], down);
    }
}

// ------------------------------------------------------------------------------------------ pieces

__device__ __forceinline__ void bulk_load(void *dst, const void *src, uint32_t bytes, unsigned long long *bar)
{
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
                 ::"r"(smem_u32(dst)), "l"(src), "r"(bytes), "r"(smem_u32(bar)) : "memory");
}
// 16 or 4 bytes; live false: zeros.
__device__ __forceinline__ void copy16(uint32_t dst, const void *src, bool live)
{
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(live ? 16u : 0u) : "memory");
}
__device__ __forceinline__ void copy4(uint32_t dst, const void *src, bool live)
{
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(dst), "l"(src), "r"(live ? 4u : 0u) : "memory");
}

// Products of the K = 16 steps from .. from + COUNT - 1 of a chunk into one accumulator, the small ones first.  open: it holds a chunk already.
template <int PLANES, int COUNT>
__device__ __forceinline__ void issue_products(uint32_t d, uint32_t w_hi, uint32_t w_lo, uint32_t x_hi, uint32_t x_lo, uint32_t sub16, uint32_t instr, uint32_t from, bool open)
{
    auto x_at = [&](uint32_t x, uint32_t j) { return x + ((from + j) / 4) * sub16 + ((from + j) % 4) * 2u; };
    auto w_at = [&](uint32_t w, uint32_t j) { return w + (from + j) * 8u; };
    if (PLANES == 2) {                                          // never two chunks per accumulator
        umma_f16_ts<false>(d, w_at(w_hi, 0), x_at(x_lo, 0), instr);
#pragma unroll
        for (uint32_t j = 1; j < COUNT; j++) umma_f16_ts<true>(d, w_at(w_hi, j), x_at(x_lo, j), instr);
        umma_f16_ts_scaled<kLowShift>(d, w_at(w_lo, 0), x_at(x_hi, 0), instr);
    } else if (open) umma_f16_ts<true>(d, w_at(w_lo, 0), x_at(x_hi, 0), instr);
    else             umma_f16_ts<false>(d, w_at(w_lo, 0), x_at(x_hi, 0), instr);
#pragma unroll
    for (uint32_t j = 1; j < COUNT; j++) umma_f16_ts<true>(d, w_at(w_lo, j), x_at(x_hi, j), instr);
#pragma unroll
    for (uint32_t j = 0; j < COUNT; j++) umma_f16_ts<true>(d, w_at(w_hi, j), x_at(x_hi, j), instr);
}
// kind::f16 instruction descriptor: D f32, A and B f16, both K-major.
__device__ __forceinline__ uint32_t split_instr(uint32_t n) { return (1u << 4) | ((n >> 3) << 17) | ((kCols >> 4) << 24); }

__device__ __forceinline__ __half2 as_half2(uint32_t v) { return *reinterpret_cast<const __half2 *>(&v); }
__device__ __forceinline__ uint32_t as_word(__half2 v) { return *reinterpret_cast<const uint32_t *>(&v); }

// Two codes as f16 1024 + c in one word -> exact parts of (c - offset) * d.
__device__ __forceinline__ void split_codes(uint32_t magic, __half2 offset, __half2 d, uint32_t &hi, uint32_t &lo)
{
    const __half2 c = __hsub2(as_half2(magic), offset);
    const __half2 h = __hmul2_rn(c, d);                         // never contracted into the fma below
    hi = as_word(h);
    lo = as_word(__hfma2(c, d, __hneg2(h)));
}

// a - c and a * b + c of f16 values and an f32, rounded once.
__device__ __forceinline__ float sub_mixed(__half a, float c)
{
    float d;
    asm("sub.rn.f32.f16 %0, %1, %2;" : "=f"(d) : "h"(__half_as_ushort(a)), "f"(c));
    return d;
}
__device__ __forceinline__ float fma_mixed(__half a, __half b, float c)
{
    float d;
    asm("fma.rn.f32.f16 %0, %1, %2, %3;" : "=f"(d) : "h"(__half_as_ushort(a)), "h"(__half_as_ushort(b)), "f"(c));
    return d;
}
// Two codes as f16 1024 + c in one word -> parts of c * d + m: the first rounded to nearest, the second what is left of it.
__device__ __forceinline__ void split_affine(uint32_t magic, __half2 d, __half2 m, float m32, uint32_t &hi, uint32_t &lo)
{
    const __half2 c = __hsub2(as_half2(magic), __float2half2_rn(1024.f));
    const __half2 h = __hfma2(c, d, m);
    hi = as_word(h);
    lo = as_word(__floats2half2_rn(fma_mixed(__low2half(c), __low2half(d), -sub_mixed(__low2half(h), m32)),
                                   fma_mixed(__high2half(c), __low2half(d), -sub_mixed(__high2half(h), m32))));
}

// The element (row, col) in plain f32, the way the tiled kernel sums it.
template <int FMT>
__device__ __forceinline__ float plain_element(const SplitParams &p, bool bf16, uint32_t row, uint32_t col)
{
    float acc = 0.f;
    const uint32_t *w32 = reinterpret_cast<const uint32_t *>(p.w);
    for (uint32_t b = 0; b < p.bpc; b++) {
        const unsigned long long g = (unsigned long long)col * p.bpc + b;
        float d, lo = 0.f;
        const uint32_t *q;
        if (FMT == MGQ_FMT_Q4) {
            const float2 dm = __half22float2(as_half2(w32[g]));
            d = dm.x; lo = dm.y;
            q = w32 + p.num_blocks + g * 4;
        } else {
            d = __half2float(__ushort_as_half((unsigned short)(w32[g * 9] & 0xFFFFu)));
            q = w32 + g * 9 + 1;
        }
        for (uint32_t i = 0; i < 32; i++) {
            const float code = FMT == MGQ_FMT_Q4 ? (float)((q[i >> 3] >> (4 * (i & 7u))) & 0xFu) : (float)(int)(signed char)((q[i >> 2] >> (8 * (i & 3u))) & 0xFFu);
            const float w = FMT == MGQ_FMT_Q4 ? code * d + lo : code * d;
            acc = fmaf(load_act(p.a, (size_t)row * p.k + b * 32u + i, bf16), w, acc);
        }
    }
    return acc;
}

// The sums that a drain warp has noted, tile by tile: a thread its own column, the rows one after another.
template <int FMT>
__device__ __noinline__ void redo_odd(const SplitParams &p, bool bf16, uint32_t u_begin, uint32_t u_end, uint32_t warp, uint32_t lane)
{
    for (uint32_t tile = u_begin / p.chunks; tile <= (u_end - 1) / p.chunks; tile++) {
        uint32_t by = lane == 0 ? p.odd_by[tile * 8 + warp] : 0u;
        if (__shfl_sync(0xffffffffu, by, 0) != blockIdx.x + 1) continue;
        const unsigned long long odd = p.odd[((size_t)tile * 8 + warp) * 32 + lane];
        const uint32_t groups = p.tok / 16, m0 = (tile % p.m_tiles) * p.tok + (warp >= 4 ? (groups + 1) / 2 * 16 : 0);
        const uint32_t col = (tile / p.m_tiles) * kCols + (warp & 3u) * 32 + lane;
        for (uint32_t r = 0; r < 64; r++) {
            const bool mine = odd >> r & 1u;
            if (!__any_sync(0xffffffffu, mine)) continue;
            const uint32_t row = m0 + r;
            bool nan = false;                                   // NaN times any weight is NaN, and so is the sum
            for (uint32_t k0 = 0; k0 < p.k && !nan; k0 += 256) {
                bool found = false;
#pragma unroll
                for (uint32_t x = 0; x < 256; x += 32)
                    if (k0 + x < p.k) found |= isnan(load_act(p.a, (size_t)row * p.k + k0 + x + lane, bf16));
                nan = __any_sync(0xffffffffu, found);
            }
            if (!mine) continue;
            const float v = nan ? __uint_as_float(0x7FC00000u) : plain_element<FMT>(p, bf16, row, col);
            const size_t o = (size_t)row * p.n + col;
            p.c[o] = p.addend ? v + p.addend[o] : v;
        }
    }
}

// Asynchronous copy of the packed bytes that a warp's 32 columns (from col0) hold of a chunk; neighbouring lanes copy
// neighbouring pieces of a column, and a lane's addresses advance by constants.  Blocks beyond K read as zeros; columns
// beyond N are left out (a weight column is a row of the product: nothing else depends on it).
template <int FMT>
__device__ __forceinline__ void fetch_weights(const SplitParams &p, uint32_t dst, uint32_t col0, uint32_t chunk, uint32_t lane)
{
    constexpr uint32_t kBytes = raw_bytes(FMT);
    const uint32_t b0 = chunk * 4, cols = col0 < p.n ? min(32u, p.n - col0) : 0u;
    const unsigned long long block = (unsigned long long)col0 * p.bpc + b0;
    if (FMT == MGQ_FMT_Q8) {
        const uint8_t *src = p.w + block * 36u;
        const size_t pitch = (size_t)p.bpc * 36u;
        if (p.wide) {                                           // 9 pieces of 16 bytes: three lanes per column
            const uint32_t c = lane / 3, piece = (lane % 3) * 16u;
            const uint8_t *from = src + c * pitch + piece;
            const uint32_t to = dst + c * kBytes + piece;
#pragma unroll
            for (uint32_t i = 0; i < 3; i++)
                if (c < 10 && c + i * 10 < cols) {
#pragma unroll
                    for (uint32_t x = 0; x < 3; x++) copy16(to + i * 10 * kBytes + x * 48u, from + i * 10 * pitch + x * 48u, true);
                }
            const uint32_t rest = 30 + lane / 9;                // columns 30 and 31: 18 lanes
            if (lane < 18 && rest < cols) copy16(dst + rest * kBytes + (lane % 9) * 16u, src + rest * pitch + (lane % 9) * 16u, true);
        } else {                                                // 36 words: a whole warp per column, the last four words of eight columns at a time
            const bool live = b0 + lane / 9 < p.bpc;
            const uint8_t *from = live ? src + lane * 4u : p.w;
            const size_t step = live ? pitch : 0;
            const uint32_t to = dst + lane * 4u;
#pragma unroll 8
            for (uint32_t c = 0; c < cols; c++) copy4(to + c * kBytes, from + c * step, live);
            const uint32_t c = lane / 4, word = 32 + lane % 4;
            const bool rest = b0 + 3 < p.bpc;
#pragma unroll
            for (uint32_t i = 0; i < 4; i++)
                if (c + i * 8 < cols) copy4(dst + (c + i * 8) * kBytes + word * 4u, rest ? src + (c + i * 8) * pitch + word * 4u : p.w, rest);
        }
    } else {
        const uint32_t c = lane / 4, b = lane % 4;              // four blocks of eight columns at a time
        const bool live = b0 + b < p.bpc;
        const uint8_t *hdr = p.w + (block + (unsigned long long)c * p.bpc + b) * 4u, *nib = p.w + (p.num_blocks + (block + (unsigned long long)c * p.bpc + b) * 4u) * 4u;
#pragma unroll
        for (uint32_t i = 0; i < 4; i++)
            if (c + i * 8 < cols) copy4(dst + (c + i * 8) * kBytes + b * 4u, live ? hdr + (size_t)i * 8 * p.bpc * 4u : p.w, live);
        if (p.wide) {
#pragma unroll
            for (uint32_t i = 0; i < 4; i++)
                if (c + i * 8 < cols) copy16(dst + (c + i * 8) * kBytes + 16u + b * 16u, live ? nib + (size_t)i * 8 * p.bpc * 16u : p.w, live);
        } else {
            const uint32_t c2 = lane / 16, word = lane % 16;
            const bool live2 = b0 + word / 4 < p.bpc;
            const uint8_t *from = p.w + (p.num_blocks + (block + (unsigned long long)c2 * p.bpc) * 4u + word) * 4u;
#pragma unroll 4
            for (uint32_t i = 0; i < 16; i++)
                if (c2 + i * 2 < cols) copy4(dst + (c2 + i * 2) * kBytes + 16u + word * 4u, live2 ? from + (size_t)i * 2 * p.bpc * 16u : p.w, live2);
        }
    }
}

// COUNT groups of 16 tokens: sums += accumulator * scale.
template <int G0, int COUNT>
__device__ __forceinline__ void drain_part(uint32_t from, const uint8_t *scale, float (&acc)[4][16])
{
    uint32_t r[COUNT][16];
#pragma unroll
    for (int g = 0; g < COUNT; g++)
        asm volatile("tcgen05.ld.sync.aligned.32x32b.x16.b32 "
                     "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
                     : "=r"(r[g][0]), "=r"(r[g][1]), "=r"(r[g][2]), "=r"(r[g][3]), "=r"(r[g][4]), "=r"(r[g][5]), "=r"(r[g][6]), "=r"(r[g][7]),
                       "=r"(r[g][8]), "=r"(r[g][9]), "=r"(r[g][10]), "=r"(r[g][11]), "=r"(r[g][12]), "=r"(r[g][13]), "=r"(r[g][14]), "=r"(r[g][15])
                     : "r"(from + (G0 + g) * 16) : "memory");
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
    for (int g = 0; g < COUNT; g++)
#pragma unroll
        for (int e = 0; e < 16; e += 4) {
            const float4 s = *reinterpret_cast<const float4 *>(scale + ((G0 + g) * 16 + e) * 4);
            fma_pair(acc[G0 + g][e], acc[G0 + g][e + 1], __uint_as_float(r[g][e]), __uint_as_float(r[g][e + 1]), s.x, s.y);
            fma_pair(acc[G0 + g][e + 2], acc[G0 + g][e + 3], __uint_as_float(r[g][e + 2]), __uint_as_float(r[g][e + 3]), s.z, s.w);
        }
}

// sum += x; low collects what the sums round away.
__device__ __forceinline__ void add_exact(float &sum, float &low, float x)
{
    const float s = __fadd_rn(sum, x), b = __fsub_rn(s, sum);
    low = __fadd_rn(low, __fadd_rn(__fsub_rn(sum, __fsub_rn(s, b)), __fsub_rn(x, b)));
    sum = s;
}

// drain_part for one group of 16 tokens; the scales are powers of two, so that the products are exact.
__device__ __forceinline__ void drain_fine(uint32_t from, const uint8_t *scale, float (&sum)[16], float (&low)[16])
{
    uint32_t r[16];
    tmem_ld16(from, r);
#pragma unroll
    for (int e = 0; e < 16; e++) add_exact(sum[e], low[e], __uint_as_float(r[e]) * *reinterpret_cast<const float *>(scale + e * 4));
}

// acc += the sums that another CTA has left.
__device__ __forceinline__ void add_part(const float *src, uint32_t groups, float (&acc)[4][16])
{
#pragma unroll
    for (int g = 0; g < 4; g++)
        if (g < (int)groups) {
            float v[16];
#pragma unroll
            for (int e = 0; e < 16; e++) v[e] = __ldcg(src + (g * 16 + e) * kCols);
#pragma unroll
            for (int e = 0; e < 16; e++) acc[g][e] += v[e];
        }
}

// FINE: an accumulator per 32 k, compensated sums; one group of 16 tokens only.
template <int FMT, int PLANES, bool FINE>
__global__ void __launch_bounds__(kSplitThreads, 1) gemm_split_kernel(const __grid_constant__ SplitParams p)
{
    extern __shared__ uint8_t smem_raw[];
    __shared__ SplitShared sh;
    constexpr uint32_t kRawChunk = kCols * raw_bytes(FMT);
    constexpr uint32_t kParts = 2 * PLANES, kDepth = kSlots / kParts;       // sub-tiles of a chunk, chunks in the ring
    const uint32_t group = PLANES == 1 ? group_of(PLANES, p.k) : 1;
    uint8_t *ring = reinterpret_cast<uint8_t *>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
    const uint32_t sub = p.tok * 128u;                          // bytes of a token sub-tile, a multiple of 2048
    const uint32_t scale_bytes = p.tok * 4u;                    // a multiple of 64
    uint8_t *scale_ring = ring + kSlots * sub;
    uint8_t *raw = scale_ring + kScaleSlots * scale_bytes;
    const uint32_t tid = threadIdx.x, warp = tid >> 5, lane = tid & 31u;
    const uint32_t u_begin = unit_start(blockIdx.x, p.units, gridDim.x), u_end = unit_start(blockIdx.x + 1, p.units, gridDim.x);

    if (tid == 0) {
        for (uint32_t s = 0; s < kSlots; s++) mbar_init(&sh.slot_full[s], 1);
        for (uint32_t s = 0; s < kDepth; s++) mbar_init(&sh.slot_empty[s], 1);
        for (uint32_t s = 0; s < kScaleSlots; s++) { mbar_init(&sh.sc_full[s], 1); mbar_init(&sh.sc_empty[s], 8); }
        for (uint32_t s = 0; s < 2; s++) {
            mbar_init(&sh.w_full[s], 4);
            mbar_init(&sh.d_empty[s], 8);
            mbar_init(&sh.w_empty[s], 1);
            mbar_init(&sh.d_full[s], 1);
        }
        mbar_init(&sh.flushed, 1);
        sh.failed = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 1) tmem_alloc(&sh.tmem_base, 512);
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = sh.tmem_base;
    const uint32_t tmem_w = tmem + 2 * kMaxTok;                 // stage s: hi at +128 s, lo at +128 s + 64

    bool redo = false;                                          // a drain warp has noted sums that are not finite
    if (warp < 4) {
        asm volatile("setmaxnreg.dec.sync.aligned.u32 56;");
        if (warp == 0) {
            // ------------------------------------------------------------------ token planes and scales
            // lane x: the x-th sub-tile of every chunk; lane kParts: scales.  One lane for all of them was late: a
            // wait, an arrival and a copy take it 300 cycles.
            if (lane <= kParts) {
                pdl_wait();
                const uint32_t depth = lane < kParts ? kDepth : kScaleSlots, count = u_end - u_begin;
                const uint32_t bytes = lane < kParts ? sub : scale_bytes, pitch = lane < kParts ? kParts * sub : scale_bytes;
                const uint8_t *base = lane < kParts ? p.planes + lane * sub : reinterpret_cast<const uint8_t *>(p.scales);
                // [m tile][chunk]: the tiles of a column strip follow one another
                uint32_t at = u_begin / p.chunks % p.m_tiles * p.chunks + u_begin % p.chunks, armed = 0;
                const uint32_t wrap = p.m_tiles * p.chunks;
                for (uint32_t i = 0; i < count; i++, at = at + 1 == wrap ? 0 : at + 1) {
                    const uint32_t s = i % depth, slot = s * kParts + lane;
                    unsigned long long *full = lane < kParts ? &sh.slot_full[slot] : &sh.sc_full[s], *empty = lane < kParts ? &sh.slot_empty[s] : &sh.sc_empty[s];
                    if (!mbar_wait(empty, ((i / depth) & 1u) ^ 1u, &sh.failed, &g_split_error)) continue;
                    mbar_arrive_expect_tx(full, bytes);
                    bulk_load(lane < kParts ? ring + slot * sub : scale_ring + s * scale_bytes, base + (size_t)at * pitch, bytes, full);
                    armed = i + 1;
                }
                if (sh.failed)                                  // let this lane's own copies land before the CTA exits
                    for (uint32_t j = armed > depth ? armed - depth : 0; j < armed; j++) {
                        unsigned long long *full = lane < kParts ? &sh.slot_full[j % depth * kParts + lane] : &sh.sc_full[j % depth];
                        for (uint32_t i = 0; i < kWaitLimit && !mbar_try_wait(full, (j / depth) & 1u); i++) { }
                    }
            }
        } else if (warp == 1) {
            // ------------------------------------------------------------------ MMA issue
            // The whole warp runs the loop and one elected lane issues: addresses and descriptors then stay in uniform registers (a
            // lane in a branch of its own took 100 cycles per MMA, N = 128 needs 64).  All waits of a chunk at once and two
            // commits per chunk (each takes the warp 170 cycles).
            const uint32_t instr = split_instr(p.tok);
            const uint32_t tm = __shfl_sync(0xffffffffu, tmem, 0), count = __shfl_sync(0xffffffffu, u_end - u_begin, 0);
            const bool leader = elect_one();
            const uint32_t ring16 = smem_u32(ring) >> 4;
            const uint32_t sub16 = sub >> 4;
            uint32_t chunk = __shfl_sync(0xffffffffu, u_begin % p.chunks, 0), filled = 0;      // accumulators so far
            bool ok = true, open = false;                       // open: the accumulator holds a chunk already
            for (uint32_t i = 0; i < count; i++) {
                const uint32_t stage = i & 1u, ph = (i >> 1) & 1u, s = i % kDepth;
                uint32_t b = filled & 1u;
                const bool close = group == 1 || chunk % group == group - 1 || chunk + 1 == p.chunks || i + 1 == count;
                const uint32_t w_hi = tm + 2 * kMaxTok + stage * 128u, w_lo = w_hi + 64u;
                // lane 0: accumulator, 1: weights, 4..: the chunk's sub-tiles
                unsigned long long *bar = lane == 0 ? &sh.d_empty[b] : lane == 1 ? &sh.w_full[stage] : &sh.slot_full[(s * kParts + lane - 4u) % kSlots];
                const uint32_t parity = lane == 0 ? ((filled >> 1) & 1u) ^ 1u : lane == 1 ? ph : (i / kDepth) & 1u;
                ok = mbar_wait_lanes(bar, parity, lane < 2 || (lane >= 4 && lane < 4 + kParts), &sh.failed, &g_split_error);
                if (!ok) break;
                tc_fence_after();
                const uint32_t x_lo = ring16 + s * kParts * sub16, x_hi = x_lo + (kParts - 2) * sub16;
                if (FINE) {                                     // all quarters of the chunk but the last
                    for (uint32_t from = 0; from < 6; from += 2) {
                        if (leader) {
                            issue_products<PLANES, 2>(tm + b * kMaxTok, w_hi, w_lo, x_hi, x_lo, sub16, instr, from, false);
                            umma_commit(&sh.d_full[b]);
                        }
                        __syncwarp();
                        filled++;
                        b = filled & 1u;
                        ok = ok && mbar_wait_lanes(&sh.d_empty[b], ((filled >> 1) & 1u) ^ 1u, lane == 0, &sh.failed, &g_split_error);
                        tc_fence_after();
                    }
                    if (!ok) break;
                }
                if (leader) {
                    if (FINE) issue_products<PLANES, 2>(tm + b * kMaxTok, w_hi, w_lo, x_hi, x_lo, sub16, instr, 6, false);
                    else      issue_products<PLANES, 8>(tm + b * kMaxTok, w_hi, w_lo, x_hi, x_lo, sub16, instr, 0, open);
                    umma_commit(&sh.w_empty[stage]);
                    umma_commit(&sh.slot_empty[s]);
                    if (close) umma_commit(&sh.d_full[b]);
                }
                __syncwarp();
                open = !close;
                if (close) filled++;
                if (++chunk == p.chunks) chunk = 0;
            }
            if (!ok && leader) {                                // products in flight end before the CTA does
                umma_commit(&sh.flushed);
                for (uint32_t i = 0; i < kWaitLimit && !mbar_try_wait(&sh.flushed, 0); i++) { }
            }
        }
    } else if (warp < 12) {
        asm volatile("setmaxnreg.inc.sync.aligned.u32 128;");
        // ---------------------------------------------------------------------- drain and results
        const uint32_t quad = warp & 3u, wg = (warp - 4) >> 2;
        const uint32_t lane_addr = (quad * 32u) << 16;
        // the first four warps take the first half of the tile's groups of 16 tokens, the others the rest
        const uint32_t groups = p.tok / 16, half = (groups + 1) / 2;
        const uint32_t first = wg * half * 16, mine = wg ? groups - half : half;
        const uint32_t j = quad * 32 + lane;                    // weight column within the tile
        float acc[4][16];                                       // tokens first + 16 g + e
        uint32_t i = 0, filled = 0;                             // chunks, accumulators so far
        for (uint32_t u = u_begin; u < u_end;) {
            const uint32_t tile = u / p.chunks, c0 = u % p.chunks;
            const uint32_t c1 = min(p.chunks, c0 + (u_end - u));
#pragma unroll
            for (int g = 0; g < 4; g++)
#pragma unroll
                for (int e = 0; e < 16; e++) acc[g][e] = 0.f;
            for (uint32_t c = c0; c < c1; c++, i++) {
                if (group > 1 && c % group != group - 1 && c + 1 != c1) continue;            // the next chunk goes into the same accumulator
                const uint32_t sc = i % kScaleSlots, span = group > 1 ? min(c % group, c - c0) + 1 : 1;
                const uint32_t x = i + 1 - lane;                // lane 0: the accumulator, 1..span: scales of its chunks
                const uint8_t *scale = scale_ring + sc * scale_bytes + first * 4u;
                for (uint32_t h = FINE ? 0 : 3; h < 4; h++) {
                    const uint32_t b = filled & 1u;
                    mbar_wait_lanes(lane == 0 ? &sh.d_full[b] : &sh.sc_full[x % kScaleSlots], lane == 0 ? (filled >> 1) & 1u : (x / kScaleSlots) & 1u, lane <= span, &sh.failed, &g_split_error);
                    filled++;
                    __syncwarp();                               // tcgen05.ld is warp-collective
                    tc_fence_after();
                    const uint32_t from = tmem + lane_addr + b * kMaxTok + first;
                    if (FINE) {
                        if (mine > 0) drain_fine(from, scale, acc[0], acc[1]);
                    } else {
                        if (mine > 1) drain_part<0, 2>(from, scale, acc);
                        else if (mine > 0) drain_part<0, 1>(from, scale, acc);
                        if (mine > 3) drain_part<2, 2>(from, scale, acc);
                        else if (mine > 2) drain_part<2, 1>(from, scale, acc);
                    }
                    tc_fence_before();
                    __syncwarp();
                    if (lane == 0) mbar_arrive(&sh.d_empty[b]);
                }
                if (lane == 0)
                    for (uint32_t y = 0; y < span; y++) mbar_arrive(&sh.sc_empty[(i - y) % kScaleSlots]);
            }
            u += c1 - c0;
            if (FINE)                                           // before any part is added: the sum of two must not depend on which comes last
#pragma unroll
                for (int e = 0; e < 16; e++) acc[0][e] += acc[1][e];

            bool finish = true;
            if (c0 != 0 || c1 != p.chunks) {
                // part of a tile: leave the sums, the last CTA to get here adds all parts in the order of their chunks
                const uint32_t head = unit_owner(tile * p.chunks, p.units, gridDim.x), tail = unit_owner((tile + 1) * p.chunks - 1, p.units, gridDim.x);
                auto part_of = [&](uint32_t s) {
                    return p.partial + ((size_t)s * 2 + (unit_start(s, p.units, gridDim.x) <= tile * p.chunks ? 1 : 0)) * (kMaxTok * kCols) + first * kCols + j;
                };
                bool waiting = false;                           // the other one of two parts is there already: no need to leave this one
                if (tail == head + 1) {
                    if (tid == 128) {
                        uint32_t seen;
                        asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(seen) : "l"(p.counters + tile) : "memory");
                        sh.last = seen;
                    }
                    asm volatile("bar.sync 1, 256;" ::: "memory");
                    waiting = sh.last != 0;
                    asm volatile("bar.sync 1, 256;" ::: "memory");      // sh.last may be written again
                }
                if (waiting) {
                    add_part(part_of(blockIdx.x == head ? tail : head), mine, acc);
                } else {
                    float *part = part_of(blockIdx.x);
#pragma unroll
                    for (int g = 0; g < 4; g++)
                        if (g < (int)mine)
#pragma unroll
                            for (int e = 0; e < 16; e++) __stcg(part + (g * 16 + e) * kCols, acc[g][e]);
                    __threadfence();
                    asm volatile("bar.sync 1, 256;" ::: "memory");
                    if (tid == 128) {
                        sh.last = atomicAdd(p.counters + tile, 1u) == tail - head ? 1u : 0u;
                        __threadfence();
                    }
                    asm volatile("bar.sync 1, 256;" ::: "memory");
                    finish = sh.last != 0;
                    asm volatile("bar.sync 1, 256;" ::: "memory");      // sh.last may be written again
                    if (finish) {
                        __threadfence();
#pragma unroll
                        for (int g = 0; g < 4; g++)
#pragma unroll
                            for (int e = 0; e < 16; e++) acc[g][e] = 0.f;
                        if (FINE) {
                            for (uint32_t s = head; s <= tail && mine > 0; s++) {
                                const float *part = part_of(s);
                                float v[16];
#pragma unroll
                                for (int e = 0; e < 16; e++) v[e] = __ldcg(part + e * kCols);
#pragma unroll
                                for (int e = 0; e < 16; e++) add_exact(acc[0][e], acc[1][e], v[e]);
                            }
#pragma unroll
                            for (int e = 0; e < 16; e++) acc[0][e] += acc[1][e];
                        } else {
                            for (uint32_t s = head; s <= tail; s++) add_part(part_of(s), mine, acc);      // this CTA's own part among them
                        }
                    }
                }
            }
            if (finish) {
                const uint32_t col = (tile / p.m_tiles) * kCols + j, m0 = (tile % p.m_tiles) * p.tok + first;
                const uint32_t rows = col < p.n && m0 < p.m ? min(mine * 16u, p.m - m0) : 0u;
                const size_t o0 = (size_t)m0 * p.n + col;
                unsigned long long odd = 0;                     // sums that are not finite
#pragma unroll
                for (int g = 0; g < 4; g++) {
#pragma unroll
                    for (int e = 0; e < 16; e++)
                        if (!(fabsf(acc[g][e]) < __uint_as_float(0x7F800000u))) odd |= 1ull << (g * 16 + e);
                    if (p.addend) {
                        float v[16];
#pragma unroll
                        for (int e = 0; e < 16; e++) v[e] = g * 16 + e < (int)rows ? p.addend[o0 + (size_t)(g * 16 + e) * p.n] : 0.f;
#pragma unroll
                        for (int e = 0; e < 16; e++) acc[g][e] += v[e];
                    }
#pragma unroll
                    for (int e = 0; e < 16; e++)
                        if (g * 16 + e < (int)rows && !(odd >> (g * 16 + e) & 1u)) p.c[o0 + (size_t)(g * 16 + e) * p.n] = acc[g][e];
                }
                if (rows < 64) odd &= (1ull << rows) - 1;
                if (__any_sync(0xffffffffu, odd != 0)) {
                    p.odd[((size_t)tile * 8 + warp - 4) * 32 + lane] = odd;
                    if (lane == 0) p.odd_by[tile * 8 + warp - 4] = blockIdx.x + 1;
                    redo = true;
                }
            }
        }
    } else {
        asm volatile("setmaxnreg.dec.sync.aligned.u32 80;");
        // ---------------------------------------------------------------------- weights
        const uint32_t group = (warp - 12) >> 2, quad = warp & 3u;
        const uint32_t count = u_end - u_begin;
        const uint32_t mine = smem_u32(raw) + quad * 32u * raw_bytes(FMT);     // + place * kRawChunk
        uint32_t next = group, tile = (u_begin + group) / p.chunks, chunk = (u_begin + group) % p.chunks, col0 = (tile / p.m_tiles) * kCols + quad * 32;
        auto fetch = [&] {                                      // this group's next chunk, into the ring's place for it
            if (next < count) fetch_weights<FMT>(p, mine + (next % kRaw) * kRawChunk, col0, chunk, lane);
            asm volatile("cp.async.commit_group;" ::: "memory");
            next += 2;
            chunk += 2;
            if (chunk >= p.chunks) {
                tile += chunk / p.chunks;
                chunk %= p.chunks;
                col0 = (tile / p.m_tiles) * kCols + quad * 32;
            }
        };
        fetch();
        fetch();
        for (uint32_t i = group; i < count; i += 2) {
            asm volatile("cp.async.wait_group 1;" ::: "memory");
            __syncwarp();
            const uint8_t *src = raw + (i % kRaw) * kRawChunk + (quad * 32 + lane) * raw_bytes(FMT);
            mbar_wait(&sh.w_empty[group], ((i >> 1) & 1u) ^ 1u, &sh.failed, &g_split_error);
            __syncwarp();
            tc_fence_after();
            const uint32_t dst = tmem_w + ((quad * 32u) << 16) + group * 128u;
            if (FMT == MGQ_FMT_Q4) {
                const uint4 head = *reinterpret_cast<const uint4 *>(src);
                const uint32_t h[4] = {head.x, head.y, head.z, head.w};
#pragma unroll
                for (int blk = 0; blk < 4; blk++) {
                    uint32_t hi[16], lo[16];
                    const __half2 d = __half2half2(__low2half(as_half2(h[blk]))), m = __half2half2(__high2half(as_half2(h[blk])));
                    const float m32 = __high2float(as_half2(h[blk]));
                    const uint4 q4 = *reinterpret_cast<const uint4 *>(src + 16u + blk * 16u);
                    const uint32_t q[4] = {q4.x, q4.y, q4.z, q4.w};
#pragma unroll
                    for (int e = 0; e < 4; e++)
#pragma unroll
                        for (int s = 0; s < 4; s++)             // codes s and s + 4 of eight
                            split_affine(((q[e] >> (4 * s)) & 0x000F000Fu) | 0x64006400u, d, m, m32, hi[e * 4 + s], lo[e * 4 + s]);
                    tmem_st16(dst + blk * 16u, hi);
                    tmem_st16(dst + 64u + blk * 16u, lo);
                }
            } else {
                uint32_t words[36];                             // four blocks of 9
#pragma unroll
                for (int x = 0; x < 9; x++) {
                    const uint4 v = *reinterpret_cast<const uint4 *>(src + x * 16);
                    words[4 * x] = v.x; words[4 * x + 1] = v.y; words[4 * x + 2] = v.z; words[4 * x + 3] = v.w;
                }
                const __half2 offset = __float2half2_rn(1152.f);
#pragma unroll
                for (int blk = 0; blk < 4; blk++) {
                    uint32_t hi[16], lo[16];
                    const __half2 d = __half2half2(__low2half(as_half2(words[blk * 9])));
#pragma unroll
                    for (int e = 0; e < 8; e++) {
                        const uint32_t c = words[blk * 9 + 1 + e] ^ 0x80808080u;      // code + 128
                        split_codes(__byte_perm(c, 0x64646464u, 0x4140), offset, d, hi[e * 2], lo[e * 2]);
                        split_codes(__byte_perm(c, 0x64646464u, 0x4342), offset, d, hi[e * 2 + 1], lo[e * 2 + 1]);
                    }
                    tmem_st16(dst + blk * 16u, hi);
                    tmem_st16(dst + 64u + blk * 16u, lo);
                }
            }
            asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
            tc_fence_before();
            __syncwarp();                                       // every lane has read its bytes and stored its weights
            if (lane == 0) mbar_arrive(&sh.w_full[group]);
            fetch();
        }
        asm volatile("cp.async.wait_group 0;" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 1) {
        __syncwarp();
        tc_fence_after();
        tmem_free(tmem, 512);
    }
    // out here the call costs the drain no registers: 512 x 4096 x 12288 Q4 f32 131 us in a tight loop, 140 with the call at the drain's end
    if (redo) redo_odd<FMT>(p, PLANES == 1, u_begin, u_end, warp - 4, lane);
}

// ------------------------------------------------------------------------------------------ workspace

struct RelaxedCapture {                            // what this thread calls meanwhile is no part of any capture
    cudaStreamCaptureMode mode = cudaStreamCaptureModeRelaxed;
    RelaxedCapture() { cudaThreadExchangeStreamCaptureMode(&mode); }
    ~RelaxedCapture() { cudaThreadExchangeStreamCaptureMode(&mode); }
};

// Outside of captures: stream-ordered, so calls on different streams and threads never share a block; up to kKeep bytes stay with the pool
// between calls, the rest goes back to the device.
constexpr unsigned long long kKeep = 256ull << 20;
cudaMemPool_t g_pool[64] = {};
std::mutex g_pool_mu;

cudaMemPool_t workspace_pool(int dev)
{
    if (dev < 0 || dev >= 64) return nullptr;
    std::lock_guard<std::mutex> lock(g_pool_mu);
    if (!g_pool[dev]) {
        cudaMemPoolProps props{};
        props.allocType = cudaMemAllocationTypePinned;
        props.location.type = cudaMemLocationTypeDevice;
        props.location.id = dev;
        cudaMemPool_t pool = nullptr;
        RelaxedCapture relaxed;                    // another thread may be capturing
        unsigned long long keep = kKeep;
        if (cudaMemPoolCreate(&pool, &props) != cudaSuccess) { cudaGetLastError(); return nullptr; }
        if (cudaMemPoolSetAttribute(pool, cudaMemPoolAttrReleaseThreshold, &keep) != cudaSuccess) {
            cudaGetLastError();
            cudaMemPoolDestroy(pool);
            return nullptr;
        }
        g_pool[dev] = pool;
    }
    return g_pool[dev];
}

// Inside of a capture an allocation would become a node of the graph, and graphs with such nodes can be neither child graphs
// nor bodies of conditional nodes.  The workspace is then ordinary memory that the graph owns (a user object), shared by the calls that
// were captured on one stream, which run one after another; it goes back to the device with the first call, or the first session
// that ends, after the last executable of the graph is gone (a user object's destructor may not call CUDA itself).
struct CaptureSpace {
    unsigned long long capture;
    cudaStream_t stream;
    size_t bytes;
    void *ptr;
};
struct GraphSpaces {
    std::vector<CaptureSpace> captured;            // their graphs are alive
    std::vector<void *> orphans;                   // their graphs are gone
    std::mutex mu;
};
// Never destroyed: a destructor may run on a thread of the driver's while the process ends.
GraphSpaces &graph_spaces()
{
    static GraphSpaces *spaces = new GraphSpaces;
    return *spaces;
}

void CUDART_CB graph_gone(void *ptr)
{
    GraphSpaces &g = graph_spaces();
    std::lock_guard<std::mutex> lock(g.mu);
    g.captured.erase(std::remove_if(g.captured.begin(), g.captured.end(), [&](const CaptureSpace &c) { return c.ptr == ptr; }), g.captured.end());
    g.orphans.push_back(ptr);
}

// Null: no room.
void *capture_workspace(unsigned long long capture, cudaGraph_t graph, cudaStream_t stream, size_t bytes)
{
    GraphSpaces &g = graph_spaces();
    {
        std::lock_guard<std::mutex> lock(g.mu);
        for (const CaptureSpace &c : g.captured)
            if (c.capture == capture && c.stream == stream && c.bytes >= bytes) return c.ptr;
    }
    RelaxedCapture relaxed;
    void *ptr = nullptr;
    cudaUserObject_t owner = nullptr;
    if (cudaMalloc(&ptr, bytes) != cudaSuccess) { cudaGetLastError(); return nullptr; }
    if (cudaUserObjectCreate(&owner, ptr, graph_gone, 1, cudaUserObjectNoDestructorSync) != cudaSuccess) {
        cudaGetLastError();
        cudaFree(ptr);
        return nullptr;
    }
    {
        std::lock_guard<std::mutex> lock(g.mu);
        g.captured.push_back({capture, stream, bytes, ptr});
    }
    if (cudaGraphRetainUserObject(graph, owner, 1, cudaGraphUserObjectMove) != cudaSuccess) {
        cudaGetLastError();
        cudaUserObjectRelease(owner, 1);
        return nullptr;
    }
    return ptr;
}

template <int FMT, int PLANES, bool FINE = false>
int launch_split(const SplitParams &p, uint32_t ctas, cudaStream_t stream)
{
    const size_t smem = 1024 + (size_t)kSlots * p.tok * 128 + (size_t)kScaleSlots * p.tok * 4 + (size_t)kRaw * kCols * raw_bytes(FMT);
    if (int rc = allow_smem(gemm_split_kernel<FMT, PLANES, FINE>, smem)) return rc;
    return launch(gemm_split_kernel<FMT, PLANES, FINE>, dim3(ctas), dim3(kSplitThreads), smem, stream, p);
}

}  // namespace

void release_graph_workspaces()
{
    std::vector<void *> gone;
    {
        std::lock_guard<std::mutex> lock(graph_spaces().mu);
        gone.swap(graph_spaces().orphans);
    }
    if (gone.empty()) return;
    RelaxedCapture relaxed;
    for (void *p : gone) cudaFree(p);
}

// When there is no room for the workspace, nothing is launched for the rows from *done on.
int launch_gemm_split(int fmt, const void *a, int a_dtype, const void *w, const float *addend, float *c,
                      uint32_t m, uint32_t k, uint32_t n, void *stream_v, uint32_t *done)
{
    cudaStream_t stream = static_cast<cudaStream_t>(stream_v);
    int dev = 0, sms = 0;
    MGQ_CUDA(cudaGetDevice(&dev));
    MGQ_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
    *done = 0;
    cudaStreamCaptureStatus capturing = cudaStreamCaptureStatusNone;
    unsigned long long capture = 0;
    cudaGraph_t graph = nullptr;
    MGQ_CUDA(cudaStreamGetCaptureInfo(stream, &capturing, &capture, &graph));
    const bool captured = capturing == cudaStreamCaptureStatusActive;
    if (!captured) release_graph_workspaces();
    cudaMemPool_t pool = captured ? nullptr : workspace_pool(dev);
    if (!captured && !pool) return MGQ_OK;
    const bool bf16 = a_dtype == MGQ_A_BF16, q4 = fmt == MGQ_FMT_Q4;
    const uint32_t planes = bf16 ? 1 : 2;
    const size_t elem = bf16 ? 2 : 4;
    uint32_t pass = kPassElems / k / kMaxTok * kMaxTok;
    if (pass < kMaxTok) pass = kMaxTok;
    for (uint32_t r0 = 0; r0 < m; r0 += *done - r0) {
        SplitParams p{};
        p.m = m - r0 < pass ? m - r0 : pass;
        p.k = k; p.n = n; p.bpc = k / 32;
        p.num_blocks = (unsigned long long)p.bpc * n;
        p.w = static_cast<const uint8_t *>(w);
        p.a = static_cast<const uint8_t *>(a) + (size_t)r0 * k * elem;
        p.addend = addend ? addend + (size_t)r0 * n : nullptr;
        p.c = c + (size_t)r0 * n;
        // tiles of equal numbers of tokens, in steps of the MMA's 16
        p.m_tiles = (p.m + kMaxTok - 1) / kMaxTok;
        p.tok = ((p.m + p.m_tiles - 1) / p.m_tiles + 15) / 16 * 16;
        p.m_tiles = (p.m + p.tok - 1) / p.tok;
        p.chunks = (k + kChunk - 1) / kChunk;
        const unsigned long long units = (unsigned long long)p.m_tiles * ((n + kCols - 1) / kCols) * p.chunks;
        if (units >= (1ull << 31)) return MGQ_OK;
        p.tiles = (uint32_t)(units / p.chunks);
        p.units = (uint32_t)units;
        // Q8: whole 16-byte pieces of 4 blocks; Q4: nibbles behind num_blocks header words
        p.wide = q4 ? p.num_blocks % 4 == 0 : p.bpc % 4 == 0;
        const bool fine = !q4 && !bf16 && m <= MGQ_GEMV_MAX_M && !gemv_streamable(fmt, a, k, n) && !gemv_mma_eligible(m, k, n, a, w);
        const uint32_t ctas = p.units / 2 < 1 ? 1 : p.units / 2 < (uint32_t)sms ? p.units / 2 : (uint32_t)sms;

        const size_t plane_bytes = (size_t)p.m_tiles * p.chunks * 2 * planes * p.tok * 128;
        const size_t scale_bytes = ((size_t)p.m_tiles * p.chunks * p.tok * 4 + 255) / 256 * 256;
        const size_t part_bytes = (size_t)ctas * 2 * kMaxTok * kCols * 4, odd_bytes = (size_t)p.tiles * 256 * 8, words = (size_t)p.tiles * 9;
        const size_t all_bytes = plane_bytes + scale_bytes + part_bytes + odd_bytes + words * 4;
        uint8_t *ws = nullptr;
        if (captured) ws = static_cast<uint8_t *>(capture_workspace(capture, graph, stream, all_bytes));
        else if (cudaMallocFromPoolAsync(reinterpret_cast<void **>(&ws), all_bytes, pool, stream) != cudaSuccess) cudaGetLastError(), ws = nullptr;
        if (!ws) return MGQ_OK;
        float *scales = reinterpret_cast<float *>(ws + plane_bytes);
        p.planes = ws;
        p.scales = scales;
        p.partial = reinterpret_cast<float *>(ws + plane_bytes + scale_bytes);
        p.odd = reinterpret_cast<unsigned long long *>(ws + plane_bytes + scale_bytes + part_bytes);
        p.counters = reinterpret_cast<unsigned int *>(ws + plane_bytes + scale_bytes + part_bytes + odd_bytes);
        p.odd_by = p.counters + p.tiles;
        const bool vec = reinterpret_cast<uintptr_t>(p.a) % 16 == 0;
        const unsigned long long warps = (unsigned long long)p.m * ((p.chunks + group_of(planes, k) - 1) / group_of(planes, k));
        split_rows_kernel<<<(uint32_t)((warps + 7) / 8), 256, 0, stream>>>(p.a, bf16, vec, ws, scales, p.counters, (uint32_t)words, p.m, k, p.tok, p.chunks, planes, q4);
        int rc = cuda_check((int)cudaGetLastError(), "split_rows_kernel", __FILE__, __LINE__);
        if (rc == MGQ_OK)
            rc = q4 ? (bf16 ? launch_split<MGQ_FMT_Q4, 1>(p, ctas, stream) : launch_split<MGQ_FMT_Q4, 2>(p, ctas, stream))
                    : (bf16 ? launch_split<MGQ_FMT_Q8, 1>(p, ctas, stream) : fine ? launch_split<MGQ_FMT_Q8, 2, true>(p, ctas, stream) : launch_split<MGQ_FMT_Q8, 2>(p, ctas, stream));
        const int freed = captured ? MGQ_OK : cuda_check((int)cudaFreeAsync(ws, stream), "cudaFreeAsync", __FILE__, __LINE__);
        if (rc != MGQ_OK) return rc;
        if (freed != MGQ_OK) return freed;
        *done = r0 + p.m;
    }
    return MGQ_OK;
}

int tc_device_status()
{
    unsigned int err = 0;
    MGQ_CUDA(cudaMemcpyFromSymbol(&err, g_split_error, sizeof err));
    if (err) {
        const unsigned int zero = 0;
        MGQ_CUDA(cudaMemcpyToSymbol(g_split_error, &zero, sizeof zero));
        return fail(MGQ_ERR_TIMEOUT, "a bounded wait inside the tensor-core GEMM ran out");
    }
    return linear_tc_status();
}

}  // namespace mgq
