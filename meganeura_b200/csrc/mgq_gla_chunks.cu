// Recurrences over many tokens in chunks of 16 on the tensor cores: gated linear attention, RWKV-style time mixing, mLSTM.
//
// Inside a chunk, with a_t the decays per key channel, L_t = a_1 .. a_t, G_s = a_(s+1) .. a_16 and the
// state S in front of the chunk:
//     o_t = S^T (L_t q_t) + sum_(s <= t) A_ts v_s,      A_ts = sum_d q_t k_s a_(s+1) .. a_t
//     S'  = diag(L_16) S + sum_s (G_s k_s) v_s^T
// Only products of decays appear, never a quotient, so nothing overflows however strong the decay is.
// Time mixing reads the state before a token's decay and update: L_t = a_1 .. a_(t-1), A_ts = sum_d q_t k_s a_(s+1) .. a_(t-1)
// for s < t and A_tt = sum_d q_t u k_t.  mLSTM: with the maxima m_t (a scan over the gates, mlstm_gates_kernel) all channels of a head decay by
// exp(f_t + m_(t-1) - m_t), keys count exp(i_t - m_t), and the normaliser is one more value column that holds ones.
//   gla_prepare_kernel  CTA = chunk x head: the decays from their low-rank projection, then A, L q, G k and L_16
//                       into a record that the next kernel copies as it is
//   gla_chunks_kernel   a warp keeps S^T for 16 value columns and all keys in registers, as f32 accumulators of
//                       mma.sync whose layout is also that of the products' left operand, and walks the chunks;
//                       the records come through a ring of cp.async copies
// State, decays and sums are f32.  Where the state is read it enters as the sum of three bf16, i.e. with all its
// bits; the decayed queries and keys, A and the values as sums of two, three products each: 16 to 17 significant bits
// of numbers whose factors are projections, with the range of f32.  Time mixing and mLSTM take sums of three everywhere and six of
// the nine products (what is left out is below 2^-26 of a product).  The tensor cores truncate what they accumulate, so there every
// block of 16 keys is summed by itself and added in f32.  Against 64 bits, this and token by token: time mixing 64 x 64 with
// decays around 0.95 1.24e-7 / 1.21e-7, 0.999 3.7e-7 / 4.5e-7, mLSTM 128 x 256 6.3e-7 / 8.2e-7 (all blocks in one
// accumulator: 4.4e-7, 6.9e-7, 1.8e-6).  A long portion is cut into segments:
// a first pass leaves the end state of every segment but the last, each started from nothing, gla_combine_kernel
// turns them into the segments' start states, and a second pass runs all segments with outputs.
// 2048 tokens, all launches: mLSTM 8 x 128 x 256 190 us against 311 token by token, time mixing 32 x 64 x 64 about 100 against 138.
#include <algorithm>

#include "mgq_mixer.cuh"

namespace mgq {
namespace {

constexpr uint32_t kChunk = 16, kStages = 3, kMaxWarps = 8, kMaxSegs = 16;
// Time mixing and mLSTM take longer portions in pieces, whose records (31 KB per token with 32 heads of 64 channels) then share 64 MB; a
// piece fills the chip.
constexpr uint32_t kPieceRows = 2048;

enum { kGla = 0, kWkv = 1, kMlstm = 2 };
__host__ __device__ constexpr int parts_of(int mode) { return mode == kGla ? 2 : 3; }

// Record of a chunk of a head: G k (parts, the highest first), L_16, L q (parts), A (parts); rows padded for ldmatrix.
template <int D, int PARTS> struct Record {
    static constexpr uint32_t pitch = D + 8, matrix = kChunk * pitch * 2;
    static constexpr uint32_t lam = PARTS * matrix, ql = lam + D * 4, a = ql + PARTS * matrix, bytes = a + PARTS * kChunk * kChunk * 2;
    static constexpr uint32_t state_part = ql;           // what a pass without outputs needs
};

struct Chunks {
    const float *q, *k, *v, *w;                          // w: decays, or null: from d
    Decay d;
    const float *u;                                      // time mixing: bonus [heads, dim]
    const float *gi, *gf;                                // mLSTM: gate pre-activations [rows, heads]
    float4 *gates;                                       // mLSTM: decay, key weight, exp(-m) [heads][rows]
    float *den;                                          // mLSTM: normaliser . q [rows, heads]
    float *shift_state;
    float *o, *state, *segments, *products;              // products: of a segment's decays, [segment][heads][D]
    uint8_t *records;
    uint32_t rows, heads, dim, vdim, chunks;
    uint32_t cols;                                       // value columns with the normaliser's
    uint32_t blocks, norm_pitch, shift_width;            // mLSTM: copies of n and m behind the state, floats from one to the next
    uint32_t seg_len, segs, states_only;                 // chunks per segment; the first pass leaves end states only
    float qscale, cap;
};

// Normaliser of a head (n, then m), copy b: behind the heads' states.
__device__ __forceinline__ float *normalizer(const Chunks &p, uint32_t head, uint32_t b)
{
    const uint32_t kp = (p.dim + 3u) & ~3u;
    return p.state + (size_t)p.heads * p.vdim * kp + (size_t)(head * p.blocks + b) * p.norm_pitch;
}

__device__ __forceinline__ void split2(float x, float y, uint32_t &hi, uint32_t &lo)
{
    const __nv_bfloat162 h = __floats2bfloat162_rn(x, y);
    const float2 f = __bfloat1622float2(h);
    const __nv_bfloat162 l = __floats2bfloat162_rn(x - f.x, y - f.y);
    hi = *reinterpret_cast<const uint32_t *>(&h);
    lo = *reinterpret_cast<const uint32_t *>(&l);
}
__device__ __forceinline__ void split3(float x, float y, uint32_t &hi, uint32_t &mid, uint32_t &lo)
{
    const __nv_bfloat162 h = __floats2bfloat162_rn(x, y);
    const float2 f = __bfloat1622float2(h);
    hi = *reinterpret_cast<const uint32_t *>(&h);
    split2(x - f.x, y - f.y, mid, lo);
}

// The parts of two neighbours, the highest first.
template <int PARTS>
__device__ __forceinline__ void split_parts(float x, float y, uint32_t (&part)[3])
{
    if (PARTS == 3) split3(x, y, part[0], part[1], part[2]);
    else            split2(x, y, part[0], part[1]);
}

// m_t = max(f_t + m_(t-1), i_t) is a scan of (sum of f, max) pairs.  CTA = head; 1024 tokens at a time.
__global__ void __launch_bounds__(1024) mlstm_gates_kernel(const __grid_constant__ Chunks p)
{
    __shared__ float s_f[32], s_m[32], s_last;
    const uint32_t t = threadIdx.x, lane = t & 31u, warp = t >> 5, head = blockIdx.x, kp = (p.dim + 3u) & ~3u;
    pdl_launch_dependents();
    pdl_wait();
    float m = normalizer(p, head, 0)[kp];
    __syncthreads();                                     // read by all before it is replaced below
    for (uint32_t r0 = 0; r0 < p.rows; r0 += 1024) {
        const uint32_t row = r0 + t;
        const bool in = row < p.rows;
        const size_t at = (size_t)row * p.heads + head;
        const float li = in ? p.cap * tanhf(p.gi[at] / p.cap) : -INFINITY, lf = in ? log_sigmoid(p.cap * tanhf(p.gf[at] / p.cap)) : 0.f;
        float F = lf, M = li;
#pragma unroll
        for (int off = 1; off < 32; off <<= 1) {
            const float Fp = __shfl_up_sync(0xffffffffu, F, off), Mp = __shfl_up_sync(0xffffffffu, M, off);
            if (lane >= (uint32_t)off) { M = fmaxf(M, F + Mp); F += Fp; }
        }
        if (lane == 31) { s_f[warp] = F; s_m[warp] = M; }
        __syncthreads();
        float before = m;                                // m in front of this warp
        for (uint32_t w = 0; w < warp; w++) before = fmaxf(s_f[w] + before, s_m[w]);
        const float mt = fmaxf(F + before, M);
        float prev = __shfl_up_sync(0xffffffffu, mt, 1);
        if (lane == 0) prev = before;
        if (in) p.gates[(size_t)head * p.rows + row] = make_float4(expf(lf + (prev - mt)), expf(li - mt), expf(-mt), 0.f);
        if (t == 1023) s_last = mt;                      // tokens beyond the portion leave it as it is
        __syncthreads();
        m = s_last;
        __syncthreads();
    }
    if (t < p.blocks) normalizer(p, head, t)[kp] = m;
}

template <int D, int MODE>
__global__ void __launch_bounds__(256) gla_prepare_kernel(const __grid_constant__ Chunks p)
{
    constexpr uint32_t P = D + 4, SLICES = D / 4 < 16 ? D / 4 : 16;
    constexpr int PARTS = parts_of(MODE);
    using R = Record<D, PARTS>;
    extern __shared__ __align__(16) float smem[];        // q, k, w [16][P], partial sums of A [SLICES][16 t][16 s]
    float *sq = smem, *sk = sq + kChunk * P, *sw = sk + kChunk * P, *sa = sw + kChunk * P;
    const uint32_t t = threadIdx.x, chunk = blockIdx.x, head = blockIdx.y, row0 = chunk * kChunk, kpitch = p.heads * p.dim;
    pdl_launch_dependents();
    pdl_wait();
    if (MODE == kWkv && p.shift_state && chunk == 0)     // what token shift has left for the next step
        for (uint32_t j = head * 256 + t; j < p.shift_width; j += p.heads * 256) p.shift_state[j] = p.shift_state[p.shift_width + j];
    const float4 *gates = MODE == kMlstm ? p.gates + (size_t)head * p.rows + row0 : nullptr;
    // beyond the portion and beyond the head's channels: nothing decays and nothing is added
    if (p.dim % 4 == 0) {
#pragma unroll
        for (uint32_t j = 0; j < (kChunk * D / 4 + 255) / 256; j++) {
            const uint32_t i = t + 256 * j, r = i / (D / 4), d = i % (D / 4) * 4;
            if (i >= kChunk * D / 4) break;
            const bool in = row0 + r < p.rows && d < p.dim;
            const size_t at = (size_t)(row0 + r) * kpitch + head * p.dim + d;
            float4 q = make_float4(0.f, 0.f, 0.f, 0.f), k = q;
            if (in) { q = *reinterpret_cast<const float4 *>(p.q + at); k = *reinterpret_cast<const float4 *>(p.k + at); }
            if (MODE == kMlstm && in) {
                const float b = gates[r].y;
                k.x *= b; k.y *= b; k.z *= b; k.w *= b;
            }
            *reinterpret_cast<float4 *>(sq + r * P + d) = make_float4(q.x * p.qscale, q.y * p.qscale, q.z * p.qscale, q.w * p.qscale);
            *reinterpret_cast<float4 *>(sk + r * P + d) = k;
        }
    } else {
#pragma unroll 4
        for (uint32_t i = t; i < kChunk * D; i += 256) {
            const uint32_t r = i / D, d = i % D;
            const bool in = row0 + r < p.rows && d < p.dim;
            const size_t at = (size_t)(row0 + r) * kpitch + head * p.dim + d;
            sq[r * P + d] = in ? p.q[at] * p.qscale : 0.f;
            sk[r * P + d] = in ? p.k[at] * (MODE == kMlstm ? gates[r].y : 1.f) : 0.f;
        }
    }
    if (MODE == kMlstm) {
        for (uint32_t i = t; i < kChunk * D; i += 256) {
            const uint32_t r = i / D, d = i % D;
            sw[r * P + d] = row0 + r < p.rows ? gates[r].x : 1.f;
        }
    } else if (p.w) {
#pragma unroll 4
        for (uint32_t i = t; i < kChunk * D; i += 256) {
            const uint32_t r = i / D, d = i % D;
            const bool in = row0 + r < p.rows && d < p.dim;
            sw[r * P + d] = in ? p.w[(size_t)(row0 + r) * kpitch + head * p.dim + d] : 1.f;
        }
    } else {
        // thread = channel x a share of the tokens; the low-rank inputs lie where the partial sums of A go later
        constexpr uint32_t GROUPS = 256 / D, PER = kChunk / GROUPS;
        const uint32_t d = t % D, r0 = t / D * PER, ranks = p.d.rank;
        float z[PER];
        for (uint32_t j0 = 0; j0 < ranks; j0 += 128) {
            const uint32_t nj = min(128u, ranks - j0);
            __syncthreads();
            for (uint32_t i = t; i < kChunk * nj; i += 256) {
                const uint32_t r = i / nj, j = i % nj;
                sa[r * 128 + j] = row0 + r < p.rows ? decay_input(p.d.low[(size_t)(row0 + r) * ranks + j0 + j], p.d.inv_tau) : 0.f;
            }
            __syncthreads();
            if (d < p.dim) {
                if (j0 == 0)
#pragma unroll
                    for (int i = 0; i < (int)PER; i++) z[i] = p.d.w0[head * p.dim + d];
                const __nv_bfloat16 *w2 = static_cast<const __nv_bfloat16 *>(p.d.w2) + (size_t)(head * p.dim + d) * ranks + j0;
                if (ranks % 8 == 0 && reinterpret_cast<uintptr_t>(p.d.w2) % 16 == 0) {      // eight ranks per load: 288 -> 89 us for the whole kernel with 32 x 64 channels, rank 64, 2048 tokens
#pragma unroll 2
                    for (uint32_t j = 0; j < nj; j += 8) {
                        float x[8];
                        unpack8(__ldg(reinterpret_cast<const uint4 *>(w2 + j)), x);
#pragma unroll
                        for (int i = 0; i < (int)PER; i++) {
                            const float4 a = *reinterpret_cast<const float4 *>(sa + (r0 + i) * 128 + j), b = *reinterpret_cast<const float4 *>(sa + (r0 + i) * 128 + j + 4);
                            z[i] = fmaf(x[3], a.w, fmaf(x[2], a.z, fmaf(x[1], a.y, fmaf(x[0], a.x, z[i]))));
                            z[i] = fmaf(x[7], b.w, fmaf(x[6], b.z, fmaf(x[5], b.y, fmaf(x[4], b.x, z[i]))));
                        }
                    }
                } else {
#pragma unroll 8
                    for (uint32_t j = 0; j < nj; j++) {
                        const float x = __bfloat162float(w2[j]);
#pragma unroll
                        for (int i = 0; i < (int)PER; i++) z[i] = fmaf(x, sa[(r0 + i) * 128 + j], z[i]);
                    }
                }
            }
        }
#pragma unroll
        for (int i = 0; i < (int)PER; i++) sw[(r0 + i) * P + d] = d < p.dim && row0 + r0 + i < p.rows ? decay_value(z[i], p.d.inv_tau) : 1.f;
    }
    __syncthreads();
    uint8_t *rec = p.records + ((size_t)head * p.chunks + chunk) * R::bytes;
    // A: thread = key token s x a share of the channels; the key decays from token to token
    {
        const uint32_t s = t & 15u, slice = t >> 4;
        float acc[kChunk];
#pragma unroll
        for (int i = 0; i < (int)kChunk; i++) acc[i] = 0.f;
        for (uint32_t d = slice * 4; d < (uint32_t)D; d += 64) {
            const float4 k4 = *reinterpret_cast<const float4 *>(sk + s * P + d);
            float4 u4 = make_float4(0.f, 0.f, 0.f, 0.f);
            if (MODE == kWkv) {
                const float *u = p.u + head * p.dim + d;
                u4 = make_float4(d < p.dim ? u[0] * k4.x : 0.f, d + 1 < p.dim ? u[1] * k4.y : 0.f, d + 2 < p.dim ? u[2] * k4.z : 0.f, d + 3 < p.dim ? u[3] * k4.w : 0.f);
            }
            float4 r = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
            for (int i = 0; i < (int)kChunk; i++) {
                const float4 w4 = *reinterpret_cast<const float4 *>(sw + i * P + d), q4 = *reinterpret_cast<const float4 *>(sq + i * P + d);
                const bool own = (uint32_t)i == s;
                if (MODE == kWkv) {                      // the state before this token, and the bonus
                    const float4 x = own ? u4 : r;
                    acc[i] = fmaf(x.x, q4.x, acc[i]); acc[i] = fmaf(x.y, q4.y, acc[i]); acc[i] = fmaf(x.z, q4.z, acc[i]); acc[i] = fmaf(x.w, q4.w, acc[i]);
                }
                r.x = own ? k4.x : r.x * w4.x; r.y = own ? k4.y : r.y * w4.y; r.z = own ? k4.z : r.z * w4.z; r.w = own ? k4.w : r.w * w4.w;
                if (MODE != kWkv) {
                    acc[i] = fmaf(r.x, q4.x, acc[i]); acc[i] = fmaf(r.y, q4.y, acc[i]); acc[i] = fmaf(r.z, q4.z, acc[i]); acc[i] = fmaf(r.w, q4.w, acc[i]);
                }
            }
        }
        if (slice < SLICES)
#pragma unroll
            for (int i = 0; i < (int)kChunk; i++) sa[(slice * kChunk + i) * kChunk + s] = acc[i];
    }
    // L q by the first half of the threads, G k and L_16 by the second, two channels each
    {
        const uint32_t d = (t & 127u) * 2;
        if (d < (uint32_t)D) {
            float2 f = make_float2(1.f, 1.f);
            if (t < 128) {
#pragma unroll
                for (int i = 0; i < (int)kChunk; i++) {
                    const float2 w2 = *reinterpret_cast<const float2 *>(sw + i * P + d), x = *reinterpret_cast<const float2 *>(sq + i * P + d);
                    if (MODE != kWkv) { f.x *= w2.x; f.y *= w2.y; }
                    uint32_t part[3];
                    split_parts<PARTS>(x.x * f.x, x.y * f.y, part);
#pragma unroll
                    for (int h = 0; h < PARTS; h++) *reinterpret_cast<uint32_t *>(rec + R::ql + h * R::matrix + (i * R::pitch + d) * 2) = part[h];
                    if (MODE == kWkv) { f.x *= w2.x; f.y *= w2.y; }
                }
            } else {
#pragma unroll
                for (int i = (int)kChunk - 1; i >= 0; i--) {
                    const float2 w2 = *reinterpret_cast<const float2 *>(sw + i * P + d), x = *reinterpret_cast<const float2 *>(sk + i * P + d);
                    uint32_t part[3];
                    split_parts<PARTS>(x.x * f.x, x.y * f.y, part);
#pragma unroll
                    for (int h = 0; h < PARTS; h++) *reinterpret_cast<uint32_t *>(rec + h * R::matrix + (i * R::pitch + d) * 2) = part[h];
                    f.x *= w2.x; f.y *= w2.y;
                }
                *reinterpret_cast<float2 *>(rec + R::lam + d * 4) = f;
            }
        }
    }
    __syncthreads();
    if (t < 128) {                                       // two neighbouring keys of one query
        float2 sum[4] = {};                              // three parts: four short sums round less than one
#pragma unroll
        for (int i = 0; i < (int)SLICES; i++) {
            const float2 y = *reinterpret_cast<const float2 *>(sa + i * kChunk * kChunk + 2 * t);
            float2 &x = sum[PARTS == 3 ? i % 4 : 0];
            x.x += y.x; x.y += y.y;
        }
        uint32_t part[3];
        split_parts<PARTS>((sum[0].x + sum[1].x) + (sum[2].x + sum[3].x), (sum[0].y + sum[1].y) + (sum[2].y + sum[3].y), part);
#pragma unroll
        for (int h = 0; h < PARTS; h++) *reinterpret_cast<uint32_t *>(rec + R::a + h * kChunk * kChunk * 2 + 4 * t) = part[h];
    }
}

__device__ __forceinline__ uint32_t smem_addr(const void *p) { return (uint32_t)__cvta_generic_to_shared(p); }
__device__ __forceinline__ void ldmatrix4(uint32_t addr, uint32_t (&r)[4])
{
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0, %1, %2, %3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr) : "memory");
}
__device__ __forceinline__ void ldmatrix4_t(uint32_t addr, uint32_t (&r)[4])
{
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0, %1, %2, %3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr) : "memory");
}
__device__ __forceinline__ void mma16816(float (&c)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1)
{
    asm("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
                 : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3]) : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
// CTA = head (x) x value columns (y), 16 per warp, x segment (z).
template <int D, int MODE>
__global__ void __launch_bounds__(256, 1) gla_chunks_kernel(const __grid_constant__ Chunks p)
{
    constexpr int PARTS = parts_of(MODE);
    using R = Record<D, PARTS>;
    extern __shared__ __align__(16) uint8_t ring[];      // kStages records
    __shared__ float s_f[D];                             // product of the decays so far (first pass)
    const uint32_t t = threadIdx.x, threads = blockDim.x, lane = t & 31u, warp = t >> 5, g = lane >> 2, tq = lane & 3u;
    const uint32_t head = blockIdx.x, v0 = (blockIdx.y * (threads >> 5) + warp) * 16, kp = (p.dim + 3u) & ~3u, vpitch = p.heads * p.vdim;
    const uint32_t seg = blockIdx.z, c0 = seg * p.seg_len, c1 = min(c0 + p.seg_len, p.chunks);
    const bool outputs = !p.states_only;
    const uint32_t vr[2] = {v0 + g, v0 + g + 8};         // this thread's value columns
    const bool live[2] = {vr[0] < p.cols, vr[1] < p.cols};
    const bool ones[2] = {MODE == kMlstm && vr[0] == p.vdim, MODE == kMlstm && vr[1] == p.vdim};      // the normaliser's column
    pdl_launch_dependents();
    pdl_wait();
    const uint8_t *records = p.records + (size_t)head * p.chunks * R::bytes;
    auto stage = [&](uint32_t c) {                       // always one commit
        if (c < c1) {
            const uint8_t *src = records + (size_t)c * R::bytes;
            const uint32_t dst = smem_addr(ring + (c - c0) % kStages * R::bytes), bytes = outputs ? R::bytes : R::state_part;
            for (uint32_t i = t * 16; i < bytes; i += threads * 16)
                asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(dst + i), "l"(src + i) : "memory");
        }
        asm volatile("cp.async.commit_group;\n" ::: "memory");
    };
    stage(c0);
    stage(c0 + 1);
    const float *vbase = p.v + head * p.vdim;
    float v[8];
    auto load_values = [&](uint32_t c) {                 // [token pair low / high half][column], two tokens each
#pragma unroll
        for (int h = 0; h < 2; h++)
#pragma unroll
            for (int i = 0; i < 2; i++)
#pragma unroll
                for (int e = 0; e < 2; e++) {
                    const uint32_t row = c * kChunk + h * 8 + tq * 2 + e;
                    v[(h * 2 + i) * 2 + e] = c < c1 && row < p.rows && live[i] ? ones[i] ? 1.f : vbase[(size_t)row * vpitch + vr[i]] : 0.f;
                }
    };
    load_values(c0);

    // S^T: rows are value columns, columns are keys
    float S[D / 8][4];
#pragma unroll
    for (int n = 0; n < D / 8; n++)
#pragma unroll
        for (int e = 0; e < 4; e++) S[n][e] = 0.f;
    if (seg == 0 || outputs) {                           // start state: the sequence's, or what the combination left
        const bool own = seg == 0 && (p.segs == 1 || !outputs);
        const uint32_t slot = seg == 0 ? p.segs - 1 : seg - 1, pitch = own ? kp : D;
        const float *start = own ? p.state + (size_t)head * p.vdim * kp : p.segments + ((size_t)slot * p.heads + head) * p.cols * D;
#pragma unroll
        for (int n = 0; n < D / 8; n++)
#pragma unroll
            for (int i = 0; i < 2; i++) {
                const uint32_t d = n * 8 + tq * 2;
                if (d < pitch && live[i]) {
                    const float2 x = *reinterpret_cast<const float2 *>((own && ones[i] ? normalizer(p, head, 0) : start + (size_t)vr[i] * pitch) + d);
                    S[n][2 * i] = x.x; S[n][2 * i + 1] = x.y;
                }
            }
    }

    const bool product = !outputs && blockIdx.y == 0;
    if (product)
        for (uint32_t d = t; d < (uint32_t)D; d += threads) s_f[d] = 1.f;      // a thread only ever touches its own entries
    const uint32_t q_off = R::ql + (((lane & 7u) + (lane >> 4) * 8) * R::pitch + ((lane >> 3) & 1u) * 8) * 2;
    const uint32_t k_off = (((lane & 7u) + ((lane >> 3) & 1u) * 8) * R::pitch + (lane >> 4) * 8) * 2;
    for (uint32_t c = c0; c < c1; c++) {
        asm volatile("cp.async.wait_group 1;\n" ::: "memory");
        __syncthreads();                                 // everyone's copies, and everyone has left the buffer that is filled now
        stage(c + 2);
        const uint8_t *rec = ring + (c - c0) % kStages * R::bytes;
        const uint32_t base = smem_addr(rec);
        uint32_t vp[3][4];                               // V^T as left operand: rows value columns, columns tokens
#pragma unroll
        for (int i = 0; i < 4; i++) {
            uint32_t part[3];
            split_parts<PARTS>(v[2 * i], v[2 * i + 1], part);
#pragma unroll
            for (int h = 0; h < PARTS; h++) vp[h][i] = part[h];
        }
        load_values(c + 1);
        float o[2][4] = {{0.f, 0.f, 0.f, 0.f}, {0.f, 0.f, 0.f, 0.f}};          // o^T: rows value columns, columns tokens
#pragma unroll
        for (int j = 0; j < D / 16; j++) {
            uint32_t sp[3][4], qp[3][4], kq[3][4];
            if (outputs) {
#pragma unroll
                for (int i = 0; i < 4; i++) split3(S[2 * j + i / 2][i % 2 * 2], S[2 * j + i / 2][i % 2 * 2 + 1], sp[0][i], sp[1][i], sp[2][i]);
#pragma unroll
                for (int h = 0; h < PARTS; h++) ldmatrix4(base + q_off + h * R::matrix + j * 32, qp[h]);
            }
#pragma unroll
            for (int h = 0; h < PARTS; h++) ldmatrix4_t(base + k_off + h * R::matrix + j * 32, kq[h]);
            float add[2][4] = {}, out[2][4] = {};        // three parts: each block of 16 keys by itself, added in f32
            float f[2][2];                               // the chunk's decay of this thread's keys
#pragma unroll
            for (int n = 0; n < 2; n++) {
                const float2 l = *reinterpret_cast<const float2 *>(rec + R::lam + (j * 16 + n * 8 + tq * 2) * 4);
                f[n][0] = l.x; f[n][1] = l.y;
                if (PARTS == 2)
#pragma unroll
                    for (int e = 0; e < 4; e++) S[2 * j + n][e] *= f[n][e & 1];
            }
            // small products first (the two factors' parts count 2^-8 each); the sums are independent of each other
#pragma unroll
            for (int order = 2; order >= 0; order--)
#pragma unroll
                for (int x = 0; x <= order; x++) {       // part x of the left operand, order - x of the right
                    const int y = order - x;
                    if (y >= PARTS) continue;
                    if (outputs) {
                        mma16816(PARTS == 3 ? out[0] : o[0], sp[x], qp[y][0], qp[y][1]);
                        mma16816(PARTS == 3 ? out[1] : o[1], sp[x], qp[y][2], qp[y][3]);
                    }
                    if (PARTS == 2 && (order == 2 || x >= PARTS)) continue;
                    mma16816(PARTS == 3 ? add[0] : S[2 * j], vp[x], kq[y][0], kq[y][1]);
                    mma16816(PARTS == 3 ? add[1] : S[2 * j + 1], vp[x], kq[y][2], kq[y][3]);
                }
            if (PARTS == 3)
#pragma unroll
                for (int n = 0; n < 2; n++)
#pragma unroll
                    for (int e = 0; e < 4; e++) {
                        S[2 * j + n][e] = fmaf(S[2 * j + n][e], f[n][e & 1], add[n][e]);
                        o[n][e] += out[n][e];
                    }
        }
        if (product)
            for (uint32_t d = t; d < (uint32_t)D; d += threads) s_f[d] *= *reinterpret_cast<const float *>(rec + R::lam + d * 4);
        if (!outputs) continue;
#pragma unroll
        for (int n = 0; n < 2; n++) {                    // tokens n * 8 + g as columns, keys of the chunk as the sum
            const uint8_t *a = rec + R::a + ((n * 8 + g) * kChunk + tq * 2) * 2;
            uint32_t ap[3][2];
#pragma unroll
            for (int h = 0; h < PARTS; h++) {
                ap[h][0] = *reinterpret_cast<const uint32_t *>(a + h * kChunk * kChunk * 2);
                ap[h][1] = *reinterpret_cast<const uint32_t *>(a + h * kChunk * kChunk * 2 + 16);
            }
            float in[4] = {};                            // from inside the chunk
#pragma unroll
            for (int order = PARTS - 1; order >= 0; order--)
#pragma unroll
                for (int x = 0; x <= order; x++) mma16816(PARTS == 3 ? in : o[n], vp[x], ap[order - x][0], ap[order - x][1]);
            if (PARTS == 3)
#pragma unroll
                for (int e = 0; e < 4; e++) o[n][e] += in[e];
#pragma unroll
            for (int e = 0; e < 4; e++) {
                const uint32_t row = c * kChunk + n * 8 + tq * 2 + (e & 1);
                if (row >= p.rows || !live[e >> 1]) continue;
                if (ones[e >> 1]) p.den[(size_t)row * p.heads + head] = o[n][e];
                else              p.o[(size_t)row * vpitch + head * p.vdim + vr[e >> 1]] = o[n][e];
            }
        }
    }
    if (outputs && c1 != p.chunks) return;
    if (product)
        for (uint32_t d = t; d < (uint32_t)D; d += threads) p.products[((size_t)seg * p.heads + head) * D + d] = s_f[d];
#pragma unroll
    for (int n = 0; n < D / 8; n++)
#pragma unroll
        for (int i = 0; i < 2; i++) {
            const uint32_t d = n * 8 + tq * 2;
            if (!live[i]) continue;
            const float2 x = make_float2(S[n][2 * i], S[n][2 * i + 1]);
            if (!outputs)    *reinterpret_cast<float2 *>(p.segments + (((size_t)seg * p.heads + head) * p.cols + vr[i]) * D + d) = x;
            else if (ones[i]) {
                for (uint32_t b = 0; d < kp && b < p.blocks; b++) *reinterpret_cast<float2 *>(normalizer(p, head, b) + d) = x;
            }
            else if (d < kp) *reinterpret_cast<float2 *>(p.state + ((size_t)head * p.vdim + vr[i]) * kp + d) = x;
        }
}

// End states of segments that started from nothing (the first one: from the state) -> states behind them, in place.
// The last slot receives a copy of the sequence's state, which the last segment of the second pass overwrites.
// CTA = head x kCombineCols value columns; thread = 4 keys of a share of the columns.
constexpr uint32_t kCombineCols = 16;
template <int D>
__global__ void __launch_bounds__(256) gla_combine_kernel(const __grid_constant__ Chunks p)
{
    const uint32_t t = threadIdx.x, head = blockIdx.x, v0 = blockIdx.y * kCombineCols;
    pdl_launch_dependents();
    pdl_wait();
    const size_t step = (size_t)p.heads * p.cols * D;
    const uint32_t kp = (p.dim + 3u) & ~3u;
    for (uint32_t i = t; i < kCombineCols * D / 4; i += 256) {
        const uint32_t v = v0 + i / (D / 4), d = i % (D / 4) * 4;
        if (v >= p.cols) break;
        float *at = p.segments + ((size_t)head * p.cols + v) * D + d;
        float4 S = *reinterpret_cast<const float4 *>(at);
        *reinterpret_cast<float4 *>(at + (p.segs - 1) * step) =
            d < kp ? *reinterpret_cast<const float4 *>((v < p.vdim ? p.state + ((size_t)head * p.vdim + v) * kp : normalizer(p, head, 0)) + d) : make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll 4
        for (uint32_t s = 1; s + 1 < p.segs; s++) {
            const float4 x = *reinterpret_cast<const float4 *>(at + s * step), f = *reinterpret_cast<const float4 *>(p.products + ((size_t)s * p.heads + head) * D + d);
            S = make_float4(fmaf(f.x, S.x, x.x), fmaf(f.y, S.y, x.y), fmaf(f.z, S.z, x.z), fmaf(f.w, S.w, x.w));
            *reinterpret_cast<float4 *>(at + s * step) = S;
        }
    }
}

// o = o / (max(|n . q|, exp(-m)) + 1e-6): a thread per four columns.
__global__ void __launch_bounds__(256) mlstm_divide_kernel(const __grid_constant__ Chunks p)
{
    pdl_launch_dependents();
    pdl_wait();
    const uint32_t row = blockIdx.x;
    for (uint32_t i = threadIdx.x; i < p.heads * p.vdim; i += 256) {
        const uint32_t head = i / p.vdim;
        const float d = fmaxf(fabsf(p.den[(size_t)row * p.heads + head]), p.gates[(size_t)head * p.rows + row].z) + 1e-6f;
        p.o[(size_t)row * p.heads * p.vdim + i] /= d;
    }
}

uint32_t padded(uint32_t dim) { return dim <= 32 ? 32 : dim <= 64 ? 64 : dim <= 128 ? 128 : 256; }
// Two CTAs of up to 5 warps fit an SM where the state of a warp is no more than 128 keys wide.  More and shorter segments pay for
// time mixing (32 x 64 x 64, 2048 tokens, both passes: 59 against 85 us), not for mLSTM, whose 17 blocks then need a fourth CTA
// (8 x 128 x 256: 182 against 135 us).
uint32_t ctas_per_sm(int mode, uint32_t dim) { return mode == kWkv && padded(dim) <= 128 ? 2 : 1; }
// Blocks of 16 value columns, shared out evenly over as few CTAs as can take them.
uint32_t warps_for(int mode, uint32_t dim, uint32_t cols)
{
    const uint32_t most = ctas_per_sm(mode, dim) == 2 ? 5 : kMaxWarps, blocks = (cols + 15) / 16, ctas = (blocks + most - 1) / most;
    return (blocks + ctas - 1) / ctas;
}
size_t align256(size_t n) { return (n + 255) & ~(size_t)255; }
template <int PARTS> size_t record_bytes_of(uint32_t dim)
{
    const uint32_t d = padded(dim);
    return d == 32 ? Record<32, PARTS>::bytes : d == 64 ? Record<64, PARTS>::bytes : d == 128 ? Record<128, PARTS>::bytes : Record<256, PARTS>::bytes;
}
size_t record_bytes(int mode, uint32_t dim) { return parts_of(mode) == 2 ? record_bytes_of<2>(dim) : record_bytes_of<3>(dim); }

// Chunks per segment; all of them: one pass.  Two passes pay from three segments on.
uint32_t segment_chunks(int mode, uint32_t chunks, uint32_t heads, uint32_t dim, uint32_t cols)
{
    const uint32_t w = warps_for(mode, dim, cols), ctas = heads * ((cols + 16 * w - 1) / (16 * w)), want = std::min(kMaxSegs, 148u * ctas_per_sm(mode, dim) / ctas);
    if (want < 3 || chunks < 12) return chunks;
    const uint32_t len = std::max(4u, (chunks + want - 1) / want);
    return (chunks + len - 1) / len < 3 ? chunks : len;
}

template <int D, int MODE>
int launch_sized(Chunks p, cudaStream_t st)
{
    const size_t prep = (size_t)(3 * kChunk * (D + 4) + std::max(std::min(D / 4, 16) * kChunk * kChunk, kChunk * 128)) * 4, smem = (size_t)kStages * Record<D, parts_of(MODE)>::bytes;
    if (int rc = allow_smem(gla_prepare_kernel<D, MODE>, prep)) return rc;
    if (int rc = allow_smem(gla_chunks_kernel<D, MODE>, smem)) return rc;
    if (MODE == kMlstm)
        if (int rc = launch(mlstm_gates_kernel, dim3(p.heads), dim3(1024), 0, st, p)) return rc;
    if (int rc = launch(gla_prepare_kernel<D, MODE>, dim3(p.chunks, p.heads), dim3(256), prep, st, p)) return rc;
    const uint32_t w = warps_for(MODE, p.dim, p.cols);
    dim3 grid(p.heads, (p.cols + 16 * w - 1) / (16 * w), p.segs);
    if (p.segs > 1) {
        grid.z = p.segs - 1;
        p.states_only = 1;
        if (int rc = launch(gla_chunks_kernel<D, MODE>, grid, dim3(w * 32), smem, st, p)) return rc;
        if (int rc = launch(gla_combine_kernel<D>, dim3(p.heads, (p.cols + kCombineCols - 1) / kCombineCols), dim3(256), 0, st, p)) return rc;
        grid.z = p.segs;
        p.states_only = 0;
    }
    if (int rc = launch(gla_chunks_kernel<D, MODE>, grid, dim3(w * 32), smem, st, p)) return rc;
    return MODE == kMlstm ? launch(mlstm_divide_kernel, dim3(p.rows), dim3(256), 0, st, p) : MGQ_OK;
}

template <int MODE>
int launch_piece(Chunks p, void *workspace, cudaStream_t st)
{
    p.cols = p.vdim + (MODE == kMlstm ? 1 : 0);
    p.chunks = (p.rows + kChunk - 1) / kChunk;
    uint8_t *ws = static_cast<uint8_t *>(workspace);
    p.records = ws;
    ws += align256((size_t)p.chunks * p.heads * record_bytes(MODE, p.dim));
    if (MODE == kMlstm) {
        p.gates = reinterpret_cast<float4 *>(ws);
        ws += align256((size_t)p.rows * p.heads * 16);
        p.den = reinterpret_cast<float *>(ws);
        ws += align256((size_t)p.rows * p.heads * 4);
    }
    p.segments = reinterpret_cast<float *>(ws);
    p.products = p.segments + (size_t)kMaxSegs * p.heads * p.cols * padded(p.dim);
    p.seg_len = segment_chunks(MODE, p.chunks, p.heads, p.dim, p.cols);
    p.segs = (p.chunks + p.seg_len - 1) / p.seg_len;
    switch (padded(p.dim)) {
        case 32: return launch_sized<32, MODE>(p, st);
        case 64: return launch_sized<64, MODE>(p, st);
        case 128: return launch_sized<128, MODE>(p, st);
        default: return launch_sized<256, MODE>(p, st);
    }
}

template <int MODE>
int launch_chunks(const Chunks &all, void *workspace, cudaStream_t st)
{
    const uint32_t piece = MODE == kGla ? all.rows : kPieceRows;
    for (uint32_t r0 = 0; r0 < all.rows; r0 += piece) {
        Chunks p = all;
        p.rows = std::min(piece, all.rows - r0);
        const size_t keys = (size_t)r0 * p.heads * p.dim, values = (size_t)r0 * p.heads * p.vdim, gates = (size_t)r0 * p.heads;
        p.q += keys; p.k += keys; p.v += values; p.o += values;
        if (p.w) p.w += keys;
        if (p.d.low) p.d.low += (size_t)r0 * p.d.rank;
        if (MODE == kMlstm) { p.gi += gates; p.gf += gates; }
        if (r0) p.shift_state = nullptr;
        if (int rc = launch_piece<MODE>(p, workspace, st)) return rc;
    }
    return MGQ_OK;
}

size_t chunks_workspace(int mode, uint32_t max_rows, uint32_t heads, uint32_t dim, uint32_t vdim)
{
    if (max_rows < kPrefillRows) return 0;
    if (mode != kGla) max_rows = std::min(max_rows, kPieceRows);
    const size_t chunks = (max_rows + kChunk - 1) / kChunk, cols = vdim + (mode == kMlstm ? 1 : 0);
    return align256(chunks * heads * record_bytes(mode, dim)) + (mode == kMlstm ? align256((size_t)max_rows * heads * 16) + align256((size_t)max_rows * heads * 4) : 0) +
           (size_t)kMaxSegs * heads * (cols + 1) * padded(dim) * 4;
}

}  // namespace

size_t gla_chunks_workspace(uint32_t max_rows, uint32_t heads, uint32_t dim, uint32_t vdim) { return chunks_workspace(kGla, max_rows, heads, dim, vdim); }
size_t wkv_chunks_workspace(uint32_t max_rows, uint32_t heads, uint32_t dim, uint32_t vdim) { return chunks_workspace(kWkv, max_rows, heads, dim, vdim); }
size_t mlstm_chunks_workspace(uint32_t max_rows, uint32_t heads, uint32_t dim, uint32_t vdim) { return chunks_workspace(kMlstm, max_rows, heads, dim, vdim); }

// Up to rank 32 the launch saved is worth more than the preparation's extra multiply-adds whatever the operator, beyond that for few rows
// only, and for more of them the more tokens share a channel's weights (16 with 256 channels, 4 with 64).  Whole recurrence in
// microseconds, decays inside / in front: time mixing 32 x 64, 2048 tokens, rank 16 149 / 156, 32 158 / 160, 64 189 / 170; rank 64, 128
// tokens 47 / 54, 777 tokens 92 / 86; gated linear attention 8 x 128 x 256, 777 tokens, rank 64 82 / 90, 2048 tokens 146 / 145.
bool decay_in_chunks(uint32_t rank, uint32_t dim, uint32_t rows) { return rank <= 32 || rows < (dim >= 128 ? 1024u : 256u); }

int launch_channel_decay_chunks(const ChannelDecay &a, void *stream)
{
    if (a.dim > kMaxStateDim || !a.workspace) return fail(MGQ_ERR_STATE, "recurrence in chunks: no workspace");
    Chunks p{};
    p.q = a.q; p.k = a.k; p.v = a.v; p.w = a.decay_pending ? nullptr : a.d.out; p.d = a.d; p.u = a.u; p.o = a.o; p.state = a.state;
    p.shift_state = a.shift_state; p.shift_width = a.shift_width;
    p.rows = a.rows; p.heads = a.heads; p.dim = a.dim; p.vdim = a.vdim;
    p.qscale = a.u ? 1.f : (float)(1.0 / sqrt((double)a.dim));
    return a.u ? launch_chunks<kWkv>(p, a.workspace, static_cast<cudaStream_t>(stream)) : launch_chunks<kGla>(p, a.workspace, static_cast<cudaStream_t>(stream));
}

int launch_mlstm_chunks(const Mlstm &a, uint32_t blocks, void *stream)
{
    if (a.dim > kMaxStateDim || !a.workspace) return fail(MGQ_ERR_STATE, "recurrence in chunks: no workspace");
    Chunks p{};
    p.q = a.q; p.k = a.k; p.v = a.v; p.gi = a.gi; p.gf = a.gf; p.o = a.o; p.state = a.state;
    p.rows = a.rows; p.heads = a.heads; p.dim = a.dim; p.vdim = a.vdim;
    p.blocks = blocks;
    p.norm_pitch = ((a.dim + 3u) & ~3u) + 4u;
    p.cap = a.cap;
    p.qscale = (float)(1.0 / sqrt((double)a.dim));
    return launch_chunks<kMlstm>(p, a.workspace, static_cast<cudaStream_t>(stream));
}

}  // namespace mgq
