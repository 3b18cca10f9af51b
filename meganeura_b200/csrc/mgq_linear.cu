// Linear layers over bf16 weights stored [N, K]:  y[m, n] = sum_k x[m, k] W[n, k] (+ bias[n]) (+ addend[m, n]).
//
// One launch takes a GROUP of up to kMaxSegments independent layers that share M (the projections of
// one mixer: same or different inputs, different widths), so a decode step pays one kernel boundary
// for all of them.  A gated feed-forward's pair of projections runs as one segment with two weights
// whose epilogue applies the GLU.
//
//   linear_gemv_kernel   M <= 8: HBM-bound, a warp streams R weight rows with 16-byte loads for all M
//                        activation rows at once (every weight byte is read once per 8 rows).
//   linear_tiled_kernel  general: 64x64 register tiles in true f32, K split over clusters (f32 activations, sizes
//                        the tensor cores cannot take).
//   mgq_linear_tc.cu     M > 8, bf16 activations: tcgen05.
#include "mgq_linear.cuh"

namespace mgq {
namespace {

// ---------------------------------------------------------------- GEMV
// Unit = R weight rows of one segment (GLU: R/2 columns, gate and up rows of each).
template <typename XT, int M, int R, bool GLU, bool VEC>
__global__ void __launch_bounds__(128) linear_gemv_kernel(const __grid_constant__ LinearGroup g, uint32_t m, uint32_t row0)
{
    constexpr int COLS = GLU ? R / 2 : R;
    const uint32_t lane = threadIdx.x & 31u;
    uint32_t unit = blockIdx.x * 4u + (threadIdx.x >> 5), si = 0;
    pdl_launch_dependents();
    while (si < g.count) {
        const uint32_t units = (g.seg[si].n + COLS - 1) / COLS;
        if (unit < units) break;
        unit -= units;
        si++;
    }
    if (si >= g.count) return;
    const LinearSegment &s = g.seg[si];
    const uint32_t n0 = unit * COLS, k = s.k;
    const __nv_bfloat16 *w[R];
#pragma unroll
    for (int r = 0; r < R; r++) {
        const uint32_t n = min(n0 + (uint32_t)(GLU ? r / 2 : r), s.n - 1u);
        w[r] = static_cast<const __nv_bfloat16 *>((GLU && (r & 1)) ? s.w2 : s.w) + (size_t)n * k;
    }
    // weights are immutable: start moving all of the rows towards L2 before waiting for the activations, and keep eight loads of a
    // lone row in flight (Tobovik, 777 + 12 tokens: 9321 -> 9052 us; only the first 2048 k and four loads before)
    for (uint32_t c = lane * 64u; c < k; c += 2048u)
#pragma unroll
        for (int r = 0; r < R; r++) asm volatile("prefetch.global.L2 [%0];" ::"l"(w[r] + c));
    pdl_wait();
    const XT *x = static_cast<const XT *>(s.a) + (size_t)row0 * k;
    float acc[M][R];
#pragma unroll
    for (int i = 0; i < M; i++)
#pragma unroll
        for (int r = 0; r < R; r++) acc[i][r] = 0.f;
    if (VEC) {
        const uint32_t chunks = k / 8;
#pragma unroll(M <= 2 ? (R == 1 ? 8 : 4) : 2)
        for (uint32_t c = lane; c < chunks; c += 32) {
            uint4 q[R];
#pragma unroll
            for (int r = 0; r < R; r++)
                asm volatile("ld.global.nc.L1::no_allocate.v4.u32 {%0, %1, %2, %3}, [%4];"
                             : "=r"(q[r].x), "=r"(q[r].y), "=r"(q[r].z), "=r"(q[r].w) : "l"(w[r] + (size_t)c * 8));
#pragma unroll
            for (int i = 0; i < M; i++) {
                float xv[8];
                load8(x + (size_t)(i < (int)m ? i : 0) * k + (size_t)c * 8, xv);
#pragma unroll
                for (int r = 0; r < R; r++) {
                    float wv[8];
                    unpack8(q[r], wv);
#pragma unroll
                    for (int j = 0; j < 8; j++) acc[i][r] = fmaf(xv[j], wv[j], acc[i][r]);
                }
            }
        }
    } else {
        for (uint32_t c = lane; c < k; c += 32) {
            float wv[R];
#pragma unroll
            for (int r = 0; r < R; r++) wv[r] = __bfloat162float(w[r][c]);
#pragma unroll
            for (int i = 0; i < M; i++) {
                const float xv = to_f32(x[(size_t)(i < (int)m ? i : 0) * k + c]);
#pragma unroll
                for (int r = 0; r < R; r++) acc[i][r] = fmaf(xv, wv[r], acc[i][r]);
            }
        }
    }
#pragma unroll
    for (int i = 0; i < M; i++)
#pragma unroll
        for (int r = 0; r < R; r++) acc[i][r] = warp_sum(acc[i][r]);
#pragma unroll
    for (int i = 0; i < M; i++) {
        if (i >= (int)m) break;
#pragma unroll
        for (int c = 0; c < COLS; c++) {
            const uint32_t n = n0 + c;
            if (lane != (uint32_t)(i * COLS + c) % 32u || n >= s.n) continue;
            const size_t o = (size_t)(row0 + i) * s.n + n;
            if (GLU) {
                const float y = glu_f(acc[i][2 * c] + (s.bias ? s.bias[n] : 0.f), acc[i][2 * c + 1] + (s.bias ? s.bias2[n] : 0.f), g.act);
                if (g.out_bf16) static_cast<__nv_bfloat16 *>(s.out)[o] = __float2bfloat16_rn(y);
                else            static_cast<float *>(s.out)[o] = y;
            } else {
                float y = acc[i][c];
                if (s.bias) y += s.bias[n];
                if (s.addend) y += s.addend[o];
                static_cast<float *>(s.out)[o] = y;
            }
        }
    }
}

template <typename XT, int M, int R, bool GLU>
int launch_gemv_vec(const LinearGroup &g, uint32_t m, uint32_t row0, bool vec, cudaStream_t stream)
{
    constexpr uint32_t COLS = GLU ? R / 2 : R;
    uint32_t units = 0;
    for (uint32_t i = 0; i < g.count; i++) units += (g.seg[i].n + COLS - 1) / COLS;
    const dim3 grid((units + 3) / 4);
    if (vec) return launch(linear_gemv_kernel<XT, M, R, GLU, true>, grid, dim3(128), 0, stream, g, m, row0);
    return launch(linear_gemv_kernel<XT, M, R, GLU, false>, grid, dim3(128), 0, stream, g, m, row0);
}

template <typename XT, int M>
int launch_gemv_rows(const LinearGroup &g, uint32_t m, uint32_t row0, bool vec, cudaStream_t stream)
{
    // enough warps to fill the GPU before a warp takes several rows
    uint32_t rows = 0;
    for (uint32_t i = 0; i < g.count; i++) rows += g.seg[i].n * (g.glu ? 2u : 1u);
    if (g.glu) {
        if (rows >= 9472u) return launch_gemv_vec<XT, M, 4, true>(g, m, row0, vec, stream);
        return launch_gemv_vec<XT, M, 2, true>(g, m, row0, vec, stream);
    }
    if (rows >= 9472u) return launch_gemv_vec<XT, M, 4, false>(g, m, row0, vec, stream);
    if (rows >= 4736u) return launch_gemv_vec<XT, M, 2, false>(g, m, row0, vec, stream);
    return launch_gemv_vec<XT, M, 1, false>(g, m, row0, vec, stream);
}

template <typename XT>
int launch_gemv_typed(const LinearGroup &g, bool vec, cudaStream_t stream)
{
    for (uint32_t row0 = 0; row0 < g.m; row0 += 8) {
        const uint32_t m = min(8u, g.m - row0);
        int rc;
        if (m == 1)      rc = launch_gemv_rows<XT, 1>(g, m, row0, vec, stream);
        else if (m == 2) rc = launch_gemv_rows<XT, 2>(g, m, row0, vec, stream);
        else if (m <= 4) rc = launch_gemv_rows<XT, 4>(g, m, row0, vec, stream);
        else             rc = launch_gemv_rows<XT, 8>(g, m, row0, vec, stream);
        if (rc) return rc;
    }
    return MGQ_OK;
}

// ---------------------------------------------------------------- general tiled kernel (CUDA cores, f32)
// A tile of 8 RM rows x 64 columns per CTA, RM x 4 values per thread, true f32 products and sums.  Few rows make few tiles (100 x 1024
// outputs are 32), so K is shared out over a cluster of up to 8 CTAs whose partial sums meet in rank order through distributed
// shared memory; a rank finishes the rows of its share.  The next 32 k are requested while the current ones are multiplied.
// Bound by the issue of multiply-adds (two per instruction) once the SMs are full.
// A prompt of 100 tokens and 3 single ones of a 2-layer f32 Tobovik of width 1024: 2829 us with one CTA per tile and 16 k per
// step, 1160 us so.
constexpr int BN = 64, BK = 32;

__device__ __forceinline__ float4 cluster_load4(const float *p, uint32_t rank)
{
    uint32_t addr;
    float4 v;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(addr) : "r"((uint32_t)__cvta_generic_to_shared(p)), "r"(rank));
    asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(addr) : "memory");
    return v;
}

__device__ __forceinline__ void load4(const float *p, float (&v)[4])
{
    const float4 q = *reinterpret_cast<const float4 *>(p);
    v[0] = q.x; v[1] = q.y; v[2] = q.z; v[3] = q.w;
}
__device__ __forceinline__ void load4(const __nv_bfloat16 *p, float (&v)[4])
{
    const uint2 q = *reinterpret_cast<const uint2 *>(p);
    v[0] = __uint_as_float(q.x << 16); v[1] = __uint_as_float(q.x & 0xFFFF0000u);
    v[2] = __uint_as_float(q.y << 16); v[3] = __uint_as_float(q.y & 0xFFFF0000u);
}

template <bool GLU>
__device__ __forceinline__ void finish_value(const LinearGroup &g, const LinearSegment &s, uint32_t row, uint32_t n, float y, float up)
{
    if (row >= g.m || n >= s.n) return;
    const size_t o = (size_t)row * s.n + n;
    if (GLU) {
        y = glu_f(y + (s.bias ? s.bias[n] : 0.f), up + (s.bias ? s.bias2[n] : 0.f), g.act);
        if (g.out_bf16) static_cast<__nv_bfloat16 *>(s.out)[o] = __float2bfloat16_rn(y);
        else            static_cast<float *>(s.out)[o] = y;
        return;
    }
    if (s.bias) y += s.bias[n];
    if (s.addend) y += s.addend[o];
    static_cast<float *>(s.out)[o] = y;
}

// grid: column tiles of all layers x (row tiles * splits); a cluster is the splits of a tile.
template <typename XT, bool GLU, int RM>
__global__ void __launch_bounds__(128) linear_tiled_kernel(const __grid_constant__ LinearGroup g, uint32_t splits, bool vec)
{
    constexpr int BM = 8 * RM, U = GLU ? 2 : 1, LA = BM + 4, LW = BN + 4;
    constexpr int kStage = BK * LA + U * BK * LW, kPart = U * BM * LW;
    __shared__ __align__(16) float buf[kStage > kPart ? kStage : kPart];
    float *s_a = buf, *s_w = buf + BK * LA;                    // [k][row], [weight][k][column]
    uint32_t tile = blockIdx.x, si = 0;
    pdl_launch_dependents();
    while (si + 1 < g.count) {
        const uint32_t tiles = (g.seg[si].n + BN - 1) / BN;
        if (tile < tiles) break;
        tile -= tiles;
        si++;
    }
    const LinearSegment &s = g.seg[si];
    const uint32_t rank = blockIdx.y % splits;
    const uint32_t n0 = tile * BN, m0 = blockIdx.y / splits * BM, k = s.k, t = threadIdx.x;
    const uint32_t tx = t & 15u, ty = t >> 4;
    const uint32_t share = (k + splits * BK - 1) / (splits * BK) * BK, k_begin = min(k, rank * share), k_end = min(k, k_begin + share);
    const XT *a = static_cast<const XT *>(s.a);
    const __nv_bfloat16 *w[U] = {};
    w[0] = static_cast<const __nv_bfloat16 *>(s.w);
    if (GLU) w[U - 1] = static_cast<const __nv_bfloat16 *>(s.w2);
    constexpr int NA = BM * (BK / 4) / 128, NW = BN * (BK / 8) / 128;
    float ra[NA][4];
    uint4 rw[U][NW];
    auto fetch = [&](uint32_t k0) {                            // zeros beyond the matrix and beyond this rank's share
#pragma unroll
        for (int i = 0; i < NA; i++) {
            const uint32_t e = t + 128u * i, row = m0 + e % BM, kk = k0 + e / BM * 4;
#pragma unroll
            for (int x = 0; x < 4; x++) ra[i][x] = 0.f;
            if (row < g.m && kk < k_end) {
                const XT *p = a + (size_t)row * k + kk;
                if (vec) load4(p, ra[i]);
                else
#pragma unroll
                    for (int x = 0; x < 4; x++)
                        if (kk + x < k_end) ra[i][x] = to_f32(p[x]);
            }
        }
#pragma unroll
        for (int u = 0; u < U; u++)
#pragma unroll
            for (int i = 0; i < NW; i++) {
                const uint32_t e = t + 128u * i, n = n0 + e % BN, kk = k0 + e / BN * 8;
                rw[u][i] = make_uint4(0, 0, 0, 0);
                if (n < s.n && kk < k_end) {
                    const __nv_bfloat16 *p = w[u] + (size_t)n * k + kk;
                    if (vec) rw[u][i] = __ldg(reinterpret_cast<const uint4 *>(p));
                    else {
                        uint32_t v[8];
#pragma unroll
                        for (int x = 0; x < 8; x++) v[x] = kk + x < k_end ? (uint32_t)__bfloat16_as_ushort(p[x]) : 0u;
                        rw[u][i] = make_uint4(v[0] | v[1] << 16, v[2] | v[3] << 16, v[4] | v[5] << 16, v[6] | v[7] << 16);
                    }
                }
            }
    };
    float acc[U][RM][4];
#pragma unroll
    for (int u = 0; u < U; u++)
#pragma unroll
        for (int i = 0; i < RM; i++)
#pragma unroll
            for (int j = 0; j < 4; j++) acc[u][i][j] = 0.f;
    pdl_wait();
    fetch(k_begin);
    for (uint32_t k0 = k_begin; k0 < k_end; k0 += BK) {
#pragma unroll
        for (int i = 0; i < NA; i++) {
            const uint32_t e = t + 128u * i;
#pragma unroll
            for (int x = 0; x < 4; x++) s_a[(e / BM * 4 + x) * LA + e % BM] = ra[i][x];
        }
#pragma unroll
        for (int u = 0; u < U; u++)
#pragma unroll
            for (int i = 0; i < NW; i++) {
                const uint32_t e = t + 128u * i;
                float v[8];
                unpack8(rw[u][i], v);
#pragma unroll
                for (int x = 0; x < 8; x++) s_w[(u * BK + e / BN * 8 + x) * LW + e % BN] = v[x];
            }
        __syncthreads();
        if (k0 + BK < k_end) fetch(k0 + BK);
#pragma unroll 8
        for (int kk = 0; kk < BK; kk++) {
            float ar[RM];
#pragma unroll
            for (int i = 0; i < RM; i += 4) {
                const float4 v = *reinterpret_cast<const float4 *>(s_a + kk * LA + ty * RM + i);
                ar[i] = v.x; ar[i + 1] = v.y; ar[i + 2] = v.z; ar[i + 3] = v.w;
            }
#pragma unroll
            for (int u = 0; u < U; u++) {
                const float4 v = *reinterpret_cast<const float4 *>(s_w + (u * BK + kk) * LW + tx * 4);
#pragma unroll
                for (int i = 0; i < RM; i++) {
                    fma_pair(acc[u][i][0], acc[u][i][1], ar[i], ar[i], v.x, v.y);
                    fma_pair(acc[u][i][2], acc[u][i][3], ar[i], ar[i], v.z, v.w);
                }
            }
        }
        __syncthreads();
    }
    if (splits == 1) {
#pragma unroll
        for (int i = 0; i < RM; i++)
#pragma unroll
            for (int j = 0; j < 4; j++) finish_value<GLU>(g, s, m0 + ty * RM + i, n0 + tx * 4 + j, acc[0][i][j], acc[U - 1][i][j]);
        return;
    }
#pragma unroll
    for (int u = 0; u < U; u++)
#pragma unroll
        for (int i = 0; i < RM; i++) *reinterpret_cast<float4 *>(buf + (u * BM + ty * RM + i) * LW + tx * 4) = make_float4(acc[u][i][0], acc[u][i][1], acc[u][i][2], acc[u][i][3]);
    cluster_sync();
    const uint32_t rows = BM / splits;
    for (uint32_t e = t; e < rows * 16; e += 128) {
        const uint32_t row = rank * rows + e / 16, col = e % 16 * 4;
        float4 sum[U];
#pragma unroll
        for (int u = 0; u < U; u++) {
            sum[u] = cluster_load4(buf + (u * BM + row) * LW + col, 0);
            for (uint32_t r = 1; r < splits; r++) {
                const float4 v = cluster_load4(buf + (u * BM + row) * LW + col, r);
                sum[u].x += v.x; sum[u].y += v.y; sum[u].z += v.z; sum[u].w += v.w;
            }
        }
        finish_value<GLU>(g, s, m0 + row, n0 + col, sum[0].x, sum[U - 1].x);
        finish_value<GLU>(g, s, m0 + row, n0 + col + 1, sum[0].y, sum[U - 1].y);
        finish_value<GLU>(g, s, m0 + row, n0 + col + 2, sum[0].z, sum[U - 1].z);
        finish_value<GLU>(g, s, m0 + row, n0 + col + 3, sum[0].w, sum[U - 1].w);
    }
    cluster_sync();                                            // the others may still read this CTA's sums
}

template <typename XT, bool GLU, int RM>
int launch_tiled_rows(const LinearGroup &g, bool vec, cudaStream_t stream)
{
    uint32_t tiles = 0, k = 0;
    for (uint32_t i = 0; i < g.count; i++) {
        tiles += (g.seg[i].n + BN - 1) / BN;
        k = max(k, g.seg[i].k);
    }
    const uint32_t row_tiles = (g.m + 8 * RM - 1) / (8 * RM);
    // four CTAs per SM, as long as each has 128 k left to sum
    uint32_t splits = 1;
    while (splits < 8 && tiles * row_tiles * splits * 2 <= 4 * 148 && k / (splits * 2) >= 128) splits *= 2;
    return launch_clustered(linear_tiled_kernel<XT, GLU, RM>, dim3(tiles, row_tiles * splits), dim3(128), splits, 0, stream, g, splits, vec);
}

template <typename XT>
int launch_tiled_typed(const LinearGroup &g, bool vec, cudaStream_t stream)
{
    if (g.m <= 32) return g.glu ? launch_tiled_rows<XT, true, 4>(g, vec, stream) : launch_tiled_rows<XT, false, 4>(g, vec, stream);
    return g.glu ? launch_tiled_rows<XT, true, 8>(g, vec, stream) : launch_tiled_rows<XT, false, 8>(g, vec, stream);
}

int g_linear_force_tiled = 0;      // "linear.force_tiled"

}  // namespace

int set_linear_option(const char *name, long value)
{
    if (!__builtin_strcmp(name, "linear.force_tiled")) {
        g_linear_force_tiled = value ? 1 : 0;
        return MGQ_OK;
    }
    return fail(MGQ_ERR_NAME, "unknown option: %s", name);
}

int launch_linear_group(const LinearGroup &g, void *stream_v)
{
    cudaStream_t stream = static_cast<cudaStream_t>(stream_v);
    if (g.m == 0) return MGQ_OK;
    if (g.count == 0 || g.count > kMaxSegments || (g.glu && g.count != 1)) return fail(MGQ_ERR_SHAPE, "linear: %u layers", g.count);
    bool vec = true;
    for (uint32_t i = 0; i < g.count; i++) {
        const LinearSegment &s = g.seg[i];
        if (!s.a || !s.w || !s.out || (g.glu && (!s.w2 || !s.bias != !s.bias2))) return fail(MGQ_ERR_NULL, "linear: null operand");
        if (s.k == 0) return fail(MGQ_ERR_SHAPE, "linear: K is 0");
        vec = vec && s.k % 8 == 0 && reinterpret_cast<uintptr_t>(s.a) % 16 == 0 && reinterpret_cast<uintptr_t>(s.w) % 16 == 0 &&
              reinterpret_cast<uintptr_t>(s.w2) % 16 == 0;
    }
    if (g.m <= 8) return g.a_bf16 ? launch_gemv_typed<__nv_bfloat16>(g, vec, stream) : launch_gemv_typed<float>(g, vec, stream);
    if (g.a_bf16 && vec && !g_linear_force_tiled) return launch_linear_tc(g, stream_v);
    return g.a_bf16 ? launch_tiled_typed<__nv_bfloat16>(g, vec, stream) : launch_tiled_typed<float>(g, vec, stream);
}

}  // namespace mgq
