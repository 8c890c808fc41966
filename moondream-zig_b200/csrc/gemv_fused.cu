// Fused GEMV kernels of the decode step (M <= 8 activation rows).
//
// The reference runs one decoder layer for one token as LayerNorm, four GEMVs with their bias /
// GELU passes and two residual adds (text_model.zig:150-172, 182-323): ten tensor-wide passes, each
// of which is a separate kernel launch on a GPU.  At one token per step every one of them is far
// shorter than a launch-to-launch dependency, so the layer is restated as two weight-streaming
// kernels around the attention kernel, with every rounding point of the reference kept:
//
//   gemv_ln_dual_kernel   y = LayerNorm(hidden) (ops.zig:1152-1419, f16-rounded), then
//                         qkv = f16(f16(y Wqkv^T) + bqkv)                 (text_model.zig:193-196)
//                         fc1 = gelu(f16(f16(y Wfc1^T) + bfc1))           (text_model.zig:310-312)
//                         Both matrices consume the same y (the Phi block is parallel), so one grid
//                         streams both; every CTA recomputes the LayerNorm of the M rows (8 KB of L2
//                         reads) instead of waiting for a separate kernel.
//   gemv_dual_k_kernel    a   = f16(f16(attn Wout^T) + bout)              (text_model.zig:296-299)
//                         m   = f16(f16(fc1 Wfc2^T) + bfc2)               (text_model.zig:317-318)
//                         hidden = f16(hidden + f16(a + m))               (text_model.zig:170-171)
//                         One CTA owns 8 output rows and both dot products of those rows.
//
// Both use the tensor-core mapping of gemv.cu (weight rows on the M side of mma.sync.m16n8k16, the
// <= 8 activation rows on the N side).  gemv_dual_k_kernel needs more CTAs than 2048 / 16 to cover the
// SMs, so its A fragment holds the SAME 8 weight rows twice, rows 0-7 from one 32-wide k slab and rows
// 8-15 from the next; two MMAs with the two matching activation slabs then produce the valid halves
// (rows 0-7 of the first, rows 8-15 of the second).  Tensor work doubles, which is free here.
//
// All kernels are written for programmatic dependent launch: weights (never written on the stream)
// are requested before griddepcontrol.wait, activations only after it and never through the
// non-coherent path.
#include "md_internal.cuh"

namespace {

__device__ __forceinline__ uint4 ldg_stream(const void* p) {
    uint4 v;
    asm volatile("ld.global.nc.L1::no_allocate.v4.u32 {%0,%1,%2,%3}, [%4];"
                 : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w)
                 : "l"(p));
    return v;
}
__device__ __forceinline__ uint4 ld_act(const __half* p) {
    uint4 v;
    asm volatile("ld.global.cg.v4.u32 {%0,%1,%2,%3}, [%4];"
                 : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w)
                 : "l"(p)
                 : "memory");
    return v;
}
__device__ __forceinline__ float ld_act1(const __half* p) {
    unsigned short u;
    asm volatile("ld.global.cg.u16 %0, [%1];" : "=h"(u) : "l"(p) : "memory");
    __half_raw r;
    r.x = u;
    return __half2float(__half(r));
}
__device__ __forceinline__ void mma_16816(float (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3,
                                          uint32_t b0, uint32_t b1) {
    asm volatile(
        "mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
        : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
        : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}
__device__ __forceinline__ void pdl_launch_dependents() { asm volatile("griddepcontrol.launch_dependents;"); }
__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

// ---------------------------------------------------------------------------- LN + dual-N GEMV
constexpr int LN_K = 2048;                 // model dim this kernel is specialised for
constexpr int LN_WARPS = 8;                // 256 threads: one 16-byte piece of a row per thread
constexpr int LN_PITCH = LN_K + 32;        // halves; +64 bytes keeps the fragment reads conflict-free
constexpr int LN_CHUNKS = LN_K / 32;       // 64 chunks of 32 k, 8 per warp

struct LnDualParams {
    const __half* hidden;            // [M][2048]
    const __half *ln_w, *ln_b;       // [2048]
    float eps;
    const __half *w1, *b1;           // [n1][2048], [n1]
    __half* out1;                    // [M][n1]
    const __half *w2, *b2;           // [n2][2048], [n2]; GELU applied
    __half* out2;                    // [M][n2]
    int n1, n2, M;
    unsigned long long* amax;        // optional [M]: running argmax keys of out1 (greedy sampling), see below
    int gelu1;                       // GELU on segment 1 as well (fc1 alone as segment 1)
    md_ahead ahead;                  // requested beside a CTA's last tile (beside its first they hold the others up)
};

// ONE: a single row, normalised by the whole CTA; else up to eight, a warp each.
//
// The CTAs stay: two per SM, an equal share of the rows of both matrices each, 16 rows at a time.  A lane's registers always hold
// the requests of one whole tile (64 KB per CTA); as soon as a piece is multiplied its registers take the request of the same
// piece of the next tile.  With a CTA per 16 rows a third of a CTA's life went to the LayerNorm, the sum over the warps and the
// start of the next CTA, with nothing requested: 59 MB (qkv and fc1 in one launch) took 14.2 us, 11.7 now; lm_head (210 MB) 42.7,
// 32.5 now.  One CTA per SM (64 KB in flight) takes 16 us for the 59 MB.
template <bool ONE>
__global__ void __launch_bounds__(LN_WARPS * 32, 2)
gemv_ln_dual_kernel(LnDualParams p, int R) {
    __shared__ __align__(16) __half xs[8][LN_PITCH];
    __shared__ float partial[2][LN_WARPS][16][8];
    __shared__ float red[2][LN_WARPS];
    constexpr int PIECES = LN_CHUNKS / LN_WARPS;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, t = lane & 3;
    const int total = p.n1 + p.n2, first = blockIdx.x * R, end = min(first + R, total);

    pdl_launch_dependents();
    uint4 lo[PIECES], hi[PIECES];
    const __half *w_lo, *w_hi;
    bool has_lo, has_hi;
    float bias = 0.f;                  // of this thread's output row
    auto locate = [&](int row0) {      // this lane's two rows of a tile
        const int a = row0 + g, c = a + 8;
        has_lo = a < end, has_hi = c < end;
        w_lo = (a < p.n1 ? p.w1 + (size_t)a * LN_K : p.w2 + (size_t)(a - p.n1) * LN_K) + warp * 32 + t * 8;
        w_hi = (c < p.n1 ? p.w1 + (size_t)c * LN_K : p.w2 + (size_t)(c - p.n1) * LN_K) + warp * 32 + t * 8;
        const int row = row0 + (tid & 15);
        if (tid < 128 && row < end) bias = __half2float(row < p.n1 ? p.b1[row] : p.b2[row - p.n1]);
    };
    auto request = [&](int u) {
        lo[u] = has_lo ? ldg_stream(w_lo + u * LN_WARPS * 32) : make_uint4(0, 0, 0, 0);
        hi[u] = has_hi ? ldg_stream(w_hi + u * LN_WARPS * 32) : make_uint4(0, 0, 0, 0);
    };
    locate(first);
#pragma unroll
    for (int u = 0; u < PIECES; ++u) request(u);

    // ---- LayerNorm of the M rows into shared memory (two-pass f32, one f16 rounding)
    auto normalised = [&](const float (&v)[8], float mean, float rstd, const uint4& gw, const uint4& gb) {
        const __half2 *wh = reinterpret_cast<const __half2*>(&gw), *bh = reinterpret_cast<const __half2*>(&gb);
        const float mean_rstd = mean * rstd;
        uint4 o;
        __half2* oh = reinterpret_cast<__half2*>(&o);
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const float2 a = __half22float2(wh[i]), b = __half22float2(bh[i]);
            oh[i] = __floats2half2_rn((v[2 * i] * rstd - mean_rstd) * a.x + b.x, (v[2 * i + 1] * rstd - mean_rstd) * a.y + b.y);
        }
        return o;
    };
    auto unpack = [](const uint4& u, float (&v)[8]) {
        const __half2* h = reinterpret_cast<const __half2*>(&u);
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const float2 f = __half22float2(h[i]);
            v[2 * i] = f.x;
            v[2 * i + 1] = f.y;
        }
    };
    auto warp_sum = [](float x) {
#pragma unroll
        for (int o = 16; o; o >>= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
        return x;
    };
    if constexpr (ONE) {
        // LayerNorm parameters are weights too
        const uint4 gw = ldg_stream(p.ln_w + tid * 8), gb = ldg_stream(p.ln_b + tid * 8);
#pragma unroll
        for (int m = 1; m < 8; ++m) *reinterpret_cast<uint4*>(&xs[m][tid * 8]) = make_uint4(0, 0, 0, 0);
        pdl_wait();
        auto block_sum = [&](float x, int slot) {
            x = warp_sum(x);
            if (lane == 0) red[slot][warp] = x;
            __syncthreads();
            x = 0.f;
#pragma unroll
            for (int w = 0; w < LN_WARPS; ++w) x += red[slot][w];
            return x;
        };
        float v[8], s = 0.f, q = 0.f;
        unpack(ld_act(p.hidden + tid * 8), v);
#pragma unroll
        for (int i = 0; i < 4; ++i) s += v[2 * i] + v[2 * i + 1];
        const float mean = block_sum(s, 0) * (1.0f / LN_K);
#pragma unroll
        for (int i = 0; i < 8; ++i) q += (v[i] - mean) * (v[i] - mean);
        const float rstd = 1.0f / sqrtf(block_sum(q, 1) * (1.0f / LN_K) + p.eps);
        *reinterpret_cast<uint4*>(&xs[0][tid * 8]) = normalised(v, mean, rstd, gw, gb);
    } else {
        pdl_wait();
        constexpr int PER = LN_K / 256;      // 16-byte pieces of a row per lane
        if (warp < p.M) {
            uint4 row[PER];
#pragma unroll
            for (int i = 0; i < PER; ++i) row[i] = ld_act(p.hidden + (size_t)warp * LN_K + (i * 32 + lane) * 8);
            float s = 0.f, q = 0.f;
#pragma unroll
            for (int i = 0; i < PER; ++i) {
                float v[8];
                unpack(row[i], v);
#pragma unroll
                for (int j = 0; j < 4; ++j) s += v[2 * j] + v[2 * j + 1];
            }
            const float mean = warp_sum(s) * (1.0f / LN_K);
#pragma unroll
            for (int i = 0; i < PER; ++i) {
                float v[8];
                unpack(row[i], v);
#pragma unroll
                for (int j = 0; j < 8; ++j) q += (v[j] - mean) * (v[j] - mean);
            }
            const float rstd = 1.0f / sqrtf(warp_sum(q) * (1.0f / LN_K) + p.eps);
#pragma unroll
            for (int i = 0; i < PER; ++i) {
                float v[8];
                unpack(row[i], v);
                const int c = (i * 32 + lane) * 8;
                *reinterpret_cast<uint4*>(&xs[warp][c]) = normalised(v, mean, rstd, ldg_stream(p.ln_w + c), ldg_stream(p.ln_b + c));
            }
        } else {
#pragma unroll
            for (int i = 0; i < PER; ++i) *reinterpret_cast<uint4*>(&xs[warp][(i * 32 + lane) * 8]) = make_uint4(0, 0, 0, 0);
        }
    }
    __syncthreads();
    uint4 xv[PIECES];
#pragma unroll
    for (int u = 0; u < PIECES; ++u) xv[u] = *reinterpret_cast<const uint4*>(&xs[g][(warp + u * LN_WARPS) * 32 + t * 8]);  // rows >= M are zeros

    // ---- the dot products
    unsigned long long best = 0ull;
    int buf = 0;
    for (int row0 = first; row0 < end; row0 += 16, buf ^= 1) {
        const float own_bias = bias;
        if (tid == 0 && row0 + 16 >= end) md_fetch_ahead(p.ahead, blockIdx.x, gridDim.x);
        locate(row0 + 16);
        float acc[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
        for (int u = 0; u < PIECES; ++u) {
            mma_16816(acc, lo[u].x, hi[u].x, lo[u].y, hi[u].y, xv[u].x, xv[u].y);
            mma_16816(acc, lo[u].z, hi[u].z, lo[u].w, hi[u].w, xv[u].z, xv[u].w);
            request(u);
        }
        float (*mine)[16][8] = partial[buf];
        mine[warp][g][2 * t] = acc[0];
        mine[warp][g][2 * t + 1] = acc[1];
        mine[warp][g + 8][2 * t] = acc[2];
        mine[warp][g + 8][2 * t + 1] = acc[3];
        __syncthreads();
        if (tid >= 128) continue;
        const int m = tid >> 4, row = row0 + (tid & 15);
        if (m >= p.M || row >= end) continue;
        const bool seg2 = row >= p.n1;
        const int n = seg2 ? row - p.n1 : row, n_seg = seg2 ? p.n2 : p.n1;
        float sum = 0.f;
#pragma unroll
        for (int w = 0; w < LN_WARPS; ++w) sum += mine[w][tid & 15][m];
        float val = md_round_f16(sum);
        val = md_round_f16(val + own_bias);
        if (seg2 || p.gelu1) val = md_round_f16(md_gelu_f32(val));
        (seg2 ? p.out2 : p.out1)[(size_t)m * n_seg + n] = __float2half_rn(val);
        // Greedy sampling folded into the lm_head (sampling.zig:257-273: first strict maximum of the f16
        // logits): a 64-bit key orders by value, then by LOWER index; one atomicMax per CTA and row.
        const unsigned bits = __float_as_uint(val);
        const unsigned ordered = (bits & 0x80000000u) ? ~bits : (bits | 0x80000000u);
        const unsigned long long key = ((unsigned long long)ordered << 32) | (unsigned long long)(0xFFFFFFFFu - (unsigned)n);
        if (!seg2) best = key > best ? key : best;
    }
    if (p.amax && tid < 128) {
#pragma unroll
        for (int o = 8; o; o >>= 1) {
            const unsigned long long other = __shfl_xor_sync(0xffffffffu, best, o);
            best = other > best ? other : best;
        }
        if ((tid & 15) == 0 && (tid >> 4) < p.M) atomicMax(p.amax + (tid >> 4), best);
    }
}

// ---------------------------------------------------------------------------- dual-K GEMV + residuals


struct DualKParams {
    const __half *x1, *w1, *b1;   // [M][k1], [N][k1], [N]
    const __half *x2, *w2, *b2;   // [M][k2], [N][k2], [N]
    __half* hidden;               // [M][N], updated in place
    int N, k1, k2, M;
};

template <int DK_WARPS, int UNROLL>
__global__ void __launch_bounds__(DK_WARPS * 32)
gemv_dual_k_kernel(DualKParams p) {
    __shared__ float partial[DK_WARPS][2][8][8];
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, t = lane & 3;
    const int row0 = blockIdx.x * 8;
    const int r = min(row0 + g, p.N - 1);
    const int units1 = p.k1 / 64, units = units1 + p.k2 / 64;  // a unit = two consecutive 32-wide k slabs
    const bool has_x = g < p.M;

    float a1e[4] = {0.f, 0.f, 0.f, 0.f}, a1o[4] = {0.f, 0.f, 0.f, 0.f};
    float a2e[4] = {0.f, 0.f, 0.f, 0.f}, a2o[4] = {0.f, 0.f, 0.f, 0.f};

    pdl_launch_dependents();
    bool waited = false;
    for (int u0 = warp; u0 < units; u0 += UNROLL * DK_WARPS) {
        uint4 lo[UNROLL], hi[UNROLL];
#pragma unroll
        for (int j = 0; j < UNROLL; ++j) {
            const int u = u0 + j * DK_WARPS;
            if (u < units) {
                const bool s2 = u >= units1;
                const __half* wrow = s2 ? p.w2 + (size_t)r * p.k2 + (size_t)(u - units1) * 64
                                        : p.w1 + (size_t)r * p.k1 + (size_t)u * 64;
                lo[j] = ldg_stream(wrow + t * 8);        // slab A: k .. k+31
                hi[j] = ldg_stream(wrow + 32 + t * 8);   // slab B: k+32 .. k+63
            } else {
                lo[j] = hi[j] = make_uint4(0, 0, 0, 0);
            }
        }
        if (!waited) { pdl_wait(); waited = true; }
#pragma unroll
        for (int j = 0; j < UNROLL; ++j) {
            const int u = u0 + j * DK_WARPS;
            if (u >= units) continue;
            const bool s2 = u >= units1;
            const __half* xrow = s2 ? p.x2 + (size_t)(has_x ? g : 0) * p.k2 + (size_t)(u - units1) * 64
                                    : p.x1 + (size_t)(has_x ? g : 0) * p.k1 + (size_t)u * 64;
            const uint4 xa = has_x ? ld_act(xrow + t * 8) : make_uint4(0, 0, 0, 0);
            const uint4 xb = has_x ? ld_act(xrow + 32 + t * 8) : make_uint4(0, 0, 0, 0);
            if (s2) {
                mma_16816(a2e, lo[j].x, hi[j].x, lo[j].y, hi[j].y, xa.x, xa.y);
                mma_16816(a2e, lo[j].z, hi[j].z, lo[j].w, hi[j].w, xa.z, xa.w);
                mma_16816(a2o, lo[j].x, hi[j].x, lo[j].y, hi[j].y, xb.x, xb.y);
                mma_16816(a2o, lo[j].z, hi[j].z, lo[j].w, hi[j].w, xb.z, xb.w);
            } else {
                mma_16816(a1e, lo[j].x, hi[j].x, lo[j].y, hi[j].y, xa.x, xa.y);
                mma_16816(a1e, lo[j].z, hi[j].z, lo[j].w, hi[j].w, xa.z, xa.w);
                mma_16816(a1o, lo[j].x, hi[j].x, lo[j].y, hi[j].y, xb.x, xb.y);
                mma_16816(a1o, lo[j].z, hi[j].z, lo[j].w, hi[j].w, xb.z, xb.w);
            }
        }
    }
    if (!waited) pdl_wait();
    // valid halves: rows 0-7 of the "even" accumulators (c0, c1), rows 8-15 of the "odd" ones (c2, c3)
    partial[warp][0][g][2 * t] = a1e[0] + a1o[2];
    partial[warp][0][g][2 * t + 1] = a1e[1] + a1o[3];
    partial[warp][1][g][2 * t] = a2e[0] + a2o[2];
    partial[warp][1][g][2 * t + 1] = a2e[1] + a2o[3];
    __syncthreads();
    if (tid < 64) {
        const int m = tid >> 3, rr = tid & 7, n = row0 + rr;
        if (m < p.M && n < p.N) {
            float s1 = 0.f, s2 = 0.f;
#pragma unroll
            for (int w = 0; w < DK_WARPS; ++w) {
                s1 += partial[w][0][rr][m];
                s2 += partial[w][1][rr][m];
            }
            const float a = md_round_f16(md_round_f16(s1) + __half2float(p.b1[n]));
            const float mlp = md_round_f16(md_round_f16(s2) + __half2float(p.b2[n]));
            const float sum = md_round_f16(a + mlp);
            __half* h = p.hidden + (size_t)m * p.N + n;
            *h = __float2half_rn(ld_act1(h) + sum);
        }
    }
}

template <class Kern, class Params, class... More>
int launch_pdl(md_ctx* ctx, Kern kern, unsigned grid, unsigned block, const Params& p, const char* name, More... more) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(grid);
    cfg.blockDim = dim3(block);
    cfg.stream = ctx->stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = ctx->pdl ? 1 : 0;
    const cudaError_t e = cudaLaunchKernelEx(&cfg, kern, p, more...);
    if (e != cudaSuccess) return md_fail(ctx, MD_ERR_CUDA, "launch of %s failed: %s", name, cudaGetErrorString(e));
    ctx->launches++;
    return MD_OK;
}

}  // namespace

bool md_gemv_ln_dual_supported(size_t M, size_t K, size_t n1, size_t n2) {
    return M >= 1 && M <= 8 && K == LN_K && n1 % 16 == 0 && n2 % 16 == 0 && n1 > 0;
}

int md_launch_gemv_ln_dual(md_ctx* ctx, const __half* hidden, const __half* ln_w, const __half* ln_b, float eps,
                           const __half* w1, const __half* b1, __half* out1, size_t n1, const __half* w2,
                           const __half* b2, __half* out2, size_t n2, size_t M, size_t K, unsigned long long* amax,
                           bool gelu1, const md_ahead& ahead) {
    if (!md_gemv_ln_dual_supported(M, K, n1, n2))
        return md_fail(ctx, MD_ERR_UNSUPPORTED, "gemv_ln_dual: unsupported shape M=%zu K=%zu n1=%zu n2=%zu", M, K, n1, n2);
    LnDualParams p;
    p.hidden = hidden; p.ln_w = ln_w; p.ln_b = ln_b; p.eps = eps;
    p.w1 = w1; p.b1 = b1; p.out1 = out1; p.w2 = w2; p.b2 = b2; p.out2 = out2;
    p.n1 = (int)n1; p.n2 = (int)n2; p.M = (int)M;
    p.amax = amax;
    p.gelu1 = gelu1 ? 1 : 0;
    p.ahead = ahead;
    // an equal share for every CTA that fits at once, in rows (fewer tiles than that: one each)
    const int total = (int)(n1 + n2), ctas = 2 * ctx->sm_count;
    const int R = total / 16 < ctas ? 16 : (total + ctas - 1) / ctas;
    const unsigned grid = (unsigned)((total + R - 1) / R);
    return launch_pdl(ctx, M == 1 ? gemv_ln_dual_kernel<true> : gemv_ln_dual_kernel<false>, grid, LN_WARPS * 32, p, "gemv_ln_dual_kernel", R);
}

bool md_gemv_dual_k_supported(size_t M, size_t N, size_t k1, size_t k2) {
    return M >= 1 && M <= 8 && N > 0 && k1 % 64 == 0 && k2 % 64 == 0 && k1 > 0 && k2 > 0;
}

int md_launch_gemv_dual_k(md_ctx* ctx, const __half* x1, const __half* w1, const __half* b1, size_t k1,
                          const __half* x2, const __half* w2, const __half* b2, size_t k2, __half* hidden, size_t N,
                          size_t M) {
    if (!md_gemv_dual_k_supported(M, N, k1, k2))
        return md_fail(ctx, MD_ERR_UNSUPPORTED, "gemv_dual_k: unsupported shape M=%zu N=%zu k1=%zu k2=%zu", M, N, k1, k2);
    DualKParams p;
    p.x1 = x1; p.w1 = w1; p.b1 = b1; p.x2 = x2; p.w2 = w2; p.b2 = b2; p.hidden = hidden;
    p.N = (int)N; p.k1 = (int)k1; p.k2 = (int)k2; p.M = (int)M;
    const unsigned grid = (unsigned)((N + 7) / 8);
    switch (ctx->dualk_variant) {
        case 1: return launch_pdl(ctx, gemv_dual_k_kernel<16, 5>, grid, 16 * 32, p, "gemv_dual_k_kernel");
        case 2: return launch_pdl(ctx, gemv_dual_k_kernel<8, 10>, grid, 8 * 32, p, "gemv_dual_k_kernel");
        case 3: return launch_pdl(ctx, gemv_dual_k_kernel<4, 10>, grid, 4 * 32, p, "gemv_dual_k_kernel");
        case 4: return launch_pdl(ctx, gemv_dual_k_kernel<16, 10>, grid, 16 * 32, p, "gemv_dual_k_kernel");
        default: return launch_pdl(ctx, gemv_dual_k_kernel<8, 5>, grid, 8 * 32, p, "gemv_dual_k_kernel");
    }
}
