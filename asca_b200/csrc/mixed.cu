// bf16-mode companions of the f32 element-wise entry points -- the residual stream, the norms and the
// gates stay f32; what feeds a tensor-core product is written as bf16 by the kernel that produces it --
// and the delta block's prologue in both types.
#include "common.cuh"

#include <cuda_bf16.h>

namespace {

__device__ __forceinline__ uint2 pack4_bf16(float a, float b, float c, float d) {
    const __nv_bfloat162 lo = __floats2bfloat162_rn(a, b), hi = __floats2bfloat162_rn(c, d);
    return make_uint2(*reinterpret_cast<const uint32_t*>(&lo), *reinterpret_cast<const uint32_t*>(&hi));
}

__global__ void __launch_bounds__(256) cast_bf16_kernel(const float* __restrict__ src, __nv_bfloat16* __restrict__ dst,
                                                        int64_t n, int vec) {
    const int64_t n4 = vec ? n >> 2 : 0;
    const int64_t stride = (int64_t)gridDim.x * blockDim.x;
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n4; i += stride) {
        const float4 x = reinterpret_cast<const float4*>(src)[i];
        reinterpret_cast<uint2*>(dst)[i] = pack4_bf16(x.x, x.y, x.z, x.w);
    }
    for (int64_t i = n4 * 4 + (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += stride)
        dst[i] = __float2bfloat16(src[i]);
}

// Warp per row, the row held in registers (cols % 4 == 0, cols <= 128 * NV): x_mid = x (+ res), written
// when xsum is given (xsum may be x itself); xn = bf16(x_mid / sqrt(mean x_mid^2 + eps)), written to row y_row[r]
// when a row map is given (the expert-order position of the row: the MoE gather folded into the norm).
template <int NV>
__global__ void __launch_bounds__(256) rmsnorm_bf16_warp_kernel(const float* x, const float* __restrict__ res,
                                                                float* xsum, __nv_bfloat16* __restrict__ y,
                                                                int64_t rows, int cols, float eps, const int32_t* __restrict__ y_row) {
    const int lane = threadIdx.x & 31;
    const int64_t r = (int64_t)blockIdx.x * 8 + (threadIdx.x >> 5);
    pdl_wait();
    pdl_launch_dependents();
    if (r >= rows) return;
    const float4* xr = reinterpret_cast<const float4*>(x + r * (int64_t)cols);
    const int n4 = cols >> 2;
    float4 v[NV];
#pragma unroll
    for (int i = 0; i < NV; ++i) {
        const int c = lane + 32 * i;
        v[i] = c < n4 ? xr[c] : make_float4(0, 0, 0, 0);
    }
    if (res) {
        const float4* rr = reinterpret_cast<const float4*>(res + r * (int64_t)cols);
#pragma unroll
        for (int i = 0; i < NV; ++i) {
            const int c = lane + 32 * i;
            if (c < n4) {
                const float4 b = rr[c];
                v[i].x += b.x; v[i].y += b.y; v[i].z += b.z; v[i].w += b.w;
            }
        }
    }
    if (xsum) {
        float4* sr = reinterpret_cast<float4*>(xsum + r * (int64_t)cols);
#pragma unroll
        for (int i = 0; i < NV; ++i) {
            const int c = lane + 32 * i;
            if (c < n4) sr[c] = v[i];
        }
    }
    float acc = 0.0f;
#pragma unroll
    for (int i = 0; i < NV; ++i) acc += v[i].x * v[i].x + v[i].y * v[i].y + v[i].z * v[i].z + v[i].w * v[i].w;
    acc = warp_sum(acc);
    const float inv = 1.0f / sqrtf(acc / (float)cols + eps);
    uint2* yr = reinterpret_cast<uint2*>(y + (y_row ? (int64_t)y_row[r] : r) * (int64_t)cols);
#pragma unroll
    for (int i = 0; i < NV; ++i) {
        const int c = lane + 32 * i;
        if (c < n4) yr[c] = pack4_bf16(v[i].x * inv, v[i].y * inv, v[i].z * inv, v[i].w * inv);
    }
}

int residual_rmsnorm_bf16_impl(asca_ctx* ctx, const float* x, const float* yadd, float* x_mid, void* xn, int64_t rows, int64_t cols,
                               float eps, const int32_t* y_row) {
    ASCA_REQUIRE(ctx, x && xn && rows >= 0 && cols > 0, "residual_rmsnorm_bf16: bad arguments");
    ASCA_REQUIRE(ctx, (cols & 3) == 0 && cols <= 2048, "residual_rmsnorm_bf16: cols must be a multiple of 4, at most 2048");
    ASCA_REQUIRE(ctx, ((reinterpret_cast<uintptr_t>(x) | reinterpret_cast<uintptr_t>(yadd) | reinterpret_cast<uintptr_t>(x_mid)) & 15) == 0 &&
                          (reinterpret_cast<uintptr_t>(xn) & 7) == 0, "residual_rmsnorm_bf16: misaligned pointer");
    if (rows == 0) return ASCA_OK;
    const unsigned grid = (unsigned)ceil_div64(rows, 8);
    __nv_bfloat16* y = (__nv_bfloat16*)xn;
    cudaError_t e;
    if (cols <= 512) e = asca_launch(ctx, rmsnorm_bf16_warp_kernel<4>, dim3(grid), dim3(256), 0, x, yadd, x_mid, y, rows, (int)cols, eps, y_row);
    else if (cols <= 1024) e = asca_launch(ctx, rmsnorm_bf16_warp_kernel<8>, dim3(grid), dim3(256), 0, x, yadd, x_mid, y, rows, (int)cols, eps, y_row);
    else e = asca_launch(ctx, rmsnorm_bf16_warp_kernel<16>, dim3(grid), dim3(256), 0, x, yadd, x_mid, y, rows, (int)cols, eps, y_row);
    ASCA_CUDA(ctx, e);
    ctx->launches++;
    return ASCA_OK;
}

// Prologue of the delta block, rust/src/delta.rs:134-179: split, per-head L2 normalise (z / max(|z|, 1e-8)), sigmoids. A
// (row, head) belongs to DH / 4 neighbouring lanes, a float4 of q, k and v each, so that every warp reads and writes whole
// 512-byte (f32) runs whatever the head width. Bound by HBM; with a warp per (row, head) and scalar accesses a prefill's
// 14,448 rows of 12 heads of 64 took 104 us, three times this.
__device__ __forceinline__ void put4(float* p, float a, float b, float c, float d) { *reinterpret_cast<float4*>(p) = make_float4(a, b, c, d); }
__device__ __forceinline__ void put4(__nv_bfloat16* p, float a, float b, float c, float d) { *reinterpret_cast<uint2*>(p) = pack4_bf16(a, b, c, d); }

template <int DH, typename T>
__global__ void __launch_bounds__(256) delta_prep_kernel(const float* __restrict__ qkv, const float* __restrict__ gate, int64_t units, int H,
                                                         T* __restrict__ q, T* __restrict__ k, T* __restrict__ v, float* __restrict__ qn,
                                                         float* __restrict__ kn, float* __restrict__ alpha, float* __restrict__ beta) {
    constexpr int G = DH / 4;   // lanes per unit
    const int64_t u0 = ((int64_t)blockIdx.x * 256 + threadIdx.x) / G;
    const int64_t unit = u0 < units ? u0 : units - 1;   // (a ragged last warp repeats the last unit: its shuffles stay whole)
    const int lane = threadIdx.x % G, h = (int)(unit % H), d = H * DH;
    const int64_t r = unit / H;
    const float* src = qkv + r * 3 * (int64_t)d + h * DH + lane * 4;
    const float4 a = *reinterpret_cast<const float4*>(src), b = *reinterpret_cast<const float4*>(src + d), c = *reinterpret_cast<const float4*>(src + 2 * d);
    float sq = a.x * a.x + a.y * a.y + a.z * a.z + a.w * a.w, sk = b.x * b.x + b.y * b.y + b.z * b.z + b.w * b.w;
#pragma unroll
    for (int m = G / 2; m > 0; m >>= 1) {
        sq += __shfl_xor_sync(0xffffffffu, sq, m);
        sk += __shfl_xor_sync(0xffffffffu, sk, m);
    }
    const float nq = fmaxf(sqrtf(sq), 1e-8f), nk = fmaxf(sqrtf(sk), 1e-8f);
    if (u0 >= units) return;
    const int64_t o = r * (int64_t)d + h * DH + lane * 4;
    put4(q + o, a.x / nq, a.y / nq, a.z / nq, a.w / nq);
    put4(k + o, b.x / nk, b.y / nk, b.z / nk, b.w / nk);
    put4(v + o, c.x, c.y, c.z, c.w);
    if (lane == 0) {
        qn[unit] = nq;
        kn[unit] = nk;
        alpha[unit] = 1.0f / (1.0f + expf(-gate[r * 2 * H + h]));
        beta[unit] = 1.0f / (1.0f + expf(-gate[r * 2 * H + H + h]));
    }
}
// the same for any head width and alignment, one warp per (row, head)
template <typename T>
__global__ void __launch_bounds__(256) delta_prep_any_kernel(const float* __restrict__ qkv, const float* __restrict__ gate, int64_t units, int H,
                                                             int dh, T* __restrict__ q, T* __restrict__ k, T* __restrict__ v,
                                                             float* __restrict__ qn, float* __restrict__ kn, float* __restrict__ alpha,
                                                             float* __restrict__ beta) {
    const int lane = threadIdx.x & 31;
    const int64_t unit = (int64_t)blockIdx.x * 8 + (threadIdx.x >> 5);
    if (unit >= units) return;
    const int64_t r = unit / H;
    const int h = (int)(unit % H);
    const int d = H * dh;
    const float* src = qkv + r * 3 * (int64_t)d + h * dh;
    const int64_t o = r * (int64_t)d + h * dh;
    float sq = 0.0f, sk = 0.0f;
    for (int c = lane; c < dh; c += 32) {
        const float a = src[c], b = src[d + c];
        sq += a * a;
        sk += b * b;
    }
    sq = warp_sum(sq);
    sk = warp_sum(sk);
    const float nq = fmaxf(sqrtf(sq), 1e-8f), nk = fmaxf(sqrtf(sk), 1e-8f);
    for (int c = lane; c < dh; c += 32) {
        q[o + c] = from_f32<T>(src[c] / nq);
        k[o + c] = from_f32<T>(src[d + c] / nk);
        v[o + c] = from_f32<T>(src[2 * d + c]);
    }
    if (lane == 0) {
        qn[unit] = nq;
        kn[unit] = nk;
        alpha[unit] = 1.0f / (1.0f + expf(-gate[r * 2 * H + h]));
        beta[unit] = 1.0f / (1.0f + expf(-gate[r * 2 * H + H + h]));
    }
}

template <typename T>
int delta_prep(asca_ctx* ctx, const float* qkv, const float* gate, int64_t N, int64_t H, int64_t dh, void* q, void* k, void* v, float* qn,
               float* kn, float* alpha, float* beta) {
    ASCA_REQUIRE(ctx, qkv && gate && q && k && v && qn && kn && alpha && beta && N >= 0 && H > 0 && dh > 0, "delta_prep: bad arguments");
    if (N == 0) return ASCA_OK;
    const int64_t units = N * H;
    const uintptr_t out = reinterpret_cast<uintptr_t>(q) | reinterpret_cast<uintptr_t>(k) | reinterpret_cast<uintptr_t>(v);
    const bool vec = (reinterpret_cast<uintptr_t>(qkv) & 15) == 0 && (out & (4 * sizeof(T) - 1)) == 0;
#define ASCA_PREP(DH_)                                                                                                                  \
    delta_prep_kernel<DH_, T><<<(unsigned)ceil_div64(units * (DH_ / 4), 256), 256, 0, ctx->stream>>>(qkv, gate, units, (int)H, (T*)q, (T*)k, \
                                                                                                   (T*)v, qn, kn, alpha, beta)
    if (vec && dh == 128) ASCA_PREP(128);
    else if (vec && dh == 64) ASCA_PREP(64);
    else if (vec && dh == 32) ASCA_PREP(32);
    else if (vec && dh == 16) ASCA_PREP(16);
    else
        delta_prep_any_kernel<T><<<(unsigned)ceil_div64(units, 8), 256, 0, ctx->stream>>>(qkv, gate, units, (int)H, (int)dh, (T*)q, (T*)k, (T*)v,
                                                                                         qn, kn, alpha, beta);
#undef ASCA_PREP
    ASCA_CHECK_LAUNCH(ctx);
    return ASCA_OK;
}

}  // namespace

// residual + RMSNorm whose bf16 rows land in expert order: row r is written to row y_row[r] of xn
int asca_residual_rmsnorm_bf16_rows(asca_ctx* ctx, const float* x, const float* yadd, float* x_mid, void* xn, int64_t rows,
                                    int64_t cols, float eps, const int32_t* y_row) {
    if (!ctx) return ASCA_ERR_ARG;
    return residual_rmsnorm_bf16_impl(ctx, x, yadd, x_mid, xn, rows, cols, eps, y_row);
}

extern "C" {

int asca_cast_bf16(asca_ctx* ctx, const float* src, void* dst, int64_t n) {
    if (!ctx) return ASCA_ERR_ARG;
    ASCA_REQUIRE(ctx, n >= 0 && (n == 0 || (src && dst)), "cast_bf16: bad arguments");
    if (n == 0) return ASCA_OK;
    const int vec = ((reinterpret_cast<uintptr_t>(src) & 15) | (reinterpret_cast<uintptr_t>(dst) & 7)) == 0;
    const int64_t blocks = std::min<int64_t>(ceil_div64((vec ? n >> 2 : n) + 1, 256), 148 * 16);
    cast_bf16_kernel<<<(unsigned)blocks, 256, 0, ctx->stream>>>(src, (__nv_bfloat16*)dst, n, vec);
    ASCA_CHECK_LAUNCH(ctx);
    return ASCA_OK;
}

int asca_residual_rmsnorm_bf16(asca_ctx* ctx, const float* x, const float* yadd, float* x_mid, void* xn, int64_t rows,
                               int64_t cols, float eps) {
    if (!ctx) return ASCA_ERR_ARG;
    return residual_rmsnorm_bf16_impl(ctx, x, yadd, x_mid, xn, rows, cols, eps, nullptr);
}

int asca_delta_prep(asca_ctx* ctx, const float* qkv, const float* gate, int64_t N, int64_t H, int64_t dh, float* q,
                    float* k, float* v, float* qnorm, float* knorm, float* alpha, float* beta) {
    if (!ctx) return ASCA_ERR_ARG;
    return delta_prep<float>(ctx, qkv, gate, N, H, dh, q, k, v, qnorm, knorm, alpha, beta);
}

int asca_delta_prep_bf16(asca_ctx* ctx, const float* qkv, const float* gate, int64_t N, int64_t H, int64_t dh, void* q,
                         void* k, void* v, float* qnorm, float* knorm, float* alpha, float* beta) {
    if (!ctx) return ASCA_ERR_ARG;
    return delta_prep<__nv_bfloat16>(ctx, qkv, gate, N, H, dh, q, k, v, qnorm, knorm, alpha, beta);
}

}  // extern "C"
