// Hash-MoE expert FFN: grouped forward and backward products over the dispatch permutation,
// and the per-token decode step. Math of rust/src/model.rs:237-293 (forward), :417-495
// (backward), :309-337 (step); replaces Gpu::moe_forward_dev / moe_bwd_dev
// (rust/src/cuda/mod.rs:523-607, :745-824), which loop over experts with 7 + 10 launches and
// fresh allocations per expert. Here every product is ONE grouped launch over all experts:
// the row gather is fused into the operand load, bias + SiLU (forward) and SiLU' (backward)
// into the epilogue, and the un-permute scatter into the output store.
#include "gemm_simt.cuh"
#include "gemm_tc.cuh"

bool asca_tc_enabled();  // gemm.cu

namespace {

// Column sums of a bf16 matrix grouped by expert segment: a cluster of 8 CTAs owns 256 columns (a lane eight) of one segment,
// its 64 warps take every 64th row, eight 16-byte loads in flight each, and the partial sums are added in a fixed order
// through distributed shared memory. Bound by reading the matrix. (One CTA a segment left the most frequent expert of a
// skewed load, 13,000 of 65,536 rows, to a single SM for most of the launch: 242 us for 4096 columns, 104 now = 5.2 TB/s.)
constexpr int CS_CLUSTER = 8;
__global__ void __launch_bounds__(256) colsum_bf16_seg_kernel(const __nv_bfloat16* __restrict__ src, int64_t ld,
                                                              const int32_t* __restrict__ offsets, int cols,
                                                              float* __restrict__ out, int64_t out_gstride, int accumulate) {
    __shared__ __align__(16) float part[8][256];
    const int g = blockIdx.y, lane = threadIdx.x & 31, w = threadIdx.x >> 5, rank = blockIdx.z;
    const int64_t lo = offsets[g], hi = offsets[g + 1];
    const int c = blockIdx.x * 256 + 8 * lane;   // (cols is a multiple of 8)
    float acc[8] = {};
    auto add = [&](const uint4& u) {
        const __nv_bfloat162* h = reinterpret_cast<const __nv_bfloat162*>(&u);
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            acc[2 * i] += __low2float(h[i]);
            acc[2 * i + 1] += __high2float(h[i]);
        }
    };
    if (c < cols) {
        constexpr int STEP = 8 * CS_CLUSTER;
        int64_t r = lo + rank * 8 + w;
        for (; r + 7 * STEP < hi; r += 8 * STEP) {
            uint4 v[8];
#pragma unroll
            for (int i = 0; i < 8; ++i) v[i] = __ldg(reinterpret_cast<const uint4*>(src + (r + i * STEP) * ld + c));
#pragma unroll
            for (int i = 0; i < 8; ++i) add(v[i]);
        }
        for (; r < hi; r += STEP) add(__ldg(reinterpret_cast<const uint4*>(src + r * ld + c)));
    }
#pragma unroll
    for (int i = 0; i < 8; ++i) part[w][8 * lane + i] = acc[i];
    __syncthreads();
    float t = 0.0f;
#pragma unroll
    for (int i = 0; i < 8; ++i) t += part[i][threadIdx.x];
    __syncthreads();
    part[0][threadIdx.x] = t;
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
    const int col = blockIdx.x * 256 + threadIdx.x;
    if (rank == 0 && col < cols) {
        float sum = 0.0f;
#pragma unroll
        for (int r = 0; r < CS_CLUSTER; ++r) {
            uint32_t at;
            float x;
            asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(at) : "r"((uint32_t)__cvta_generic_to_shared(&part[0][threadIdx.x])), "r"(r));
            asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(x) : "r"(at));
            sum += x;
        }
        float* o = out + (int64_t)g * out_gstride + col;
        *o = accumulate ? *o + sum : sum;
    }
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");   // peers may still read
}

// Decode step: one CTA per token. rmsnorm -> pre = b1[e] + xn W1[:, e] -> silu -> out = b2 + h W2[e].
template <typename T>
__global__ void __launch_bounds__(256) moe_step_kernel(const float* __restrict__ x, const uint32_t* __restrict__ ids,
                                                       const T* __restrict__ w1, const float* __restrict__ b1,
                                                       const T* __restrict__ w2, const float* __restrict__ b2, int d,
                                                       int F, int E, float* __restrict__ out) {
    extern __shared__ float sh[];  // xn[d] | hid[F] | red[33]
    float* xn = sh;
    float* hid = sh + d;
    float* red = hid + F;
    const int s = blockIdx.x;
    uint32_t h = ids[s] * 0x9E3779B1u;
    h ^= h >> 15;
    h *= 0x85EBCA6Bu;
    h ^= h >> 13;
    const int e = (int)(h % (uint32_t)E);
    const float* xr = x + (int64_t)s * d;
    float acc = 0.0f;
    for (int c = threadIdx.x; c < d; c += blockDim.x) acc += xr[c] * xr[c];
    const float ss = block_sum(acc, red);
    const float inv = 1.0f / sqrtf(ss / (float)d + 1e-6f);
    for (int c = threadIdx.x; c < d; c += blockDim.x) xn[c] = xr[c] * inv;
    __syncthreads();
    const int64_t EF = (int64_t)E * F;
    for (int j = threadIdx.x; j < F; j += blockDim.x) {  // coalesced over j
        float a = b1[(int64_t)e * F + j];
        const T* col = w1 + (int64_t)e * F + j;
        for (int c = 0; c < d; ++c) a = fmaf(xn[c], to_f32<T>(col[(int64_t)c * EF]), a);
        hid[j] = a / (1.0f + expf(-a));
    }
    __syncthreads();
    for (int c = threadIdx.x; c < d; c += blockDim.x) {  // coalesced over c
        float a = b2[c];
        const T* col = w2 + (int64_t)e * F * d + c;
        for (int j = 0; j < F; ++j) a = fmaf(hid[j], to_f32<T>(col[(int64_t)j * d]), a);
        out[(int64_t)s * d + c] = a;
    }
}


// dst[r,:] = src[idx[r],:] for bf16 rows (cols % 8 == 0): 16-byte copies, one warp per row.
__global__ void __launch_bounds__(256) gather_rows_bf16_kernel(const __nv_bfloat16* __restrict__ src,
                                                               const int32_t* __restrict__ idx,
                                                               __nv_bfloat16* __restrict__ dst, int64_t n_rows,
                                                               int cols) {
    const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int64_t r = (int64_t)blockIdx.x * 8 + w;
    pdl_wait();
    pdl_launch_dependents();
    if (r >= n_rows) return;
    const uint4* s = reinterpret_cast<const uint4*>(src + (int64_t)idx[r] * cols);
    uint4* d = reinterpret_cast<uint4*>(dst + r * cols);
    for (int c = lane; c < cols / 8; c += 32) d[c] = s[c];
}
// dst[r,:] = bf16(src[idx[r],:]) for f32 rows (cols % 4 == 0), and the sums of src's columns over the slice of rows this block
// moves (part[slice][cols]): the output bias gradient without a second pass over src (63 + 59 us for 65,536 x 1024 apart,
// 76 us together). A thread owns four columns and has eight rows in flight; bound by HBM.
__global__ void __launch_bounds__(256) gather_colsum_kernel(const float* __restrict__ src, const int32_t* __restrict__ idx,
                                                            __nv_bfloat16* __restrict__ dst, int64_t n_rows, int cols, int64_t per_slice,
                                                            float* __restrict__ part) {
    const int c = 4 * (blockIdx.x * blockDim.x + threadIdx.x);
    if (c >= cols) return;
    const int64_t lo = blockIdx.y * per_slice, hi = min(lo + per_slice, n_rows);
    float4 sum = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    auto put = [&](int64_t r, const float4& v) {
        const __nv_bfloat162 a = __floats2bfloat162_rn(v.x, v.y), b = __floats2bfloat162_rn(v.z, v.w);
        *reinterpret_cast<uint2*>(dst + r * cols + c) = make_uint2(*reinterpret_cast<const uint32_t*>(&a), *reinterpret_cast<const uint32_t*>(&b));
        sum.x += v.x; sum.y += v.y; sum.z += v.z; sum.w += v.w;
    };
    int64_t r = lo;
    for (; r + 8 <= hi; r += 8) {
        float4 v[8];
#pragma unroll
        for (int i = 0; i < 8; ++i) v[i] = __ldg(reinterpret_cast<const float4*>(src + (int64_t)__ldg(idx + r + i) * cols + c));
#pragma unroll
        for (int i = 0; i < 8; ++i) put(r + i, v[i]);
    }
    for (; r < hi; ++r) put(r, __ldg(reinterpret_cast<const float4*>(src + (int64_t)__ldg(idx + r) * cols + c)));
    *reinterpret_cast<float4*>(part + (int64_t)blockIdx.y * cols + c) = sum;
}
// out[c] (+)= the slices' sums, in a fixed order: 32 columns a block, 32 threads a column
__global__ void __launch_bounds__(1024) colsum_parts_kernel(const float* __restrict__ part, int slices, int cols, float* __restrict__ out, int accumulate) {
    __shared__ float sh[32][33];
    const int x = threadIdx.x & 31, y = threadIdx.x >> 5, c = blockIdx.x * 32 + x;
    float a = 0.0f;
    if (c < cols) {
#pragma unroll 8
        for (int i = y; i < slices; i += 32) a += part[(int64_t)i * cols + c];
    }
    sh[y][x] = a;
    __syncthreads();
    if (y == 0 && c < cols) {
        float t = 0.0f;
#pragma unroll
        for (int i = 0; i < 32; ++i) t += sh[i][x];
        out[c] = accumulate ? out[c] + t : t;
    }
}

inline bool tc_shapes_ok(int64_t d, int64_t F) { return asca_tc_enabled() && d % 64 == 0 && F % 64 == 0; }

inline size_t align256(size_t x) { return (x + 255) & ~(size_t)255; }

// Tensor-core forward: permute xn once, then two grouped tcgen05 GEMMs. pre_p null: the pre-activations are not kept.
// res (may be out; null: nothing) is added in the second product's epilogue and out16 (nullable) takes a bf16 copy of the sum.
int moe_fwd_tc(asca_ctx* ctx, const __nv_bfloat16* xn, const __nv_bfloat16* w1, const float* b1,
               const __nv_bfloat16* w2, const float* b2, const int32_t* perm, const int32_t* offsets, int64_t N,
               int64_t d, int64_t F, int64_t E, const float* res, float* out, __nv_bfloat16* out16, float* pre_p, __nv_bfloat16* hid_p) {
    void* ws;
    ASCA_TRY(asca_workspace(ctx, align256((size_t)N * d * 2) + 256, &ws));
    __nv_bfloat16* xp = (__nv_bfloat16*)ws;
    gemm_tc::Args a{};
    a.mode = ASCA_NN;
    a.A = xp; a.lda = d; a.a_rows = N; a.a_cols = d;
    a.B = w1; a.ldb = E * F; a.b_rows = d; a.b_cols = E * F; a.b_goff_inner = (int)F;
    a.C = pre_p; a.ldc = F; a.N = (int)F; a.K = (int)d;
    a.bias = b1; a.bias_gstride = F;
    a.offsets = offsets; a.n_groups = (int)E; a.group_dim = gemm_tc::GROUP_M; a.total_rows = N;
    a.epi = gemm_tc::EPI_SILU; a.C2 = hid_p; a.ldc2 = F; a.c2_only = pre_p == nullptr;
    gemm_tc::Args b{};
    b.mode = ASCA_NN;
    b.A = hid_p; b.lda = F; b.a_rows = N; b.a_cols = F;
    b.B = w2; b.ldb = d; b.b_rows = E * F; b.b_cols = d; b.b_goff_outer = (int)F;
    b.C = out; b.ldc = d; b.N = (int)d; b.K = (int)F; b.c_idx = perm;
    b.accumulate = res != nullptr; b.res = res == out ? nullptr : res;
    b.C2 = out16; b.ldc2 = d; b.c2_mapped = out16 != nullptr;
    b.bias = b2; b.bias_gstride = 0;
    b.offsets = offsets; b.n_groups = (int)E; b.group_dim = gemm_tc::GROUP_M; b.total_rows = N;
    // nothing is launched unless the gather (16-byte copies) and every product can run here: the caller falls back as a whole
    if ((reinterpret_cast<uintptr_t>(xn) & 15) || !gemm_tc::supported(a) || !gemm_tc::supported(b)) return ASCA_ERR_UNSUPPORTED;
    ASCA_CUDA(ctx, asca_launch(ctx, gather_rows_bf16_kernel, dim3((unsigned)ceil_div64(N, 8)), dim3(256), 0, xn, perm, xp, N, (int)d));
    ctx->launches++;
    ASCA_TRY(gemm_tc::launch(ctx, a));
    return gemm_tc::launch(ctx, b);
}

// Tensor-core backward: permuted bf16 copies of xn and dout, then four grouped tcgen05 GEMMs.
int moe_bwd_tc(asca_ctx* ctx, const __nv_bfloat16* xn, const __nv_bfloat16* w1, const __nv_bfloat16* w2,
               const float* pre_p, const __nv_bfloat16* hid_p, const float* dout, const int32_t* perm,
               const int32_t* offsets, int64_t N, int64_t d, int64_t F, int64_t E, float* d_w1, float* d_b1,
               float* d_w2, float* d_b2, float* dxn, int acc) {
    cudaStream_t s = ctx->stream;
    const size_t b_xp = align256((size_t)N * d * 2), b_dp16 = align256((size_t)N * F * 2);
    void* ws;
    // slices of rows for the bias gradient: four blocks an SM, 32 rows at least
    const int threads = (int)std::min<int64_t>(256, ceil_div64(d / 4, 32) * 32);
    const int64_t col_blocks = ceil_div64(d, 4 * threads);
    const int64_t per_slice = std::max<int64_t>(32, ceil_div64(N, std::max<int64_t>(1, 4 * (ctx->sm_count > 0 ? ctx->sm_count : 148) / col_blocks)));
    const int64_t slices = ceil_div64(N, per_slice);
    const size_t b_part = align256((size_t)slices * d * 4);
    ASCA_TRY(asca_workspace(ctx, 2 * b_xp + b_dp16 + b_part + 256, &ws));
    char* w = (char*)ws;
    float* part = (float*)(w + 2 * b_xp + b_dp16);
    __nv_bfloat16* xp = (__nv_bfloat16*)w;
    __nv_bfloat16* dout_p = (__nv_bfloat16*)(w + b_xp);
    __nv_bfloat16* dpre16 = (__nv_bfloat16*)(w + 2 * b_xp);
    gemm_tc::Args g1{}, g2{}, g3{}, g4{};
    // d_w2[eF+j, c] = sum_r hid_p[r,j] dout_p[r,c]
    g1.mode = ASCA_TN;
    g1.A = hid_p; g1.lda = F; g1.a_rows = N; g1.a_cols = F;
    g1.B = dout_p; g1.ldb = d; g1.b_rows = N; g1.b_cols = d;
    g1.C = d_w2; g1.ldc = d; g1.c_gstride = F * d; g1.M = (int)F; g1.N = (int)d; g1.accumulate = acc;
    g1.offsets = offsets; g1.n_groups = (int)E; g1.group_dim = gemm_tc::GROUP_K; g1.total_rows = N;
    // dpre16[r,j] = (sum_c dout_p[r,c] W2[eF+j,c]) * silu'(pre_p[r,j]), written as bf16 only: the weight-gradient product
    // below reads bf16, and the bias gradient sums the same rounded values
    g2.mode = ASCA_NT;
    g2.A = dout_p; g2.lda = d; g2.a_rows = N; g2.a_cols = d;
    g2.B = w2; g2.ldb = d; g2.b_rows = E * F; g2.b_cols = d; g2.b_goff_outer = (int)F;
    g2.C = nullptr; g2.ldc = F; g2.N = (int)F; g2.K = (int)d; g2.c2_only = 1;
    g2.offsets = offsets; g2.n_groups = (int)E; g2.group_dim = gemm_tc::GROUP_M; g2.total_rows = N;
    g2.epi = gemm_tc::EPI_SILU_BWD; g2.aux = pre_p; g2.ldaux = F; g2.C2 = dpre16; g2.ldc2 = F;
    // d_w1[c, eF+j] = sum_r xp[r,c] dpre16[r,j]
    g3.mode = ASCA_TN;
    g3.A = xp; g3.lda = d; g3.a_rows = N; g3.a_cols = d;
    g3.B = dpre16; g3.ldb = F; g3.b_rows = N; g3.b_cols = F;
    g3.C = d_w1; g3.ldc = E * F; g3.c_gstride = F; g3.M = (int)d; g3.N = (int)F; g3.accumulate = acc;
    g3.offsets = offsets; g3.n_groups = (int)E; g3.group_dim = gemm_tc::GROUP_K; g3.total_rows = N;
    // dxn[perm[r], c] = sum_j dpre16[r,j] W1[c, eF+j]
    g4.mode = ASCA_NT;
    g4.A = dpre16; g4.lda = F; g4.a_rows = N; g4.a_cols = F;
    g4.B = w1; g4.ldb = E * F; g4.b_rows = d; g4.b_cols = E * F; g4.b_goff_inner = (int)F;
    g4.C = dxn; g4.ldc = d; g4.N = (int)d; g4.K = (int)F; g4.c_idx = perm;
    g4.offsets = offsets; g4.n_groups = (int)E; g4.group_dim = gemm_tc::GROUP_M; g4.total_rows = N;
    // nothing is launched unless the gathers (16-byte loads) and every product can run here: the caller falls back as a whole,
    // and with `acc` a partial run followed by the fallback would add some gradients twice
    if (((reinterpret_cast<uintptr_t>(xn) | reinterpret_cast<uintptr_t>(dout)) & 15) != 0) return ASCA_ERR_UNSUPPORTED;
    if (!gemm_tc::supported(g1) || !gemm_tc::supported(g2) || !gemm_tc::supported(g3) || !gemm_tc::supported(g4))
        return ASCA_ERR_UNSUPPORTED;
    gather_rows_bf16_kernel<<<(unsigned)ceil_div64(N, 8), 256, 0, s>>>(xn, perm, xp, N, (int)d);
    ASCA_CHECK_LAUNCH(ctx);
    gather_colsum_kernel<<<dim3((unsigned)col_blocks, (unsigned)slices), threads, 0, s>>>(dout, perm, dout_p, N, (int)d, per_slice, part);
    ASCA_CHECK_LAUNCH(ctx);
    colsum_parts_kernel<<<(unsigned)ceil_div64(d, 32), 1024, 0, s>>>(part, (int)slices, (int)d, d_b2, acc);
    ASCA_CHECK_LAUNCH(ctx);
    ASCA_TRY(gemm_tc::launch(ctx, g1));
    ASCA_TRY(gemm_tc::launch(ctx, g2));
    {
        cudaLaunchConfig_t cfg = {};
        cfg.gridDim = dim3((unsigned)ceil_div64(F, 256), (unsigned)E, CS_CLUSTER);
        cfg.blockDim = dim3(256);
        cfg.stream = s;
        cudaLaunchAttribute at[1];
        at[0].id = cudaLaunchAttributeClusterDimension;
        at[0].val.clusterDim.x = at[0].val.clusterDim.y = 1;
        at[0].val.clusterDim.z = CS_CLUSTER;
        cfg.attrs = at;
        cfg.numAttrs = 1;
        ASCA_CUDA(ctx, cudaLaunchKernelEx(&cfg, colsum_bf16_seg_kernel, (const __nv_bfloat16*)dpre16, F, offsets, (int)F, d_b1, F, acc));
    }
    ASCA_CHECK_LAUNCH(ctx);
    ASCA_TRY(gemm_tc::launch(ctx, g3));
    return gemm_tc::launch(ctx, g4);
}

// The two FFMA products; res (nullable, (N, d)): added to the output rows.
int moe_fwd_simt(asca_ctx* ctx, const void* xn, const void* w1, const float* b1, const void* w2, const float* b2, const int32_t* perm,
                 const int32_t* offsets, int64_t N, int64_t d, int64_t F, int64_t E, int bf, const float* res, float* out, float* pre_p,
                 void* hid_p) {
    // pre_p[r,:] = xn[perm[r],:] W1[:, eF:(e+1)F] + b1[e];  hid_p = silu(pre_p)
    gemm::Params p{};
    p.A = xn; p.lda = d; p.a_idx = perm;
    p.B = w1; p.ldb = E * F; p.b_gstride = F;
    p.C = pre_p; p.ldc = F;
    p.M = 0; p.N = (int)F; p.K = (int)d;
    p.bias = b1; p.bias_gstride = F;
    p.offsets = offsets; p.n_groups = (int)E; p.group_dim = gemm::GROUP_M;
    p.epi = gemm::EPI_SILU; p.C2 = hid_p; p.ldc2 = F;
    p.mode = ASCA_NN; p.total_rows = N;
    if (bf) ASCA_CUDA(ctx, gemm::launch<__nv_bfloat16>(ctx, p, 1, 1));
    else ASCA_CUDA(ctx, gemm::launch<float>(ctx, p, 0, 0));
    ctx->launches++;
    // out[perm[r],:] = hid_p[r,:] W2[eF:(e+1)F,:] + b2
    gemm::Params q{};
    q.A = hid_p; q.lda = F;
    q.B = w2; q.ldb = d; q.b_gstride = F * d;
    q.C = out; q.ldc = d; q.c_idx = perm;
    q.res = res;
    q.M = 0; q.N = (int)d; q.K = (int)F;
    q.bias = b2; q.bias_gstride = 0;
    q.offsets = offsets; q.n_groups = (int)E; q.group_dim = gemm::GROUP_M;
    q.epi = gemm::EPI_NONE;
    q.mode = ASCA_NN; q.total_rows = N;
    ASCA_CUDA(ctx, gemm::launch<float>(ctx, q, bf, bf));
    ctx->launches++;
    return ASCA_OK;
}

}  // namespace

// bf16 forward with the residual add in the second product's epilogue: out = res + moe(xn) (out may be res), and its bf16 copy in
// out16 (nullable). pre_p null: the pre-activations are not kept (no backward follows: a third of the first product's epilogue
// and two thirds of its bytes). ASCA_ERR_UNSUPPORTED, nothing launched, where the tensor-core products cannot run; the caller
// then uses asca_moe_fwd and adds.
int asca_moe_fwd_bf16_residual(asca_ctx* ctx, const __nv_bfloat16* xn, const __nv_bfloat16* w1, const float* b1, const __nv_bfloat16* w2, const float* b2,
                            const int32_t* perm, const int32_t* offsets, int64_t N, int64_t d, int64_t F, int64_t E, const float* res, float* out,
                               __nv_bfloat16* out16, float* pre_p, __nv_bfloat16* hid_p) {
    if (!tc_shapes_ok(d, F)) return ASCA_ERR_UNSUPPORTED;
    return moe_fwd_tc(ctx, xn, w1, b1, w2, b2, perm, offsets, N, d, F, E, res, out, out16, pre_p, hid_p);
}

// f32 forward with the residual add in the second product's store: out = res + moe(xn)
int asca_moe_fwd_f32_residual(asca_ctx* ctx, const float* xn, const float* w1, const float* b1, const float* w2, const float* b2,
                              const int32_t* perm, const int32_t* offsets, int64_t N, int64_t d, int64_t F, int64_t E, const float* res,
                              float* out, float* pre_p, float* hid_p) {
    return moe_fwd_simt(ctx, xn, w1, b1, w2, b2, perm, offsets, N, d, F, E, 0, res, out, pre_p, hid_p);
}

// Decode-step form of the layer, on bf16 rows already in expert order: x[perm[r], :] += silu(xp[r] W1_e + b1_e) W2_e + b2
// in place on the f32 residual rows, with a bf16 copy of the updated rows in x16. Two launches of the few-row
// kernel; ASCA_ERR_UNSUPPORTED (nothing launched) when that kernel does not take the shapes. check_only: launch nothing.
// packed: w1 and w2 point to the experts' weights in the kernel's streaming order (gemm_tc::skinny_pack).
int asca_moe_fwd_sorted_residual(asca_ctx* ctx, const __nv_bfloat16* xp, const __nv_bfloat16* w1, const float* b1,
                                 const __nv_bfloat16* w2, const float* b2, const int32_t* perm, const int32_t* offsets, int64_t N,
                                 int64_t d, int64_t F, int64_t E, float* x, __nv_bfloat16* x16, __nv_bfloat16* hid_p, int check_only,
                                 int packed) {
    if (!tc_shapes_ok(d, F) || N <= 0) return ASCA_ERR_UNSUPPORTED;
    gemm_tc::Args a{};
    a.mode = ASCA_NN;
    a.A = xp; a.lda = d; a.a_rows = N; a.a_cols = d;
    a.B = w1; a.ldb = E * F; a.b_rows = d; a.b_cols = E * F; a.b_goff_inner = (int)F;
    a.C = nullptr; a.ldc = F; a.N = (int)F; a.K = (int)d;
    a.bias = b1; a.bias_gstride = F;
    a.offsets = offsets; a.n_groups = (int)E; a.group_dim = gemm_tc::GROUP_M; a.total_rows = N;
    a.epi = gemm_tc::EPI_SILU; a.C2 = hid_p; a.ldc2 = F;
    gemm_tc::Args b{};
    b.mode = ASCA_NN;
    b.A = hid_p; b.lda = F; b.a_rows = N; b.a_cols = F;
    b.B = w2; b.ldb = d; b.b_rows = E * F; b.b_cols = d; b.b_goff_outer = (int)F;
    b.C = x; b.ldc = d; b.N = (int)d; b.K = (int)F; b.c_idx = perm; b.accumulate = 1;
    b.bias = b2; b.bias_gstride = 0;
    b.offsets = offsets; b.n_groups = (int)E; b.group_dim = gemm_tc::GROUP_M; b.total_rows = N;
    b.C2 = x16; b.ldc2 = d; b.c2_mapped = 1;
    a.b_early = b.b_early = 1;   // weights and the dispatch tables predate the kernel before each product
    if (packed) {   // w1 / w2 are skinny_pack buffers of the E expert matrices
        a.b_packed = 1; a.ldb = 64; a.b_cols = 64; a.b_rows = gemm_tc::skinny_packed_rows(E, d, F); a.b_goff_inner = 0;
        b.b_packed = 1; b.ldb = 64; b.b_cols = 64; b.b_rows = gemm_tc::skinny_packed_rows(E, F, d); b.b_goff_outer = 0;
    }
    if (!gemm_tc::skinny_wanted(a) || !gemm_tc::skinny_wanted(b) || !gemm_tc::supported(a) || !gemm_tc::supported(b))
        return ASCA_ERR_UNSUPPORTED;
    if (check_only) return ASCA_OK;
    ASCA_TRY(gemm_tc::launch_skinny(ctx, a));
    return gemm_tc::launch_skinny(ctx, b);
}

extern "C" {

int asca_moe_fwd(asca_ctx* ctx, const void* xn, const void* w1, const float* b1, const void* w2, const float* b2,
                 const int32_t* perm, const int32_t* offsets, int64_t N, int64_t d, int64_t F, int64_t E, int dtype,
                 float* out, float* pre_p, void* hid_p) {
    if (!ctx) return ASCA_ERR_ARG;
    ASCA_REQUIRE(ctx, xn && w1 && b1 && w2 && b2 && perm && offsets && out && pre_p && hid_p, "moe_fwd: null pointer");
    ASCA_REQUIRE(ctx, N >= 0 && d > 0 && F > 0 && E > 0 && N < (1ll << 31) && E * F < (1ll << 31), "moe_fwd: bad shape");
    ASCA_REQUIRE(ctx, dtype == ASCA_F32 || dtype == ASCA_BF16, "moe_fwd: unknown dtype");
    if (N == 0) return ASCA_OK;
    const int bf = dtype == ASCA_BF16;
    if (bf && tc_shapes_ok(d, F)) {
        const int rc = moe_fwd_tc(ctx, (const __nv_bfloat16*)xn, (const __nv_bfloat16*)w1, b1, (const __nv_bfloat16*)w2, b2,
                            perm, offsets, N, d, F, E, nullptr, out, nullptr, pre_p, (__nv_bfloat16*)hid_p);
        if (rc != ASCA_ERR_UNSUPPORTED) return rc;
    }
    return moe_fwd_simt(ctx, xn, w1, b1, w2, b2, perm, offsets, N, d, F, E, bf, nullptr, out, pre_p, hid_p);
}

static int moe_bwd_impl(asca_ctx* ctx, const void* xn, const void* w1, const void* w2, const float* pre_p, const void* hid_p,
                        const float* dout, const int32_t* perm, const int32_t* offsets, int64_t N, int64_t d, int64_t F,
                        int64_t E, int dtype, float* d_w1, float* d_b1, float* d_w2, float* d_b2, float* dxn, int acc) {
    if (!ctx) return ASCA_ERR_ARG;
    ASCA_REQUIRE(ctx, xn && w1 && w2 && pre_p && hid_p && dout && perm && offsets && d_w1 && d_b1 && d_w2 && d_b2 && dxn,
                 "moe_bwd: null pointer");
    ASCA_REQUIRE(ctx, N >= 0 && d > 0 && F > 0 && E > 0 && N < (1ll << 31) && E * F < (1ll << 31), "moe_bwd: bad shape");
    ASCA_REQUIRE(ctx, dtype == ASCA_F32 || dtype == ASCA_BF16, "moe_bwd: unknown dtype");
    const int bf = dtype == ASCA_BF16;
    cudaStream_t s = ctx->stream;
    if (N == 0 && acc) return ASCA_OK;
    if (N == 0) {
        ASCA_CUDA(ctx, cudaMemsetAsync(d_w1, 0, (size_t)(d * E * F) * 4, s));
        ASCA_CUDA(ctx, cudaMemsetAsync(d_w2, 0, (size_t)(d * E * F) * 4, s));
        ASCA_CUDA(ctx, cudaMemsetAsync(d_b1, 0, (size_t)(E * F) * 4, s));
        ASCA_CUDA(ctx, cudaMemsetAsync(d_b2, 0, (size_t)d * 4, s));
        return ASCA_OK;
    }
    if (bf && tc_shapes_ok(d, F)) {
        int rc = moe_bwd_tc(ctx, (const __nv_bfloat16*)xn, (const __nv_bfloat16*)w1, (const __nv_bfloat16*)w2, pre_p,
                            (const __nv_bfloat16*)hid_p, dout, perm, offsets, N, d, F, E, d_w1, d_b1, d_w2, d_b2, dxn, acc);
        if (rc != ASCA_ERR_UNSUPPORTED) return rc;
    }
    // scratch: dpre_p (N x F) f32, in the permuted order
    void* ws;
    ASCA_TRY(asca_workspace(ctx, (size_t)N * F * 4 + 256, &ws));
    float* dpre_p = (float*)ws;

    // first launch: d_b2, d_w2 and dpre_p, which read dout only
    gemm::Params db2{};   // d_b2[c] = sum over all tokens of dout[t,c]
    db2.mode = ASCA_TN; db2.B = dout; db2.ldb = d; db2.N = (int)d; db2.K = (int)N;
    db2.colsum = d_b2; db2.accumulate = acc;
    gemm::Params dw2{};   // d_w2[eF+j, c] = sum_r hid_p[r,j] dout[perm[r],c]      (TN, K = rows of expert e)
    dw2.mode = ASCA_TN;
    dw2.A = hid_p; dw2.lda = F;
    dw2.B = dout; dw2.ldb = d; dw2.b_idx = perm;
    dw2.C = d_w2; dw2.ldc = d; dw2.c_gstride = F * d; dw2.accumulate = acc;
    dw2.M = (int)F; dw2.N = (int)d;
    dw2.offsets = offsets; dw2.n_groups = (int)E; dw2.group_dim = gemm::GROUP_K; dw2.total_rows = N;
    gemm::Params dpre{};  // dpre_p[r,j] = (sum_c dout[perm[r],c] W2[eF+j,c]) * silu'(pre_p[r,j])   (NT)
    dpre.mode = ASCA_NT;
    dpre.A = dout; dpre.lda = d; dpre.a_idx = perm;
    dpre.B = w2; dpre.ldb = d; dpre.b_gstride = F * d;
    dpre.C = dpre_p; dpre.ldc = F;
    dpre.N = (int)F; dpre.K = (int)d;
    dpre.offsets = offsets; dpre.n_groups = (int)E; dpre.group_dim = gemm::GROUP_M; dpre.total_rows = N;
    dpre.epi = gemm::EPI_SILU_BWD; dpre.aux = pre_p; dpre.ldaux = F;
    // second launch: d_w1 with d_b1 beside it, and dxn, which read dpre_p
    gemm::Params dw1{};   // d_w1[c, eF+j] = sum_r xn[perm[r],c] dpre_p[r,j];  d_b1[eF+j] = sum_r dpre_p[r,j]   (TN)
    dw1.mode = ASCA_TN;
    dw1.A = xn; dw1.lda = d; dw1.a_idx = perm;
    dw1.B = dpre_p; dw1.ldb = F;
    dw1.C = d_w1; dw1.ldc = E * F; dw1.c_gstride = F; dw1.accumulate = acc;
    dw1.M = (int)d; dw1.N = (int)F;
    dw1.offsets = offsets; dw1.n_groups = (int)E; dw1.group_dim = gemm::GROUP_K; dw1.total_rows = N;
    dw1.colsum = d_b1; dw1.colsum_gstride = F;
    gemm::Params dx{};    // dxn[perm[r], c] = sum_j dpre_p[r,j] W1[c, eF+j]          (NT)
    dx.mode = ASCA_NT;
    dx.A = dpre_p; dx.lda = F;
    dx.B = w1; dx.ldb = E * F; dx.b_gstride = F;
    dx.C = dxn; dx.ldc = d; dx.c_idx = perm;
    dx.N = (int)d; dx.K = (int)F;
    dx.offsets = offsets; dx.n_groups = (int)E; dx.group_dim = gemm::GROUP_M; dx.total_rows = N;
    if (!bf) {
        gemm::Multi m{};
        m.n = 3;
        m.p[0] = dw2; m.p[1] = dpre; m.p[2] = db2;
        ASCA_CUDA(ctx, gemm::launch_f32(ctx, m));
        m.n = 2;
        m.p[0] = dw1; m.p[1] = dx;
        ASCA_CUDA(ctx, gemm::launch_f32(ctx, m));
        ctx->launches += 2;
        return ASCA_OK;
    }
    ASCA_CUDA(ctx, gemm::launch<float>(ctx, db2, 0, 0));
    ASCA_CUDA(ctx, gemm::launch<float>(ctx, dw2, 1, 0));
    ASCA_CUDA(ctx, gemm::launch<float>(ctx, dpre, 0, 1));
    ASCA_CUDA(ctx, gemm::launch<float>(ctx, dw1, 1, 0));
    ASCA_CUDA(ctx, gemm::launch<float>(ctx, dx, 0, 1));
    ctx->launches += 5;
    return ASCA_OK;
}

int asca_moe_bwd(asca_ctx* ctx, const void* xn, const void* w1, const void* w2, const float* pre_p, const void* hid_p,
                 const float* dout, const int32_t* perm, const int32_t* offsets, int64_t N, int64_t d, int64_t F,
                 int64_t E, int dtype, float* d_w1, float* d_b1, float* d_w2, float* d_b2, float* dxn) {
    return moe_bwd_impl(ctx, xn, w1, w2, pre_p, hid_p, dout, perm, offsets, N, d, F, E, dtype, d_w1, d_b1, d_w2, d_b2, dxn, 0);
}

int asca_moe_bwd_acc(asca_ctx* ctx, const void* xn, const void* w1, const void* w2, const float* pre_p, const void* hid_p,
                     const float* dout, const int32_t* perm, const int32_t* offsets, int64_t N, int64_t d, int64_t F,
                     int64_t E, int dtype, float* d_w1, float* d_b1, float* d_w2, float* d_b2, float* dxn) {
    return moe_bwd_impl(ctx, xn, w1, w2, pre_p, hid_p, dout, perm, offsets, N, d, F, E, dtype, d_w1, d_b1, d_w2, d_b2, dxn, 1);
}

int asca_moe_step(asca_ctx* ctx, const float* x, const uint32_t* ids, const void* w1, const float* b1, const void* w2,
                  const float* b2, int64_t n_streams, int64_t d, int64_t F, int64_t E, int dtype, float* out) {
    if (!ctx) return ASCA_ERR_ARG;
    ASCA_REQUIRE(ctx, x && ids && w1 && b1 && w2 && b2 && out && n_streams >= 0 && d > 0 && F > 0 && E > 0,
                 "moe_step: bad arguments");
    ASCA_REQUIRE(ctx, dtype == ASCA_F32 || dtype == ASCA_BF16, "moe_step: unknown dtype");
    if (n_streams == 0) return ASCA_OK;
    const size_t smem = (size_t)(d + F + 33) * 4;
    ASCA_REQUIRE(ctx, smem <= 200 * 1024, "moe_step: d + F too large for one CTA");
    if (dtype == ASCA_BF16) {
        auto kern = moe_step_kernel<__nv_bfloat16>;
        if (smem > 48 * 1024) ASCA_CUDA(ctx, cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
        kern<<<(unsigned)n_streams, 256, smem, ctx->stream>>>(x, ids, (const __nv_bfloat16*)w1, b1,
                                                              (const __nv_bfloat16*)w2, b2, (int)d, (int)F, (int)E, out);
    } else {
        auto kern = moe_step_kernel<float>;
        if (smem > 48 * 1024) ASCA_CUDA(ctx, cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
        kern<<<(unsigned)n_streams, 256, smem, ctx->stream>>>(x, ids, (const float*)w1, b1, (const float*)w2, b2, (int)d,
                                                              (int)F, (int)E, out);
    }
    ASCA_CHECK_LAUNCH(ctx);
    return ASCA_OK;
}

}  // extern "C"
