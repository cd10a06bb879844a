// Gated delta rule, bf16 mode: chunk-parallel WY/UT form on the 5th-generation tensor cores, head dim 128 or 64.
//
// Chunk of C = 64 tokens, state S (DH x DH, key x value) in f32 in TMEM for the whole sequence. With g = cumsum(log alpha) inside
// a chunk, gam = exp(g), Gam[t,i] = exp(g_t - g_i), eg = exp(g_C - g), everything that depends on neither S nor dS is taken off the
// two serial chains:
//
//   delta_prep_tc_kernel   one CTA per (chunk, chain)
//     L = strictlower(beta_t Gam K K^T), A = lower(Gam Q K^T), X = (I + L)^-1 (f32), W^ = X diag(beta gam) K, Uv = X diag(beta) V
//   delta_fwd_tc_kernel    one CTA per chain, two dependent products a chunk
//     U = Uv - W^ S          S <- gam_C S + K^T (eg U)          o = gam (Q S) + A U      (o off the serial path)
//   delta_bwd_tc_kernel    one CTA per chain in reverse, three dependent products a chunk
//     dU = A^T dO + eg (K dS)    dR = X^T dU    dS <- gam_C dS + Q^T (gam dO) - K^T (beta gam dR)    dv = beta dR    <S, dS>    dv . (S^T k)
//   delta_grad_tc_kernel   one CTA per (chunk, chain): dq, dk and the gate gradients from S, dS, U and dR, see its header
//
// Row factors (gam, eg, beta) are applied in f32 to results or to the rows of a 64-row operand just before it is rounded, never
// to copies of q, k, v: the kernels read those straight from the caller's tensors, and what travels between them per (chunk, chain) is
// W^, Uv, A, X - I (56 KB at DH 128) and, for a backward, S, U (in the checkpoint buffer) and dS, dR. A travels as two bf16
// tiles, value and remainder: the rounding of an entry of A meets a whole row of U or dO, an error common to 128 columns that was most of
// what the gate gradients and o's sums over heads had. Sums over dS and dR are taken in the chain, where these are f32.
//
// Tiles arrive by TMA (plain loads, 128-byte swizzle); a box that runs past a sequence's end is filled with zeros. Many products have
// 64 rows: they either run as M = 128 with whatever lies behind the operand as rows 64 - 127 (the results of those rows land
// in TMEM lanes that nobody reads; an M = 64 instruction takes as long), or as two M = 64 products in the two 16-lane halves of
// each TMEM lane quarter.
//
// Every mbarrier wait is bounded (tc::mbar_wait): a wait that runs out sets the context's error
// word, and the CTA still frees its TMEM and exits.
#include "common.cuh"
#include "tc_common.cuh"

namespace delta_tc {

constexpr int C = 64;     // chunk length

// Intermediate buffers, one tile per (chain, chunk), DH wide; and per-token vectors.
struct Tiles {
    __nv_bfloat16* WH;    // [tile][64][DH]  W^
    __nv_bfloat16* UV;    // [tile][64][DH]  Uv
    __nv_bfloat16* AA;    // [tile][64][64]  A
    __nv_bfloat16* AL;    // [tile][64][64]  what A loses in bf16, itself bf16
    __nv_bfloat16* TP;    // [tile][64][64]  X - I (null without a backward)
    float* GB;            // [tile][64], [64] cumulative log alpha (constant past the sequence's end), beta (0 there)
};

// 512 bytes (a tile's row of GB) into shared memory
__device__ __forceinline__ void load_vec(void* dst, const float* src, uint64_t* bar) {
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], 512, [%2];"
                 ::"r"(tc::smem_u32(dst)), "l"(src), "r"(tc::smem_u32(bar))
                 : "memory");
}
// __expf, taken whatever becomes of it: the compiler does not move it under a condition
__device__ __forceinline__ float exp_always(float x) {
    float y = __expf(x);
    asm volatile("" : "+f"(y));
    return y;
}
// 32 columns of a row, 32 bytes at a time where the rows lie on that grid
__device__ __forceinline__ void store32(float* p, const float (&v)[32], bool w32) {
    if (w32) {
#pragma unroll
        for (int j = 0; j < 32; j += 8)
            asm volatile("st.global.v8.f32 [%8], {%0, %1, %2, %3, %4, %5, %6, %7};"
                         ::"f"(v[j]), "f"(v[j + 1]), "f"(v[j + 2]), "f"(v[j + 3]), "f"(v[j + 4]), "f"(v[j + 5]), "f"(v[j + 6]), "f"(v[j + 7]), "l"(p + j)
                         : "memory");
    } else {
#pragma unroll
        for (int j = 0; j < 32; j += 4) *reinterpret_cast<float4*>(p + j) = make_float4(v[j], v[j + 1], v[j + 2], v[j + 3]);
    }
}
__device__ __forceinline__ void store16(float* p, const float (&v)[16], bool w32) {
    if (w32) {
#pragma unroll
        for (int j = 0; j < 16; j += 8)
            asm volatile("st.global.v8.f32 [%8], {%0, %1, %2, %3, %4, %5, %6, %7};"
                         ::"f"(v[j]), "f"(v[j + 1]), "f"(v[j + 2]), "f"(v[j + 3]), "f"(v[j + 4]), "f"(v[j + 5]), "f"(v[j + 6]), "f"(v[j + 7]), "l"(p + j)
                         : "memory");
    } else {
#pragma unroll
        for (int j = 0; j < 16; j += 4) *reinterpret_cast<float4*>(p + j) = make_float4(v[j], v[j + 1], v[j + 2], v[j + 3]);
    }
}
__device__ __forceinline__ void store32_bf16(__nv_bfloat16* p, const float (&v)[32], bool w32) {
    uint4 h[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) h[j] = tc::pack8_bf16(v + 8 * j);
    if (w32) {
#pragma unroll
        for (int j = 0; j < 4; j += 2)
            asm volatile("st.global.v8.b32 [%8], {%0, %1, %2, %3, %4, %5, %6, %7};"
                         ::"r"(h[j].x), "r"(h[j].y), "r"(h[j].z), "r"(h[j].w), "r"(h[j + 1].x), "r"(h[j + 1].y), "r"(h[j + 1].z), "r"(h[j + 1].w), "l"(p + 8 * j)
                         : "memory");
    } else {
#pragma unroll
        for (int j = 0; j < 4; ++j) reinterpret_cast<uint4*>(p)[j] = h[j];
    }
}

// ------------------------------------------------------------------ pre-pass
constexpr int PRE_THREADS = 256;
// The f32 matrices L and X are lower triangular: their ten 16 x 16 blocks are kept side by side, rows 20 floats apart (float4
// reads of eight rows at a time fall in different banks).
constexpr int BLD = 20, BSZ = 16 * BLD;
constexpr int TRI_BYTES = 10 * BSZ * 4;           // 12,800
constexpr int L_BYTES = 13312;                    // TRI_BYTES and two 64-float vectors; later an 8 KiB operand tile in L's place
static_assert(L_BYTES == TRI_BYTES + 512 && L_BYTES % 1024 == 0, "pre-pass shared-memory layout");
__host__ __device__ constexpr int tri(int I, int J) { return (I * (I + 1) / 2 + J) * BSZ; }
template <int DH>
constexpr size_t pre_smem() {
    return 1024 + (size_t)(DH / 64) * 24576 /*K, Q, V*/ + L_BYTES + TRI_BYTES + 64 * 4 + 64;
}

// An R x 4 tile of a 16 x 16 block product  acc += L[r..r+R)[0..16) * X[0..16)[c..c+4)  (f32, shared memory): R + 4 reads of 16 bytes
// per 16 R multiply-adds. What counts here is the shared-memory read path, so tiles of four rows on a few lanes beat strips of one
// row on all of them.
template <int R>
__device__ __forceinline__ void tile16(const float* __restrict__ l, const float* __restrict__ x, float (&acc)[R][4]) {
#pragma unroll
    for (int k4 = 0; k4 < 4; ++k4) {
        float4 lr[R], xr[4];
#pragma unroll
        for (int i = 0; i < R; ++i) lr[i] = *reinterpret_cast<const float4*>(l + i * BLD + 4 * k4);
#pragma unroll
        for (int e = 0; e < 4; ++e) xr[e] = *reinterpret_cast<const float4*>(x + (4 * k4 + e) * BLD);
#pragma unroll
        for (int i = 0; i < R; ++i) {
            const float lv[4] = {lr[i].x, lr[i].y, lr[i].z, lr[i].w};
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                acc[i][0] = fmaf(lv[e], xr[e].x, acc[i][0]);
                acc[i][1] = fmaf(lv[e], xr[e].y, acc[i][1]);
                acc[i][2] = fmaf(lv[e], xr[e].z, acc[i][2]);
                acc[i][3] = fmaf(lv[e], xr[e].w, acc[i][3]);
            }
        }
    }
}
template <int R>
__device__ __forceinline__ void put_tile(float* p, float (&acc)[R][4], float f) {
#pragma unroll
    for (int i = 0; i < R; ++i) {
        *reinterpret_cast<float4*>(p + i * BLD) = make_float4(f * acc[i][0], f * acc[i][1], f * acc[i][2], f * acc[i][3]);
#pragma unroll
        for (int e = 0; e < 4; ++e) acc[i][e] = 0.0f;
    }
}
__device__ __forceinline__ void bar_sync(int id, int threads) { asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(threads) : "memory"); }

// Three CTAs of eight warps per SM (four at head dim 64): bound by the latency of a CTA's chain -- tiles, [K;Q]K^T, the solve on four
// warps, the second products -- of which the stores are a sixth. 8192 chunks of 64 x 128: 235 us (440 with scaled copies of K, Q and V
// kept for the chains and the solve on all warps, strip by strip); 64 x 64: 193. K, Q and V come by TMA and are never copied: the factors beta gam and beta go into the
// columns of X - I, once per product, and the rows that the identity contributes are added in f32 (a rounded diagonal would be an error
// common to a whole row of W^ and Uv: 15 % of the error of o, dq and dk).
template <int DH>
__global__ void __launch_bounds__(PRE_THREADS, DH == 64 ? 4 : 3) delta_prep_tc_kernel(
    const __grid_constant__ CUtensorMap mapK, const __grid_constant__ CUtensorMap mapQ, const __grid_constant__ CUtensorMap mapV,
    const __grid_constant__ CUtensorMap mapWH, const __grid_constant__ CUtensorMap mapUV, const float* __restrict__ alpha,
    const float* __restrict__ beta, int T, int H, int n_chunks, Tiles out, int* err_word) {
    constexpr int NB = DH / 64;
    extern __shared__ uint8_t smem_raw[];
    uint8_t* base = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
    uint8_t* KQ_s = base;                         // NB boxes of 128 rows x 128 B: rows 0-63 K, 64-127 Q
    uint8_t* V_s = KQ_s + NB * 16384;             // NB boxes of 64 rows
    float* Lf = reinterpret_cast<float*>(V_s + NB * 8192);
    float* Xf = reinterpret_cast<float*>(reinterpret_cast<uint8_t*>(Lf) + L_BYTES);
    float* g_s = reinterpret_cast<float*>(reinterpret_cast<uint8_t*>(Xf) + TRI_BYTES);
    float* bg_s = Lf + TRI_BYTES / 4;             // beta gam
    float* be_s = bg_s + 64;
    uint64_t* bar = reinterpret_cast<uint64_t*>(g_s + 64);   // [0] K, Q; [1] MMA-A done; [2] MMA-B done; [3] V
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bar + 4);
    volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
    float* wtot = reinterpret_cast<float*>(tmem_slot + 2);
    uint8_t* X1_s = KQ_s + 8192;                  // (X - I) diag(beta gam) as an operand: where Q's first box was
    uint8_t* X2_s = reinterpret_cast<uint8_t*>(Lf);   // (X - I) diag(beta): where L was
    float* Yf = reinterpret_cast<float*>(X1_s);   // [4] blocks in flight

    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int wq = warp & 3, cg = warp >> 2;      // TMEM lane quarter, column group
    const int chunk = blockIdx.x, chain = blockIdx.y;
    const int b = chain / H, h = chain % H;
    const int t0 = chunk * C;
    const int n = T - t0 < C ? T - t0 : C;
    const int64_t row0 = (int64_t)b * T + t0;
    const int64_t tix = (int64_t)chain * n_chunks + chunk;

    float al = 1.0f, be = 0.0f;
    if (tid < n) {
        al = alpha[(row0 + tid) * H + h];
        be = beta[(row0 + tid) * H + h];
    }
    if (tid == 0) {
        *abort_flag = 0;
        for (int i = 0; i < 4; ++i) tc::mbar_init(&bar[i], 1);
        tc::mbar_fence_init();
        tc::mbar_expect_tx(&bar[0], NB * 16384);
#pragma unroll
        for (int kb = 0; kb < NB; ++kb) {
            tc::tma_load_3d(KQ_s + kb * 16384, &mapK, h * DH + kb * 64, t0, b, &bar[0]);
            tc::tma_load_3d(KQ_s + kb * 16384 + 8192, &mapQ, h * DH + kb * 64, t0, b, &bar[0]);
        }
        tc::mbar_expect_tx(&bar[3], NB * 8192);
#pragma unroll
        for (int kb = 0; kb < NB; ++kb) tc::tma_load_3d(V_s + kb * 8192, &mapV, h * DH + kb * 64, t0, b, &bar[3]);
    }
    if (warp == 7) tc::tmem_alloc(tmem_slot, DH);
    // g = cumsum(log alpha): warp scans over the 64 tokens
    float gx = 0.0f;
    if (tid < C) {
        be_s[tid] = be;
        gx = tid < n ? logf(al) : 0.0f;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const float y = __shfl_up_sync(0xffffffffu, gx, o);
            if (lane >= o) gx += y;
        }
        if (tid == 31) *wtot = gx;
    }
    tc::tcgen05_fence_before();
    __syncthreads();
    tc::tcgen05_fence_after();
    const uint32_t tmem = *tmem_slot;
    auto warp_wait = [&](int i) -> bool {
        int got = 1;
        if (lane == 0) got = tc::mbar_wait(&bar[i], 0, abort_flag, err_word, 200 + i) ? 1 : 0;
        return __shfl_sync(0xffffffffu, got, 0) != 0;
    };
    // ---- MMA-A: [KK ; QK] = [K ; Q] K^T   (M128 N64 K = DH)
    if (tid == 128 && tc::mbar_wait(&bar[0], 0, abort_flag, err_word, 200)) {
        constexpr uint32_t IDESC = tc::idesc_bf16_f32(128, 64, 0, 0);
        const uint32_t kq = tc::smem_u32(KQ_s);
#pragma unroll
        for (int k16 = 0; k16 < DH / 16; ++k16) {
            const uint32_t off = (k16 >> 2) * 16384 + (k16 & 3) * 32;
            tc::umma_bf16(tmem, tc::smem_desc_sw128(kq + off, 16, 1024), tc::smem_desc_sw128(kq + off, 16, 1024), IDESC, k16 > 0 ? 1u : 0u);
        }
        tc::umma_commit(&bar[1]);
    }
    if (tid < C) {
        if (tid >= 32) gx += *wtot;
        g_s[tid] = gx;
        bg_s[tid] = be * expf(gx);
        out.GB[tix * 128 + tid] = gx;
        out.GB[tix * 128 + 64 + tid] = be;
    }
    __syncthreads();   // the per-token vectors
    bool ok = warp_wait(1);
    ok = __syncthreads_and(ok ? 1 : 0) != 0;
    tc::tcgen05_fence_after();
    // ---- 32 columns per thread: L = strictlower(beta_t Gam KK) (f32, lanes 0-63); A = lower(Gam QK) (bf16, lanes 64-127)
    if (ok) {
        const int t = 32 * (wq & 1) + lane;
        const bool empty = cg > (wq & 1);         // columns 32-63 of rows 0-31
        uint32_t r[32];
        float e[32];
        if (!empty) {
            tc::tmem_ld_32x32(tmem + ((uint32_t)(wq * 32) << 16) + cg * 32, r);
            const float gt = g_s[t];
#pragma unroll
            for (int j4 = 0; j4 < 8; ++j4) {   // (every one, also above the diagonal: branches around them cost more)
                const float4 g4 = *reinterpret_cast<const float4*>(g_s + cg * 32 + 4 * j4);
                e[4 * j4] = exp_always(gt - g4.x);
                e[4 * j4 + 1] = exp_always(gt - g4.y);
                e[4 * j4 + 2] = exp_always(gt - g4.z);
                e[4 * j4 + 3] = exp_always(gt - g4.w);
            }
            tc::tmem_ld_wait();
        }
        if (wq < 2) {
            const float bt = be_s[t];
            if (!empty) {
#pragma unroll
                for (int j4 = 0; j4 < 8; ++j4) {
                    const int J = cg * 2 + (j4 >> 2);
                    if (J <= (t >> 4)) {
                        float l[4];
#pragma unroll
                        for (int i = 0; i < 4; ++i) l[i] = cg * 32 + 4 * j4 + i < t ? bt * e[4 * j4 + i] * __uint_as_float(r[4 * j4 + i]) : 0.0f;
                        *reinterpret_cast<float4*>(&Lf[tri(t >> 4, J) + (t & 15) * BLD + 4 * (j4 & 3)]) = make_float4(l[0], l[1], l[2], l[3]);
                    }
                }
            }
        } else {
#pragma unroll
            for (int j = 0; j < 32; ++j) e[j] = !empty && cg * 32 + j <= t ? e[j] * __uint_as_float(r[j]) : 0.0f;
            store32_bf16(out.AA + (tix * 64 + t) * 64 + cg * 32, e, true);
#pragma unroll
            for (int j = 0; j < 32; ++j) e[j] -= __bfloat162float(__float2bfloat16(e[j]));
            store32_bf16(out.AL + (tix * 64 + t) * 64 + cg * 32, e, true);
        }
        if (wq < 2) bar_sync(2, 128);   // the four warps that hold L
    }

    // ---- X = (I + L)^-1 in f32 on warps 0 - 3, while the others finish. Warps 0 and 1: two diagonal blocks each, one column per lane, and
    //      the block below them; then warp 2I + J the block (2 + I, J) of the lower left quarter
    if (warp < 2 && ok) {
        {
            const int I = tid >> 4, jj = tid & 15;
            const float* Lb = Lf + tri(I, I);
            float x[16];
#pragma unroll
            for (int t = 0; t < 16; ++t) x[t] = t == jj ? 1.0f : 0.0f;
#pragma unroll
            for (int kb = 0; kb < 4; ++kb) {
                float4 l[16];
#pragma unroll
                for (int t = 4 * kb + 1; t < 16; ++t) l[t] = *reinterpret_cast<const float4*>(Lb + t * BLD + 4 * kb);
#pragma unroll
                for (int t = 4 * kb + 1; t < 16; ++t) x[t] = fmaf(-l[t].x, x[4 * kb], x[t]);
#pragma unroll
                for (int t = 4 * kb + 2; t < 16; ++t) x[t] = fmaf(-l[t].y, x[4 * kb + 1], x[t]);
#pragma unroll
                for (int t = 4 * kb + 3; t < 16; ++t) x[t] = fmaf(-l[t].z, x[4 * kb + 2], x[t]);
#pragma unroll
                for (int t = 4 * kb + 4; t < 16; ++t) x[t] = fmaf(-l[t].w, x[4 * kb + 3], x[t]);
            }
#pragma unroll
            for (int t = 0; t < 16; ++t) Xf[tri(I, I) + t * BLD + jj] = x[t];
        }
        __syncwarp();
        const int tr = lane >> 2, c4 = (lane & 3) * 4;
        {
            const int I = 2 * warp + 1, J = 2 * warp;
            float acc[2][4] = {};
            tile16(Lf + tri(I, J) + 2 * tr * BLD, Xf + tri(J, J) + c4, acc);
            put_tile(&Yf[warp * BSZ + 2 * tr * BLD + c4], acc, 1.0f);
            __syncwarp();
            tile16(Xf + tri(I, I) + 2 * tr * BLD, Yf + warp * BSZ + c4, acc);
            put_tile(&Xf[tri(I, J) + 2 * tr * BLD + c4], acc, -1.0f);
        }
    }
    if (warp < 4 && ok) {
        const int tr = lane >> 2, c4 = (lane & 3) * 4, I = warp >> 1, J = warp & 1;
        float acc[2][4] = {};
        bar_sync(1, 128);
        if (J == 0) tile16(Lf + tri(2 + I, 0) + 2 * tr * BLD, Xf + tri(0, 0) + c4, acc);
        tile16(Lf + tri(2 + I, 1) + 2 * tr * BLD, Xf + tri(1, J) + c4, acc);
        put_tile(&Yf[(2 * J + I) * BSZ + 2 * tr * BLD + c4], acc, 1.0f);
        bar_sync(1, 128);
        tile16(Xf + tri(2 + I, 2) + 2 * tr * BLD, Yf + 2 * J * BSZ + c4, acc);
        if (I == 1) tile16(Xf + tri(3, 3) + 2 * tr * BLD, Yf + (2 * J + 1) * BSZ + c4, acc);
        put_tile(&Xf[tri(2 + I, J) + 2 * tr * BLD + c4], acc, -1.0f);
    }
    tc::tcgen05_fence_before();
    __syncthreads();
    // ---- (X - I) diag(beta gam), (X - I) diag(beta) -> bf16 operand tiles (K-major) and, for the backward, X - I row-major
    float bg8[8], be8[8];
#pragma unroll
    for (int e = 0; e < 8; ++e) {
        bg8[e] = bg_s[(tid & 7) * 8 + e];
        be8[e] = be_s[(tid & 7) * 8 + e];
    }
#pragma unroll
    for (int it = 0; it < 512 / PRE_THREADS; ++it) {
        const int idx = tid + it * PRE_THREADS, t = idx >> 3, jc = tid & 7;
        float x8[8], y8[8];
        if ((jc >> 1) <= (t >> 4)) {
            const float* src = &Xf[tri(t >> 4, jc >> 1) + (t & 15) * BLD + (jc & 1) * 8];
            const float4 a = *reinterpret_cast<const float4*>(src);
            const float4 c = *reinterpret_cast<const float4*>(src + 4);
            x8[0] = a.x, x8[1] = a.y, x8[2] = a.z, x8[3] = a.w, x8[4] = c.x, x8[5] = c.y, x8[6] = c.z, x8[7] = c.w;
        } else {
#pragma unroll
            for (int e = 0; e < 8; ++e) x8[e] = 0.0f;
        }
#pragma unroll
        for (int e = 0; e < 8; ++e)
            if (jc * 8 + e == t) x8[e] = 0.0f;
#pragma unroll
        for (int e = 0; e < 8; ++e) y8[e] = x8[e] * bg8[e];
        *reinterpret_cast<uint4*>(X1_s + tc::sw128_off(t, jc)) = tc::pack8_bf16(y8);
#pragma unroll
        for (int e = 0; e < 8; ++e) y8[e] = x8[e] * be8[e];
        *reinterpret_cast<uint4*>(X2_s + tc::sw128_off(t, jc)) = tc::pack8_bf16(y8);
        if (out.TP) *reinterpret_cast<uint4*>(out.TP + (tix * 64 + t) * 64 + jc * 8) = tc::pack8_bf16(x8);
    }
    tc::fence_proxy_async_smem();
    __syncthreads();

    // ---- MMA-B: X1 K in lane half 0, X2 V in lane half 1   (2 x M64 N = DH K64)
    if (tid == 0 && ok && tc::mbar_wait(&bar[3], 0, abort_flag, err_word, 203)) {
        constexpr uint32_t IDESC = tc::idesc_bf16_f32(64, DH, 0, 1);
        const uint32_t x1 = tc::smem_u32(X1_s), x2 = tc::smem_u32(X2_s), kb = tc::smem_u32(KQ_s), vb = tc::smem_u32(V_s);
        tc::tcgen05_fence_after();
#pragma unroll
        for (int k16 = 0; k16 < C / 16; ++k16)
            tc::umma_bf16(tmem, tc::smem_desc_sw128(x1 + k16 * 32, 16, 1024), tc::smem_desc_sw128(kb + k16 * 2048, 16384, 1024), IDESC, k16 > 0 ? 1u : 0u);
#pragma unroll
        for (int k16 = 0; k16 < C / 16; ++k16)
            tc::umma_bf16(tmem + (16u << 16), tc::smem_desc_sw128(x2 + k16 * 32, 16, 1024), tc::smem_desc_sw128(vb + k16 * 2048, 8192, 1024), IDESC,
                          k16 > 0 ? 1u : 0u);
        tc::umma_commit(&bar[2]);
    }
    if (ok) ok = warp_wait(2);
    ok = __syncthreads_and(ok ? 1 : 0) != 0;
    tc::tcgen05_fence_after();
    // + the identity's rows; into the (consumed) operand tiles of K and V, and out by TMA
    if (ok) {
        const int half = lane >> 4, row = 16 * wq + (lane & 15);
        const float f = half == 0 ? bg_s[row] : be_s[row];
#pragma unroll
        for (int cc = 0; cc < DH / 64; ++cc) {
            const int col = cg * (DH / 2) + cc * 32;
            uint32_t r[32];
            tc::tmem_ld_32x32(tmem + ((uint32_t)(wq * 32) << 16) + col, r);
            tc::tmem_ld_wait();
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const int c16 = (col >> 3) + j;
                uint4* at = reinterpret_cast<uint4*>((half == 0 ? KQ_s + (c16 >> 3) * 16384 : V_s + (c16 >> 3) * 8192) + tc::sw128_off(row, c16 & 7));
                float o8[8];
                tc::unpack8_bf16(*at, o8);
#pragma unroll
                for (int e = 0; e < 8; ++e) o8[e] = fmaf(f, o8[e], __uint_as_float(r[8 * j + e]));
                *at = tc::pack8_bf16(o8);
            }
        }
        tc::fence_proxy_async_smem();
    }
    tc::tcgen05_fence_before();
    __syncthreads();
    if (tid == 0 && ok) {
#pragma unroll
        for (int kb = 0; kb < NB; ++kb) {
            tc::tma_store_2d(&mapWH, KQ_s + kb * 16384, kb * 64, (int)(tix * 64));
            tc::tma_store_2d(&mapUV, V_s + kb * 8192, kb * 64, (int)(tix * 64));
        }
        tc::bulk_commit_group();
        tc::bulk_wait_read();
    }
    if (warp == 7) tc::tmem_dealloc(tmem, DH);
    if (*abort_flag) __nanosleep(20000);   // (a load that never arrived must not land in another CTA's shared memory)
}

// ------------------------------------------------------------------ forward chain
// Threads: 4 warps per 32 columns of the state (warp w: TMEM lane quarter w & 3, columns 32 (w >> 2) ..), one that issues the products
// and one that moves tiles in and out (a TMA instruction waits for its turn at a busy memory: in the issuing thread's loop twelve of
// them were a thousand cycles of every chunk).
// Quarters 0 and 1 hold the 64 rows of U, quarters 2 and 3 those of o; the state's DH rows are all four quarters (DH 128) or 0 and 1.
template <int DH>
struct ChainCfg {
    static constexpr int NB = DH / 64, NG = DH / 32, COMPUTE = 128 * NG, THREADS = COMPUTE + 64;
    static constexpr int S_WARPS = (DH == 128 ? 4 : 2) * NG, ROW_WARPS = 2 * NG;
    static constexpr int S_BYTES = NB * DH * 128;
    static constexpr int F_STAGE = NB * 32768 + 16384, F_K = NB * 16384, F_UV = NB * 24576, F_A = NB * 32768, F_AL = F_A + 8192;   // (W^, Q from 0)
    static constexpr size_t F_SMEM = 1024 + 2 * F_STAGE + S_BYTES + 4 * 512 + 128;
    static constexpr int B_STAGE = NB * 24576 + 24576, B_KQ = 0, B_DO = NB * 16384, B_A = NB * 24576, B_AL = B_A + 8192, B_TP = B_AL + 8192;
    static constexpr int B_RS = DH == 128 ? B_AL : B_TP;   // beta gam dR, where X - I (and AL) were
    // behind the stages: dS and, at 128, dU (then dR) and S; at 64 these lie where A and its remainder were
    static constexpr size_t B_SMEM = 1024 + 2 * B_STAGE + S_BYTES + (DH == 128 ? 16384 + S_BYTES : 0) + 2 * 512 + 192;
};

// What bounds it: at 128 chains HBM (145 KB per chunk with a backward to follow: 5.8 TB/s at 203 us for 64 chunks, 281 before), at few
// chains the two products and two register passes of a chunk (2.9 us).
template <int DH>
__global__ void __launch_bounds__(ChainCfg<DH>::THREADS, DH == 128 ? 1 : 2) delta_fwd_tc_kernel(
    const __grid_constant__ CUtensorMap mapWH, const __grid_constant__ CUtensorMap mapQ, const __grid_constant__ CUtensorMap mapK,
    const __grid_constant__ CUtensorMap mapUV, const __grid_constant__ CUtensorMap mapAA, const __grid_constant__ CUtensorMap mapAL,
    const __grid_constant__ CUtensorMap mapS0, const __grid_constant__ CUtensorMap mapU, const float* __restrict__ GB, int T, int H, int n_chunks, __nv_bfloat16* __restrict__ o,
    const float* s_init, float* s_final /* may be s_init */, int keep /* states and U go out */, int ahead /* L2 prefetch */, int* err_word) {
    using Cfg = ChainCfg<DH>;
    constexpr int NB = Cfg::NB;
    extern __shared__ uint8_t smem_raw[];
    uint8_t* base = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
    uint8_t* S_s = base + 2 * Cfg::F_STAGE;      // NB n-boxes x (DH k-rows x 128 B)
    auto U_s = [&](int s) { return base + s * Cfg::F_STAGE + Cfg::F_UV; };   // U takes Uv's place: NB n-boxes x (64 k-rows x 128 B)
    auto Ue_s = [&](int s) { return base + s * Cfg::F_STAGE; };              // eg U takes W^'s place: n-boxes 16 KiB apart
    float* gb_s = reinterpret_cast<float*>(S_s + Cfg::S_BYTES);   // [4][128]: loaded with the stages, read two chunks longer
    uint64_t* bars = reinterpret_cast<uint64_t*>(gb_s + 512);
    // mma3_done per stage: the moving thread may see it late, and its next phase needs tiles only that thread loads. Every other barrier's
    // next phase needs an arrival or a product of who waits for it.
    uint64_t *full = bars, *mma1_done = bars + 2, *u_ready = bars + 3, *mma2_done = bars + 4, *s_ready = bars + 5, *mma3_done = bars + 6 /*[2]*/,
             *o_done = bars + 8, *s_stored = bars + 9;
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 10);
    volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int chain = blockIdx.x;
    const int b = chain / H, h = chain % H;
    const int d = H * DH;
    const int64_t tile0 = (int64_t)chain * n_chunks;

    if (tid == 0) {
        *abort_flag = 0;
        for (int i = 0; i < 10; ++i) {
            const uint64_t* w = bars + i;
            tc::mbar_init(&bars[i], w == u_ready || w == o_done ? Cfg::ROW_WARPS : w == s_ready ? Cfg::S_WARPS : 1);
        }
        tc::mbar_fence_init();
    }
    if (warp == Cfg::COMPUTE / 32) tc::tmem_alloc(tmem_slot, 4 * DH);
    tc::tcgen05_fence_before();
    __syncthreads();
    tc::tcgen05_fence_after();
    const uint32_t tmem_S = *tmem_slot, tmem_D1 = tmem_S + DH /* two, in turn */, tmem_D2 = tmem_S + 3 * DH;

    if (warp == Cfg::COMPUTE / 32) {
        // ------------------------------------------------------------ MMA issuer (one thread)
        if (lane == 0) {
            constexpr uint32_t ID_KM = tc::idesc_bf16_f32(128, DH, 0, 1);   // A K-major, B MN-major
            constexpr uint32_t ID_MM = tc::idesc_bf16_f32(128, DH, 1, 1);   // A MN-major, B MN-major
            const uint32_t s_addr = tc::smem_u32(S_s);
            for (int c = 0; c < n_chunks; ++c) {
                const int s = c & 1;
                const uint32_t st = tc::smem_u32(base + s * Cfg::F_STAGE);
                if (!tc::mbar_wait(&full[s], (c >> 1) & 1, abort_flag, err_word, 211)) break;
                if (!tc::mbar_wait(s_ready, c & 1, abort_flag, err_word, 212)) break;
                tc::tcgen05_fence_after();
                // D1 = [W^ ; Q] S
                const uint32_t d1 = tmem_D1 + s * DH;
#pragma unroll
                for (int k16 = 0; k16 < DH / 16; ++k16)
                    tc::umma_bf16(d1, tc::smem_desc_sw128(st + (k16 >> 2) * 16384 + (k16 & 3) * 32, 16, 1024),
                                  tc::smem_desc_sw128(s_addr + k16 * 2048, DH * 128, 1024), ID_KM, k16 > 0 ? 1u : 0u);
                tc::umma_commit(mma1_done);
                if (!tc::mbar_wait(u_ready, c & 1, abort_flag, err_word, 213)) break;
                tc::tcgen05_fence_after();
                // S += K^T (eg U)   (head dim 64: rows 64-127 multiply what lies behind K and are not read)
#pragma unroll
                for (int k16 = 0; k16 < C / 16; ++k16)
                    tc::umma_bf16(tmem_S, tc::smem_desc_sw128(st + Cfg::F_K + k16 * 2048, 8192, 1024),
                                  tc::smem_desc_sw128(st + k16 * 2048, 16384, 1024), ID_MM, 1u);
                tc::umma_commit(mma2_done);
                // D2 = [.. ; A] U + [.. ; AL] U   (rows 0-63 multiply what lies in front and are not read)
                if (!tc::mbar_wait(o_done, c & 1, abort_flag, err_word, 214)) break;
                tc::tcgen05_fence_after();
#pragma unroll
                for (int k16 = 0; k16 < C / 16; ++k16)
                    tc::umma_bf16(tmem_D2, tc::smem_desc_sw128(st + Cfg::F_A - 8192 + k16 * 32, 16, 1024),
                                  tc::smem_desc_sw128(st + Cfg::F_UV + k16 * 2048, 8192, 1024), ID_KM, k16 > 0 ? 1u : 0u);
#pragma unroll
                for (int k16 = 0; k16 < C / 16; ++k16)
                    tc::umma_bf16(tmem_D2, tc::smem_desc_sw128(st + Cfg::F_A + k16 * 32, 16, 1024),
                                  tc::smem_desc_sw128(st + Cfg::F_UV + k16 * 2048, 8192, 1024), ID_KM, 1u);
                tc::umma_commit(&mma3_done[s]);
            }
        }
    } else if (warp > Cfg::COMPUTE / 32) {
        // ------------------------------------------------------------ everything that moves (one thread): tiles in, state and U out
        if (lane == 0) {
            auto load = [&](int c, int s) {
                uint8_t* st = base + s * Cfg::F_STAGE;
                const int t = (int)(tile0 + c);
                tc::mbar_expect_tx(&full[s], Cfg::F_STAGE + 512);
                load_vec(gb_s + (c & 3) * 128, GB + (int64_t)t * 128, &full[s]);
#pragma unroll
                for (int kb = 0; kb < NB; ++kb) {
                    tc::tma_load_2d(st + kb * 16384, &mapWH, kb * 64, t * 64, &full[s]);
                    tc::tma_load_3d(st + kb * 16384 + 8192, &mapQ, h * DH + kb * 64, c * C, b, &full[s]);
                    tc::tma_load_2d(st + Cfg::F_UV + kb * 8192, &mapUV, kb * 64, t * 64, &full[s]);
                    tc::tma_load_3d(st + Cfg::F_K + kb * 8192, &mapK, h * DH + kb * 64, c * C, b, &full[s]);
                }
                tc::tma_load_2d(st + Cfg::F_A, &mapAA, 0, t * 64, &full[s]);
                tc::tma_load_2d(st + Cfg::F_AL, &mapAL, 0, t * 64, &full[s]);
            };
            // With one chain per SM two stages in flight do not cover the memory's latency: the next chunk's tiles are asked into L2
            auto prefetch = [&](int c) {
                if (c >= n_chunks) return;
                const int t = (int)(tile0 + c);
#pragma unroll
                for (int kb = 0; kb < NB; ++kb) {
                    tc::tma_prefetch_2d(&mapWH, kb * 64, t * 64);
                    tc::tma_prefetch_3d(&mapQ, h * DH + kb * 64, c * C, b);
                    tc::tma_prefetch_2d(&mapUV, kb * 64, t * 64);
                    tc::tma_prefetch_3d(&mapK, h * DH + kb * 64, c * C, b);
                }
                tc::tma_prefetch_2d(&mapAA, 0, t * 64);
                tc::tma_prefetch_2d(&mapAL, 0, t * 64);
            };
            load(0, 0);
            if (n_chunks > 1) load(1, 1);
            if (ahead) prefetch(2);
            for (int c = 0; c < n_chunks; ++c) {
                if (keep) {   // straight from the operand tiles
                    if (!tc::mbar_wait(s_ready, c & 1, abort_flag, err_word, 215)) break;
#pragma unroll
                    for (int nb = 0; nb < NB; ++nb) tc::tma_store_2d(&mapS0, S_s + nb * (DH * 128), nb * 64, (int)(tile0 + c) * DH);
                    tc::bulk_commit_group();
                    tc::bulk_wait_read();
                    if (!tc::mbar_wait(u_ready, c & 1, abort_flag, err_word, 216)) break;
                    tc::mbar_arrive(s_stored);   // (the new state, whose update needs U as well, may take the old one's place)
#pragma unroll
                    for (int nb = 0; nb < NB; ++nb) tc::tma_store_2d(&mapU, U_s(c & 1) + nb * 8192, nb * 64, (int)(tile0 + c) * 64);
                    tc::bulk_commit_group();
                    tc::bulk_wait_read();
                }
                if (c + 2 < n_chunks) {
                    if (!tc::mbar_wait(&mma3_done[c & 1], (c >> 1) & 1, abort_flag, err_word, 217)) break;
                    load(c + 2, c & 1);
                    if (ahead) prefetch(c + 3);
                }
            }
        }
    } else {
        const int wq = warp & 3, cg = warp >> 2, arow = 32 * wq + lane, row = arow & 63;
        const uint32_t lane_addr = (uint32_t)(wq * 32) << 16;
        const int col = cg * 32;
        const bool s_warp = DH == 128 || wq < 2;
        const bool w32 = (reinterpret_cast<uintptr_t>(o) & 31) == 0;
        auto warp_wait = [&](uint64_t* bar, uint32_t parity, int code) -> bool {
            int got = 1;
            if (lane == 0) got = tc::mbar_wait(bar, parity, abort_flag, err_word, code) ? 1 : 0;
            got = __shfl_sync(0xffffffffu, got, 0);
            tc::tcgen05_fence_after();
            return got != 0;
        };
        auto arrive = [&](uint64_t* bar) {   // one arrival per warp, after every lane's accesses
            tc::fence_proxy_async_smem();
            tc::tcgen05_fence_before();
            __syncwarp();
            if (lane == 0) tc::mbar_arrive(bar);
        };
        bool ok = warp_wait(&full[0], 0, 220);
        if (wq >= 2 && lane == 0) tc::mbar_arrive(o_done);   // phase c: D2 and the other D1 are free for chunk c
        if (s_warp && ok) {   // initial state: bf16 operand copy, and f32 scaled by the first chunk's decay
            const float g0 = expf(gb_s[C - 1]);
            const float* si = s_init ? s_init + ((int64_t)chain * DH + arow) * DH + col : nullptr;
            uint32_t r[32];
            float f[32];
#pragma unroll
            for (int j = 0; j < 32; ++j) f[j] = si ? si[j] : 0.0f;
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const int c16 = cg * 4 + j;
                *reinterpret_cast<uint4*>(S_s + (c16 >> 3) * (DH * 128) + tc::sw128_off(arow, c16 & 7)) = tc::pack8_bf16(f + 8 * j);
            }
#pragma unroll
            for (int j = 0; j < 32; ++j) r[j] = __float_as_uint(g0 * f[j]);
            tc::tmem_st_32x32(tmem_S + lane_addr + col, r);
            tc::tmem_st_wait();
            arrive(s_ready);
        }
        for (int c = 0; ok && c < n_chunks; ++c) {   // (entered with the chunk's tiles in their stage)
            const int s = c & 1;
            const bool last = c + 1 == n_chunks;
            const float g_row = gb_s[(c & 3) * 128 + row], g_last = gb_s[(c & 3) * 128 + C - 1];
            uint32_t r[32];
            if (wq < 2) {
                // U = Uv - W^ S  ->  bf16 operands U and eg U (k rows = tokens, n = value columns)
                const float eg = expf(g_last - g_row);
                if (!warp_wait(mma1_done, c & 1, 222)) break;
                tc::tmem_ld_32x32(tmem_D1 + s * DH + lane_addr + col, r);
                tc::tmem_ld_wait();
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    const int c16 = cg * 4 + j;
                    const uint32_t off = tc::sw128_off(row, c16 & 7);
                    uint4* at = reinterpret_cast<uint4*>(U_s(s) + (c16 >> 3) * 8192 + off);
                    float uv[8], u8[8];
                    tc::unpack8_bf16(*at, uv);
#pragma unroll
                    for (int e = 0; e < 8; ++e) u8[e] = uv[e] - __uint_as_float(r[8 * j + e]);
                    *at = tc::pack8_bf16(u8);
#pragma unroll
                    for (int e = 0; e < 8; ++e) u8[e] *= eg;
                    *reinterpret_cast<uint4*>(Ue_s(s) + (c16 >> 3) * 16384 + off) = tc::pack8_bf16(u8);
                }
                arrive(u_ready);
            }
            const float gam = expf(g_row);
            if (!last && !warp_wait(&full[s ^ 1], ((c + 1) >> 1) & 1, 223)) break;
            if (s_warp) {
                // new state: final state (f32), or bf16 operand copy and pre-scale for the next chunk
                const float gnext = expf(gb_s[((c + 1) & 3) * 128 + C - 1]);
                if (keep && !warp_wait(s_stored, c & 1, 224)) break;
                if (!warp_wait(mma2_done, c & 1, 225)) break;
                tc::tmem_ld_32x32(tmem_S + lane_addr + col, r);
                tc::tmem_ld_wait();
                float f[32];
#pragma unroll
                for (int j = 0; j < 32; ++j) f[j] = __uint_as_float(r[j]);
                if (last) {
                    if (s_final) store32(s_final + ((int64_t)chain * DH + arow) * DH + col, f, false);
                } else {
#pragma unroll
                    for (int j = 0; j < 4; ++j) {
                        const int c16 = cg * 4 + j;
                        *reinterpret_cast<uint4*>(S_s + (c16 >> 3) * (DH * 128) + tc::sw128_off(arow, c16 & 7)) = tc::pack8_bf16(f + 8 * j);
                    }
#pragma unroll
                    for (int j = 0; j < 32; ++j) r[j] = __float_as_uint(gnext * f[j]);
                    tc::tmem_st_32x32(tmem_S + lane_addr + col, r);
                    tc::tmem_st_wait();
                    arrive(s_ready);
                }
            }
            if (wq >= 2) {
                // o = gam (Q S) + A U: TMEM lanes 64-127
                if (!warp_wait(&mma3_done[s], (c >> 1) & 1, 226)) break;
                uint32_t q[32];
                tc::tmem_ld_32x32(tmem_D1 + s * DH + lane_addr + col, q);
                tc::tmem_ld_32x32(tmem_D2 + lane_addr + col, r);
                tc::tmem_ld_wait();
                tc::tcgen05_fence_before();
                __syncwarp();
                if (lane == 0) tc::mbar_arrive(o_done);
                if (c * C + row < T) {
                    float f[32];
#pragma unroll
                    for (int j = 0; j < 32; ++j) f[j] = fmaf(gam, __uint_as_float(q[j]), __uint_as_float(r[j]));
                    store32_bf16(o + ((int64_t)b * T + c * C + row) * d + h * DH + col, f, w32);
                }
            }
        }
    }
    tc::tcgen05_fence_before();
    __syncthreads();
    if (*abort_flag) __nanosleep(20000);
    if (warp == Cfg::COMPUTE / 32) tc::tmem_dealloc(tmem_S, 4 * DH);
}

// ------------------------------------------------------------------ backward chain
// Same threads as the forward: quarters 0 and 1 hold the 64 rows of dU and dR, quarters 2 and 3 scale the rows of dO by gam in place
// (after A^T dO has read them), dS is held like S. TMEM: dS, D1 = K dS and later (X - I)^T dU, D2 = A^T dO, D3 = K S. 202 KB of HBM per chunk
// (dv in f32 among them) at 3.9 TB/s: 420 us for 64 chunks of 128 chains, three products and their register passes one after another. The 32 KB of
// S are there for two sums over f32 values, <S, dS> and dv . (S^T k): without them 371 us, of the difference most is the load.
// With the gradients on the same chain a chunk was nine groups of products: 914 us.
template <int DH>
__global__ void __launch_bounds__(ChainCfg<DH>::THREADS, DH == 128 ? 1 : 2) delta_bwd_tc_kernel(
    const __grid_constant__ CUtensorMap mapK, const __grid_constant__ CUtensorMap mapQ, const __grid_constant__ CUtensorMap mapDO,
    const __grid_constant__ CUtensorMap mapAA, const __grid_constant__ CUtensorMap mapAL, const __grid_constant__ CUtensorMap mapTP,
    const __grid_constant__ CUtensorMap mapDS,
    const __grid_constant__ CUtensorMap mapDR, const __grid_constant__ CUtensorMap mapV, const __grid_constant__ CUtensorMap mapS0,
    const float* __restrict__ GB, const __nv_bfloat16* __restrict__ v, int T, int H, int n_chunks, float* __restrict__ d_qkv,
    float* __restrict__ VD /* [tile][2][NG][64]: v . dv and -gam dv . (S^T k) over 32 columns */, float* __restrict__ SD /* [tile][S_WARPS]: parts of <S, dS> */, int ahead, int* err_word) {
    using Cfg = ChainCfg<DH>;
    constexpr int NB = Cfg::NB, NG = Cfg::NG;
    extern __shared__ uint8_t smem_raw[];
    uint8_t* base = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
    uint8_t* S_s = base + 2 * Cfg::B_STAGE;      // dS: NB n-boxes x (DH k-rows x 128 B)
    auto R_s = [&](int s) {                      // dU, then dR: NB n-boxes x (64 k-rows x 128 B)
        return DH == 128 ? S_s + Cfg::S_BYTES : base + s * Cfg::B_STAGE + Cfg::B_A;
    };
    auto Rs_s = [&](int s) { return base + s * Cfg::B_STAGE + Cfg::B_RS; };
    // S at the start of step it's chunk, which meets dS in the step before: a buffer of its own, or at head dim 64 the place that the
    // remainder of A has left in that step's stage
    auto S0_s = [&](int it) { return DH == 128 ? S_s + Cfg::S_BYTES + 16384 : base + ((it & 1) ^ 1) * Cfg::B_STAGE + Cfg::B_AL; };
    float* gb_s = reinterpret_cast<float*>(S_s + Cfg::S_BYTES + (DH == 128 ? 16384 + Cfg::S_BYTES : 0));   // [2][128], with the stages
    uint64_t* bars = reinterpret_cast<uint64_t*>(gb_s + 256);
    uint64_t *full = bars, *mma0_done = bars + 2, *mma1_done = bars + 3, *mma2_done = bars + 4, *mma3_done = bars + 5 /*[2], per stage as in the forward*/,
             *s_ready = bars + 7, *do_ready = bars + 8, *du_ready = bars + 9, *dr_ready = bars + 10, *s_stored = bars + 11, *r_stored = bars + 12,
             *s0_full = bars + 13, *ks_done = bars + 14, *ks_read = bars + 15;
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 16);
    volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int chain = blockIdx.x;
    const int b = chain / H, h = chain % H;
    const int d = H * DH;
    const int64_t tile0 = (int64_t)chain * n_chunks;

    if (tid == 0) {
        *abort_flag = 0;
        for (int i = 0; i < 16; ++i) {
            const uint64_t* w = bars + i;
            tc::mbar_init(&bars[i], w == s_ready ? Cfg::S_WARPS : w == do_ready || w == du_ready || w == dr_ready || w == ks_read ? Cfg::ROW_WARPS : 1);
        }
        tc::mbar_fence_init();
    }
    constexpr int TMEM_COLS = 4 * DH;
    if (warp == Cfg::COMPUTE / 32) tc::tmem_alloc(tmem_slot, TMEM_COLS);
    tc::tcgen05_fence_before();
    __syncthreads();
    tc::tcgen05_fence_after();
    const uint32_t tmem_S = *tmem_slot, tmem_D1 = tmem_S + DH, tmem_D2 = tmem_S + 2 * DH, tmem_D3 = tmem_S + 3 * DH;

    if (warp == Cfg::COMPUTE / 32) {
        // ------------------------------------------------------------ MMA issuer (one thread)
        if (lane == 0) {
            constexpr uint32_t ID_KM = tc::idesc_bf16_f32(128, DH, 0, 1), ID_MM = tc::idesc_bf16_f32(128, DH, 1, 1), ID_MM_NEG = ID_MM | (1u << 13);
            const uint32_t s_addr = tc::smem_u32(S_s);
            // D2 = (A + AL)^T dO of step `it`   (rows 64-127 multiply what lies behind and are not read)
            auto mma0 = [&](int it) -> bool {
                const int s = it & 1;
                if (!tc::mbar_wait(&full[s], (it >> 1) & 1, abort_flag, err_word, 301)) return false;
                const uint32_t st = tc::smem_u32(base + s * Cfg::B_STAGE);
                tc::tcgen05_fence_after();
#pragma unroll
                for (int k16 = 0; k16 < C / 16; ++k16)
                    tc::umma_bf16(tmem_D2, tc::smem_desc_sw128(st + Cfg::B_A + k16 * 2048, 8192, 1024),
                                  tc::smem_desc_sw128(st + Cfg::B_DO + k16 * 2048, 8192, 1024), ID_MM, k16 > 0 ? 1u : 0u);
#pragma unroll
                for (int k16 = 0; k16 < C / 16; ++k16)
                    tc::umma_bf16(tmem_D2, tc::smem_desc_sw128(st + Cfg::B_AL + k16 * 2048, 8192, 1024),
                                  tc::smem_desc_sw128(st + Cfg::B_DO + k16 * 2048, 8192, 1024), ID_MM, 1u);
                tc::umma_commit(mma0_done);
                return true;
            };
            // D3 = K S of step `it`, off the serial path
            auto mma_ks = [&](int it) -> bool {
                if (!tc::mbar_wait(s0_full, it & 1, abort_flag, err_word, 319)) return false;
                if (it > 0 && !tc::mbar_wait(ks_read, (it - 1) & 1, abort_flag, err_word, 300)) return false;
                const uint32_t st = tc::smem_u32(base + (it & 1) * Cfg::B_STAGE), s0 = tc::smem_u32(S0_s(it));
                tc::tcgen05_fence_after();
#pragma unroll
                for (int k16 = 0; k16 < DH / 16; ++k16)
                    tc::umma_bf16(tmem_D3, tc::smem_desc_sw128(st + (k16 >> 2) * 16384 + (k16 & 3) * 32, 16, 1024),
                                  tc::smem_desc_sw128(s0 + k16 * 2048, DH * 128, 1024), ID_KM, k16 > 0 ? 1u : 0u);
                tc::umma_commit(ks_done);
                return true;
            };
            bool ok = mma0(0) && mma_ks(0);
            for (int it = 0; ok && it < n_chunks; ++it) {
                const int c = n_chunks - 1 - it, par = it & 1;
                const uint32_t st = tc::smem_u32(base + par * Cfg::B_STAGE), r_addr = tc::smem_u32(R_s(par)), rs_addr = tc::smem_u32(Rs_s(par));
                if (!tc::mbar_wait(s_ready, par, abort_flag, err_word, 302)) break;
                tc::tcgen05_fence_after();
                // D1 = K dS   (rows 64-127 multiply Q and are not read)
#pragma unroll
                for (int k16 = 0; k16 < DH / 16; ++k16)
                    tc::umma_bf16(tmem_D1, tc::smem_desc_sw128(st + (k16 >> 2) * 16384 + (k16 & 3) * 32, 16, 1024),
                                  tc::smem_desc_sw128(s_addr + k16 * 2048, DH * 128, 1024), ID_KM, k16 > 0 ? 1u : 0u);
                tc::umma_commit(mma1_done);
                if (!tc::mbar_wait(du_ready, par, abort_flag, err_word, 303)) break;
                tc::tcgen05_fence_after();
                // D1 = (X - I)^T dU
#pragma unroll
                for (int k16 = 0; k16 < C / 16; ++k16)
                    tc::umma_bf16(tmem_D1, tc::smem_desc_sw128(st + Cfg::B_TP + k16 * 2048, 8192, 1024),
                                  tc::smem_desc_sw128(r_addr + k16 * 2048, 8192, 1024), ID_MM, k16 > 0 ? 1u : 0u);
                tc::umma_commit(mma2_done);
                if (c == 0) break;
                // dS += Q^T (gam dO), while dR is formed
                if (!tc::mbar_wait(do_ready, par, abort_flag, err_word, 304)) break;
                tc::tcgen05_fence_after();
#pragma unroll
                for (int k16 = 0; k16 < C / 16; ++k16)
                    tc::umma_bf16(tmem_S, tc::smem_desc_sw128(st + 8192 + k16 * 2048, 16384, 1024),
                                  tc::smem_desc_sw128(st + Cfg::B_DO + k16 * 2048, 8192, 1024), ID_MM, 1u);
                if (!tc::mbar_wait(dr_ready, par, abort_flag, err_word, 305)) break;
                tc::tcgen05_fence_after();
                // dS -= K^T (beta gam dR)
#pragma unroll
                for (int k16 = 0; k16 < C / 16; ++k16)
                    tc::umma_bf16(tmem_S, tc::smem_desc_sw128(st + k16 * 2048, 16384, 1024),
                                  tc::smem_desc_sw128(rs_addr + k16 * 2048, 8192, 1024), ID_MM_NEG, 1u);
                tc::umma_commit(&mma3_done[par]);
                if (!mma0(it + 1) || !mma_ks(it + 1)) break;
            }
        }
    } else if (warp > Cfg::COMPUTE / 32) {
        // ------------------------------------------------------------ everything that moves (one thread): tiles in, dS and dR out
        if (lane == 0) {
            auto load_al = [&](int it) {   // (counted in its stage's bytes)
                tc::tma_load_2d(base + (it & 1) * Cfg::B_STAGE + Cfg::B_AL, &mapAL, 0, (int)(tile0 + n_chunks - 1 - it) * 64, &full[it & 1]);
            };
            auto load_s0 = [&](int it) {
                tc::mbar_expect_tx(s0_full, Cfg::S_BYTES);
#pragma unroll
                for (int nb = 0; nb < NB; ++nb)
                    tc::tma_load_2d(S0_s(it) + nb * (DH * 128), &mapS0, nb * 64, (int)(tile0 + n_chunks - 1 - it) * DH, s0_full);
            };
            auto load = [&](int it) {
                const int c = n_chunks - 1 - it, s = it & 1;
                uint8_t* st = base + s * Cfg::B_STAGE;
                const int t = (int)(tile0 + c);
                tc::mbar_expect_tx(&full[s], Cfg::B_STAGE + 512);
                load_vec(gb_s + s * 128, GB + (int64_t)t * 128, &full[s]);
#pragma unroll
                for (int kb = 0; kb < NB; ++kb) tc::tma_load_3d(st + Cfg::B_DO + kb * 8192, &mapDO, h * DH + kb * 64, c * C, b, &full[s]);
                tc::tma_load_2d(st + Cfg::B_A, &mapAA, 0, t * 64, &full[s]);
                if (DH == 128 || it == 0) load_al(it);
#pragma unroll
                for (int kb = 0; kb < NB; ++kb) {
                    tc::tma_load_3d(st + kb * 16384, &mapK, h * DH + kb * 64, c * C, b, &full[s]);
                    tc::tma_load_3d(st + kb * 16384 + 8192, &mapQ, h * DH + kb * 64, c * C, b, &full[s]);
                }
                tc::tma_load_2d(st + Cfg::B_TP, &mapTP, 0, t * 64, &full[s]);
            };
            auto prefetch = [&](int it) {   // into L2, as in the forward; v is read from there by the threads
                const int c = n_chunks - 1 - it, t = (int)(tile0 + c);
                if (c < 0) return;
#pragma unroll
                for (int kb = 0; kb < NB; ++kb) {
                    tc::tma_prefetch_3d(&mapDO, h * DH + kb * 64, c * C, b);
                    tc::tma_prefetch_3d(&mapK, h * DH + kb * 64, c * C, b);
                    tc::tma_prefetch_3d(&mapQ, h * DH + kb * 64, c * C, b);
                    tc::tma_prefetch_3d(&mapV, h * DH + kb * 64, c * C, b);
                }
                tc::tma_prefetch_2d(&mapAA, 0, t * 64);
                tc::tma_prefetch_2d(&mapAL, 0, t * 64);
                tc::tma_prefetch_2d(&mapTP, 0, t * 64);
#pragma unroll
                for (int nb = 0; nb < NB; ++nb) tc::tma_prefetch_2d(&mapS0, nb * 64, t * DH);
            };
            load(0);
            load_s0(0);
            if (n_chunks > 1) load(1);
            if (ahead) prefetch(2);
            for (int it = 0; it < n_chunks; ++it) {
                const int c = n_chunks - 1 - it, par = it & 1;
                if (!tc::mbar_wait(s_ready, par, abort_flag, err_word, 306)) break;
#pragma unroll
                for (int nb = 0; nb < NB; ++nb) tc::tma_store_2d(&mapDS, S_s + nb * (DH * 128), nb * 64, (int)(tile0 + c) * DH);
                tc::bulk_commit_group();
                if (it + 1 < n_chunks) {   // this step's S has met dS (s_ready) and K; at head dim 64 the remainder of A gives up its place
                    if (!tc::mbar_wait(ks_done, par, abort_flag, err_word, 309)) break;   // (and A^T dO before it)
                    load_s0(it + 1);
                    if (DH == 64) load_al(it + 1);
                }
                tc::bulk_wait_read();
                tc::mbar_arrive(s_stored);
                if (!tc::mbar_wait(dr_ready, par, abort_flag, err_word, 307)) break;
#pragma unroll
                for (int nb = 0; nb < NB; ++nb) tc::tma_store_2d(&mapDR, R_s(par) + nb * 8192, nb * 64, (int)(tile0 + c) * 64);
                tc::bulk_commit_group();
                tc::bulk_wait_read();
                tc::mbar_arrive(r_stored);
                if (it + 2 < n_chunks) {
                    if (!tc::mbar_wait(&mma3_done[par], (it >> 1) & 1, abort_flag, err_word, 308)) break;
                    load(it + 2);
                    if (ahead) prefetch(it + 3);
                }
            }
        }
    } else {
        const int wq = warp & 3, cg = warp >> 2, arow = 32 * wq + lane, row = arow & 63;
        const uint32_t lane_addr = (uint32_t)(wq * 32) << 16;
        const int col = cg * 32;
        const bool s_warp = DH == 128 || wq < 2;
        const bool w32 = (reinterpret_cast<uintptr_t>(d_qkv) & 31) == 0;
        auto warp_wait = [&](uint64_t* bar, uint32_t parity, int code) -> bool {
            int got = 1;
            if (lane == 0) got = tc::mbar_wait(bar, parity, abort_flag, err_word, code) ? 1 : 0;
            got = __shfl_sync(0xffffffffu, got, 0);
            tc::tcgen05_fence_after();
            return got != 0;
        };
        auto arrive = [&](uint64_t* bar) {   // one arrival per warp, after every lane's accesses
            tc::fence_proxy_async_smem();
            tc::tcgen05_fence_before();
            __syncwarp();
            if (lane == 0) tc::mbar_arrive(bar);
        };
        if (s_warp) {   // dS = 0
            uint32_t z[32];
#pragma unroll
            for (int j = 0; j < 32; ++j) z[j] = 0u;
            tc::tmem_st_32x32(tmem_S + lane_addr + col, z);
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const int c16 = cg * 4 + j;
                *reinterpret_cast<uint4*>(S_s + (c16 >> 3) * (DH * 128) + tc::sw128_off(arow, c16 & 7)) = make_uint4(0, 0, 0, 0);
            }
            tc::tmem_st_wait();
            arrive(s_ready);
        }
        bool ok = warp_wait(&full[0], 0, 310);
        for (int it = 0; ok && it < n_chunks; ++it) {   // (entered with the chunk's tiles in their stage)
            const int c = n_chunks - 1 - it, par = it & 1;
            uint8_t* st = base + par * Cfg::B_STAGE;
            const float g_row = gb_s[par * 128 + row], be_row = gb_s[par * 128 + 64 + row], gam = expf(g_row);
            float du[32];
            // The row of v, used behind the state's update: at head dim 64 asked for before it (265 us for 128 chains of 64 chunks, 279 behind it), at
            // 128 behind it, where the update needs the registers (438 and 420).
            uint4 v4[4];
            auto ask_v = [&] {
                const __nv_bfloat16* vr = v + ((int64_t)b * T + c * C + row) * d + h * DH + col;
#pragma unroll
                for (int j = 0; j < 4; ++j) v4[j] = c * C + row < T ? reinterpret_cast<const uint4*>(vr)[j] : make_uint4(0, 0, 0, 0);
            };
            if (wq >= 2) {
                if (c > 0) {   // gam dO in place, once A^T dO is done
                    if (!warp_wait(mma0_done, par, 311)) break;
                    uint8_t* dot = st + Cfg::B_DO;
#pragma unroll
                    for (int j = 0; j < 4; ++j) {
                        const int c16 = cg * 4 + j;
                        uint4* at = reinterpret_cast<uint4*>(dot + (c16 >> 3) * 8192 + tc::sw128_off(row, c16 & 7));
                        float x8[8];
                        tc::unpack8_bf16(*at, x8);
#pragma unroll
                        for (int e = 0; e < 8; ++e) x8[e] *= gam;
                        *at = tc::pack8_bf16(x8);
                    }
                    arrive(do_ready);
                }
            } else {
                // dU = A^T dO + eg (K dS)
                const float eg = expf(gb_s[par * 128 + C - 1] - g_row);
                if (it > 0 && !warp_wait(r_stored, (it - 1) & 1, 312)) break;
                if (!warp_wait(mma1_done, par, 313)) break;   // (and A^T dO before it)
#pragma unroll
                for (int i = 0; i < 2; ++i) {
                    uint32_t a[16], r[16];
                    tc::tmem_ld_32x16(tmem_D2 + lane_addr + col + 16 * i, a);
                    tc::tmem_ld_32x16(tmem_D1 + lane_addr + col + 16 * i, r);
                    tc::tmem_ld_wait();
#pragma unroll
                    for (int j = 0; j < 16; ++j) du[16 * i + j] = fmaf(eg, __uint_as_float(r[j]), __uint_as_float(a[j]));
#pragma unroll
                    for (int j = 0; j < 2; ++j) {
                        const int c16 = cg * 4 + 2 * i + j;
                        *reinterpret_cast<uint4*>(R_s(par) + (c16 >> 3) * 8192 + tc::sw128_off(row, c16 & 7)) = tc::pack8_bf16(du + 16 * i + 8 * j);
                    }
                }
                arrive(du_ready);
                // dR = dU + (X - I)^T dU
                if (!warp_wait(mma2_done, par, 314)) break;
                const float bg = be_row * gam;
#pragma unroll
                for (int i = 0; i < 2; ++i) {
                    uint32_t r[16];
                    tc::tmem_ld_32x16(tmem_D1 + lane_addr + col + 16 * i, r);
                    tc::tmem_ld_wait();
#pragma unroll
                    for (int j = 0; j < 16; ++j) du[16 * i + j] += __uint_as_float(r[j]);
#pragma unroll
                    for (int j = 0; j < 2; ++j) {
                        const int c16 = cg * 4 + 2 * i + j;
                        const uint32_t off = (c16 >> 3) * 8192 + tc::sw128_off(row, c16 & 7);
                        *reinterpret_cast<uint4*>(R_s(par) + off) = tc::pack8_bf16(du + 16 * i + 8 * j);
                        float x8[8];
#pragma unroll
                        for (int e = 0; e < 8; ++e) x8[e] = bg * du[16 * i + 8 * j + e];
                        *reinterpret_cast<uint4*>(Rs_s(par) + off) = tc::pack8_bf16(x8);
                    }
                }
                arrive(dr_ready);
                if (DH == 64) ask_v();
                // -beta gam dR . (S^T k)   (K S was done before K dS)
                float ky = 0.0f;
#pragma unroll
                for (int i = 0; i < 2; ++i) {
                    uint32_t r[16];
                    tc::tmem_ld_32x16(tmem_D3 + lane_addr + col + 16 * i, r);
                    tc::tmem_ld_wait();
#pragma unroll
                    for (int j = 0; j < 16; ++j) ky = fmaf(du[16 * i + j], __uint_as_float(r[j]), ky);
                }
                arrive(ks_read);
                VD[(((tile0 + c) * 2 + 1) * NG + cg) * 64 + row] = -bg * ky;
            }
            float sd = 0.0f;
            if (c > 0) {
                if (!warp_wait(&full[par ^ 1], ((it + 1) >> 1) & 1, 315)) break;
                if (s_warp) {   // dS at the start of the chunk: bf16 operand copy, f32 scaled by the chunk before's decay, and <S, dS> for that chunk
                    const float gC = expf(gb_s[(par ^ 1) * 128 + C - 1]);
                    if (!warp_wait(s0_full, par ^ 1, 318)) break;
                    if (!warp_wait(s_stored, par, 316)) break;
                    if (!warp_wait(&mma3_done[par], (it >> 1) & 1, 317)) break;
#pragma unroll
                    for (int i = 0; i < 2; ++i) {
                        uint32_t r[16];
                        float f[16];
                        tc::tmem_ld_32x16(tmem_S + lane_addr + col + 16 * i, r);
                        tc::tmem_ld_wait();
#pragma unroll
                        for (int j = 0; j < 16; ++j) f[j] = __uint_as_float(r[j]);
#pragma unroll
                        for (int j = 0; j < 2; ++j) {
                            const int c16 = cg * 4 + 2 * i + j;
                            const uint32_t off = (c16 >> 3) * (DH * 128) + tc::sw128_off(arow, c16 & 7);
                            *reinterpret_cast<uint4*>(S_s + off) = tc::pack8_bf16(f + 8 * j);
                            float s8[8];
                            tc::unpack8_bf16(*reinterpret_cast<const uint4*>(S0_s(it + 1) + off), s8);
#pragma unroll
                            for (int e = 0; e < 8; ++e) sd = fmaf(s8[e], f[8 * j + e], sd);
                        }
#pragma unroll
                        for (int j = 0; j < 16; ++j) r[j] = __float_as_uint(gC * f[j]);
                        tc::tmem_st_32x16(tmem_S + lane_addr + col + 16 * i, r);
                    }
                    tc::tmem_st_wait();
                    arrive(s_ready);
                    sd = warp_sum(sd);
                    if (lane == 0) SD[(tile0 + c - 1) * Cfg::S_WARPS + cg * (Cfg::S_WARPS / NG) + wq] = sd;
                }
            }
            if (wq < 2) {   // dv = beta dR, and this thread's part of v . dv
                if (DH == 128) ask_v();
                float vd = 0.0f;
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    float x8[8];
                    tc::unpack8_bf16(v4[j], x8);
#pragma unroll
                    for (int e = 0; e < 8; ++e) {
                        du[8 * j + e] *= be_row;
                        vd = fmaf(x8[e], du[8 * j + e], vd);
                    }
                }
                VD[((tile0 + c) * 2 * NG + cg) * 64 + row] = vd;
                if (c * C + row < T) store32(d_qkv + ((int64_t)b * T + c * C + row) * 3 * d + 2 * d + h * DH + col, du, w32);
            }
        }
    }
    tc::tcgen05_fence_before();
    __syncthreads();
    if (*abort_flag) __nanosleep(20000);
    if (warp == Cfg::COMPUTE / 32) tc::tmem_dealloc(tmem_S, TMEM_COLS);
}

// ------------------------------------------------------------------ gradients per chunk
// One CTA per (chunk, chain), two per SM; nothing here depends on another chunk. 209 KB of HBM a chunk: 410 us for 8192 of 64 x 128
// (4.2 TB/s, 394 us with the gates' sums over the bf16 tiles M and P; two CTAs per SM are what 103 KB of tiles allow, and one's loads and stores hide the other's register passes). With S and dS the (bf16) state at the chunk's start
// and gradient at its end:
//   dL = dR U^T,  dA = dO U^T,  X = dO S^T,  Y = dR S^T,  dW = U dS^T              one group of products, value columns 64 at a time
//   M = -beta Gam dL (strictly lower),  P = Gam dA (lower);  X *= gam,  Y *= -beta gam   (in TMEM)
//   dq = X + P K,   dk = Y + M^T K + P^T Q + M K, + eg dW                          second group, on top of X and Y
// and the gate gradients from f32 values alone, with KK = K K^T and QK = Q K^T formed once more:
//   w_t = rowsum(M o KK)_t + k_t . Y_t
//   d log alpha_t = sum over t' >= t of (w + rowsum(P o QK) + q . X - colsum(M o KK + P o QK) - eg k . dW)_t'
//                   + gam_C <S, dS> + sum over t' of eg k . dW          (<S, dS> and k . Y = -gam dv . (S^T k) from the chain
//                                                                        kernel, which holds dS and dR in f32)
//   d beta_t = (v_t . dv_t + w_t) / beta_t
// TMEM halves: thread (warp, lane) sees row 16 (warp & 3) + (lane & 15) of the product in half lane >> 4.
constexpr int GR_THREADS = 256;
template <int DH>
struct GradCfg {
    // Value columns are taken 64 at a time. Head dim 128: rows (dR, U, dO) of both halves, S and the first half of dS come at once; what
    // the first half's products have consumed makes room for the second half of dS, K and Q. Head dim 64: everything at once.
    static constexpr int NB = DH / 64, SB = DH * 128 /*64 columns of S*/, R_DR = 0, R_U = 8192, R_DO = 16384, R_ROWS = 24576 /*per half*/,
                         R_S = NB * R_ROWS, R_DS = R_S + SB, R_S1 = R_DS + SB, R_DS1 = R_S,
                         R_K = DH == 128 ? R_DS : R_DS + SB, R_Q = DH == 128 ? R_DR : R_K + 8192, R_END = DH == 128 ? R_S1 + SB : R_Q + 8192,
                         R_M = (NB - 1) * R_ROWS + R_DR, R_P = (NB - 1) * R_ROWS + R_DO;
    static constexpr int NVEC = 64 /*g*/ + 64 /*beta*/ + 64 /*alpha*/ + 128 /*norms*/ + 2 * 128 * 2 /*dots, row sums*/ + 4 * 64 /*column sums*/ +
                                2 * 64 * 2 /*q.X, k.dW*/ + 64 * 2 /*v.dv, k.Y*/;
    static constexpr size_t SMEM = 1024 + R_END + NVEC * 4 + 96;
};

template <int DH>
__global__ void __launch_bounds__(GR_THREADS, 2) delta_grad_tc_kernel(
    const __grid_constant__ CUtensorMap mapK, const __grid_constant__ CUtensorMap mapQ, const __grid_constant__ CUtensorMap mapDO,
    const __grid_constant__ CUtensorMap mapDR, const __grid_constant__ CUtensorMap mapU, const __grid_constant__ CUtensorMap mapS0,
    const __grid_constant__ CUtensorMap mapDS, const float* __restrict__ GB, const float* __restrict__ VD, const float* __restrict__ SD, const float* __restrict__ alpha,
    const float* __restrict__ qnorm, const float* __restrict__ knorm, int T, int H, int n_chunks,
    float* __restrict__ d_qkv, float* __restrict__ d_gate, int* err_word) {
    using Cfg = GradCfg<DH>;
    constexpr int NB = Cfg::NB, CW = DH / 2 /*columns of a row per thread*/;
    extern __shared__ uint8_t smem_raw[];
    uint8_t* sm = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
    float* g_s = reinterpret_cast<float*>(sm + Cfg::R_END);
    float *be_s = g_s + 64, *al_s = be_s + 64, *nrm_s = al_s + 64 /*q rows, k rows*/, *dot_s = nrm_s + 128 /*[2][128]*/,
          *rs_s = dot_s + 256 /*[2][128]*/, *qx_s = rs_s + 256 /*[2][64]*/, *cs_s = qx_s + 128 /*[4][64]*/, *kw_s = cs_s + 256 /*[2][64]*/, *vd_s = kw_s + 128,
          *ky_s = vd_s + 64;
    // tiles: [0], [1] by half, [2] dS's second, [3] K, Q; products: [4], [5] by half, [6] second group, [7] K K^T, Q K^T
    uint64_t* bars = reinterpret_cast<uint64_t*>(ky_s + 64);
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 8);
    volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int wq = warp & 3, cg = warp >> 2, half = lane >> 4, row = 16 * wq + (lane & 15);
    const int chunk = blockIdx.x, chain = blockIdx.y;
    const int b = chain / H, h = chain % H;
    const int d = H * DH;
    const int t0 = chunk * C;
    const int n = T - t0 < C ? T - t0 : C;
    const int64_t grow = (int64_t)b * T + t0;
    const int64_t tix = (int64_t)chain * n_chunks + chunk;
    const bool w32 = (reinterpret_cast<uintptr_t>(d_qkv) & 31) == 0;

    auto load_rows = [&](int hv, uint64_t* bar) {
        tc::tma_load_2d(sm + hv * Cfg::R_ROWS + Cfg::R_DR, &mapDR, hv * 64, (int)tix * 64, bar);
        tc::tma_load_2d(sm + hv * Cfg::R_ROWS + Cfg::R_U, &mapU, hv * 64, (int)tix * 64, bar);
        tc::tma_load_3d(sm + hv * Cfg::R_ROWS + Cfg::R_DO, &mapDO, h * DH + hv * 64, t0, b, bar);
    };
    auto load_kq = [&] {
        tc::mbar_expect_tx(&bars[3], NB * 16384);
#pragma unroll
        for (int kb = 0; kb < NB; ++kb) {
            tc::tma_load_3d(sm + Cfg::R_K + kb * 8192, &mapK, h * DH + kb * 64, t0, b, &bars[3]);
            tc::tma_load_3d(sm + Cfg::R_Q + kb * 8192, &mapQ, h * DH + kb * 64, t0, b, &bars[3]);
        }
    };
    if (tid == 0) {
        *abort_flag = 0;
        for (int i = 0; i < 8; ++i) tc::mbar_init(&bars[i], 1);
        tc::mbar_fence_init();
        tc::mbar_expect_tx(&bars[0], Cfg::R_ROWS + 2 * Cfg::SB);
        load_rows(0, &bars[0]);
        tc::tma_load_2d(sm + Cfg::R_S, &mapS0, 0, (int)tix * DH, &bars[0]);
        tc::tma_load_2d(sm + Cfg::R_DS, &mapDS, 0, (int)tix * DH, &bars[0]);
        if constexpr (DH == 128) {
            tc::mbar_expect_tx(&bars[1], Cfg::R_ROWS + Cfg::SB);
            load_rows(1, &bars[1]);
            tc::tma_load_2d(sm + Cfg::R_S1, &mapS0, 64, (int)tix * DH, &bars[1]);
        } else {
            load_kq();
        }
    }
    if (warp == 0) tc::tmem_alloc(tmem_slot, 256);
    constexpr int SDN = ChainCfg<DH>::S_WARPS;
    const float sds = warp == 0 && lane < SDN && chunk + 1 < n_chunks ? SD[tix * SDN + lane] : 0.0f;   // <S, dS>'s parts (dS = 0 at the end)
    {
        const int t = tid & 63;
        const bool live = t < n;
        const int64_t r = (grow + (live ? t : 0)) * H + h;
        if (tid < 64) {
            g_s[t] = GB[tix * 128 + t];
            be_s[t] = GB[tix * 128 + 64 + t];
        } else if (tid < 128) {
            al_s[t] = alpha[r];
            float s = 0.0f, y = 0.0f;
#pragma unroll
            for (int i = 0; i < DH / 32; ++i) {
                s += VD[(tix * 2 * (DH / 32) + i) * 64 + t];
                y += VD[((tix * 2 + 1) * (DH / 32) + i) * 64 + t];
            }
            vd_s[t] = s;
            ky_s[t] = y;
        } else if (tid < 192) {
            nrm_s[t] = qnorm[r];
        } else {
            nrm_s[64 + t] = knorm[r];
        }
    }
    tc::tcgen05_fence_before();
    __syncthreads();
    tc::tcgen05_fence_after();
    const uint32_t tm = *tmem_slot;
    const uint32_t ACC_A = tm /* X | Y, then dq | dk */, ACC_D = tm + DH /* dL | dA, then K K^T | Q K^T */, ACC_W = tm + DH + 64 /* dW */;
    constexpr uint32_t H1 = 16u << 16;                    // lane offset of the second half
    const uint32_t lane_addr = (uint32_t)(wq * 32) << 16;
    const uint32_t sb = tc::smem_u32(sm);
    auto kmaj = [&](uint32_t off, int k16) { return tc::smem_desc_sw128(sb + off + k16 * 32, 16, 1024); };          // one 64-wide k box
    auto mnmaj = [&](uint32_t off, int k16) { return tc::smem_desc_sw128(sb + off + k16 * 2048, 8192, 1024); };     // 64 k rows, boxes 8 KiB apart
    auto tile = [&](uint32_t off, int r, int c16) -> uint4* {
        return reinterpret_cast<uint4*>(sm + off + (c16 >> 3) * 8192 + tc::sw128_off(r, c16 & 7));
    };
    // A wait that gives up raises *abort_flag; the CTA then runs to its end on whatever it has (every block barrier is reached by
    // every thread). The host sees the error word.
    auto wait_bar = [&](int i, uint32_t parity) {
        if (lane == 0) tc::mbar_wait(&bars[i], parity, abort_flag, err_word, 320 + i);
        __syncwarp();
        tc::tcgen05_fence_after();
    };

    // ---- first group
    constexpr uint32_t I64 = tc::idesc_bf16_f32(64, 64, 0, 0), IDH = tc::idesc_bf16_f32(64, DH, 0, 0);
    auto group1 = [&](int hv) {
        const uint32_t rows = hv * Cfg::R_ROWS, s0 = hv == 0 ? Cfg::R_S : Cfg::R_S1;
#pragma unroll
        for (int k16 = 0; k16 < 4; ++k16) {
            const uint32_t acc = hv > 0 || k16 > 0;
            const uint64_t dr = kmaj(rows + Cfg::R_DR, k16), dO = kmaj(rows + Cfg::R_DO, k16), u = kmaj(rows + Cfg::R_U, k16);
            tc::umma_bf16(ACC_D, dr, u, I64, acc);
            tc::umma_bf16(ACC_D + H1, dO, u, I64, acc);
            tc::umma_bf16(ACC_A, dO, kmaj(s0, k16), IDH, acc);
            tc::umma_bf16(ACC_A + H1, dr, kmaj(s0, k16), IDH, acc);
        }
    };
    auto products_dw = [&](int hv) {
        const uint32_t rows = hv * Cfg::R_ROWS, ds = hv == 0 ? Cfg::R_DS : Cfg::R_DS1;
#pragma unroll
        for (int k16 = 0; k16 < 4; ++k16) {
            const uint32_t acc = hv > 0 || k16 > 0;
            const uint64_t u = kmaj(rows + Cfg::R_U, k16);
            if constexpr (DH == 128) {   // keys 0-63 in half 0, 64-127 in half 1
                tc::umma_bf16(ACC_W, u, kmaj(ds, k16), I64, acc);
                tc::umma_bf16(ACC_W + H1, u, kmaj(ds + 8192, k16), I64, acc);
            } else {
                tc::umma_bf16(ACC_W + H1, u, kmaj(ds, k16), I64, acc);
            }
        }
    };
    wait_bar(0, 0);
    if (tid == 0) {
        group1(0);
        products_dw(0);
        tc::umma_commit(&bars[4]);
        if constexpr (DH == 128) {
            tc::mbar_wait(&bars[1], 0, abort_flag, err_word, 321);
            group1(1);
            tc::umma_commit(&bars[5]);
            if (tc::mbar_wait(&bars[4], 0, abort_flag, err_word, 324)) {
                tc::fence_proxy_async_smem();
                tc::mbar_expect_tx(&bars[2], Cfg::SB);
                tc::tma_load_2d(sm + Cfg::R_DS1, &mapDS, 64, (int)tix * DH, &bars[2]);
                load_kq();
            }
        }
    }
    const float g_row = g_s[row], be_row = be_s[row], gam = __expf(g_row), eg = __expf(g_s[C - 1] - g_row);
    wait_bar(3 + NB, 0);
    // ---- M (half 0) and P (half 1): 32 columns of a row per thread, rounded where the last dR and dO were
    float mp[32];
    {
        uint32_t r[32];
        tc::tmem_ld_32x32(ACC_D + lane_addr + cg * 32, r);
        tc::tmem_ld_wait();
        const float f = half == 0 ? -be_row : 1.0f;
        const int lim = row + half - cg * 32;   // M: i < row; P: i <= row
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            float x8[8];
            const float4 ga = *reinterpret_cast<const float4*>(g_s + cg * 32 + 8 * j), gb = *reinterpret_cast<const float4*>(g_s + cg * 32 + 8 * j + 4);
            const float g8[8] = {ga.x, ga.y, ga.z, ga.w, gb.x, gb.y, gb.z, gb.w};
            // Masked exponentials are skipped one by one at head dim 128 and all taken at 64, where the branches cost more than the
            // exponentials (64: 264 -> 228 us at 8192 chunks; 128 the other way about: 449 and 411).
#pragma unroll
            for (int e = 0; e < 8; ++e) x8[e] = DH == 64 ? exp_always(g_row - g8[e]) : 8 * j + e < lim ? __expf(g_row - g8[e]) : 0.0f;
#pragma unroll
            for (int e = 0; e < 8; ++e) mp[8 * j + e] = x8[e] = 8 * j + e < lim ? f * x8[e] * __uint_as_float(r[8 * j + e]) : 0.0f;
            *reinterpret_cast<uint4*>(sm + (half == 0 ? Cfg::R_M : Cfg::R_P) + tc::sw128_off(row, cg * 4 + j)) = tc::pack8_bf16(x8);
        }
    }
    tc::tcgen05_fence_before();
    __syncthreads();   // everybody has dL and dA
    wait_bar(3, 0);
    if (tid == 0) {
#pragma unroll
        for (int k16 = 0; k16 < DH / 16; ++k16) {
            const uint32_t off = (k16 >> 2) * 8192;
            tc::umma_bf16(ACC_D, kmaj(Cfg::R_K + off, k16 & 3), kmaj(Cfg::R_K + off, k16 & 3), I64, k16 > 0);
            tc::umma_bf16(ACC_D + H1, kmaj(Cfg::R_Q + off, k16 & 3), kmaj(Cfg::R_K + off, k16 & 3), I64, k16 > 0);
        }
        tc::umma_commit(&bars[7]);
        if constexpr (DH == 128) {
            tc::mbar_wait(&bars[2], 0, abort_flag, err_word, 322);
            products_dw(1);   // (finished when the second group is)
        }
    }
    __syncwarp();
    // ---- X *= gam, Y *= -beta gam; q . X
    {
        const float f = half == 0 ? gam : -be_row * gam;
        float qx = 0.0f;
#pragma unroll
        for (int pc = 0; pc < CW / 16; ++pc) {
            const int col = cg * CW + pc * 16;
            uint32_t r[16];
            tc::tmem_ld_32x16(ACC_A + lane_addr + col, r);
            tc::tmem_ld_wait();
#pragma unroll
            for (int j = 0; j < 2; ++j) {
                float q8[8];
                tc::unpack8_bf16(*tile(Cfg::R_Q, row, (col >> 3) + j), q8);
#pragma unroll
                for (int e = 0; e < 8; ++e) {
                    const float x = f * __uint_as_float(r[8 * j + e]);
                    qx = fmaf(q8[e], x, qx);
                    r[8 * j + e] = __float_as_uint(x);
                }
            }
            tc::tmem_st_32x16(ACC_A + lane_addr + col, r);
        }
        if (half == 0) qx_s[cg * 64 + row] = qx;
        tc::tmem_st_wait();
    }
    tc::fence_proxy_async_smem();
    tc::tcgen05_fence_before();
    __syncthreads();
    // ---- second group
    if (tid == 0) {
        constexpr uint32_t IKM = tc::idesc_bf16_f32(64, DH, 0, 1), IMM = tc::idesc_bf16_f32(64, DH, 1, 1);
        tc::tcgen05_fence_after();
#pragma unroll
        for (int k16 = 0; k16 < 4; ++k16) {
            const uint64_t kk = mnmaj(Cfg::R_K, k16);
            tc::umma_bf16(ACC_A, kmaj(Cfg::R_P, k16), kk, IKM, 1u);                                  // P K
            tc::umma_bf16(ACC_A + H1, mnmaj(Cfg::R_M, k16), kk, IMM, 1u);                            // M^T K
            tc::umma_bf16(ACC_A + H1, mnmaj(Cfg::R_P, k16), mnmaj(Cfg::R_Q, k16), IMM, 1u);          // P^T Q
            tc::umma_bf16(ACC_A + H1, kmaj(Cfg::R_M, k16), kk, IKM, 1u);                             // M K
        }
        tc::umma_commit(&bars[6]);
    }
    // ---- row and column sums of M o K K^T and P o Q K^T, while the second group runs
    wait_bar(7, 0);
    {
        uint32_t r[32];
        tc::tmem_ld_32x32(ACC_D + lane_addr + cg * 32, r);
        tc::tmem_ld_wait();
        float s = 0.0f;
#pragma unroll
        for (int j = 0; j < 32; ++j) {
            mp[j] *= __uint_as_float(r[j]);
            s += mp[j];
        }
        rs_s[cg * 128 + half * 64 + row] = s;
        // columns, over the warp's 16 rows of both: lane l ends with column l
#pragma unroll
        for (int w = 16; w > 0; w >>= 1) {
            const bool up = lane & w;
#pragma unroll
            for (int j = 0; j < w; ++j) {
                const float give = up ? mp[j] : mp[j + w];
                mp[j] = (up ? mp[j + w] : mp[j]) + __shfl_xor_sync(0xffffffffu, give, w);
            }
        }
        cs_s[wq * 64 + cg * 32 + lane] = mp[0];
    }
    wait_bar(6, 0);
    // ---- dq (half 0) and dk (half 1) before the norm's backward: back to TMEM; row sums
    const uint32_t ytile = half == 0 ? Cfg::R_Q : Cfg::R_K;
    {
        float dot = 0.0f, kws = 0.0f;
#pragma unroll
        for (int pc = 0; pc < CW / 16; ++pc) {
            const int col = cg * CW + pc * 16;
            uint32_t x[16], w[16];
            tc::tmem_ld_32x16(ACC_A + lane_addr + col, x);
            tc::tmem_ld_32x16(ACC_W + lane_addr + (DH == 128 ? pc * 16 : col), w);
            tc::tmem_ld_wait();
            if constexpr (DH == 128) {   // keys 64 cg .. of a row sit in half cg
                const int src = (lane & 15) | (cg << 4);
#pragma unroll
                for (int j = 0; j < 16; ++j) w[j] = __shfl_sync(0xffffffffu, w[j], src);
            }
#pragma unroll
            for (int j = 0; j < 2; ++j) {
                float y8[8];
                tc::unpack8_bf16(*tile(ytile, row, (col >> 3) + j), y8);
#pragma unroll
                for (int e = 0; e < 8; ++e) {
                    float g = __uint_as_float(x[8 * j + e]);
                    if (half == 1) {
                        const float w_ = eg * __uint_as_float(w[8 * j + e]);
                        g += w_;
                        kws = fmaf(y8[e], w_, kws);
                    }
                    dot = fmaf(y8[e], g, dot);
                    x[8 * j + e] = __float_as_uint(g);
                }
            }
            tc::tmem_st_32x16(ACC_A + lane_addr + col, x);
        }
        dot_s[cg * 128 + half * 64 + row] = dot;
        if (half == 1) kw_s[cg * 64 + row] = kws;
        tc::tmem_st_wait();
    }
    __syncthreads();
    // ---- L2-norm backward and store
    {
        const float dot = dot_s[half * 64 + row] + dot_s[128 + half * 64 + row], inv = 1.0f / nrm_s[half * 64 + row];
        float* dst = d_qkv + (grow + row) * 3 * d + half * d + h * DH;
#pragma unroll
        for (int pc = 0; pc < CW / 16; ++pc) {
            const int col = cg * CW + pc * 16;
            uint32_t x[16];
            tc::tmem_ld_32x16(ACC_A + lane_addr + col, x);
            tc::tmem_ld_wait();
            float f[16];
#pragma unroll
            for (int j = 0; j < 2; ++j) {
                float y8[8];
                tc::unpack8_bf16(*tile(ytile, row, (col >> 3) + j), y8);
#pragma unroll
                for (int e = 0; e < 8; ++e) f[8 * j + e] = (__uint_as_float(x[8 * j + e]) - y8[e] * dot) * inv;
            }
            if (row < n) store16(dst + col, f, w32);
        }
    }
    // ---- gates (warp 0): reverse cumulative sum, sigmoid backward
    if (warp == 0) {
        float s[2], w[2], kw = 0.0f;
#pragma unroll
        for (int i = 0; i < 2; ++i) {
            const int t = lane + 32 * i;
            const float kw_t = kw_s[t] + kw_s[64 + t];
            w[i] = rs_s[t] + rs_s[128 + t] + ky_s[t];
            s[i] = w[i] + (rs_s[64 + t] + rs_s[192 + t]) + (qx_s[t] + qx_s[64 + t]) - (cs_s[t] + cs_s[64 + t] + cs_s[128 + t] + cs_s[192 + t]) - kw_t;
            kw += kw_t;
        }
        const float extra = __expf(g_s[C - 1]) * warp_sum(sds) + warp_sum(kw);
        if (lane == 31) s[1] += extra;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {   // suffix sums over t = 0..63
            const float nb = __shfl_down_sync(0xffffffffu, s[1], o), na = __shfl_down_sync(0xffffffffu, s[0], o);
            if (lane + o < 32) {
                s[1] += nb;
                s[0] += na;
            }
        }
        s[0] += __shfl_sync(0xffffffffu, s[1], 0);
#pragma unroll
        for (int i = 0; i < 2; ++i) {
            const int t = lane + 32 * i;
            if (t < n) {
                float* dst = d_gate + (grow + t) * 2 * H + h;
                dst[0] = s[i] * (1.0f - al_s[t]);
                dst[H] = (vd_s[t] + w[i]) * (1.0f - be_s[t]);
            }
        }
    }
    tc::tcgen05_fence_before();
    __syncthreads();
    if (warp == 0) tc::tmem_dealloc(tm, 256);
    if (*abort_flag) __nanosleep(20000);
}

// ------------------------------------------------------------------ host side
typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                  const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                  CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
static EncodeTiledFn encode_fn() {
    static EncodeTiledFn fn = nullptr;
    if (!fn) {
        void* p = nullptr;
        cudaDriverEntryPointQueryResult qr;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &qr) == cudaSuccess &&
            qr == cudaDriverEntryPointSuccess)
            fn = (EncodeTiledFn)p;
    }
    return fn;
}
static bool make_map(CUtensorMap* m, const void* base, int64_t rows, int64_t cols, int box_cols, int box_rows) {
    EncodeTiledFn fn = encode_fn();
    if (!fn) return false;
    cuuint64_t dims[2] = {(cuuint64_t)cols, (cuuint64_t)rows};
    cuuint64_t strides[1] = {(cuuint64_t)cols * 2};
    cuuint32_t box[2] = {(cuuint32_t)box_cols, (cuuint32_t)box_rows};
    cuuint32_t estr[2] = {1, 1};
    return fn(m, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void*>(base), dims, strides, box, estr,
              CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
              CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

static bool make_map3(CUtensorMap* m, const void* base, int64_t B, int64_t T, int64_t cols) {   // (columns, tokens, sequences), 64 x 64 boxes
    EncodeTiledFn fn = encode_fn();
    if (!fn) return false;
    cuuint64_t dims[3] = {(cuuint64_t)cols, (cuuint64_t)T, (cuuint64_t)B};
    cuuint64_t strides[2] = {(cuuint64_t)cols * 2, (cuuint64_t)(T * cols) * 2};
    cuuint32_t box[3] = {64, C, 1};
    cuuint32_t estr[3] = {1, 1, 1};
    return fn(m, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3, const_cast<void*>(base), dims, strides, box, estr,
              CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
              CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

static inline size_t al(size_t x) { return (x + 1023) & ~(size_t)1023; }
static inline char* al_ptr(void* p) { return reinterpret_cast<char*>(al(reinterpret_cast<size_t>(p))); }

bool available() { return encode_fn() != nullptr; }

// Carves the per-(chain, chunk) buffers out of memory that starts on a 1024-byte boundary (null: counts).
struct Carver {
    char* base;
    size_t at = 0;
    template <typename P>
    P* take(int64_t n) {
        P* r = base ? reinterpret_cast<P*>(base + at) : nullptr;
        at += al((size_t)n * sizeof(P));
        return r;
    }
};
static void carve_kept(Carver& w, int64_t n_tiles, bool full, Tiles* t) {   // what a backward reads again
    t->AA = w.take<__nv_bfloat16>(n_tiles * C * C);
    t->AL = w.take<__nv_bfloat16>(n_tiles * C * C);
    t->TP = full ? w.take<__nv_bfloat16>(n_tiles * C * C) : nullptr;
    t->GB = w.take<float>(n_tiles * 2 * C);
}
static void carve_rows(Carver& w, int64_t n_tiles, int64_t dh, Tiles* t) {
    t->WH = w.take<__nv_bfloat16>(n_tiles * C * dh);
    t->UV = w.take<__nv_bfloat16>(n_tiles * C * dh);
}

template <int DH>
static int run_prepass(asca_ctx* ctx, const void* q, const void* k, const void* v, const float* alpha, const float* beta, int64_t B, int64_t T,
                       int64_t H, int64_t n_chunks, const Tiles& t) {
    CUtensorMap mK, mQ, mV, mWH, mUV;
    const int64_t n_tiles = B * H * n_chunks;
    if (!make_map3(&mK, k, B, T, H * DH) || !make_map3(&mQ, q, B, T, H * DH) || !make_map3(&mV, v, B, T, H * DH) ||
        !make_map(&mWH, t.WH, n_tiles * C, DH, 64, C) || !make_map(&mUV, t.UV, n_tiles * C, DH, 64, C))
        return asca_fail(ctx, ASCA_ERR_CUDA, "delta_tc: cuTensorMapEncodeTiled failed");
    auto kern = delta_prep_tc_kernel<DH>;
    ASCA_CUDA(ctx, cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)pre_smem<DH>()));
    {
        asca_span sp(ctx, "delta_prep_tc_kernel");
        kern<<<dim3((unsigned)n_chunks, (unsigned)(B * H)), PRE_THREADS, pre_smem<DH>(), ctx->stream>>>(
            mK, mQ, mV, mWH, mUV, alpha, beta, (int)T, (int)H, (int)n_chunks, t, ctx->err_word);
    }
    ASCA_CHECK_LAUNCH(ctx);
    return ASCA_OK;
}

// Forward for bf16 q, k, v. o is bf16. When checkpoints are requested (a backward will follow) the buffer receives, as bf16, the
// chunk-start states (B, H, n_chunks, dh, dh) in its first half and the rows U (B, H, n_chunks, 64, dh) behind them; A, X - I and the
// decays stay in a context-owned buffer keyed by the checkpoint pointer, so that the backward does not repeat the pre-pass.
template <int DH>
static int forward_dh(asca_ctx* ctx, const void* q, const void* k, const void* v, const float* alpha, const float* beta,
                      int64_t B, int64_t T, int64_t H, void* o, const float* s_init, float* s_final, float* ckpt) {
    const int64_t n_chunks = (T + C - 1) / C, chains = B * H, n_tiles = chains * n_chunks;
    Tiles t{};
    const bool keep = ckpt != nullptr;
    int slot = -1;
    void* ws;
    if (keep) {
        Carver kept{nullptr}, rows{nullptr};
        carve_kept(kept, n_tiles, true, &t);
        carve_rows(rows, n_tiles, DH, &t);
        const size_t need = kept.at + 1024;
        auto& dt = ctx->dtiles;
        for (size_t i = 0; i < dt.size(); ++i)
            if (dt[i].buf && dt[i].ckpt == (const void*)ckpt) slot = (int)i;
        if (slot < 0) {   // a free entry, a new one, or the least recently used one
            for (size_t i = 0; i < dt.size() && slot < 0; ++i)
                if (!dt[i].ckpt) slot = (int)i;
            size_t total = 0;
            for (auto& e : dt) total += e.bytes;
            if (slot < 0 && dt.size() < 32 && total + need <= ctx->dtiles_cap) {
                dt.emplace_back();
                slot = (int)dt.size() - 1;
            }
            if (slot < 0) {
                slot = 0;
                for (size_t i = 1; i < dt.size(); ++i)
                    if (dt[i].stamp < dt[slot].stamp) slot = (int)i;
            }
        }
        auto& e = dt[slot];
        e.ckpt = nullptr;   // invalid until this forward has been queued
        if (need > e.bytes) {
            ASCA_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
            if (e.buf) cudaFree(e.buf);
            e.buf = nullptr;
            e.bytes = 0;
            ASCA_CUDA(ctx, cudaMalloc(&e.buf, need));
            e.bytes = need;
        }
        kept = Carver{al_ptr(e.buf)};
        carve_kept(kept, n_tiles, true, &t);
        ASCA_TRY(asca_workspace(ctx, rows.at + 1024, &ws));
        rows = Carver{al_ptr(ws)};
        carve_rows(rows, n_tiles, DH, &t);
    } else {
        Carver w{nullptr};
        carve_kept(w, n_tiles, false, &t);
        carve_rows(w, n_tiles, DH, &t);
        ASCA_TRY(asca_workspace(ctx, w.at + 1024, &ws));
        w = Carver{al_ptr(ws)};
        carve_kept(w, n_tiles, false, &t);
        carve_rows(w, n_tiles, DH, &t);
    }
    ASCA_TRY((run_prepass<DH>(ctx, q, k, v, alpha, beta, B, T, H, n_chunks, t)));
    CUtensorMap mWH, mQ, mK, mUV, mAA, mAL, mS0, mU;
    const char* u_rows = reinterpret_cast<const char*>(ckpt) + (size_t)n_tiles * DH * DH * 2;
    if (!make_map(&mWH, t.WH, n_tiles * C, DH, 64, C) || !make_map3(&mQ, q, B, T, H * DH) || !make_map3(&mK, k, B, T, H * DH) ||
        !make_map(&mUV, t.UV, n_tiles * C, DH, 64, C) || !make_map(&mAA, t.AA, n_tiles * C, C, 64, C) ||
        !make_map(&mAL, t.AL, n_tiles * C, C, 64, C) ||
        !(keep ? make_map(&mS0, ckpt, n_tiles * DH, DH, 64, DH) && make_map(&mU, u_rows, n_tiles * C, DH, 64, C)
               : make_map(&mS0, t.WH, n_tiles * C, DH, 64, C) && make_map(&mU, t.WH, n_tiles * C, DH, 64, C)))   // (unused)
        return asca_fail(ctx, ASCA_ERR_CUDA, "delta_tc: cuTensorMapEncodeTiled failed");
    using Cfg = ChainCfg<DH>;
    auto kern = delta_fwd_tc_kernel<DH>;
    ASCA_CUDA(ctx, cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)Cfg::F_SMEM));
    {
        asca_span sp(ctx, "delta_fwd_tc_kernel");
        kern<<<(unsigned)chains, Cfg::THREADS, Cfg::F_SMEM, ctx->stream>>>(mWH, mQ, mK, mUV, mAA, mAL, mS0, mU, t.GB, (int)T, (int)H, (int)n_chunks,
                                                                           (__nv_bfloat16*)o, s_init, s_final, keep ? 1 : 0, chains <= ctx->sm_count, ctx->err_word);
    }
    ASCA_CHECK_LAUNCH(ctx);
    if (keep) {
        auto& e = ctx->dtiles[slot];
        e.ckpt = ckpt;
        e.q = q; e.k = k; e.v = v; e.alpha = alpha; e.beta = beta;
        e.B = B;
        e.T = T;
        e.H = H * 1024 + DH;   // heads and head dim in one key field
        e.stamp = ++ctx->dtiles_clock;
    }
    return ASCA_OK;
}

int forward(asca_ctx* ctx, const void* q, const void* k, const void* v, const float* alpha, const float* beta,
            int64_t B, int64_t T, int64_t H, int64_t dh, void* o, const float* s_init, float* s_final, float* ckpt) {
    if (s_final && (reinterpret_cast<uintptr_t>(s_final) & 15)) {   // the kernel writes the final state 16 bytes at a time
        const size_t bytes = (size_t)(B * H * dh * dh) * 4;
        void* fin;
        ASCA_TRY(asca_malloc(ctx, bytes, &fin));
        int rc = forward(ctx, q, k, v, alpha, beta, B, T, H, dh, o, s_init, (float*)fin, ckpt);
        if (rc == ASCA_OK && cudaMemcpyAsync(s_final, fin, bytes, cudaMemcpyDeviceToDevice, ctx->stream) != cudaSuccess)
            rc = asca_fail(ctx, ASCA_ERR_CUDA, "delta_fwd: cannot copy the final state");
        asca_free(ctx, fin);   // (reused by later work on the stream only)
        return rc;
    }
    return dh == 128 ? forward_dh<128>(ctx, q, k, v, alpha, beta, B, T, H, o, s_init, s_final, ckpt)
                     : forward_dh<64>(ctx, q, k, v, alpha, beta, B, T, H, o, s_init, s_final, ckpt);
}

// Backward for bf16 q, k, v, d_o (checkpoints every 64 tokens from the forward).
template <int DH>
static int backward_dh(asca_ctx* ctx, const void* q, const void* k, const void* v, const float* alpha, const float* beta,
                       const float* qnorm, const float* knorm, const void* d_o, const float* ckpt, int64_t B, int64_t T, int64_t H,
                       float* d_qkv, float* d_gate) {
    const int64_t n_chunks = (T + C - 1) / C, chains = B * H, n_tiles = chains * n_chunks;
    Tiles t{};
    int slot = -1;
    for (size_t i = 0; i < ctx->dtiles.size(); ++i) {
        const auto& e = ctx->dtiles[i];
        // the tiles are functions of q, k, v, alpha, beta: the same buffers must come back (their contents are the
        // caller's contract, see the header); anything else rebuilds the tiles
        if (e.buf && e.ckpt == (const void*)ckpt && e.q == q && e.k == k && e.v == v && e.alpha == (const void*)alpha &&
            e.beta == (const void*)beta && e.B == B && e.T == T && e.H == H * 1024 + DH)
            slot = (int)i;
    }
    __nv_bfloat16 *dS, *dR;
    float *VD, *SD;
    void* ws;
    for (int pass = 0; pass < 2; ++pass) {   // count, then carve
        Carver w{pass ? al_ptr(ws) : nullptr};
        dS = w.take<__nv_bfloat16>(n_tiles * DH * DH);
        dR = w.take<__nv_bfloat16>(n_tiles * C * DH);
        VD = w.take<float>(n_tiles * 2 * C * (DH / 32));
        SD = w.take<float>(n_tiles * ChainCfg<DH>::S_WARPS);
        if (slot < 0) {
            carve_kept(w, n_tiles, true, &t);
            carve_rows(w, n_tiles, DH, &t);
        }
        if (!pass) ASCA_TRY(asca_workspace(ctx, w.at + 1024, &ws));
    }
    if (slot >= 0) {   // the forward that wrote `ckpt` left its tiles here
        ctx->dtiles[slot].stamp = ++ctx->dtiles_clock;
        Carver kept{al_ptr(ctx->dtiles[slot].buf)};
        carve_kept(kept, n_tiles, true, &t);
    } else {
        ASCA_TRY((run_prepass<DH>(ctx, q, k, v, alpha, beta, B, T, H, n_chunks, t)));
    }
    CUtensorMap mK, mQ, mV, mDO, mAA, mAL, mTP, mDS, mDR, mS0, mU;
    const char* u_rows = reinterpret_cast<const char*>(ckpt) + (size_t)n_tiles * DH * DH * 2;
    if (!make_map3(&mK, k, B, T, H * DH) || !make_map3(&mQ, q, B, T, H * DH) || !make_map3(&mV, v, B, T, H * DH) || !make_map3(&mDO, d_o, B, T, H * DH) ||
        !make_map(&mAA, t.AA, n_tiles * C, C, 64, C) || !make_map(&mAL, t.AL, n_tiles * C, C, 64, C) ||
        !make_map(&mTP, t.TP, n_tiles * C, C, 64, C) ||
        !make_map(&mDS, dS, n_tiles * DH, DH, 64, DH) || !make_map(&mDR, dR, n_tiles * C, DH, 64, C) ||
        !make_map(&mS0, ckpt, n_tiles * DH, DH, 64, DH) || !make_map(&mU, u_rows, n_tiles * C, DH, 64, C))
        return asca_fail(ctx, ASCA_ERR_CUDA, "delta_tc: cuTensorMapEncodeTiled failed");
    using Cfg = ChainCfg<DH>;
    auto chain = delta_bwd_tc_kernel<DH>;
    ASCA_CUDA(ctx, cudaFuncSetAttribute(chain, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)Cfg::B_SMEM));
    {
        asca_span sp(ctx, "delta_bwd_tc_kernel");
        chain<<<(unsigned)chains, Cfg::THREADS, Cfg::B_SMEM, ctx->stream>>>(mK, mQ, mDO, mAA, mAL, mTP, mDS, mDR, mV, mS0, t.GB, (const __nv_bfloat16*)v,
                                                                            (int)T, (int)H, (int)n_chunks, d_qkv, VD, SD, chains <= ctx->sm_count, ctx->err_word);
    }
    ASCA_CHECK_LAUNCH(ctx);
    auto grad = delta_grad_tc_kernel<DH>;
    ASCA_CUDA(ctx, cudaFuncSetAttribute(grad, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)GradCfg<DH>::SMEM));
    {
        asca_span sp(ctx, "delta_grad_tc_kernel");
        grad<<<dim3((unsigned)n_chunks, (unsigned)chains), GR_THREADS, GradCfg<DH>::SMEM, ctx->stream>>>(
            mK, mQ, mDO, mDR, mU, mS0, mDS, t.GB, VD, SD, alpha, qnorm, knorm, (int)T, (int)H, (int)n_chunks, d_qkv, d_gate, ctx->err_word);
    }
    ASCA_CHECK_LAUNCH(ctx);
    return ASCA_OK;
}

int backward(asca_ctx* ctx, const void* q, const void* k, const void* v, const float* alpha, const float* beta,
             const float* qnorm, const float* knorm, const void* d_o, const float* ckpt, int64_t B, int64_t T, int64_t H,
             int64_t dh, float* d_qkv, float* d_gate) {
    ASCA_REQUIRE(ctx, (reinterpret_cast<uintptr_t>(d_qkv) & 15) == 0, "delta_bwd: d_qkv must be 16-byte aligned in tensor-core mode");
    return dh == 128 ? backward_dh<128>(ctx, q, k, v, alpha, beta, qnorm, knorm, d_o, ckpt, B, T, H, d_qkv, d_gate)
                     : backward_dh<64>(ctx, q, k, v, alpha, beta, qnorm, knorm, d_o, ckpt, B, T, H, d_qkv, d_gate);
}

}  // namespace delta_tc
