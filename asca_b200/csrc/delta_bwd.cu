// Gated delta rule, BPTT backward, f32-exact, as a reverse CHUNKED scan.
//
// The reference walks time backwards one step at a time and reads two full dh x dh states per
// step from a (T+1)*dh*dh history (rust/src/delta.rs:485-572, rust/kernels/asca.cu:340-485).
// Here no per-step state exists. The forward leaves one state per `chunk` tokens; one CTA per
// (sequence, head) walks those checkpoints in reverse, and inside a checkpoint interval works
// on sub-chunks of C tokens in the WY/UT form:
//
//   g_t = sum_{j<=t} log(alpha_j), gam = exp(g), Gam[t,i] = exp(g_t - g_i) (i <= t, always <= 1)
//   L = strictlower(beta_t Gam (K K^T)),  A = lower(Gam (Q K^T)),  eg_t = exp(g_last - g_t)
//   Z = V - diag(gam) K S0,  U = (I+L)^-1 diag(beta) Z            (forward recompute)
//   dU  = A^T dO + diag(eg) K dS          dR = (I+L)^-T dU        dV = diag(beta) dR = dZ
//   dL  = -strictlower(dR U^T)            dA = lower(dO U^T)
//   dbeta_t = dR_t.Z_t + sum_i dL[t,i] Gam[t,i] (k_t.k_i)
//   dQ  = diag(gam) dO S0^T + (dA.Gam) K
//   dK  = (dA.Gam)^T Q + (M + M^T) K + diag(eg) U dS^T - diag(gam) dZ S0^T,  M = dL.beta_t.Gam
//   dg_t = rowsum_t(P) - colsum_t(P) + gam_t q_t.(S0 dO_t) + gam_t k_t.dKg_t - eg_t k_t.dW_t,
//          P = (dA.Gam).(Q K^T) + M.(K K^T);  dg_last += sum_t eg_t k_t.dW_t + gam_last <S0,dS>
//   dlogalpha_j = sum_{t>=j} dg_t;   d_gate_alpha = dlogalpha (1 - alpha)
//   dS0 = gam_last dS + (diag(gam) Q)^T dO - (diag(gam) K)^T dZ    -> dS of the previous sub-chunk
//
// followed in the same kernel by the per-head L2-norm backward (rust/src/delta.rs:678-698), the
// sigmoid backward and the [dq|dk|dv] concat (rust/src/delta.rs:594-611). When a checkpoint
// interval spans several sub-chunks, the states at the inner boundaries are first recomputed
// forward (S_C = gam_last S0 + (diag(eg) K)^T U) into a small per-CTA scratch that stays in L2.
//
// All products are FFMA with f32 accumulation from shared memory; row strides are padded by 4
// floats so float4 reads along a row are aligned and rows fall in different banks.
#include "common.cuh"

#include <algorithm>

bool asca_tc_enabled();  // gemm.cu
namespace delta_tc {
bool available();
int backward(asca_ctx* ctx, const void* q, const void* k, const void* v, const float* alpha, const float* beta,
             const float* qnorm, const float* knorm, const void* d_o, const float* ckpt, int64_t B, int64_t T, int64_t H,
             int64_t dh, float* d_qkv, float* d_gate);
}  // namespace delta_tc

namespace {

constexpr int BT = 256;  // threads per CTA

enum { L_MK = 0, L_KM = 1 };  // A operand layout: [m][k] or [k][m]
enum { L_KN = 0, L_NK = 1 };  // B operand layout: [k][n] or [n][k]

// C[m][n] = sum_k A(m,k) B(k,n) for an M x N output with N % 4 == 0 and operands in shared
// memory (lda/ldb multiples of 4, 16-byte aligned). Threads tile the output TM x 4; `epi(m, n,
// acc)` receives each finished element. K % 4 == 0 where an operand is contiguous along k.
template <int M, int N, int K, int ALAY, int BLAY, class Epi>
__device__ __forceinline__ void cta_gemm(const float* __restrict__ A, int lda, const float* __restrict__ B, int ldb,
                                         Epi epi) {
    constexpr int TN = 4;
    constexpr int THR_N = N / TN;
    constexpr int THR_M_MAX = BT / THR_N > 0 ? BT / THR_N : 1;
    constexpr int THR_M = THR_M_MAX < M ? THR_M_MAX : M;
    constexpr int TM = M / THR_M;
    constexpr bool KM_VEC = ALAY == L_KM && BLAY == L_KN && TM % 4 == 0 && THR_N % 32 == 0;
    static_assert(N % TN == 0 && THR_N <= BT && M % THR_M == 0, "tile shape");
    const int tid = threadIdx.x;
    if (tid >= THR_N * THR_M) return;
    const int tn = tid % THR_N, tm = tid / THR_N;
    const int n0 = tn * TN;
    // rows of this thread: m = tm + THR_M * i  (interleaved so KM loads stay scalar-broadcast)
    float acc[TM][TN];
#pragma unroll
    for (int i = 0; i < TM; ++i)
#pragma unroll
        for (int j = 0; j < TN; ++j) acc[i][j] = 0.0f;
    constexpr int UNR = TM <= 2 ? 4 : 2;   // small register tiles: more k-steps of loads in flight per warp
    if (ALAY == L_MK && BLAY == L_KN) {
#pragma unroll UNR
        for (int k = 0; k < K; k += 4) {
            float4 a[TM];
#pragma unroll
            for (int i = 0; i < TM; ++i) a[i] = *reinterpret_cast<const float4*>(A + (tm + THR_M * i) * lda + k);
#pragma unroll
            for (int kk = 0; kk < 4; ++kk) {
                const float4 b = *reinterpret_cast<const float4*>(B + (k + kk) * ldb + n0);
#pragma unroll
                for (int i = 0; i < TM; ++i) {
                    const float av = kk == 0 ? a[i].x : kk == 1 ? a[i].y : kk == 2 ? a[i].z : a[i].w;
                    acc[i][0] = fmaf(av, b.x, acc[i][0]);
                    acc[i][1] = fmaf(av, b.y, acc[i][1]);
                    acc[i][2] = fmaf(av, b.z, acc[i][2]);
                    acc[i][3] = fmaf(av, b.w, acc[i][3]);
                }
            }
        }
    } else if (ALAY == L_KM && BLAY == L_KN) {
        if (KM_VEC) {   // rows tm * TM + i: the lanes of a warp share tm, so A arrives as broadcast float4 loads
#pragma unroll 2
            for (int k = 0; k < K; ++k) {
                const float4 b = *reinterpret_cast<const float4*>(B + k * ldb + n0);
#pragma unroll
                for (int i4 = 0; i4 < TM / 4; ++i4) {
                    const float4 a4 = *reinterpret_cast<const float4*>(A + k * lda + tm * TM + 4 * i4);
                    const float av[4] = {a4.x, a4.y, a4.z, a4.w};
#pragma unroll
                    for (int e = 0; e < 4; ++e) {
                        acc[4 * i4 + e][0] = fmaf(av[e], b.x, acc[4 * i4 + e][0]);
                        acc[4 * i4 + e][1] = fmaf(av[e], b.y, acc[4 * i4 + e][1]);
                        acc[4 * i4 + e][2] = fmaf(av[e], b.z, acc[4 * i4 + e][2]);
                        acc[4 * i4 + e][3] = fmaf(av[e], b.w, acc[4 * i4 + e][3]);
                    }
                }
            }
        } else {
#pragma unroll 4
            for (int k = 0; k < K; ++k) {
                const float4 b = *reinterpret_cast<const float4*>(B + k * ldb + n0);
#pragma unroll
                for (int i = 0; i < TM; ++i) {
                    const float av = A[k * lda + tm + THR_M * i];
                    acc[i][0] = fmaf(av, b.x, acc[i][0]);
                    acc[i][1] = fmaf(av, b.y, acc[i][1]);
                    acc[i][2] = fmaf(av, b.z, acc[i][2]);
                    acc[i][3] = fmaf(av, b.w, acc[i][3]);
                }
            }
        }
    } else {  // L_MK x L_NK: both contiguous along k; this thread's columns are tn + THR_N * j, so that the lanes of a
              // quarter warp read 8 consecutive rows of B (row stride = 4 banks: all 32 banks, no conflict)
#pragma unroll UNR
        for (int k = 0; k < K; k += 4) {
            float4 b[TN];
#pragma unroll
            for (int j = 0; j < TN; ++j) b[j] = *reinterpret_cast<const float4*>(B + (tn + THR_N * j) * ldb + k);
#pragma unroll
            for (int i = 0; i < TM; ++i) {
                const float4 a = *reinterpret_cast<const float4*>(A + (tm + THR_M * i) * lda + k);
#pragma unroll
                for (int j = 0; j < TN; ++j) {
                    acc[i][j] = fmaf(a.x, b[j].x, acc[i][j]);
                    acc[i][j] = fmaf(a.y, b[j].y, acc[i][j]);
                    acc[i][j] = fmaf(a.z, b[j].z, acc[i][j]);
                    acc[i][j] = fmaf(a.w, b[j].w, acc[i][j]);
                }
            }
        }
    }
#pragma unroll
    for (int i = 0; i < TM; ++i)
#pragma unroll
        for (int j = 0; j < TN; ++j)
            epi(KM_VEC ? tm * TM + i : tm + THR_M * i, (ALAY == L_MK && BLAY == L_NK) ? tn + THR_N * j : n0 + j, acc[i][j]);
}

// dst[t][c] = src[(row0 + t) ld + col0 + c] for t < n, zero for n <= t < C
template <typename T>
__device__ __forceinline__ void load_rows(const T* __restrict__ src, int64_t row0, int64_t ld, int col0, int n, int C,
                                          int W, float* __restrict__ dst, int ldd) {
    // dst[t][c] = src[(row0+t)*ld + col0 + c] for t < n, zero for n <= t < C.  W % 4 == 0.
    const int w4 = W / 4;
    for (int idx = threadIdx.x; idx < C * w4; idx += BT) {
        const int t = idx / w4, c = (idx % w4) * 4;
        float4 val = make_float4(0, 0, 0, 0);
        if (t < n) {
            const T* p = src + (row0 + t) * ld + col0 + c;
            if (sizeof(T) == 4) {
                val = *reinterpret_cast<const float4*>(p);
            } else {
                uint2 raw = *reinterpret_cast<const uint2*>(p);
                __nv_bfloat162 a = *reinterpret_cast<__nv_bfloat162*>(&raw.x),
                               b = *reinterpret_cast<__nv_bfloat162*>(&raw.y);
                val = make_float4(__low2float(a), __high2float(a), __low2float(b), __high2float(b));
            }
        }
        *reinterpret_cast<float4*>(dst + t * ldd + c) = val;
    }
}

template <int DH, int C>
struct BwdSmem {
    static constexpr int LDK = DH + 4;   // K, Q, bufA, bufB rows
    static constexpr int LDV = DH + 4;   // value-width rows (Z, U, dO, dR, S0, dS)
    static constexpr int LDC = C + 4;    // C x C rows
    static constexpr int N_CC = 7;       // KK, QK, Gam, L, A, dL/M, dA
    static constexpr int floats = 2 * C * LDK      /* K, Q */
                                  + 4 * C * LDV    /* Z, U, dO, dR */
                                  + 2 * DH * LDV   /* S0, dS */
                                  + 2 * C * LDK    /* bufA, bufB */
                                  + N_CC * C * LDC + 16 * C + 64;
    static constexpr size_t bytes = (size_t)floats * 4;
};

template <int DH, int C, typename T>
__global__ void __launch_bounds__(BT, 1) delta_bwd_kernel(
    const T* __restrict__ q, const T* __restrict__ k, const T* __restrict__ v, const float* __restrict__ alpha,
    const float* __restrict__ beta, const float* __restrict__ qnorm, const float* __restrict__ knorm,
    const T* __restrict__ d_o, const float* __restrict__ ckpt, float* __restrict__ sub_ckpt, int B, int Tlen, int H,
    int chunk, float* __restrict__ d_qkv, float* __restrict__ d_gate) {
    using SM = BwdSmem<DH, C>;
    constexpr int LDK = SM::LDK, LDV = SM::LDV, LDC = SM::LDC;
    static_assert(C <= 32, "the gate scans run in one warp");
    extern __shared__ __align__(16) float smem[];
    float* Ks = smem;
    float* Qs = Ks + C * LDK;
    float* Zs = Qs + C * LDK;     // V, then Z = V - gam K S0
    float* Us = Zs + C * LDV;     // R = beta Z, then U
    float* dOs = Us + C * LDV;
    float* dRs = dOs + C * LDV;   // dU -> dR -> dZ
    float* S0 = dRs + C * LDV;
    float* dS = S0 + DH * LDV;
    float* bufA = dS + DH * LDV;
    float* bufB = bufA + C * LDK;
    float* KK = bufB + C * LDK;
    float* QK = KK + C * LDC;
    float* Gm = QK + C * LDC;
    float* Lm = Gm + C * LDC;
    float* Am = Lm + C * LDC;
    float* dLm = Am + C * LDC;
    float* dAm = dLm + C * LDC;
    float* vec = dAm + C * LDC;
    float* g_s = vec;             // cumulative log alpha
    float* gam_s = vec + C;       // exp(g)
    float* eg_s = vec + 2 * C;    // exp(g_last - g)
    float* be_s = vec + 3 * C;    // beta (0 on padded steps)
    float* al_s = vec + 4 * C;    // alpha (1 on padded steps)
    float* r_qs = vec + 5 * C;    // gam_t q_t.(S0 dO_t)
    float* r_kg = vec + 6 * C;    // gam_t k_t.dKg_t
    float* r_kw = vec + 7 * C;    // eg_t k_t.dW_t
    float* dbe_s = vec + 8 * C;   // dbeta
    float* dg_s = vec + 9 * C;    // dg
    float* red = vec + 16 * C;    // 33 floats

    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int chain = blockIdx.x;
    const int bi = chain / H, h = chain % H;
    const int d = H * DH;
    const int64_t row0 = (int64_t)bi * Tlen;
    const int n_ck = (Tlen + chunk - 1) / chunk;
    const int sub_per_ck = (chunk + C - 1) / C;
    float* my_sub = sub_ckpt + (int64_t)chain * sub_per_ck * DH * DH;

    for (int i = tid; i < DH * LDV; i += BT) dS[i] = 0.0f;

    auto load_state = [&](const float* src) {
        for (int idx = tid; idx < DH * (DH / 4); idx += BT) {
            const int a = idx / (DH / 4), c = (idx % (DH / 4)) * 4;
            *reinterpret_cast<float4*>(S0 + a * LDV + c) = *reinterpret_cast<const float4*>(src + a * DH + c);
        }
    };
    auto store_state = [&](float* dst) {
        for (int idx = tid; idx < DH * (DH / 4); idx += BT) {
            const int a = idx / (DH / 4), c = (idx % (DH / 4)) * 4;
            *reinterpret_cast<float4*>(dst + a * DH + c) = *reinterpret_cast<const float4*>(S0 + a * LDV + c);
        }
    };

    // Shared front part of a sub-chunk starting at token t0 with n live steps: loads K (and Q,
    // dO when `full`), V, gates; builds g, gam, eg, Gam, KK, L (and QK, A); Z, R; solves U.
    auto chunk_front = [&](int t0, int n, bool full) {
        load_rows<T>(k, row0 + t0, d, h * DH, n, C, DH, Ks, LDK);
        load_rows<T>(v, row0 + t0, d, h * DH, n, C, DH, Zs, LDV);
        if (full) {
            load_rows<T>(q, row0 + t0, d, h * DH, n, C, DH, Qs, LDK);
            load_rows<T>(d_o, row0 + t0, d, h * DH, n, C, DH, dOs, LDV);
        }
        if (tid < C) {
            const bool live = tid < n;
            const float a = live ? alpha[(row0 + t0 + tid) * H + h] : 1.0f;
            al_s[tid] = a;
            be_s[tid] = live ? beta[(row0 + t0 + tid) * H + h] : 0.0f;
            g_s[tid] = logf(a);
        }
        __syncthreads();
        if (warp == 0) {   // inclusive scan of the C (<= 32) log alphas, left to right
            float gx = lane < C ? g_s[lane] : 0.0f;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const float y = __shfl_up_sync(0xffffffffu, gx, o);
                if (lane >= o) gx += y;
            }
            if (lane < C) g_s[lane] = gx;
        }
        __syncthreads();
        if (tid < C) {
            gam_s[tid] = expf(g_s[tid]);
            eg_s[tid] = expf(g_s[C - 1] - g_s[tid]);
        }
        for (int idx = tid; idx < C * C; idx += BT) {
            const int t = idx / C, i = idx % C;
            Gm[t * LDC + i] = i <= t ? expf(g_s[t] - g_s[i]) : 0.0f;
        }
        __syncthreads();
        // KK = K K^T (and QK = Q K^T): one output element per thread pass
        for (int idx = tid; idx < C * C; idx += BT) {
            const int t = idx / C, i = idx % C;
            float s1 = 0.0f, s2 = 0.0f;
            const float* kt = Ks + t * LDK;
            const float* ki = Ks + i * LDK;
            const float* qt = Qs + t * LDK;
#pragma unroll 4
            for (int a = 0; a < DH; a += 4) {
                const float4 x = *reinterpret_cast<const float4*>(kt + a), y = *reinterpret_cast<const float4*>(ki + a);
                s1 = fmaf(x.x, y.x, s1); s1 = fmaf(x.y, y.y, s1); s1 = fmaf(x.z, y.z, s1); s1 = fmaf(x.w, y.w, s1);
                if (full) {
                    const float4 z = *reinterpret_cast<const float4*>(qt + a);
                    s2 = fmaf(z.x, y.x, s2); s2 = fmaf(z.y, y.y, s2); s2 = fmaf(z.z, y.z, s2); s2 = fmaf(z.w, y.w, s2);
                }
            }
            const float gm = Gm[t * LDC + i];
            KK[t * LDC + i] = s1;
            Lm[t * LDC + i] = i < t ? be_s[t] * gm * s1 : 0.0f;
            if (full) {
                QK[t * LDC + i] = s2;
                Am[t * LDC + i] = gm * s2;  // gm is 0 above the diagonal
            }
        }
        // Z = V - gam K S0 ; R = beta Z
        cta_gemm<C, DH, DH, L_MK, L_KN>(Ks, LDK, S0, LDV, [&](int t, int c, float acc) {
            const float z = Zs[t * LDV + c] - gam_s[t] * acc;
            Zs[t * LDV + c] = z;
            Us[t * LDV + c] = be_s[t] * z;
        });
        __syncthreads();
        // U = (I + L)^-1 R : one thread per value column, forward substitution in registers
        if (tid < DH) {
            float x[C];
#pragma unroll
            for (int t = 0; t < C; ++t) {
                float s = Us[t * LDV + tid];
#pragma unroll
                for (int i = 0; i < t; ++i) s = fmaf(-Lm[t * LDC + i], x[i], s);
                x[t] = s;
                Us[t * LDV + tid] = s;
            }
        }
        __syncthreads();
    };

    for (int ck = n_ck - 1; ck >= 0; --ck) {
        const int t_lo = ck * chunk;
        const int t_hi = t_lo + chunk < Tlen ? t_lo + chunk : Tlen;
        const int nsub = (t_hi - t_lo + C - 1) / C;
        const float* ck_state = ckpt + ((int64_t)chain * n_ck + ck) * DH * DH;

        // ---- phase F: states at the inner sub-chunk boundaries
        if (nsub > 1) {
            __syncthreads();
            load_state(ck_state);
            __syncthreads();
            for (int j = 0; j + 1 < nsub; ++j) {
                chunk_front(t_lo + j * C, C, false);
                // S0 <- gam_last S0 + (diag(eg) K)^T U
                for (int idx = tid; idx < C * DH; idx += BT) {
                    const int t = idx / DH, a = idx % DH;
                    bufA[t * LDK + a] = eg_s[t] * Ks[t * LDK + a];
                }
                __syncthreads();
                const float gl = gam_s[C - 1];
                cta_gemm<DH, DH, C, L_KM, L_KN>(bufA, LDK, Us, LDV, [&](int a, int c, float acc) {
                    S0[a * LDV + c] = fmaf(gl, S0[a * LDV + c], acc);
                });
                __syncthreads();
                store_state(my_sub + (int64_t)(j + 1) * DH * DH);
                __syncthreads();
            }
        }

        // the interval processed next (the one before this): its k, v rows and its checkpoint are requested into L2 now,
        // so that its phase F does not start on DRAM latency (q and dO of an interval are re-read shortly after phase F)
        if (ck > 0) {
            const int p_lo = (ck - 1) * chunk;
            constexpr int LPR = DH * (int)sizeof(T) / 128 > 0 ? DH * (int)sizeof(T) / 128 : 1;   // 128-byte lines per row
            for (int idx = tid; idx < chunk * LPR * 2; idx += BT) {
                const int which = idx / (chunk * LPR), rem = idx % (chunk * LPR);
                const T* base = which == 0 ? k : v;
                const char* ptr = reinterpret_cast<const char*>(base + (row0 + p_lo + rem / LPR) * d + h * DH) + (rem % LPR) * 128;
                asm volatile("prefetch.global.L2 [%0];" ::"l"(ptr));
            }
            const char* st = reinterpret_cast<const char*>(ckpt + ((int64_t)chain * n_ck + ck - 1) * DH * DH);
            for (int idx = tid; idx < DH * DH * 4 / 128; idx += BT) asm volatile("prefetch.global.L2 [%0];" ::"l"(st + idx * 128));
        }
        // ---- phase B: sub-chunks in reverse
        for (int j = nsub - 1; j >= 0; --j) {
            const int t0 = t_lo + j * C;
            const int n = t_hi - t0 < C ? t_hi - t0 : C;
            __syncthreads();
            load_state(j == 0 ? ck_state : my_sub + (int64_t)j * DH * DH);
            __syncthreads();
            chunk_front(t0, n, true);

            // dU = A^T dO + diag(eg) K dS
            cta_gemm<C, DH, C, L_KM, L_KN>(Am, LDC, dOs, LDV, [&](int i, int c, float acc) { dRs[i * LDV + c] = acc; });
            __syncthreads();
            cta_gemm<C, DH, DH, L_MK, L_KN>(Ks, LDK, dS, LDV,
                                            [&](int i, int c, float acc) { dRs[i * LDV + c] += eg_s[i] * acc; });
            __syncthreads();
            // dR = (I + L)^-T dU : back substitution, one thread per value column
            if (tid < DH) {
                float y[C];
#pragma unroll
                for (int t = C - 1; t >= 0; --t) {
                    float s = dRs[t * LDV + tid];
#pragma unroll
                    for (int jj = C - 1; jj > t; --jj) s = fmaf(-Lm[jj * LDC + t], y[jj], s);
                    y[t] = s;
                    dRs[t * LDV + tid] = s;
                }
            }
            __syncthreads();
            // dL = -strictlower(dR U^T), dA = lower(dO U^T); then M = dL beta Gam, dAG = dA Gam
            for (int idx = tid; idx < C * C; idx += BT) {
                const int t = idx / C, i = idx % C;
                float s1 = 0.0f, s2 = 0.0f;
                if (i <= t) {
                    const float* rt = dRs + t * LDV;
                    const float* ot = dOs + t * LDV;
                    const float* ui = Us + i * LDV;
#pragma unroll 4
                    for (int c = 0; c < DH; c += 4) {
                        const float4 u4 = *reinterpret_cast<const float4*>(ui + c);
                        const float4 r4 = *reinterpret_cast<const float4*>(rt + c);
                        const float4 o4 = *reinterpret_cast<const float4*>(ot + c);
                        s1 = fmaf(r4.x, u4.x, s1); s1 = fmaf(r4.y, u4.y, s1); s1 = fmaf(r4.z, u4.z, s1); s1 = fmaf(r4.w, u4.w, s1);
                        s2 = fmaf(o4.x, u4.x, s2); s2 = fmaf(o4.y, u4.y, s2); s2 = fmaf(o4.z, u4.z, s2); s2 = fmaf(o4.w, u4.w, s2);
                    }
                }
                const float gm = Gm[t * LDC + i];
                const float dl = i < t ? -s1 : 0.0f;
                dLm[t * LDC + i] = dl * gm;               // dL Gam  (times beta_t below -> M)
                dAm[t * LDC + i] = s2 * gm;               // dA Gam  (gm = 0 above the diagonal)
            }
            __syncthreads();
            // dbeta_t = dR_t.Z_t + sum_i (dL Gam)[t,i] KK[t,i]; then M = (dL Gam) beta_t.
            // per-row P sums: rowP[t] = sum_i dAG[t,i] QK[t,i] + M[t,i] KK[t,i]
            for (int t = warp; t < C; t += BT / 32) {
                float s = 0.0f;
                for (int c = lane; c < DH; c += 32) s = fmaf(dRs[t * LDV + c], Zs[t * LDV + c], s);
                float s2 = 0.0f;
                for (int i = lane; i < C; i += 32) s2 = fmaf(dLm[t * LDC + i], KK[t * LDC + i], s2);
                s = warp_sum(s);
                s2 = warp_sum(s2);
                if (lane == 0) dbe_s[t] = s + s2;
            }
            __syncthreads();
            for (int idx = tid; idx < C * C; idx += BT) {
                const int t = idx / C, i = idx % C;
                dLm[t * LDC + i] *= be_s[t];
            }
            // dV = beta dR (written out), dZ = dV kept in dRs
            for (int idx = tid; idx < C * DH; idx += BT) {
                const int t = idx / DH, c = idx % DH;
                const float dz = be_s[t] * dRs[t * LDV + c];
                dRs[t * LDV + c] = dz;
                if (t < n) d_qkv[(row0 + t0 + t) * 3 * d + 2 * d + h * DH + c] = dz;
            }
            __syncthreads();
            // bufA = dO S0^T (dQ inter, unscaled) ; bufB = -dZ S0^T (dKg)
            cta_gemm<C, DH, DH, L_MK, L_NK>(dOs, LDV, S0, LDV, [&](int t, int a, float acc) { bufA[t * LDK + a] = acc; });
            cta_gemm<C, DH, DH, L_MK, L_NK>(dRs, LDV, S0, LDV, [&](int t, int a, float acc) { bufB[t * LDK + a] = -acc; });
            __syncthreads();
            for (int t = warp; t < C; t += BT / 32) {
                float s1 = 0.0f, s2 = 0.0f;
                for (int a = lane; a < DH; a += 32) {
                    s1 = fmaf(Qs[t * LDK + a], bufA[t * LDK + a], s1);
                    s2 = fmaf(Ks[t * LDK + a], bufB[t * LDK + a], s2);
                }
                s1 = warp_sum(s1);
                s2 = warp_sum(s2);
                if (lane == 0) {
                    r_qs[t] = gam_s[t] * s1;
                    r_kg[t] = gam_s[t] * s2;
                }
            }
            __syncthreads();
            // dQ = gam bufA + dAG K  (in bufA)
            cta_gemm<C, DH, C, L_MK, L_KN>(dAm, LDC, Ks, LDK, [&](int t, int a, float acc) {
                bufA[t * LDK + a] = fmaf(gam_s[t], bufA[t * LDK + a], acc);
            });
            __syncthreads();
            // L2-norm backward of dq rows and store: (g - y (y.g)) / norm   (y = normalised q)
            for (int t = warp; t < n; t += BT / 32) {
                float s = 0.0f;
                for (int a = lane; a < DH; a += 32) s = fmaf(Qs[t * LDK + a], bufA[t * LDK + a], s);
                s = warp_sum(s);
                const float nq = qnorm[(row0 + t0 + t) * H + h];
                float* dst = d_qkv + (row0 + t0 + t) * 3 * d + h * DH;
                for (int a = lane; a < DH; a += 32) dst[a] = (bufA[t * LDK + a] - Qs[t * LDK + a] * s) / nq;
            }
            __syncthreads();
            // bufA = dW = U dS^T ; r_kw[t] = eg_t k_t.dW_t
            cta_gemm<C, DH, DH, L_MK, L_NK>(Us, LDV, dS, LDV, [&](int t, int a, float acc) { bufA[t * LDK + a] = acc; });
            __syncthreads();
            for (int t = warp; t < C; t += BT / 32) {
                float s = 0.0f;
                for (int a = lane; a < DH; a += 32) s = fmaf(Ks[t * LDK + a], bufA[t * LDK + a], s);
                s = warp_sum(s);
                if (lane == 0) r_kw[t] = eg_s[t] * s;
            }
            // dK = gam dKg + eg dW  (into bufB), then += dAG^T Q + (M + M^T) K
            for (int idx = tid; idx < C * DH; idx += BT) {
                const int t = idx / DH, a = idx % DH;
                bufB[t * LDK + a] = fmaf(gam_s[t], bufB[t * LDK + a], eg_s[t] * bufA[t * LDK + a]);
            }
            __syncthreads();
            cta_gemm<C, DH, C, L_KM, L_KN>(dAm, LDC, Qs, LDK, [&](int i, int a, float acc) { bufB[i * LDK + a] += acc; });
            __syncthreads();
            // P row/col sums before M is symmetrised: rowP, colP over P = dAG.QK + M.KK
            if (tid < C) {
                const int t = tid;
                float rs = 0.0f, cs = 0.0f;
                for (int i = 0; i < C; ++i) {
                    rs = fmaf(dAm[t * LDC + i], QK[t * LDC + i], rs);
                    rs = fmaf(dLm[t * LDC + i], KK[t * LDC + i], rs);
                    cs = fmaf(dAm[i * LDC + t], QK[i * LDC + t], cs);
                    cs = fmaf(dLm[i * LDC + t], KK[i * LDC + t], cs);
                }
                dg_s[t] = rs - cs + r_qs[t] + r_kg[t] - r_kw[t];
            }
            __syncthreads();
            // Msym = M + M^T into Am (A is no longer needed)
            for (int idx = tid; idx < C * C; idx += BT) {
                const int t = idx / C, i = idx % C;
                Am[t * LDC + i] = dLm[t * LDC + i] + dLm[i * LDC + t];
            }
            __syncthreads();
            cta_gemm<C, DH, C, L_MK, L_KN>(Am, LDC, Ks, LDK, [&](int i, int a, float acc) { bufB[i * LDK + a] += acc; });
            // <S0, dS> for dg_last (all threads), meanwhile nothing else writes S0/dS
            float part = 0.0f;
            for (int idx = tid; idx < DH * DH; idx += BT) {
                const int a = idx / DH, c = idx % DH;
                part = fmaf(S0[a * LDV + c], dS[a * LDV + c], part);
            }
            const float sds = block_sum(part, red);  // contains __syncthreads
            // gates: dg_last += sum_t r_kw[t] + gam_last <S0,dS>; reverse cumsum; sigmoid backward
            if (warp == 0) {
                float kw = lane < C ? r_kw[lane] : 0.0f;
                kw = warp_sum(kw);
                float gx = lane < C ? dg_s[lane] : 0.0f;
                if (lane == C - 1) gx += gam_s[C - 1] * sds + kw;
#pragma unroll
                for (int o = 1; o < 32; o <<= 1) {   // suffix sums: dlogalpha_t = sum_{j >= t} dg_j
                    const float y = __shfl_down_sync(0xffffffffu, gx, o);
                    if (lane + o < 32) gx += y;
                }
                if (lane < C) dg_s[lane] = gx;
            }
            __syncthreads();
            if (tid < n) {
                const int64_t r = row0 + t0 + tid;
                const float al = al_s[tid], be = be_s[tid];
                d_gate[r * 2 * H + h] = dg_s[tid] * (1.0f - al);            // (dlogalpha/alpha) alpha (1-alpha)
                d_gate[r * 2 * H + H + h] = dbe_s[tid] * be * (1.0f - be);
            }
            // L2-norm backward of dk rows and store
            for (int t = warp; t < n; t += BT / 32) {
                float s = 0.0f;
                for (int a = lane; a < DH; a += 32) s = fmaf(Ks[t * LDK + a], bufB[t * LDK + a], s);
                s = warp_sum(s);
                const float nk = knorm[(row0 + t0 + t) * H + h];
                float* dst = d_qkv + (row0 + t0 + t) * 3 * d + d + h * DH;
                for (int a = lane; a < DH; a += 32) dst[a] = (bufB[t * LDK + a] - Ks[t * LDK + a] * s) / nk;
            }
            __syncthreads();
            // dS <- gam_last dS + (gam Q)^T dO - (gam K)^T dZ
            for (int idx = tid; idx < C * DH; idx += BT) {
                const int t = idx / DH, a = idx % DH;
                bufA[t * LDK + a] = gam_s[t] * Qs[t * LDK + a];
                bufB[t * LDK + a] = -gam_s[t] * Ks[t * LDK + a];
            }
            __syncthreads();
            const float gl = gam_s[C - 1];
            cta_gemm<DH, DH, C, L_KM, L_KN>(bufA, LDK, dOs, LDV, [&](int a, int c, float acc) {
                dS[a * LDV + c] = fmaf(gl, dS[a * LDV + c], acc);
            });
            __syncthreads();
            cta_gemm<DH, DH, C, L_KM, L_KN>(bufB, LDK, dRs, LDV, [&](int a, int c, float acc) { dS[a * LDV + c] += acc; });
            __syncthreads();
        }
    }
}

// ------------------------------------------------------------------ checkpoints every 64 tokens: three kernels
// With one sub-chunk per checkpoint interval (C = chunk = 64) only dS itself runs from chunk to chunk, and by VALUE column
// that recurrence splits without communication. So:
//   pre    one CTA per (chain, chunk), all chunks at once:  A, LG = strictlower(Gam K K^T), T = (I + L)^-1 (16-wide diagonal
//          blocks by substitution, then doubled twice by block products), D = beta T^T A^T dO, Hm = beta T^T diag(eg) K,
//          Y = (gam Q)^T dO
//   chain  one CTA per (chain, block of value columns), chunks in reverse:  dZ = D + Hm dS;  dS' = gam_last dS + Y - (gam K)^T dZ
//   grad   one CTA per (chain, chunk), all chunks at once: everything else, from S0 (the checkpoint), dS and dZ
// Two products a chunk are left on the serial path where the single kernel above has thirteen and the recomputation of inner
// states; a launch of few chains (the small models, host calls) fills the GPU with its chunks. Work per token and head is about
// 13 dh^2 multiply-adds against 21. Every dL and dA appears times beta or L, so nothing is divided by beta:
//   beta dL = -strictlower(dZ U^T),  beta dbeta_t = dZ_t.Z_t - sum_i (dZ U^T)[t,i] LG[t,i]
// A launch takes a group of chains and a segment of their chunks (`Range`), last segment first, so that the scratch between the
// kernels stays bounded; the chain kernel hands dS from segment to segment through `carry`.
// Bound: shared-memory return bandwidth of the 8 x 4 thread tiles (0.375 loads per FFMA), one CTA per SM at dh 128.
constexpr int CC = 64;   // tokens per chunk
constexpr int LX = CC + 4;

// dst[t][c] = src[(row0 + t) ld + col0 + c] for t < n, zero for n <= t < ROWS: asynchronous copies (f32), or every load of the
// tile in flight before the first store (bf16). tile_wait() makes all tiles asked for so far visible to the CTA.
template <typename T, int ROWS, int W>
__device__ __forceinline__ void load_tile(const T* __restrict__ src, int64_t row0, int64_t ld, int col0, int n, float* __restrict__ dst, int ldd) {
    constexpr int Q = W / 4, IT = (ROWS * Q + BT - 1) / BT;
    src += row0 * ld + col0;
    if (sizeof(T) == 4) {
#pragma unroll
        for (int i = 0; i < IT; ++i) {
            const int idx = threadIdx.x + i * BT, t = idx / Q, c = idx % Q * 4;
            if (ROWS * Q % BT == 0 || idx < ROWS * Q)
                asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"((uint32_t)__cvta_generic_to_shared(dst + t * ldd + c)),
                             "l"(src + (t < n ? t : 0) * ld + c), "r"(t < n ? 16 : 0) : "memory");
        }
    } else {
        uint2 v[IT];
#pragma unroll
        for (int i = 0; i < IT; ++i) {
            const int idx = threadIdx.x + i * BT, t = idx / Q, c = idx % Q * 4;
            v[i] = t < n && idx < ROWS * Q ? *reinterpret_cast<const uint2*>(src + t * ld + c) : make_uint2(0, 0);
        }
#pragma unroll
        for (int i = 0; i < IT; ++i) {
            const int idx = threadIdx.x + i * BT, t = idx / Q, c = idx % Q * 4;
            const __nv_bfloat162 a = *reinterpret_cast<__nv_bfloat162*>(&v[i].x), b = *reinterpret_cast<__nv_bfloat162*>(&v[i].y);
            if (idx < ROWS * Q)
                *reinterpret_cast<float4*>(dst + t * ldd + c) = make_float4(__low2float(a), __high2float(a), __low2float(b), __high2float(b));
        }
    }
}
__device__ __forceinline__ void tile_wait() {
    asm volatile("cp.async.wait_all;" ::: "memory");
    __syncthreads();
}
// asks for `rows` runs of `bytes` (a multiple of 128 when above it), `pitch` bytes apart, in L2
__device__ __forceinline__ void prefetch_l2(const void* p, int rows, int bytes, int64_t pitch) {
    const int lines = (bytes + 127) / 128;
    for (int i = threadIdx.x; i < rows * lines; i += BT)
        asm volatile("prefetch.global.L2 [%0];" ::"l"(reinterpret_cast<const char*>(p) + i / lines * pitch + i % lines * 128));
}

// acc += A B for an M x N output in BT threads' registers, K deep, operands in shared memory (row pitches multiples of 4).
// Thread (tm, tn) owns columns tn + THR_N j and rows in groups of four (tm + THR_M i where it has fewer than four).
// 8 x 4 tiles run at two thirds of the FFMA rate (64 x 128 x 128 on one CTA per SM: 12.2 thousand cycles of 8.2); 8 x 8 tiles over lanes that
// share k, which read a third less shared memory, were no faster (13 - 15), nor were operands read a step ahead or packed pairs of k.
template <int M, int N>
struct MM {
    static constexpr int TN = 4, THR_N = N / TN, THR_M = BT / THR_N < M ? BT / THR_N : M, TM = M / THR_M;
    static constexpr bool R4 = TM % 4 == 0;
    static_assert(N % 4 == 0 && BT % THR_N == 0 && M % THR_M == 0, "tile shape");
    float acc[TM][TN];
    int tn, tm;
    bool on, first;   // first: the one lane of a row that speaks for it
    __device__ __forceinline__ MM() {
        tn = threadIdx.x % THR_N;
        tm = threadIdx.x / THR_N;
        on = tm < THR_M;
        first = tn == 0;
        clear();
    }
    __device__ __forceinline__ void clear() {
#pragma unroll
        for (int i = 0; i < TM; ++i)
#pragma unroll
            for (int j = 0; j < TN; ++j) acc[i][j] = 0.0f;
    }
    __device__ __forceinline__ int row(int i) const { return R4 ? (i >> 2) * (4 * THR_M) + tm * 4 + (i & 3) : tm + THR_M * i; }
    __device__ __forceinline__ int col(int j) const { return tn + THR_N * j; }
    template <int K, int ALAY, int BLAY>
    __device__ __forceinline__ void mul(const float* __restrict__ A, int lda, const float* __restrict__ B, int ldb) {
        if (!on) return;
#pragma unroll (TM > 8 ? 1 : TM > 4 ? 2 : TM > 2 ? 4 : 8)
        for (int k = 0; k < K; k += 4) {
            float b[4][TN];   // [k][column]
            if (BLAY == L_NK) {
#pragma unroll
                for (int j = 0; j < TN; ++j) {
                    const float4 v = *reinterpret_cast<const float4*>(B + col(j) * ldb + k);
                    b[0][j] = v.x; b[1][j] = v.y; b[2][j] = v.z; b[3][j] = v.w;
                }
            } else {
#pragma unroll
                for (int kk = 0; kk < 4; ++kk)
#pragma unroll
                    for (int j = 0; j < TN; ++j) b[kk][j] = B[(k + kk) * ldb + col(j)];
            }
            if (ALAY == L_MK) {
#pragma unroll
                for (int i = 0; i < TM; ++i) {
                    const float4 a = *reinterpret_cast<const float4*>(A + row(i) * lda + k);
#pragma unroll
                    for (int j = 0; j < TN; ++j) {
                        acc[i][j] = fmaf(a.x, b[0][j], acc[i][j]);
                        acc[i][j] = fmaf(a.y, b[1][j], acc[i][j]);
                        acc[i][j] = fmaf(a.z, b[2][j], acc[i][j]);
                        acc[i][j] = fmaf(a.w, b[3][j], acc[i][j]);
                    }
                }
            } else {
#pragma unroll
                for (int kk = 0; kk < 4; ++kk) {
                    float a[TM];
                    if (R4) {
#pragma unroll
                        for (int i = 0; i < TM; i += 4) {
                            const float4 v = *reinterpret_cast<const float4*>(A + (k + kk) * lda + row(i));
                            a[i] = v.x; a[(i + 1) % TM] = v.y; a[(i + 2) % TM] = v.z; a[(i + 3) % TM] = v.w;
                        }
                    } else {
#pragma unroll
                        for (int i = 0; i < TM; ++i) a[i] = A[(k + kk) * lda + row(i)];
                    }
#pragma unroll
                    for (int i = 0; i < TM; ++i)
#pragma unroll
                        for (int j = 0; j < TN; ++j) acc[i][j] = fmaf(a[i], b[kk][j], acc[i][j]);
                }
            }
        }
    }
    // f(row, column, value) of every element of this thread
    template <class F>
    __device__ __forceinline__ void each(F f) {
        if (!on) return;
#pragma unroll
        for (int i = 0; i < TM; ++i)
#pragma unroll
            for (int j = 0; j < TN; ++j) f(row(i), col(j), acc[i][j]);
    }
    template <class F>
    __device__ __forceinline__ void each_index(F f) {   // f(row, column, index of the row, of the column)
        if (!on) return;
#pragma unroll
        for (int i = 0; i < TM; ++i)
#pragma unroll
            for (int j = 0; j < TN; ++j) f(row(i), col(j), i, j);
    }
    // the sum over a row's columns of f(row, column, value, index of the column), in every lane that shares the row (THR_N neighbouring lanes)
    template <class F>
    __device__ __forceinline__ float row_sum(int i, F f) {
        float s = 0.0f;
#pragma unroll
        for (int j = 0; j < TN; ++j) s += f(row(i), col(j), acc[i][j], j);
        return lanes_sum(s);
    }
    __device__ __forceinline__ float lanes_sum(float s) const {
#pragma unroll
        for (int m = THR_N / 2; m > 0; m >>= 1) s += __shfl_xor_sync(0xffffffffu, s, m);
        return s;
    }
};

// Gates of a chunk of n live steps (alpha 1, beta 0 behind them): cumulative log alpha g, gam = exp(g), eg = exp(g_last - g).
struct ChunkGates {
    float g[CC], gam[CC], eg[CC], be[CC], al[CC];
};
__device__ __forceinline__ void load_gates(const float* alpha, const float* beta, int64_t row0, int n, int H, int h, ChunkGates& s) {
    const int t = threadIdx.x;
    if (t < CC) {
        s.al[t] = t < n ? alpha[(row0 + t) * H + h] : 1.0f;
        s.be[t] = t < n ? beta[(row0 + t) * H + h] : 0.0f;
    }
    __syncthreads();
    if (t < 32) {   // two steps a lane, left to right
        const float a = logf(s.al[2 * t]), b = logf(s.al[2 * t + 1]);
        float x = a + b;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const float y = __shfl_up_sync(0xffffffffu, x, o);
            if (t >= o) x += y;
        }
        const float before = __shfl_up_sync(0xffffffffu, x, 1);
        s.g[2 * t] = (t ? before : 0.0f) + a;
        s.g[2 * t + 1] = x;
    }
    __syncthreads();
    if (t < CC) {
        s.gam[t] = expf(s.g[t]);
        s.eg[t] = expf(s.g[CC - 1] - s.g[t]);
    }
    __syncthreads();
}

// Per (chain, chunk) scratch, in floats: A, LG, T (CC x CC each), D -> dZ and Hm (CC x DH), Y -> dS at the chunk's end (DH x DH),
// gam (CC)
template <int DH>
struct ChunkScratch {
    static constexpr int64_t A = 0, LG = CC * CC, T = 2 * CC * CC, D = 3 * CC * CC, HM = D + CC * DH, Y = HM + CC * DH, GAM = Y + DH * DH, SIZE = GAM + CC;
};

// The chains [chain0, chain0 + gridDim.y) and chunks [ck0, ck0 + n) of a launch; scratch tiles are numbered inside it.
struct Range {
    int chain0, ck0, n;
    __device__ __forceinline__ int64_t tile(int chain, int ck) const { return (int64_t)(chain - chain0) * n + (ck - ck0); }
};

template <int DH, typename T>
struct PreSmem {
    static constexpr int LD = DH + 4;
    static constexpr size_t bytes = (size_t)(4 * CC * LD + 3 * CC * LX) * 4 + sizeof(ChunkGates);
};

template <int DH, typename T>
__global__ void __launch_bounds__(BT, DH == 128 ? 1 : DH == 64 ? 2 : 3) delta_bwd_pre_kernel(const T* __restrict__ q, const T* __restrict__ k, const float* __restrict__ alpha,
                                                           const float* __restrict__ beta, const T* __restrict__ d_o,
                                                           float* __restrict__ scratch, int Tlen, int H, const Range range) {
    using SC = ChunkScratch<DH>;
    constexpr int LD = DH + 4;
    extern __shared__ __align__(16) float smem[];
    float *Ks = smem, *Qs = Ks + CC * LD, *Os = Qs + CC * LD, *Xs = Os + CC * LD, *Ls = Xs + CC * LD, *Ts = Ls + CC * LX, *As = Ts + CC * LX;
    ChunkGates& gt = *reinterpret_cast<ChunkGates*>(As + CC * LX);
    const int tid = threadIdx.x, ck = range.ck0 + blockIdx.x, chain = range.chain0 + blockIdx.y, bi = chain / H, h = chain % H, d = H * DH;
    const int n = min(CC, Tlen - ck * CC);
    const int64_t row0 = (int64_t)bi * Tlen + ck * CC;
    float* out = scratch + range.tile(chain, ck) * SC::SIZE;
    load_tile<T, CC, DH>(k, row0, d, h * DH, n, Ks, LD);
    load_tile<T, CC, DH>(q, row0, d, h * DH, n, Qs, LD);
    load_tile<T, CC, DH>(d_o, row0, d, h * DH, n, Os, LD);
    load_gates(alpha, beta, row0, n, H, h, gt);
    if (tid < CC) out[SC::GAM + tid] = gt.gam[tid];
    tile_wait();
    {
        MM<CC, CC> kk, qk;
        kk.template mul<DH, L_MK, L_NK>(Ks, LD, Ks, LD);
        kk.each([&](int t, int i, float v) {
            const float lg = i < t ? expf(gt.g[t] - gt.g[i]) * v : 0.0f;
            out[SC::LG + t * CC + i] = lg;
            Ls[t * LX + i] = gt.be[t] * lg;
            Ts[t * LX + i] = t == i ? 1.0f : 0.0f;
        });
        qk.template mul<DH, L_MK, L_NK>(Qs, LD, Ks, LD);
        qk.each([&](int t, int i, float v) {
            const float a = i <= t ? expf(gt.g[t] - gt.g[i]) * v : 0.0f;
            out[SC::A + t * CC + i] = a;
            As[t * LX + i] = a;
        });
    }
    __syncthreads();
    // T: the four 16 x 16 diagonal blocks, a thread per column
    if (tid < CC) {
        const int b0 = tid & ~15, c = tid & 15;
        float x[16];
#pragma unroll
        for (int t = 0; t < 16; ++t) {
            float v[4] = {t == c ? 1.0f : 0.0f, 0.0f, 0.0f, 0.0f};   // (four partial sums: the chain is the rows', not the terms')
#pragma unroll
            for (int i = 0; i < t; i += 4) {
                const float4 l = *reinterpret_cast<const float4*>(Ls + (b0 + t) * LX + b0 + i);   // zeros from the diagonal on
                v[0] = fmaf(-l.x, x[i], v[0]);
                if (i + 1 < t) v[1] = fmaf(-l.y, x[i + 1], v[1]);
                if (i + 2 < t) v[2] = fmaf(-l.z, x[i + 2], v[2]);
                if (i + 3 < t) v[3] = fmaf(-l.w, x[i + 3], v[3]);
            }
            x[t] = (v[0] + v[1]) + (v[2] + v[3]);
            Ts[(b0 + t) * LX + b0 + c] = x[t];
        }
    }
    __syncthreads();
    // ... doubled: T21 = -T2 (L21 T1), the inner product in the not yet needed X area; a thread takes four columns of a row
#pragma unroll
    for (int w = 16; w < CC; w *= 2) {
        const int at = tid * 4, b = at / (w * w) * 2 * w, t = at / w % w, c = at % w;
        const bool on = at < CC / 2 * w;   // (CC / 2w blocks of w x w)
        auto product = [&](const float* A, const float* B, int ldb) {   // row of A times w rows of B
            float4 v = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
#pragma unroll 8
            for (int i = 0; i < w; ++i) {
                const float a = A[i];
                const float4 x = *reinterpret_cast<const float4*>(B + i * ldb);
                v.x = fmaf(a, x.x, v.x); v.y = fmaf(a, x.y, v.y); v.z = fmaf(a, x.z, v.z); v.w = fmaf(a, x.w, v.w);
            }
            return v;
        };
        if (on) *reinterpret_cast<float4*>(Xs + at) = product(Ls + (b + w + t) * LX + b, Ts + b * LX + b + c, LX);
        __syncthreads();
        if (on) {
            const float4 v = product(Ts + (b + w + t) * LX + b + w, Xs + at - t * w, w);
            *reinterpret_cast<float4*>(Ts + (b + w + t) * LX + b + c) = make_float4(-v.x, -v.y, -v.z, -v.w);
        }
        __syncthreads();
    }
    for (int idx = tid; idx < CC * CC / 4; idx += BT)
        *reinterpret_cast<float4*>(out + SC::T + idx * 4) = *reinterpret_cast<const float4*>(Ts + idx / (CC / 4) * LX + idx % (CC / 4) * 4);
    MM<CC, DH> m;
    m.template mul<CC, L_KM, L_KN>(As, LX, Os, LD);   // A^T dO
    m.each([&](int t, int c, float v) { Xs[t * LD + c] = v; });
    __syncthreads();
    m.clear();
    m.template mul<CC, L_KM, L_KN>(Ts, LX, Xs, LD);   // D
    m.each([&](int t, int c, float v) { out[SC::D + t * DH + c] = gt.be[t] * v; });
    __syncthreads();
    for (int idx = tid; idx < CC * DH; idx += BT) {
        const int t = idx / DH, c = idx % DH;
        Xs[t * LD + c] = gt.eg[t] * Ks[t * LD + c];
        Qs[t * LD + c] *= gt.gam[t];
    }
    __syncthreads();
    m.clear();
    m.template mul<CC, L_KM, L_KN>(Ts, LX, Xs, LD);   // Hm
    m.each([&](int t, int c, float v) { out[SC::HM + t * DH + c] = gt.be[t] * v; });
    MM<DH, DH> y;
    y.template mul<CC, L_KM, L_KN>(Qs, LD, Os, LD);
    y.each([&](int a, int c, float v) { out[SC::Y + a * DH + c] = v; });
}

// Where the tiles are small the next chunk's are copied while this one is worked on (two buffers, D and Y in registers);
// elsewhere they are only asked for in L2.
template <int DH, int W>
struct ChainSmem {
    static constexpr bool AHEAD = DH * W <= 64 * 64;
    static constexpr int LD = DH + 4, LW = W + 4, STAGE = 2 * CC * LD + CC;   // Hm, K, gam
    static constexpr size_t bytes = (size_t)((AHEAD ? 2 : 1) * STAGE + DH * LW + CC * LW) * 4;
};

template <int DH, int W, typename T>
__global__ void __launch_bounds__(BT, DH >= 64 ? 1 : 2) delta_bwd_chain_kernel(const T* __restrict__ k, float* __restrict__ scratch, float* __restrict__ carry,
                                                             int Tlen, int H, const Range range, int last) {
    using SC = ChunkScratch<DH>;
    using SM = ChainSmem<DH, W>;
    constexpr int LD = SM::LD, LW = SM::LW;
    constexpr bool AHEAD = SM::AHEAD;
    extern __shared__ __align__(16) float smem[];
    float *dS = smem + (AHEAD ? 2 : 1) * SM::STAGE, *dZ = dS + DH * LW;
    const int tid = threadIdx.x, c0 = blockIdx.x * W, chain = range.chain0 + blockIdx.y, bi = chain / H, h = chain % H, d = H * DH;
    const int ck_end = range.ck0 + range.n;
    carry += (int64_t)blockIdx.y * DH * DH + c0;   // dS between segments: `last` starts from zero, the first leaves none behind
    for (int i = tid; i < DH * W; i += BT) dS[i / W * LW + i % W] = last ? 0.0f : carry[i / W * DH + i % W];
    MM<DH, W> s_in;   // Y and D of the chunk to come
    MM<CC, W> z_in;
    auto request = [&](int ck, float* st) {
        float* at = scratch + range.tile(chain, ck) * SC::SIZE;
        load_tile<float, CC, DH>(at + SC::HM, 0, DH, 0, CC, st, LD);
        load_tile<T, CC, DH>(k, (int64_t)bi * Tlen + ck * CC, d, h * DH, min(CC, Tlen - ck * CC), st + CC * LD, LD);
        if (tid < CC / 4)
            asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((uint32_t)__cvta_generic_to_shared(st + 2 * CC * LD + tid * 4)),
                         "l"(at + SC::GAM + tid * 4) : "memory");
        s_in.each([&](int a, int c, float& v) { v = at[SC::Y + a * DH + c0 + c]; });
        z_in.each([&](int t, int c, float& v) { v = at[SC::D + t * DH + c0 + c]; });
    };
    if (AHEAD) request(ck_end - 1, smem + ((ck_end - 1) & 1) * SM::STAGE);
    for (int ck = ck_end - 1; ck >= range.ck0; --ck) {
        float* at = scratch + range.tile(chain, ck) * SC::SIZE;
        float* Hs = smem + (AHEAD ? (ck & 1) * SM::STAGE : 0);
        const float *Ks = Hs + CC * LD, *gam = Hs + 2 * CC * LD;
        if (!AHEAD) request(ck, Hs);
        if (!AHEAD && ck > range.ck0) {
            prefetch_l2(at - SC::SIZE + SC::HM, 1, CC * DH * 4, 0);
            prefetch_l2(at - SC::SIZE + SC::D + c0, CC, W * 4, DH * 4);
            prefetch_l2(at - SC::SIZE + SC::Y + c0, DH, W * 4, DH * 4);
            prefetch_l2(k + ((int64_t)bi * Tlen + (ck - 1) * CC) * d + h * DH, CC, DH * (int)sizeof(T), (int64_t)d * sizeof(T));
        }
        tile_wait();
        MM<DH, W> s = s_in;
        MM<CC, W> z = z_in;
        if (AHEAD && ck > range.ck0) request(ck - 1, smem + ((ck - 1) & 1) * SM::STAGE);
        s.each([&](int a, int c, float) { at[SC::Y + a * DH + c0 + c] = dS[a * LW + c]; });   // dS at the end of this chunk
        z.template mul<DH, L_MK, L_KN>(Hs, LD, dS, LW);
        z.each([&](int t, int c, float v) {
            at[SC::D + t * DH + c0 + c] = v;
            dZ[t * LW + c] = -gam[t] * v;
        });
        if (ck == 0) break;   // (dS before the first token is nobody's)
        __syncthreads();
        const float gl = gam[CC - 1];
        s.each([&](int a, int c, float& v) { v = fmaf(gl, dS[a * LW + c], v); });
        s.template mul<CC, L_KM, L_KN>(Ks, LD, dZ, LW);
        __syncthreads();
        if (ck == range.ck0) {
            s.each([&](int a, int c, float v) { carry[a * DH + c] = v; });
            break;
        }
        s.each([&](int a, int c, float v) { dS[a * LW + c] = v; });
        if (!AHEAD) __syncthreads();   // (with two buffers the next tile_wait is the barrier)
    }
}

// x / n for a row's common n: one Newton step on the quotient by its reciprocal, within a rounding of a division; the plain quotient where the
// step is not finite (n zero or infinite, or an overflow). Below 2^-128 n has no finite reciprocal, so both sides of a small n are scaled by
// a power of two first (an x that overflows by it has an infinite quotient).
struct RowDiv {
    float scale, n, inv;
    __device__ __forceinline__ explicit RowDiv(float norm) {
        scale = fabsf(norm) < 0x1p-100f ? 0x1p100f : 1.0f;
        n = norm * scale;
        inv = 1.0f / n;
    }
    __device__ __forceinline__ float operator()(float x) const {
        x *= scale;
        const float q = x * inv, e = fmaf(-n, q, x);
        return fabsf(e) < INFINITY ? fmaf(e, inv, q) : q;
    }
};

template <int DH>
struct GradSmem {
    static constexpr int LD = DH + 4;
    static constexpr size_t bytes = (size_t)(4 * CC * LD + DH * LD + CC * LX + 8 * CC + 8 * CC + 64) * 4 + sizeof(ChunkGates);
};

// 7.35 M multiply-adds per chunk at head dim 128, where one CTA fills an SM and may use every register. Of its 127 thousand cycles 93 are
// products at two thirds of the FFMA rate; what it reads beside them (A, LG, dS, norms) is asked for ahead of a product, since eight warps
// wait for each such load (171 thousand cycles, 4.78 -> 3.69 ms for 8192 chunks; launched together with L2 requests for the CTA
// that follows on the SM: 4.6).
template <int DH, typename T>
__global__ void __launch_bounds__(BT, DH == 128 ? 1 : DH == 64 ? 2 : 3) delta_bwd_grad_kernel(
    const T* __restrict__ q, const T* __restrict__ k, const T* __restrict__ v, const float* __restrict__ alpha,
    const float* __restrict__ beta, const float* __restrict__ qnorm, const float* __restrict__ knorm, const T* __restrict__ d_o,
    const float* __restrict__ ckpt, const float* __restrict__ scratch, int Tlen, int H, int n_ck, const Range range,
    float* __restrict__ d_qkv, float* __restrict__ d_gate) {
    using SC = ChunkScratch<DH>;
    constexpr int LD = DH + 4;
    extern __shared__ __align__(16) float smem[];
    float *Ks = smem, *Bs = Ks + CC * LD /* V, Z, then dO, then Q */, *Us = Bs + CC * LD, *Zs = Us + CC * LD /* dZ */, *Ss = Zs + CC * LD /* S0, then dS */,
          *Xs = Ss + DH * LD /* T, then dA Gam, then M + M^T */, *col_part = Xs + CC * LX, *vec = col_part + 8 * CC, *red = vec + 8 * CC;
    float *row_p = vec, *col_p = vec + CC, *r_qs = vec + 2 * CC, *r_kg = vec + 3 * CC, *r_kw = vec + 4 * CC, *dbe = vec + 5 * CC,
          *nq_s = vec + 6 * CC, *nk_s = vec + 7 * CC;
    ChunkGates& gt = *reinterpret_cast<ChunkGates*>(red + 64);
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, ck = range.ck0 + blockIdx.x, chain = range.chain0 + blockIdx.y, bi = chain / H,
              h = chain % H, d = H * DH;
    const int n = min(CC, Tlen - ck * CC);
    const int64_t row0 = (int64_t)bi * Tlen + ck * CC;
    const float* in = scratch + range.tile(chain, ck) * SC::SIZE;
    const float* S0 = ckpt + ((int64_t)chain * n_ck + ck) * DH * DH;
    load_tile<T, CC, DH>(k, row0, d, h * DH, n, Ks, LD);
    load_tile<float, DH, DH>(S0, 0, DH, 0, DH, Ss, LD);
    load_tile<T, CC, DH>(v, row0, d, h * DH, n, Bs, LD);
    load_tile<float, CC, DH>(in + SC::D, 0, DH, 0, CC, Zs, LD);
    load_tile<float, CC, CC>(in + SC::T, 0, CC, 0, CC, Xs, LX);
    if (tid < 2 * CC) {
        const int t = tid & (CC - 1);
        (tid < CC ? nq_s : nk_s)[t] = t < n ? (tid < CC ? qnorm : knorm)[(row0 + t) * H + h] : 1.0f;
    }
    load_gates(alpha, beta, row0, n, H, h, gt);
    tile_wait();
    // what comes into these buffers later is on its way to L2
    prefetch_l2(in + SC::A, 1, 2 * CC * CC * 4, 0);
    prefetch_l2(in + SC::Y, 1, DH * DH * 4, 0);
    prefetch_l2(d_o + row0 * d + h * DH, n, DH * (int)sizeof(T), (int64_t)d * sizeof(T));
    prefetch_l2(q + row0 * d + h * DH, n, DH * (int)sizeof(T), (int64_t)d * sizeof(T));
    using MD = MM<CC, DH>;
    using MX = MM<CC, CC>;
    {   // Z = V - gam K S0 (beta Z is what U wants), dZ.Z; dV = dZ goes out
        MD m;
        m.template mul<DH, L_MK, L_KN>(Ks, LD, Ss, LD);
#pragma unroll
        for (int i = 0; i < MD::TM; ++i) {
            const int t = m.row(i);
            const float s = m.row_sum(i, [&](int tt, int c, float& x, int j) {
                const float z = Bs[tt * LD + c] - gt.gam[tt] * x, dz = Zs[tt * LD + c];
                Bs[tt * LD + c] = gt.be[tt] * z;
                if (tt < n) d_qkv[(row0 + tt) * 3 * d + 2 * d + h * DH + c] = dz;
                return z * dz;
            });
            if (m.first) dbe[t] = s;
        }
    }
    __syncthreads();
    {   // U = T beta Z
        MD m;
        m.template mul<CC, L_MK, L_KN>(Xs, LX, Bs, LD);
        m.each([&](int t, int c, float x) { Us[t * LD + c] = x; });
    }
    __syncthreads();
    load_tile<T, CC, DH>(d_o, row0, d, h * DH, n, Bs, LD);
    tile_wait();
    // a C x C matrix of products P = e(acc) o other: row sums and column sums in a fixed order
    auto sums = [&](auto& m, auto f, bool first) {
        float cp[MX::TN] = {};
#pragma unroll
        for (int i = 0; i < MX::TM; ++i) {
            float p[MX::TN], s = 0.0f;
#pragma unroll
            for (int j = 0; j < MX::TN; ++j) {
                p[j] = f(m.row(i), m.col(j), m.acc[i][j], i, j);
                cp[j] += p[j];
                s += p[j];
            }
            s = m.lanes_sum(s);
            if (m.first) {
                if (first) row_p[m.row(i)] = s;
                else {
                    row_p[m.row(i)] += s;
                    dbe[m.row(i)] += s;   // (the second matrix is beta dL o L: it belongs to dbeta as well)
                }
            }
        }
#pragma unroll
        for (int j = 0; j < MX::TN; ++j) {
            cp[j] += __shfl_xor_sync(0xffffffffu, cp[j], 16);   // the warp's two row groups
            if (lane < 16) col_part[warp * CC + m.col(j)] = cp[j];
        }
        __syncthreads();
        if (tid < CC) {
            float s = 0.0f;
#pragma unroll
            for (int w = 0; w < 8; ++w) s += col_part[w * CC + tid];
            col_p[tid] = first ? s : col_p[tid] + s;
        }
    };
    {   // dA Gam
        MX m;
        float a[MX::TM][MX::TN];   // A, asked for ahead of the product
        m.each_index([&](int t, int i, int ti, int tj) { a[ti][tj] = in[SC::A + t * CC + i]; });
        m.template mul<DH, L_MK, L_NK>(Bs, LD, Us, LD);
        sums(m, [&](int t, int i, float x, int ti, int tj) {
            Xs[t * LX + i] = i <= t ? expf(gt.g[t] - gt.g[i]) * x : 0.0f;
            return i <= t ? x * a[ti][tj] : 0.0f;
        }, true);
    }
    {   // dQ = gam dO S0^T + (dA Gam) K, L2-norm backward, out
        MD m;
        m.template mul<DH, L_MK, L_NK>(Bs, LD, Ss, LD);
        float qv[MD::TM][MD::TN];
#pragma unroll
        for (int i = 0; i < MD::TM; ++i) {
            const int t = m.row(i);
            const float s = m.row_sum(i, [&](int tt, int c, float& x, int j) {
                x *= gt.gam[tt];
                return x * (qv[i][j] = tt < n ? to_f32<T>(q[(row0 + tt) * d + h * DH + c]) : 0.0f);
            });
            if (m.first) r_qs[t] = s;
        }
        __syncthreads();   // dA Gam is in place
        m.template mul<CC, L_MK, L_KN>(Xs, LX, Ks, LD);
#pragma unroll
        for (int i = 0; i < MD::TM; ++i) {
            const int t = m.row(i);
            const float s = m.row_sum(i, [&](int, int, float x, int j) { return x * qv[i][j]; });
            if (t < n) {
                const RowDiv by(nq_s[t]);
#pragma unroll
                for (int j = 0; j < MD::TN; ++j) d_qkv[(row0 + t) * 3 * d + h * DH + m.col(j)] = by(m.acc[i][j] - qv[i][j] * s);
            }
        }
    }
    constexpr int IT = (DH * DH / 4 + BT - 1) / BT, BATCH = IT < 8 ? IT : 8;
    float4 ds[BATCH];   // dS; the first batch is asked for ahead of the product
    auto ask = [&](int i0) {
#pragma unroll
        for (int i = 0; i < BATCH; ++i) {
            const int idx = tid + (i0 + i) * BT;
            ds[i] = idx < DH * DH / 4 ? *reinterpret_cast<const float4*>(in + SC::Y + idx * 4) : make_float4(0, 0, 0, 0);
        }
    };
    ask(0);
    MD dk;   // dK = -gam dZ S0^T + eg U dS^T + (dA Gam)^T Q + (M + M^T) K
    dk.template mul<DH, L_MK, L_NK>(Zs, LD, Ss, LD);
#pragma unroll
    for (int i = 0; i < MD::TM; ++i) {
        const int t = dk.row(i);
        const float s = dk.row_sum(i, [&](int tt, int c, float& x, int j) {
            x *= -gt.gam[tt];
            return x * Ks[tt * LD + c];
        });
        if (dk.first) r_kg[t] = s;
    }
    __syncthreads();   // S0 and dO are done with
    load_tile<T, CC, DH>(q, row0, d, h * DH, n, Bs, LD);
    float part = 0.0f;   // <S0, dS>
#pragma unroll
    for (int i0 = 0; i0 < IT; i0 += BATCH) {
        if (i0) ask(i0);
#pragma unroll
        for (int i = 0; i < BATCH; ++i) {
            const int idx = tid + (i0 + i) * BT;
            if (idx >= DH * DH / 4) continue;
            float4* at = reinterpret_cast<float4*>(Ss + idx / (DH / 4) * LD + idx % (DH / 4) * 4);
            const float4 a = *at;
            part = fmaf(a.x, ds[i].x, part); part = fmaf(a.y, ds[i].y, part); part = fmaf(a.z, ds[i].z, part); part = fmaf(a.w, ds[i].w, part);
            *at = ds[i];
        }
    }
    asm volatile("cp.async.wait_all;" ::: "memory");
    const float sds = block_sum(part, red);   // (holds barriers: dS and Q are in place)
    {
        MD m;
        m.template mul<DH, L_MK, L_NK>(Us, LD, Ss, LD);
#pragma unroll
        for (int i = 0; i < MD::TM; ++i) {
            const int t = m.row(i);
            const float s = m.row_sum(i, [&](int tt, int c, float& x, int j) {
                x *= gt.eg[tt];
                return x * Ks[tt * LD + c];
            });
            if (m.first) r_kw[t] = s;
#pragma unroll
            for (int j = 0; j < MD::TN; ++j) dk.acc[i][j] += m.acc[i][j];
        }
    }
    dk.template mul<CC, L_KM, L_KN>(Xs, LX, Bs, LD);
    {
        MX m;   // dZ U^T
        float lg[MX::TM][MX::TN];
        m.each_index([&](int t, int i, int ti, int tj) { lg[ti][tj] = in[SC::LG + t * CC + i]; });
        m.template mul<DH, L_MK, L_NK>(Zs, LD, Us, LD);
        __syncthreads();   // every reader of dA Gam is done
        m.each([&](int t, int i, float x) {
            if (i <= t) Xs[t * LX + i] = i < t ? -expf(gt.g[t] - gt.g[i]) * x : 0.0f;   // M
        });
        sums(m, [&](int t, int i, float x, int ti, int tj) { return i < t ? -x * lg[ti][tj] : 0.0f; }, false);   // (holds a barrier)
    }
    for (int idx = tid; idx < CC * CC; idx += BT) {   // M + M^T: the upper triangle is the mirror of the lower
        const int t = idx / CC, i = idx % CC;
        if (i > t) Xs[t * LX + i] = Xs[i * LX + t];
    }
    __syncthreads();
    dk.template mul<CC, L_MK, L_KN>(Xs, LX, Ks, LD);
#pragma unroll
    for (int i = 0; i < MD::TM; ++i) {
        const int t = dk.row(i);
        const float s = dk.row_sum(i, [&](int tt, int c, float x, int) { return x * Ks[tt * LD + c]; });
        if (t < n) {
            const RowDiv by(nk_s[t]);
#pragma unroll
            for (int j = 0; j < MD::TN; ++j) d_qkv[(row0 + t) * 3 * d + d + h * DH + dk.col(j)] = by(dk.acc[i][j] - Ks[t * LD + dk.col(j)] * s);
        }
    }
    // gates: dg, its suffix sums (two steps a lane), sigmoid backward
    if (warp == 0) {
        auto dg = [&](int t) { return row_p[t] - col_p[t] + r_qs[t] + r_kg[t] - r_kw[t]; };
        const float kw = warp_sum(r_kw[2 * lane] + r_kw[2 * lane + 1]);
        const float a = dg(2 * lane);
        float b = dg(2 * lane + 1);
        if (lane == 31) b += gt.gam[CC - 1] * sds + kw;
        float x = a + b;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const float y = __shfl_down_sync(0xffffffffu, x, o);
            if (lane + o < 32) x += y;
        }
        const float behind = __shfl_down_sync(0xffffffffu, x, 1);
        if (lane < 31) b += behind;
#pragma unroll
        for (int e = 0; e < 2; ++e) {
            const int t = 2 * lane + e;
            if (t < n) {
                d_gate[(row0 + t) * 2 * H + h] = (e ? b : x) * (1.0f - gt.al[t]);   // (dlogalpha / alpha) alpha (1 - alpha)
                d_gate[(row0 + t) * 2 * H + H + h] = dbe[t] * (1.0f - gt.be[t]);
            }
        }
    }
}

template <int DH, int C, typename T>
int launch_bwd(asca_ctx* ctx, const void* q, const void* k, const void* v, const float* alpha, const float* beta,
               const float* qnorm, const float* knorm, const void* d_o, const float* ckpt, int B, int Tlen, int H,
               int chunk, float* d_qkv, float* d_gate) {
    using SM = BwdSmem<DH, C>;
    static_assert(SM::bytes <= 227 * 1024, "shared memory budget");
    const int sub_per_ck = (chunk + C - 1) / C;
    void* ws;
    ASCA_TRY(asca_workspace(ctx, (size_t)B * H * sub_per_ck * DH * DH * 4 + 256, &ws));
    auto kern = delta_bwd_kernel<DH, C, T>;
    ASCA_CUDA(ctx, cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)SM::bytes));
    asca_span sp(ctx, "delta_bwd_kernel");
    kern<<<B * H, BT, SM::bytes, ctx->stream>>>((const T*)q, (const T*)k, (const T*)v, alpha, beta, qnorm, knorm,
                                                (const T*)d_o, ckpt, (float*)ws, B, Tlen, H, chunk, d_qkv, d_gate);
    ASCA_CHECK_LAUNCH(ctx);
    return ASCA_OK;
}

template <int DH, int W, typename T>
int launch_chain(asca_ctx* ctx, const void* k, float* ws, float* carry, int chains, int Tlen, int H, const Range& range, bool last) {
    auto kern = delta_bwd_chain_kernel<DH, W, T>;
    ASCA_CUDA(ctx, cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)ChainSmem<DH, W>::bytes));
    kern<<<dim3(DH / W, chains), BT, ChainSmem<DH, W>::bytes, ctx->stream>>>((const T*)k, ws, carry, Tlen, H, range, last ? 1 : 0);
    ASCA_CHECK_LAUNCH(ctx);
    return ASCA_OK;
}

// Scratch of a launch of the three kernels at most. 8,192 tiles at dh 128 (8 x 4096 tokens of 16 heads) are 1.48 GB and stay one launch;
// a launch this size is 60 waves of the chunk kernels, whose ends then cost nothing that shows. Where the device has no room
// for it, a fourth, and a sixteenth, and then the single kernel, which needs a few states per chain.
constexpr int64_t BWD64_SCRATCH = (int64_t)3 << 29;
constexpr int MIN_SEGMENT = 16;   // chunks a launch takes of a chain before it takes fewer chains (the chain kernel's start-up)

template <int DH, typename T>
int launch_bwd64(asca_ctx* ctx, const void* q, const void* k, const void* v, const float* alpha, const float* beta, const float* qnorm,
                 const float* knorm, const void* d_o, const float* ckpt, int B, int Tlen, int H, float* d_qkv, float* d_gate) {
    const int n_ck = (Tlen + CC - 1) / CC, n_chains = B * H;
    static_assert(PreSmem<DH, T>::bytes <= 227 * 1024 && GradSmem<DH>::bytes <= 227 * 1024, "shared memory budget");
    int chains = n_chains, seg = n_ck;   // of a launch
    void* p = nullptr;
    for (int64_t room = BWD64_SCRATCH;; room /= 4) {
        if (room < BWD64_SCRATCH / 16)
            return launch_bwd<DH, DH == 128 ? 16 : 32, T>(ctx, q, k, v, alpha, beta, qnorm, knorm, d_o, ckpt, B, Tlen, H, CC, d_qkv, d_gate);
        const int64_t tiles = room / (ChunkScratch<DH>::SIZE * 4);
        if ((int64_t)n_chains * n_ck > tiles) {   // even groups of chains, even segments
            const int64_t groups = ceil_div64(n_chains, std::max<int64_t>(1, tiles / std::min(MIN_SEGMENT, n_ck)));
            chains = (int)ceil_div64(n_chains, groups);
            const int64_t segs = ceil_div64(n_ck, std::max<int64_t>(1, tiles / chains));
            seg = (int)ceil_div64(n_ck, segs);
        }
        const int rc = asca_workspace(ctx, ((size_t)chains * seg * ChunkScratch<DH>::SIZE + (seg < n_ck ? (size_t)chains * DH * DH : 0)) * 4 + 256, &p);
        if (rc == ASCA_OK) break;
        if (rc != ASCA_ERR_OOM) return rc;
    }
    float *ws = (float*)p, *carry = ws + (int64_t)chains * seg * ChunkScratch<DH>::SIZE;
    auto pre = delta_bwd_pre_kernel<DH, T>;
    auto grad = delta_bwd_grad_kernel<DH, T>;
    ASCA_CUDA(ctx, cudaFuncSetAttribute(pre, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)PreSmem<DH, T>::bytes));
    ASCA_CUDA(ctx, cudaFuncSetAttribute(grad, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)GradSmem<DH>::bytes));
    const int n_sm = ctx->sm_count > 0 ? ctx->sm_count : 148;
    for (int chain0 = 0; chain0 < n_chains; chain0 += chains) {
        const int nc = std::min(chains, n_chains - chain0);
        for (int end = n_ck; end > 0;) {
            const int ck0 = std::max(0, end - seg), n = end - ck0;
            const Range range = {chain0, ck0, n};
            {
                asca_span sp(ctx, "delta_bwd_pre_kernel");
                pre<<<dim3(n, nc), BT, PreSmem<DH, T>::bytes, ctx->stream>>>((const T*)q, (const T*)k, alpha, beta, (const T*)d_o, ws, Tlen, H, range);
                ASCA_CHECK_LAUNCH(ctx);
            }
            {   // value columns per CTA: as many as leave every SM a CTA, since wider tiles read less shared memory per FFMA
                asca_span sp(ctx, "delta_bwd_chain_kernel");
                const bool last = end == n_ck;
                int w = DH;
                while (w > 16 && nc * (DH / w) * 2 <= n_sm) w /= 2;
                if (w == 128) ASCA_TRY((launch_chain<DH, DH < 128 ? DH : 128, T>(ctx, k, ws, carry, nc, Tlen, H, range, last)));
                else if (w == 64) ASCA_TRY((launch_chain<DH, DH < 64 ? DH : 64, T>(ctx, k, ws, carry, nc, Tlen, H, range, last)));
                else if (w == 32) ASCA_TRY((launch_chain<DH, DH < 32 ? DH : 32, T>(ctx, k, ws, carry, nc, Tlen, H, range, last)));
                else ASCA_TRY((launch_chain<DH, 16, T>(ctx, k, ws, carry, nc, Tlen, H, range, last)));
            }
            asca_span sp(ctx, "delta_bwd_grad_kernel");
            grad<<<dim3(n, nc), BT, GradSmem<DH>::bytes, ctx->stream>>>((const T*)q, (const T*)k, (const T*)v, alpha, beta, qnorm, knorm,
                                                                        (const T*)d_o, ckpt, ws, Tlen, H, n_ck, range, d_qkv, d_gate);
            ASCA_CHECK_LAUNCH(ctx);
            end = ck0;
        }
    }
    return ASCA_OK;
}

}  // namespace

extern "C" int asca_delta_bwd(asca_ctx* ctx, const void* q, const void* k, const void* v, const float* alpha,
                              const float* beta, const float* qnorm, const float* knorm, const void* d_o,
                              const float* ckpt, int64_t B, int64_t T, int64_t H, int64_t dh, int64_t chunk, int dtype,
                              float* d_qkv, float* d_gate) {
    if (!ctx) return ASCA_ERR_ARG;
    ASCA_REQUIRE(ctx, q && k && v && alpha && beta && qnorm && knorm && d_o && ckpt && d_qkv && d_gate,
                 "delta_bwd: null pointer");
    ASCA_REQUIRE(ctx, B >= 0 && T >= 0 && H > 0 && chunk >= 1 && B * T < (1ll << 31), "delta_bwd: bad shape");
    ASCA_REQUIRE(ctx, dtype == ASCA_F32 || dtype == ASCA_BF16, "delta_bwd: unknown dtype");
    if (dh != 16 && dh != 32 && dh != 64 && dh != 128)
        return asca_fail(ctx, ASCA_ERR_UNSUPPORTED, "delta_bwd: dh must be 16, 32, 64 or 128 (got %lld)", (long long)dh);
    const uintptr_t al = (uintptr_t)q | (uintptr_t)k | (uintptr_t)v | (uintptr_t)d_o | (uintptr_t)ckpt;
    ASCA_REQUIRE(ctx, (al & 15) == 0, "delta_bwd: q, k, v, d_o, ckpt must be 16-byte aligned");
    if (B == 0 || T == 0) return ASCA_OK;
    // bf16 mode, dh = 128, checkpoints every 64 tokens: reverse chunked scan on the tensor cores
    if (dtype == ASCA_BF16 && (dh == 128 || dh == 64) && chunk == 64 && asca_tc_enabled() && delta_tc::available())
        return delta_tc::backward(ctx, q, k, v, alpha, beta, qnorm, knorm, d_o, ckpt, B, T, H, dh, d_qkv, d_gate);
    if (chunk == CC && B * H < 65536) {
#define ASCA_BWD64(DH_)                                                                                                          \
    return dtype == ASCA_BF16 ? launch_bwd64<DH_, __nv_bfloat16>(ctx, q, k, v, alpha, beta, qnorm, knorm, d_o, ckpt, (int)B, (int)T, (int)H, \
                                                                 d_qkv, d_gate)                                                  \
                              : launch_bwd64<DH_, float>(ctx, q, k, v, alpha, beta, qnorm, knorm, d_o, ckpt, (int)B, (int)T, (int)H, d_qkv, d_gate)
        switch (dh) {
            case 16: ASCA_BWD64(16);
            case 32: ASCA_BWD64(32);
            case 64: ASCA_BWD64(64);
            default: ASCA_BWD64(128);
        }
#undef ASCA_BWD64
    }
#define ASCA_BWD(DH_, C_)                                                                                             \
    return dtype == ASCA_BF16                                                                                         \
               ? launch_bwd<DH_, C_, __nv_bfloat16>(ctx, q, k, v, alpha, beta, qnorm, knorm, d_o, ckpt, (int)B, (int)T, \
                                                    (int)H, (int)chunk, d_qkv, d_gate)                                \
               : launch_bwd<DH_, C_, float>(ctx, q, k, v, alpha, beta, qnorm, knorm, d_o, ckpt, (int)B, (int)T, (int)H, \
                                            (int)chunk, d_qkv, d_gate)
    switch (dh) {
        case 16: ASCA_BWD(16, 32);
        case 32: ASCA_BWD(32, 32);
        case 64: ASCA_BWD(64, 32);
        default: ASCA_BWD(128, 16);
    }
#undef ASCA_BWD
}
