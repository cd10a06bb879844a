// Gated delta rule, forward direction, f32-exact kernels:
//   * delta_fwd_rec_kernel -- the per-step recurrence of rust/src/delta.rs:281-315 with the
//     dh x dh state split by VALUE column. Column i of S evolves independently of the others
//     (u_i, S[.][i] and o_i only touch column i), so a chain (sequence, head) is cut into
//     groups of 4 or 8 lanes (and CTAs) that share nothing; the state lives in registers and the
//     whole sequence runs without a block barrier inside a 16-step stage. State is written to HBM
//     only at chunk boundaries (checkpoints for the backward) and once at the end -- never per step
//     as the reference kernel (rust/kernels/asca.cu:276-312) does.
//   * delta_step_kernel -- the O(1) decode step (rust/src/delta.rs:356-406): one CTA per
//     (stream, head) streams S through registers once (read + write = the HBM floor).
#include "common.cuh"

#include <type_traits>

#include <algorithm>

#include <cuda_bf16.h>

bool asca_tc_enabled();  // gemm.cu
namespace delta_tc {
bool available();
int forward(asca_ctx* ctx, const void* q, const void* k, const void* v, const float* alpha, const float* beta,
            int64_t B, int64_t T, int64_t H, int64_t dh, void* o, const float* s_init, float* s_final, float* ckpt);
}  // namespace delta_tc

namespace {

template <typename T>
__device__ __forceinline__ float4 ld4(const T* p);
template <>
__device__ __forceinline__ float4 ld4<float>(const float* p) { return *reinterpret_cast<const float4*>(p); }
template <>
__device__ __forceinline__ float4 ld4<__nv_bfloat16>(const __nv_bfloat16* p) {
    uint2 raw = *reinterpret_cast<const uint2*>(p);
    __nv_bfloat162 a = *reinterpret_cast<__nv_bfloat162*>(&raw.x), b = *reinterpret_cast<__nv_bfloat162*>(&raw.y);
    return make_float4(__low2float(a), __high2float(a), __low2float(b), __high2float(b));
}

// Two f32 in one 64-bit register pair. The pairs stay 64-bit values from the load to the store: built from scalars at each use
// they cost two moves per FFMA.
typedef unsigned long long pair_t;
__device__ __forceinline__ pair_t make_pair(float lo, float hi) {
    pair_t p;
    asm("mov.b64 %0, {%1, %2};" : "=l"(p) : "f"(lo), "f"(hi));
    return p;
}
__device__ __forceinline__ float2 unpair(pair_t p) {
    float2 v;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(v.x), "=f"(v.y) : "l"(p));
    return v;
}
__device__ __forceinline__ void fma2(pair_t& d, pair_t a, pair_t b) { asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(d) : "l"(a), "l"(b)); }

// LANES neighbouring lanes share COLS value columns: a lane holds DH / LANES rows of each. NT: threads per CTA.
template <int DH, int COLS>
struct RecCfg {
    static constexpr int LANES = DH == 128 ? 8 : 4, RPT = DH / LANES;
    static constexpr int ALL = DH / COLS * LANES;             // threads that hold a whole state
    static constexpr int NT = ALL < 256 ? ALL : (COLS == 1 ? 128 : 256);
    static constexpr int FW = NT / LANES * COLS;              // value columns per CTA
    static constexpr int HT = DH == 128 && COLS < 4 ? 128 : 64;           // helper threads: they stage the inputs and store the outputs
    static constexpr int FTS = DH == 128 && COLS > 1 ? 8 : 16;   // timesteps per staged block (48 KiB of shared memory)
    static_assert(RPT % 4 == 0 && NT >= 32, "tile shape");
};

// One step: sk = S^T k and sq = S^T q from the SAME pass over the old state, u = beta v - alpha beta sk,
// o = alpha sq + (k.q) u, S = alpha S + k u: the output needs no second reduction, and only sk is on the chain from step to
// step. Rows are held in pairs (k and q arrive as pairs), so all three passes are packed two-lane FFMAs. With COLS > 1 the
// 2 COLS sums of a lane group are exchanged by halves: after log2 COLS rounds a lane holds the two sums of one column.
// What bounds it: with COLS = 1 the reads of k and q (8 bytes per state element and step) once a few chains share an SM, the
// step's latency before that; COLS = 4 reads a quarter and is bound by FFMA issue.
template <int DH, int COLS, typename T>
__global__ void __launch_bounds__(RecCfg<DH, COLS>::NT + RecCfg<DH, COLS>::HT) delta_fwd_rec_kernel(
    const T* __restrict__ q, const T* __restrict__ k, const T* __restrict__ v, const float* __restrict__ alpha,
    const float* __restrict__ beta, int B, int Tlen, int H, int chunk, T* __restrict__ o,
    const float* s_init, float* s_final /* may be s_init */, float* __restrict__ ckpt) {
    using C = RecCfg<DH, COLS>;
    constexpr int LANES = C::LANES, RPT = C::RPT, NT = C::NT, HT = C::HT, FW = C::FW, FTS = C::FTS;
    constexpr int KQ4 = FTS * DH / 4;        // float4 units of k (or q) per stage
    constexpr int KQ_PT = (KQ4 + HT - 1) / HT, V_PT = (FTS * FW + HT - 1) / HT;
    static_assert(KQ4 % HT == 0, "whole rows per pass");
    __shared__ __align__(16) float k_s[2][FTS][DH];
    __shared__ __align__(16) float q_s[2][FTS][DH];
    __shared__ float v_s[2][FTS][FW];        // beta v
    // per step: product of the stage's alphas up to and with it, its inverse, -alpha beta times the product before it, k.q
    __shared__ __align__(16) float4 g_s[2][FTS];
    __shared__ float2 ab_s[2][FTS];          // alpha, beta
    __shared__ float decay_s[2];             // product of all the stage's alphas
    __shared__ float o_s[2][FTS][FW];

    const int tid = threadIdx.x;
    const int ag = tid % LANES, cg = tid / LANES;
    const int chain = blockIdx.y;              // b*H + h
    const int bi = chain / H, h = chain % H;
    const int i0 = blockIdx.x * FW;            // first value column of this CTA
    const int d = H * DH;
    const int64_t row0 = (int64_t)bi * Tlen;
    const int n_chunks = (Tlen + chunk - 1) / chunk;

    const int n_stages = (Tlen + FTS - 1) / FTS;
    if (tid >= NT) {
        const int ht = tid - NT;
        // ---- helpers: while a stage is worked on they store the outputs of the one before it, put the one after it into shared
        // memory and request the one after that; the working threads see one barrier per stage
        float4 pk[KQ_PT], pq[KQ_PT];
        float pv[V_PT], pbv[V_PT], pa = 0.0f, pb = 0.0f;
        auto fetch = [&](int t0) {
#pragma unroll
            for (int u = 0; u < KQ_PT; ++u) {
                const int idx = ht + u * HT;
                int t = idx / (DH / 4), c4 = idx % (DH / 4);
                if (idx < KQ4 && t0 + t < Tlen) {
                    int64_t off = (row0 + t0 + t) * d + h * DH + c4 * 4;
                    pk[u] = ld4<T>(k + off);
                    pq[u] = ld4<T>(q + off);
                } else {
                    pk[u] = make_float4(0, 0, 0, 0);
                    pq[u] = make_float4(0, 0, 0, 0);
                }
            }
#pragma unroll
            for (int u = 0; u < V_PT; ++u) {
                const int idx = ht + u * HT;
                int t = idx / FW, c = idx % FW;
                const bool ok = idx < FTS * FW && t0 + t < Tlen;
                pv[u] = ok ? to_f32<T>(v[(row0 + t0 + t) * d + h * DH + i0 + c]) : 0.0f;
                pbv[u] = ok ? beta[(row0 + t0 + t) * H + h] : 0.0f;
            }
            if (ht < FTS && t0 + ht < Tlen) {
                pa = alpha[(row0 + t0 + ht) * H + h];
                pb = beta[(row0 + t0 + ht) * H + h];
            }
        };
        auto stash = [&](int buf) {
#pragma unroll
            for (int u = 0; u < KQ_PT; ++u) {
                const int idx = ht + u * HT;
                int t = idx / (DH / 4), c4 = idx % (DH / 4);
                float kq = pk[u].x * pq[u].x + pk[u].y * pq[u].y + pk[u].z * pq[u].z + pk[u].w * pq[u].w;   // the row's lanes: one warp
#pragma unroll
                for (int m = (DH / 4 < 32 ? DH / 4 : 32) / 2; m > 0; m >>= 1) kq += __shfl_xor_sync(0xffffffffu, kq, m);
                if (idx < KQ4) {
                    *reinterpret_cast<float4*>(&k_s[buf][t][c4 * 4]) = pk[u];
                    *reinterpret_cast<float4*>(&q_s[buf][t][c4 * 4]) = pq[u];
                    if (c4 == 0) g_s[buf][t].w = kq;
                }
            }
#pragma unroll
            for (int u = 0; u < V_PT; ++u) {
                const int idx = ht + u * HT;
                if (idx < FTS * FW) v_s[buf][idx / FW][idx % FW] = pbv[u] * pv[u];
            }
            if (ht < 32) {
                float dec = ht < FTS ? pa : 1.0f;
#pragma unroll
                for (int m = 1; m < FTS; m <<= 1) {
                    const float x = __shfl_up_sync(0xffffffffu, dec, m);
                    if (ht >= m) dec *= x;
                }
                const float before = __shfl_up_sync(0xffffffffu, dec, 1);
                if (ht < FTS) {
                    g_s[buf][ht].x = dec;
                    g_s[buf][ht].y = 1.0f / dec;
                    g_s[buf][ht].z = -pa * pb * (ht ? before : 1.0f);
                    ab_s[buf][ht] = make_float2(pa, pb);
                }
                if (ht == FTS - 1) decay_s[buf] = dec;
            }
        };
        auto store = [&](int stage) {
            const int t0 = stage * FTS, steps = Tlen - t0 < FTS ? Tlen - t0 : FTS;
            for (int idx = ht; idx < steps * FW; idx += HT) {
                const int ts = idx / FW, c = idx % FW;
                o[(row0 + t0 + ts) * d + h * DH + i0 + c] = from_f32<T>(o_s[stage & 1][ts][c]);
            }
        };
        fetch(0);
        stash(0);
        if (n_stages > 1) fetch(FTS);
        __syncthreads();
        for (int st = 0; st < n_stages; ++st) {
            if (st > 0) store(st - 1);
            if (st + 1 < n_stages) stash((st + 1) & 1);
            if (st + 2 < n_stages) fetch((st + 2) * FTS);
            __syncthreads();
        }
        store(n_stages - 1);
        return;
    }

    auto row_of = [&](int p) { return ((p >> 1) * LANES + ag) * 4 + (p & 1) * 2; };   // rows (r, r + 1) of pair p
    pair_t S[RPT / 2][COLS];
#pragma unroll
    for (int p = 0; p < RPT / 2; ++p)
#pragma unroll
        for (int c = 0; c < COLS; ++c) {
            const float* si = s_init + (int64_t)chain * DH * DH + i0 + cg * COLS + c;
            S[p][c] = s_init ? make_pair(si[row_of(p) * DH], si[(row_of(p) + 1) * DH]) : 0;
        }
    // The decay is kept out of the registers: inside a stage the state is the product of the alphas so far times S, and a step
    // adds k (u / product) -- one FFMA per element where alpha S + k u takes a multiply besides. The product is folded in at the
    // end of the stage; a stage whose product falls below 1e-4 (u / product stays far inside the f32 range above it) folds in
    // every step's alpha instead.
    auto fold = [&](float by) {
#pragma unroll
        for (int p = 0; p < RPT / 2; ++p)
#pragma unroll
            for (int c = 0; c < COLS; ++c) S[p][c] = make_pair(unpair(S[p][c]).x * by, unpair(S[p][c]).y * by);
    };
    int mine = 0;   // the column of its group whose sums a lane ends up with
#pragma unroll
    for (int w = COLS / 2, bit = 1; w > 0; w >>= 1, bit <<= 1) mine = mine * 2 + (ag & bit ? 1 : 0);
    auto write_state = [&](float* dst) {  // dst: dh x dh row-major, the caller's buffer: of any alignment
        const bool vec = COLS == 4 && (reinterpret_cast<uintptr_t>(dst) & 15) == 0;
#pragma unroll
        for (int p = 0; p < RPT / 2; ++p)
#pragma unroll
            for (int e = 0; e < 2; ++e) {
                float* at = dst + (row_of(p) + e) * DH + i0 + cg * COLS;
                float x[COLS];
#pragma unroll
                for (int c = 0; c < COLS; ++c) x[c] = e ? unpair(S[p][c]).y : unpair(S[p][c]).x;
                if (vec) {
                    *reinterpret_cast<float4*>(at) = make_float4(x[0], x[1 % COLS], x[2 % COLS], x[3 % COLS]);
                } else {
#pragma unroll
                    for (int c = 0; c < COLS; ++c) at[c] = x[c];
                }
            }
    };

    int next_ck = ckpt ? 0 : Tlen;
    __syncthreads();
    for (int st = 0; st < n_stages; ++st) {
        const int t0 = st * FTS, buf = st & 1, steps = Tlen - t0 < FTS ? Tlen - t0 : FTS;
        if (t0 == next_ck) {
            write_state(ckpt + ((int64_t)chain * n_chunks + t0 / chunk) * DH * DH);
            next_ck += chunk;
        }
        struct Row {
            pair_t k[RPT / 2], q[RPT / 2];
            float4 g;
            float v;
        };
        auto read = [&](int ts, Row& x) {
            x.g = g_s[buf][ts];
            x.v = v_s[buf][ts][cg * COLS + mine];
#pragma unroll
            for (int r = 0; r < RPT / 4; ++r) {
                const ulonglong2 a = *reinterpret_cast<const ulonglong2*>(&k_s[buf][ts][(r * LANES + ag) * 4]),
                                 b = *reinterpret_cast<const ulonglong2*>(&q_s[buf][ts][(r * LANES + ag) * 4]);
                x.k[2 * r] = a.x; x.k[2 * r + 1] = a.y;
                x.q[2 * r] = b.x; x.q[2 * r + 1] = b.y;
            }
        };
        // dec: the decay folded in after this step, inv: its inverse, nab: -alpha beta times the decay before it
        auto step = [&](int ts, const Row& x, float dec, float inv, float nab) {
            float val[2 * COLS];   // (sk, sq) of each column
#pragma unroll
            for (int c = 0; c < COLS; ++c) {
                pair_t sk = 0, sq = 0;
#pragma unroll
                for (int p = 0; p < RPT / 2; ++p) {
                    fma2(sk, S[p][c], x.k[p]);
                    fma2(sq, S[p][c], x.q[p]);
                }
                val[2 * c] = unpair(sk).x + unpair(sk).y;
                val[2 * c + 1] = unpair(sq).x + unpair(sq).y;
            }
            // exchange by halves: round i keeps the columns whose bit i matches the lane's
#pragma unroll
            for (int w = COLS / 2, bit = 1; w > 0; w >>= 1, bit <<= 1) {
                const bool up = ag & bit;
#pragma unroll
                for (int j = 0; j < 2 * w; ++j) {
                    const float send = up ? val[j] : val[2 * w + j], keep = up ? val[2 * w + j] : val[j];
                    val[j] = keep + __shfl_xor_sync(0xffffffffu, send, bit);
                }
            }
#pragma unroll
            for (int bit = COLS; bit < LANES; bit <<= 1) {
                val[0] += __shfl_xor_sync(0xffffffffu, val[0], bit);
                val[1] += __shfl_xor_sync(0xffffffffu, val[1], bit);
            }
            const float u = fmaf(nab, val[0], x.v), us = u * inv;
            if (ag < COLS) o_s[buf][ts][cg * COLS + mine] = fmaf(dec, val[1], x.g.w * u);
#pragma unroll
            for (int c = 0; c < COLS; ++c) {
                // the lane of the group that holds column c: its bits, most significant column bit first
                const int src = COLS == 4 ? ((c >> 1) | ((c & 1) << 1)) : c;
                const float uc = COLS == 1 ? us : __shfl_sync(0xffffffffu, us, ((tid & 31) & ~(LANES - 1)) | src);
                const pair_t u2 = make_pair(uc, uc);
#pragma unroll
                for (int p = 0; p < RPT / 2; ++p) fma2(S[p][c], x.k[p], u2);
            }
        };
        Row ra, rb;
        read(0, ra);
        if (steps == FTS && decay_s[buf] > 1e-4f && next_ck >= t0 + FTS) {
            // a step's rows are read while the one before it is worked on
#pragma unroll 1
            for (int ts = 0; ts < FTS; ts += 2) {
                read(ts + 1, rb);
                step(ts, ra, ra.g.x, ra.g.y, ra.g.z);
                read((ts + 2) % FTS, ra);   // (past the last step: a read of no use, but an unconditional one)
                step(ts + 1, rb, rb.g.x, rb.g.y, rb.g.z);
            }
            fold(decay_s[buf]);
        } else {   // ragged stages, checkpoints inside a stage, strong decay: folded in at every step
#pragma unroll 1
            for (int ts = 0; ts < steps; ++ts) {
                if (t0 + ts == next_ck) {
                    write_state(ckpt + ((int64_t)chain * n_chunks + (t0 + ts) / chunk) * DH * DH);
                    next_ck += chunk;
                }
                read(ts, ra);
                const float2 ab = ab_s[buf][ts];
                fold(ab.x);   // (alpha S)^T k = alpha (S^T k): the decayed state takes the step with decay 1
                step(ts, ra, 1.0f, 1.0f, -ab.y);
            }
        }
        __syncthreads();
    }
    if (s_final) write_state(s_final + (int64_t)chain * DH * DH);
}

// ------------------------------------------------------------------ decode step
template <int DH>
struct StepCfg {
    static constexpr int THREADS = DH >= 32 ? 256 : 64;
    static constexpr int CV = DH / 4;            // float4 columns
    static constexpr int RG = THREADS / CV;      // row groups
    static constexpr int RPT = DH / RG;          // rows per thread
};

template <int DH>
__global__ void __launch_bounds__(StepCfg<DH>::THREADS) delta_step_kernel(
    const float* __restrict__ q, const float* __restrict__ k, const float* __restrict__ v,
    const float* __restrict__ alpha, const float* __restrict__ beta, float* __restrict__ S, int H, int fused,
    float* __restrict__ o) {
    using C = StepCfg<DH>;
    __shared__ __align__(16) float qs[DH], ks[DH], vs[DH];
    __shared__ __align__(16) float red[C::RG][DH];
    __shared__ float rsum[33];
    __shared__ float ab[2];
    const int tid = threadIdx.x;
    const int unit = blockIdx.x;  // stream*H + h
    const int s = unit / H, h = unit % H;
    const int d = H * DH;
    // ---- inputs (optionally the fused prologue: L2 normalise + sigmoid)
    if (fused) {
        const float* row = q + (int64_t)s * 3 * d + h * DH;
        float qv = 0.0f, kv = 0.0f;
        if (tid < DH) {
            qv = row[tid];
            kv = row[d + tid];
            vs[tid] = row[2 * d + tid];
        }
        const float qq = block_sum(qv * qv, rsum);
        const float kk2 = block_sum(kv * kv, rsum);
        const float qi = 1.0f / fmaxf(sqrtf(qq), 1e-8f), ki = 1.0f / fmaxf(sqrtf(kk2), 1e-8f);
        if (tid < DH) {
            qs[tid] = qv * qi;
            ks[tid] = kv * ki;
        }
        if (tid == 0) {
            ab[0] = 1.0f / (1.0f + expf(-alpha[(int64_t)s * 2 * H + h]));
            ab[1] = 1.0f / (1.0f + expf(-alpha[(int64_t)s * 2 * H + H + h]));
        }
    } else {
        if (tid < DH) {
            qs[tid] = q[(int64_t)s * d + h * DH + tid];
            ks[tid] = k[(int64_t)s * d + h * DH + tid];
            vs[tid] = v[(int64_t)s * d + h * DH + tid];
        }
        if (tid == 0) {
            ab[0] = alpha[(int64_t)s * H + h];
            ab[1] = beta[(int64_t)s * H + h];
        }
    }
    const int cv = tid % C::CV, rg = tid / C::CV;
    float4* Sg = reinterpret_cast<float4*>(S + (int64_t)unit * DH * DH);
    float4 st[C::RPT];
#pragma unroll
    for (int r = 0; r < C::RPT; ++r) st[r] = Sg[(rg + C::RG * r) * C::CV + cv];  // loads in flight over the sync
    __syncthreads();
    const float a = ab[0], b = ab[1];
    float4 acc = make_float4(0, 0, 0, 0);
#pragma unroll
    for (int r = 0; r < C::RPT; ++r) {
        const float ka = ks[rg + C::RG * r];
        acc.x = fmaf(st[r].x, ka, acc.x); acc.y = fmaf(st[r].y, ka, acc.y);
        acc.z = fmaf(st[r].z, ka, acc.z); acc.w = fmaf(st[r].w, ka, acc.w);
    }
    *reinterpret_cast<float4*>(&red[rg][cv * 4]) = acc;
    __syncthreads();
    float4 sk = make_float4(0, 0, 0, 0);
#pragma unroll
    for (int g = 0; g < C::RG; ++g) {
        float4 t = *reinterpret_cast<const float4*>(&red[g][cv * 4]);
        sk.x += t.x; sk.y += t.y; sk.z += t.z; sk.w += t.w;
    }
    const float4 vv = *reinterpret_cast<const float4*>(&vs[cv * 4]);
    const float4 u = make_float4(b * (vv.x - a * sk.x), b * (vv.y - a * sk.y), b * (vv.z - a * sk.z),
                                 b * (vv.w - a * sk.w));
    acc = make_float4(0, 0, 0, 0);
#pragma unroll
    for (int r = 0; r < C::RPT; ++r) {
        const int row = rg + C::RG * r;
        const float ka = ks[row], qa = qs[row];
        st[r].x = fmaf(ka, u.x, a * st[r].x); st[r].y = fmaf(ka, u.y, a * st[r].y);
        st[r].z = fmaf(ka, u.z, a * st[r].z); st[r].w = fmaf(ka, u.w, a * st[r].w);
        Sg[row * C::CV + cv] = st[r];
        acc.x = fmaf(st[r].x, qa, acc.x); acc.y = fmaf(st[r].y, qa, acc.y);
        acc.z = fmaf(st[r].z, qa, acc.z); acc.w = fmaf(st[r].w, qa, acc.w);
    }
    __syncthreads();  // everyone has finished reading red[] for sk
    *reinterpret_cast<float4*>(&red[rg][cv * 4]) = acc;
    __syncthreads();
    if (rg == 0) {
        float4 ov = make_float4(0, 0, 0, 0);
#pragma unroll
        for (int g = 0; g < C::RG; ++g) {
            float4 t = *reinterpret_cast<const float4*>(&red[g][cv * 4]);
            ov.x += t.x; ov.y += t.y; ov.z += t.z; ov.w += t.w;
        }
        *reinterpret_cast<float4*>(o + (int64_t)s * d + h * DH + cv * 4) = ov;
    }
}

// Decode step for head dim 64, one WARP per (stream, head): lane l owns value columns 2l and 2l+1 of the 64 x 64
// state, all 64 rows (64 float2 loads issued back to back, 256 contiguous bytes per row across the warp). Every
// per-column quantity (S^T k, u, the update, S^T q) is local to the lane, so the step needs no block barrier and
// no cross-lane reduction except the two norms of the fused prologue; k and q are broadcast from the warp's slice
// of shared memory. qkv / gate may be the two parts of one wider row (row pitches ld_qkv, ld_gate); o16, when
// given, receives a bf16 copy of the output for a following tensor-core product.
constexpr int SW_WARPS = 8;
__global__ void __launch_bounds__(SW_WARPS * 32) delta_step_warp64_kernel(
    const float* __restrict__ q, const float* __restrict__ k, const float* __restrict__ v, const float* __restrict__ alpha,
    const float* __restrict__ beta, float* __restrict__ S, int64_t n_units, int H, int fused, int64_t ld_qkv,
    int64_t ld_gate, float* __restrict__ o, __nv_bfloat16* __restrict__ o16) {
    constexpr int DH = 64;
    __shared__ __align__(16) float kq_s[SW_WARPS][2][DH];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    bool waited = false;   // the state is this kernel's own (last written a step ago): the first unit's loads are issued
                           // before the wait for the previous kernel, whose output is only q, k, v and the gates
    // The grid is at most one block per SM and block b owns the units [b n / G, (b + 1) n / G): every SM streams the same
    // number of state bytes (within one unit), which is what it takes to reach the HBM rate -- an SM cannot pull more
    // than its share, so a grid of fixed-size blocks that leaves some SMs a block short loses that share.
    const int64_t lo = n_units * blockIdx.x / gridDim.x, hi = n_units * (blockIdx.x + 1) / gridDim.x;
    for (int64_t unit = lo + w; unit < hi; unit += SW_WARPS) {   // unit = stream * H + h
    __syncwarp();   // the previous unit's k and q have been read by every lane
    const int64_t s = unit / H;
    const int h = (int)(unit % H);
    const int d = H * DH;
    float2* Sg = reinterpret_cast<float2*>(S + unit * DH * DH);
    float2 st[DH];
#pragma unroll
    for (int a = 0; a < DH; ++a) st[a] = Sg[a * 32 + lane];   // in flight while the inputs are prepared
    if (!waited) {
        pdl_wait();
        pdl_launch_dependents();
        waited = true;
    }
    float2 q2, k2, v2;
    float al, be;
    if (fused) {
        const float* row = q + s * ld_qkv + h * DH + 2 * lane;
        q2 = *reinterpret_cast<const float2*>(row);
        k2 = *reinterpret_cast<const float2*>(row + d);
        v2 = *reinterpret_cast<const float2*>(row + 2 * d);
        const float qq = warp_sum(q2.x * q2.x + q2.y * q2.y), kk = warp_sum(k2.x * k2.x + k2.y * k2.y);
        const float qi = 1.0f / fmaxf(sqrtf(qq), 1e-8f), ki = 1.0f / fmaxf(sqrtf(kk), 1e-8f);
        q2.x *= qi; q2.y *= qi; k2.x *= ki; k2.y *= ki;
        al = 1.0f / (1.0f + expf(-alpha[s * ld_gate + h]));
        be = 1.0f / (1.0f + expf(-alpha[s * ld_gate + H + h]));
    } else {
        const int64_t off = s * d + h * DH + 2 * lane;
        q2 = *reinterpret_cast<const float2*>(q + off);
        k2 = *reinterpret_cast<const float2*>(k + off);
        v2 = *reinterpret_cast<const float2*>(v + off);
        al = alpha[s * H + h];
        be = beta[s * H + h];
    }
    *reinterpret_cast<float2*>(&kq_s[w][0][2 * lane]) = k2;
    *reinterpret_cast<float2*>(&kq_s[w][1][2 * lane]) = q2;
    __syncwarp();
    const float* ks = kq_s[w][0];
    const float* qs = kq_s[w][1];
    float2 sk = make_float2(0.0f, 0.0f);
#pragma unroll
    for (int a4 = 0; a4 < DH; a4 += 4) {
        const float4 k4 = *reinterpret_cast<const float4*>(ks + a4);
        sk.x = fmaf(st[a4].x, k4.x, sk.x);         sk.y = fmaf(st[a4].y, k4.x, sk.y);
        sk.x = fmaf(st[a4 + 1].x, k4.y, sk.x);     sk.y = fmaf(st[a4 + 1].y, k4.y, sk.y);
        sk.x = fmaf(st[a4 + 2].x, k4.z, sk.x);     sk.y = fmaf(st[a4 + 2].y, k4.z, sk.y);
        sk.x = fmaf(st[a4 + 3].x, k4.w, sk.x);     sk.y = fmaf(st[a4 + 3].y, k4.w, sk.y);
    }
    const float2 u = make_float2(be * (v2.x - al * sk.x), be * (v2.y - al * sk.y));
    float2 acc = make_float2(0.0f, 0.0f);
#pragma unroll
    for (int a4 = 0; a4 < DH; a4 += 4) {
        const float4 k4 = *reinterpret_cast<const float4*>(ks + a4), q4 = *reinterpret_cast<const float4*>(qs + a4);
        const float kk[4] = {k4.x, k4.y, k4.z, k4.w}, qq[4] = {q4.x, q4.y, q4.z, q4.w};
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            float2 t = st[a4 + e];
            t.x = fmaf(kk[e], u.x, al * t.x);
            t.y = fmaf(kk[e], u.y, al * t.y);
            Sg[(a4 + e) * 32 + lane] = t;
            acc.x = fmaf(t.x, qq[e], acc.x);
            acc.y = fmaf(t.y, qq[e], acc.y);
        }
    }
    *reinterpret_cast<float2*>(o + s * d + h * DH + 2 * lane) = acc;
    if (o16) *reinterpret_cast<__nv_bfloat162*>(o16 + s * d + h * DH + 2 * lane) = __floats2bfloat162_rn(acc.x, acc.y);
    }
    if (!waited) {   // a warp without a unit
        pdl_wait();
        pdl_launch_dependents();
    }
}

template <int DH, int COLS, typename T>
cudaError_t launch_fwd_cols(asca_ctx* ctx, const void* q, const void* k, const void* v, const float* alpha, const float* beta, int B,
                            int T_, int H, int chunk, void* o, const float* s_init, float* s_final, float* ckpt) {
    using C = RecCfg<DH, COLS>;
    delta_fwd_rec_kernel<DH, COLS, T><<<dim3(DH / C::FW, B * H), C::NT + C::HT, 0, ctx->stream>>>(
        (const T*)q, (const T*)k, (const T*)v, alpha, beta, B, T_, H, chunk, (T*)o, s_init, s_final, ckpt);
    return cudaGetLastError();
}
// Value columns per lane group: one while the chains leave the SMs idle (a step then takes its latency), more once the reads
// of k and q fill shared memory. `load`: states of 128 x 128 per SM.
template <int DH, typename T>
cudaError_t launch_fwd(asca_ctx* ctx, const void* q, const void* k, const void* v, const float* alpha, const float* beta, int B, int T_,
                       int H, int chunk, void* o, const float* s_init, float* s_final, float* ckpt) {
    const double n_sm = ctx->sm_count > 0 ? ctx->sm_count : 148, load = (double)B * H * DH * DH / (128 * 128) / n_sm;
    if (DH >= 32 && load > 0.5)
        return launch_fwd_cols<DH, DH >= 32 ? 4 : 1, T>(ctx, q, k, v, alpha, beta, B, T_, H, chunk, o, s_init, s_final, ckpt);
    if (DH >= 32 && load > 0.25)
        return launch_fwd_cols<DH, DH >= 32 ? 2 : 1, T>(ctx, q, k, v, alpha, beta, B, T_, H, chunk, o, s_init, s_final, ckpt);
    return launch_fwd_cols<DH, 1, T>(ctx, q, k, v, alpha, beta, B, T_, H, chunk, o, s_init, s_final, ckpt);
}

}  // namespace

template <typename... A>
std::integral_constant<int, sizeof...(A)> n_args(void (*)(A...));
// A recorded launch of delta_step_warp64_kernel goes to the states at S from now on (launches under way keep theirs).
int asca_delta_step_repoint(asca_ctx* ctx, cudaGraphExec_t exec, cudaGraphNode_t node, float* S) {
    constexpr int N_ARGS = decltype(n_args(delta_step_warp64_kernel))::value, S_ARG = 5;   // (q, k, v, alpha, beta, S, ...)
    cudaKernelNodeParams kp;
    ASCA_CUDA(ctx, cudaGraphKernelNodeGetParams(node, &kp));
    void* args[N_ARGS];
    for (int i = 0; i < N_ARGS; ++i) args[i] = kp.kernelParams[i];
    args[S_ARG] = &S;
    kp.kernelParams = args;
    ASCA_CUDA(ctx, cudaGraphExecKernelNodeSetParams(exec, node, &kp));
    return ASCA_OK;
}

extern "C" {

int64_t asca_delta_ckpt_floats(int64_t B, int64_t T, int64_t H, int64_t dh, int64_t chunk) {
    if (B <= 0 || T <= 0 || H <= 0 || dh <= 0 || chunk <= 0) return 0;
    return B * H * ((T + chunk - 1) / chunk) * dh * dh;
}

int asca_delta_fwd(asca_ctx* ctx, const void* q, const void* k, const void* v, const float* alpha, const float* beta,
                   int64_t B, int64_t T, int64_t H, int64_t dh, int64_t chunk, int dtype, void* o, const float* s_init,
                   float* s_final, float* ckpt) {
    if (!ctx) return ASCA_ERR_ARG;
    ASCA_REQUIRE(ctx, q && k && v && alpha && beta && o, "delta_fwd: null pointer");
    ASCA_REQUIRE(ctx, B >= 0 && T >= 0 && H > 0 && B * H < 65536 && B * T < (1ll << 31), "delta_fwd: bad shape");
    ASCA_REQUIRE(ctx, dtype == ASCA_F32 || dtype == ASCA_BF16, "delta_fwd: unknown dtype");
    ASCA_REQUIRE(ctx, !ckpt || chunk >= 1, "delta_fwd: chunk must be >= 1 when checkpoints are requested");
    if (dh != 16 && dh != 32 && dh != 64 && dh != 128)
        return asca_fail(ctx, ASCA_ERR_UNSUPPORTED, "delta_fwd: dh must be 16, 32, 64 or 128 (got %lld)", (long long)dh);
    const uintptr_t al = (uintptr_t)q | (uintptr_t)k | (uintptr_t)v | (uintptr_t)o;
    ASCA_REQUIRE(ctx, (al & 15) == 0, "delta_fwd: q, k, v, o must be 16-byte aligned");
    if (B == 0) return ASCA_OK;
    if (T == 0) {
        if (s_final) {
            if (s_init) ASCA_CUDA(ctx, cudaMemcpyAsync(s_final, s_init, (size_t)(B * H * dh * dh) * 4, cudaMemcpyDeviceToDevice, ctx->stream));
            else ASCA_CUDA(ctx, cudaMemsetAsync(s_final, 0, (size_t)(B * H * dh * dh) * 4, ctx->stream));
        }
        return ASCA_OK;
    }
    // bf16 mode, dh = 128 or 64: chunk-parallel WY/UT form on the tensor cores (checkpoints every 64)
    if (dtype == ASCA_BF16 && (dh == 128 || dh == 64) && (!ckpt || chunk == 64) && asca_tc_enabled() && delta_tc::available())
        return delta_tc::forward(ctx, q, k, v, alpha, beta, B, T, H, dh, o, s_init, s_final, ckpt);
    if (ckpt)
        for (auto& e : ctx->dtiles)
            if (e.ckpt == (const void*)ckpt) e.ckpt = nullptr;   // kept tiles no longer match this buffer
    const int ch = ckpt ? (int)chunk : 1;
    cudaError_t e;
    asca_span sp(ctx, "delta_fwd_rec_kernel");
#define ASCA_FWD(DH_)                                                                                              \
    e = dtype == ASCA_BF16                                                                                         \
            ? launch_fwd<DH_, __nv_bfloat16>(ctx, q, k, v, alpha, beta, (int)B, (int)T, (int)H, ch, o, s_init, \
                                             s_final, ckpt)                                                        \
            : launch_fwd<DH_, float>(ctx, q, k, v, alpha, beta, (int)B, (int)T, (int)H, ch, o, s_init,     \
                                     s_final, ckpt)
    switch (dh) {
        case 16: ASCA_FWD(16); break;
        case 32: ASCA_FWD(32); break;
        case 64: ASCA_FWD(64); break;
        default: ASCA_FWD(128); break;
    }
#undef ASCA_FWD
    ASCA_CUDA(ctx, e);
    ctx->launches++;
    return ASCA_OK;
}

// fused = 1 only: qkv rows of pitch ld_qkv, gate rows of pitch ld_gate (both may point into one wider buffer);
// o16 (nullable) gets a bf16 copy of o. dh = 64.
int asca_delta_step_strided(asca_ctx* ctx, const float* qkv, int64_t ld_qkv, const float* gate, int64_t ld_gate, float* S,
                            int64_t n_streams, int64_t H, float* o, void* o16) {
    if (!ctx) return ASCA_ERR_ARG;
    ASCA_REQUIRE(ctx, qkv && gate && S && o && n_streams >= 0 && H > 0, "delta_step_strided: bad arguments");
    ASCA_REQUIRE(ctx, ld_qkv >= 3 * H * 64 && ld_gate >= 2 * H && (ld_qkv & 1) == 0, "delta_step_strided: bad row pitch");
    ASCA_REQUIRE(ctx, (((uintptr_t)S | (uintptr_t)o | (uintptr_t)qkv) & 7) == 0 && ((uintptr_t)o16 & 3) == 0,
                 "delta_step_strided: misaligned pointer");
    if (n_streams == 0) return ASCA_OK;
    const int64_t units = n_streams * H;
    const int64_t n_sm = ctx->sm_count > 0 ? ctx->sm_count : 148;
    asca_span sp(ctx, "delta_step_warp64_kernel", (double)units * 2.0 * 64 * 64 * 4);   // state bytes read + written
    ASCA_CUDA(ctx, asca_launch(ctx, delta_step_warp64_kernel, dim3((unsigned)std::min(n_sm, ceil_div64(units, SW_WARPS))), dim3(SW_WARPS * 32), 0,
                               qkv, nullptr, nullptr, gate, nullptr, S, units, (int)H, 1, ld_qkv, ld_gate, o, (__nv_bfloat16*)o16));
    ctx->launches++;
    return ASCA_OK;
}

int asca_delta_step(asca_ctx* ctx, const float* q, const float* k, const float* v, const float* alpha,
                    const float* beta, float* S, int64_t n_streams, int64_t H, int64_t dh, int fused, float* o) {
    if (!ctx) return ASCA_ERR_ARG;
    ASCA_REQUIRE(ctx, q && alpha && S && o && (fused || (k && v && beta)), "delta_step: null pointer");
    ASCA_REQUIRE(ctx, n_streams >= 0 && H > 0 && n_streams * H < (1ll << 31), "delta_step: bad shape");
    if (dh != 16 && dh != 32 && dh != 64 && dh != 128)
        return asca_fail(ctx, ASCA_ERR_UNSUPPORTED, "delta_step: dh must be 16, 32, 64 or 128 (got %lld)", (long long)dh);
    ASCA_REQUIRE(ctx, (((uintptr_t)S | (uintptr_t)o) & 15) == 0, "delta_step: S and o must be 16-byte aligned");
    if (n_streams == 0) return ASCA_OK;
    const unsigned grid = (unsigned)(n_streams * H);
    const bool in8 = fused ? ((uintptr_t)q & 7) == 0 : (((uintptr_t)q | (uintptr_t)k | (uintptr_t)v) & 7) == 0;
    if (dh == 64 && in8) {   // one warp per (stream, head), no block barrier
        const int64_t units = n_streams * H;
        const int64_t n_sm = ctx->sm_count > 0 ? ctx->sm_count : 148;
        delta_step_warp64_kernel<<<(unsigned)std::min(n_sm, ceil_div64(units, SW_WARPS)), SW_WARPS * 32, 0, ctx->stream>>>(
            q, k, v, alpha, beta, S, units, (int)H, fused, 3 * H * dh, 2 * H, o, nullptr);
        ASCA_CHECK_LAUNCH(ctx);
        return ASCA_OK;
    }
    switch (dh) {
        case 16: delta_step_kernel<16><<<grid, StepCfg<16>::THREADS, 0, ctx->stream>>>(q, k, v, alpha, beta, S, (int)H, fused, o); break;
        case 32: delta_step_kernel<32><<<grid, StepCfg<32>::THREADS, 0, ctx->stream>>>(q, k, v, alpha, beta, S, (int)H, fused, o); break;
        case 64: delta_step_kernel<64><<<grid, StepCfg<64>::THREADS, 0, ctx->stream>>>(q, k, v, alpha, beta, S, (int)H, fused, o); break;
        default: delta_step_kernel<128><<<grid, StepCfg<128>::THREADS, 0, ctx->stream>>>(q, k, v, alpha, beta, S, (int)H, fused, o); break;
    }
    ASCA_CHECK_LAUNCH(ctx);
    return ASCA_OK;
}

}  // extern "C"
