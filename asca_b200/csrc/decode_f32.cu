// f32 decode: the whole of Model::step (rust/src/model.rs:631-649) for any number of steps in one launch.
//
// Streams are independent, so a stream gets a thread-block cluster of its own (8 CTAs for a few streams, fewer when the
// streams alone fill the GPU) and nothing ever waits for another stream. What bounds a step of one stream is latency -- a
// 331k-parameter model needs 116 k multiply-adds a token -- so the step is organised to synchronise as little as possible:
//   * every CTA keeps the residual row in its own shared memory; a block is two exchanges. A CTA owns some heads: it projects
//     their q, k, v and gates, updates their states and multiplies their o with its ROWS of W_o; the partial rows (d floats)
//     go to every CTA through distributed shared memory, one cluster barrier, and every CTA adds them up in the same order.
//     The expert layer is cut the same way: a slice of the hidden features, then those rows of W2.
//   * the recurrent states stay in shared memory over all steps (transposed: a warp owns value columns, its lanes the rows).
//   * S^T k and S^T q are taken from the same pass over the old state: o = a S^T q + (k.q) u, one reduction instead of two.
//   * a product's weights are requested before the barrier in front of it: they do not depend on it.
//   * the RMSNorm factor multiplies the finished sums (a row's norm is needed only there).
// Weights come through L1: a 331k model's share of a CTA stays there over the steps.
// One stream of the 331k model: 17.6 us a token (128 a call); step by step through the single kernels 106.
#include "model.cuh"

#include <algorithm>

namespace {

constexpr int DT = 512;   // threads per CTA
constexpr int NR = 10;    // weight rows of a thread that are requested ahead

struct DecodeArgs {
    const float* P;
    int64_t embed, head, layer_stride;
    Lyr l0;                       // offsets in the first block; block i adds i * layer_stride
    int d, H, L, E, F, V, ns;
    int64_t n_steps;
    float* state;                 // (L, ns, H, dh, dh)
    const uint32_t* ids;          // first step's tokens
    uint32_t* tokens;             // (n_steps, ns)
    float* logits;                // (ns, V) of the last step, nullable
    int fl, vl;                   // hidden features / vocabulary entries per CTA, multiples of 4
};

__device__ __forceinline__ void cluster_arrive() { asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory"); }
__device__ __forceinline__ void cluster_wait() { asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory"); }

// One product x (K) times W (K x N): a thread takes four neighbouring columns of every ks-th row of its slice of k.
struct Product {
    const float* w;   // this thread's first four columns of row 0; null: no part in it
    int64_t ld;
    int K, ks, stride, out;   // rows ks, ks + stride, ...; first output of the four
};
struct Split {   // how the threads share a product with nq column quads and K rows
    int nq, slices;
    __device__ Split(int nq_, int K) : nq(nq_), slices(max(1, min(DT / max(nq_, 1), (K + 3) / 4))) {}
};

__device__ __forceinline__ void request(const Product& p, float4 (&w)[NR]) {
#pragma unroll
    for (int i = 0; i < NR; ++i) {
        const int k = p.ks + i * p.stride;
        if (p.w && k < p.K) w[i] = __ldg(reinterpret_cast<const float4*>(p.w + (int64_t)k * p.ld));
    }
}
// partial sums of this thread's rows -> red[slice][out .. out + 3]
__device__ __forceinline__ void multiply(const Product& p, const float4 (&w)[NR], const float* x, float* red, int n_out) {
    if (!p.w) return;
    float4 a = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
#pragma unroll
    for (int i = 0; i < NR; ++i) {
        const int k = p.ks + i * p.stride;
        if (k < p.K) {
            const float v = x[k];
            a.x = fmaf(v, w[i].x, a.x); a.y = fmaf(v, w[i].y, a.y); a.z = fmaf(v, w[i].z, a.z); a.w = fmaf(v, w[i].w, a.w);
        }
    }
    for (int k = p.ks + NR * p.stride; k < p.K; k += p.stride) {
        const float4 t = __ldg(reinterpret_cast<const float4*>(p.w + (int64_t)k * p.ld));
        const float v = x[k];
        a.x = fmaf(v, t.x, a.x); a.y = fmaf(v, t.y, a.y); a.z = fmaf(v, t.z, a.z); a.w = fmaf(v, t.w, a.w);
    }
    *reinterpret_cast<float4*>(red + p.ks * n_out + p.out) = a;
}
__device__ __forceinline__ float add_slices(const float* red, int slices, int n_out, int j) {
    float t = 0.0f;
#pragma unroll 4
    for (int s = 0; s < slices; ++s) t += red[s * n_out + j];
    return t;
}

template <int DH>
__global__ void __launch_bounds__(DT, 1) decode_f32_kernel(const __grid_constant__ DecodeArgs g) {
    constexpr int RPL = DH < 32 ? 1 : DH / 32;   // state rows per lane
    constexpr int CPW = DH < 32 ? 2 : 1;         // value columns a warp holds at a time
    extern __shared__ __align__(16) float sm[];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    uint32_t rank, cs;
    asm("mov.u32 %0, %%cluster_ctarank;" : "=r"(rank));
    asm("mov.u32 %0, %%cluster_nctarank;" : "=r"(cs));
    const int s = blockIdx.x / cs, d = g.d;
    const int h0 = g.H * rank / cs, h1 = g.H * (rank + 1) / cs, nh = h1 - h0;   // this CTA's heads
    const int f0 = min(g.F, (int)rank * g.fl), nf = min(g.fl, g.F - f0), v0 = min(g.V, (int)rank * g.vl), nv = min(g.vl, g.V - v0);
    const int nh_max = (g.H + cs - 1) / cs;

    float* x = sm;                          // residual row
    float* part_a = x + d;                  // cs partial rows of the delta block
    float* part_b = part_a + cs * d;        // cs partial rows of the expert layer
    float* red = part_b + cs * d;           // partial sums of a product
    float* qkv = red + 4 * DT;              // this CTA's heads: q, k, v
    float* gates = qkv + nh_max * 3 * DH;   // alpha, beta
    float* o = gates + 2 * nh_max;
    float* hid = o + nh_max * DH + (2 * nh_max & 2);   // (16-byte aligned again)
    float* best = hid + max(g.fl, g.vl);    // cs (value, index) pairs
    float* S = best + 2 * cs;               // [layer][head][value column][key row]

    // states in, transposed
    for (int li = 0; li < g.L; ++li)
        for (int i = tid; i < nh * DH * DH; i += DT) {
            const int hh = i / (DH * DH), e = i % (DH * DH);
            S[(li * nh + hh) * DH * DH + (e % DH) * DH + e / DH] = g.state[(((int64_t)li * g.ns + s) * g.H + h0 + hh) * DH * DH + e];
        }

    // the thread's part of each product (weight pointers of block 0, expert 0)
    Product p_qkv{}, p_o{}, p_w1{}, p_w2{}, p_head{};
    auto share = [&](Product& p, int nq, int K, const float* w, int64_t ld, int col) {   // col: of this thread's quad
        const Split sp(nq, K);
        p.ks = tid / max(nq, 1);
        p.K = K; p.ld = ld; p.stride = sp.slices;
        p.out = nq ? (tid % nq) * 4 : 0;
        p.w = nq > 0 && p.ks < sp.slices ? w + col : nullptr;
        return sp.slices;
    };
    const int n1 = nh * 3 * DH;   // outputs of the q, k, v projection
    int c1 = 0;
    if (nh) {
        const int j = (tid % (n1 / 4)) * 4, hh = j / (3 * DH), e = j % (3 * DH);
        c1 = (e / DH) * d + (h0 + hh) * DH + e % DH;
    }
    const int s_qkv = share(p_qkv, n1 / 4, d, g.P + g.l0.w_qkv, 3 * d, c1);
    const int s_o = share(p_o, nh ? d / 4 : 0, nh * DH, g.P + g.l0.w_o + (int64_t)h0 * DH * d, d, (tid % (d / 4)) * 4);
    const int s_w1 = share(p_w1, nf / 4, d, g.P + g.l0.w1 + f0, (int64_t)g.E * g.F, nf ? (tid % (nf / 4)) * 4 : 0);
    const int s_w2 = share(p_w2, nf ? d / 4 : 0, nf, g.P + g.l0.w2 + (int64_t)f0 * d, d, (tid % (d / 4)) * 4);
    const int s_head = share(p_head, nv / 4, d, g.P + g.head + v0, g.V, nv ? (tid % (nv / 4)) * 4 : 0);
    auto at = [&](Product p, int64_t off) {
        if (p.w) p.w += off;
        return p;
    };
    // d floats of this CTA's partial row (thread t: element t) into every CTA's row `rank` of a partial buffer
    auto send = [&](float* buf, int j, float v) {
        const uint32_t a = (uint32_t)__cvta_generic_to_shared(buf + rank * d + j);
        for (uint32_t c = 0; c < cs; ++c) {
            uint32_t to;
            asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(to) : "r"(a), "r"(c));
            asm volatile("st.shared::cluster.f32 [%0], %1;" ::"r"(to), "f"(v) : "memory");
        }
    };
    // the factor of the RMSNorm of row v, in every warp by itself
    auto norm_of = [&](const float* v) {
        float a = 0.0f;
        for (int i = lane; i < d; i += 32) a = fmaf(v[i], v[i], a);
        return 1.0f / sqrtf(warp_sum(a) / (float)d + 1e-6f);
    };

    float4 w[NR];
    uint32_t id = g.ids[s];
    request(p_qkv, w);
    cluster_arrive();   // every CTA of the cluster runs before anyone writes to it
    cluster_wait();
    for (int64_t step = 0; step < g.n_steps; ++step) {
        for (int i = tid; i < d; i += DT) x[i] = g.P[g.embed + (int64_t)id * d + i];
        uint32_t hsh = id * 0x9E3779B1u;   // rust/src/model.rs:69-77
        hsh ^= hsh >> 15;
        hsh *= 0x85EBCA6Bu;
        hsh ^= hsh >> 13;
        const int e = (int)(hsh % (uint32_t)g.E);
        __syncthreads();
        for (int li = 0; li < g.L; ++li) {
            const int64_t lo = li * g.layer_stride;
            // ---- q, k, v and gates of this CTA's heads
            multiply(at(p_qkv, lo), w, x, red, n1);
            request(at(p_o, lo), w);
            for (int gi = warp; gi < 2 * nh; gi += DT / 32) {   // alpha, beta of each head: a warp each
                const int col = (gi & 1) * g.H + h0 + (gi >> 1);
                float a = 0.0f;
                for (int k = lane; k < d; k += 32) a = fmaf(x[k], __ldg(g.P + g.l0.w_gate + lo + (int64_t)k * 2 * g.H + col), a);
                a = warp_sum(a) + g.P[g.l0.b_gate + lo + col];
                if (lane == 0) gates[gi] = 1.0f / (1.0f + expf(-a));
            }
            __syncthreads();
            for (int j = tid; j < n1; j += DT) {
                const int hh = j / (3 * DH), ee = j % (3 * DH);
                qkv[j] = add_slices(red, s_qkv, n1, j) + g.P[g.l0.b_qkv + lo + (ee / DH) * d + (h0 + hh) * DH + ee % DH];
            }
            __syncthreads();
            // ---- state update: a warp per value column (two of 16 rows at dh 16), lanes over the key rows
            for (int hh = 0; hh < nh; ++hh) {
                const float* q = qkv + hh * 3 * DH;
                float kr[RPL], qr[RPL], qq = 0.0f, kk = 0.0f, kq = 0.0f;
#pragma unroll
                for (int r = 0; r < RPL; ++r) {
                    qr[r] = q[(lane % DH) + 32 * r];
                    kr[r] = q[DH + (lane % DH) + 32 * r];
                    qq = fmaf(qr[r], qr[r], qq);
                    kk = fmaf(kr[r], kr[r], kk);
                    kq = fmaf(kr[r], qr[r], kq);
                }
#pragma unroll
                for (int m = (DH < 32 ? DH : 32) / 2; m > 0; m >>= 1) {
                    qq += __shfl_xor_sync(0xffffffffu, qq, m);
                    kk += __shfl_xor_sync(0xffffffffu, kk, m);
                    kq += __shfl_xor_sync(0xffffffffu, kq, m);
                }
                const float qi = 1.0f / fmaxf(sqrtf(qq), 1e-8f), ki = 1.0f / fmaxf(sqrtf(kk), 1e-8f);
                kq *= qi * ki;
#pragma unroll
                for (int r = 0; r < RPL; ++r) qr[r] *= qi, kr[r] *= ki;
                const float al = gates[2 * hh], be = gates[2 * hh + 1];
                float* Sh = S + (li * nh + hh) * DH * DH;
                for (int c = warp * CPW; c < DH; c += DT / 32 * CPW) {
                    const int col = c + (CPW == 2 ? lane / DH : 0);
                    float st[RPL], sk = 0.0f, sq = 0.0f;
#pragma unroll
                    for (int r = 0; r < RPL; ++r) {
                        st[r] = Sh[col * DH + (lane % DH) + 32 * r];
                        sk = fmaf(st[r], kr[r], sk);
                        sq = fmaf(st[r], qr[r], sq);
                    }
#pragma unroll
                    for (int m = (DH < 32 ? DH : 32) / 2; m > 0; m >>= 1) {
                        sk += __shfl_xor_sync(0xffffffffu, sk, m);
                        sq += __shfl_xor_sync(0xffffffffu, sq, m);
                    }
                    const float u = be * (q[2 * DH + col] - al * sk);
#pragma unroll
                    for (int r = 0; r < RPL; ++r) Sh[col * DH + (lane % DH) + 32 * r] = fmaf(kr[r], u, al * st[r]);
                    if (lane % DH == 0) o[hh * DH + col] = fmaf(kq, u, al * sq);
                }
            }
            __syncthreads();
            // ---- this CTA's rows of W_o
            multiply(at(p_o, lo), w, o, red, d);
            request(at(p_w1, lo + (int64_t)e * g.F), w);
            __syncthreads();
            if (nh)
                for (int j = tid; j < d; j += DT) send(part_a, j, add_slices(red, s_o, d, j));
            cluster_arrive();
            cluster_wait();
            for (int j = tid; j < d; j += DT) {
                float v = 0.0f;
                for (uint32_t c = 0; c < cs; ++c)
                    if (g.H * (c + 1) / cs > g.H * c / cs) v += part_a[c * d + j];
                x[j] += v + g.P[g.l0.b_o + lo + j];
            }
            __syncthreads();
            // ---- expert layer: a slice of the hidden features, then those rows of W2
            const float inv = norm_of(x);
            multiply(at(p_w1, lo + (int64_t)e * g.F), w, x, red, nf);
            request(at(p_w2, lo + (int64_t)e * g.F * d), w);
            __syncthreads();
            for (int j = tid; j < nf; j += DT) {
                const float a = inv * add_slices(red, s_w1, nf, j) + g.P[g.l0.b1 + lo + (int64_t)e * g.F + f0 + j];
                hid[j] = a / (1.0f + expf(-a));
            }
            __syncthreads();
            multiply(at(p_w2, lo + (int64_t)e * g.F * d), w, hid, red, d);
            request(li + 1 < g.L ? at(p_qkv, lo + g.layer_stride) : p_head, w);
            __syncthreads();
            if (nf > 0)
                for (int j = tid; j < d; j += DT) send(part_b, j, add_slices(red, s_w2, d, j));
            cluster_arrive();
            cluster_wait();
            for (int j = tid; j < d; j += DT) {
                float v = 0.0f;
                for (uint32_t c = 0; c < cs; ++c)
                    if ((int)c * g.fl < g.F) v += part_b[c * d + j];
                x[j] += v + g.P[g.l0.b2 + lo + j];
            }
            __syncthreads();
        }
        // ---- final norm, head, argmax (lowest index on ties)
        const float inv = norm_of(x);
        multiply(p_head, w, x, red, nv);
        request(p_qkv, w);
        __syncthreads();
        for (int j = tid; j < nv; j += DT) {
            const float a = inv * add_slices(red, s_head, nv, j);
            hid[j] = a;
            if (g.logits && step + 1 == g.n_steps) g.logits[(int64_t)s * g.V + v0 + j] = a;
        }
        __syncthreads();
        if (warp == 0) {
            float bv = -INFINITY;
            int bi = lane < nv ? v0 + lane : 0x7fffffff;   // (a row of NaNs or of -inf: the lowest index)
            for (int j = lane; j < nv; j += 32)
                if (hid[j] > bv) {
                    bv = hid[j];
                    bi = v0 + j;
                }
#pragma unroll
            for (int m = 16; m > 0; m >>= 1) {
                const float ov = __shfl_xor_sync(0xffffffffu, bv, m);
                const int oi = __shfl_xor_sync(0xffffffffu, bi, m);
                if (ov > bv || (ov == bv && oi < bi)) {
                    bv = ov;
                    bi = oi;
                }
            }
            if (lane < (int)cs) {
                uint32_t to;
                asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(to) : "r"((uint32_t)__cvta_generic_to_shared(best + 2 * rank)), "r"(lane));
                asm volatile("st.shared::cluster.v2.f32 [%0], {%1, %2};" ::"r"(to), "f"(bv), "f"(__int_as_float(bi)) : "memory");
            }
        }
        cluster_arrive();
        cluster_wait();
        float bv = -INFINITY;
        int bi = 0x7fffffff;
        for (uint32_t c = 0; c < cs; ++c) {   // ascending index ranges: the first of equals is the lowest index
            const float v = best[2 * c];
            const int i = __float_as_int(best[2 * c + 1]);
            if (v > bv || (v == bv && i < bi)) {
                bv = v;
                bi = i;
            }
        }
        id = (uint32_t)bi;
        if (rank == 0 && tid == 0) g.tokens[step * g.ns + s] = id;
    }
    for (int li = 0; li < g.L; ++li)
        for (int i = tid; i < nh * DH * DH; i += DT) {
            const int hh = i / (DH * DH), e = i % (DH * DH);
            g.state[(((int64_t)li * g.ns + s) * g.H + h0 + hh) * DH * DH + e] = S[(li * nh + hh) * DH * DH + (e % DH) * DH + e / DH];
        }
}

// Whether a call of n_steps steps is better off in this launch (`cs` CTAs a stream, so many streams at a time) than step by step
// through the single kernels. Each stream of a launch reads all its weights by itself: once every SM has one, the launch takes
// wave after wave, while a batched step shares the weights' way through L2 and is bound by its kernels' latencies. In microseconds:
//   a wave, per step   5 a block (its exchanges) + the stream's weight bytes at 37.8 kB/us an SM;  once  its states at 1 kB/us
//   a batched step     45 a block + 0.065 (a model of up to 32 MB, measured at 1 - 11) or 0.165 (measured at 51) for each dependent load of
//                      the expert kernel's two matrix-vector products, which is most of it
// Measured, us a step in one launch / batched, 32 steps a call: d 64, 2 blocks (331k) 512 streams 88 / 126, 740: 112 / 134, 1024:
// 155 / 146, 2048: 307 / 197; d 192, 6 blocks (12.7m) 296: 566 / 1315, 592: 1129 / 1459, 740: 1412 / 1513, 1024: 1952 / 1600; d 256, 4 heads,
// 2 blocks, expert width 512: 148: 127 / 226, 149: 233 / 227, 297: 349 / 235, 1024: 872 / 494. One step a call: 12.7m 296: 1233 / 1321,
// 384: 1702 / 1359; 331k 592: 135 / 148, 740: 161 / 160, 1024: 212 / 174. Of 102 points the rule takes the slower side at three: by 4 % at a
// d 96 model, by 25 and 32 % for one step a call of 384 and 444 streams of the 12.7m model, whose states then cost more than the
// estimate. Up to one wave the launch was ahead by 1.8 and more everywhere.
bool one_launch_pays(const asca_model* m, int64_t ns, int64_t n_steps, int cs, int n_sm) {
    const int64_t at_once = std::max<int64_t>(1, n_sm / cs), waves = ceil_div64(ns, at_once);
    if (waves <= 1) return true;
    const double d = (double)m->d, dh = d / (double)m->H, F = (double)m->F, L = (double)m->L, n = (double)n_steps;
    const double weights = 4.0 * (L * (4.0 * d * d + 2.0 * d * (double)m->H + 2.0 * d * F) + d * (double)m->vocab) / cs;
    const double states = 4.0 * L * (double)m->H * dh * dh / cs;
    const double loads = (double)ceil_div64(m->F, 256) * d + (double)ceil_div64(m->d, 256) * F;
    const double batched = L * (45.0 + (m->n_params * 4 <= ((int64_t)32 << 20) ? 0.065 : 0.165) * loads);
    return (double)waves * (n * (5.0 * L + weights / 37.8e3) + states / 1e3) <= n * batched;
}

size_t smem_bytes(const asca_model* m, int cs, int fl, int vl) {
    const int64_t d = m->d, dh = d / m->H, nh = (m->H + cs - 1) / cs;
    return (size_t)(d + 2 * cs * d + 4 * DT + nh * 3 * dh + 2 * nh + nh * dh + 2 + std::max(fl, vl) + 2 * cs + m->L * nh * dh * dh) * 4;
}

}  // namespace

// n_steps greedy steps of ns streams from ids (device); tokens (device, n_steps x ns), logits (device, nullable) of the last
// step. ASCA_ERR_UNSUPPORTED, nothing launched: a stream's states do not fit its cluster's shared memory, the shapes rule
// out 16-byte weight loads, or there are more streams than this form is good for (the caller steps through the single kernels then).
int asca_decode_f32(asca_ctx* ctx, asca_model* m, float* state, const uint32_t* ids, int64_t ns, int64_t n_steps, uint32_t* tokens,
                    float* logits) {
    const int64_t d = m->d, H = m->H, dh = d / H, F = m->F, V = m->vocab;
    const Lyr& a = m->lay[0];
    int64_t off = m->embed | m->head | a.w_qkv | a.w_o | a.w1 | a.w2 | F | V | d;
    const int64_t stride = m->L > 1 ? m->lay[1].w_qkv - a.w_qkv : 0;
    off |= stride;
    if ((off & 3) || d > 4 * DT || ns >= (1 << 20)) return ASCA_ERR_UNSUPPORTED;
    // the widest cluster with which all streams still run at once
    const int n_sm = ctx->sm_count > 0 ? ctx->sm_count : 148;
    int cs = 8;
    while (cs > 1 && ns * cs > n_sm) cs >>= 1;
    DecodeArgs g{};
    size_t smem;
    for (;; cs <<= 1) {   // ... and wide enough for a stream's states and a thread per column quad
        g.fl = (int)(ceil_div64(F, 4 * cs) * 4);
        g.vl = (int)(ceil_div64(V, 4 * cs) * 4);
        smem = smem_bytes(m, cs, g.fl, g.vl);
        if (smem <= ctx->smem_optin && ceil_div64(H, cs) * 3 * dh <= 4 * DT && std::max(g.fl, g.vl) <= 4 * DT) break;
        if (cs == 8) return ASCA_ERR_UNSUPPORTED;
    }
    if (!one_launch_pays(m, ns, n_steps, cs, n_sm)) return ASCA_ERR_UNSUPPORTED;
    g.P = m->params; g.embed = m->embed; g.head = m->head; g.layer_stride = stride; g.l0 = a;
    g.d = (int)d; g.H = (int)H; g.L = (int)m->L; g.E = (int)m->E; g.F = (int)F; g.V = (int)V; g.ns = (int)ns;
    g.n_steps = n_steps; g.state = state; g.ids = ids; g.tokens = tokens; g.logits = logits;
    auto kern = dh == 16 ? decode_f32_kernel<16> : dh == 32 ? decode_f32_kernel<32> : dh == 64 ? decode_f32_kernel<64> : decode_f32_kernel<128>;
    ASCA_CUDA(ctx, cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)(ns * cs));
    cfg.blockDim = dim3(DT);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = ctx->stream;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = (unsigned)cs;
    at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    ASCA_CUDA(ctx, cudaLaunchKernelEx(&cfg, kern, (const DecodeArgs)g));
    ctx->launches++;
    return ASCA_OK;
}
