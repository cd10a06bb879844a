// f32-accurate SIMT products (FFMA, f32 accumulate) with optional row gather / scatter maps and
// expert grouping. It is the exact-mode (1e-5) engine behind asca_matmul / asca_gemm and the
// grouped expert products of the hash-MoE; operands may be f32 or bf16 and are widened to f32
// on the way into shared memory.
//
// One launch takes up to four independent products of any operand form (a training step's products
// are microseconds long: what is launched together is paid for once), in one of three tile shapes:
//   128 x 128 x 16                256 threads x (8 x 8)    large products: FFMA issue bound
//    64 x  64 x 32  4 k-groups of  64 threads x (8 x 8)    a few hundred rows and up
//    32 x  32 x 64  8 k-groups of  32 threads x (4 x 8)    latency bound: few tiles, short k
// and a k-split over the CTAs of a cluster (1, 2, 4 or 8): the partial tiles stay in shared memory
// and are added across the cluster in rank order, so a weight gradient over thousands of rows with
// a handful of output tiles fills the GPU without a scratch buffer or a second launch. Results do
// not depend on scheduling. plan() picks tile shape and split from the launch's tiles and slabs.
//
// Operands go to shared memory with cp.async, STAGES slabs deep. What bounds the
// inner loop is the 128 bytes a cycle that shared memory returns to an SM's registers, broadcast or
// not: an 8 x 8 thread tile needs 64 bytes for 64 FFMAs (both limits met at once), a 4 x 4 tile twice
// that. Hence the k-groups: a small CTA tile keeps the large thread tile, and its warps divide k.
#pragma once
#include "common.cuh"

#include <algorithm>

namespace gemm {

enum { EPI_NONE = 0, EPI_SILU = 1, EPI_SILU_BWD = 2 };
enum { GROUP_NONE = 0, GROUP_M = 1, GROUP_K = 2 };

struct Params {
    const void* A;
    const void* B;
    float* C;
    int64_t lda, ldb, ldc;
    int M, N, K;
    const float* bias;      // per output column, nullable
    int accumulate;         // C += result
    const float* res;       // C = res + result, rows and pitch of C; nullable
    // optional maps from a logical "token" row to a memory row (int32), nullable:
    //   a_idx: rows of A's memory layout; b_idx: rows of B's memory layout (TN only);
    //   c_idx: rows of C.
    const int32_t* a_idx;
    const int32_t* b_idx;
    const int32_t* c_idx;
    // grouping (hash-MoE experts): offsets[n_groups+1] are row ranges in the permuted order.
    //   GROUP_M: group g owns logical rows [offsets[g], offsets[g+1]) of A and C (M varies).
    //   GROUP_K: group g owns memory rows  [offsets[g], offsets[g+1]) of A and B (K varies).
    // The operand that is not token-indexed moves by *_gstride elements per group.
    const int32_t* offsets;
    int n_groups;
    int group_dim;
    int64_t b_gstride, c_gstride, bias_gstride;
    // epilogue: EPI_SILU writes the pre-activation to C and silu to C2 (type TC2);
    // EPI_SILU_BWD multiplies by silu'(aux[row][col]) (aux rows follow the logical row).
    int epi;
    const float* aux;
    int64_t ldaux;
    void* C2;
    int64_t ldc2;
    int mode;               // ASCA_NN / ASCA_TN / ASCA_NT
    int64_t total_rows;     // grouped: token rows over all groups (bounds the grid and the k range)
    // a second operand pair with its own k, added to the same result (ungrouped, no maps)
    const void* A2;
    const void* B2;
    int64_t lda2, ldb2;
    int K2;
    // TN: the column sums of B (a bias gradient) beside the product; with A null, the sums alone (f32, K rows of B)
    float* colsum;
    int64_t colsum_gstride;
};

constexpr int MAX_PROBLEMS = 4;
constexpr int THREADS = 256;

struct Multi {
    Params p[MAX_PROBLEMS];
    int split[MAX_PROBLEMS];      // CTAs that share a tile's k: 1, 2, 4 or 8, at most the launch's cluster size
    int cta0[MAX_PROBLEMS + 1];   // first CTA of each problem (a multiple of the cluster size: a cluster works on one problem)
    int n;
};

template <int BM_, int BN_, int BK_, int TM_, int TN_, int KG_, int STAGES_>
struct Cfg {
    static constexpr int BM = BM_, BN = BN_, BK = BK_, TM = TM_, TN = TN_, KG = KG_, STAGES = STAGES_;
    static constexpr int THR_M = BM / TM, THR_N = BN / TN;
    static_assert(THR_M * THR_N * KG == THREADS && TM % 4 == 0 && TN % 4 == 0 && BK % (4 * KG) == 0, "tile shape");
    // row pitches: 16-byte aligned, 8 consecutive rows start in 8 different bank groups
    static constexpr bool TRANSPOSE = KG == 1;   // operands along k are transposed on their way into shared memory
    static constexpr int A_FLOATS = BM * (BK + 4) > BK * (BM + 8) ? BM * (BK + 4) : BK * (BM + 8);
    static constexpr int B_FLOATS = BN * (BK + 4) > BK * (BN + 8) ? BN * (BK + 4) : BK * (BN + 8);
    static constexpr int STAGE_FLOATS = A_FLOATS + B_FLOATS;
    static constexpr int RED_FLOATS = KG * (BM * BN + BN);   // partial tiles + column sums, over the (finished) stages
    static constexpr int SMEM_FLOATS = STAGES * STAGE_FLOATS > RED_FLOATS ? STAGES * STAGE_FLOATS : RED_FLOATS;
    static constexpr size_t SMEM = (size_t)SMEM_FLOATS * 4;
};
using CfgL = Cfg<128, 128, 16, 8, 8, 1, 3>;
using CfgM = Cfg<64, 64, 32, 8, 8, 4, 3>;
using CfgS = Cfg<32, 32, 64, 4, 8, 8, 3>;

__device__ __forceinline__ float silu_f(float x) { return x / (1.0f + expf(-x)); }
__device__ __forceinline__ float silu_grad_f(float p) {
    float sg = 1.0f / (1.0f + expf(-p));
    return sg * (1.0f + p * (1.0f - sg));
}

// two independent FFMAs in one instruction (the rounding of two scalar ones, half the issue slots)
__device__ __forceinline__ void fma2(float2& d, const float2& a, const float2& b) {
    asm("fma.rn.f32x2 %0, %1, %2, %0;"
        : "+l"(reinterpret_cast<uint64_t&>(d))
        : "l"(reinterpret_cast<const uint64_t&>(a)), "l"(reinterpret_cast<const uint64_t&>(b)));
}

// Four elements of a row into shared memory, the first `valid` of them from p and zeros behind.
__device__ __forceinline__ void stage4(float* dst, const float* p, bool vec_ok, int valid) {
    const uint32_t s = (uint32_t)__cvta_generic_to_shared(dst);
    if (vec_ok) {
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(s), "l"(p), "r"(valid * 4) : "memory");
    } else {
#pragma unroll
        for (int j = 0; j < 4; ++j)
            asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(s + 4 * j), "l"(j < valid ? p + j : p), "r"(j < valid ? 4 : 0)
                         : "memory");
    }
}
__device__ __forceinline__ void stage4(float* dst, const __nv_bfloat16* p, bool vec_ok, int valid) {
    float4 v = make_float4(0, 0, 0, 0);
    if (vec_ok && valid == 4) {
        const uint2 raw = *reinterpret_cast<const uint2*>(p);
        const __nv_bfloat162 a = *reinterpret_cast<const __nv_bfloat162*>(&raw.x), b = *reinterpret_cast<const __nv_bfloat162*>(&raw.y);
        v = make_float4(__low2float(a), __high2float(a), __low2float(b), __high2float(b));
    } else {
        if (valid > 0) v.x = __bfloat162float(p[0]);
        if (valid > 1) v.y = __bfloat162float(p[1]);
        if (valid > 2) v.z = __bfloat162float(p[2]);
        if (valid > 3) v.w = __bfloat162float(p[3]);
    }
    *reinterpret_cast<float4*>(dst) = v;
}

__device__ __forceinline__ void stage1(float* dst, const float* p, bool valid) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(p), "r"(valid ? 4 : 0)
                 : "memory");
}
__device__ __forceinline__ void stage1(float* dst, const __nv_bfloat16* p, bool valid) { *dst = valid ? __bfloat162float(*p) : 0.0f; }

// One operand's slabs on their way into shared memory, laid out as in memory: [row][k] where k is contiguous there (ALONG_K;
// row = output row or column of the tile), [k][row] otherwise. A thread copies CH runs of four elements per slab.
template <typename T, int ROWS, int BK, bool ALONG_K>
struct Stager {
    static constexpr int LD = (ALONG_K ? BK : ROWS) + 4, CH = ROWS * BK / 4 / THREADS;
    static constexpr int RUNS = (ALONG_K ? BK : ROWS) / 4, STEP = THREADS / RUNS;   // runs per memory row; rows covered by one pass
    static_assert(CH >= 1 && THREADS % RUNS == 0, "tile shape");
    const T* ptr[ALONG_K ? CH : 1];   // ALONG_K: this thread's runs at k = 0 of the slab sequence; else its run of memory row 0
    const int32_t* idx;               // !ALONG_K: memory row of each k, from the group's first row
    int64_t ld;
    int K, next_row[ALONG_K ? 1 : CH];
    int valid_rows;                   // !ALONG_K: elements of the run that exist; ALONG_K: bit c: row of run c exists
    bool vec;

    // row0: first tile row; n: rows that exist; idx_base: logical position of the first row (ALONG_K) or of k = 0
    __device__ __forceinline__ void init(const T* b, int64_t ld_, int row0, int n, int K_, const int32_t* idx_, int64_t idx_base) {
        const int tid = threadIdx.x;
        K = K_;
        vec = (ld_ & 3) == 0 && (reinterpret_cast<uintptr_t>(b) & (sizeof(T) * 4 - 1)) == 0;
        if (ALONG_K) {
            valid_rows = 0;
#pragma unroll
            for (int c = 0; c < CH; ++c) {
                const int r = row0 + tid / RUNS + c * STEP;
                if (r < n) valid_rows |= 1 << c;
                ptr[c] = b + (r < n ? (idx_ ? (int64_t)idx_[idx_base + r] : idx_base + r) : 0) * ld_;
            }
        } else {
            const int r = row0 + (tid % RUNS) * 4;
            valid_rows = max(0, min(4, n - r));
            ptr[0] = b + (valid_rows ? r : 0) + (idx_ ? 0 : idx_base * ld_);
            idx = idx_ ? idx_ + idx_base : nullptr;
            ld = ld_;
        }
    }
    // !ALONG_K with a row map: the memory rows of the slab starting at k0 (asked for a slab ahead of the copy)
    __device__ __forceinline__ void look_up(int k0) {
        if (!ALONG_K && idx) {
#pragma unroll
            for (int c = 0; c < CH; ++c) {
                const int k = k0 + (int)threadIdx.x / RUNS + c * STEP;
                next_row[ALONG_K ? 0 : c] = k < K ? idx[k] : 0;
            }
        }
    }
    __device__ __forceinline__ void put(float* dst, int k0) {
        const int tid = threadIdx.x, first = tid / RUNS, run = tid % RUNS;
        float* d = dst + first * LD + run * 4;
        if (ALONG_K) {
            const int k = k0 + run * 4, left = K - k, valid = left < 0 ? 0 : (left > 4 ? 4 : left), at = left > 0 ? k : 0;
#pragma unroll
            for (int c = 0; c < CH; ++c) stage4(d + c * STEP * LD, ptr[c] + at, vec, (valid_rows >> c & 1) ? valid : 0);
        } else {
#pragma unroll
            for (int c = 0; c < CH; ++c) {
                const int k = k0 + first + c * STEP;
                const bool ok = k < K;
                stage4(d + c * STEP * LD, ptr[0] + (int64_t)(ok ? (idx ? next_row[ALONG_K ? 0 : c] : k) : 0) * ld, vec, ok ? valid_rows : 0);
            }
        }
    }
};

template <typename TC2>
__device__ __forceinline__ void emit(const Params& p, float* crow, const float* bias, int64_t lr, int n, float v) {
    if (bias) v += bias[n];
    if (p.epi == EPI_SILU_BWD) v *= silu_grad_f(p.aux[lr * p.ldaux + n]);
    if (p.accumulate) v += crow[n];
    if (p.res) v += p.res[crow - p.C + n];
    crow[n] = v;
    if (p.epi == EPI_SILU) reinterpret_cast<TC2*>(p.C2)[lr * p.ldc2 + n] = from_f32<TC2>(silu_f(v));
}

// four columns n .. n + 3 of one row, 16-byte accesses (row pitches and pointers allow them: vec4_ok)
template <typename TC2>
__device__ __forceinline__ bool vec4_ok(const Params& p, const float* C, const float* bias) {
    int64_t pitch = p.ldc;
    uintptr_t at = reinterpret_cast<uintptr_t>(C) | reinterpret_cast<uintptr_t>(bias) | reinterpret_cast<uintptr_t>(p.res);
    if (p.epi == EPI_SILU_BWD) pitch |= p.ldaux, at |= reinterpret_cast<uintptr_t>(p.aux);
    if (p.epi == EPI_SILU) pitch |= p.ldc2, at |= reinterpret_cast<uintptr_t>(p.C2);
    return ((pitch & 3) | (at & 15)) == 0;
}
template <typename TC2>
__device__ __forceinline__ void emit4(const Params& p, float* crow, const float* bias, int64_t lr, int n, float4 v) {
    if (bias) {
        const float4 b = *reinterpret_cast<const float4*>(bias + n);
        v.x += b.x; v.y += b.y; v.z += b.z; v.w += b.w;
    }
    if (p.epi == EPI_SILU_BWD) {
        const float4 x = *reinterpret_cast<const float4*>(p.aux + lr * p.ldaux + n);
        v.x *= silu_grad_f(x.x); v.y *= silu_grad_f(x.y); v.z *= silu_grad_f(x.z); v.w *= silu_grad_f(x.w);
    }
    if (p.accumulate) {
        const float4 c = *reinterpret_cast<const float4*>(crow + n);
        v.x += c.x; v.y += c.y; v.z += c.z; v.w += c.w;
    }
    if (p.res) {
        const float4 c = *reinterpret_cast<const float4*>(p.res + (crow - p.C) + n);
        v.x += c.x; v.y += c.y; v.z += c.z; v.w += c.w;
    }
    *reinterpret_cast<float4*>(crow + n) = v;
    if (p.epi == EPI_SILU) {
        TC2* c2 = reinterpret_cast<TC2*>(p.C2) + lr * p.ldc2 + n;
        const float s[4] = {silu_f(v.x), silu_f(v.y), silu_f(v.z), silu_f(v.w)};
        if (sizeof(TC2) == 4) {
            *reinterpret_cast<float4*>(c2) = make_float4(s[0], s[1], s[2], s[3]);
        } else {
#pragma unroll
            for (int j = 0; j < 4; ++j) c2[j] = from_f32<TC2>(s[j]);
        }
    }
}

// Column sums alone: 8 columns (one sector) of all rows per CTA, 32 rows a pass, 8 passes in flight, a fixed tree.
__device__ __forceinline__ void colsum_tile(const Params& p, int tile, float* smem) {
    const float* B = reinterpret_cast<const float*>(p.B);
    const int tid = threadIdx.x, c = tile * 8 + (tid & 7), w = tid >> 3;
    float acc = 0.0f;
    if (c < p.N) {
        int r = w;
        for (; r + 224 < p.K; r += 256) {
            float x[8];
#pragma unroll
            for (int i = 0; i < 8; ++i) x[i] = B[(int64_t)(r + 32 * i) * p.ldb + c];
            acc += ((x[0] + x[1]) + (x[2] + x[3])) + ((x[4] + x[5]) + (x[6] + x[7]));
        }
        for (; r < p.K; r += 32) acc += B[(int64_t)r * p.ldb + c];
    }
    smem[w * 8 + (tid & 7)] = acc;
    __syncthreads();
    if (tid < 8 && c < p.N) {
        float t = 0.0f;
#pragma unroll
        for (int i = 0; i < 32; ++i) t += smem[i * 8 + tid];
        p.colsum[c] = p.accumulate ? p.colsum[c] + t : t;
    }
}

// Values of T rows at k of a staged operand.
template <int T, bool ALONG_K, class Of>
__device__ __forceinline__ void read_rows(const float* s, int ld, int k, const Of& of, float (&v)[T]) {
    if (ALONG_K) {
#pragma unroll
        for (int i = 0; i < T; ++i) v[i] = s[of(i) * ld + k];
    } else {
#pragma unroll
        for (int i = 0; i < T; i += 4) {
            const float4 x = *reinterpret_cast<const float4*>(s + k * ld + of(i));
            v[i] = x.x; v[i + 1] = x.y; v[i + 2] = x.z; v[i + 3] = x.w;
        }
    }
}

// The same for an operand that is contiguous along k, transposed to [k][row] by the copy: a warp takes 8 rows x 4 k at a time
// (pitch ROWS + 8: 32 different banks). The largest tile shape reads its operands along the rows in every form, since
// reading 16 values one by one costs it more issue slots than the 4-byte copies do.
template <typename T, int ROWS, int BK>
struct TransposingStager {
    static constexpr int CH = ROWS * BK / THREADS, KB = BK / 4, WR = 8 / KB * 8;
    const T* base;
    int64_t ld;
    int K, kl, row[CH];   // memory rows of this thread's elements, -1: none
    __device__ __forceinline__ void init(const T* b, int64_t ld_, int row0, int n, int K_, const int32_t* idx, int64_t idx_base) {
        const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
        base = b; ld = ld_; K = K_;
        kl = (w % KB) * 4 + (lane >> 3);
#pragma unroll
        for (int c = 0; c < CH; ++c) {
            const int r = row0 + w / KB * 8 + (lane & 7) + c * WR;
            row[c] = r < n ? (int)(idx ? (int64_t)idx[idx_base + r] : idx_base + r) : -1;
        }
    }
    __device__ __forceinline__ void look_up(int) {}
    __device__ __forceinline__ void put(float* dst, int k0) {
        const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
        float* d = dst + kl * (ROWS + 8) + w / KB * 8 + (lane & 7);
        const T* p = base + (k0 + kl < K ? k0 + kl : 0);
#pragma unroll
        for (int c = 0; c < CH; ++c) stage1(d + c * WR, p + (int64_t)max(row[c], 0) * ld, row[c] >= 0 && k0 + kl < K);
    }
};
template <class C, typename T, int ROWS, bool ALONG_K, bool TR = C::TRANSPOSE && ALONG_K>
struct StagerOf {
    using type = Stager<T, ROWS, C::BK, ALONG_K>;
};
template <class C, typename T, int ROWS, bool ALONG_K>
struct StagerOf<C, T, ROWS, ALONG_K, true> {
    using type = TransposingStager<T, ROWS, C::BK>;
};

__device__ __forceinline__ void cluster_sync() {
    asm volatile("barrier.cluster.arrive.aligned;\nbarrier.cluster.wait.aligned;" ::: "memory");
}

// What the end of a tile needs to know.
struct Out {
    float* C;
    const float* bias;
    float* colsum;   // null: none wanted
    int64_t m_base;
    int m0, n0, M, N;
};

// The product of a tile up to its partial sums in shared memory; true where finish() is left to do. The three operand forms of a mixed
// launch are three copies of this in one kernel, run side by side: what is the same for all of them is kept out (finish) and the
// staging code is there once, not once per prologue stage (12.7M-parameter step 2552 -> 2515 us, expert layer of 4000 tokens, 256 -> 1024,
// 519 -> 495). Rolling up the loop over k as well cost 4 %.
template <class C, int MODE, typename TA, typename TB, typename TC2>
__device__ __forceinline__ bool tile_product(const Params& p, int tile, bool live, int rank, int split, float* smem, int* sh_group, Out& out) {
    constexpr int BM = C::BM, BN = C::BN, BK = C::BK, TM = C::TM, TN = C::TN, KG = C::KG, STAGES = C::STAGES;
    constexpr bool A_KC = !C::TRANSPOSE && MODE != ASCA_TN, B_KC = !C::TRANSPOSE && MODE == ASCA_NT;   // along k in shared memory
    constexpr int LDA = A_KC ? BK + 4 : BM + (C::TRANSPOSE && MODE != ASCA_TN ? 8 : 4),
                  LDB = B_KC ? BK + 4 : BN + (C::TRANSPOSE && MODE == ASCA_NT ? 8 : 4);

    int M = p.M, N = p.N, K = p.K;
    const TA* A = reinterpret_cast<const TA*>(p.A);
    const TB* B = reinterpret_cast<const TB*>(p.B);
    float* Cp = p.C;
    const float* bias = p.bias;
    float* colsum = p.colsum;
    const int tiles_n = (N + BN - 1) / BN, tid = threadIdx.x;
    int64_t row_base = 0;   // logical row offset of this group (GROUP_M) or its k offset (GROUP_K)
    int g = 0, t = tile;
    if (p.group_dim != GROUP_NONE && live) {
        // locate (group, tile): warp 0 scans the per-group tile counts
        if (tid < 32) {
            const int lane = tid;
            int found_g = -1, found_t = 0, base = 0;
            for (int g0 = 0; g0 < p.n_groups && found_g < 0; g0 += 32) {
                const int gi = g0 + lane;
                int cnt = 0;
                if (gi < p.n_groups) {
                    const int n_g = p.offsets[gi + 1] - p.offsets[gi];
                    cnt = p.group_dim == GROUP_M ? ((n_g + BM - 1) / BM) * tiles_n : ((M + BM - 1) / BM) * tiles_n;
                }
                int inc = cnt;
#pragma unroll
                for (int o = 1; o < 32; o <<= 1) {
                    const int x = __shfl_up_sync(0xffffffffu, inc, o);
                    if (lane >= o) inc += x;
                }
                const int start = base + inc - cnt;
                const unsigned m = __ballot_sync(0xffffffffu, tile >= start && tile < start + cnt);
                if (m) {
                    const int src = __ffs(m) - 1;
                    found_g = __shfl_sync(0xffffffffu, gi, src);
                    found_t = tile - __shfl_sync(0xffffffffu, start, src);
                }
                base += __shfl_sync(0xffffffffu, inc, 31);
            }
            if (lane == 0) {
                sh_group[0] = found_g;
                sh_group[1] = found_t;
            }
        }
        __syncthreads();
        g = sh_group[0];
        t = sh_group[1];
        live = g >= 0;       // else a surplus tile of the upper-bound grid
    }
    if (!live) {
        if (split > 1) {   // (other tiles of the cluster are waiting for it)
            cluster_sync();
            cluster_sync();
        }
        return false;
    }
    if (p.group_dim != GROUP_NONE) {
        const int lo = p.offsets[g], n_g = p.offsets[g + 1] - lo;
        row_base = lo;
        if (p.group_dim == GROUP_M) {
            M = n_g;
            B += (int64_t)g * p.b_gstride;
        } else {
            K = n_g;
            Cp += (int64_t)g * p.c_gstride;
            if (colsum) colsum += (int64_t)g * p.colsum_gstride;
        }
        if (bias) bias += (int64_t)g * p.bias_gstride;
    }
    const int tile_n = t % tiles_n, tile_m = t / tiles_n;
    const int m0 = tile_m * BM, n0 = tile_n * BN;
    const int64_t m_base = p.group_dim == GROUP_M ? row_base : 0, k_base = p.group_dim == GROUP_K ? row_base : 0;
    const bool want_cs = MODE == ASCA_TN && colsum && tile_m == 0;

    typename StagerOf<C, TA, BM, MODE != ASCA_TN>::type sa;
    typename StagerOf<C, TB, BN, MODE == ASCA_NT>::type sb;
    sa.init(A, p.lda, m0, M, K, p.a_idx, MODE != ASCA_TN ? m_base : k_base);
    sb.init(B, p.ldb, n0, N, K, MODE == ASCA_TN ? p.b_idx : nullptr, MODE == ASCA_TN ? k_base : 0);
    const int slabs1 = (K + BK - 1) / BK, slabs = slabs1 + (p.K2 + BK - 1) / BK;
    const int s_lo = (int)((int64_t)slabs * rank / split), s_hi = (int)((int64_t)slabs * (rank + 1) / split);
    int staged = s_lo;   // next slab to stage
    bool second = false;   // the slabs come from the second operand pair
    sa.look_up(s_lo * BK);
    sb.look_up(s_lo * BK);
    auto stage_next = [&]() {
        if (staged < s_hi) {
            if (p.K2 > 0 && staged >= slabs1 && !second) {
                sa.init(reinterpret_cast<const TA*>(p.A2), p.lda2, m0, M, p.K2, nullptr, 0);
                sb.init(reinterpret_cast<const TB*>(p.B2), p.ldb2, n0, N, p.K2, nullptr, 0);
                second = true;
            }
            const int k0 = (staged >= slabs1 ? staged - slabs1 : staged) * BK;
            float* As = smem + ((staged - s_lo) % STAGES) * C::STAGE_FLOATS;
            sa.put(As, k0);
            sb.put(As + C::A_FLOATS, k0);
            ++staged;
            sa.look_up(k0 + BK);
            sb.look_up(k0 + BK);
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };

    const int kg = tid / (C::THR_M * C::THR_N), tt = tid % (C::THR_M * C::THR_N);
    const int tn = tt % C::THR_N, tm = tt / C::THR_N;
    // this thread's output rows and columns: interleaved where the operand is read along k (the lanes of a phase then read
    // rows a pitch apart: no bank conflict), groups of four where it is read along the row
    auto m_of = [&](int i) { return A_KC ? tm + C::THR_M * i : (i >> 2) * (BM * 4 / TM) + tm * 4 + (i & 3); };
    auto n_of = [&](int j) { return B_KC ? tn + C::THR_N * j : (j >> 2) * (BN * 4 / TN) + tn * 4 + (j & 3); };

    float2 acc[TM][TN / 2];   // columns (j, j + 1)
#pragma unroll
    for (int i = 0; i < TM; ++i)
#pragma unroll
        for (int j = 0; j < TN / 2; ++j) acc[i][j] = make_float2(0.0f, 0.0f);
    float cs[TN];
#pragma unroll
    for (int j = 0; j < TN; ++j) cs[j] = 0.0f;

#pragma unroll 1
    for (int slab = s_lo - (STAGES - 1); slab < s_hi; ++slab) {
        if (slab >= s_lo) {
            asm volatile("cp.async.wait_group %0;" ::"n"(STAGES - 2) : "memory");
            __syncthreads();   // the slab has landed for every thread, and the stage filled next is no longer being read
        }
        stage_next();
        if (slab < s_lo) continue;   // (the first stages)
        const float* As = smem + ((slab - s_lo) % STAGES) * C::STAGE_FLOATS;
        const float* Bs = As + C::A_FLOATS;
        // the operands of the next k are read while this one is multiplied; the k-groups take turns four k wide
        float a[2][TM], b[2][TN];
        auto read = [&](int kk) {
            const int k = ((kk >> 2) * KG + kg) * 4 + (kk & 3);
            read_rows<TM, A_KC>(As, LDA, k, m_of, a[kk & 1]);
            read_rows<TN, B_KC>(Bs, LDB, k, n_of, b[kk & 1]);
        };
        read(0);
#pragma unroll
        for (int kk = 0; kk < BK / KG; ++kk) {
            if (kk + 1 < BK / KG) read(kk + 1);
            if (MODE == ASCA_TN && want_cs) {
#pragma unroll
                for (int j = 0; j < TN; ++j) cs[j] += b[kk & 1][j];
            }
#pragma unroll
            for (int i = 0; i < TM; ++i)
#pragma unroll
                for (int j = 0; j < TN / 2; ++j) {
                    const float2 bb = make_float2(b[kk & 1][2 * j], b[kk & 1][2 * j + 1]);
                    if (B_KC) {   // (the two columns come from separate loads: pairing them would cost moves)
                        acc[i][j].x = fmaf(a[kk & 1][i], bb.x, acc[i][j].x);
                        acc[i][j].y = fmaf(a[kk & 1][i], bb.y, acc[i][j].y);
                    } else {
                        fma2(acc[i][j], make_float2(a[kk & 1][i], a[kk & 1][i]), bb);
                    }
                }
        }
    }
    auto value = [&](int i, int j) -> float { return (j & 1) ? acc[i][j >> 1].y : acc[i][j >> 1].x; };

    if (KG == 1 && split == 1 && !want_cs) {   // straight from the registers
        const bool vec = vec4_ok<TC2>(p, Cp, bias);
#pragma unroll
        for (int i = 0; i < TM; ++i) {
            const int m = m0 + m_of(i);
            if (m >= M) continue;
            const int64_t lr = m_base + m;
            float* crow = Cp + (p.c_idx ? (int64_t)p.c_idx[lr] : lr) * p.ldc;
            if (!B_KC && vec) {
#pragma unroll
                for (int j = 0; j < TN; j += 4)
                    if (n0 + n_of(j) + 3 < N)
                        emit4<TC2>(p, crow, bias, lr, n0 + n_of(j), make_float4(value(i, j), value(i, j + 1), value(i, j + 2), value(i, j + 3)));
                    else
                        for (int jj = 0; jj < 3; ++jj)
                            if (n0 + n_of(j) + jj < N) emit<TC2>(p, crow, bias, lr, n0 + n_of(j) + jj, jj == 0 ? value(i, j) : jj == 1 ? value(i, j + 1) : value(i, j + 2));
                continue;
            }
#pragma unroll
            for (int j = 0; j < TN; ++j) {
                const int n = n0 + n_of(j);
                if (n < N) emit<TC2>(p, crow, bias, lr, n, value(i, j));
            }
        }
        return false;
    }
    // partial tiles to shared memory, added over the cluster's CTAs and their k-groups in order
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    __syncthreads();   // the stages are free
    float* red = smem;
    float* red_cs = smem + KG * BM * BN;
#pragma unroll
    for (int i = 0; i < TM; ++i) {
        float* row = red + kg * BM * BN + m_of(i) * BN;
        if (B_KC) {
#pragma unroll
            for (int j = 0; j < TN; ++j) row[n_of(j)] = value(i, j);
        } else {
#pragma unroll
            for (int j = 0; j < TN; j += 4)
                *reinterpret_cast<float4*>(row + n_of(j)) = make_float4(value(i, j), value(i, j + 1), value(i, j + 2), value(i, j + 3));
        }
    }
    if (want_cs && tm == 0) {
#pragma unroll
        for (int j = 0; j < TN; ++j) red_cs[kg * BN + n_of(j)] = cs[j];
    }
    out.C = Cp; out.bias = bias; out.colsum = want_cs ? colsum : nullptr;
    out.m_base = m_base; out.m0 = m0; out.n0 = n0; out.M = M; out.N = N;
    return true;
}

// The partial tiles added over the cluster's CTAs and their k-groups, and stored.
template <class C, typename TC2>
__device__ __forceinline__ void finish(const Params& p, const Out& out, int rank, int split, float* smem) {
    constexpr int BM = C::BM, BN = C::BN, KG = C::KG;
    const int tid = threadIdx.x, m0 = out.m0, n0 = out.n0, M = out.M, N = out.N;
    const int64_t m_base = out.m_base;
    float* Cp = out.C;
    const float* bias = out.bias;
    const bool vec = vec4_ok<TC2>(p, Cp, bias);
    const uint32_t mine = (uint32_t)__cvta_generic_to_shared(smem);
    uint32_t base;   // first CTA of this tile in its cluster: itself where the tile is not split, whatever the launch's clusters
    asm("mov.u32 %0, %%cluster_ctarank;" : "=r"(base));
    base = base / split * split;
    if (split > 1) cluster_sync();
    else __syncthreads();
    // v + the KG values at off, off + stride, ... (floats) of every CTA, in order
    auto add_all = [&](float4 v, int off, int stride) -> float4 {
        for (int r = 0; r < split; ++r) {
            float4 x[KG];
            uint32_t at;
            asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(at) : "r"(mine), "r"(base + r));
#pragma unroll
            for (int q = 0; q < KG; ++q)
                asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];"
                             : "=f"(x[q].x), "=f"(x[q].y), "=f"(x[q].z), "=f"(x[q].w) : "r"(at + (uint32_t)(off + q * stride) * 4));
#pragma unroll
            for (int q = 0; q < KG; ++q) v.x += x[q].x, v.y += x[q].y, v.z += x[q].z, v.w += x[q].w;
        }
        return v;
    };
    const int rows = BM / split;   // this CTA finishes its share of the tile's rows
    for (int e = tid; e < rows * BN / 4; e += THREADS) {
        const int mi = rank * rows + e / (BN / 4), ni = e % (BN / 4) * 4, m = m0 + mi, n = n0 + ni;
        if (m >= M || n >= N) continue;
        const float4 v = add_all(make_float4(0.0f, 0.0f, 0.0f, 0.0f), mi * BN + ni, BM * BN);
        const int64_t lr = m_base + m;
        float* crow = Cp + (p.c_idx ? (int64_t)p.c_idx[lr] : lr) * p.ldc;
        if (vec && n + 3 < N) {
            emit4<TC2>(p, crow, bias, lr, n, v);
        } else {
            emit<TC2>(p, crow, bias, lr, n, v.x);
            if (n + 1 < N) emit<TC2>(p, crow, bias, lr, n + 1, v.y);
            if (n + 2 < N) emit<TC2>(p, crow, bias, lr, n + 2, v.z);
            if (n + 3 < N) emit<TC2>(p, crow, bias, lr, n + 3, v.w);
        }
    }
    if (out.colsum && rank == 0 && tid < BN / 4) {
        const float4 v = add_all(make_float4(0.0f, 0.0f, 0.0f, 0.0f), KG * BM * BN + tid * 4, BN);
        const float x[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
        for (int j = 0; j < 4; ++j)
            if (n0 + tid * 4 + j < N) {
                float* o = out.colsum + n0 + tid * 4 + j;
                *o = p.accumulate ? *o + x[j] : x[j];
            }
    }
    if (split > 1) cluster_sync();   // peers may still read
}

// MODE: the operand form of every problem of the launch, or ANY_MODE (mixed forms; costs registers).
constexpr int ANY_MODE = -1;
template <class C, int MODE, typename TA, typename TB, typename TC2>
__global__ void __launch_bounds__(THREADS, 2) gemm_kernel(const __grid_constant__ Multi mp) {
    extern __shared__ __align__(16) float smem[];
    __shared__ int sh_group[2];
    int i = 0;
#pragma unroll
    for (int q = 1; q < MAX_PROBLEMS; ++q)
        if (q < mp.n && (int)blockIdx.x >= mp.cta0[q]) i = q;
    const Params& p = mp.p[i];
    const int split = mp.split[i], at = blockIdx.x - mp.cta0[i], t = at / split, rank = at % split;
    const int mode = MODE == ANY_MODE ? p.mode : MODE;
    if (mode == ASCA_TN && p.A == nullptr) {
        colsum_tile(p, t, smem);   // (split 1; tiles past the last column do nothing)
        return;
    }
    const bool live = p.group_dim != GROUP_NONE || t < ((p.M + C::BM - 1) / C::BM) * ((p.N + C::BN - 1) / C::BN);
    Out out;
    bool left;
    if (mode == ASCA_NN) left = tile_product<C, ASCA_NN, TA, TB, TC2>(p, t, live, rank, split, smem, sh_group, out);
    else if (mode == ASCA_TN) left = tile_product<C, ASCA_TN, TA, TB, TC2>(p, t, live, rank, split, smem, sh_group, out);
    else left = tile_product<C, ASCA_NT, TA, TB, TC2>(p, t, live, rank, split, smem, sh_group, out);
    if (left) finish<C, TC2>(p, out, rank, split, smem);
}

// Tiles of one problem (upper bound for GROUP_M: every group can add one ragged tile).
template <class C>
inline int64_t tiles_of(const Params& p) {
    if (p.mode == ASCA_TN && !p.A) return (p.N + 7) / 8;
    const int64_t tn = (p.N + C::BN - 1) / C::BN, tm = std::max<int64_t>(1, (p.M + C::BM - 1) / C::BM);
    if (p.group_dim == GROUP_NONE) return tm * tn;
    if (p.group_dim == GROUP_M) return (p.total_rows / C::BM + p.n_groups) * tn;
    return (int64_t)p.n_groups * tm * tn;
}

template <class C, int MODE, typename TA, typename TB, typename TC2>
inline cudaError_t launch_mode(asca_ctx* ctx, Multi& m) {
    int64_t ctas = 0;
    int cluster = 1;
    for (int i = 0; i < m.n; ++i) cluster = std::max(cluster, m.split[i]);
    for (int i = 0; i < m.n; ++i) {
        m.cta0[i] = (int)ctas;
        ctas += (tiles_of<C>(m.p[i]) * m.split[i] + cluster - 1) / cluster * cluster;
    }
    m.cta0[m.n] = (int)ctas;
    if (ctas == 0) return cudaSuccess;
    auto kern = gemm_kernel<C, MODE, TA, TB, TC2>;
    if (C::SMEM > 48 * 1024) {
        const cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)C::SMEM);
        if (e != cudaSuccess) return e;
    }
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)ctas);
    cfg.blockDim = dim3(THREADS);
    cfg.dynamicSmemBytes = C::SMEM;
    cfg.stream = ctx->stream;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = (unsigned)cluster;
    at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
    cfg.attrs = at;
    cfg.numAttrs = cluster > 1 ? 1 : 0;
    return cudaLaunchKernelEx(&cfg, kern, (const Multi)m);
}

template <class C, typename TA, typename TB, typename TC2>
inline cudaError_t launch_cfg(asca_ctx* ctx, Multi& m) {
    for (int i = 1; i < m.n; ++i)
        if (m.p[i].mode != m.p[0].mode) return launch_mode<C, ANY_MODE, TA, TB, TC2>(ctx, m);
    if (m.p[0].mode == ASCA_NN) return launch_mode<C, ASCA_NN, TA, TB, TC2>(ctx, m);
    if (m.p[0].mode == ASCA_TN) return launch_mode<C, ASCA_TN, TA, TB, TC2>(ctx, m);
    return launch_mode<C, ASCA_NT, TA, TB, TC2>(ctx, m);
}

// Estimated microseconds of a launch, from the measured time of a slab on an SM (CTAs that share an SM add their slabs: the
// kernel is bound by its own issue, not by latency), of a CTA's prologue and epilogue, and of a launch. Measured on B200,
// back to back in a graph: 64 x 64 tiles 1.0 us a slab (2048 x 576 x 192: 16 us = 28 TFLOP/s; 8192-long
// weight gradients with the k-split 65 us, 272 without), 32 x 32 tiles 0.81 us (2048 x 64 x 64: 3.5 us), 128 x 128 tiles
// 1.6 us (4096^3: 2.7 - 2.9 ms = 47 - 51 TFLOP/s). A k-split pays for the cluster's two barriers and the exchange.
struct Shape {
    double slab, cta, cta_split, launch;
};
// The best estimate for one tile shape; split: how the problems' k is shared out.
template <class C>
inline double estimate(const Multi& m, int n_sm, int max_split, const Shape& c, int (&split)[MAX_PROBLEMS]) {
    double tiles[MAX_PROBLEMS], slabs[MAX_PROBLEMS];
    for (int i = 0; i < m.n; ++i) {
        const Params& p = m.p[i];
        split[i] = 1;
        tiles[i] = slabs[i] = 0.0;
        if (p.mode == ASCA_TN && !p.A) continue;
        const double tn = (p.N + C::BN - 1) / C::BN, groups = p.group_dim == GROUP_NONE ? 1 : p.n_groups;
        const double mean = (double)p.total_rows / groups;   // token rows of a group
        const double tm = p.group_dim == GROUP_M ? mean / C::BM + 0.5 : std::ceil((double)p.M / C::BM);   // (ragged last tiles)
        const double k = (p.group_dim == GROUP_K ? mean : (double)p.K) + p.K2;
        tiles[i] = groups * tm * tn;
        slabs[i] = std::max(1.0, std::ceil(k / C::BK));
    }
    auto time = [&]() {
        double ctas = 0.0, work = 0.0, longest = 0.0;
        for (int i = 0; i < m.n; ++i) {
            const double one = std::max(1.0, slabs[i] / split[i]) * c.slab + (split[i] > 1 ? c.cta_split : c.cta), n = tiles[i] * split[i];
            if (n == 0.0) continue;
            ctas += n;
            work += n * one;
            longest = std::max(longest, one);
        }
        return ctas == 0.0 ? c.launch : c.launch + std::max(longest, std::ceil(ctas / n_sm) * work / ctas);
    };
    // every chain length a split can reach is tried as the bound for all problems (halving the longest one while that helps
    // stops early where two problems are equally long: a 576 x 64 x 2048 gradient beside a short product took 34 us, 16 so)
    double best = 1e300;
    int found[MAX_PROBLEMS] = {};
    for (int i = 0; i < m.n; ++i)
        for (int s = 1; s <= max_split; s *= 2) {
            const double bound = slabs[i] / s;
            for (int j = 0; j < m.n; ++j)
                for (split[j] = 1; split[j] < max_split && slabs[j] / split[j] > bound && slabs[j] >= 2.0 * split[j];) split[j] *= 2;
            const double t = time();
            if (t < best) {
                best = t;
                for (int j = 0; j < m.n; ++j) found[j] = split[j];
            }
        }
    for (int j = 0; j < m.n; ++j) split[j] = found[j];
    return best;
}

// Tile shape of a launch (0: 128, 1: 64, 2: 32 wide); fills in the k-splits.
inline int plan(const asca_ctx* ctx, Multi& m) {
    const int n_sm = ctx->sm_count > 0 ? ctx->sm_count : 148;
    int split[3][MAX_PROBLEMS];
    const double e[3] = {estimate<CfgL>(m, n_sm, 1, {1.6, 7.0, 0.0, 3.3}, split[0]), estimate<CfgM>(m, n_sm, 8, {1.0, 0.8, 3.8, 3.3}, split[1]),
                         estimate<CfgS>(m, n_sm, 8, {0.81, 0.8, 2.3, 2.6}, split[2])};
    const int shape = e[0] < e[1] ? (e[0] < e[2] ? 0 : 2) : (e[1] < e[2] ? 1 : 2);
    for (int i = 0; i < m.n; ++i) m.split[i] = split[shape][i];
    return shape;
}

// One launch of up to MAX_PROBLEMS f32 products.
inline cudaError_t launch_f32(asca_ctx* ctx, Multi& m) {
    const int shape = plan(ctx, m);
    if (shape == 0) return launch_cfg<CfgL, float, float, float>(ctx, m);
    if (shape == 1) return launch_cfg<CfgM, float, float, float>(ctx, m);
    return launch_cfg<CfgS, float, float, float>(ctx, m);
}

// One product with operands of either type. bf16 operands come here only where the tensor-core kernels cannot take the
// shape (odd pitches, few columns), so they have the middle tile shape alone.
template <typename TC2 = float>
inline cudaError_t launch(asca_ctx* ctx, const Params& p, int a_bf16, int b_bf16) {
    Multi m{};
    m.p[0] = p;
    m.n = 1;
    m.split[0] = 1;
    if (!a_bf16 && !b_bf16) return launch_f32(ctx, m);
    if (a_bf16 && b_bf16) return launch_cfg<CfgM, __nv_bfloat16, __nv_bfloat16, TC2>(ctx, m);
    if (a_bf16) return launch_cfg<CfgM, __nv_bfloat16, float, TC2>(ctx, m);
    return launch_cfg<CfgM, float, __nv_bfloat16, TC2>(ctx, m);
}

}  // namespace gemm
