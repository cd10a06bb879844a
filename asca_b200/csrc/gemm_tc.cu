// bf16 GEMM on the 5th-generation tensor cores (tcgen05) for sm_100a.
//
// Persistent: two CTAs per SM work through the 128 x 128 f32 output tiles, each claiming the next unclaimed tile when it
// starts one (KP::dyn_ctr below; a fixed walk t, t + grid, ... with ASCA_GEMM_DYNAMIC=0). Warp roles (192 threads):
//   warp 0      TMA producer: one thread streams 128x64 A and 64x128 B bf16 tiles (128-byte
//               swizzle, plain non-multicast cp.async.bulk.tensor) through a 3-stage ring of
//               mbarriers, running ahead across tile boundaries;
//   warp 1      allocates two accumulator buffers in TMEM, and one thread issues
//               tcgen05.mma (M128 N128 K16, 4 per k-tile) into the buffer of the current tile;
//               tcgen05.commit releases ring slots and hands the finished buffer to the epilogue;
//   warps 2-5   epilogue (2-9 in the pair shape's eight-warp form): tcgen05.ld the accumulator (each warp its 32-lane quarter), 32
//               columns of a row per lane; bias / SiLU / SiLU' / accumulate are applied in registers; f32 output (and an
//               optional bf16 second output), optionally through a row map (the un-permute scatter of the MoE combine). The
//               buffer is released after the last tcgen05.ld, and the main loop of the next tile runs meanwhile in the other.
//
// Operand majorness covers the three modes without any transposed copy: NN = A K-major, B
// MN-major; TN = A MN-major, B MN-major; NT = A K-major, B K-major. Expert grouping: GROUP_M
// tiles the rows of each expert's segment (rows past the segment end are computed and not
// stored); GROUP_K runs the k-loop over an expert's rows and zeroes the ragged last k-tile in
// shared memory before it is multiplied.
//
// Every mbarrier wait is bounded; a wait that runs out raises an error word that the host reads
// back as ASCA_ERR_DEVICE, and the CTA still frees its TMEM and exits.
#include "gemm_tc.cuh"

#include <algorithm>
#include <cstdlib>
#include "tc_common.cuh"

namespace gemm_tc {
namespace {

constexpr int BM = 128, BK = 64;
constexpr int A_BYTES = BM * BK * 2;
// Two tile shapes. 128 x 128: 3-stage ring, 256 TMEM columns, two CTAs per SM (two independent MMA streams keep the
// tensor pipe fed).
// DEEP: a problem of at most one 128 x 128 tile per SM (a decode step's products) runs one CTA per SM with a
// 7-stage ring: its k-loop streams weights that are cold in L2, and three stages do not cover the HBM latency.
// PAIR: a cluster of two CTAs computes 256 x 256 tiles with cta_group::2 instructions (M = 256, N = 256). Each CTA
// loads its own 128 rows of A and its own 128 of the tile's 256 B columns: 32 KiB per k-tile for 4.2 MFLOP on this SM where the
// 128 x 128 tile has 32 KiB per 2.1, so the shared-memory traffic per FLOP, which is what bounds the single-CTA shape, is half of
// its. 7-stage ring, all 512 TMEM columns, one CTA per SM. What bounds its main loop is the round trip of a stage (slot free ->
// load -> barrier -> instruction) against the ring's depth: the odd CTA's loads complete on the even CTA's barrier and the
// ring is as deep as shared memory allows. 65,536 x 4096 x 1024: 400 us, 1375 TFLOP/s (433 us with six stages and the odd CTA's
// loads reported by one of its threads); 32,768 x 6144 x 2048: tensor pipe 76 % busy.
template <int BN, bool DEEP = false, bool PAIR = false, bool EW8 = false> struct Shape {
    static constexpr int STAGES = PAIR || DEEP ? 7 : 3;   // (one fewer where the tile table needs the room)
    static constexpr int B_BYTES = (PAIR ? BN / 2 : BN) * BK * 2;
    static constexpr int STAGE_BYTES = A_BYTES + B_BYTES;
    static constexpr int TMEM_COLS = 2 * BN;      // two accumulator buffers
    static constexpr int CTAS_PER_SM = PAIR || DEEP ? 1 : 2;
    // epilogue warps: one per TMEM lane quarter. EW8 (pair shape): two warps share each quarter and split the 256 columns -- for
    // the row-grouped expert products, whose epilogues (activation, two outputs, row scatter) would otherwise outlast the
    // main loop, and for the fused qkv epilogue (a warp's 128 columns are one head, or two of 64). Plain dense and k-grouped
    // products are faster with four (14,448 x 768 -> 2304: 56 against 68 us).
    static constexpr int EPI_WARPS = (PAIR && EW8) ? 8 : 4;
    // A warp of its own (the k-grouped products run in this shape or on single CTAs) clears what a ragged k-tile holds of the next
    // group's rows as soon as the tile has landed, while the issuer is still at earlier ones: see there
    static constexpr bool RAG_WARP = PAIR && !EW8;
    static constexpr int THREADS = 64 + 32 * EPI_WARPS + (RAG_WARP ? 32 : 0);
    static constexpr size_t SMEM_FIXED = 1024 /*alignment slack*/ + 416 /*barriers, claims, ragged k-tiles*/;   // + stages + tile table
};
constexpr int MAX_GROUPS = 2048, MAX_STAGES = 7;
constexpr int RAG_Q = 8;               // ragged k-tiles under way in a CTA at most: each holds a ring slot until it has been cleared and used
static_assert(RAG_Q >= MAX_STAGES, "every ring slot may hold a ragged k-tile");

struct KP {
    float* C;
    int64_t ldc;
    int M, N, K;
    const float* bias;
    const float* old;                  // added to the product, rows and pitch like C's (C itself where it accumulates); null: nothing
    const int32_t* c_idx;
    const int32_t* offsets;
    int n_groups, group_dim;
    int b_goff_inner, b_goff_outer;
    int64_t c_gstride, bias_gstride;
    int epi;
    const float* aux;
    int64_t ldaux;
    __nv_bfloat16* C2;
    int64_t ldc2;
    int c2_only, c2_mapped;
    __nv_bfloat16 *qkv_q, *qkv_k, *qkv_v;
    float *qkv_qn, *qkv_kn;
    int qkv_d, qkv_dh;
    const uint32_t* ce_targets;
    float* ce_loss;
    float ce_scale;
    // Dynamic tile claims (null: every walker takes tiles walker, walker + n_walkers, ...). With them a walker -- a CTA,
    // or a CTA pair -- takes the next unclaimed tile whenever it starts one, so CTAs that find their SM occupied by
    // another stream's kernels (a collective running beside the step) simply claim fewer tiles instead of holding the
    // launch up with a fixed share. The producer thread of the walker's first CTA claims (atomicAdd) and publishes the
    // claim in a small ring in the shared memory of both CTAs, tagged with its number; every other role reads it from
    // there (through global memory the read took 2,000 of an epilogue's 22,000 cycles a tile).
    int* dyn_ctr;                      // this launch's counter (zero at launch)
    int* dyn_reset;                    // the next launch's counter, zeroed by this launch
    int* err_word;
    uint32_t stages;                   // ring depth: what the shared memory holds beside the tile table, at most MAX_STAGES
};
constexpr int DYN_Q = 16;              // claims a walker's producer can be ahead of its slowest role, with room to spare

// 1 / (1 + 2^(-x log2 e)), in the two approximate instructions whose errors the PTX manual bounds (2^-22 relative for ex2, one unit
// in the last place for rcp): within (|x| + 5) 2^-23 of the sigmoid, and 0 or 1 where 2^(-x log2 e) leaves the range of f32. Its
// results are rounded to bf16 or multiply bf16 products, and an epilogue is bound by its instructions.
__device__ __forceinline__ float sigmoid_f(float x) {
    float e, r;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(e) : "f"(x * -1.4426950408889634f));
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(1.0f + e));
    return r;
}
__device__ __forceinline__ float silu_f(float x) { return x * sigmoid_f(x); }
__device__ __forceinline__ float silu_grad_f(float p) {
    const float sg = sigmoid_f(p);
    return sg * fmaf(p, 1.0f - sg, 1.0f);
}

// Up to 32 columns of a row between global memory and a lane's registers, `n` of them inside the matrix: 32 bytes at once where
// every row starts on a 32-byte boundary (w = 8), else 16 (w = 4), else one element.
__device__ __forceinline__ void load_row(float (&v)[32], const float* p, int n, int w) {
    if (w == 8 && n >= 32) {
#pragma unroll
        for (int j = 0; j < 32; j += 8)
            asm volatile("ld.global.v8.f32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
                         : "=f"(v[j]), "=f"(v[j + 1]), "=f"(v[j + 2]), "=f"(v[j + 3]), "=f"(v[j + 4]), "=f"(v[j + 5]), "=f"(v[j + 6]), "=f"(v[j + 7])
                         : "l"(p + j));
        return;
    }
#pragma unroll
    for (int j = 0; j < 32; j += 4) {
        if (w >= 4 && j + 4 <= n) {
            const float4 t = *reinterpret_cast<const float4*>(p + j);
            v[j] = t.x; v[j + 1] = t.y; v[j + 2] = t.z; v[j + 3] = t.w;
        } else {
#pragma unroll
            for (int i = j; i < j + 4; ++i) v[i] = i < n ? p[i] : 0.0f;
        }
    }
}
__device__ __forceinline__ void store_row(float* p, const float (&v)[32], int n, int w) {
    if (w == 8 && n >= 32) {
#pragma unroll
        for (int j = 0; j < 32; j += 8)
            asm volatile("st.global.v8.f32 [%8], {%0, %1, %2, %3, %4, %5, %6, %7};"
                         ::"f"(v[j]), "f"(v[j + 1]), "f"(v[j + 2]), "f"(v[j + 3]), "f"(v[j + 4]), "f"(v[j + 5]), "f"(v[j + 6]), "f"(v[j + 7]),
                         "l"(p + j)
                         : "memory");
        return;
    }
#pragma unroll
    for (int j = 0; j < 32; j += 4) {
        if (w >= 4 && j + 4 <= n) {
            *reinterpret_cast<float4*>(p + j) = make_float4(v[j], v[j + 1], v[j + 2], v[j + 3]);
        } else {
#pragma unroll
            for (int i = j; i < j + 4; ++i)
                if (i < n) p[i] = v[i];
        }
    }
}
__device__ __forceinline__ void store_row(__nv_bfloat16* p, const float (&v)[32], int n, int w) {
    if (w >= 4 && n >= 32) {
        uint32_t h[16];
#pragma unroll
        for (int j = 0; j < 16; ++j) {
            const __nv_bfloat162 t = __floats2bfloat162_rn(v[2 * j], v[2 * j + 1]);
            h[j] = *reinterpret_cast<const uint32_t*>(&t);
        }
        if (w == 8) {
#pragma unroll
            for (int j = 0; j < 16; j += 8)
                asm volatile("st.global.v8.b32 [%8], {%0, %1, %2, %3, %4, %5, %6, %7};"
                             ::"r"(h[j]), "r"(h[j + 1]), "r"(h[j + 2]), "r"(h[j + 3]), "r"(h[j + 4]), "r"(h[j + 5]), "r"(h[j + 6]), "r"(h[j + 7]),
                             "l"(p + 2 * j)
                             : "memory");
        } else {
#pragma unroll
            for (int j = 0; j < 16; j += 4) *reinterpret_cast<uint4*>(p + 2 * j) = make_uint4(h[j], h[j + 1], h[j + 2], h[j + 3]);
        }
        return;
    }
#pragma unroll
    for (int j = 0; j < 32; ++j)
        if (j < n) p[j] = __float2bfloat16(v[j]);
}

// 32 columns of the rows of two neighbouring lanes: 32-byte pieces are exchanged first, so that a store instruction's lane pairs
// write 64 consecutive bytes. even_row, odd_row: where the even and the odd lane's columns go.
__device__ __forceinline__ void store_row_pair(float* even_row, float* odd_row, const float (&v)[32], bool odd) {
#pragma unroll
    for (int h = 0; h < 32; h += 16) {
        float e[8], o[8];
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            const float a = v[h + j], b = v[h + 8 + j], got = __shfl_xor_sync(0xffffffffu, odd ? a : b, 1);
            e[j] = odd ? got : a;
            o[j] = odd ? b : got;
        }
        const int at = h + (odd ? 8 : 0);
        asm volatile("st.global.v8.f32 [%8], {%0, %1, %2, %3, %4, %5, %6, %7};"
                     ::"f"(e[0]), "f"(e[1]), "f"(e[2]), "f"(e[3]), "f"(e[4]), "f"(e[5]), "f"(e[6]), "f"(e[7]), "l"(even_row + at)
                     : "memory");
        asm volatile("st.global.v8.f32 [%8], {%0, %1, %2, %3, %4, %5, %6, %7};"
                     ::"f"(o[0]), "f"(o[1]), "f"(o[2]), "f"(o[3]), "f"(o[4]), "f"(o[5]), "f"(o[6]), "f"(o[7]), "l"(odd_row + at)
                     : "memory");
    }
}

template <int MODE, int BN, bool DEEP, bool PAIR, bool EW8>
__global__ void __launch_bounds__(Shape<BN, DEEP, PAIR, EW8>::THREADS, Shape<BN, DEEP, PAIR, EW8>::CTAS_PER_SM) gemm_tc_kernel(const __grid_constant__ CUtensorMap mapA,
                                                             const __grid_constant__ CUtensorMap mapB, const KP p) {
    constexpr bool A_MN = (MODE == ASCA_TN);   // A operand MN-major
    constexpr bool B_MN = (MODE != ASCA_NT);   // B operand MN-major
    using SH = Shape<BN, DEEP, PAIR, EW8>;
    constexpr int STAGE_BYTES = SH::STAGE_BYTES, TMEM_COLS = SH::TMEM_COLS;
    const uint32_t STAGES = p.stages;
    constexpr int TM = PAIR ? 2 * BM : BM;       // rows of an output tile (both CTAs of a pair)
    constexpr int BNL = PAIR ? BN / 2 : BN;      // B columns this CTA loads per tile
    const int rank = PAIR ? (int)tc::cluster_ctarank() : 0;   // 0 = the CTA that issues the pair's instructions
    const int n_walkers = PAIR ? (int)gridDim.x / 2 : (int)gridDim.x, walker = PAIR ? (int)blockIdx.x / 2 : (int)blockIdx.x;
    extern __shared__ uint8_t smem_raw[];
    uint8_t* tiles = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
    uint64_t* full = reinterpret_cast<uint64_t*>(tiles + STAGES * STAGE_BYTES);
    uint64_t* empty = full + MAX_STAGES;
    uint64_t* acc_full = empty + MAX_STAGES; // [2] accumulator buffer written (MMA -> epilogue)
    uint64_t* acc_empty = acc_full + 2;      // [2] accumulator buffer read out (epilogue -> MMA)
    uint64_t* rag_full = acc_empty + 2;      // [stage] PAIR: this CTA's bytes of a ragged k-tile have landed (`full` takes the others)
    uint64_t* rag_clear = rag_full + MAX_STAGES;   // [stage] PAIR, even CTA: both CTAs have cleared the end of their ragged k-tile
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(rag_clear + MAX_STAGES);
    volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
    volatile unsigned long long* claims = reinterpret_cast<volatile unsigned long long*>(tmem_slot + 2);   // [DYN_Q] (number + 1) << 32 | tile
    volatile int* rag_word = reinterpret_cast<volatile int*>(claims + DYN_Q);        // [0] 2 x ragged k-tiles handed over (+ 1: no more come), [1] tiles
    volatile uint16_t* rag_q = reinterpret_cast<volatile uint16_t*>(rag_word + 2);   // [RAG_Q] ring slot << 8 | rows of k that are the expert's
    int* prefix = reinterpret_cast<int*>(const_cast<uint16_t*>(rag_q) + RAG_Q);      // [n_groups + 1] first tile of every group

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int tiles_n = (p.N + BN - 1) / BN;
    const int n_groups = p.group_dim == GROUP_NONE ? 1 : p.n_groups;

    // ---- tile table: group g owns tiles [prefix[g], prefix[g+1]), tile = tile_m * tiles_n + tile_n within it
    if (warp == 1) {
        if (PAIR) tc::tmem_alloc_pair(tmem_slot, TMEM_COLS);
        else tc::tmem_alloc(tmem_slot, TMEM_COLS);
    }
    pdl_wait();   // the group offsets below may be the previous kernel's output
    if (warp == 0) {
        int base = 0;
        for (int g0 = 0; g0 < n_groups; g0 += 32) {
            const int g = g0 + lane;
            int cnt = 0;
            if (g < n_groups) {
                if (p.group_dim == GROUP_M) cnt = ((p.offsets[g + 1] - p.offsets[g] + TM - 1) / TM) * tiles_n;
                else cnt = ((p.M + TM - 1) / TM) * tiles_n;
            }
            int inc = cnt;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const int nb = __shfl_up_sync(0xffffffffu, inc, o);
                if (lane >= o) inc += nb;
            }
            if (g < n_groups) prefix[g] = base + inc - cnt;
            base += __shfl_sync(0xffffffffu, inc, 31);
        }
        if (p.group_dim != GROUP_NONE)   // the group offsets once more in shared memory: locate() runs per tile and role
            for (int g = lane; g <= n_groups; g += 32) prefix[n_groups + 1 + g] = p.offsets[g];
        if (lane == 0) {
            prefix[n_groups] = base;
            *abort_flag = 0;
            for (int i = 0; i < DYN_Q; ++i) claims[i] = 0;
            rag_word[0] = rag_word[1] = 0;
            for (uint32_t s = 0; s < STAGES; ++s) {
                tc::mbar_init(&full[s], 1);
                tc::mbar_init(&empty[s], 1);
                tc::mbar_init(&rag_full[s], 1);
                tc::mbar_init(&rag_clear[s], 2);
            }
            for (int b = 0; b < 2; ++b) {
                tc::mbar_init(&acc_full[b], 1);
                tc::mbar_init(&acc_empty[b], PAIR ? 2 * SH::EPI_WARPS : SH::EPI_WARPS);   // epilogue warps (of both CTAs)
            }
            tc::mbar_fence_init();
            tc::prefetch_tensormap(&mapA);
            tc::prefetch_tensormap(&mapB);
        }
    }
    tc::tcgen05_fence_before();
    __syncthreads();
    if (PAIR) tc::cluster_sync_all();   // the peer's barriers exist before anything is signalled across
    tc::tcgen05_fence_after();
    pdl_launch_dependents();   // after this CTA holds its TMEM: a dependent that becomes resident early cannot take it
    const uint32_t tmem_base = *tmem_slot;
    const int total_tiles = prefix[n_groups];

    // Geometry of one tile; every role walks the same tile sequence blockIdx.x, + gridDim.x, ...
    struct Tile {
        int g, m0, n0, M, num_k, K, row_base_m, row_base_k, b_in, b_out;
    };
    auto locate = [&](int t) {
        int lo = 0, hi = n_groups - 1;   // last group with prefix[g] <= t
        while (lo < hi) {
            const int mid = (lo + hi + 1) >> 1;
            if (prefix[mid] <= t) lo = mid; else hi = mid - 1;
        }
        Tile x;
        x.g = lo;
        const int in = t - prefix[lo];
        x.m0 = (in / tiles_n) * TM + rank * BM;   // this CTA's 128 rows of the tile
        x.n0 = (in % tiles_n) * BN;
        int seg_lo = 0;
        x.M = p.M;
        x.K = p.K;
        if (p.group_dim != GROUP_NONE) {
            seg_lo = prefix[n_groups + 1 + lo];
            const int n_g = prefix[n_groups + 2 + lo] - seg_lo;
            if (p.group_dim == GROUP_M) x.M = n_g; else x.K = n_g;
        }
        x.num_k = (x.K + BK - 1) / BK;
        x.row_base_m = p.group_dim == GROUP_M ? seg_lo : 0;   // added to A/C row coordinates
        x.row_base_k = p.group_dim == GROUP_K ? seg_lo : 0;   // added to k-row coordinates (TN)
        x.b_in = lo * p.b_goff_inner;
        x.b_out = lo * p.b_goff_outer;
        return x;
    };

    // The i-th tile of this walker (-1: none left). claim_tile is for the walker's claiming thread only.
    const bool dyn = p.dyn_ctr != nullptr;
    auto publish_claim = [&](int i, int t) {   // claim i = tile t (-1: none left)
        if (t >= total_tiles) t = -1;
        const unsigned long long v = ((unsigned long long)(uint32_t)(i + 1) << 32) | (uint32_t)t;
        claims[i % DYN_Q] = v;
        if (PAIR)
            asm volatile("st.relaxed.cluster.shared::cluster.u64 [%0], %1;"
                         ::"r"(tc::mapa_u32(tc::smem_u32(const_cast<unsigned long long*>(claims + i % DYN_Q)), 1)), "l"(v)
                         : "memory");
    };
    auto read_tile = [&](int i) -> int {   // one thread polls; bounded like every other wait of the kernel
        if (!dyn) {
            const int t = walker + i * n_walkers;
            return t < total_tiles ? t : -1;
        }
        const long long t0 = clock64();
        while (true) {
            const unsigned long long v = claims[i % DYN_Q];
            if ((uint32_t)(v >> 32) == (uint32_t)(i + 1)) return (int)(uint32_t)v;
            if (*abort_flag) return -1;
            if (clock64() - t0 > tc::WAIT_LIMIT_CYCLES) {
                *abort_flag = 1;
                if (p.err_word) atomicExch(p.err_word, 107);
                return -1;
            }
        }
    };
    if (dyn && blockIdx.x == 0 && threadIdx.x == 0) *p.dyn_reset = 0;   // the launch after this one starts from zero
    // A ragged k-tile of an expert's tokens: the instructions take whole sixteens of k rows, so A's rows from `valid` to the next
    // sixteen, which are the next expert's, are cleared by one warp (a row of k is 128 bytes in each of two boxes)
    auto clear_rows = [&](uint32_t s, int valid) {
        uint8_t* a_s = tiles + s * STAGE_BYTES + ((lane >> 3) & 1) * 8192 + (lane & 7) * 16;
        for (int kr = valid + (lane >> 4); kr < ((valid + 15) & ~15); kr += 2) *reinterpret_cast<uint4*>(a_s + kr * 128) = make_uint4(0, 0, 0, 0);
        tc::fence_proxy_async_smem();
        __syncwarp();
    };

    if (warp == 0) {
        // ------------------------------------------------------------ TMA producer (one thread)
        if (lane == 0) {
            uint32_t s = 0, round = 0;   // ring slot of the next k-tile and how often the ring has been around
            int n_rag = 0;
            bool ok = true;
            // The claiming thread asks for claim ci + 1 half way through claim ci's loads and publishes it after them: the
            // atomic's round trip hides behind the loads, and no other role needs the next claim before this one is used up.
            // (Not earlier: with about as many tiles as walkers the first to start would take two each, 190 us against 110 for
            // 64 tiles.)
            const bool claimer = dyn && rank == 0, may_be_empty = p.group_dim == GROUP_K || p.K == 0;
            int cur = 0;
            Tile ahead{};            // the claimer's next tile, where it has been located already
            bool located = false;
            if (claimer) {
                cur = atomicAdd(p.dyn_ctr, 1);
                publish_claim(0, cur);
            }
            for (int ci = 0; ok; ++ci) {
                const int t = claimer ? (cur < total_tiles ? cur : -1) : read_tile(ci);
                if (t < 0) break;
                int nxt = 0;
                const Tile x = located ? ahead : locate(t);
                located = false;
                const int nl0 = x.n0 + rank * BNL;   // first B column this CTA loads
                if (claimer && x.num_k == 0) nxt = atomicAdd(p.dyn_ctr, 1);
                for (int kt = 0; kt < x.num_k; ++kt) {
                    if (claimer && kt == x.num_k / 2) nxt = atomicAdd(p.dyn_ctr, 1);
                    if (round > 0 && !tc::mbar_wait(&empty[s], (round - 1) & 1, abort_flag, p.err_word, 101)) {
                        ok = false;
                        break;
                    }
                    uint8_t* a_s = tiles + s * STAGE_BYTES;
                    uint8_t* b_s = a_s + A_BYTES;
                    // A pair's stage completes on the even CTA's barrier, for both CTAs' bytes at once. A ragged k-tile is zeroed
                    // in part by each CTA first, so each waits for its own bytes, on a barrier of its own.
                    const bool joint = PAIR && !(p.group_dim == GROUP_K && kt + 1 == x.num_k && (x.K % BK) != 0);
                    const uint32_t bar = tc::smem_u32(PAIR && !joint ? &rag_full[s] : &full[s]), bar0 = joint && rank ? tc::mapa_u32(bar, 0) : bar;
                    if (!joint) tc::mbar_expect_tx(PAIR ? &rag_full[s] : &full[s], STAGE_BYTES);
                    else if (rank == 0) tc::mbar_expect_tx(&full[s], 2 * STAGE_BYTES);
                    auto load = [&](uint8_t* dst, const CUtensorMap* map, int c0, int c1) {
                        if (PAIR) tc::tma_load_2d_pair(dst, map, c0, c1, bar0);
                        else tc::tma_load_2d(dst, map, c0, c1, &full[s]);
                    };
                    const int k0 = kt * BK;
                    if (A_MN) {   // memory (k rows x M): two boxes of 64 columns
                        load(a_s, &mapA, x.m0, x.row_base_k + k0);
                        load(a_s + 8192, &mapA, x.m0 + 64, x.row_base_k + k0);
                    } else {      // memory (rows x K): one box 64 k x 128 rows
                        load(a_s, &mapA, k0, x.row_base_m + x.m0);
                    }
                    if (B_MN) {   // memory (k rows x N)
                        const int kr = (MODE == ASCA_TN ? x.row_base_k : 0) + k0 + x.b_out;
#pragma unroll
                        for (int nb = 0; nb < BNL / 64; ++nb)   // boxes of 64 columns
                            load(b_s + nb * 8192, &mapB, nl0 + nb * 64 + x.b_in, kr);
                    } else {      // memory (N rows x K)
                        load(b_s, &mapB, k0 + x.b_in, nl0 + x.b_out);
                    }
                    if (SH::RAG_WARP && !joint) {   // to the warp that clears its end
                        rag_q[n_rag++ % RAG_Q] = (uint16_t)(s << 8 | (uint32_t)(x.K % BK));
                        __threadfence_block();
                        rag_word[0] = 2 * n_rag;
                    }
                    if (++s == STAGES) s = 0, ++round;
                }
                if (SH::RAG_WARP) rag_word[1] = ci + 1;
                if (claimer) {
                    // A tile without k-tiles takes no ring slot, so nothing above holds the claims of a run of them back: each waits
                    // for the epilogue to release its accumulator buffer once more (of the tile two before it, or of one before that
                    // where ring slots have let the claims run further ahead; the distance then stays). The wait stands in front of
                    // the publication: behind it, the epilogues could be through the new tile already, and the parity would
                    // mean a tile that is yet to be claimed.
                    const int c = ci + 1;
                    if (ok && may_be_empty && nxt < total_tiles) {
                        ahead = locate(nxt);
                        located = true;
                        if (ahead.num_k == 0 && c >= 2) ok = tc::mbar_wait(&acc_empty[c & 1], ((c >> 1) - 1) & 1, abort_flag, p.err_word, 108);
                    }
                    cur = ok ? nxt : total_tiles;   // (after a wait that gave up: "none left", so that the other roles stop too)
                    publish_claim(c, cur);
                }
            }
            if (SH::RAG_WARP) rag_word[0] = 2 * n_rag + 1;
        }
    } else if (warp == 1) {
        // ------------------------------------------------------------ MMA issuer
        // One thread of the even CTA runs the loop (in single CTAs the rest of the warp joins to clear a ragged k-tile): wait for the
        // stage, four tcgen05.mma whose descriptors are the stage's base descriptor plus a constant, commit.
        // The loop's own dependent instructions are what bounds a single MMA stream, so it is kept short.
        constexpr uint32_t IDESC = tc::idesc_bf16_f32(TM, BN, A_MN ? 1 : 0, B_MN ? 1 : 0);
        constexpr uint32_t DESC_HI = (1024u >> 4) | (1u << 14) | (2u << 29);          // SBO 1024, version 1, 128-byte swizzle
        constexpr uint32_t A_LBO = (A_MN ? 8192u : 16u) >> 4, B_LBO = (B_MN ? 8192u : 16u) >> 4;
        constexpr uint32_t A_K16 = (A_MN ? 2048u : 32u) >> 4, B_K16 = (B_MN ? 2048u : 32u) >> 4;   // per k16 step, in 16-byte units
        const uint32_t a_lo0 = ((tc::smem_u32(tiles) >> 4) & 0x3FFF) | (A_LBO << 16);
        const uint32_t b_lo0 = (((tc::smem_u32(tiles) + A_BYTES) >> 4) & 0x3FFF) | (B_LBO << 16);
        bool ok = true;
        uint32_t s = 0;                      // ring slot of the next k-tile
        uint32_t par = 0, rag_par = 0;       // parity of every slot's next wait on `full` and on `rag_clear` (a bit each)
        for (int tl = 0; rank == 0; ++tl) {   // tiles done by this CTA: accumulator buffer tl & 1
            int t = lane == 0 && ok ? read_tile(tl) : -1;
            t = __shfl_sync(0xffffffffu, t, 0);
            if (t < 0) break;
            const Tile x = locate(t);
            const int buf = tl & 1;
            const uint32_t tmem_acc = tmem_base + buf * BN;
            const bool ragged = p.group_dim == GROUP_K && (x.K % BK) != 0;   // warp-uniform
            const int n_plain = ragged ? x.num_k - 1 : x.num_k;
            auto next = [&] {
                if (++s == STAGES) s = 0;
            };
            auto issue = [&](int kt, int rows) {   // one k-tile's instructions (on the first `rows` of its k), slot release, tile hand-over
                const uint32_t a_lo = a_lo0 + s * (STAGE_BYTES >> 4), b_lo = b_lo0 + s * (STAGE_BYTES >> 4);
#pragma unroll
                for (int k16 = 0; k16 < BK / 16; ++k16) {
                    if (k16 * 16 >= rows) break;
                    const uint64_t da = ((uint64_t)DESC_HI << 32) | (a_lo + k16 * A_K16), db = ((uint64_t)DESC_HI << 32) | (b_lo + k16 * B_K16);
                    if (PAIR) tc::umma_bf16_pair(tmem_acc, da, db, IDESC, (kt > 0 || k16 > 0) ? 1u : 0u);
                    else tc::umma_bf16(tmem_acc, da, db, IDESC, (kt > 0 || k16 > 0) ? 1u : 0u);
                }
                if (PAIR) {
                    tc::umma_commit_pair(&empty[s]);              // the slot is free in both CTAs once these MMAs retire
                    if (kt == x.num_k - 1) tc::umma_commit_pair(&acc_full[buf]);
                } else {
                    tc::umma_commit(&empty[s]);                   // slot free once these MMAs retire
                    if (kt == x.num_k - 1) tc::umma_commit(&acc_full[buf]);
                }
            };
            if (lane == 0) {
                if (tl >= 2) {   // the epilogue (of both CTAs) has read this buffer's previous tile out
                    ok = PAIR ? tc::mbar_wait_cluster(&acc_empty[buf], ((tl >> 1) - 1) & 1, abort_flag, p.err_word, 104)
                              : tc::mbar_wait(&acc_empty[buf], ((tl >> 1) - 1) & 1, abort_flag, p.err_word, 104);
                }
                tc::tcgen05_fence_after();
                for (int kt = 0; kt < n_plain && ok; ++kt) {
                    ok = tc::mbar_wait(&full[s], (par >> s) & 1, abort_flag, p.err_word, 102);
                    if (!ok) break;
                    tc::tcgen05_fence_after();
                    issue(kt, BK);
                    par ^= 1u << s;
                    next();
                }
                if (PAIR && ragged && ok) {
                    ok = tc::mbar_wait_cluster(&rag_clear[s], (rag_par >> s) & 1, abort_flag, p.err_word, 106);
                    if (ok) {
                        tc::tcgen05_fence_after();
                        issue(n_plain, x.K - n_plain * BK);
                        rag_par ^= 1u << s;
                        next();
                    }
                }
            }
            if (!PAIR && ragged) {
                // last k-tile of this expert: rows past it belong to the next expert and are cleared by the whole warp
                s = __shfl_sync(0xffffffffu, s, 0);
                int got = 0;
                if (lane == 0) got = ok && tc::mbar_wait(&full[s], (par >> s) & 1, abort_flag, p.err_word, 105) ? 1 : 0;
                got = __shfl_sync(0xffffffffu, got, 0);
                ok = got != 0;
                if (ok) {
                    clear_rows(s, x.K - n_plain * BK);
                    if (lane == 0) {
                        tc::tcgen05_fence_after();
                        issue(n_plain, x.K - n_plain * BK);
                    }
                }
                par ^= 1u << s;
                next();
            }
            if (lane == 0 && ok && x.num_k == 0) {   // empty expert: the epilogue stores zeros
                tc::mbar_arrive(&acc_full[buf]);
                if (PAIR) tc::mbar_arrive_cluster(tc::mapa_u32(tc::smem_u32(&acc_full[buf]), 1));
            }
            ok = __shfl_sync(0xffffffffu, ok ? 1 : 0, 0) != 0;   // lane 0's verdict; keeps the warp's tile loops in step
        }
    } else if (SH::RAG_WARP && warp == 2 + SH::EPI_WARPS) {
        // ------------------------------------------------------------ ragged k-tiles of a pair (both CTAs)
        // Clears the end of an expert's last k-tile when the tile lands, up to a ring's depth ahead of the instructions that read it.
        // In the issuing warp, all 64 rows' ends at a time, it held the instructions of the tile and of the next one up by 3 us a
        // tile: C = 1024 x 4096 for 64 experts of 512 tokens took 350 us where every count is a multiple of 64 and 498 where none
        // is (1,024 tokens: 520 and 718); now 367 and 377 (527 and 590).
        // The producer hands the ragged k-tiles over one by one, so this warp need not follow the claims, which nothing would hold for
        // it over a run of tiles without a ragged end.
        uint32_t par = 0;   // parity of every slot's next ragged k-tile (a bit each)
        if (p.group_dim == GROUP_K) {
            for (int done = 0;; ++done) {
                int item = -1;   // none left, or a wait gave up
                if (lane == 0) {
                    long long t0 = clock64();
                    for (int beat = 0;;) {
                        const int w = rag_word[0], tiles_done = rag_word[1];
                        if ((w >> 1) > done) {
                            __threadfence_block();
                            item = rag_q[done % RAG_Q];
                            if (!tc::mbar_wait(&rag_full[item >> 8], (par >> (item >> 8)) & 1, abort_flag, p.err_word, 105)) item = -1;
                            break;
                        }
                        if ((w & 1) || *abort_flag) break;
                        if (tiles_done != beat) beat = tiles_done, t0 = clock64();
                        if (clock64() - t0 > tc::WAIT_LIMIT_CYCLES) {   // (no tile for as long as any wait of the producer may take)
                            *abort_flag = 1;
                            if (p.err_word) atomicExch(p.err_word, 109);
                            break;
                        }
                        __nanosleep(100);
                    }
                }
                item = __shfl_sync(0xffffffffu, item, 0);
                if (item < 0) break;
                const uint32_t slot = (uint32_t)item >> 8;
                clear_rows(slot, item & 255);
                if (lane == 0) tc::mbar_arrive_cluster(tc::mapa_u32(tc::smem_u32(&rag_clear[slot]), 0));
                par ^= 1u << slot;
            }
        }
    } else {
        // ------------------------------------------------------------ epilogue (warps 2..5, EW8: 2..9)
        // A lane holds a row: tcgen05.ld hands it 32 columns of its row, bias / activation / accumulation are applied to those
        // 32 independent values, and they leave as 32-byte stores -- whole sectors, so neither a transpose through shared memory nor
        // row maps and ragged rows (a lane's own address, a lane's own predicate) cost anything. What bounds an epilogue of one
        // or two warps per scheduler is the latency of its instructions, not the bytes: hence the 32-wide straight-line code and
        // the loads of `aux` / of the old C a column group or two ahead, the first before the accumulator is awaited. Measured on the
        // expert products of 65,536 tokens, 1024 -> 4096 (two outputs, SiLU; SiLU' with its f32 read), whose tiles have 6 us of main
        // loop: 670 and 730 us, against 1076 and 1166 with results staged through shared memory. The TMEM buffer is released after
        // the last tcgen05.ld; the next tile's main loop runs meanwhile in the other buffer.
        const int q = warp & 3;                 // TMEM lane quarter this warp may read
        const int ew = warp - 2;                // epilogue warp index; warps ew and ew + 4 share lane quarter q
        constexpr int C_PER_WARP = (BN / 32) / (SH::EPI_WARPS / 4);   // 32-column groups of a row per warp
        const int c_lo = (ew >> 2) * C_PER_WARP;
        // elements a lane may move at once: 8 (32 bytes), 4 or 1
        auto width = [](const void* base, int64_t ld, int64_t gstride, int unit) {
            const uintptr_t a = reinterpret_cast<uintptr_t>(base) | (uintptr_t)(ld * unit) | (uintptr_t)(gstride * unit);
            return (a & 31) == 0 ? 8 : (a & 15) == 0 ? 4 : 1;
        };
        const int c_w = min(width(p.C, p.ldc, p.group_dim == GROUP_K ? p.c_gstride : 0, 4), width(p.old, 0, 0, 4));
        const int aux_w = width(p.aux, p.ldaux, 0, 4);
        const int bias_w = width(p.bias, 0, p.bias_gstride, 4);
        const int c2_w = width(p.C2, p.ldc2, 0, 2);
        const int qkv_w = min(width(p.qkv_q, p.qkv_d, 0, 2), min(width(p.qkv_k, 0, 0, 2), width(p.qkv_v, 0, 0, 2)));
        const bool with_aux = p.epi == EPI_SILU_BWD;
        bool ok = true;
        for (int tl = 0; ok; ++tl) {
            int t = lane == 0 ? read_tile(tl) : -1;
            t = __shfl_sync(0xffffffffu, t, 0);
            if (t < 0) break;
            const Tile x = locate(t);
            const int buf = tl & 1;
            const uint32_t tmem_acc = tmem_base + buf * BN + ((uint32_t)(q * 32) << 16);
            const bool live = x.M - (x.m0 + q * 32) > lane;   // rows past the matrix's or the expert's end are computed, not stored
            const int64_t lr = (int64_t)x.row_base_m + x.m0 + (live ? q * 32 + lane : 0);
            const int64_t cr = p.c_idx && live ? (int64_t)p.c_idx[lr] : lr;
            const int64_t c_off = (p.group_dim == GROUP_K ? (int64_t)x.g * p.c_gstride : 0) + cr * p.ldc + x.n0;
            float* crow = p.C + c_off;
            const float* orow = p.old + c_off;
            const float* arow = p.aux + lr * p.ldaux + x.n0;
            const float* brow = p.bias ? p.bias + (int64_t)x.g * p.bias_gstride + x.n0 : nullptr;
            // aux, or where there is none the rows to add, ahead of their use (an add of the residual here, with the bf16 copy the
            // next block reads, hides behind the next tile's instructions: a prefill of 14,448 tokens x 12 blocks took 6.06 ms with
            // the adds in passes of their own, 5.92 with them here; a training step of 32,768 x 2048 15.95 and 15.82 ms)
            const float* prow = with_aux ? arow : orow;
            const bool ahead = live && (with_aux || p.old);
            const int p_w = with_aux ? aux_w : c_w;
            constexpr int AHEAD = PAIR && !EW8 ? 2 : 1;   // (registers: 255 with four epilogue warps, 168 with eight)
            float pre[AHEAD][32];
            if (ahead) {
#pragma unroll
                for (int g = 0; g < AHEAD; ++g) load_row(pre[g], prow + (c_lo + g) * 32, p.N - x.n0 - (c_lo + g) * 32, p_w);
            }
            if (brow && lane < C_PER_WARP && x.n0 + (c_lo + lane) * 32 < p.N)   // this warp's bias on its way into L1
                asm volatile("prefetch.global.L1 [%0];" ::"l"(brow + (c_lo + lane) * 32));
            int got = 0;
            if (lane == 0)
                got = (PAIR ? tc::mbar_wait_cluster(&acc_full[buf], (tl >> 1) & 1, abort_flag, p.err_word, 103)
                            : tc::mbar_wait(&acc_full[buf], (tl >> 1) & 1, abort_flag, p.err_word, 103)) ? 1 : 0;
            ok = __shfl_sync(0xffffffffu, got, 0) != 0;  // uniform: tcgen05.ld below is warp-aligned
            if (!ok) break;
            tc::tcgen05_fence_after();
            // fused qkv epilogue (pair shape): this warp's 128 columns are one head of q, k or v, or two of 64
            const bool qkv = PAIR && EW8 && p.epi == EPI_QKV;
            float qkv_scale[2] = {1.0f, 1.0f};      // 1 / max(|z|, 1e-8) of this lane's row (q, k), 1 for v; per 64 columns
            __nv_bfloat16* hrow = p.C2 + (p.c2_mapped ? cr : lr) * p.ldc2 + x.n0;
            if (qkv) {
                const int hc0 = x.n0 + c_lo * 32;   // first column of the head
                const int sec = hc0 / p.qkv_d;      // 0 q, 1 k, 2 v
                hrow = (sec == 0 ? p.qkv_q : sec == 1 ? p.qkv_k : p.qkv_v) + lr * p.qkv_d + (x.n0 - sec * p.qkv_d);
                if (sec < 2) {
                    float ss[2] = {0.0f, 0.0f};
#pragma unroll 1
                    for (int c = 0; c < C_PER_WARP; ++c) {
                        uint32_t r[32];
                        tc::tmem_ld_32x32(tmem_acc + (uint32_t)((c_lo + c) * 32), r);
                        tc::tmem_ld_wait();
                        const float4* bb = reinterpret_cast<const float4*>(p.bias + hc0 + c * 32);
                        float sq = 0.0f;
#pragma unroll
                        for (int j = 0; j < 8; ++j) {
                            const float4 b4 = bb[j];
                            const float v0 = __uint_as_float(r[4 * j]) + b4.x, v1 = __uint_as_float(r[4 * j + 1]) + b4.y,
                                        v2 = __uint_as_float(r[4 * j + 2]) + b4.z, v3 = __uint_as_float(r[4 * j + 3]) + b4.w;
                            sq += (v0 * v0 + v1 * v1) + (v2 * v2 + v3 * v3);
                        }
                        if (c < C_PER_WARP / 2) ss[0] += sq;
                        else ss[1] += sq;
                    }
                    const bool two = p.qkv_dh == 64;
                    if (!two) ss[0] += ss[1];
                    const int heads = p.qkv_d / p.qkv_dh, head = (hc0 - sec * p.qkv_d) / p.qkv_dh;
                    float* norms = (sec == 0 ? p.qkv_qn : p.qkv_kn) + lr * heads + head;
                    const float n0 = fmaxf(sqrtf(ss[0]), 1e-8f), n1 = two ? fmaxf(sqrtf(ss[1]), 1e-8f) : n0;
                    qkv_scale[0] = 1.0f / n0;
                    qkv_scale[1] = 1.0f / n1;
                    if (live) norms[0] = n0;
                    if (live && two) norms[1] = n1;
                }
            }
            // fused cross-entropy (pair shape, four epilogue warps: a warp's lanes hold whole rows of 256 logits)
            const bool ce = PAIR && !EW8 && p.epi == EPI_CE;
            float ce_max = 0.0f, ce_inv = 0.0f;
            int ce_t = 0;
            if (ce) {
                ce_t = (int)p.ce_targets[lr];
                float mx = -INFINITY, sum = 0.0f, zt = 0.0f;
#pragma unroll 1
                for (int c = 0; c < BN / 32; ++c) {   // online max / sum of exponentials over the row
                    uint32_t r[32];
                    tc::tmem_ld_32x32(tmem_acc + (uint32_t)(c * 32), r);
                    tc::tmem_ld_wait();
                    float cm = mx;
#pragma unroll
                    for (int j = 0; j < 32; ++j) {
                        const float z = __uint_as_float(r[j]);
                        cm = fmaxf(cm, z);
                        if (c * 32 + j == ce_t) zt = z;
                    }
                    float part = 0.0f;
#pragma unroll
                    for (int j = 0; j < 32; ++j) part += expf(__uint_as_float(r[j]) - cm);
                    sum = sum * expf(mx - cm) + part;
                    mx = cm;
                }
                p.ce_loss[lr] = (mx + logf(sum)) - zt;
                ce_max = mx;
                ce_inv = 1.0f / sum;
            }
            const bool c_out = !(p.c2_only || qkv || ce), h_out = qkv || ce || p.C2;
            const int h_w = qkv ? qkv_w : c2_w;
            // Every 32-byte piece that a store instruction writes to a line of its own is a request to L2, and with f32 results the
            // requests bound these epilogues; lane pairs that write 64 bytes halve them. 64 experts of about 1,024 tokens, C = 1024 x
            // 4096: 563 -> 531 us, and of about 512 tokens, 2048 x 4096: 790 -> 700. Not with eight warps, whose bf16 second results or
            // reads weigh as much and whose registers are full: SiLU' 727 -> 775 us, the fused qkv form 70 -> 76. Groups of four lanes and
            // 128 bytes cost more in exchanges than they save (734 -> 781).
            const bool odd = lane & 1, c_pair = PAIR && !EW8 && c_out && c_w == 8 && __all_sync(0xffffffffu, live);
            float* const nb_row = reinterpret_cast<float*>(__shfl_xor_sync(0xffffffffu, reinterpret_cast<unsigned long long>(crow), 1));
            float *const even_row = odd ? nb_row : crow, *const odd_row = odd ? crow : nb_row;
            // A tcgen05.ld takes about 1,000 cycles beside the next tile's instructions, so the next group's is under way while one is
            // processed. (Unrolled to the end: what it loads may not pass through a loop's register moves before the wait. The four-warp
            // form loads in turn: two under way took 66 us against 51 for 14,448 x 768 x 768 with a residual.)
            constexpr bool TWO = C_PER_WARP <= 4;
            uint32_t acc[TWO ? 2 : 1][32];
            if (TWO) tc::tmem_ld_32x32(tmem_acc + (uint32_t)(c_lo * 32), acc[0]);
#pragma unroll(TWO ? C_PER_WARP : 2)
            for (int i = 0; i < C_PER_WARP; ++i) {
                const int c = c_lo + i;
                const int n_left = p.N - x.n0 - c * 32;   // columns of the matrix from here on
                float v[32];
                if (!TWO) tc::tmem_ld_32x32(tmem_acc + (uint32_t)(c * 32), acc[0]);
                tc::tmem_ld_wait();
#pragma unroll
                for (int j = 0; j < 32; ++j) v[j] = x.num_k > 0 ? __uint_as_float(acc[TWO ? i & 1 : 0][j]) : 0.0f;
                if (TWO && i + 1 < C_PER_WARP) tc::tmem_ld_32x32(tmem_acc + (uint32_t)((c + 1) * 32), acc[(i + 1) & 1]);
                if (c + 1 == c_lo + C_PER_WARP) {   // this warp's share of the buffer is free for the tile after next
                    tc::tcgen05_fence_before();
                    __syncwarp();
                    if (lane == 0) {
                        if (PAIR) tc::mbar_arrive_cluster(tc::mapa_u32(tc::smem_u32(&acc_empty[buf]), 0));   // counted by the even CTA
                        else tc::mbar_arrive(&acc_empty[buf]);
                    }
                }
                if (n_left <= 0) continue;
                if (ce) {    // dlogits = (softmax - onehot) * scale
#pragma unroll
                    for (int j = 0; j < 32; ++j) {
                        float pr = expf(v[j] - ce_max) * ce_inv;
                        if (c * 32 + j == ce_t) pr -= 1.0f;
                        v[j] = pr * p.ce_scale;
                    }
                }
                if (brow) {
                    float b[32];
                    load_row(b, brow + c * 32, n_left, bias_w);
#pragma unroll
                    for (int j = 0; j < 32; ++j) v[j] += b[j];
                }
                if (qkv) {
#pragma unroll
                    for (int j = 0; j < 32; ++j) v[j] *= qkv_scale[2 * i / C_PER_WARP];
                }
                if (with_aux) {
#pragma unroll
                    for (int j = 0; j < 32; ++j) v[j] *= silu_grad_f(pre[i % AHEAD][j]);
                    if (p.old && live) {
                        float old[32];
                        load_row(old, orow + c * 32, n_left, c_w);
#pragma unroll
                        for (int j = 0; j < 32; ++j) v[j] += old[j];
                    }
                } else if (p.old) {
#pragma unroll
                    for (int j = 0; j < 32; ++j) v[j] += pre[i % AHEAD][j];
                }
                if (ahead && i + AHEAD < C_PER_WARP) load_row(pre[i % AHEAD], prow + (c + AHEAD) * 32, n_left - 32 * AHEAD, p_w);
                if (PAIR && !EW8 && c_pair && n_left >= 32) store_row_pair(even_row + c * 32, odd_row + c * 32, v, odd);
                else if (c_out && live) store_row(crow + c * 32, v, n_left, c_w);
                if (h_out && live) {
                    if (p.epi == EPI_SILU) {
#pragma unroll
                        for (int j = 0; j < 32; ++j) v[j] = silu_f(v[j]);
                    }
                    store_row(hrow + c * 32, v, n_left, h_w);
                }
            }
        }
    }
    // ---- teardown: everyone meets, then the allocating warp frees TMEM
    tc::tcgen05_fence_before();
    __syncthreads();
    if (PAIR) tc::cluster_sync_all();     // neither CTA leaves (or frees TMEM) while its peer may still signal it
    if (*abort_flag) __nanosleep(20000);  // let copies already in flight land before the CTA exits
    if (warp == 1) {
        if (PAIR) tc::tmem_dealloc_pair(tmem_base, TMEM_COLS);
        else tc::tmem_dealloc(tmem_base, TMEM_COLS);
    }
}

typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                  const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                  CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

EncodeTiledFn encode_fn() {
    static EncodeTiledFn fn = nullptr;
    if (!fn) {
        void* p = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) == cudaSuccess &&
            q == cudaDriverEntryPointSuccess)
            fn = (EncodeTiledFn)p;
    }
    return fn;
}

// 2-D bf16 tensor map: `cols` contiguous elements per row, `rows` rows, row pitch `ld` elements.
bool make_map(CUtensorMap* m, const void* base, int64_t rows, int64_t cols, int64_t ld, int box_cols, int box_rows) {
    EncodeTiledFn fn = encode_fn();
    if (!fn) return false;
    cuuint64_t dims[2] = {(cuuint64_t)cols, (cuuint64_t)rows};
    cuuint64_t strides[1] = {(cuuint64_t)ld * 2};
    cuuint32_t box[2] = {(cuuint32_t)box_cols, (cuuint32_t)box_rows};
    cuuint32_t estr[2] = {1, 1};
    return fn(m, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void*>(base), dims, strides, box, estr,
              CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
              CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

}  // namespace

bool supported(const Args& a) {
    if (!encode_fn()) return false;
    if ((reinterpret_cast<uintptr_t>(a.A) & 15) || (reinterpret_cast<uintptr_t>(a.B) & 15)) return false;
    if ((a.lda & 7) || (a.ldb & 7)) return false;                       // row pitch multiple of 16 bytes
    if ((a.b_goff_inner & 7)) return false;                             // TMA inner coordinate: 16-byte aligned
    if (a.a_rows <= 0 || a.b_rows <= 0 || a.a_cols <= 0 || a.b_cols <= 0) return false;
    // grouped coordinate offsets must not let a ragged tile read a neighbouring expert's k range
    if (a.group_dim == GROUP_M && a.mode == ASCA_NT && a.b_goff_inner != 0 && (a.K % BK) != 0) return false;
    if (a.group_dim == GROUP_M && a.mode == ASCA_NN && a.b_goff_outer != 0 && (a.K % BK) != 0) return false;
    if (a.group_dim != GROUP_NONE && a.n_groups > MAX_GROUPS) return false;
    if (a.group_dim == GROUP_K && a.mode != ASCA_TN) return false;
    if (a.group_dim == GROUP_M && a.mode == ASCA_TN) return false;
    if (a.c2_only && (!a.C2 || a.accumulate || (a.epi != EPI_NONE && a.epi != EPI_SILU && a.epi != EPI_SILU_BWD) || a.c_idx || skinny_wanted(a))) return false;
    if (a.b_packed && !skinny_wanted(a)) return false;
    if (a.res && (!a.accumulate || a.group_dim == GROUP_K || skinny_wanted(a))) return false;
    return true;
}

template <int BN, bool DEEP, bool PAIR = false, bool EW8 = false>
static int launch_shape(asca_ctx* ctx, const Args& a, int64_t grid) {
    CUtensorMap mapA, mapB;
    bool ok;
    if (a.mode == ASCA_TN) ok = make_map(&mapA, a.A, a.a_rows, a.a_cols, a.lda, 64, 64);
    else ok = make_map(&mapA, a.A, a.a_rows, a.a_cols, a.lda, 64, 128);
    if (a.mode == ASCA_NT) ok = ok && make_map(&mapB, a.B, a.b_rows, a.b_cols, a.ldb, 64, PAIR ? BN / 2 : BN);
    else ok = ok && make_map(&mapB, a.B, a.b_rows, a.b_cols, a.ldb, 64, 64);
    if (!ok) return asca_fail(ctx, ASCA_ERR_CUDA, "gemm_tc: cuTensorMapEncodeTiled failed");
    KP p{};
    p.C = a.C; p.ldc = a.ldc; p.M = a.M; p.N = a.N; p.K = a.K;
    p.bias = a.bias; p.old = a.accumulate ? (a.res ? a.res : a.C) : nullptr; p.c_idx = a.c_idx;
    p.offsets = a.offsets; p.n_groups = a.n_groups; p.group_dim = a.group_dim;
    p.b_goff_inner = a.b_goff_inner; p.b_goff_outer = a.b_goff_outer;
    p.c_gstride = a.c_gstride; p.bias_gstride = a.bias_gstride;
    p.epi = a.epi; p.aux = a.aux; p.ldaux = a.ldaux; p.C2 = a.C2; p.ldc2 = a.ldc2; p.c2_only = a.c2_only; p.c2_mapped = a.c2_mapped;
    p.ce_targets = a.ce_targets; p.ce_loss = a.ce_loss; p.ce_scale = a.ce_scale;
    p.qkv_q = a.qkv_q; p.qkv_k = a.qkv_k; p.qkv_v = a.qkv_v; p.qkv_qn = a.qkv_qn; p.qkv_kn = a.qkv_kn; p.qkv_d = a.qkv_d; p.qkv_dh = a.qkv_dh;
    p.err_word = ctx->err_word;
    {   // dynamic tile claims: not under programmatic dependent launch (the counter hand-over relies on stream order)
        static const int dyn_env = [] { const char* e = getenv("ASCA_GEMM_DYNAMIC"); return e ? atoi(e) : 1; }();
        const bool want = dyn_env != 0;   // on unless ASCA_GEMM_DYNAMIC=0
        if (want && !ctx->pdl) {
            if (!ctx->dyn_buf) {
                if (cudaMalloc(&ctx->dyn_buf, 256) != cudaSuccess) return asca_fail(ctx, ASCA_ERR_OOM, "gemm_tc: cannot allocate the tile counters");
                ASCA_CUDA(ctx, cudaMemsetAsync(ctx->dyn_buf, 0, 256, ctx->stream));
                ctx->dyn_seq = 0;
            }
            // One tile per claim: with several consecutive ones (8 where a walker has > 128 tiles) a train step took 355.4 ms
            // against 335.9 -- neighbouring walkers then do not work on neighbouring tiles at the same time, which is what
            // lets them share operand tiles in L2.
            const uint32_t seq = ++ctx->dyn_seq;
            int* ctrs = static_cast<int*>(ctx->dyn_buf);
            p.dyn_ctr = ctrs + (seq & 1) * 32;          // the two counters sit in different 128-byte lines
            p.dyn_reset = ctrs + ((seq + 1) & 1) * 32;
        }
    }
    using SH = Shape<BN, DEEP, PAIR, EW8>;
    const size_t table = (size_t)(2 * (a.group_dim == GROUP_NONE ? 1 : a.n_groups) + 4) * 4;   // tile table + group offsets
    p.stages = (uint32_t)std::min<size_t>(SH::STAGES, (ctx->smem_optin - SH::SMEM_FIXED - table) / SH::STAGE_BYTES);
    const size_t smem = SH::SMEM_FIXED + p.stages * SH::STAGE_BYTES + table;
    auto go = [&](auto kern) -> cudaError_t {
        cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        if (e != cudaSuccess) return e;
        if (!PAIR) return asca_launch(ctx, kern, dim3((unsigned)grid), dim3(SH::THREADS), smem, mapA, mapB, p);
        // pairs of CTAs: a cluster of two per walker (grid = 2 x walkers)
        cudaLaunchConfig_t cfg = {};
        cfg.gridDim = dim3((unsigned)grid);
        cfg.blockDim = dim3(SH::THREADS);
        cfg.dynamicSmemBytes = smem;
        cfg.stream = ctx->stream;
        cudaLaunchAttribute at[2];
        at[0].id = cudaLaunchAttributeClusterDimension;
        at[0].val.clusterDim.x = 2;
        at[0].val.clusterDim.y = 1;
        at[0].val.clusterDim.z = 1;
        at[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        at[1].val.programmaticStreamSerializationAllowed = 1;
        cfg.attrs = at;
        cfg.numAttrs = ctx->pdl ? 2 : 1;
        return cudaLaunchKernelEx(&cfg, kern, mapA, mapB, p);
    };
    cudaError_t e = a.mode == ASCA_NN ? go(gemm_tc_kernel<ASCA_NN, BN, DEEP, PAIR, EW8>)
                    : a.mode == ASCA_TN ? go(gemm_tc_kernel<ASCA_TN, BN, DEEP, PAIR, EW8>) : go(gemm_tc_kernel<ASCA_NT, BN, DEEP, PAIR, EW8>);
    ASCA_CUDA(ctx, e);
    ctx->launches++;
    return ASCA_OK;
}

// upper bound on the number of bm x bn tiles (exact unless rows are grouped by expert)
static int64_t tile_bound(const Args& a, int bn, int bm = BM) {
    const int64_t tn = (a.N + bn - 1) / bn;
    if (a.group_dim == GROUP_NONE) return ((int64_t)(a.M + bm - 1) / bm) * tn;
    if (a.group_dim == GROUP_M) return (a.total_rows / bm + a.n_groups) * tn;
    return (int64_t)a.n_groups * ((a.M + bm - 1) / bm) * tn;
}

// ASCA_GEMM_PAIR=0 switches the CTA-pair shape off (A/B measurements); read once.
static bool pair_enabled() {
    static const bool on = [] {
        const char* e = getenv("ASCA_GEMM_PAIR");
        return !(e && e[0] == '0');
    }();
    return on;
}

static bool pair_wanted(asca_ctx* ctx, const Args& a);

bool qkv_fusable(asca_ctx* ctx, const Args& a) {
    return supported(a) && !skinny_wanted(a) && a.group_dim == GROUP_NONE && a.mode == ASCA_NN && pair_wanted(ctx, a) && a.qkv_d > 0 &&
           a.qkv_d % 256 == 0 && (a.qkv_dh == 128 || a.qkv_dh == 64) && a.N == 3 * a.qkv_d && a.bias && (reinterpret_cast<uintptr_t>(a.bias) & 15) == 0 &&
           a.qkv_q && a.qkv_k && a.qkv_v && a.qkv_qn && a.qkv_kn && !a.accumulate && !a.c_idx &&
           ((reinterpret_cast<uintptr_t>(a.qkv_q) | reinterpret_cast<uintptr_t>(a.qkv_k) | reinterpret_cast<uintptr_t>(a.qkv_v)) & 7) == 0;
}

bool ce_fusable(asca_ctx* ctx, const Args& a) {
    return supported(a) && !skinny_wanted(a) && a.group_dim == GROUP_NONE && a.mode == ASCA_NN && pair_wanted(ctx, a) && a.N == 256 &&
           a.M % 256 == 0 && !a.bias && !a.accumulate && !a.c_idx && a.C2 && a.ldc2 == 256 && (reinterpret_cast<uintptr_t>(a.C2) & 7) == 0 &&
           a.ce_targets && a.ce_loss;
}

int launch(asca_ctx* ctx, const Args& a) {
    if (a.epi == EPI_CE && !ce_fusable(ctx, a)) return asca_fail(ctx, ASCA_ERR_UNSUPPORTED, "gemm_tc: this product cannot take the fused cross-entropy epilogue");
    if (a.epi == EPI_QKV && !qkv_fusable(ctx, a)) return asca_fail(ctx, ASCA_ERR_UNSUPPORTED, "gemm_tc: this product cannot take the fused qkv epilogue");
    if (skinny_wanted(a)) return launch_skinny(ctx, a);
    // measurement harnesses: the product's algorithmic FLOPs go with the timed span
    const double rows_m = a.group_dim == GROUP_M ? (double)a.total_rows : (double)a.M;
    const double rows_k = a.group_dim == GROUP_K ? (double)a.total_rows : (double)a.K;
    asca_span sp(ctx, a.group_dim == GROUP_NONE ? "gemm_tc_kernel (dense)"
                      : a.group_dim == GROUP_M  ? "gemm_tc_kernel (expert-grouped rows)"
                                                : "gemm_tc_kernel (expert-grouped k)",
                 2.0 * rows_m * (double)a.N * rows_k);
    const int n_sm = ctx->sm_count > 0 ? ctx->sm_count : 148;
    // persistent: the CTAs (or pairs, on 256 x 256 tiles) claim tile after tile
    if (pair_wanted(ctx, a)) {
        const int64_t g2 = 2 * std::min<int64_t>(tile_bound(a, 256, 256), n_sm / 2);
        if (a.group_dim == GROUP_M || a.epi == EPI_QKV) return launch_shape<256, false, true, true>(ctx, a, g2);
        return launch_shape<256, false, true, false>(ctx, a, g2);
    }
    const int64_t grid = tile_bound(a, 128);
    if (grid <= 0) return ASCA_OK;
    if (grid <= n_sm) return launch_shape<128, true>(ctx, a, grid);
    return launch_shape<128, false>(ctx, a, std::min<int64_t>(grid, 2 * n_sm));
}

// A pair runs a 256 x 256 tile 1.6 times as fast as two SMs run its four quarters in the 128 x 128 shape (two CTAs an SM), so pairs win
// from half of them busy on; below that, each quarter has an SM of its own in the deep 128 x 128 form. With 64 tiles (1024 x 65,536 x
// 4096, A^T B): 402 us in pairs, 906 in quarters. Rows grouped by expert need 512 rows an expert, or padding to 256 rows costs more than that.
static bool pair_wanted(asca_ctx* ctx, const Args& a) {
    const int n_sm = ctx->sm_count > 0 ? ctx->sm_count : 148;
    const int64_t pairs = tile_bound(a, 256, 256);
    static const bool pair_rows = [] { const char* e = getenv("ASCA_GEMM_PAIR"); return !(e && e[0] == '1'); }();
    const bool pair_shape = a.group_dim == GROUP_M ? (pair_rows && a.total_rows >= 512 * (int64_t)a.n_groups) : a.M >= 256;
    return pair_enabled() && pair_shape && a.N >= 256 && (a.group_dim == GROUP_M ? pairs >= n_sm / 2 : pairs > n_sm / 4);
}

}  // namespace gemm_tc
