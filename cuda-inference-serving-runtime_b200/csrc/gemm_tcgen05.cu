// Matrix product on the 5th-generation tensor cores: out[M, N] (float) = a[M, K] * w[N, K]^T, bfloat16
// operands, float accumulation in tensor memory.  Used for steps with more tokens than the weight-streaming
// kernels take (prompt portions, large decode batches).
//
//   * few tiles: gemm_tcgen05_split_kernel, a tile per CTA, K cut over a cluster
//   * more: gemm_tcgen05_pair_kernel, persistent, tiles of 256 rows on two SMs
//   * routed experts: gemm_tcgen05_experts_kernel, weight rows as the rows of a tile, an expert's tokens as its columns
//   * grouped products, and narrow ones with many rows: gemm_tcgen05_kernel, persistent CTAs that walk output tiles of 128 x BN
//     (BN = 256, 128 or 64) with two accumulators of BN columns in tensor memory, so that the epilogue of one tile runs under the
//     products of the next
// All of them have the same roles (here those of gemm_tcgen05_kernel):
//   * warp 0: one thread issues TMA loads (cp.async.bulk.tensor.2d, 128-byte swizzle) of the A tile
//     [128 rows x 64 k] and the B tile [BN rows x 64 k] into a STAGES-deep ring of shared memory (3 to 8
//     stages), each load completing on the stage's "full" mbarrier
//   * warp 1: allocates 2 * BN columns of tensor memory; one thread issues tcgen05.mma (kind::f16, M = 128,
//     N = BN, K = 16, four per 64-wide k block) on shared-memory descriptors and commits each stage to its
//     "empty" mbarrier, and each finished tile to its "accumulator ready" mbarrier
//   * warps 2..5: read the accumulator with tcgen05.ld (32 lanes x 32 columns per warp and step) and run the
//     epilogue: PLAIN writes float rows of `out` (or adds them to it: the residual form); SWIGLU (the B tile is
//     gate rows and the up rows of the same features) writes silu(gate) * up as bfloat16; ROPE (the tile is
//     whole heads of the stacked q/k/v projection) rotates q and k heads and writes q rows and the k, v cache
//     pages as bfloat16
//
// Rows and columns beyond M, N or K are zero-filled by TMA on the way in and skipped on the way out, so any
// M and N work; K must be a multiple of 8 (16-byte rows for the tensor map).  Every wait on an mbarrier
// gives up after a bounded number of polls: the kernel then sets `*error`, skips the rest of its work,
// frees its tensor memory and returns, and the host reports the failure.
//
// Parity: this is the product runtime/blas.py:41-56 of the reference hands to cuBLAS (C^T = W * X^T).
#include <limits.h>

#include "tcgen05.cuh"

namespace {
typedef __nv_bfloat16 bf16;
enum : int { EPI_PLAIN = 0, EPI_SWIGLU = 1, EPI_ROPE = 2, EPI_RELU2 = 3, EPI_GATED = 4 };
// SWIGLU and GATED: the B tile is BN / 2 gate rows and the BN / 2 up rows of the same features
__host__ __device__ constexpr bool paired_rows(int epi) { return epi == EPI_SWIGLU || epi == EPI_GATED; }
constexpr int BK = 64, UMMA_K = 16;     // BM = 128 (tcgen05.cuh)

// Where a role is in a ring of `stages`: the stage, and the parity of the turn it is on.
struct RingAt {
    int stage = 0; uint32_t turn = 0;
    __device__ __forceinline__ void next(int stages) { if (++stage == stages) { stage = 0; turn ^= 1u; } }
};

struct Epilogue {                       // what the epilogue variants need beyond the accumulator
    float* out_f32; bf16* out_bf16; int inter;
    float limit, alpha;                 // GATED: g' = min(g, limit), u' = clamp(u, +-limit), g' sigmoid(alpha g') (u' + 1)
    int act;                            // RELU2's activation: 0 max(z, 0)^2, 1 the exact gelu z Phi(z); SWIGLU's gate: 0 silu, 1 the tanh form of gelu
    int accumulate;                     // PLAIN: out += product
    float out_mult;                     // PLAIN: the product is multiplied by it first (a constant factor of the residual branch); 0: no factor (the residual stream, in place) instead of out = product
    const float* cos_t; const float* sin_t; bf16* q_out; bf16* k_cache; bf16* v_cache; const int* positions;
    const int* token_req; const int* req_slot; const int* block_table; int table_width; int page_size; int hq; int hkv; int dim;
    // Grouped product: the rows of `a` are sorted by group (an expert), each group's rows padded to whole 128-row tiles;
    // tile_group[i] is the group of row tile i (-1: the tile holds no rows and is skipped), and group g multiplies with
    // rows [g * n, (g + 1) * n) of `w`.  Null: one weight matrix for all rows.
    const int* tile_group;
};
// 32 floats -> 32 bfloat16 (64 bytes) at dst; `count` of them are valid
__device__ __forceinline__ void store_bf16x32(bf16* dst, const float (&v)[32], int count) {
    if (count >= 32 && ((uintptr_t)dst & 15) == 0) {
#pragma unroll
        for (int j = 0; j < 32; j += 8) {
            uint4 p;
            __nv_bfloat162 a = __floats2bfloat162_rn(v[j], v[j + 1]), b = __floats2bfloat162_rn(v[j + 2], v[j + 3]);
            __nv_bfloat162 c = __floats2bfloat162_rn(v[j + 4], v[j + 5]), d = __floats2bfloat162_rn(v[j + 6], v[j + 7]);
            p.x = *reinterpret_cast<uint32_t*>(&a); p.y = *reinterpret_cast<uint32_t*>(&b);
            p.z = *reinterpret_cast<uint32_t*>(&c); p.w = *reinterpret_cast<uint32_t*>(&d);
            *reinterpret_cast<uint4*>(dst + j) = p;
        }
    } else {
#pragma unroll
        for (int j = 0; j < 32; ++j)
            if (j < count) dst[j] = __float2bfloat16_rn(v[j]);
    }
}

// A warp's results leave by way of a patch of shared memory (STAGE_BYTES, 16-byte units of a row exchanged among eight rows against
// bank conflicts): in registers a lane has a row, and stores of 16 bytes each to 32 rows reach L2 as half-filled sectors; from the patch
// four to eight rows leave as whole runs.  us, persistent kernel, without and with: 2533 rows of 6144 x 2048 67 and 58, 4096 rows of 8192 x
// 2048 116 and 106; few tiles, 2048 rows of 2048 x 2048 19.0 and 17.8.  Gated results, half as many bytes, go straight out of the kernel
// for few tiles (200 rows of 4096 x 1024 8.4 us, 8.8 through the patch); in the pair kernel there is no difference.
constexpr size_t STAGE_BYTES = 4096;
// 32 bfloat16 per lane and row to dst + 32-column runs: `to(r)` is where row r of the warp's 32 goes (null: nowhere); units of eight
// columns, `units` of them valid
template <typename To>
__device__ __forceinline__ void store_rows_bf16(unsigned char* patch, const float (&v)[32], To to, int units) {
    const int lane = threadIdx.x & 31;
    __syncwarp();                                        // the run before has been read
#pragma unroll
    for (int u = 0; u < 4; ++u) {
        uint32_t w[4];
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            const __nv_bfloat162 p = __floats2bfloat162_rn(v[8 * u + 2 * e], v[8 * u + 2 * e + 1]);
            w[e] = *reinterpret_cast<const uint32_t*>(&p);
        }
        *reinterpret_cast<uint4*>(patch + lane * 64 + ((u ^ (lane >> 1)) & 3) * 16) = make_uint4(w[0], w[1], w[2], w[3]);
    }
    __syncwarp();
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const int r = 8 * i + (lane >> 2), u = lane & 3;
        bf16* dst = to(r);
        const uint4 w = *reinterpret_cast<const uint4*>(patch + r * 64 + ((u ^ (r >> 1)) & 3) * 16);
        if (dst && u < units) *reinterpret_cast<uint4*>(dst + 8 * u) = w;
    }
}

// Columns of tensor memory for two accumulators of `bn` columns: allocations are powers of two.
__host__ __device__ constexpr int tmem_columns(int bn) { return 2 * bn <= 32 ? 32 : 2 * bn <= 64 ? 64 : 2 * bn <= 128 ? 128 : 2 * bn <= 256 ? 256 : 512; }

template <int BN, int STAGES>
struct Smem {
    static constexpr size_t A_BYTES = (size_t)BM * BK * sizeof(bf16);
    static constexpr size_t B_BYTES = (size_t)BN * BK * sizeof(bf16);
    static constexpr size_t TILES = STAGES * (A_BYTES + B_BYTES);
    static constexpr bool PATCHES = BN != 128;      // tiles of 128 columns: two CTAs share an SM, which leaves no room for them
    static constexpr size_t TOTAL = TILES + 1024 /* alignment slack */ + 256 /* barriers */ + (PATCHES ? 4 * STAGE_BYTES : 0);
};

// 32 activations per lane and row into out [m, width] at column `col`
__device__ __forceinline__ void store_activations(bf16* out, int width, int col, const float (&act)[32], unsigned char* patch, int row, int m) {
    if (col >= width) return;
    if (patch && (width & 7) == 0 && ((uintptr_t)out & 15) == 0) {
        const int row0 = row - (int)(threadIdx.x & 31);
        store_rows_bf16(patch, act, [&](int r) { return row0 + r < m ? out + (size_t)(row0 + r) * width + col : nullptr; }, (width - col) >> 3);
    } else if (row < m) store_bf16x32(out + (size_t)row * width + col, act, width - col);
}

// A tile's result is taken 32 columns at a time: in units of 32 columns (PLAIN, RELU2), of 32 gate and the 32 up columns of
// the same features (SWIGLU, GATED; where half the tile is no multiple of 32 the last unit begins early and makes some columns a
// second time), or of 32 rotation pairs of a head (ROPE: columns c and c + dim / 2).
template <int EPI>
__device__ __forceinline__ constexpr int epilogue_units(int bn) {
    return EPI == EPI_PLAIN || EPI == EPI_RELU2 ? bn / 32 : paired_rows(EPI) ? (bn / 2 + 31) / 32 : bn / 64;
}
template <int EPI>
__device__ __forceinline__ void unit_columns(const Epilogue& ep, int bn, int unit, int& lo, int& hi) {
    lo = 32 * unit; hi = 0;
    if (paired_rows(EPI)) { lo = min(lo, bn / 2 - 32); hi = bn / 2 + lo; }
    if (EPI == EPI_ROPE) {
        const int per_head = ep.dim / 64;
        lo = (unit / per_head) * ep.dim + (unit % per_head) * 32;
        hi = lo + ep.dim / 2;
    }
}
// The epilogue of units [u0, u1) of an output tile of `bn` columns for one thread: `row` is the thread's output row, n0 the tile's first column
// (feature); load(column, v) gives 32 columns of the row's sums (called by whole warps).
// `pos`, `page` (ROPE): the row's position and the cache page it is written to, looked up by the caller while the tile
// was still being accumulated (-1: a padding row, or a row beyond the step).
template <int EPI, typename Load>
__device__ __forceinline__ void epilogue_tile(const Epilogue& ep, int bn, Load load, int u0, int u1, int row, int m, int n, int n0, int pos, int page,
                                              unsigned char* patch) {
    const int lane = threadIdx.x & 31, row0 = row - lane;
#pragma unroll 1
    for (int unit = u0; unit < u1; ++unit) {
        int lo_col, hi_col;
        unit_columns<EPI>(ep, bn, unit, lo_col, hi_col);
        uint32_t v[32];
        load(lo_col, v);
        if (EPI == EPI_PLAIN) {
            if (ep.out_mult != 0.f) {
#pragma unroll
                for (int j = 0; j < 32; ++j) v[j] = __float_as_uint(__uint_as_float(v[j]) * ep.out_mult);
            }
            const int c = lo_col;
            if (patch && (n & 3) == 0) {
                __syncwarp();                            // the run before has been read
#pragma unroll
                for (int u = 0; u < 8; ++u)
                    *reinterpret_cast<uint4*>(patch + lane * 128 + ((u ^ lane) & 7) * 16) = make_uint4(v[4 * u], v[4 * u + 1], v[4 * u + 2], v[4 * u + 3]);
                __syncwarp();
                const int u = lane & 7, col = n0 + c + 4 * u;
#pragma unroll
                for (int i = 0; i < 8; ++i) {
                    const int r = 4 * i + (lane >> 3);
                    const float4 x = *reinterpret_cast<const float4*>(patch + r * 128 + ((u ^ r) & 7) * 16);
                    if (row0 + r >= m || col >= n) continue;
                    float* dst = ep.out_f32 + (size_t)(row0 + r) * n + col;
                    // The add is done where the element lives (a reduction in L2), so the epilogue does not wait for a load: every
                    // element belongs to this thread alone, and one float add in round-to-nearest is the same sum wherever it is made.
                    if (ep.accumulate) asm volatile("red.global.add.v4.f32 [%0], {%1, %2, %3, %4};" ::"l"(dst), "f"(x.x), "f"(x.y), "f"(x.z), "f"(x.w) : "memory");
                    else *reinterpret_cast<float4*>(dst) = x;
                }
            } else if (row < m) {
                float* dst = ep.out_f32 + (size_t)row * n + n0 + c;
                if (n0 + c + 32 <= n && (n & 3) == 0) {
                    if (ep.accumulate) {
#pragma unroll
                        for (int j = 0; j < 32; j += 4)
                            asm volatile("red.global.add.v4.f32 [%0], {%1, %2, %3, %4};" ::"l"(dst + j), "f"(__uint_as_float(v[j])),
                                         "f"(__uint_as_float(v[j + 1])), "f"(__uint_as_float(v[j + 2])), "f"(__uint_as_float(v[j + 3])) : "memory");
                    } else {
#pragma unroll
                        for (int j = 0; j < 32; j += 4)
                            *reinterpret_cast<float4*>(dst + j) = make_float4(__uint_as_float(v[j]), __uint_as_float(v[j + 1]),
                                                                              __uint_as_float(v[j + 2]), __uint_as_float(v[j + 3]));
                    }
                } else {
#pragma unroll
                    for (int j = 0; j < 32; ++j)
                        if (n0 + c + j < n) dst[j] = ep.accumulate ? dst[j] + __uint_as_float(v[j]) : __uint_as_float(v[j]);
                }
            }
        } else if (EPI == EPI_RELU2) {
            // out = act(product) as bfloat16 [m, n]: the activation of an expert's first product (max(z, 0)^2, or the exact gelu)
            const bool gelu = ep.act == 1;
            float act[32];
#pragma unroll
            for (int j = 0; j < 32; ++j) {
                const float z = __uint_as_float(v[j]), r = fmaxf(z, 0.f);
                act[j] = gelu ? 0.5f * z * (1.f + erff(z * 0.70710678118654752f)) : r * r;
            }
            store_activations(ep.out_bf16, n, n0 + lo_col, act, patch, row, m);
        } else if (paired_rows(EPI)) {
            uint32_t u[32];
            load(hi_col, u);
            float act[32];
            if (EPI == EPI_GATED) {
                // the clamped gated activation of stacked gate and up rows, as bfloat16 [m, inter]
                const float limit = ep.limit, alpha = ep.alpha;
#pragma unroll
                for (int j = 0; j < 32; ++j) {
                    const float gv = fminf(__uint_as_float(v[j]), limit), uv = fminf(fmaxf(__uint_as_float(u[j]), -limit), limit);
                    act[j] = quotient(gv, 1.f + expf(-alpha * gv)) * (uv + 1.f);
                }
            } else {
                // silu(z) = z / (1 + exp(-z)) and gelu(z) = z / (1 + exp(-2 sqrt(2 / pi) (z + 0.044715 z^3))) differ in the exponent only
                const float lin = ep.act == 1 ? 2.f * 0.7978845608028654f : 1.f, cub = ep.act == 1 ? 0.044715f : 0.f;
#pragma unroll
                for (int j = 0; j < 32; ++j) {
                    const float gv = __uint_as_float(v[j]);
                    act[j] = quotient(gv, 1.f + expf(-lin * (gv + cub * gv * gv * gv))) * __uint_as_float(u[j]);
                }
            }
            store_activations(ep.out_bf16, ep.inter, n0 + lo_col, act, patch, row, m);
        } else {
            // whole heads of the stacked q, k, v projection: BN / dim heads per tile, rotation pairs (i, i + dim / 2)
            const int dim = ep.dim, half = dim / 2;
            const int hh = (n0 + lo_col) / dim, c = lo_col % dim;  // head index in the stacked projection, first pair of the unit
            uint32_t hi[32];
            load(hi_col, hi);
            if (hh >= ep.hq + 2 * ep.hkv) break;
            const bool is_q = hh < ep.hq, is_k = !is_q && hh < ep.hq + ep.hkv;
            bf16* dst = nullptr;
            if (row < m) {
                if (is_q) dst = ep.q_out + ((size_t)row * ep.hq + hh) * dim;
                else if (page >= 0) {                               // a missing page entry: a padding row, nothing to write
                    const int kvh = is_k ? hh - ep.hq : hh - ep.hq - ep.hkv;
                    dst = (is_k ? ep.k_cache : ep.v_cache) +
                          (((size_t)page * ep.hkv + kvh) * ep.page_size + pos % ep.page_size) * dim;
                }
            }
            float first[32], second[32];
            if ((is_q || is_k) && row < m) {
                const float4* cs = reinterpret_cast<const float4*>(ep.cos_t + (size_t)row * half + c);   // half is a multiple of 32
                const float4* sn = reinterpret_cast<const float4*>(ep.sin_t + (size_t)row * half + c);
#pragma unroll
                for (int j = 0; j < 32; j += 4) {
                    const float4 cv = cs[j >> 2], sv = sn[j >> 2];
                    const float cc[4] = {cv.x, cv.y, cv.z, cv.w}, ss[4] = {sv.x, sv.y, sv.z, sv.w};
#pragma unroll
                    for (int e = 0; e < 4; ++e) {
                        const float x = __uint_as_float(v[j + e]), y = __uint_as_float(hi[j + e]);
                        first[j + e] = x * cc[e] - y * ss[e];
                        second[j + e] = y * cc[e] + x * ss[e];
                    }
                }
            } else {
#pragma unroll
                for (int j = 0; j < 32; ++j) { first[j] = __uint_as_float(v[j]); second[j] = __uint_as_float(hi[j]); }
            }
            if (patch && !(((uintptr_t)ep.q_out | (uintptr_t)ep.k_cache | (uintptr_t)ep.v_cache) & 15)) {      // heads are 128 bytes and more
                const auto place = [&](int r) { return reinterpret_cast<bf16*>(__shfl_sync(0xffffffffu, reinterpret_cast<unsigned long long>(dst), r)); };
                store_rows_bf16(patch, first, [&](int r) { bf16* p = place(r); return p ? p + c : p; }, 4);
                store_rows_bf16(patch, second, [&](int r) { bf16* p = place(r); return p ? p + half + c : p; }, 4);
            } else if (dst) {
                store_bf16x32(dst + c, first, 32);
                store_bf16x32(dst + half + c, second, 32);
            }
        }
    }
}

// Persistent: a CTA walks output tiles blockIdx.x, blockIdx.x + gridDim.x, ...; the accumulator is double-buffered in
// tensor memory, so the MMA thread fills one buffer while the epilogue warps drain the other.  For PLAIN and RELU2 epilogues.
template <int BN, int STAGES, int EPI>
__global__ void __launch_bounds__(192)
gemm_tcgen05_kernel(const __grid_constant__ CUtensorMap map_a, const __grid_constant__ CUtensorMap map_w,
                    const Epilogue ep, int m, int n, int k, int tiles_m, int tiles_n, int* __restrict__ error) {
    CISR_TRACE_SCOPE(TRACE_GEMM_TCGEN05);
    extern __shared__ unsigned char smem_raw[];
    typedef Smem<BN, STAGES> S;
    unsigned char* tiles = reinterpret_cast<unsigned char*>(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);   // swizzle atoms are 1024-byte aligned
    uint64_t* full_bar = reinterpret_cast<uint64_t*>(tiles + S::TILES);
    uint64_t* empty_bar = full_bar + STAGES;
    uint64_t* acc_full = empty_bar + STAGES;       // [2]: the MMAs of a tile are done
    uint64_t* acc_empty = acc_full + 2;            // [2]: the epilogue has read the buffer
    uint64_t* done = acc_empty + 2;                // giving up: every product issued is done
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(done + 1);

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int k_blocks = (k + BK - 1) / BK;
    const int total_tiles = tiles_m * tiles_n;
    static_assert(EPI == EPI_PLAIN || EPI == EPI_RELU2, "the other epilogues are the split and the pair kernel's");
    // One weight matrix: neighbouring tiles share its rows (and the CTAs running together share few weight tiles and all
    // activations).  Grouped: neighbours share a row tile and its group's weights; in the other order the CTAs running
    // together read every group's activations, more than L2 holds, once per column of tiles (64 experts of 1792 x 4096,
    // 2048 tokens, eight experts each: 385 us, 281 in this order; the products back 235 -> 195).
    const int grouped = ep.tile_group != nullptr;
    auto row_tile = [&](int tile) { return grouped ? tile / tiles_n : tile % tiles_m; };
    auto col_tile = [&](int tile) { return grouped ? tile % tiles_n : tile / tiles_m; };

    if (threadIdx.x == 0) {
        for (int s = 0; s < STAGES; ++s) { mbar_init(full_bar + s, 1); mbar_init(empty_bar + s, 1); }
        for (int b = 0; b < 2; ++b) { mbar_init(acc_full + b, 1); mbar_init(acc_empty + b, 4); }
        mbar_init(done, 1);
        mbar_init_fence();
    }
    if (warp == 1) {    // one warp allocates two accumulators' columns of tensor memory
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)), "r"(tmem_columns(BN)) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    tcgen05_fence_before();
    __syncthreads();
    tcgen05_fence_after();
    const uint32_t tmem_base = *tmem_slot;
    bool ok = true;
    int requested = 0;                             // warp 0: k blocks, over all tiles
    pdl_trigger();      // under programmatic dependent launch the next kernel may begin its own set-up now

    if (warp == 0) {
        if (lane == 0) {
            auto load_b = [&](int s, int kb, int n0) {
                tma_load_2d(tiles + s * (S::A_BYTES + S::B_BYTES) + S::A_BYTES, &map_w, kb * BK, n0, full_bar + s);
            };
            // The weights do not come from the kernel before this one: the first stages' weight tiles are requested
            // before the wait on that kernel, the activation tiles after it.
            // (a grouped product learns its weight rows from the kernel before: nothing is requested early)
            const int early = ep.tile_group ? 0 : (k_blocks < STAGES ? k_blocks : STAGES);
            if (early && (int)blockIdx.x < total_tiles) {
                const int n0 = ((int)blockIdx.x / tiles_m) * BN;
                for (int kb = 0; kb < early; ++kb) {
                    mbar_expect_tx(full_bar + kb, (uint32_t)(S::A_BYTES + S::B_BYTES));
                    load_b(kb, kb, n0);
                }
            }
            pdl_wait();
            CISR_TRACE_WAITED();
            for (int tile = blockIdx.x; tile < total_tiles && ok; tile += gridDim.x) {
                const int m0 = row_tile(tile) * BM, n0 = col_tile(tile) * BN;
                int w_row = n0;
                if (ep.tile_group) {
                    const int group = ep.tile_group[row_tile(tile)];
                    if (group < 0) continue;
                    w_row = group * n + n0;
                }
                for (int kb = 0; kb < k_blocks; ++kb, ++requested) {
                    const int s = requested % STAGES;
                    if (requested < early) {        // this stage's barrier is armed and its weight tile on the way already
                        tma_load_2d(tiles + s * (S::A_BYTES + S::B_BYTES), &map_a, kb * BK, m0, full_bar + s);
                        continue;
                    }
                    ok = mbar_wait(empty_bar + s, ((requested / STAGES) & 1) ^ 1);  // the MMAs that read this stage are done
                    if (!ok) break;
                    mbar_expect_tx(full_bar + s, (uint32_t)(S::A_BYTES + S::B_BYTES));
                    tma_load_2d(tiles + s * (S::A_BYTES + S::B_BYTES), &map_a, kb * BK, m0, full_bar + s);
                    load_b(s, kb, w_row);
                }
            }
        }
    } else if (warp == 1) {
        if (lane == 0) {
            constexpr uint32_t idesc = umma_idesc(BN);
            int kbg = 0, it = 0;
            if (ep.tile_group) pdl_wait();      // the tile list comes from the kernel before
            for (int tile = blockIdx.x; tile < total_tiles && ok; tile += gridDim.x) {
                if (grouped && ep.tile_group[row_tile(tile)] < 0) continue;      // an empty row tile: skipped by every role alike
                const int acc = it & 1;
                ok = mbar_wait(acc_empty + acc, ((it >> 1) & 1) ^ 1);          // the epilogue has drained this buffer
                if (!ok) break;
                tcgen05_fence_after();
                const uint32_t tmem_acc = tmem_base + (uint32_t)(acc * BN);
                for (int kb = 0; kb < k_blocks; ++kb, ++kbg) {
                    const int s = kbg % STAGES;
                    ok = mbar_wait(full_bar + s, (kbg / STAGES) & 1);          // both tiles of this stage have landed
                    if (!ok) break;
                    tcgen05_fence_after();
                    const uint64_t desc_a = umma_desc(tiles + s * (S::A_BYTES + S::B_BYTES));
                    const uint64_t desc_b = umma_desc(tiles + s * (S::A_BYTES + S::B_BYTES) + S::A_BYTES);
#pragma unroll
                    for (int kk = 0; kk < BK / UMMA_K; ++kk)                    // 32 bytes further along K per step
                        umma_bf16(tmem_acc, desc_a + 2 * kk, desc_b + 2 * kk, idesc, (kb | kk) != 0);
                    umma_commit(empty_bar + s);                                // frees the stage when these MMAs finish
                }
                if (ok) umma_commit(acc_full + acc);                           // the whole tile is accumulated
                ++it;
            }
        }
    } else {
        const int quarter = warp & 3;                                          // the 32 lanes this warp may read
        int it = 0;
        pdl_wait();      // outputs may alias what the kernel before still reads
        for (int tile = blockIdx.x; tile < total_tiles && ok; tile += gridDim.x) {
            if (grouped && ep.tile_group[row_tile(tile)] < 0) continue;
            const int acc = it & 1;
            const int m0 = row_tile(tile) * BM, n0 = col_tile(tile) * BN;
            const int row = m0 + quarter * 32 + lane;
            ok = mbar_wait(acc_full + acc, (it >> 1) & 1);
            if (!ok) break;
            tcgen05_fence_after();
            const uint32_t lane_base = tmem_base + (uint32_t)(acc * BN) + ((uint32_t)(quarter * 32) << 16);
            epilogue_tile<EPI>(ep, BN, [&](int c, uint32_t (&v)[32]) { tmem_load32(lane_base + (uint32_t)c, v); }, 0, epilogue_units<EPI>(BN), row, m, n, n0, 0, -1,
                                        S::PATCHES && EPI == EPI_PLAIN ? tiles + S::TILES + 256 + (warp - 2) * STAGE_BYTES : nullptr);
            tcgen05_fence_before();
            __syncwarp();
            if (lane == 0) asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(acc_empty + acc)) : "memory");
            ++it;
        }
    }
    if (!ok && lane == 0) atomicExch(error, 1);
    tcgen05_fence_before();
    if (__syncthreads_or(!ok)) {
        if (threadIdx.x == 0) wait_for_copies(full_bar, requested, STAGES);
        if (threadIdx.x == 32) wait_for_products(done);
        __syncthreads();
    }
    if (warp == 1) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(tmem_columns(BN)) : "memory");
}

// ---------------------------------------------------------------- few tiles: one per CTA, K over a cluster
// For products of one round of CTAs.  A CTA has MT tiles of 128 rows by BN columns (MT accumulators side by side in tensor memory,
// which share every weight tile), and the CTAs of a cluster (1, 2 or 4, along z) an equal share of K each.  The cluster's partial
// sums meet in shared memory: each CTA lays down the units that each other one finishes, in the ring, which its own products have
// left; one barrier.cluster says that every inbox is free; bulk copies bring the runs over; and each CTA adds its units' shares in
// the order of K.  A last barrier.cluster keeps every CTA until its own runs are read.
//
// What bounds it: one SM takes 110 to 150 B/ns from L2, whatever the tile, so a tile's K takes its time however few tiles there
// are.  Narrow tiles (64 columns) and K cut over a cluster put more SMs on the same bytes; the meeting costs 2 us.  us with the
// weights in L2, before (the persistent kernel) and in this one, 64 / 200 / 512 rows: 4096 x 14336 66 / 69 / 75, 28 / 35 / 55;
// 4096 x 4096 22 / 23 / 25, 12 / 14 / 19; 2048 x 8192 38 / 40 / 42, 14 / 16 / 22; 576 x 576 6.6 / 7.2 / 7.4, 4.8 / 6.0 / 6.1.
// The shares of a unit are added 32 columns at a time: with the loop over the shares inside the loop over the columns the
// compiler read them one after the other, 15 us a launch.
template <int BN, int MT, int STAGES>
struct SplitSmem {
    static constexpr size_t A_BYTES = (size_t)MT * BM * BK * sizeof(bf16);
    static constexpr size_t B_BYTES = (size_t)BN * BK * sizeof(bf16);
    static constexpr size_t STAGE = A_BYTES + B_BYTES, TILES = STAGES * STAGE;
    static constexpr size_t TOTAL = TILES + 1024 /* alignment slack */ + 256 /* barriers */;
    // what a CTA sends away and what it receives, (shares - 1) / shares of the tile each, lie side by side in the ring
    static constexpr bool CAN_SPLIT = MT == 1 && BN <= 128;
    static constexpr size_t PATCHES = TILES - 4 * STAGE_BYTES;      // the ring is free by then, but for the runs
    static_assert(!CAN_SPLIT || 2 * (size_t)BN * BM * sizeof(float) * 3 / 4 <= PATCHES, "the runs of four shares");
};

__device__ __forceinline__ void cluster_meet() {
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}

template <int BN, int MT, int STAGES, int EPI>
__global__ void __launch_bounds__(192, 1)
gemm_tcgen05_split_kernel(const __grid_constant__ CUtensorMap map_a, const __grid_constant__ CUtensorMap map_w,
                          const Epilogue ep, int m, int n, int k, int* __restrict__ error) {
    CISR_TRACE_SCOPE(TRACE_GEMM_TCGEN05);
    extern __shared__ unsigned char smem_raw[];
    typedef SplitSmem<BN, MT, STAGES> S;
    unsigned char* tiles = reinterpret_cast<unsigned char*>(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
    uint64_t* full_bar = reinterpret_cast<uint64_t*>(tiles + S::TILES);
    uint64_t* empty_bar = full_bar + STAGES;
    uint64_t* acc_full = empty_bar + STAGES;
    uint64_t* inbox_full = acc_full + 1;                                       // the other CTAs' shares have arrived
    uint64_t* done = inbox_full + 1;                                           // giving up: every product issued is done
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(done + 1);
    constexpr int TILE_N = paired_rows(EPI) ? BN / 2 : BN;
    constexpr int COLUMNS = MT * BN;                                           // of tensor memory: 64 to 512, a power of two
    const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0), lane = threadIdx.x & 31;
    const int shares = (int)gridDim.z, rank = (int)blockIdx.z;                 // the cluster is the z dimension
    const int n0 = (int)blockIdx.x * TILE_N, m0 = (int)blockIdx.y * MT * BM;
    const int all_blocks = (k + BK - 1) / BK, kb0 = all_blocks * rank / shares, k_blocks = all_blocks * (rank + 1) / shares - kb0;

    if (threadIdx.x == 0) {
        for (int s = 0; s < STAGES; ++s) { mbar_init(full_bar + s, 1); mbar_init(empty_bar + s, 1); }
        mbar_init(acc_full, 1);
        mbar_init(inbox_full, 1);
        mbar_init(done, 1);
        mbar_init_fence();
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)), "r"(COLUMNS) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    tcgen05_fence_before();
    __syncthreads();
    tcgen05_fence_after();
    const uint32_t tmem_base = __shfl_sync(0xffffffffu, *tmem_slot, 0);
    bool ok = true;
    int requested = 0;                                                         // warp 0: blocks of K
    pdl_trigger();

    if (warp == 0) {
        auto load_b = [&](int s, int kb) {
            unsigned char* b_tile = tiles + s * S::STAGE + S::A_BYTES;
            if (paired_rows(EPI)) {       // two boxes of BN/2 rows: gate rows n0.., up rows inter + n0..
                tma_load_2d_elect(b_tile, &map_w, (kb0 + kb) * BK, n0, full_bar + s);
                tma_load_2d_elect(b_tile + S::B_BYTES / 2, &map_w, (kb0 + kb) * BK, ep.inter + n0, full_bar + s);
            } else {
                tma_load_2d_elect(b_tile, &map_w, (kb0 + kb) * BK, n0, full_bar + s);
            }
        };
        auto load_a = [&](int s, int kb) {
#pragma unroll
            for (int t = 0; t < MT; ++t) tma_load_2d_elect(tiles + s * S::STAGE + t * (S::A_BYTES / MT), &map_a, (kb0 + kb) * BK, m0 + t * BM, full_bar + s);
        };
        // the weights do not come from the kernel before: the first stages' tiles of them are requested before the wait on it
        const int early = k_blocks < STAGES ? k_blocks : STAGES;
        for (int kb = 0; kb < early; ++kb) {
            mbar_expect_tx_elect(full_bar + kb, (uint32_t)S::STAGE);
            load_b(kb, kb);
        }
        pdl_wait();
        CISR_TRACE_WAITED();
        for (int kb = 0; kb < early; ++kb) load_a(kb, kb);
        requested = early;
        RingAt at{0, 1u};                                    // the second turn
        for (int kb = early; kb < k_blocks; ++kb, at.next(STAGES)) {
            ok = __all_sync(0xffffffffu, mbar_wait(empty_bar + at.stage, at.turn ^ 1));
            if (!ok) break;
            mbar_expect_tx_elect(full_bar + at.stage, (uint32_t)S::STAGE);
            load_a(at.stage, kb);
            load_b(at.stage, kb);
            ++requested;
        }
    } else if (warp == 1) {
        constexpr uint32_t idesc = umma_idesc(BN);
        const uint64_t desc_a = umma_desc(tiles), desc_b = umma_desc(tiles + S::A_BYTES);      // addresses below 256 KB: sums stay in the field
        RingAt ring;
        for (int kb = 0; kb < k_blocks; ++kb, ring.next(STAGES)) {
            ok = __all_sync(0xffffffffu, mbar_wait(full_bar + ring.stage, ring.turn));
            if (!ok) break;
            tcgen05_fence_after();
            const uint64_t at = (uint64_t)ring.stage * (S::STAGE >> 4);
#pragma unroll
            for (int t = 0; t < MT; ++t)
#pragma unroll
                for (int kk = 0; kk < BK / UMMA_K; ++kk)
                    umma_bf16_elect(tmem_base + (uint32_t)(t * BN), desc_a + at + t * (S::A_BYTES / MT >> 4) + 2 * kk, desc_b + at + 2 * kk, idesc, (kb | kk) != 0);
            umma_commit_elect(empty_bar + ring.stage);
        }
        if (ok) umma_commit_elect(acc_full);
    }
    const int quarter = warp & 3;                                              // epilogue warps: the 32 lanes this warp may read
    int pos[MT], page[MT];
    if (warp >= 2) {
        pdl_wait();      // outputs may alias what the kernel before still reads; step metadata is older than that kernel
        // ROPE: where a row's key and value go hangs on four dependent loads of step metadata; they run while the tile is still being accumulated
#pragma unroll
        for (int t = 0; t < MT; ++t) {
            const int row = m0 + t * BM + quarter * 32 + lane;
            pos[t] = 0; page[t] = -1;
            if (EPI == EPI_ROPE && row < m) {
                pos[t] = ep.positions[row];
                page[t] = ep.block_table[(size_t)ep.req_slot[ep.token_req[row]] * ep.table_width + pos[t] / ep.page_size];
            }
        }
        ok = mbar_wait(acc_full, 0);
        tcgen05_fence_after();
    }
    const uint32_t lanes = (uint32_t)(quarter * 32) << 16;
    unsigned char* patch = paired_rows(EPI) ? nullptr : tiles + S::PATCHES + quarter * STAGE_BYTES;
    constexpr int UNITS = epilogue_units<EPI>(BN);
    if (S::CAN_SPLIT && shares > 1) {
        // every thread meets the barriers, also where a wait ran out (its sums are then not written)
        __syncwarp();
        const int per_cta = UNITS / shares, sides = EPI == EPI_PLAIN || EPI == EPI_RELU2 ? 1 : 2;
        const int run = per_cta * sides * 32 * BM;                             // floats that one CTA sends another: [unit][side][32 columns][128 rows]
        float* outbox = reinterpret_cast<float*>(tiles);                       // [shares - 1] runs, by receiver
        float* inbox = outbox + (size_t)(shares - 1) * run;                    // [shares - 1] runs, by sender
        const int row_in = quarter * 32 + lane;
        if (warp >= 2) {
            for (int to = 0; to < shares; ++to) {
                if (to == rank) continue;
                float* box = outbox + (size_t)(to < rank ? to : to - 1) * run + row_in;
                for (int u = 0; u < per_cta; ++u) {
                    int lo, hi;
                    unit_columns<EPI>(ep, BN, to * per_cta + u, lo, hi);
                    for (int side = 0; side < sides; ++side) {
                        uint32_t v[32];
                        tmem_load32(tmem_base + lanes + (uint32_t)(side ? hi : lo), v);
#pragma unroll
                        for (int j = 0; j < 32; ++j) box[j * BM] = __uint_as_float(v[j]);
                        box += 32 * BM;
                    }
                }
            }
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");      // the runs before the copies that read them
            if (warp == 2 && lane == 0) mbar_expect_tx(inbox_full, (uint32_t)((shares - 1) * run * sizeof(float)));
            __syncwarp();
        }
        cluster_meet();                                                        // every CTA's products are done and its runs are written: the inboxes are free
        if (warp == 2 && lane == 0) {
            for (int to = 0; to < shares; ++to) {
                if (to == rank) continue;
                uint32_t there, bar;
                asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(there) : "r"(smem_u32(inbox + (size_t)(rank < to ? rank : rank - 1) * run)), "r"(to));
                asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(bar) : "r"(smem_u32(inbox_full)), "r"(to));
                asm volatile("cp.async.bulk.shared::cluster.shared::cta.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
                             ::"r"(there), "r"(smem_u32(outbox + (size_t)(to < rank ? to : to - 1) * run)), "r"((uint32_t)(run * sizeof(float))), "r"(bar) : "memory");
            }
        }
        __syncwarp();
        if (warp >= 2) {
            ok = mbar_wait(inbox_full, 0) && ok;
            if (__all_sync(0xffffffffu, ok)) {
                const float* next = inbox + row_in;                            // loads come in the order unit, side
                epilogue_tile<EPI>(ep, BN, [&](int c, uint32_t (&v)[32]) {
                    const float* from = next;
                    next += 32 * BM;
#pragma unroll
                    for (int j = 0; j < 32; ++j) v[j] = 0u;
#pragma unroll 1
                    for (int r = 0; r < shares; ++r) {                         // the shares in the order of K
                        uint32_t share[32];
                        if (r == rank) {
                            tmem_load32(tmem_base + lanes + (uint32_t)c, share);
                        } else {
#pragma unroll
                            for (int j = 0; j < 32; ++j) share[j] = __float_as_uint(from[j * BM]);
                            from += run;
                        }
#pragma unroll
                        for (int j = 0; j < 32; ++j) v[j] = __float_as_uint(__uint_as_float(v[j]) + __uint_as_float(share[j]));
                    }
                }, rank * per_cta, (rank + 1) * per_cta, m0 + row_in, m, n, n0, pos[0], page[0], patch);
            }
        }
        __syncwarp();
        cluster_meet();                                                        // every run has arrived: no CTA leaves while its own are read
    } else if (warp >= 2 && ok) {
#pragma unroll
        for (int t = 0; t < MT; ++t) {
            const uint32_t lane_base = tmem_base + lanes + (uint32_t)(t * BN);
            epilogue_tile<EPI>(ep, BN, [&](int c, uint32_t (&v)[32]) { tmem_load32(lane_base + (uint32_t)c, v); }, 0, UNITS,
                                   m0 + t * BM + quarter * 32 + lane, m, n, n0, pos[t], page[t], patch);
        }
    }
    if (!ok && lane == 0) atomicExch(error, 1);
    tcgen05_fence_before();
    if (__syncthreads_or(!ok)) {
        if (warp == 0) wait_for_copies(full_bar, requested, STAGES);
        if (warp == 1) wait_for_products_elect(done);
        __syncthreads();
    }
    if (warp == 1) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(COLUMNS) : "memory");
}

// ---------------------------------------------------------------- large products: a tile on two SMs
// Tiles of 256 rows x bn columns (bn a multiple of 32 up to 256, chosen by pair_choice), one per pair of CTAs that share a TPC.  Each
// CTA brings its 128 rows of A and half of the weight rows into its own shared memory; the products (tcgen05.mma.cta_group::2, M = 256)
// are issued by the pair's first CTA and read both halves, and each CTA's tensor memory receives its own 128 rows by all columns, so
// the epilogue is the one of a 128-row tile.  Persistent, two accumulators per CTA, eight epilogue warps (four per half of the columns).
//
// Barriers: `full` (in the first CTA) counts both CTAs' copies; `empty` and `acc_full` are in both and told by commits that reach both;
// `acc_empty` (in the first CTA) hears the epilogue warps of both.
//
// What bounds it: an SM brings 110 to 150 B/ns from L2, and a 128 x 256 tile on one SM wants 48 KB per 64 of K (512 cycles of products);
// a pair's 256 x 256 tile wants 32 KB per SM.  From there on the tensor cores, at the clock that the power leaves them (a block of K of a 256
// x 256 tile 0.29 us on an idle chip, 0.38 on a busy one), and the last round.  us, 128 x 256 tiles on one SM each and so: gated 14336 x 4096,
// 2048 rows 330 and 315, 1000 rows 201 and 157, 512 rows 111 and 90; gated 8192 x 2048, 2048 rows 100 and 90; plain 6144 x 2048, 2533 rows 67 and
// 50; 8192 x 2048, 2048 rows 65 and 52; 4096 x 14336, 2048 rows 184 and 166.
constexpr int PAIR_STAGES = 6, PAIR_THREADS = 320, PAIR_BN = 256;      // stages of one block of K; half as many of two
struct PairSmem {
    static constexpr size_t A_BYTES = (size_t)BM * BK * sizeof(bf16), B_BYTES = (size_t)PAIR_BN / 2 * BK * sizeof(bf16);
    static constexpr size_t STAGE = A_BYTES + B_BYTES, TILES = PAIR_STAGES * STAGE;
    static constexpr size_t TOTAL = TILES + 1024 /* alignment slack */ + 256 /* barriers */ + 8 * STAGE_BYTES;
};

// The end of a pair's kernel: neither CTA leaves while the other's products read its tiles or its barriers are told.  Where a wait ran out, the first CTA,
// on whose barriers the copies of both complete and which issues the products, waits for both before it meets the other.
__device__ __forceinline__ void meet_pair(bool ok, int rank, int warp, uint64_t* full_bar, int requested, int stages, uint64_t* done, int* error) {
    if (!ok && (threadIdx.x & 31) == 0) atomicExch(error, 1);
    __syncwarp();
    tcgen05_fence_before();
    if (__syncthreads_or(!ok) && rank == 0) {
        if (warp == 0) wait_for_copies(full_bar, requested, stages);
        if (warp == 1) wait_for_products_pair_elect(done);
        __syncwarp();
    }
    cluster_meet();
}

template <int EPI>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(PAIR_THREADS, 1)
gemm_tcgen05_pair_kernel(const __grid_constant__ CUtensorMap map_a, const __grid_constant__ CUtensorMap map_w,
                         const Epilogue ep, int m, int n, int k, int bn, int tiles_m, int tiles_n, int per, int* __restrict__ error) {
    CISR_TRACE_SCOPE(TRACE_GEMM_TCGEN05);
    extern __shared__ unsigned char smem_raw[];
    typedef PairSmem S;
    unsigned char* tiles = reinterpret_cast<unsigned char*>(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
    uint64_t* full_bar = reinterpret_cast<uint64_t*>(tiles + S::TILES);
    uint64_t* empty_bar = full_bar + PAIR_STAGES;
    uint64_t* acc_full = empty_bar + PAIR_STAGES;
    uint64_t* acc_empty = acc_full + 2;
    uint64_t* done = acc_empty + 2;
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(done + 1);

    const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0), lane = threadIdx.x & 31;
    const int rank = (int)blockIdx.x & 1, pair = (int)blockIdx.x >> 1, pairs = (int)gridDim.x >> 1;
    const int stages = PAIR_STAGES / per, k_blocks = (k + per * BK - 1) / (per * BK), total_tiles = tiles_m * tiles_n;
    const int tile_n = paired_rows(EPI) ? bn / 2 : bn;

    if (threadIdx.x == 0) {
        for (int s = 0; s < PAIR_STAGES; ++s) { mbar_init(full_bar + s, 1); mbar_init(empty_bar + s, 1); }
        for (int b = 0; b < 2; ++b) { mbar_init(acc_full + b, 1); mbar_init(acc_empty + b, 16); }
        mbar_init(done, 1);
        mbar_init_fence();
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)), "r"(2 * PAIR_BN) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
    }
    tcgen05_fence_before();
    cluster_meet();                      // both CTAs' barriers are there before either is told anything
    tcgen05_fence_after();
    const uint32_t tmem_base = __shfl_sync(0xffffffffu, *tmem_slot, 0);
    bool ok = true;
    int requested = 0;                   // warp 0: blocks of K, over all tiles
    pdl_trigger();

    if (warp == 0) {
        const uint32_t full_first = in_cluster(full_bar, 0);
        const uint32_t stage_bytes = 2 * per * (uint32_t)(S::A_BYTES + (size_t)bn / 2 * BK * sizeof(bf16));       // of both CTAs
        // this CTA's half of the weight rows: of a tile's columns, or (paired) the gate rows here and the up rows there
        const int w_off = paired_rows(EPI) ? rank * ep.inter : rank * (bn / 2);
        auto load = [&](unsigned char* to, const CUtensorMap* map, int kb, int row, uint32_t bar) {
            if (per == 2) tma_load_3d_pair(to, map, 0, row, 2 * kb, bar);
            else tma_load_2d_pair(to, map, kb * BK, row, bar);
        };
        auto load_b = [&](int s, int kb, int n0) { load(tiles + per * (s * S::STAGE + S::A_BYTES), &map_w, kb, n0 + w_off, full_first + 8 * s); };
        auto load_a = [&](int s, int kb, int m0) { load(tiles + per * s * S::STAGE, &map_a, kb, m0 + rank * BM, full_first + 8 * s); };
        // the first stages' weights are requested before the wait on the kernel before, the activations after it
        const int early = pair < total_tiles ? min(k_blocks, stages) : 0;
        for (int kb = 0; kb < early; ++kb) {
            if (rank == 0) mbar_expect_tx_elect(full_bar + kb, stage_bytes);
            load_b(kb, kb, pair / tiles_m * tile_n);
        }
        pdl_wait();
        CISR_TRACE_WAITED();
        int asked = early;                                       // blocks of the first tile whose weights are on their way
        RingAt at;
        for (int tile = pair; tile < total_tiles && ok; tile += pairs) {
            const int m0 = tile % tiles_m * 2 * BM, n0 = tile / tiles_m * tile_n;
            for (int kb = 0; kb < k_blocks; ++kb, at.next(stages)) {
                if (asked) --asked;
                else {
                    ok = __all_sync(0xffffffffu, mbar_wait(empty_bar + at.stage, at.turn ^ 1));
                    if (!ok) break;
                    if (rank == 0) mbar_expect_tx_elect(full_bar + at.stage, stage_bytes);
                    load_b(at.stage, kb, n0);
                }
                load_a(at.stage, kb, m0);
                ++requested;
            }
        }
    } else if (warp == 1) {
        if (rank == 0) {
            const uint32_t idesc = umma_idesc_pair(bn);
            const uint64_t desc_a = umma_desc(tiles), desc_b = umma_desc(tiles + per * S::A_BYTES);
            const uint32_t b_group = (uint32_t)bn / 2 * BK * sizeof(bf16) >> 4;
            RingAt ring;
            int it = 0;
            for (int tile = pair; tile < total_tiles && ok; tile += pairs, ++it) {
                const int acc = it & 1;
                ok = __all_sync(0xffffffffu, mbar_wait(acc_empty + acc, ((it >> 1) & 1) ^ 1));
                if (!ok) break;
                tcgen05_fence_after();
                const uint32_t tmem_acc = tmem_base + (uint32_t)(acc * PAIR_BN);
                for (int kb = 0; kb < k_blocks; ++kb, ring.next(stages)) {
                    ok = __all_sync(0xffffffffu, mbar_wait(full_bar + ring.stage, ring.turn));
                    if (!ok) break;
                    tcgen05_fence_after();
                    const uint64_t at = (uint64_t)ring.stage * per * (S::STAGE >> 4);
                    for (int g = 0; g < per; ++g)
#pragma unroll
                        for (int kk = 0; kk < BK / UMMA_K; ++kk)
                            umma_bf16_pair_elect(tmem_acc, desc_a + at + g * (S::A_BYTES >> 4) + 2 * kk, desc_b + at + g * b_group + 2 * kk, idesc, (kb | g | kk) != 0);
                    umma_commit_pair_elect(empty_bar + ring.stage);
                }
                if (ok) umma_commit_pair_elect(acc_full + acc);
            }
        }
    } else {
        const int quarter = warp & 3, half = (warp - 2) >> 2;                  // the 32 lanes this warp may read; its half of the columns
        const int units = epilogue_units<EPI>(bn), u0 = half ? (units + 1) / 2 : 0, u1 = half ? units : (units + 1) / 2;
        int it = 0;
        pdl_wait();      // outputs may alias what the kernel before still reads; step metadata is older than that kernel
        for (int tile = pair; tile < total_tiles && ok; tile += pairs, ++it) {
            const int acc = it & 1;
            const int m0 = tile % tiles_m * 2 * BM + rank * BM, n0 = tile / tiles_m * tile_n;
            const int row = m0 + quarter * 32 + lane;
            int pos = 0, page = -1;
            if (EPI == EPI_ROPE && row < m) {
                pos = ep.positions[row];
                page = ep.block_table[(size_t)ep.req_slot[ep.token_req[row]] * ep.table_width + pos / ep.page_size];
            }
            ok = __all_sync(0xffffffffu, mbar_wait(acc_full + acc, (it >> 1) & 1));
            if (!ok) break;
            tcgen05_fence_after();
            const uint32_t lane_base = tmem_base + (uint32_t)(acc * PAIR_BN) + ((uint32_t)(quarter * 32) << 16);
            epilogue_tile<EPI>(ep, bn, [&](int c, uint32_t (&v)[32]) { tmem_load32(lane_base + (uint32_t)c, v); }, u0, u1, row, m, n, n0, pos, page,
                                        tiles + S::TILES + 256 + (warp - 2) * STAGE_BYTES);
            tcgen05_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive_cluster(in_cluster(acc_empty + acc, 0));
        }
    }
    meet_pair(ok, rank, warp, full_bar, requested, stages, done, error);
    if (warp == 1) asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(2 * PAIR_BN) : "memory");
}

// two warps that exchange values meet at a named barrier; both_ok: and whether both are
__device__ __forceinline__ void meet_two(int barrier) { asm volatile("bar.sync %0, 64;" ::"r"(barrier) : "memory"); }
__device__ __forceinline__ bool both_ok(int barrier, bool ok) {
    uint32_t all;
    asm volatile("{\n\t.reg .pred p, q;\n\tsetp.ne.b32 p, %1, 0;\n\tbar.red.and.pred q, %2, 64, p;\n\tselp.u32 %0, 1, 0, q;\n\t}"
                 : "=r"(all) : "r"((uint32_t)ok), "r"(barrier) : "memory");
    return all != 0;
}
// A lane has feature f of the tokens row0, row0 + 1, ...: neighbours put their features together, a lane of two writes every other
// token's.  `left` tokens are there; width (features per row) is even.
template <int TOKENS>
__device__ __forceinline__ void store_columns_bf16(bf16* out, int width, int row0, int left, int f, const float (&act)[TOKENS]) {
    const bool odd = threadIdx.x & 1;
    bf16* dst = out + (size_t)(row0 + odd) * width + (f & ~1);
#pragma unroll
    for (int j = 0; j < TOKENS; j += 2) {
        const float other = __shfl_xor_sync(0xffffffffu, odd ? act[j] : act[j + 1], 1);
        const __nv_bfloat162 p = odd ? __floats2bfloat162_rn(other, act[j + 1]) : __floats2bfloat162_rn(act[j], other);
        if (f < width && j + odd < left) *reinterpret_cast<__nv_bfloat162*>(dst + (size_t)j * width) = p;
    }
}

// ---------------------------------------------------------------- experts: weight rows on the lanes, tokens as columns
// The products of rows sorted by expert (moe_sort), each expert's with its own matrix.  Where the rows are the 128 lanes of a tile an expert's
// rows are padded to whole tiles, a quarter of all products for 256 rows an expert; here a pair of CTAs has 256 weight rows (A) and up to
// 256 of an expert's rows as the columns (B), in steps of 32: tiles [i] = (expert, first row, rows, -), rows 0 from the last one on.  An expert's
// further tiles follow one another, so its weights come from memory once.  Ring, barriers and accumulators as in the pair kernel.
//   PLAIN   out float [rows, n]
//   RELU2   out bfloat16 [rows, n], an activation of the product
//   GATED   w has an expert's gate rows and then its up rows; a CTA's 128 lanes are 64 gate rows and the 64 up rows of the same features,
//           and two epilogue warps exchange halves of their columns, so that each has both for 16 of 32 tokens; out bfloat16 [rows, n / 2]
// us, 2048 tokens, 64 experts of which each token has eight, on rows padded to 128 and so: gated 1792 x 4096 253 and 229, 4096 x 896 165
// and 145 (of which 113 are the bytes at the rate of memory, the float rows most of them).
struct ExpertMaps { CUtensorMap w, rows[8]; };          // rows[i]: boxes of 16 (i + 1) of the sorted rows
template <int EPI>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(PAIR_THREADS, 1)
gemm_tcgen05_experts_kernel(const __grid_constant__ ExpertMaps maps, const Epilogue ep, int n, int k, const int4* __restrict__ tiles_list, int max_tiles,
                            int per, int* __restrict__ error) {
    CISR_TRACE_SCOPE(TRACE_GEMM_TCGEN05);
    extern __shared__ unsigned char smem_raw[];
    typedef PairSmem S;
    unsigned char* tiles = reinterpret_cast<unsigned char*>(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
    uint64_t* full_bar = reinterpret_cast<uint64_t*>(tiles + S::TILES);
    uint64_t* empty_bar = full_bar + PAIR_STAGES;
    uint64_t* acc_full = empty_bar + PAIR_STAGES;
    uint64_t* acc_empty = acc_full + 2;
    uint64_t* done = acc_empty + 2;
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(done + 1);

    const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0), lane = threadIdx.x & 31;
    const int rank = (int)blockIdx.x & 1, pair = (int)blockIdx.x >> 1, pairs = (int)gridDim.x >> 1;
    const int stages = PAIR_STAGES / per, k_blocks = (k + per * BK - 1) / (per * BK);
    const int cols = EPI == EPI_GATED ? n / 2 : n, tile_cols = EPI == EPI_GATED ? BM : 2 * BM, tiles_n = (cols + tile_cols - 1) / tile_cols;
    const int total = max_tiles * tiles_n;

    if (threadIdx.x == 0) {
        for (int s = 0; s < PAIR_STAGES; ++s) { mbar_init(full_bar + s, 1); mbar_init(empty_bar + s, 1); }
        for (int b = 0; b < 2; ++b) { mbar_init(acc_full + b, 1); mbar_init(acc_empty + b, 16); }
        mbar_init(done, 1);
        mbar_init_fence();
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)), "r"(2 * PAIR_BN) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
    }
    tcgen05_fence_before();
    cluster_meet();
    tcgen05_fence_after();
    const uint32_t tmem_base = __shfl_sync(0xffffffffu, *tmem_slot, 0);
    bool ok = true;
    int requested = 0;                   // warp 0: blocks of K, over all tiles
    pdl_trigger();
    pdl_wait();                          // the tiles come from a kernel before
    // item i: the rows of tiles_list[i / tiles_n] with column tile i % tiles_n; every role walks the same items, and asks for the next one's rows early
    const auto rows_of = [&](int item) { return item < total ? tiles_list[item / tiles_n] : make_int4(0, 0, 0, 0); };

    if (warp == 0) {
        const uint32_t full_first = in_cluster(full_bar, 0);
        RingAt at;
        int4 t = rows_of(pair), next;
        for (int item = pair; t.z && ok; item += pairs, t = next) {
            next = rows_of(item + pairs);
            const int f0 = item % tiles_n * tile_cols, half = (t.z + 31) / 32 * 16;      // rows of the tile that each CTA brings
            const int row0 = t.y + rank * half, w_row = t.x * n + f0 + rank * BM, side = f0 + rank * (BM / 2);
            const uint32_t stage_bytes = 2 * per * (uint32_t)(S::A_BYTES + half * BK * sizeof(bf16));
            const CUtensorMap* rows = &maps.rows[half / 16 - 1];
            for (int kb = 0; kb < k_blocks; ++kb, at.next(stages)) {
                unsigned char* stage = tiles + per * at.stage * S::STAGE;
                ok = __all_sync(0xffffffffu, mbar_wait(empty_bar + at.stage, at.turn ^ 1));
                if (!ok) break;
                if (rank == 0) mbar_expect_tx_elect(full_bar + at.stage, stage_bytes);
                const uint32_t bar = full_first + 8 * at.stage;
                if (per == 2) {
                    if (EPI == EPI_GATED) tma_load_4d_pair(stage, &maps.w, 0, side, 2 * t.x, 2 * kb, bar);
                    else tma_load_3d_pair(stage, &maps.w, 0, w_row, 2 * kb, bar);
                    tma_load_3d_pair(stage + 2 * S::A_BYTES, rows, 0, row0, 2 * kb, bar);
                } else {
                    if (EPI == EPI_GATED) {
                        tma_load_2d_pair(stage, &maps.w, kb * BK, t.x * n + side, bar);
                        tma_load_2d_pair(stage + S::A_BYTES / 2, &maps.w, kb * BK, t.x * n + cols + side, bar);
                    } else {
                        tma_load_2d_pair(stage, &maps.w, kb * BK, w_row, bar);
                    }
                    tma_load_2d_pair(stage + S::A_BYTES, rows, kb * BK, row0, bar);
                }
                ++requested;
            }
        }
    } else if (warp == 1) {
        if (rank == 0) {
            const uint64_t desc_a = umma_desc(tiles), desc_b = umma_desc(tiles + per * S::A_BYTES);
            RingAt ring;
            int it = 0;
            int4 t = rows_of(pair), next;
            for (int item = pair; t.z && ok; item += pairs, ++it, t = next) {
                next = rows_of(item + pairs);
                const int acc = it & 1;
                const uint32_t idesc = umma_idesc_pair((t.z + 31) / 32 * 32), b_group = (uint32_t)((t.z + 31) / 32 * 16) * BK * sizeof(bf16) >> 4;
                ok = __all_sync(0xffffffffu, mbar_wait(acc_empty + acc, ((it >> 1) & 1) ^ 1));
                if (!ok) break;
                tcgen05_fence_after();
                const uint32_t tmem_acc = tmem_base + (uint32_t)(acc * PAIR_BN);
                for (int kb = 0; kb < k_blocks; ++kb, ring.next(stages)) {
                    ok = __all_sync(0xffffffffu, mbar_wait(full_bar + ring.stage, ring.turn));
                    if (!ok) break;
                    tcgen05_fence_after();
                    const uint64_t at = (uint64_t)ring.stage * per * (S::STAGE >> 4);
                    for (int g = 0; g < per; ++g)
#pragma unroll
                        for (int kk = 0; kk < BK / UMMA_K; ++kk)
                            umma_bf16_pair_elect(tmem_acc, desc_a + at + g * (S::A_BYTES >> 4) + 2 * kk, desc_b + at + g * b_group + 2 * kk, idesc, (kb | g | kk) != 0);
                    umma_commit_pair_elect(empty_bar + ring.stage);
                }
                if (ok) umma_commit_pair_elect(acc_full + acc);
            }
        }
    } else {
        const int quarter = warp & 3, half = (warp - 2) >> 2;
        unsigned char* patches = tiles + S::TILES + 256;
        float* mine = reinterpret_cast<float*>(patches + (warp - 2) * STAGE_BYTES);      // [2][16 tokens][32 features]: GATED
        const float* theirs = reinterpret_cast<const float*>(patches + ((warp - 2) ^ 2) * STAGE_BYTES);
        const bool up = EPI == EPI_GATED && quarter >= 2;
        const int meeting = 1 + half * 2 + (quarter & 1);                      // the named barrier of two warps that exchange
        int it = 0, turn = 0;
        int4 t = rows_of(pair), next;
        for (int item = pair; t.z && ok; item += pairs, ++it, t = next) {
            next = rows_of(item + pairs);
            const int acc = it & 1, count = t.z, units = (count + 31) / 32;
            const int u0 = half ? (units + 1) / 2 : 0, u1 = half ? units : (units + 1) / 2;
            const int lane_feature = EPI == EPI_GATED ? rank * (BM / 2) + (quarter & 1) * 32 + lane : rank * BM + quarter * 32 + lane;
            const int f = item % tiles_n * tile_cols + lane_feature;
            ok = __all_sync(0xffffffffu, mbar_wait(acc_full + acc, (it >> 1) & 1));
            if (EPI == EPI_GATED) ok = both_ok(meeting, ok);                   // or the one would wait for the other
            if (!ok) break;
            tcgen05_fence_after();
            const uint32_t lane_base = tmem_base + (uint32_t)(acc * PAIR_BN) + ((uint32_t)(quarter * 32) << 16);
            for (int u = u0; u < u1; ++u) {
                uint32_t v[32];
                tmem_load32(lane_base + 32 * u, v);
                if (EPI == EPI_PLAIN) {
                    float* dst = ep.out_f32 + (size_t)(t.y + 32 * u) * n + f;
                    const int left = f < n ? count - 32 * u : 0;
#pragma unroll
                    for (int j = 0; j < 32; ++j)
                        if (j < left) dst[(size_t)j * n] = __uint_as_float(v[j]);
                } else if (EPI == EPI_RELU2) {
                    const bool gelu = ep.act == 1;
                    float act[32];
#pragma unroll
                    for (int j = 0; j < 32; ++j) {
                        const float z = __uint_as_float(v[j]), r = fmaxf(z, 0.f);
                        act[j] = gelu ? 0.5f * z * (1.f + erff(z * 0.70710678118654752f)) : r * r;
                    }
                    store_columns_bf16(ep.out_bf16, n, t.y + 32 * u, count - 32 * u, f, act);
                } else {
                    // the gate warp keeps tokens 0..15 and sends the gates of 16..31, the up warp the other way round
                    float* box = mine + turn * 512;
                    const float* from = theirs + turn * 512;
                    turn ^= 1;
#pragma unroll
                    for (int j = 0; j < 16; ++j) box[j * 32 + lane] = __uint_as_float(up ? v[j] : v[16 + j]);
                    meet_two(meeting);
                    float act[16];
#pragma unroll
                    for (int j = 0; j < 16; ++j) {
                        const float own = __uint_as_float(up ? v[16 + j] : v[j]), other = from[j * 32 + lane];
                        const float gv = fminf(up ? other : own, ep.limit), uv = fminf(fmaxf(up ? own : other, -ep.limit), ep.limit);
                        act[j] = quotient(gv, 1.f + expf(-ep.alpha * gv)) * (uv + 1.f);
                    }
                    const int j0 = 32 * u + (up ? 16 : 0);
                    store_columns_bf16(ep.out_bf16, cols, t.y + j0, count - j0, f, act);
                }
            }
            tcgen05_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive_cluster(in_cluster(acc_empty + acc, 0));
        }
    }
    meet_pair(ok, rank, warp, full_bar, requested, stages, done, error);
    if (warp == 1) asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(2 * PAIR_BN) : "memory");
}

// ---------------------------------------------------------------- host side
bool g_pdl = false;
int* g_error = nullptr;          // device flag, owned by the caller (see cisr_gemm_tcgen05_init)

template <int BN, int STAGES, int EPI>
int launch(const void* a, const void* w, const Epilogue& ep, int m, int n, int k, int tiles_n, cudaStream_t s, int groups = 1) {
    CUtensorMap map_a, map_w;
    int status = cached_map(&map_a, a, m, k, BM);
    if (status) return status;
    if ((status = cached_map(&map_w, w, (long long)groups * n, k, BN))) return status;
    typedef Smem<BN, STAGES> S;
    static bool configured = false;
    if (!configured) {
        cudaError_t e = cudaFuncSetAttribute(gemm_tcgen05_kernel<BN, STAGES, EPI>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)S::TOTAL);
        if (e != cudaSuccess) return (int)e;
        configured = true;
    }
    static int slots = 0;                        // CTAs that fit on the device at once
    if (!slots) {
        int device = 0, sms = 0, per_sm = 0;
        cudaGetDevice(&device);
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device);
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, gemm_tcgen05_kernel<BN, STAGES, EPI>, 192, S::TOTAL);
        per_sm = per_sm < 1 ? 1 : per_sm;
        if (per_sm * tmem_columns(BN) > 512) per_sm = 512 / tmem_columns(BN);      // tensor memory: 512 columns per SM
        slots = sms * per_sm;
    }
    const int tiles_m = (m + BM - 1) / BM, total = tiles_m * tiles_n;
    return launch_kernel(gemm_tcgen05_kernel<BN, STAGES, EPI>, dim3(total < slots ? total : slots), dim3(192), S::TOTAL, s, g_pdl,
                         map_a, map_w, ep, m, n, k, tiles_m, tiles_n, g_error);
}

// Grouped products: 128 x 256 tiles read a third less from L2 per flop than 128 x 128; worth it once there are enough of them to occupy
// most of the device (one CTA per SM at that size).  Three stages of 128 x 128 tiles keep a CTA near 100 KB of shared memory, so that two share an SM
// and one's epilogue overlaps the other's main loop.
bool wide_tiles(int m, int tiles_n256) { return (long long)((m + BM - 1) / BM) * tiles_n256 >= 120; }

template <int BN, int MT, int STAGES, int EPI>
int launch_split(const void* a, const void* w, const Epilogue& ep, int m, int n, int k, int shares, cudaStream_t s) {
    CUtensorMap map_a, map_w;
    int status = cached_map(&map_a, a, m, k, BM);
    if (status) return status;
    if ((status = cached_map(&map_w, w, n, k, paired_rows(EPI) ? BN / 2 : BN))) return status;
    typedef SplitSmem<BN, MT, STAGES> S;
    static bool configured = false;
    if (!configured) {
        cudaError_t e = cudaFuncSetAttribute(gemm_tcgen05_split_kernel<BN, MT, STAGES, EPI>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)S::TOTAL);
        if (e != cudaSuccess) return (int)e;
        configured = true;
    }
    const int cols = paired_rows(EPI) ? n / 2 : n, tile_n = paired_rows(EPI) ? BN / 2 : BN;
    return launch_kernel_cluster(gemm_tcgen05_split_kernel<BN, MT, STAGES, EPI>, dim3((cols + tile_n - 1) / tile_n, (m + MT * BM - 1) / (MT * BM), shares),
                                 dim3(192), S::TOTAL, s, g_pdl, shares, map_a, map_w, ep, m, n, k, g_error);
}

// How the kernel for few tiles takes a product of m rows and cols64 tiles of 64 columns, max64 and max128 the shares of K that tiles
// of 64 and 128 columns can be cut in (0: no such tiles); mt 0: not at all, the pair kernel is better (or CISR_GEMM_DEEP=0).
// - K to 2048 and tiles of 64 columns fit the SMs at one each: those, cut in two from 24 blocks of K on where there is room.  us,
//   64 and 128 columns wide: 576 x 576, 200 rows 6.0 and 7.6; 2048 x 2048, 64 rows 7.6 and 8.7; 512 rows 9.9 and 10.4.
// - tiles of 128 columns fit: K cut in as many shares as fit, of at least eight blocks each.  A longer K wants the wider tiles,
//   which read the activations half as often: 2048 x 8192, 64 rows, 64 CTAs either way: 14 us, 17 with 64 columns.
// - K to 1024 and tiles of 256 columns fit, or do for two row tiles that share them: those, which are done before a pair of CTAs has met.
//   us, here and in the pair kernel: gated 1536 x 576, 1400 rows 9.5 and 10.7; gated 3072 x 1024, 700 rows 12.0 and 12.6; a longer K
//   is the pairs': gated 14336 x 4096, 200 rows 57 and 53.
// - more rows or columns: the pair kernel (2048 x 2048, 700 rows 11.3 here and 13.2 there, 1400 rows 17.2 and 14.9).
// A plain product of at most 64 columns (a router's few outputs) is a column of row tiles: a long K is cut in two where the tiles
// leave room for it (us, 2048 rows of K 2048 12.6 in the persistent kernel and 7.5, of K 4096 21.0 and 10.3; 9472 rows 13.0 and 8.3,
// 21.5 and 11.3); a shorter one, or more row tiles, go to the persistent kernel with tiles of 64 columns (K 1024: 8.3).
struct SplitChoice { int bn, mt, shares; };
SplitChoice split_choice(int m, int cols64, int k, int max64, int max128, int sms) {
    static int on = -1;
    if (on < 0) { const char* e = getenv("CISR_GEMM_DEEP"); on = !(e && e[0] == '0'); }
    const int blocks = (k + BK - 1) / BK, cols128 = (cols64 + 1) / 2;
    const long long tiles_m = (m + BM - 1) / BM, tiles64 = tiles_m * cols64, tiles128 = tiles_m * cols128;
    if (!on) return {0, 0, 0};
    if (cols64 == 1 && max64 >= 2) {
        if (k >= 32 * BK && 2 * tiles64 <= sms) return {64, 1, 2};
        return {0, 0, 0};
    }
    if (max64 && blocks <= 32 && tiles64 <= sms) return {64, 1, max64 >= 2 && blocks >= 24 && 2 * tiles64 <= sms ? 2 : 1};
    if (tiles128 <= sms) {
        int shares = 1;
        while (2 * shares <= max128 && 2 * shares * tiles128 <= sms && blocks >= 16 * shares) shares *= 2;
        return {128, 1, shares};
    }
    if (blocks > 16) return {0, 0, 0};
    if (tiles_m * ((cols128 + 1) / 2) <= sms) return {256, 1, 1};
    if (tiles_m == 2 && (cols128 + 1) / 2 <= sms) return {256, 2, 1};
    return {0, 0, 0};
}
SplitChoice split_choice(int m, int cols64, int k, int max64, int max128) {
    static int sms = 0;
    if (!sms) { int device = 0; cudaGetDevice(&device); cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device); }
    return split_choice(m, cols64, k, max64, max128, sms);
}
template <int EPI>
int launch_split_choice(SplitChoice c, const void* a, const void* w, const Epilogue& ep, int m, int n, int k, cudaStream_t s) {
    if (c.bn == 64) return launch_split<64, 1, 8, EPI>(a, w, ep, m, n, k, c.shares, s);
    if (c.bn == 128) return launch_split<128, 1, 6, EPI>(a, w, ep, m, n, k, c.shares, s);
    return c.mt == 1 ? launch_split<256, 1, 4, EPI>(a, w, ep, m, n, k, 1, s) : launch_split<256, 2, 3, EPI>(a, w, ep, m, n, k, 1, s);
}

// The tile width of the pair kernel for m rows and `cols` output columns (features of a gated product), of the first `widths` bits'
// widths: the one with the least estimate, 3.7 + bn / 59 + c b (r + 0.45 t) us with b blocks of K,
// r rounds and t rounds' worth of tiles over the pairs (a busy chip runs at a lower clock) and c below.  The constants were fitted to 620 plain
// products of 11 sizes and 11 numbers of rows (4.5 %); the width they pick is behind the best of five by 0.2 % on the average of 173 products, plain and
// gated.
int pair_width(int m, int cols, int k, bool paired, unsigned widths, int pairs) {
    static const struct { int bn; double block; } WIDTHS[] = {{256, .254}, {224, .2255}, {192, .199}, {160, .183}, {128, .162}};
    const long long tiles_m = (m + 2 * BM - 1) / (2 * BM);
    int best = 0;
    double least = 0.;
    for (int i = 0; i < 5; ++i) {
        if (!(widths >> i & 1)) continue;
        const int bn = WIDTHS[i].bn, tile = paired ? bn / 2 : bn;
        const long long tiles = tiles_m * ((cols + tile - 1) / tile), rounds = (tiles + pairs - 1) / pairs;
        const double us = 3.7 + bn / 59. + WIDTHS[i].block * ((k + BK - 1) / BK) * (rounds + .45 * tiles / pairs);
        if (!best || us < least) { best = bn; least = us; }
    }
    return best;
}
// rotated: whole heads per tile, 256, 192 or 128 columns, at head size 128 not 192
unsigned pair_widths(int dim) { return dim == 0 ? 0x1f : dim == 64 ? 0x15 : 0x11; }
int device_pairs() {
    static int pairs = 0;
    if (!pairs) { int device = 0, sms = 0; cudaGetDevice(&device); cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device); pairs = sms / 2; }
    return pairs;
}
template <int EPI>
int launch_pair(const void* a, const void* w, const Epilogue& ep, int m, int n, int k, int bn, cudaStream_t s) {
    // Two blocks of K per stage, a box of each operand for both, in the narrowest tiles, whose boxes are small and whose products are done before the next
    // two boxes are on their way: a block of K 0.16 us on an idle chip, 0.21 with a box for each.  Wider ones want the finer ring (3 % at 192).
    const int per = bn < 160 && k % BK == 0 ? 2 : 1;
    CUtensorMap map_a, map_w;
    int status = cached_map(&map_a, a, m, k, BM, per * BK);
    if (status) return status;
    if ((status = cached_map(&map_w, w, n, k, bn / 2, per * BK))) return status;
    static bool configured = false;
    if (!configured) {
        cudaError_t e = cudaFuncSetAttribute(gemm_tcgen05_pair_kernel<EPI>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)PairSmem::TOTAL);
        if (e != cudaSuccess) return (int)e;
        configured = true;
    }
    const int tile_n = paired_rows(EPI) ? bn / 2 : bn, cols = paired_rows(EPI) ? n / 2 : n;
    const int tiles_m = (m + 2 * BM - 1) / (2 * BM), tiles_n = (cols + tile_n - 1) / tile_n, total = tiles_m * tiles_n, pairs = device_pairs();
    return launch_kernel(gemm_tcgen05_pair_kernel<EPI>, dim3(2 * (total < pairs ? total : pairs)), dim3(PAIR_THREADS), PairSmem::TOTAL, s,
                         g_pdl, map_a, map_w, ep, m, n, k, bn, tiles_m, tiles_n, per, g_error);
}

template <int EPI>
int launch_experts(const ExpertMaps& maps, const Epilogue& ep, int n, int k, const int4* tiles, int max_tiles, int items, cudaStream_t s) {
    static bool configured = false;
    if (!configured) {
        const cudaError_t e = cudaFuncSetAttribute(gemm_tcgen05_experts_kernel<EPI>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)PairSmem::TOTAL);
        if (e != cudaSuccess) return (int)e;
        configured = true;
    }
    const int pairs = device_pairs();
    return launch_kernel(gemm_tcgen05_experts_kernel<EPI>, dim3(2 * (items < pairs ? items : pairs)), dim3(PAIR_THREADS), PairSmem::TOTAL, s, g_pdl, maps,
                         ep, n, k, tiles, max_tiles, k % BK ? 1 : 2, g_error);
}

bool operands_ok(const void* a, const void* w, int k) {
    return g_encode && g_error && k > 0 && k % 8 == 0 && !(((uintptr_t)a | (uintptr_t)w) & 15);
}
}  // namespace

// `error_flag`: one zeroed int in device memory that a kernel sets when one of its waits ran out.
CISR_EXPORT int cisr_gemm_tcgen05_init(int* error_flag) {
    if (int status = tma_load_encoder()) return status;
    g_error = error_flag;
    return 0;
}

CISR_EXPORT void cisr_gemm_tcgen05_set_pdl(int on) { g_pdl = on != 0; }

// How the plain product of these sizes is made on a device of `sms` SMs: 0 by a persistent kernel, else the columns of a tile x 100
// + its row tiles x 10 + the shares of K.
CISR_EXPORT int cisr_gemm_tcgen05_plain_choice(int m, int n, int k, int sms) {
    const SplitChoice c = split_choice(m, (n + 63) / 64, k, 2, 4, sms);
    return c.bn * 100 + c.mt * 10 + c.shares;
}

// The columns of the pair kernel's tiles on a device of `sms` SMs; paired: of a gated product of `cols` features; dim: of the rotated projection with
// heads of that size, else 0.
CISR_EXPORT int cisr_gemm_tcgen05_pair_width(int m, int cols, int k, int paired, int dim, int sms) {
    return pair_width(m, cols, k, paired != 0, pair_widths(dim), sms / 2);
}

// How many tensor maps the library remembers before it empties its cache (tests lower it to force evictions).
CISR_EXPORT void cisr_gemm_tcgen05_set_map_cache_limit(int entries) { g_map_cache_limit = entries < 1 ? 1 : (size_t)entries; }

// accumulate != 0: out += a w^T (each output element is read, added to in float and written by the one thread that
// owns it: what the residual add of a layer does, without a pass of its own).  out_mult: the product is multiplied by it
// before it is written or added (1: as it is).
CISR_EXPORT int cisr_gemm_tcgen05(const void* a, const void* w, float* out, int m, int n, int k, int accumulate, float out_mult,
                                  void* stream) {
    if (m <= 0 || n <= 0) return 0;
    if (!g_encode || !g_error) return -13;
    if (!operands_ok(a, w, k) || ((uintptr_t)out & 15)) return -2;
    Epilogue ep = {};
    ep.out_f32 = out; ep.accumulate = accumulate != 0; ep.out_mult = out_mult == 1.f ? 0.f : out_mult;
    cudaStream_t s = (cudaStream_t)stream;
    if (const SplitChoice c = split_choice(m, (n + 63) / 64, k, 2, 4); c.mt) return launch_split_choice<EPI_PLAIN>(c, a, w, ep, m, n, k, s);
    if (n <= 64) return launch<64, 8, EPI_PLAIN>(a, w, ep, m, n, k, 1, s);
    return launch_pair<EPI_PLAIN>(a, w, ep, m, n, k, pair_width(m, n, k, false, pair_widths(0), device_pairs()), s);
}

// w stacks gate rows [0, inter) over up rows [inter, 2 * inter); out (bfloat16 [m, inter]) = act(a gate^T) * (a up^T), act silu (gate_act 0)
// or the tanh form of gelu (1); gate_act 2: the clamped form, g' sigmoid(1.702 g') (u' + 1) with g' = min(g, limit), u' = clamp(u, -limit, limit).
CISR_EXPORT int cisr_gemm_tcgen05_swiglu(const void* a, const void* w, void* out, int m, int inter, int k, int gate_act, float gate_limit,
                                         void* stream) {
    if (m <= 0 || inter <= 0) return 0;
    if (!g_encode || !g_error) return -13;
    if (!operands_ok(a, w, k)) return -2;
    Epilogue ep = {};
    ep.out_bf16 = (bf16*)out; ep.inter = inter; ep.act = gate_act;
    const SplitChoice few = split_choice(m, (inter + 31) / 32, k, 1, 2);
    const int bn = pair_width(m, inter, k, true, pair_widths(0), device_pairs());
    if (gate_act == 2) {
        ep.limit = gate_limit; ep.alpha = 1.702f;
        if (few.mt) return launch_split_choice<EPI_GATED>(few, a, w, ep, m, 2 * inter, k, (cudaStream_t)stream);
        return launch_pair<EPI_GATED>(a, w, ep, m, 2 * inter, k, bn, (cudaStream_t)stream);
    }
    if (few.mt) return launch_split_choice<EPI_SWIGLU>(few, a, w, ep, m, 2 * inter, k, (cudaStream_t)stream);
    return launch_pair<EPI_SWIGLU>(a, w, ep, m, 2 * inter, k, bn, (cudaStream_t)stream);
}

// w stacks the q, k and v heads; q and k heads are rotated (pairs (i, i + dim / 2), cos/sin [m, dim / 2]); q goes to
// q_out [m, hq, dim], k and v to their cache pages.  Takes dim 64 or 128 (whole heads per 128-column tile and 32-column
// halves of the rotation); other head sizes use the plain product and the separate rotation kernel.
CISR_EXPORT int cisr_gemm_tcgen05_rope(const void* a, const void* w, int m, int k, const float* cos_t, const float* sin_t,
                                       void* q_out, void* k_cache, void* v_cache, const int* positions,
                                       const int* token_req, const int* req_slot, const int* block_table,
                                       int table_width, int page_size, int hq, int hkv, int dim, void* stream) {
    if (m <= 0) return 0;
    if (!g_encode || !g_error) return -13;
    if (!operands_ok(a, w, k) || (dim != 64 && dim != 128)) return -2;
    Epilogue ep = {};
    ep.cos_t = cos_t; ep.sin_t = sin_t; ep.q_out = (bf16*)q_out; ep.k_cache = (bf16*)k_cache; ep.v_cache = (bf16*)v_cache;
    ep.positions = positions; ep.token_req = token_req; ep.req_slot = req_slot; ep.block_table = block_table;
    ep.table_width = table_width; ep.page_size = page_size; ep.hq = hq; ep.hkv = hkv; ep.dim = dim;
    const int n = (hq + 2 * hkv) * dim;
    if (const SplitChoice c = split_choice(m, (n + 63) / 64, k, dim == 64 ? 1 : 0, 2); c.mt) return launch_split_choice<EPI_ROPE>(c, a, w, ep, m, n, k, (cudaStream_t)stream);
    return launch_pair<EPI_ROPE>(a, w, ep, m, n, k, pair_width(m, n, k, false, pair_widths(dim), device_pairs()), (cudaStream_t)stream);
}

// The product of rows sorted by group with each group's own weight matrix: a [m, k] with every group's rows padded to
// whole 128-row tiles, w [groups * n, k] (group g's matrix in rows g * n ..), tile_group [m / 128] as described at
// `Epilogue::tile_group`.  relu2 == 0: out is float [m, n] = a_g w_g^T; 1: out is bfloat16 [m, n] = max(a_g w_g^T, 0)^2;
// 2: out is bfloat16 [m, n] = gelu(a_g w_g^T), the exact gelu z Phi(z).
CISR_EXPORT int cisr_gemm_tcgen05_grouped(const void* a, const void* w, void* out, int m, int n, int k, int groups,
                                          const int* tile_group, int relu2, void* stream) {
    if (m <= 0 || n <= 0) return 0;
    if (!g_encode || !g_error) return -13;
    if (!operands_ok(a, w, k) || ((uintptr_t)out & 15) || m % BM || !tile_group || groups <= 0) return -2;
    Epilogue ep = {};
    ep.tile_group = tile_group;
    cudaStream_t s = (cudaStream_t)stream;
    const bool wide = wide_tiles(m, (n + 255) / 256);
    if (relu2) {
        ep.out_bf16 = (bf16*)out;
        ep.act = relu2 == 2 ? 1 : 0;
        if (wide) return launch<256, 4, EPI_RELU2>(a, w, ep, m, n, k, (n + 255) / 256, s, groups);
        return launch<128, 3, EPI_RELU2>(a, w, ep, m, n, k, (n + 127) / 128, s, groups);
    }
    ep.out_f32 = (float*)out;
    if (wide) return launch<256, 4, EPI_PLAIN>(a, w, ep, m, n, k, (n + 255) / 256, s, groups);
    return launch<128, 3, EPI_PLAIN>(a, w, ep, m, n, k, (n + 127) / 128, s, groups);
}

// The products of rows sorted by expert: a [m, k], w [experts * n, k], tiles int4 [max_tiles] = (expert, first row, rows (at most 256), -), compact: rows 0
// from the first unused one on.  act < 0: out float [m, n] = a_e w_e^T; 0, 1: out bfloat16 [m, n] = max(z, 0)^2 or the exact gelu;
// 2: w holds an expert's n / 2 gate and then its n / 2 up rows, out bfloat16 [m, n / 2] = g' sigmoid(alpha g') (u' + 1).
CISR_EXPORT int cisr_gemm_tcgen05_experts(const void* a, const void* w, void* out, int m, int n, int k, int experts, const int* tiles, int max_tiles,
                                          int act, float limit, float alpha, void* stream) {
    if (m <= 0 || n <= 0 || max_tiles <= 0) return 0;
    if (!g_encode || !g_error) return -13;
    if (!operands_ok(a, w, k) || (((uintptr_t)out | (uintptr_t)tiles) & 15) || !tiles || experts <= 0 || n % 4) return -2;
    Epilogue ep = {};
    ep.out_f32 = (float*)out; ep.out_bf16 = (bf16*)out; ep.act = act; ep.limit = limit; ep.alpha = alpha;
    const bool gated = act == 2;
    const int box_cols = k % BK ? BK : 2 * BK;
    ExpertMaps maps;
    int status = cached_map(&maps.w, w, (long long)experts * n, k, gated ? BM / 2 : BM, box_cols, gated && box_cols > BK ? 2 * experts : 1, 2);
    for (int i = 0; i < 8 && !status; ++i) status = cached_map(&maps.rows[i], a, m, k, 16 * (i + 1), box_cols);
    if (status) return status;
    const long long items = (long long)max_tiles * ((n + 2 * BM - 1) / (2 * BM));
    if (items > INT_MAX) return -2;
    const auto go = act < 0 ? launch_experts<EPI_PLAIN> : act == 2 ? launch_experts<EPI_GATED> : launch_experts<EPI_RELU2>;
    return go(maps, ep, n, k, (const int4*)tiles, max_tiles, (int)items, (cudaStream_t)stream);
}
