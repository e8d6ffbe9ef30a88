// Matrix products of few tokens with large weight matrices (bfloat16, float sums): out[M, N] = act[M, K] * w[N, K]^T, M <= 16, on the
// 5th-generation tensor cores with the weight rows as the 128 rows of an accumulator and the tokens as its 16 columns.
//
//   * grid (blocks of 128 weight rows, 1, shares of K); the shares of a block are a cluster.  A block is 128 rows of w (PLAIN, ROPE: one head of
//     128 or two of 64), or 64 gate rows and the 64 up rows of the same features (SWIGLU)
//   * warp 0: TMA copies of 128 of K at a time: the block's rows in ONE box of 32 KB and the tokens in one of 4 KB, into a ring of three stages;
//     the first stages' weights are requested before the wait on the kernel before
//   * warp 1: tcgen05.mma (M = 128, N = 16), the eight products of a block into eight accumulators.  The tensor core cuts a sum instead of
//     rounding it: with all of K in one accumulator the error against 64 bits was 3.6 to 4.5 times that of stream_gemm.cu's eight slices of K (49152 x
//     576 5.2e-7, there 1.5e-7, so 0.9e-7; 16 tokens 13.5 us with one, 13.8 with eight)
//   * warps 2..5: the accumulators, added in float, are a share's sums; they go to shared memory, one barrier.cluster, and each CTA adds the shares of
//     its part of the rows, in the order of K, and runs the epilogue on them
// Two CTAs share an SM: one streams while the other starts or ends.
//
// What bounds it: the weights at the rate of memory.  The persistent kernel of stream_gemm.cu, whose warps multiply by mma.sync, takes longer with
// every token and splits no K.  us in a graph with 1, 8 and 16 tokens, that kernel and this one (floor at 6.55 TB/s): 28672 x 4096 gated 43.7, 50.8,
// 85.2 and 37.5, 38.3, 39.1 (35.9); 4096 x 4096 9.1, 11.7, 17.8 and 7.5, 7.8, 8.1 (5.1); 2048 x 8192 13.7, 24.6, - and 8.6, 8.8, 9.0 (5.1);
// 49152 x 576 17.0, 19.3, 26.8 and 12.0, 12.4, 12.5 (8.6).  Smaller matrices are the latency kernel's (skinny_gemm.cu): 960 x 2560 3.2 there, 3.7 here.
// A share that is all of K writes its sums from tensor memory: through shared memory 49152 x 576 takes 15.8 at 16 tokens, 128256 x 4096 161 (159).
// With 32 or 64 columns it is no longer the better one: 49152 x 576 17.4 and 22.6, the library 12.8 and 13.4.
// Every wait is bounded; one that runs out sets the error flag (code 4), and what the call wrote is not to be used.
#include "skinny_call.cuh"
#include "tcgen05.cuh"

namespace {
typedef __nv_bfloat16 bf16;
enum : int { EPI_PLAIN = 0, EPI_SWIGLU = 1, EPI_ROPE = 2 };
constexpr int TN = 16, BK2 = 128, STAGES = 3, THREADS = 192, EPI_THREADS = 128;
constexpr int SLICES = BK2 / 16, TMEM_COLUMNS = SLICES * TN;      // an accumulator for each sixteen of a block's K
constexpr size_t A_BYTES = (size_t)BM * BK2 * sizeof(bf16), B_BYTES = (size_t)TN * BK2 * sizeof(bf16), STAGE = A_BYTES + B_BYTES;
constexpr size_t SMEM = STAGES * STAGE + 1024 /* alignment slack */ + 128 /* barriers */;
bool g_pdl = false;
int* g_error = nullptr;

struct FewArgs {
    float* out_f32; bf16* out_bf16;
    const float* cos_t; const float* sin_t; bf16* q_out; bf16* k_cache; bf16* v_cache;
    const int* positions; const int* token_req; const int* req_slot; const int* block_table;
    float out_mult, gate_limit;
    int n, m, blocks_k, accumulate, gate_act, table_width, page_size, hq, hkv, dim;
};

__device__ __forceinline__ void cluster_meet() { asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory"); }
__device__ __forceinline__ float load_cluster(uint32_t at) {
    float v;
    asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(v) : "r"(at) : "memory");
    return v;
}

template <int EPI>
__global__ void __launch_bounds__(THREADS, 2)
few_gemm_kernel(const __grid_constant__ CUtensorMap map_w, const __grid_constant__ CUtensorMap map_a, const __grid_constant__ FewArgs a, int* __restrict__ error) {
    CISR_TRACE_SCOPE(TRACE_STREAM_GEMM);
    extern __shared__ unsigned char smem_raw[];
    __shared__ long long cache_row[TN];                    // ROPE: where a token's keys and values go
    unsigned char* ring = reinterpret_cast<unsigned char*>(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
    float* part = reinterpret_cast<float*>(ring);          // [TN][128] this share's sums, where the ring was
    uint64_t* full = reinterpret_cast<uint64_t*>(ring + STAGES * STAGE);
    uint64_t* empty = full + STAGES;
    uint64_t* acc_full = empty + STAGES;
    uint64_t* done = acc_full + 1;                         // giving up: every product issued is done
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(done + 1);
    const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0), lane = threadIdx.x & 31;
    const int block = blockIdx.x, share = blockIdx.z, shares = gridDim.z;
    const int kb0 = a.blocks_k * share / shares, blocks = a.blocks_k * (share + 1) / shares - kb0;
    if (threadIdx.x == 0) {
        for (int s = 0; s < STAGES; ++s) { mbar_init(full + s, 1); mbar_init(empty + s, 1); }
        mbar_init(acc_full, 1);
        mbar_init(done, 1);
        mbar_init_fence();
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)), "r"(TMEM_COLUMNS) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    tcgen05_fence_before();
    __syncthreads();
    tcgen05_fence_after();
    const uint32_t tmem = __shfl_sync(0xffffffffu, *tmem_slot, 0);
    bool ok = true;
    int requested = 0;                                     // warp 0: blocks of K
    pdl_trigger();

    const bool whole = EPI == EPI_PLAIN && shares == 1;    // sums that are the results: from tensor memory to the output
    const auto put = [&](int j, int col, float v) {        // one thread owns an element
        float* dst = a.out_f32 + (size_t)j * a.n + col;
        *dst = a.accumulate ? *dst + v * a.out_mult : v * a.out_mult;
    };
    if (warp == 0) {
        const auto load_w = [&](int s, int kb) {
            if (EPI == EPI_SWIGLU) tma_load_4d_elect(ring + s * STAGE, &map_w, 0, 64 * block, 0, 2 * (kb0 + kb), full + s);
            else tma_load_3d_elect(ring + s * STAGE, &map_w, 0, BM * block, 2 * (kb0 + kb), full + s);
        };
        const auto load_a = [&](int s, int kb) { tma_load_3d_elect(ring + s * STAGE + A_BYTES, &map_a, 0, 0, 2 * (kb0 + kb), full + s); };
        const int early = min(blocks, STAGES);
        for (int kb = 0; kb < early; ++kb) {
            mbar_expect_tx_elect(full + kb, (uint32_t)STAGE);
            load_w(kb, kb);
        }
        pdl_wait();
        CISR_TRACE_WAITED();
        for (int kb = 0; kb < early; ++kb) load_a(kb, kb);
        requested = early;
        int s = 0;
        uint32_t turn = 0;
        for (int kb = early; kb < blocks; ++kb) {
            ok = __all_sync(0xffffffffu, mbar_wait(empty + s, turn));
            if (!ok) break;
            mbar_expect_tx_elect(full + s, (uint32_t)STAGE);
            load_w(s, kb);
            load_a(s, kb);
            ++requested;
            if (++s == STAGES) { s = 0; turn ^= 1u; }
        }
    } else if (warp == 1) {
        constexpr uint32_t idesc = umma_idesc(TN);
        const uint64_t desc_a = umma_desc(ring), desc_b = umma_desc(ring + A_BYTES);
        int s = 0;
        uint32_t turn = 0;
        for (int kb = 0; kb < blocks; ++kb) {
            ok = __all_sync(0xffffffffu, mbar_wait(full + s, turn));
            if (!ok) break;
            tcgen05_fence_after();
            const uint64_t at = (uint64_t)s * (STAGE >> 4);
#pragma unroll
            for (int kk = 0; kk < SLICES; ++kk)
                umma_bf16_elect(tmem + (uint32_t)(kk * TN), desc_a + at + kk / 4 * (A_BYTES / 2 >> 4) + 2 * (kk % 4), desc_b + at + kk / 4 * (B_BYTES / 2 >> 4) + 2 * (kk % 4),
                                idesc, kb != 0);
            umma_commit_elect(empty + s);
            if (++s == STAGES) { s = 0; turn ^= 1u; }
        }
        if (ok) umma_commit_elect(acc_full);
    } else {
        const int quarter = warp & 3;
        pdl_wait();      // outputs may alias what the kernel before still reads
        const int token = threadIdx.x - (THREADS - EPI_THREADS);
        if (EPI == EPI_ROPE && token < a.m) {
            const int pos = a.positions[token], page = a.block_table[(size_t)a.req_slot[a.token_req[token]] * a.table_width + pos / a.page_size];
            cache_row[token] = page < 0 ? -1 : (long long)page * a.hkv * a.page_size + pos % a.page_size;
        }
        __syncwarp();
        ok = __all_sync(0xffffffffu, mbar_wait(acc_full, 0));
        tcgen05_fence_after();
        const int col = block * BM + quarter * 32 + lane;
        if (ok) {
            float v[TN];
#pragma unroll
            for (int q = 0; q < SLICES; q += 2) {              // the slices' sums, rounded where they meet
                uint32_t two[2 * TN];
                tmem_load32(tmem + ((uint32_t)(quarter * 32) << 16) + (uint32_t)(q * TN), two);
#pragma unroll
                for (int j = 0; j < TN; ++j) {
                    const float pair = __uint_as_float(two[j]) + __uint_as_float(two[TN + j]);
                    v[j] = q ? v[j] + pair : pair;
                }
            }
            if (whole) {
#pragma unroll
                for (int j = 0; j < TN; ++j) if (j < a.m && col < a.n) put(j, col, v[j]);
            } else {
#pragma unroll
                for (int j = 0; j < TN; ++j) part[j * BM + quarter * 32 + lane] = v[j];
            }
        }
    }
    __syncwarp();
    tcgen05_fence_before();
    ok = !__syncthreads_or(!ok);
    if (!ok) {
        if (threadIdx.x == 0) atomicExch(error, 4);
        if (warp == 0) wait_for_copies(full, requested, STAGES);
        if (warp == 1) wait_for_products_elect(done);
        __syncthreads();
    }
    if (warp == 1) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(TMEM_COLUMNS) : "memory");
    __syncwarp();
    if (shares > 1) cluster_meet();                        // every share's sums lie in its shared memory
    if (warp >= 2 && ok && !whole) {
        const int tid = threadIdx.x - (THREADS - EPI_THREADS);
        uint32_t from[8];
#pragma unroll
        for (int q = 0; q < 8; ++q) from[q] = in_cluster(part, q < shares ? q : 0);
        const auto sum = [&](int j, int row) {             // over the shares, in the order of K
            if (shares == 1) return part[j * BM + row];
            const uint32_t at = (uint32_t)(j * BM + row) * 4u;
            float v[8];
#pragma unroll
            for (int q = 0; q < 8; ++q) v[q] = q < shares ? load_cluster(from[q] + at) : 0.f;
            float s = v[0];
#pragma unroll
            for (int q = 1; q < 8; ++q) if (q < shares) s += v[q];
            return s;
        };
        const int rows = (EPI == EPI_PLAIN ? BM : BM / 2) / shares, r = share * rows + (tid & (rows - 1));    // this CTA's rows (or pairs of rows) of the block
        const int j0 = tid >> (31 - __clz(rows)), step = EPI_THREADS >> (31 - __clz(rows));
        if (EPI == EPI_PLAIN) {
            const int col = block * BM + r;
            if (col < a.n)
#pragma unroll 1
                for (int j = j0; j < a.m; j += step) put(j, col, sum(j, r));
        } else if (EPI == EPI_SWIGLU) {
            const int f = block * 64 + r, inter = a.n / 2;
            if (f < inter)
#pragma unroll 1
                for (int j = j0; j < a.m; j += step)
                    a.out_bf16[(size_t)j * inter + f] = __float2bfloat16_rn(gated_product(sum(j, r), sum(j, 64 + r), a.gate_act, a.gate_limit));
        } else {
            const int half = a.dim / 2, in_block = r / half, d = r - in_block * half, hh = block * (BM / a.dim) + in_block, lo = in_block * a.dim + d;
            const bool is_q = hh < a.hq, is_k = !is_q && hh < a.hq + a.hkv;
            const int kvh = is_k ? hh - a.hq : hh - a.hq - a.hkv;
            if (hh < a.hq + 2 * a.hkv)
#pragma unroll 1
                for (int j = j0; j < a.m; j += step) {
                    const float x = sum(j, lo), y = sum(j, lo + half);
                    float turned = x, second = y;
                    if (is_q || is_k) {
                        const float c = a.cos_t[(size_t)j * half + d], s = a.sin_t[(size_t)j * half + d];
                        turned = x * c - y * s;
                        second = y * c + x * s;
                    }
                    if (!is_q && cache_row[j] < 0) continue;        // a padding row: its slot holds no pages
                    bf16* dst = is_q ? a.q_out + ((size_t)j * a.hq + hh) * a.dim + d
                                     : (is_k ? a.k_cache : a.v_cache) + ((size_t)cache_row[j] + (size_t)kvh * a.page_size) * a.dim + d;
                    dst[0] = __float2bfloat16_rn(turned);
                    dst[half] = __float2bfloat16_rn(second);
                }
        }
    }
    __syncwarp();
    if (shares > 1) cluster_meet();                        // no CTA leaves while its sums are read
}

int device_sms() {
    static int sms = 0;
    if (!sms) { int device = 0; cudaGetDevice(&device); cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device); }
    return sms;
}
// Shares of K for `blocks` blocks of rows and blocks_k blocks of 128 of K: the most of 1, 2, 4, 8 whose CTAs are on the chip at once, two an SM, with
// two blocks of K each.  us alone with 1, 2, 4, 8 shares, 4 tokens: 2048 x 2048
// 7.8, 6.7, 5.5, 5.5; 4096 x 14336 45.8, 28.8, 23.4, 21.9; 6144 x 2048 (48 blocks) 10.2, 9.5, 8.3, 11.3; 16384 x 2048 gated (128 blocks) 14.1, 14.2,
// 17.2, 22.1.
int few_shares(int blocks, int blocks_k, int sms) {
    int shares = 1;
    while (shares < 8 && 2 * shares * blocks <= 2 * sms && blocks_k >= 4 * shares) shares *= 2;
    return shares;
}

template <int EPI>
int launch(const SkinnyCall& c, const FewArgs& a, int blocks, int shares) {
    CUtensorMap map_w, map_a;
    const bool paired = EPI == EPI_SWIGLU;
    int status = cached_map(&map_w, c.w, c.n, c.k, paired ? BM / 2 : BM, 2 * 64, paired ? 2 : 1, 2);
    if (!status) status = cached_map(&map_a, c.act, c.m, c.k, TN, 2 * 64);
    if (status) return status;
    static bool configured = false;
    if (!configured) {
        const cudaError_t e = cudaFuncSetAttribute(few_gemm_kernel<EPI>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)SMEM);
        if (e != cudaSuccess) return (int)e;
        configured = true;
    }
    return launch_kernel_cluster(few_gemm_kernel<EPI>, dim3(blocks, 1, shares), dim3(THREADS), SMEM, (cudaStream_t)c.stream, g_pdl, shares, map_w, map_a, a, g_error);
}
}  // namespace

CISR_EXPORT int cisr_few_init(int* error_flag) {
    if (int status = tma_load_encoder()) return status;
    g_error = error_flag;
    return 0;
}
CISR_EXPORT void cisr_few_set_pdl(int on) { g_pdl = on != 0; }
CISR_EXPORT int cisr_few_shares(int blocks, int blocks_k, int sms) { return few_shares(blocks, blocks_k, sms); }

// The packed arguments of a weight-streaming product with finished activations (no norm in front).  shares: 0 by the rule.  -2: not a call it takes.
CISR_EXPORT int cisr_few_gemm(const SkinnyCall* call, int shares) {
    const SkinnyCall& c = *call;
    if (c.m <= 0) return 0;
    if (!g_encode || !g_error) return -13;
    if (!c.act || c.m > TN || c.k <= 0 || c.k % 64 || c.n <= 0 || (((uintptr_t)c.w | (uintptr_t)c.act) & 15) || shares < 0 || shares > 8 || (shares & (shares - 1))) return -2;
    FewArgs a = {};
    a.n = c.n; a.m = c.m; a.blocks_k = (c.k + BK2 - 1) / BK2;
    a.out_f32 = (float*)c.out_f32; a.out_bf16 = (bf16*)c.out_bf16; a.out_mult = (float)c.out_mult; a.accumulate = c.accumulate;
    a.gate_act = c.gate_act; a.gate_limit = (float)c.gate_limit;
    a.cos_t = (const float*)c.cos_t; a.sin_t = (const float*)c.sin_t; a.q_out = (bf16*)c.q_out; a.k_cache = (bf16*)c.k_cache; a.v_cache = (bf16*)c.v_cache;
    a.positions = (const int*)c.positions; a.token_req = (const int*)c.token_req; a.req_slot = (const int*)c.req_slot; a.block_table = (const int*)c.block_table;
    a.table_width = c.table_width; a.page_size = c.page_size; a.hq = c.hq; a.hkv = c.hkv; a.dim = c.dim;
    if (c.epilogue == EPI_SWIGLU && c.n != 2 * c.inter) return -2;
    if (c.epilogue == EPI_ROPE && ((c.dim != 64 && c.dim != 128) || 2 * c.rot_half != c.dim || c.interleaved || c.n != (c.hq + 2 * c.hkv) * c.dim)) return -2;
    const int rows = c.epilogue == EPI_SWIGLU ? c.inter : c.n, per = c.epilogue == EPI_SWIGLU ? BM / 2 : BM, blocks = (rows + per - 1) / per;
    if (!shares) shares = few_shares(blocks, a.blocks_k, device_sms());
    if (shares > a.blocks_k) return -2;
    return c.epilogue == EPI_PLAIN ? launch<EPI_PLAIN>(c, a, blocks, shares) : c.epilogue == EPI_SWIGLU
        ? launch<EPI_SWIGLU>(c, a, blocks, shares) : launch<EPI_ROPE>(c, a, blocks, shares);
}
