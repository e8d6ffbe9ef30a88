// Matrix product of float tensors on the 5th-generation tensor cores: out[M, N] = a[M, K] * w[N, K]^T, all float.
//
// Every operand is split into three bfloat16 parts on its way to shared memory, and the six largest of the nine products of parts are taken
// (split_mma.cuh, which says what is lost: a float's own rounding).  A CTA has a tile of 128 x TN (128 or 64) columns and walks K in blocks of 64:
//   * eight warps read the block's rows of both operands (16 bytes an access, a block ahead in registers), split them and lay the parts
//     down as K-major tiles in the 128-byte swizzle, two blocks' worth of room
//   * eight warps add each block's sums to their own in registers, and one of them issues the next block's products before (tcgen05.mma,
//     kind::f16, a block's 24 into one of two accumulators, the smallest parts first).  The tensor core cuts a sum instead of rounding it, so no sum stays there
//     for longer than a block: one rounding per 64 terms, and four of the large products between two
// Sums that are not finite (an infinity, or a float that rounds to a bfloat16 infinity, has NaN among its parts), and sums other than zero below 2^-64
// (operands below about 2^-110 run out of exponents for their parts), are made once more by float multiply-adds.
//
// What bounds it: shared memory, whose 128 bytes a cycle serve the products (8 KB per 128 x 128 x 16), the parts as they are laid down, and
// nothing else: 2300 cycles a block, measured 2700 (1.45 us; 64 columns 1.07).  us, cuBLAS and here: 1000 rows of 960 x 576 29 and 15; 512 rows
// of 16384 x 2048 624 and 236 (146 TFLOP/s, where float multiply-adds reach 74), of 4096 x 14336 1065 and 348.  Error against 64 bits 1.0e-7 at K 576, 1.3e-7
// at 2048, 2.9e-7 at 14336; cuBLAS from 64 rows on 1.6e-7 to 1.1e-6.
#include "split_mma.cuh"
#include "tcgen05.cuh"

namespace {
constexpr int BK = 64, ADD_WARPS = 8, SPLIT_WARPS = 8, THREADS = 32 * (ADD_WARPS + SPLIT_WARPS);
int* g_error = nullptr;          // device flag, owned by the caller

template <int TN>
struct FloatSmem {
    static constexpr size_t A_PLANE = (size_t)BM * BK * 2, B_PLANE = (size_t)TN * BK * 2, BLOCK = 3 * (A_PLANE + B_PLANE);
    static constexpr size_t TOTAL = 2 * BLOCK + 1024 /* alignment slack */ + 128 /* barriers */;
};

__device__ __forceinline__ void arrive(uint64_t* bar) { asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory"); }

// the tile's elements [rows][TN] that the parts may not have carried, by float multiply-adds
__device__ __noinline__ void plain_tile(const float* __restrict__ a, const float* __restrict__ w, float* __restrict__ out, int m0, int n0, int tn, int m, int n, int k) {
    for (int e = threadIdx.x; e < BM * tn; e += THREADS) {
        const int row = m0 + e / tn, col = n0 + e % tn;
        if (row >= m || col >= n || oddness(out[(size_t)row * n + col]) < ODD) continue;
        float sum = 0.f;
        for (int i = 0; i < k; ++i) sum = fmaf(a[(size_t)row * k + i], w[(size_t)col * k + i], sum);
        out[(size_t)row * n + col] = sum;
    }
}

// grid (column tiles, row tiles)
template <int TN>
__global__ void __launch_bounds__(THREADS, 1)
gemm_float_kernel(const float* __restrict__ a, const float* __restrict__ w, float* __restrict__ out, int m, int n, int k, int* __restrict__ error) {
    extern __shared__ unsigned char smem_raw[];
    typedef FloatSmem<TN> S;
    unsigned char* planes = reinterpret_cast<unsigned char*>(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
    uint64_t* full = reinterpret_cast<uint64_t*>(planes + 2 * S::BLOCK);       // [2]: a block's parts are laid down
    uint64_t* empty = full + 2;                                                // [2]: its products have read them
    uint64_t* acc_full = empty + 2;                                            // [2]: its sums are there
    uint64_t* acc_empty = acc_full + 2;                                        // [2]: and have been added
    uint64_t* done = acc_empty + 2;                                            // giving up: every product issued is done
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(done + 1);
    const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0), lane = threadIdx.x & 31;
    const int n0 = (int)blockIdx.x * TN, m0 = (int)blockIdx.y * BM, blocks = (k + BK - 1) / BK;
    if (threadIdx.x == 0) {
        for (int b = 0; b < 2; ++b) { mbar_init(full + b, SPLIT_WARPS); mbar_init(empty + b, 1); mbar_init(acc_full + b, 1); mbar_init(acc_empty + b, ADD_WARPS); }
        mbar_init(done, 1);
        mbar_init_fence();
    }
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)), "r"(2 * TN) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    tcgen05_fence_before();
    __syncthreads();
    tcgen05_fence_after();
    const uint32_t tmem_base = __shfl_sync(0xffffffffu, *tmem_slot, 0);
    bool ok = true, odd = false;

    if (warp < ADD_WARPS) {
        constexpr int COLS = TN / 2;
        const int quarter = warp & 3, half = warp >> 2;                        // the 32 lanes this warp may read; its half of the columns
        const uint32_t mine = tmem_base + ((uint32_t)(quarter * 32) << 16) + (uint32_t)(half * COLS);
        const uint64_t desc_a = umma_desc(planes), desc_b = umma_desc(planes + 3 * S::A_PLANE);
        const auto issue = [&](int kb) {                                       // by warp 0
            constexpr int PART_A[6] = {2, 0, 1, 1, 0, 0}, PART_B[6] = {0, 2, 1, 0, 1, 0};
            constexpr uint32_t idesc = umma_idesc(TN);
            const int b = kb & 1;
            const uint32_t turn = (kb >> 1) & 1;
            if (!__all_sync(0xffffffffu, mbar_wait(full + b, turn) && mbar_wait(acc_empty + b, turn ^ 1))) return false;
            tcgen05_fence_after();
            const uint64_t at = (uint64_t)b * (S::BLOCK >> 4);
#pragma unroll
            for (int p = 0; p < 6; ++p)
#pragma unroll
                for (int kk = 0; kk < BK / 16; ++kk)
                    umma_bf16_elect(tmem_base + (uint32_t)(b * TN), desc_a + at + PART_A[p] * (S::A_PLANE >> 4) + 2 * kk, desc_b + at + PART_B[p] * (S::B_PLANE >> 4) + 2 * kk,
                                    idesc, (p | kk) != 0);
            umma_commit_elect(empty + b);
            umma_commit_elect(acc_full + b);
            return true;
        };
        float sums[COLS];
#pragma unroll
        for (int j = 0; j < COLS; ++j) sums[j] = 0.f;
        if (warp == 0) ok = issue(0);
        for (int kb = 0; kb < blocks && ok; ++kb) {
            const int b = kb & 1;
            if (warp == 0 && kb + 1 < blocks) ok = issue(kb + 1);
            ok = __all_sync(0xffffffffu, mbar_wait(acc_full + b, (kb >> 1) & 1)) && ok;
            if (!ok) break;
            tcgen05_fence_after();
#pragma unroll
            for (int c = 0; c < COLS; c += 32) {
                uint32_t v[32];
                tmem_load32(mine + (uint32_t)(b * TN + c), v);
#pragma unroll
                for (int j = 0; j < 32; ++j) sums[c + j] += __uint_as_float(v[j]);
            }
            tcgen05_fence_before();
            __syncwarp();
            if (lane == 0) arrive(acc_empty + b);
        }
        const int row = m0 + quarter * 32 + lane, col = n0 + half * COLS;
        if (ok && row < m) {
            uint32_t most[2] = {};
#pragma unroll
            for (int j = 0; j < COLS; ++j) most[j & 1] = max(most[j & 1], oddness(sums[j]));
            odd = max(most[0], most[1]) >= ODD;
            float* dst = out + (size_t)row * n + col;
            const bool runs = (n & 3) == 0 && ((uintptr_t)out & 15) == 0;
#pragma unroll
            for (int j = 0; j < COLS; j += 4) {
                if (runs) { if (col + j < n) *reinterpret_cast<float4*>(dst + j) = make_float4(sums[j], sums[j + 1], sums[j + 2], sums[j + 3]); }
                else {
#pragma unroll
                    for (int e = 0; e < 4; ++e) if (col + j + e < n) dst[j + e] = sums[j + e];
                }
            }
        }
    } else {
        // thread t: 16-byte run t % 16 of every sixteenth row
        const int t = threadIdx.x - 32 * ADD_WARPS, r0 = t >> 4, c = (t & 15) * 4;
        constexpr int A_RUNS = BM / 16, B_RUNS = TN / 16;
        float4 ra[A_RUNS], rb[B_RUNS];
        const auto fetch = [&](int kb) {
            const int col = kb * BK + c;
            const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
            for (int i = 0; i < A_RUNS; ++i) {
                const int row = m0 + r0 + 16 * i;
                ra[i] = row < m && col < k ? *reinterpret_cast<const float4*>(a + (size_t)row * k + col) : zero;
            }
#pragma unroll
            for (int i = 0; i < B_RUNS; ++i) {
                const int row = n0 + r0 + 16 * i;
                rb[i] = row < n && col < k ? __ldg(reinterpret_cast<const float4*>(w + (size_t)row * k + col)) : zero;
            }
        };
        const auto put = [&](unsigned char* plane, size_t next, int row, float4 v) {
            uint32_t x[3], y[3];
            split_pair(v.x, v.y, x);
            split_pair(v.z, v.w, y);
            unsigned char* at = plane + row * 128 + (((c >> 3) ^ (row & 7)) << 4) + (c & 4) * 2;
#pragma unroll
            for (int p = 0; p < 3; ++p) *reinterpret_cast<uint2*>(at + p * next) = make_uint2(x[p], y[p]);
        };
        fetch(0);
        for (int kb = 0; kb < blocks; ++kb) {
            const int b = kb & 1;
            ok = __all_sync(0xffffffffu, mbar_wait(empty + b, ((kb >> 1) & 1) ^ 1));
            if (!ok) break;
            unsigned char* to = planes + b * S::BLOCK;
#pragma unroll
            for (int i = 0; i < A_RUNS; ++i) put(to, S::A_PLANE, r0 + 16 * i, ra[i]);
#pragma unroll
            for (int i = 0; i < B_RUNS; ++i) put(to + 3 * S::A_PLANE, S::B_PLANE, r0 + 16 * i, rb[i]);
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");      // the parts before the tensor core reads them
            __syncwarp();
            if (lane == 0) arrive(full + b);
            if (kb + 1 < blocks) fetch(kb + 1);
        }
    }
    if (!ok && lane == 0) atomicExch(error, 1);
    __syncwarp();
    tcgen05_fence_before();
    const int again = __syncthreads_or(odd);
    if (__syncthreads_or(!ok)) {
        if (warp == 0) wait_for_products_elect(done);
        __syncthreads();
    }
    if (warp == 0) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(2 * TN) : "memory");
    if (again) plain_tile(a, w, out, m0, n0, TN, m, n, k);
}

template <int TN>
int launch(const float* a, const float* w, float* out, int m, int n, int k, cudaStream_t s) {
    static bool configured = false;
    if (!configured) {
        const cudaError_t e = cudaFuncSetAttribute(gemm_float_kernel<TN>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)FloatSmem<TN>::TOTAL);
        if (e != cudaSuccess) return (int)e;
        configured = true;
    }
    return launch_kernel(gemm_float_kernel<TN>, dim3((n + TN - 1) / TN, (m + BM - 1) / BM), dim3(THREADS), FloatSmem<TN>::TOTAL, s, false, a, w, out, m, n, k, g_error);
}
}  // namespace

// `error_flag`: one zeroed int in device memory that a kernel sets when one of its waits ran out.
CISR_EXPORT int cisr_gemm_float_init(int* error_flag) { g_error = error_flag; return 0; }

// `narrow`: tiles of 64 columns.  K a multiple of 4, a and w 16-byte aligned.
CISR_EXPORT int cisr_gemm_float(const float* a, const float* w, float* out, int m, int n, int k, int narrow, void* stream) {
    if (m <= 0 || n <= 0) return 0;
    if (!g_error) return -13;
    if (k <= 0 || k % 4 || (((uintptr_t)a | (uintptr_t)w) & 15) || (m + BM - 1) / BM > 65535) return -2;
    return narrow ? launch<64>(a, w, out, m, n, k, (cudaStream_t)stream) : launch<128>(a, w, out, m, n, k, (cudaStream_t)stream);
}
