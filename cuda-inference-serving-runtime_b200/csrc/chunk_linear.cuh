// The chunk products of the recurrences with a matrix state per head (gated_linear.cu, lightning.cu).  For a chunk of n <= 64
// tokens with S0 the state before it, L_t the sum of the logarithms of the decays up to token t, and gains g:
//     gain    sum_i exp(L_n - L_i) g_i k_i v_i^T             128 columns of [N, dv] per CTA
//     scores  q_t . k_i                                      in the gain's CTAs of a group's first head, which have the keys at hand
//     read    exp(L_t) S0^T q_t + sum_{i <= t} exp(L_t - L_i) g_i (q_t . k_i) v_i     64 tokens x 128 value columns per CTA
// Every product is 64 x 64 x 64 at a time, float on the tensor cores (split_mma.cuh), 256 threads, two CTAs an SM.  Few chunks and heads: 64
// columns and one tile of rows per CTA (ChunkArgs::narrow).
// What bounds it: the products (0.48 of mma.sync an SM and cycle: 17,000 of a CTA's 38,000 cycles in `gains`, two CTAs an SM), and the loads in
// front of them, which all CTAs of a round wait for together (10,000).
// Measured at 2048 tokens: lightning, 16 heads of 128 x 128, gains with scores 50 us and reads 45 (a CTA per tile of 64 x 64, which loads
// and splits every operand tile two to four times: 57 and 48; on the CUDA cores 57 without scores and 141); a matrix memory
// of 8 heads of 128 x 256, 2100 tokens, 39 and 44 (46 and 47).
#pragma once
#include "split_mma.cuh"

namespace {
constexpr int CHUNK = 64;
constexpr int CHUNK_THREADS = 256;
constexpr int CHUNK_COLUMNS = 128;                     // value columns per CTA: two tiles
constexpr size_t GAINS_SMEM = 4 * sizeof(SplitTile), READS_SMEM = 3 * sizeof(SplitTile);

struct ChunkArgs {
    const float* q; const float* k; const float* v;      // at their first column; rows of `*_stride` floats
    int q_stride, k_stride, v_stride;
    const float* la; const float* g;                     // [tokens][heads]: logarithms of the decays, gains; null:
    const float* decay;                                  // [heads] one decay per head, gains of one
    float* state; long long state_stride;
    const int* req_slot; const int* q_start; const int* q_len;
    const int* chunk_req; const int* chunk_t0; const int* req_chunk0;
    float* scores;                                       // [chunks][groups][CHUNK][CHUNK]
    float* blocks;                                       // [chunks][heads][N * dv (+ N)]
    float* chunk_decay;                                  // [chunks][heads] (may be null)
    float* y; float* yn;                                 // [tokens][heads][dv], [tokens][heads]
    float q_scale;
    int heads, groups, N, dv, least;
    int narrow;                                          // few CTAs: 64 value columns and one tile of rows in each, the scores in CTAs of their own
};

__device__ __forceinline__ float chunk_silu(float z) { return quotient(z, 1.f + expf(-z)); }

// Rows [0, nr) x columns [0, nc) of src (row stride `stride`), zeros elsewhere: asked for, and later put into a tile, so that
// several tiles' loads are on their way together.  put: silu of each where asked, then each row times weight(row).
constexpr int PER_THREAD = CHUNK * CHUNK / 4 / CHUNK_THREADS;        // runs of four floats of a tile per thread
struct RawTile { float4 v[PER_THREAD]; };
template <bool VEC>
__device__ __forceinline__ void fetch_tile(RawTile& raw, const float* __restrict__ src, size_t stride, int nr, int nc) {
#pragma unroll
    for (int u = 0; u < PER_THREAD; ++u) {
        const int i = threadIdx.x + u * CHUNK_THREADS, r = i >> 4, c = (i & 15) * 4;
        const float* p = src + (size_t)r * stride + c;
        if (VEC) {
            raw.v[u] = (r < nr && c < nc) ? *reinterpret_cast<const float4*>(p) : make_float4(0.f, 0.f, 0.f, 0.f);
        } else {
            raw.v[u].x = (r < nr && c < nc) ? p[0] : 0.f; raw.v[u].y = (r < nr && c + 1 < nc) ? p[1] : 0.f;
            raw.v[u].z = (r < nr && c + 2 < nc) ? p[2] : 0.f; raw.v[u].w = (r < nr && c + 3 < nc) ? p[3] : 0.f;
        }
    }
}
template <bool SILU, bool PLAIN, typename W>
__device__ __forceinline__ void put_tile(SplitTile& dst, const RawTile& raw, W weight) {
#pragma unroll
    for (int u = 0; u < PER_THREAD; ++u) {
        const int i = threadIdx.x + u * CHUNK_THREADS, r = i >> 4, c = (i & 15) * 4;
        float4 v = raw.v[u];
        if (SILU) { v.x = chunk_silu(v.x); v.y = chunk_silu(v.y); v.z = chunk_silu(v.z); v.w = chunk_silu(v.w); }
        const float w = weight(r);
        tile_store4<PLAIN>(dst, r, c, make_float4(v.x * w, v.y * w, v.z * w, v.w * w));
    }
}
struct One { __device__ __forceinline__ float operator()(int) const { return 1.f; } };

// L [CHUNK]: sums of the logarithms up to each token of the chunk, in double: their differences are what counts, and behind a
// run of strong decays a float sum would have lost the digits of the weak ones.  Tokens beyond the portion add nothing.
// `gain` receives g (zero beyond the portion).
__device__ __forceinline__ void stage_decays(const ChunkArgs& a, int h, int token0, int n, double* L, float* gain) {
    if (threadIdx.x < 32) {
        const int t = 2 * threadIdx.x;
        if (a.decay) {
            // a decay of zero: a logarithm whose differences are 0 for a token itself and give a factor of 0 before it
            const double lg = a.decay[h] == 0.f ? -1e5 : log((double)a.decay[h]);
            L[t] = lg * min(t + 1, n);
            L[t + 1] = lg * min(t + 2, n);
        } else {
            const double x = t < n ? (double)a.la[(size_t)(token0 + t) * a.heads + h] : 0.0;
            const double y = t + 1 < n ? (double)a.la[(size_t)(token0 + t + 1) * a.heads + h] : 0.0;
            double sum = x + y;
#pragma unroll
            for (int off = 1; off < 32; off <<= 1) {
                const double before = __shfl_up_sync(0xffffffffu, sum, off);
                if ((int)threadIdx.x >= off) sum += before;
            }
            L[t + 1] = sum;
            L[t] = sum - y;
        }
    } else if (threadIdx.x >= 64 && threadIdx.x < 64 + CHUNK) {
        const int t = threadIdx.x - 64;
        gain[t] = t < n ? (a.decay ? 1.f : a.g[(size_t)(token0 + t) * a.heads + h]) : 0.f;
    }
}

// a warp's 16 x 32 part of a 64 x 64 result, element pairs (row, col, col + 1) handed to `put`
template <typename P>
__device__ __forceinline__ void for_result(const float (&acc)[4][4], int m0, int n0, P put) {
    const int lane = threadIdx.x & 31;
#pragma unroll
    for (int half = 0; half < 2; ++half)
#pragma unroll
        for (int j = 0; j < 4; ++j) put(m0 + 8 * half + (lane >> 2), n0 + 8 * j + 2 * (lane & 3), acc[j][2 * half], acc[j][2 * half + 1]);
}
template <bool VEC>
__device__ __forceinline__ void put_pair(float* dst, int left, float x, float y) {       // `left` columns are there (VEC: an even number)
    if (VEC) {
        if (left > 0) *reinterpret_cast<float2*>(dst) = make_float2(x, y);
    } else {
        if (left > 0) dst[0] = x;
        if (left > 1) dst[1] = y;
    }
}

// How a launch of few chunks and heads is cut: with the wide CTAs (a tile of the values split once for all of a head's rows) it would leave
// SMs empty.  us, narrow and wide: two portions of 500 tokens, 8 heads of 128 x 64, gains 6.1 and 9.9; 2048 tokens, 16 heads of 128 x 128,
// gains 57 and 50, reads 48 and 45.
inline bool chunk_narrow(const ChunkArgs& a, int n_chunks) {
    static int sms = 0;
    if (!sms) { int device = 0; cudaGetDevice(&device); cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device); }
    return (long long)n_chunks * a.heads * ((a.dv + CHUNK_COLUMNS - 1) / CHUNK_COLUMNS) < 2 * sms;
}

// grid (chunk, head, 128 value columns): the gain, and in the CTAs of a group's first head the group's scores q_t . k_i, every pair of tokens
struct GainShared { double L[CHUNK]; float w[CHUNK], sums[4][CHUNK]; };
template <bool VEC, bool NORM, bool SILU, bool PLAIN>
__device__ __forceinline__ int gains_pass(const ChunkArgs& a, GainShared& sh) {
    extern __shared__ __align__(16) unsigned char chunk_smem[];
    double* L = sh.L;
    float* w = sh.w;
    SplitTile* V = reinterpret_cast<SplitTile*>(chunk_smem);       // [2]
    SplitTile &K = V[2], &Q = V[3];
    const int chunk = blockIdx.x, h = blockIdx.y, z = blockIdx.z, tid = threadIdx.x, warp = tid >> 5, m0 = 16 * (warp >> 1), n0w = 32 * (warp & 1);
    const int per_group = a.heads / a.groups, grp = h / per_group, row_tiles = (a.N + CHUNK - 1) / CHUNK;
    const bool only_scores = a.narrow && z == (int)gridDim.z - 1;
    const int c0 = only_scores ? 0 : a.narrow ? z / row_tiles * CHUNK : z * CHUNK_COLUMNS;
    const int row0 = a.narrow && !only_scores ? z % row_tiles * CHUNK : 0, row1 = a.narrow && !only_scores ? min(a.N, row0 + CHUNK) : a.N;
    const bool scores = (a.narrow ? only_scores : z == 0) && h == grp * per_group, norm_here = NORM && c0 == 0 && !only_scores;
    if (only_scores && !scores) return 0;
    const int r = a.chunk_req[chunk], t0 = a.chunk_t0[chunk], n = min(CHUNK, a.q_len[r] - t0);
    const int token0 = a.q_start[r] + t0, n_tiles = only_scores ? 0 : a.narrow || a.dv - c0 <= CHUNK ? 1 : 2;
    const float* ks = a.k + (size_t)token0 * a.k_stride + grp * a.N;
    const float* qs = a.q + (size_t)token0 * a.q_stride + grp * a.N;
    const float* vs = a.v + (size_t)token0 * a.v_stride + h * a.dv + c0;
    if (!PLAIN) pdl_wait();
    RawTile k, q;
    float sc[4][4] = {};
    int bad = 0;
    {
        RawTile v[2];
        fetch_tile<VEC>(k, ks + row0, a.k_stride, n, min(CHUNK, a.N - row0));
#pragma unroll
        for (int t = 0; t < 2; ++t) fetch_tile<VEC>(v[t], vs + t * CHUNK, a.v_stride, n, t < n_tiles ? a.dv - c0 - t * CHUNK : 0);
        if (scores) fetch_tile<VEC>(q, qs, a.q_stride, n, min(CHUNK, a.N));
        stage_decays(a, h, token0, n, L, w);
        __syncthreads();
        if (tid < CHUNK) w[tid] *= expf((float)(L[CHUNK - 1] - L[tid]));
        if (a.chunk_decay && z == 0 && tid == 0) a.chunk_decay[(size_t)chunk * a.heads + h] = expf((float)L[CHUNK - 1]);
        __syncthreads();
#pragma unroll
        for (int t = 0; t < 2; ++t)
            if (t < n_tiles) put_tile<SILU, PLAIN>(V[t], v[t], [&](int i) { return w[i]; });
    }
    const size_t per_head = (size_t)a.N * a.dv + (NORM ? a.N : 0);
    float* out = a.blocks + ((size_t)chunk * a.heads + h) * per_head;
    for (int n0 = row0; n0 < row1; n0 += CHUNK) {
        const int nr = min(CHUNK, a.N - n0);
        if (n0 > row0) __syncthreads();                              // the tiles before have been multiplied
        put_tile<SILU, PLAIN>(K, k, One());
        if (scores) put_tile<SILU, PLAIN>(Q, q, One());
        __syncthreads();
        if (n0 + CHUNK < row1) {                                     // on their way during the products
            fetch_tile<VEC>(k, ks + n0 + CHUNK, a.k_stride, n, a.N - n0 - CHUNK);
            if (scores) fetch_tile<VEC>(q, qs + n0 + CHUNK, a.q_stride, n, a.N - n0 - CHUNK);
        }
        for (int t = 0; t < n_tiles; ++t) {
            float acc[4][4] = {};
            tile_product<PLAIN, true, true>(acc, K, V[t], m0, n0w, (n + 15) >> 4);
            const int c1 = c0 + t * CHUNK, nc = a.dv - c1;
            for_result(acc, m0, n0w, [&](int row, int c, float x, float y) {
                if (row < nr) put_pair<VEC>(out + (size_t)(n0 + row) * a.dv + c1 + c, nc - c, x, y);
            });
            bad |= not_finite(acc);
        }
        if (scores && n0w <= m0 + 15) tile_product<PLAIN, false, false>(sc, Q, K, m0, n0w, (nr + 15) >> 4);      // pairs with i > t are never read
        if (norm_here) {                                             // four threads a column, sixteen tokens each
            const int c = tid & 63, part = tid >> 6;
            float sum = 0.f;
#pragma unroll 4
            for (int i = 16 * part; i < 16 * part + 16; ++i) sum = fmaf(w[i], tile_value<PLAIN>(K, i, c), sum);
            sh.sums[part][c] = sum;
            __syncthreads();
            if (tid < nr) out[(size_t)a.N * a.dv + n0 + tid] = (sh.sums[0][tid] + sh.sums[1][tid]) + (sh.sums[2][tid] + sh.sums[3][tid]);
        }
    }
    if (scores) {
        float* to = a.scores + ((size_t)chunk * a.groups + grp) * CHUNK * CHUNK;
        for_result(sc, m0, n0w, [&](int t, int i, float x, float y) { *reinterpret_cast<float2*>(to + t * CHUNK + i) = make_float2(x, y); });
        bad |= not_finite(sc);
    }
    return bad;
}
template <bool VEC, bool NORM, bool SILU>
__device__ __noinline__ void gains_plain(const ChunkArgs& a, GainShared& sh) { gains_pass<VEC, NORM, SILU, true>(a, sh); }
template <bool VEC, bool NORM, bool SILU>
__global__ void __launch_bounds__(CHUNK_THREADS, 2)
chunk_gains_kernel(const __grid_constant__ ChunkArgs a) {
    __shared__ GainShared sh;
    pdl_trigger();
    if (__syncthreads_or(gains_pass<VEC, NORM, SILU, false>(a, sh))) gains_plain<VEC, NORM, SILU>(a, sh);
}

// grid (chunk, head, 128 value columns): the running product of [q exp(L) | scores with their decays] and [S0 ; v]
struct ReadShared { double L[CHUNK]; float gain[CHUNK], carried[CHUNK], nvec[CHUNK]; };
template <bool VEC, bool NORM, bool SILU, bool PLAIN>
__device__ __forceinline__ int reads_pass(const ChunkArgs& a, ReadShared& sh) {
    extern __shared__ __align__(16) unsigned char chunk_smem[];
    double* L = sh.L;
    float *gain = sh.gain, *carried = sh.carried, *nvec = sh.nvec;
    SplitTile& A = reinterpret_cast<SplitTile*>(chunk_smem)[0];
    SplitTile* B = reinterpret_cast<SplitTile*>(chunk_smem) + 1;   // [2]
    const int chunk = blockIdx.x, h = blockIdx.y, c0 = blockIdx.z * (a.narrow ? CHUNK : CHUNK_COLUMNS), tid = threadIdx.x, warp = tid >> 5, m0 = 16 * (warp >> 1), n0w = 32 * (warp & 1);
    const int grp = h / (a.heads / a.groups), n_tiles = a.narrow || a.dv - c0 <= CHUNK ? 1 : 2;
    const int r = a.chunk_req[chunk], t0 = a.chunk_t0[chunk], n = min(CHUNK, a.q_len[r] - t0);
    const int token0 = a.q_start[r] + t0;
    const size_t per_head = (size_t)a.N * a.dv + (NORM ? a.N : 0);
    const float* block = a.blocks + ((size_t)chunk * a.heads + h) * per_head;
    const bool norm_here = NORM && c0 == 0;
    const int nt = tid >> 2, nq = (tid & 3) * 16;             // normaliser: four threads per token, a quarter of a row each
    if (!PLAIN) pdl_wait();
    float norm = 0.f;
    stage_decays(a, h, token0, n, L, gain);
    float acc[2][4][4] = {};
    for (int n0 = 0; n0 < a.N; n0 += CHUNK) {
        const int nr = min(CHUNK, a.N - n0);
        RawTile q, s0[2];
        fetch_tile<VEC>(q, a.q + (size_t)token0 * a.q_stride + grp * a.N + n0, a.q_stride, n, nr);
#pragma unroll
        for (int t = 0; t < 2; ++t) fetch_tile<VEC>(s0[t], block + (size_t)n0 * a.dv + c0 + t * CHUNK, a.dv, nr, t < n_tiles ? a.dv - c0 - t * CHUNK : 0);
        if (n0) __syncthreads();
        put_tile<SILU, PLAIN>(A, q, One());
#pragma unroll
        for (int t = 0; t < 2; ++t)
            if (t < n_tiles) put_tile<false, PLAIN>(B[t], s0[t], One());
        if (norm_here && tid < CHUNK) nvec[tid] = tid < nr ? block[(size_t)a.N * a.dv + n0 + tid] : 0.f;
        __syncthreads();
#pragma unroll
        for (int t = 0; t < 2; ++t)
            if (t < n_tiles) tile_product<PLAIN, false, true>(acc[t], A, B[t], m0, n0w, (nr + 15) >> 4);
        if (norm_here)
            for (int i = 0; i < 16; i += 8) {
                float q[8];
                tile_read8<PLAIN>(A, nt, nq + i, q);
#pragma unroll
                for (int e = 0; e < 8; ++e) norm = fmaf(q[e], nvec[nq + i + e], norm);
            }
    }
    const float* G = a.scores + ((size_t)chunk * a.groups + grp) * CHUNK * CHUNK;
    RawTile v[2], sc;
#pragma unroll
    for (int t = 0; t < 2; ++t) fetch_tile<VEC>(v[t], a.v + (size_t)token0 * a.v_stride + h * a.dv + c0 + t * CHUNK, a.v_stride, n, t < n_tiles ? a.dv - c0 - t * CHUNK : 0);
    fetch_tile<true>(sc, G, CHUNK, CHUNK, CHUNK);
    if (tid < CHUNK) carried[tid] = expf((float)L[tid]);
    __syncthreads();
#pragma unroll
    for (int half = 0; half < 2; ++half) {
        const float f = carried[m0 + 8 * half + ((tid & 31) >> 2)];
#pragma unroll
        for (int t = 0; t < 2; ++t)
#pragma unroll
            for (int j = 0; j < 4; ++j) { acc[t][j][2 * half] *= f; acc[t][j][2 * half + 1] *= f; }
    }
    norm *= carried[nt];
#pragma unroll
    for (int t = 0; t < 2; ++t)
        if (t < n_tiles) put_tile<SILU, PLAIN>(B[t], v[t], One());
#pragma unroll
    for (int u = 0; u < PER_THREAD; ++u) {
        const int i4 = tid + u * CHUNK_THREADS, t = i4 >> 4, i = (i4 & 15) * 4;
        float p[4] = {0.f, 0.f, 0.f, 0.f};
        if (i <= t) {
            const float sv[4] = {sc.v[u].x, sc.v[u].y, sc.v[u].z, sc.v[u].w};
            const double Lt = L[t];
#pragma unroll
            for (int e = 0; e < 4; ++e) p[e] = i + e <= t ? sv[e] * gain[i + e] * expf((float)(Lt - L[i + e])) : 0.f;
        }
        tile_store4<PLAIN>(A, t, i, make_float4(p[0], p[1], p[2], p[3]));
    }
    __syncthreads();
    int bad = 0;
#pragma unroll
    for (int t = 0; t < 2; ++t) {
        if (t >= n_tiles) break;
        tile_product<PLAIN, false, true, true>(acc[t], A, B[t], m0, n0w, m0 / 16 + 1);         // P holds nothing right of the diagonal
        const int c1 = c0 + t * CHUNK, nc = a.dv - c1;
        for_result(acc[t], m0, n0w, [&](int i, int c, float x, float y) {
            if (i < n) put_pair<VEC>(a.y + ((size_t)(token0 + i) * a.heads + h) * a.dv + c1 + c, nc - c, x * a.q_scale, y * a.q_scale);
        });
        bad |= not_finite(acc[t]);
    }
    if (norm_here) {
        for (int i = 0; i < 16; i += 8) {
            float p[8];
            tile_read8<PLAIN>(A, nt, nq + i, p);
#pragma unroll
            for (int e = 0; e < 8; ++e) norm += p[e];
        }
        norm += __shfl_xor_sync(0xffffffffu, norm, 1);
        norm += __shfl_xor_sync(0xffffffffu, norm, 2);
        if (nq == 0 && nt < n) a.yn[(size_t)(token0 + nt) * a.heads + h] = norm * a.q_scale;
    }
    return bad;
}
template <bool VEC, bool NORM, bool SILU>
__device__ __noinline__ void reads_plain(const ChunkArgs& a, ReadShared& sh) { reads_pass<VEC, NORM, SILU, true>(a, sh); }
template <bool VEC, bool NORM, bool SILU>
__global__ void __launch_bounds__(CHUNK_THREADS, 2)
chunk_reads_kernel(const __grid_constant__ ChunkArgs a) {
    __shared__ ReadShared sh;
    pdl_trigger();
    if (__syncthreads_or(reads_pass<VEC, NORM, SILU, false>(a, sh))) reads_plain<VEC, NORM, SILU>(a, sh);
}

// Whether rows of four floats may be read (and pairs written) as one: widths, strides and addresses that allow it.
inline bool chunk_vectors_ok(const ChunkArgs& a) {
    return a.N % 4 == 0 && a.dv % 4 == 0 && a.q_stride % 4 == 0 && a.k_stride % 4 == 0 && a.v_stride % 4 == 0 &&
           !(((uintptr_t)a.q | (uintptr_t)a.k | (uintptr_t)a.v | (uintptr_t)a.blocks | (uintptr_t)a.y) & 15);
}
template <bool VEC, bool NORM, bool SILU>
int launch_chunk_gains(const ChunkArgs& a, int n_chunks, cudaStream_t s, bool pdl) {
    static bool configured = false;
    if (!configured) {
        cudaError_t e = cudaFuncSetAttribute(chunk_gains_kernel<VEC, NORM, SILU>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)GAINS_SMEM);
        if (e == cudaSuccess) e = cudaFuncSetAttribute(chunk_gains_kernel<VEC, NORM, SILU>, cudaFuncAttributePreferredSharedMemoryCarveout, cudaSharedmemCarveoutMaxShared);
        if (e != cudaSuccess) return (int)e;
        configured = true;
    }
    ChunkArgs args = a;
    args.narrow = chunk_narrow(a, n_chunks);
    const int blocks = (a.dv + CHUNK_COLUMNS - 1) / CHUNK_COLUMNS, tiles = ((a.N + CHUNK - 1) / CHUNK) * ((a.dv + CHUNK - 1) / CHUNK);
    return launch_kernel(chunk_gains_kernel<VEC, NORM, SILU>, dim3(n_chunks, a.heads, args.narrow ? tiles + 1 : blocks), dim3(CHUNK_THREADS), GAINS_SMEM, s, pdl, args);
}
template <bool VEC, bool NORM, bool SILU>
int launch_chunk_reads(const ChunkArgs& a, int n_chunks, cudaStream_t s, bool pdl) {
    static bool configured = false;
    if (!configured) {
        cudaError_t e = cudaFuncSetAttribute(chunk_reads_kernel<VEC, NORM, SILU>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)READS_SMEM);
        if (e == cudaSuccess) e = cudaFuncSetAttribute(chunk_reads_kernel<VEC, NORM, SILU>, cudaFuncAttributePreferredSharedMemoryCarveout, cudaSharedmemCarveoutMaxShared);
        if (e != cudaSuccess) return (int)e;
        configured = true;
    }
    ChunkArgs args = a;
    args.narrow = chunk_narrow(a, n_chunks);
    const int columns = args.narrow ? CHUNK : CHUNK_COLUMNS;
    return launch_kernel(chunk_reads_kernel<VEC, NORM, SILU>, dim3(n_chunks, a.heads, (a.dv + columns - 1) / columns), dim3(CHUNK_THREADS), READS_SMEM, s, pdl, args);
}
}  // namespace
