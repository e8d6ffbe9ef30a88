// Prompt attention of float tensors on the tensor cores, heads of up to 128: every float three bfloat16 parts, six products each
// (split_mma.cuh), softmax, probabilities and sums in float.
//
// A CTA has 32 queries of one head and walks tiles of KEYS keys (64, or 32 beyond head size 64): a warp has 16 queries and 16 of
// every tile's keys, with a running softmax of its own, and the shares are merged at the end.  A tile's keys and values arrive as
// floats by cp.async while the tile before is multiplied, and are split into parts once for all warps; the probabilities are split
// in the registers in which the scores came out, which are the operand's.
//
// What bounds it: products at the rate of mma.sync (six where float has one: 91 TFLOP/s), the splitting beside them, and the longest
// row of key tiles: tiles of 32 queries make 288 CTAs of 1000 tokens x 9 heads, two per SM, the longest first.
// 1000 tokens, 9 heads of 64: 41 us; with four warps a CTA, each for 32 keys of a tile, 73; on the CUDA cores (64 queries a CTA, transposed
// operands in shared memory) 137.
//
// Scores or outputs that are not finite (an infinity among the inputs, or a float that rounds to a bfloat16 infinity, has NaN among its
// parts), and outputs other than zero below 2^-64 (values below about 2^-110 run out of exponents for their parts), send the CTA through plain_rows,
// which has float multiply-adds only.
//
// Compiled once per HEAD_DIM, a multiple of 16 up to 128; with -DSOFTCAP=1 a score becomes cap tanh(score / cap) before the softmax.  Wider heads,
// and single tokens, are attention.cu's, whose formulas these are.
#include "split_mma.cuh"
#include "softcap.cuh"

#if !defined(HEAD_DIM) || (HEAD_DIM % 16) || (HEAD_DIM > 128) || (HEAD_DIM < 16)
#error "compile with -DHEAD_DIM=<multiple of 16 between 16 and 128>"
#endif

namespace {
constexpr int D = HEAD_DIM;
constexpr int TILE = 64;                            // queries of a listed tile
constexpr int SPLIT_ROWS = 32, WARP_KEYS = 16, KEYS = D <= 64 ? 64 : 32, SHARES = KEYS / WARP_KEYS;
constexpr int SPLIT_THREADS = 2 * 32 * SHARES;
constexpr int PLD = D + 8;                          // row stride of a plane: an odd number of 16-byte units, eight rows in different banks
constexpr int Q_PLANE = SPLIT_ROWS * PLD, KV_PLANE = KEYS * PLD;
constexpr int N_BLOCK = D % 32 == 0 ? 4 : 2;        // column tiles of the output that are made together
constexpr size_t SPLIT_SMEM = sizeof(__nv_bfloat16) * 3 * (Q_PLANE + 2 * KV_PLANE) + sizeof(float) * 2 * KEYS * D;
static_assert((SHARES - 1) * 2 * 32 * (D / 2 + 4) * sizeof(float) <= sizeof(__nv_bfloat16) * 6 * KV_PLANE, "the shares meet where the planes were");

struct SplitAttention {
    const float* q; float* out; const float* k_cache; const float* v_cache;
    const int* req_slot; const int* block_table; const int* tile_req; const int* tile_q0; const int* q_start; const int* q_len; const int* ctx_len;
    const float* sink_heads;
    int table_width, hq, hkv, page_size, window, keep_first, one_round;
    float scale, softcap, sink;
};
// the CTA's queries and keys
struct SplitRows {
    int rows, tok0, qpos0, ctx, kvh, head; const int* table;
    __device__ __forceinline__ SplitRows(const SplitAttention& a) {
        // Listed longest first.  Where all CTAs run at once, two to an SM (one_round: the SMs), the second ones are taken from the short
        // end: an SM's second CTA comes with the longest first ones.
        const int at = blockIdx.x, cta = a.one_round && at >= a.one_round ? (int)gridDim.x - 1 - (at - a.one_round) : at;
        const int part = cta / a.hq, tile = part >> 1, half = 1 - (part & 1);      // the later half of a tile sees more keys
        const int req = a.tile_req[tile], q0 = a.tile_q0[tile] + SPLIT_ROWS * half, n = a.q_len[req];
        head = cta - part * a.hq;
        rows = min(SPLIT_ROWS, n - q0);
        tok0 = a.q_start[req] + q0;
        ctx = a.ctx_len[req];
        qpos0 = ctx - n + q0;
        kvh = head / (a.hq / a.hkv);
        table = a.block_table + (size_t)a.req_slot[req] * a.table_width;
    }
    __device__ __forceinline__ long long cache_row(const SplitAttention& a, int kpos) const {      // -1: no such key, or a page the window has passed
        const int page = kpos < ctx ? table[kpos / a.page_size] : -1;
        return page < 0 ? -1 : (((long long)page * a.hkv + kvh) * a.page_size + kpos % a.page_size) * D;
    }
};
__device__ __forceinline__ bool sees(const SplitAttention& a, int qpos, int kpos) {
    return kpos <= qpos && (a.window <= 0 || kpos + a.window > qpos || kpos < a.keep_first);
}
// key tiles: those that hold kept first keys, then from the window's first tile on (the two runs never overlap)
struct KeyTiles {
    int begin, kept, count;
    __device__ __forceinline__ KeyTiles(const SplitAttention& a, const SplitRows& r) {
        const int first = a.window > 0 ? max(0, r.qpos0 - a.window + 1) : 0;
        begin = first / KEYS * KEYS;
        kept = (a.window > 0 && a.keep_first > 0) ? min((a.keep_first + KEYS - 1) / KEYS, begin / KEYS) : 0;
        count = kept + (r.qpos0 + r.rows - begin + KEYS - 1) / KEYS;
    }
    __device__ __forceinline__ int key0(int tile) const { return tile < kept ? tile * KEYS : begin + (tile - kept) * KEYS; }
};

// The rows key by key with float multiply-adds, four or eight threads a row.
__device__ __noinline__ void plain_rows(const SplitAttention& a, const SplitRows& r) {
    constexpr int PER_ROW = SPLIT_THREADS / SPLIT_ROWS, N = D / PER_ROW;
    const int row = threadIdx.x / PER_ROW, part = threadIdx.x % PER_ROW;
    const bool live = row < r.rows;
    const float* q = a.q + ((size_t)(r.tok0 + (live ? row : 0)) * a.hq + r.head) * D + part * N;
    float o[N], m = -INFINITY, l = 0.f;
    for (int d = 0; d < N; ++d) o[d] = 0.f;
    const KeyTiles tiles(a, r);
    for (int t = 0; t < tiles.count; ++t)
        for (int j = 0; j < KEYS; ++j) {
            const int kpos = tiles.key0(t) + j;
            const long long at = r.cache_row(a, kpos);
            const float *k = a.k_cache + at + part * N, *v = a.v_cache + at + part * N;
            float s = 0.f;
            for (int d = 0; at >= 0 && d < N; ++d) s = fmaf(q[d] * a.scale, k[d], s);
#pragma unroll
            for (int lanes = 1; lanes < PER_ROW; lanes *= 2) s += __shfl_xor_sync(0xffffffffu, s, lanes);
            if (SOFTCAP) s = a.softcap * tanhf(s / a.softcap);
            if (!live || !sees(a, r.qpos0 + row, kpos)) continue;
            const float m_new = fmaxf(m, s), m_use = m_new == -INFINITY ? 0.f : m_new, alpha = expf(m - m_use), p = expf(s - m_use);
            l = l * alpha + p;
            m = m_new;
            for (int d = 0; d < N; ++d) o[d] = fmaf(p, at >= 0 ? v[d] : 0.f, o[d] * alpha);
        }
    if (!live) return;
    const float sk = a.sink_heads ? a.sink_heads[r.head] : a.sink;
    const float inv = 1.f / (sk > -INFINITY ? l + expf(sk - m) : l);
    float* dst = a.out + ((size_t)(r.tok0 + row) * a.hq + r.head) * D + part * N;
    for (int d = 0; d < N; ++d) dst[d] = o[d] * inv;
}

// one 16-deep step of acc += A B, B_TILES column tiles of 8: the products of parts from the smallest up, from zero, then one add
template <int N_TILES>
__device__ __forceinline__ void split_step(float (*acc)[4], const uint32_t (&a)[3][4], const uint32_t (&b)[3][N_TILES / 2][4]) {
    constexpr int PART_A[6] = {2, 0, 1, 1, 0, 0}, PART_B[6] = {0, 2, 1, 0, 1, 0};
    float t[N_TILES][4] = {};
#pragma unroll
    for (int p = 0; p < 6; ++p)
#pragma unroll
        for (int j = 0; j < N_TILES; ++j) mma_bf16(t[j], a[PART_A[p]], b[PART_B[p]][j >> 1][2 * (j & 1)], b[PART_B[p]][j >> 1][2 * (j & 1) + 1]);
#pragma unroll
    for (int j = 0; j < N_TILES; ++j)
#pragma unroll
        for (int e = 0; e < 4; ++e) acc[j][e] += t[j][e];
}
// four floats as three parts at `at` of a plane triple
__device__ __forceinline__ void put_parts(__nv_bfloat16* at, int plane, float4 v) {
    uint32_t x[3], y[3];
    split_pair(v.x, v.y, x);
    split_pair(v.z, v.w, y);
#pragma unroll
    for (int p = 0; p < 3; ++p) *reinterpret_cast<uint2*>(at + p * plane) = make_uint2(x[p], y[p]);
}

__global__ void __launch_bounds__(SPLIT_THREADS, 2)
attn_prefill_split_kernel(const __grid_constant__ SplitAttention a) {
    CISR_TRACE_SCOPE(TRACE_ATTN_SIMT);
    extern __shared__ __align__(16) float smem[];
    __nv_bfloat16* Qp = reinterpret_cast<__nv_bfloat16*>(smem);       // [3][32][PLD]
    __nv_bfloat16* Kp = Qp + 3 * Q_PLANE;                             // [3][KEYS][PLD]
    __nv_bfloat16* Vp = Kp + 3 * KV_PLANE;
    float* raw = reinterpret_cast<float*>(Vp + 3 * KV_PLANE);         // keys, then values, as they arrive: [2][KEYS][D]
    __shared__ long long rows_at[2][KEYS];                            // where a tile's keys lie in the cache, found a tile ahead
    const SplitRows r(a);
    if (r.rows <= 0) return;
    const KeyTiles tiles(a, r);
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, m0 = 16 * (warp & 1), key0 = WARP_KEYS * (warp >> 1);
    const int l7 = lane & 7, lo = (lane >> 3) & 1, hi = lane >> 4;
    constexpr int RUNS = D / 4;                                       // 16-byte runs of a row
    constexpr int COPIES = KEYS * RUNS / SPLIT_THREADS;               // of keys (and of values) per thread and tile
    static_assert(KEYS * RUNS % SPLIT_THREADS == 0, "whole runs per thread");

    // a thread copies, and later splits, the same runs
    auto request = [&](int tile) {
#pragma unroll
        for (int u = 0; u < COPIES; ++u) {
            const int e = tid + u * SPLIT_THREADS, row = e / RUNS, c = (e - row * RUNS) * 4;
            const long long at = rows_at[tile & 1][row];
            const uint32_t bytes = at < 0 ? 0u : 16u;                 // 0: zeros
            const size_t from = at < 0 ? 0 : (size_t)at + c;
            asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"((uint32_t)__cvta_generic_to_shared(raw + row * D + c)), "l"(a.k_cache + from), "r"(bytes) : "memory");
            asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"((uint32_t)__cvta_generic_to_shared(raw + KEYS * D + row * D + c)), "l"(a.v_cache + from), "r"(bytes) : "memory");
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    auto find = [&](int tile) { if (tid < KEYS && tile < tiles.count) rows_at[tile & 1][tid] = r.cache_row(a, tiles.key0(tile) + tid); };
    find(0);
    find(1);
    __syncthreads();
    request(0);
    for (int e = tid; e < SPLIT_ROWS * RUNS; e += SPLIT_THREADS) {
        const int row = e / RUNS, c = (e - row * RUNS) * 4;
        float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
        if (row < r.rows) v = *reinterpret_cast<const float4*>(a.q + ((size_t)(r.tok0 + row) * a.hq + r.head) * D + c);
        put_parts(Qp + row * PLD + c, Q_PLANE, make_float4(v.x * a.scale, v.y * a.scale, v.z * a.scale, v.w * a.scale));
    }

    // lane: rows m0 + lane / 4 (+ 8); of every eight columns 2 (lane % 4) and the next
    float o[D / 8][4] = {}, m_run[2] = {-INFINITY, -INFINITY}, l_run[2] = {0.f, 0.f}, odd = 0.f;
    const int row0 = m0 + (lane >> 2);
    for (int tile = 0; tile < tiles.count; ++tile) {
        asm volatile("cp.async.wait_group 0;" ::: "memory");
        __syncthreads();                                              // the tile before has been multiplied
#pragma unroll
        for (int u = 0; u < COPIES; ++u) {
            const int e = tid + u * SPLIT_THREADS, row = e / RUNS, c = (e - row * RUNS) * 4;
            put_parts(Kp + row * PLD + c, KV_PLANE, *reinterpret_cast<const float4*>(raw + row * D + c));
            put_parts(Vp + row * PLD + c, KV_PLANE, *reinterpret_cast<const float4*>(raw + KEYS * D + row * D + c));
        }
        __syncthreads();
        if (tile + 1 < tiles.count) request(tile + 1);
        find(tile + 2);                                               // in the place of this tile's, which have been used

        constexpr int S_TILES = WARP_KEYS / 8;
        float s[S_TILES][4] = {};
#pragma unroll
        for (int k = 0; k < D; k += 16) {
            uint32_t qa[3][4], kb[3][S_TILES / 2][4];
#pragma unroll
            for (int p = 0; p < 3; ++p) {
                load_matrices<false>(qa[p], Qp + p * Q_PLANE + (m0 + l7 + 8 * lo) * PLD + k + 8 * hi);
#pragma unroll
                for (int j = 0; j < S_TILES / 2; ++j) load_matrices<false>(kb[p][j], Kp + p * KV_PLANE + (key0 + 16 * j + l7 + 8 * hi) * PLD + k + 8 * lo);
            }
            split_step<S_TILES>(s, qa, kb);
        }
        const int kpos0 = tiles.key0(tile) + key0 + 2 * (lane & 3);
        uint32_t pa[WARP_KEYS / 16][3][4];                            // the probabilities' parts, as the operand of the second product
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const int row = row0 + 8 * h, qpos = r.qpos0 + row;
            float top = -INFINITY;
#pragma unroll
            for (int j = 0; j < S_TILES; ++j)
#pragma unroll
                for (int e = 0; e < 2; ++e) {
                    float& x = s[j][2 * h + e];
                    odd = fmaf(x, 0.f, odd);
                    if (SOFTCAP) x = a.softcap * tanhf(x / a.softcap);
                    if (!(row < r.rows && sees(a, qpos, kpos0 + 8 * j + e))) x = -INFINITY;
                    top = fmaxf(top, x);
                }
            top = fmaxf(top, __shfl_xor_sync(0xffffffffu, top, 1));
            top = fmaxf(top, __shfl_xor_sync(0xffffffffu, top, 2));
            const float m_new = fmaxf(m_run[h], top), m_use = m_new == -INFINITY ? 0.f : m_new, alpha = expf(m_run[h] - m_use);
            float sum = 0.f;
#pragma unroll
            for (int j = 0; j < S_TILES; ++j) {
                const float x = expf(s[j][2 * h] - m_use), y = expf(s[j][2 * h + 1] - m_use);
                sum += x + y;
                uint32_t parts[3];
                split_pair(x, y, parts);
#pragma unroll
                for (int p = 0; p < 3; ++p) pa[j >> 1][p][2 * (j & 1) + h] = parts[p];
            }
            sum += __shfl_xor_sync(0xffffffffu, sum, 1);
            sum += __shfl_xor_sync(0xffffffffu, sum, 2);
            l_run[h] = l_run[h] * alpha + sum;
            m_run[h] = m_new;
#pragma unroll
            for (int j = 0; j < D / 8; ++j) { o[j][2 * h] *= alpha; o[j][2 * h + 1] *= alpha; }
        }
#pragma unroll
        for (int k = 0; k < WARP_KEYS; k += 16)
#pragma unroll
            for (int n = 0; n < D / 8; n += N_BLOCK) {
                uint32_t vb[3][N_BLOCK / 2][4];
#pragma unroll
                for (int p = 0; p < 3; ++p)
#pragma unroll
                    for (int j = 0; j < N_BLOCK / 2; ++j)
                        load_matrices<true>(vb[p][j], Vp + p * KV_PLANE + (key0 + k + l7 + 8 * lo) * PLD + 8 * n + 16 * j + 8 * hi);
                split_step<N_BLOCK>(o + n, pa[k / 16], vb);
            }
    }
    // the other shares of the keys hand their sums to the first through the planes' place: per thread D / 2 sums, two maxima, two denominators
    constexpr int HAND = D / 2 + 4;
    const int share = warp >> 1;
    auto hand = [&](int from) { return reinterpret_cast<float*>(Kp) + ((from - 1) * 2 + (warp & 1)) * 32 * HAND + lane; };
    __syncthreads();
    if (share) {
        float* to = hand(share);
#pragma unroll
        for (int h = 0; h < 2; ++h) { to[32 * h] = m_run[h]; to[32 * (2 + h)] = l_run[h]; }
#pragma unroll
        for (int j = 0; j < D / 8; ++j)
#pragma unroll
            for (int e = 0; e < 4; ++e) to[32 * (4 + 4 * j + e)] = o[j][e];
    }
    __syncthreads();
    if (!share) {
        const float sk = a.sink_heads ? a.sink_heads[r.head] : a.sink;
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            float m_all = m_run[h];
            for (int from = 1; from < SHARES; ++from) m_all = fmaxf(m_all, hand(from)[32 * h]);
            const float m_use = m_all == -INFINITY ? 0.f : m_all, mine = expf(m_run[h] - m_use);
            float l = l_run[h] * mine;
#pragma unroll
            for (int j = 0; j < D / 8; ++j) { o[j][2 * h] *= mine; o[j][2 * h + 1] *= mine; }
            for (int from = 1; from < SHARES; ++from) {
                const float* in = hand(from);
                const float w = expf(in[32 * h] - m_use);
                l = fmaf(in[32 * (2 + h)], w, l);
#pragma unroll
                for (int j = 0; j < D / 8; ++j)
#pragma unroll
                    for (int e = 0; e < 2; ++e) o[j][2 * h + e] = fmaf(in[32 * (4 + 4 * j + 2 * h + e)], w, o[j][2 * h + e]);
            }
            // a sink is one more term of the denominator, exp(sink), with no value (sink -inf: none); one per head where given
            const float inv = 1.f / (sk > -INFINITY ? l + expf(sk - m_use) : l);
#pragma unroll
            for (int j = 0; j < D / 8; ++j) { o[j][2 * h] *= inv; o[j][2 * h + 1] *= inv; }
        }
    }
    uint32_t most[2] = {};
    if (!share) {
        const bool pairs = ((uintptr_t)a.out & 7) == 0;
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const int row = row0 + 8 * h;
            if (row >= r.rows) continue;
            float* dst = a.out + ((size_t)(r.tok0 + row) * a.hq + r.head) * D + 2 * (lane & 3);
#pragma unroll
            for (int j = 0; j < D / 8; ++j) {
                const float x = o[j][2 * h], y = o[j][2 * h + 1];
                most[0] = max(most[0], oddness(x));
                most[1] = max(most[1], oddness(y));
                if (pairs) *reinterpret_cast<float2*>(dst + 8 * j) = make_float2(x, y);
                else { dst[8 * j] = x; dst[8 * j + 1] = y; }
            }
        }
    }
    // a score that is not finite (0 x finite is 0, else NaN, and a NaN stays), or such an output or a tiny one: all rows again
    if (__syncthreads_or(odd != 0.f || max(most[0], most[1]) >= ODD)) plain_rows(a, r);
}
}  // namespace

CISR_EXPORT int cisr_attn_float_head_dim() { return D; }
CISR_EXPORT int cisr_attn_float_tile() { return TILE; }

CISR_EXPORT int cisr_attn_prefill_float(const void* q, void* out, const void* k_cache, const void* v_cache,
                                        const int* req_slot, const int* block_table, int table_width, const int* tile_req, const int* tile_q0,
                                        int n_tiles, const int* q_start, const int* q_len, const int* ctx_len, int hq,
                                        int hkv, int page_size, float scale, float softcap, int window, int keep_first, float sink,
                                        const float* sink_heads, void* stream) {
    if (n_tiles <= 0) return 0;
    if (hq % hkv || (SOFTCAP ? !(softcap > 0.f) : softcap != 0.f)) return -2;
    if (((uintptr_t)q | (uintptr_t)k_cache | (uintptr_t)v_cache) & 15) return -2;      // rows are read by 16 bytes
    static bool configured = false;
    static int sms = 0;
    if (!configured) {
        const cudaError_t e = cudaFuncSetAttribute(attn_prefill_split_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)SPLIT_SMEM);
        if (e != cudaSuccess) return (int)e;
        int device = 0;
        cudaGetDevice(&device);
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device);
        configured = true;
    }
    const int ctas = hq * n_tiles * (TILE / SPLIT_ROWS);
    SplitAttention a = {};
    a.q = (const float*)q; a.out = (float*)out; a.k_cache = (const float*)k_cache; a.v_cache = (const float*)v_cache;
    a.req_slot = req_slot; a.block_table = block_table; a.table_width = table_width; a.tile_req = tile_req; a.tile_q0 = tile_q0;
    a.q_start = q_start; a.q_len = q_len; a.ctx_len = ctx_len; a.sink_heads = sink_heads; a.hq = hq; a.hkv = hkv; a.page_size = page_size;
    a.window = window; a.keep_first = keep_first; a.scale = scale; a.softcap = softcap; a.sink = sink; a.one_round = ctas > sms && ctas <= 2 * sms ? sms : 0;
    attn_prefill_split_kernel<<<dim3(ctas), SPLIT_THREADS, SPLIT_SMEM, (cudaStream_t)stream>>>(a);
    return launch_status();
}
