// Lightning attention: linear attention with one fixed decay per head and a matrix state per head.
//
//   q = silu(W_q h), k = silu(W_k h) [heads x key_dim], v = silu(W_v h) [heads x value_dim]
//   per head:  S <- decay_h S + k v^T;  o = S^T q          (S [key_dim, value_dim], zero when the request starts)
//   out = o / sqrt(mean(o^2) + eps) * w_norm * sigmoid(W_g h), the mean over all heads of the token at once
//
// The projections arrive as float sums (proj [tokens, columns]: q | k | v | gate from given columns); silu, the decay and
// its powers, the state and every step of its recurrence, the norm and the gate are float arithmetic.  A request's state
// is one float row of a state tensor, laid out [heads, value_dim, key_dim] (a column of S is contiguous).
//
// Two forms of the same recurrence, which differ by rounding only:
//   walk    single tokens and short portions: a warp per column of S, its lanes holding the column's rows in registers,
//           token after token.
//   chunks  portions of LIGHTNING_CHUNK tokens and more, C = LIGHTNING_CHUNK tokens at a time.  With t, i counted inside a
//           chunk of n tokens and S0 the state before it:
//               o_t = decay^(t+1) S0^T q_t + sum_{i <= t} decay^(t-i) (q_t . k_i) v_i
//               S   = decay^n S0 + sum_i decay^(n-1-i) k_i v_i^T
//           The second sum of S (a chunk's gain) needs no state, so it is made for every chunk of the step at once; a short
//           scan then carries the state from chunk to chunk, element by element; and the read-outs of every chunk are made
//           at once from the state before each.  The products are chunk_linear.cuh's, 64 x 64 x 64 at a time, float
//           through the tensor cores, with silu taken as the operands are staged.
#include "chunk_linear.cuh"

static bool g_pdl = false;
CISR_EXPORT void cisr_lightning_set_pdl(int on) { g_pdl = on != 0; }

constexpr int LIGHTNING_CHUNK = CHUNK;
constexpr int WALK_WARPS = 8;
constexpr int MAX_KEY_DIM = 256;
CISR_EXPORT int cisr_lightning_chunk_tokens() { return LIGHTNING_CHUNK; }
CISR_EXPORT int cisr_lightning_max_key_dim() { return MAX_KEY_DIM; }

__device__ __forceinline__ float silu_f(float z) { return chunk_silu(z); }

// ---------------------------------------------------------------- token by token
// grid (requests, heads, value columns / WALK_WARPS); a warp owns column c of its head's state, lane l the rows l, l + 32, ...
// `least` > 0: requests that bring at least that many tokens are left to the chunked kernel.
template <int R>
__global__ void __launch_bounds__(32 * WALK_WARPS)
lightning_walk_kernel(const float* __restrict__ proj, int stride, int q_col, int k_col, int v_col, const float* __restrict__ decay,
                      float* __restrict__ state, long long state_stride, const int* __restrict__ req_slot,
                      const int* __restrict__ q_start, const int* __restrict__ q_len, float* __restrict__ o, int heads, int key_dim,
                      int value_dim, int least) {
    pdl_trigger();
    pdl_wait();
    const int r = blockIdx.x, h = blockIdx.y, lane = threadIdx.x & 31, c = blockIdx.z * WALK_WARPS + (threadIdx.x >> 5);
    const int n = q_len[r];
    if (n <= 0 || (least > 0 && n >= least) || c >= value_dim) return;
    float* column = state + (size_t)req_slot[r] * state_stride + ((size_t)h * value_dim + c) * key_dim;
    float S[R], k_now[R], q_now[R], k_next[R], q_next[R], v_now, v_next = 0.f;
#pragma unroll
    for (int i = 0; i < R; ++i) { const int row = lane + 32 * i; S[i] = row < key_dim ? column[row] : 0.f; k_next[i] = q_next[i] = 0.f; }
    const float dec = decay[h];
    const int t0 = q_start[r];
    auto fetch = [&](int t) {
        const float* row_p = proj + (size_t)(t0 + t) * stride;
        v_next = row_p[v_col + h * value_dim + c];
#pragma unroll
        for (int i = 0; i < R; ++i) {
            const int row = lane + 32 * i;
            k_next[i] = row < key_dim ? row_p[k_col + h * key_dim + row] : 0.f;
            q_next[i] = row < key_dim ? row_p[q_col + h * key_dim + row] : 0.f;
        }
    };
    fetch(0);
    for (int t = 0; t < n; ++t) {
        v_now = v_next;
#pragma unroll
        for (int i = 0; i < R; ++i) { k_now[i] = k_next[i]; q_now[i] = q_next[i]; }
        if (t + 1 < n) fetch(t + 1);                  // the next token's operands are on their way during this token's sums
        const float v = silu_f(v_now);
        float acc = 0.f;
#pragma unroll
        for (int i = 0; i < R; ++i) {
            S[i] = dec * S[i] + silu_f(k_now[i]) * v;
            acc += S[i] * silu_f(q_now[i]);
        }
        acc = warp_sum(acc);
        if (lane == 0) o[(size_t)(t0 + t) * heads * value_dim + h * value_dim + c] = acc;
    }
#pragma unroll
    for (int i = 0; i < R; ++i) { const int row = lane + 32 * i; if (row < key_dim) column[row] = S[i]; }
}

// ---------------------------------------------------------------- chunk by chunk
// Three launches over the chunks of the step's long portions (chunk_req, chunk_t0: a chunk's request and its first token
// inside the portion; req_chunk0: a request's first chunk), with a scratch of one state-sized block per (chunk, head) and
// one of a chunk's scores:
//   gains   every chunk's own contribution to the state, sum_i decay^(n-1-i) k_i v_i^T, into the chunk's block [key_dim][value_dim],
//           and its scores q_t . k_i
//   scan    (request, head): walks the request's chunks element by element: the scratch block receives the state BEFORE
//           its chunk, the running state becomes decay^n S + gain; the last one goes back to the request's slot.
//   reads   every chunk's read-outs, decay^(t+1) S0^T q_t + sum_{i<=t} decay^(t-i) (q_t . k_i) v_i
//           with S0 from the scratch
constexpr int C = LIGHTNING_CHUNK;

// grid (requests, heads, elements / (256 VEC)): a thread owns VEC neighbouring elements (row, col .. col + VEC - 1) of the
// head's state (VEC 4 where value_dim is a multiple of 4, so that a CTA reads 4 KB in one piece from every block; else 1)
template <int VEC>
__global__ void __launch_bounds__(256) lightning_scan_kernel(ChunkArgs a) {
    pdl_trigger();
    pdl_wait();
    const int r = blockIdx.x, h = blockIdx.y, e = (blockIdx.z * 256 + threadIdx.x) * VEC;
    const int n_all = a.q_len[r];
    if (n_all < a.least || e >= a.N * a.dv) return;
    const int row = e / a.dv, col = e - row * a.dv;
    float* kept = a.state + (size_t)a.req_slot[r] * a.state_stride + ((size_t)h * a.dv + col) * a.N + row;
    float S[VEC];
#pragma unroll
    for (int j = 0; j < VEC; ++j) S[j] = kept[(size_t)j * a.N];
    const double lg = log((double)a.decay[h]);
    const float whole = (float)exp((double)C * lg);
    const size_t step = (size_t)a.heads * a.N * a.dv;
    float* block = a.blocks + ((size_t)a.req_chunk0[r] * a.heads + h) * a.N * a.dv + e;
    const int chunks = (n_all + C - 1) / C;
    // the walk itself is one multiply-add per chunk: it goes as fast as the gains arrive, so AHEAD of them are asked for
    // together, and the next ones before the ones at hand are used
    constexpr int AHEAD = 8;
    float gain[AHEAD][VEC];
    const auto fetch = [&](int c0) {
#pragma unroll
        for (int u = 0; u < AHEAD; ++u) {
            const bool in = c0 + u < chunks;
            if (VEC == 4) {
                const float4 g = in ? *reinterpret_cast<const float4*>(block + (size_t)(c0 + u) * step) : make_float4(0.f, 0.f, 0.f, 0.f);
                gain[u][0] = g.x; gain[u][1 % VEC] = g.y; gain[u][2 % VEC] = g.z; gain[u][3 % VEC] = g.w;
            } else {
                gain[u][0] = in ? block[(size_t)(c0 + u) * step] : 0.f;
            }
        }
    };
    fetch(0);
    for (int c0 = 0; c0 < chunks; c0 += AHEAD) {
        float now[AHEAD][VEC];
#pragma unroll
        for (int u = 0; u < AHEAD; ++u)
#pragma unroll
            for (int j = 0; j < VEC; ++j) now[u][j] = gain[u][j];
        if (c0 + AHEAD < chunks) fetch(c0 + AHEAD);
#pragma unroll
        for (int u = 0; u < AHEAD; ++u) {
            const int c = c0 + u;
            if (c < chunks) {
                const int n = min(C, n_all - c * C);
                const float f = n == C ? whole : (float)exp((double)n * lg);
                if (VEC == 4) *reinterpret_cast<float4*>(block + (size_t)c * step) = make_float4(S[0], S[1 % VEC], S[2 % VEC], S[3 % VEC]);
                else block[(size_t)c * step] = S[0];
#pragma unroll
                for (int j = 0; j < VEC; ++j) S[j] = f * S[j] + now[u][j];
            }
        }
    }
#pragma unroll
    for (int j = 0; j < VEC; ++j) kept[(size_t)j * a.N] = S[j];
}

template <bool VEC>
static int launch_chunks(const ChunkArgs& a, int n_req, int n_chunks, cudaStream_t s) {
    int st = launch_chunk_gains<VEC, false, true>(a, n_chunks, s, g_pdl);
    if (st) return st;
    const int elements = a.N * a.dv;
    if (a.dv % 4 == 0 && ((uintptr_t)a.blocks & 15) == 0)
        st = launch_kernel(lightning_scan_kernel<4>, dim3(n_req, a.heads, (elements / 4 + 255) / 256), dim3(256), 0, s, g_pdl, a);
    else
        st = launch_kernel(lightning_scan_kernel<1>, dim3(n_req, a.heads, (elements + 255) / 256), dim3(256), 0, s, g_pdl, a);
    if (st) return st;
    return launch_chunk_reads<VEC, false, true>(a, n_chunks, s, g_pdl);
}

// The recurrence for a step: the requests that bring at least `least` tokens run chunk by chunk (`n_chunks` chunks listed in
// chunk_req / chunk_t0, a request's first one in req_chunk0; scratch [n_chunks][heads][key_dim][value_dim], scores
// [n_chunks][heads][LIGHTNING_CHUNK][LIGHTNING_CHUNK]), the `n_short` others token by token; least <= 0: every request
// token by token.  o float [tokens, heads * value_dim].
CISR_EXPORT int cisr_lightning_recurrence(const float* proj, int stride, int q_col, int k_col, int v_col, const float* decay, float* state,
                                          long long state_stride, const int* req_slot, const int* q_start, const int* q_len, float* o,
                                          int heads, int key_dim, int value_dim, int n_req, int least, int n_chunks, int n_short,
                                          const int* chunk_req, const int* chunk_t0, const int* req_chunk0, float* scratch, float* scores,
                                          void* stream) {
    if (n_req <= 0) return 0;
    if (key_dim <= 0 || key_dim > MAX_KEY_DIM || value_dim <= 0 || heads <= 0) return -2;
    cudaStream_t s = (cudaStream_t)stream;
    int st = 0;
    if (least > 0 && n_chunks > 0) {
        if (!chunk_req || !chunk_t0 || !req_chunk0 || !scratch || !scores || ((uintptr_t)scores & 15)) return -2;
        ChunkArgs a = {};
        a.q = proj + q_col; a.k = proj + k_col; a.v = proj + v_col; a.q_stride = a.k_stride = a.v_stride = stride;
        a.decay = decay; a.state = state; a.state_stride = state_stride; a.req_slot = req_slot; a.q_start = q_start; a.q_len = q_len;
        a.chunk_req = chunk_req; a.chunk_t0 = chunk_t0; a.req_chunk0 = req_chunk0; a.scores = scores; a.blocks = scratch; a.y = o;
        a.q_scale = 1.f; a.heads = a.groups = heads; a.N = key_dim; a.dv = value_dim; a.least = least;
        st = chunk_vectors_ok(a) ? launch_chunks<true>(a, n_req, n_chunks, s) : launch_chunks<false>(a, n_req, n_chunks, s);
        if (st) return st;
    }
    if (least <= 0 || n_short > 0) {
        const dim3 grid(n_req, heads, (value_dim + WALK_WARPS - 1) / WALK_WARPS), block(32 * WALK_WARPS);
        const int rows = (key_dim + 31) / 32;
#define LIGHTNING_WALK(R) launch_kernel(lightning_walk_kernel<R>, grid, block, 0, s, g_pdl, proj, stride, q_col, k_col, v_col, decay, state, \
                                        state_stride, req_slot, q_start, q_len, o, heads, key_dim, value_dim, least > 0 ? least : 0)
        switch (rows) {
            case 1: st = LIGHTNING_WALK(1); break;
            case 2: st = LIGHTNING_WALK(2); break;
            case 3: st = LIGHTNING_WALK(3); break;
            case 4: st = LIGHTNING_WALK(4); break;
            case 5: case 6: st = LIGHTNING_WALK(6); break;
            default: st = LIGHTNING_WALK(8); break;
        }
#undef LIGHTNING_WALK
    }
    return st;
}

// ---------------------------------------------------------------- output: norm over all heads, weight, gate
// out[t, j] = o[t, j] / sqrt(mean_j(o[t, :]^2) + eps) * norm_w[j] * sigmoid(gate[t, gate_col + j]), rounded once.
template <typename CT>
__global__ void lightning_output_kernel(const float* __restrict__ o, const float* __restrict__ gate, int gate_stride, int gate_col,
                                        const float* __restrict__ norm_w, float eps, CT* __restrict__ out, int out_stride, int width) {
    __shared__ float scratch[32];
    pdl_trigger();
    pdl_wait();
    const int t = blockIdx.x;
    const float* row = o + (size_t)t * width;
    float sq = 0.f;
    for (int j = threadIdx.x; j < width; j += blockDim.x) { const float v = row[j]; sq += v * v; }
    const float unit = rsqrtf(block_sum(sq, scratch) / (float)width + eps);
    const float* g = gate + (size_t)t * gate_stride + gate_col;
    for (int j = threadIdx.x; j < width; j += blockDim.x)
        out[(size_t)t * out_stride + j] = from_float<CT>(row[j] * unit * norm_w[j] * quotient(1.f, 1.f + expf(-g[j])));
}

// The same, four columns an access and the row and its gates in registers, all requested before the sum: bound by memory (2048
// tokens of 2048: 42 MB, 6.4 us), where single columns asked for one float a thread and the gates only after the sum:
// 18.4 us, now 11.8.
__device__ __forceinline__ void store4(float* to, const float (&v)[4]) { *reinterpret_cast<float4*>(to) = make_float4(v[0], v[1], v[2], v[3]); }
__device__ __forceinline__ void store4(__nv_bfloat16* to, const float (&v)[4]) {
    __nv_bfloat162 pair[2] = {__floats2bfloat162_rn(v[0], v[1]), __floats2bfloat162_rn(v[2], v[3])};
    *reinterpret_cast<uint2*>(to) = *reinterpret_cast<uint2*>(pair);
}
constexpr int OUT_THREADS = 256, OUT_RUNS = 4;            // rows of up to 4 * 4 * 256 columns
template <typename CT>
__global__ void __launch_bounds__(OUT_THREADS)
lightning_output_runs_kernel(const float* __restrict__ o, const float* __restrict__ gate, int gate_stride, int gate_col,
                             const float* __restrict__ norm_w, float eps, CT* __restrict__ out, int out_stride, int width) {
    __shared__ float scratch[32];
    pdl_trigger();
    pdl_wait();
    const size_t t = blockIdx.x;
    const float* row = o + t * width;
    const float* gr = gate + t * gate_stride + gate_col;
    float v[OUT_RUNS][4], g[OUT_RUNS][4], sq = 0.f;
#pragma unroll
    for (int r = 0; r < OUT_RUNS; ++r) {
        const int j = 4 * (r * OUT_THREADS + (int)threadIdx.x);
        const float4 a = j < width ? *reinterpret_cast<const float4*>(row + j) : make_float4(0.f, 0.f, 0.f, 0.f);
        const float4 b = j < width ? *reinterpret_cast<const float4*>(gr + j) : make_float4(0.f, 0.f, 0.f, 0.f);
        v[r][0] = a.x; v[r][1] = a.y; v[r][2] = a.z; v[r][3] = a.w;
        g[r][0] = b.x; g[r][1] = b.y; g[r][2] = b.z; g[r][3] = b.w;
    }
#pragma unroll
    for (int r = 0; r < OUT_RUNS; ++r)
#pragma unroll
        for (int e = 0; e < 4; ++e) sq += v[r][e] * v[r][e];
    const float unit = rsqrtf(block_sum(sq, scratch) / (float)width + eps);
#pragma unroll
    for (int r = 0; r < OUT_RUNS; ++r) {
        const int j = 4 * (r * OUT_THREADS + (int)threadIdx.x);
        if (j >= width) break;
        const float4 w = *reinterpret_cast<const float4*>(norm_w + j);
        const float ww[4] = {w.x, w.y, w.z, w.w};
#pragma unroll
        for (int e = 0; e < 4; ++e) v[r][e] = v[r][e] * unit * ww[e] * quotient(1.f, 1.f + expf(-g[r][e]));
        store4(out + t * out_stride + j, v[r]);
    }
}

CISR_EXPORT int cisr_lightning_output(const float* o, const float* gate, int gate_stride, int gate_col, const float* norm_w, float eps,
                                      void* out, int dtype, int out_stride, int width, int tokens, void* stream) {
    if (tokens <= 0) return 0;
    cudaStream_t s = (cudaStream_t)stream;
    // rows of 512 to 4096 columns in whole aligned runs of four (below, most of the threads would have none)
    const bool runs = width >= 512 && width <= 4 * OUT_THREADS * OUT_RUNS && !((width | gate_stride | gate_col | out_stride) & 3) &&
                      !(((uintptr_t)o | (uintptr_t)gate | (uintptr_t)norm_w | (uintptr_t)out) & 15);
    if (runs && dtype == CISR_BF16)
        return launch_kernel(lightning_output_runs_kernel<__nv_bfloat16>, dim3(tokens), dim3(OUT_THREADS), 0, s, g_pdl, o, gate, gate_stride,
                             gate_col, norm_w, eps, (__nv_bfloat16*)out, out_stride, width);
    if (runs)
        return launch_kernel(lightning_output_runs_kernel<float>, dim3(tokens), dim3(OUT_THREADS), 0, s, g_pdl, o, gate, gate_stride, gate_col,
                             norm_w, eps, (float*)out, out_stride, width);
    const int threads = width >= 1024 ? 256 : 128;
    if (dtype == CISR_BF16)
        return launch_kernel(lightning_output_kernel<__nv_bfloat16>, dim3(tokens), dim3(threads), 0, s, g_pdl, o, gate, gate_stride, gate_col,
                             norm_w, eps, (__nv_bfloat16*)out, out_stride, width);
    return launch_kernel(lightning_output_kernel<float>, dim3(tokens), dim3(threads), 0, s, g_pdl, o, gate, gate_stride, gate_col, norm_w,
                         eps, (float*)out, out_stride, width);
}
