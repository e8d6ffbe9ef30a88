// Causal grouped-query attention of prompt portions on the 5th-generation tensor cores, for head sizes 64 and 128
// (bfloat16 cache).  One CTA per query tile and query head, two streams of 128 query rows in it; scores, probabilities
// and outputs live in tensor memory.
//
//   warps 0, 2  producers: warp 0 the query tiles once and then the key tiles, warp 2 the value tiles (128 keys each),
//               into rings of their own (four stages each at head size 64; three key and two value stages at 128),
//               by tensor-map copies (cp.async.bulk.tensor.2d, 128-byte swizzle), one box per page and 64 columns;
//               page ids come straight from the block table
//   warps 1, 3  the products, issued by one lane each: S = Q K^T (tcgen05.mma kind::f16, M = 128, N = 128, K = 16
//               steps, Q and K both K-major) into the stream's 128 score columns, and O += P V (N = head size, P read from
//               tensor memory as the A operand, V as the MN-major B operand straight from its [key][dim] tile), 64 keys
//               at a time as their P arrives.  Head size 64: a warp per stream, the next scores as soon as the softmax
//               has the last ones; 128: warp 1 takes the streams in turn
//   warps 4..11 softmax, four warps per stream: a thread has a query row (tensor-memory lane), its running max and sum in
//               float.  The max in use moves only when a tile's is more than 8 above it (a stale max is exact arithmetic
//               as long as 2^(s - m) stays small); then the row of O is rescaled.  P = 2^(s - m) goes to tensor memory
//               as bfloat16 pairs
//
// A tile of 256 queries gives each stream 128 of them, and both read the same key and value tiles: half the copies of a CTA
// per 128 queries, and one stream's exponentials run beside the other's products.  Where a tile has 128 queries or fewer,
// both streams have the same queries and take the key tiles in turn, and a row's two parts are merged with their maxima and
// sums at the end.
//
// What bounds it: at head size 64 the exponentials (16 a clock and SM: 2048 cycles for a tile of 256 x 128, of about 3200
// that a pair of tiles takes) and the instructions around them; at 128 the chain scores - softmax - output product of a
// stream, of which the other stream hides a part (2048 cycles of products in about 3600).  There is no room in tensor memory for a second
// score buffer at 128.  Part of the exponentials as a polynomial on the multiply-add pipe made every size slower (4096
// queries, 32 heads of 64: 120 us without, 130 with a quarter of them, 152 with half).
// Measured (page size 16, causal; before: a CTA per 128 queries whose two groups of threads shared every key tile):
// 4096 queries x 32 heads of 128 239 -> 164 us, of 64 197 -> 121 us; 2048 x 32 of 128 85 -> 57 us; four portions of
// 345 to 921 behind 244 to 611 keys, 32 heads of 64, 89 -> 62 us; 300 queries x 32 of 128 15.3 -> 14.5 us.
//
// Exactness: scores are scaled by scale * log2(e) in float, exponentials are base 2 (ex2.approx), the sums and the
// maxima are float, P is rounded to bfloat16 once.  Key tiles start at multiples of 128 in absolute positions.
//
// With -DSOFTCAP=1 a score becomes cap tanh(score / cap) before the softmax (`softcap`; ignored otherwise): each thread
// bends its scores as it takes them from tensor memory.
//
// Every wait on an mbarrier is bounded; a role whose wait ran out raises the CTA's abort flag and the device flag
// (5), the other roles leave at their next wait, tensor memory is freed, and the host reports the failure.
//
// Parity: the online softmax of runtime/reference.py:18-27 and kernels/ops.cu:88-123 of the reference, tiled.
// Cache layout: [pages, kv_heads, page_size, HEAD_DIM]; page sizes: multiples of 8 that divide 128 or are multiples of it.
#include <type_traits>

#include "tcgen05.cuh"
#include "softcap.cuh"

#ifndef HEAD_DIM
#error "compile with -DHEAD_DIM=64 or 128"
#endif
#if HEAD_DIM != 64 && HEAD_DIM != 128
#error "the tcgen05 attention takes head sizes 64 and 128"
#endif

namespace {
typedef __nv_bfloat16 bf16;
constexpr int D = HEAD_DIM;
constexpr int NSUB = D / 64;                  // 64-column sub-tiles of Q, K and V rows
constexpr int BN = 128;                       // keys per tile
constexpr int SUB_BYTES = 128 * 128;          // one 128-row x 64-column sub-tile (queries)
constexpr int KV_SUB = BN * 128;              // one BN-key x 64-column sub-tile (keys, values)
constexpr int Q_BYTES = NSUB * SUB_BYTES;     // 128 queries
constexpr int KV_BYTES = NSUB * KV_SUB;       // a K tile, or a V tile
// Key tiles and value tiles have rings of their own: a key tile is free again when its score products are done, a value
// tile only after the output products, one softmax later.  A tile is 16 KB at head size 64 and 32 KB at 128.
constexpr int K_STAGES = D == 64 ? 4 : 3;
constexpr int V_STAGES = D == 64 ? 4 : 2;
// Two streams with the same queries leave room for one more value tile (stream 1's queries), which head size 128 takes.  Head
// size 64 does not: its streams take the tiles in turn and a warp of its own waits for each stream's, so a ring of five would
// hand every slot from one warp to the other, and a warp that skips a phase of a slot's barrier can pass it a phase early.
// In an even ring every slot is one stream's.
constexpr bool OWN_P = D == 64;
__host__ __device__ constexpr int value_slots(bool shared) { return V_STAGES + (shared && !OWN_P); }
static_assert(!OWN_P || (K_STAGES % 2 == 0 && value_slots(true) % 2 == 0), "a slot belongs to one stream");
constexpr size_t SMEM_FIXED = 1024 + 2 * Q_BYTES + (K_STAGES + V_STAGES) * KV_BYTES + 256 + 16;
constexpr float LOG2E = 1.4426950408889634f;
constexpr float RESCALE_STEP = 8.f;           // the max may lag by this much (base-2 exponent) before O is rescaled
constexpr int FIRST_SOFTMAX_WARP = 4;         // warps 0 and 2: key and value producers; warps 1 and 3: the products
constexpr int SOFTMAX_THREADS = 256;          // two streams of four warps: a thread has a whole query row
constexpr int THREADS = 32 * FIRST_SOFTMAX_WARP + SOFTMAX_THREADS;
// Tensor memory: the streams' scores at columns 0 and 128, their output accumulators from column 256 on.  At head size 64
// the accumulators leave room for the probabilities in a place of their own (OWN_P), so a stream's next scores are
// multiplied as soon as its threads have the scores at hand in registers; at 128 they go over the first half of the scores.
constexpr uint32_t TMEM_O = 256, TMEM_P = 384;
// A softmax thread takes its row of scores from tensor memory once and keeps it in registers (head size 64), or twice, 32
// columns at a time in a loop (128: first the max, then the exponentials).  A row in registers unrolls to four times the
// code, whose fetch shows wherever a CTA walks few tiles: 7 portions of 70 queries, 32 heads of 128: 27.4 us against 25.8,
// 2048 queries 59.0 against 56.8; at head size 64, where a stream's next scores never have to be waited for, the second
// trip shows instead: 4096 queries 138 us against 121.
constexpr bool TWO_PASSES = D == 128;
bool g_pdl = false;
int* g_error = nullptr;

__device__ __forceinline__ float fast_exp2(float x) {
    float y;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}
// Pairs of floats in one register pair: one instruction for two.
__device__ __forceinline__ uint64_t pack2(float a, float b) { uint64_t r; asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b)); return r; }
__device__ __forceinline__ void unpack2(uint64_t v, float& a, float& b) { asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(v)); }
__device__ __forceinline__ uint64_t fma2(uint64_t a, uint64_t b, uint64_t c) { uint64_t r; asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c)); return r; }
__device__ __forceinline__ uint64_t add2(uint64_t a, uint64_t b) { uint64_t r; asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b)); return r; }
__device__ __forceinline__ float max_nan(float a, float b, float c) { float r; asm("max.NaN.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c)); return r; }
__device__ __forceinline__ void mbar_arrive(uint64_t* bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}

__global__ void __launch_bounds__(THREADS, 1)
attn_prefill_tcgen05_kernel(const __grid_constant__ CUtensorMap map_q, const __grid_constant__ CUtensorMap map_k,
                            const __grid_constant__ CUtensorMap map_v, bf16* __restrict__ out, int cache_rows,
                            const int* __restrict__ req_slot, const int* __restrict__ block_table, int table_width,
                            const int* __restrict__ tile_req, const int* __restrict__ tile_q0, int span,
                            const int* __restrict__ q_start, const int* __restrict__ q_len,
                            const int* __restrict__ ctx_len, int hq, int hkv, int page_size, float scale, float softcap, int window,
                            int keep_first, float sink_all, const float* __restrict__ sink_heads, int* __restrict__ error) {
    CISR_TRACE_SCOPE(TRACE_ATTN_PREFILL);
    extern __shared__ unsigned char smem_raw[];
    unsigned char* base = reinterpret_cast<unsigned char*>(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
    unsigned char* Qs = base;                                   // [NSUB][128 queries][128 B]
    unsigned char* Kring = Qs + Q_BYTES;                        // [K_STAGES] key tiles, each [NSUB][BN keys][128 B]
    unsigned char* Vring = Kring + K_STAGES * KV_BYTES;         // [V_STAGES] value tiles, the same layout
    unsigned char* Qs1 = Vring + V_STAGES * KV_BYTES;           // stream 1's queries, or (head size 128) one more value tile where it has none of its own
    uint64_t* bars = reinterpret_cast<uint64_t*>(Qs1 + Q_BYTES);
    uint64_t* q_full = bars;                                    // [2] a stream's query tile has landed
    uint64_t* k_full = q_full + 2;                              // [K_STAGES] a key tile has landed
    uint64_t* k_empty = k_full + K_STAGES;                      // [K_STAGES] the score products that read it are done
    uint64_t* v_full = k_empty + K_STAGES;                      // [V_STAGES + 1] a value tile has landed
    uint64_t* v_empty = v_full + V_STAGES + 1;                  // [V_STAGES + 1] the output products that read it are done
    uint64_t* v_clean = v_empty + V_STAGES + 1;                 // the last value tile's rows beyond the keys are zero
    uint64_t* s_full = v_clean + 1;                             // [2] a stream's scores of its next tile are complete
    uint64_t* s_free = s_full + 2;                              // [2] (OWN_P) the scores are in registers
    uint64_t* p_full = s_free + 2;                              // [2 streams][2 halves] P of half a tile is in tensor memory (and O rescaled)
    uint64_t* o_done = p_full + 4;                              // [2] a stream's output product is done (OWN_P: of every tile; else of the last)
    static_assert(2 + 2 * (K_STAGES + V_STAGES + 1) + 11 <= 31, "the barriers and the two words behind them fit 256 bytes");
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 31);
    int* abort_flag = reinterpret_cast<int*>(tmem_slot + 1);
    uint64_t* done = bars + 32;                                 // [2] giving up: the products that warps 1 and 3 issued are done
    float* exchange = reinterpret_cast<float*>(Kring);          // once every product is done: [2][2 streams][128 rows], maxima and sums

    pdl_trigger();
    const int tile = blockIdx.x / hq, head = blockIdx.x % hq;   // neighbours share a tile's length: the long ones start first
    const int req = tile_req[tile], q0 = tile_q0[tile];
    const int rows = min(span, q_len[req] - q0);
    const int tok0 = q_start[req] + q0;
    const int ctx = ctx_len[req];
    const int qpos0 = ctx - q_len[req] + q0;
    const int kvh = head / (hq / hkv);
    const int* table = block_table + (size_t)req_slot[req] * table_width;
    const int tid = threadIdx.x, warp = __shfl_sync(0xffffffffu, tid >> 5, 0), lane = tid & 31;

    // Two streams per CTA.  More than 128 rows: stream s has the queries 128 s ... and walks every key tile they see.
    // Otherwise (`shared`) both have the same queries, stream s the key tiles s, s + 2, ..., and they are merged at the end.
    const bool shared = rows <= BM;
    const int k_end = qpos0 + rows;                                                       // the last row sees keys up to its own position
    const int k_begin = ((window > 0 ? max(0, qpos0 - window + 1) : 0) / BN) * BN;
    // key tiles: those that hold kept first keys (keys below keep_first stay in sight behind the window), then from the
    // window's first tile on; the two runs never overlap
    const int n_kept = (window > 0 && keep_first > 0) ? min((keep_first + BN - 1) / BN, k_begin / BN) : 0;
    const int n_tiles = n_kept + (k_end - k_begin + BN - 1) / BN;
    const int count0 = shared ? (n_tiles + 1) / 2 : n_kept + (qpos0 + BM - k_begin + BN - 1) / BN;      // tiles of stream 0
    // Stream 1's window begins one tile later, unless both begin with the sequence's first key: the tile that the window of
    // stream 0 begins in is none of stream 1's, which lets it go unread.  It comes first then, before the kept keys' tiles.
    const int passes = !shared && window > 0 && qpos0 - window + 1 >= 0 && keep_first <= k_begin;
    const int count1 = shared ? n_tiles / 2 : n_tiles - passes;
    auto tile_of = [&](int stream, int i) { return shared ? 2 * i + stream : i + (stream & passes); };
    // a value tile's place in its ring, and the parity of its turn there
    auto v_slot = [&](int j) { return shared ? j % value_slots(true) : j % value_slots(false); };
    auto v_turn = [&](int j) { return (uint32_t)(shared ? j / value_slots(true) : j / value_slots(false)) & 1; };
    auto tile_k0 = [&](int j) { return j < n_kept + passes && j >= passes ? (j - passes) * BN : k_begin + (j < passes ? 0 : j - n_kept) * BN; };
    if (tid == 0) {
        // a tile is free when both streams' products are done; the tiles that stream 0 no longer sees are never waited for
        for (int s = 0; s < K_STAGES; ++s) { mbar_init(k_full + s, 1); mbar_init(k_empty + s, shared ? 1 : 2); }
        for (int s = 0; s <= V_STAGES; ++s) { mbar_init(v_full + s, 1); mbar_init(v_empty + s, shared ? 1 : 2); }
        mbar_init(v_clean, 1);
        for (int s = 0; s < 2; ++s) {
            mbar_init(q_full + s, 1);
            mbar_init(s_full + s, 1);
            mbar_init(s_free + s, SOFTMAX_THREADS / 64);       // one arrival per warp of the stream, by its first lane after the warp has met
            mbar_init(p_full + 2 * s, SOFTMAX_THREADS / 64);
            mbar_init(p_full + 2 * s + 1, SOFTMAX_THREADS / 64);
            mbar_init(o_done + s, 1);
            mbar_init(done + s, 1);
        }
        *abort_flag = 0;
        mbar_init_fence();
    }
    if (warp == 1) {    // scores and outputs of two streams: 512 columns, all of this SM's tensor memory
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)), "r"(512) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    tcgen05_fence_before();
    __syncthreads();
    tcgen05_fence_after();
    const uint32_t tmem_base = __shfl_sync(0xffffffffu, *tmem_slot, 0);      // the same in every lane: kept in a uniform register
    pdl_wait();          // the queries, and this step's keys and values, come from the kernel before
    CISR_TRACE_WAITED();

    auto gave_up = [&]() {
        atomicExch(error, 5);
        *(volatile int*)abort_flag = 1;
    };
    auto wait = [&](uint64_t* bar, uint32_t parity) -> bool {     // false: leave (this or another role gave up)
        if (mbar_test(bar, parity)) return true;                  // the usual case: the phase is over already
        if (*(volatile int*)abort_flag) return false;
        if (mbar_wait(bar, parity)) return true;
        gave_up();
        return false;
    };
    int requested = 0;                                            // producers: tiles
    auto warp_wait = [&](uint64_t* bar, uint32_t parity) { return (bool)__all_sync(0xffffffffu, wait(bar, parity)); };

    if (warp == 0 || warp == 2) {
        // ------------------------------------------------------------ producers: warp 0 the queries and the keys, warp 2 the values
        const bool values = warp == 2;
        uint64_t* full = values ? v_full : k_full;
        uint64_t* empty = values ? v_empty : k_empty;
        unsigned char* ring = values ? Vring : Kring;
        const CUtensorMap* map = values ? &map_v : &map_k;
        auto load_queries = [&](int s) {
            mbar_expect_tx(q_full + s, (uint32_t)Q_BYTES);
            for (int sub = 0; sub < NSUB; ++sub) tma_load_2d((s ? Qs1 : Qs) + sub * SUB_BYTES, &map_q, head * D + sub * 64, tok0 + s * BM, q_full + s);
        };
        if (!values && lane == 0) load_queries(0);
        const int box_rows = min(page_size, BN), boxes = BN / box_rows;
        bool ok = true;
        for (int j = 0; j < n_tiles; ++j) {
            const int s = values ? v_slot(j) : j % K_STAGES;
            if (j >= (values ? value_slots(shared) : K_STAGES)) ok = warp_wait(empty + s, (values ? v_turn(j) : (j / K_STAGES) & 1) ^ 1);
            if (!ok) break;
            if (lane == 0) mbar_expect_tx(full + s, (uint32_t)KV_BYTES);
            __syncwarp();
            for (int b = lane; b < NSUB * boxes; b += 32) {       // lane b: box b (64-column half, run of box_rows keys)
                const int i = b % boxes, sub = b / boxes;
                const int kpos = tile_k0(j) + i * box_rows;
                const int page = kpos < k_end ? __ldg(table + kpos / page_size) : -1;     // the table is older than the kernel before
                const int row = page < 0 ? cache_rows : (page * hkv + kvh) * page_size + kpos % page_size;   // beyond the cache: zeros
                tma_load_2d(ring + s * KV_BYTES + sub * KV_SUB + i * box_rows * 128, map, sub * 64, row, full + s);
            }
            if (j == 0 && !values && !shared && lane == 0) load_queries(1);
            requested = j + 1;
        }
        if (values && ok && tile_k0(n_tiles - 1) + BN > k_end) {
            // Value rows beyond the last key were never written, or are left over from another request: they must not
            // meet the zero probabilities of those keys (0 * NaN).  They lie in the last tile; once it has landed its
            // rows beyond the keys are zeroed, before any output product reads them.
            const int j = n_tiles - 1, kt = tile_k0(j);
            if (warp_wait(v_full + v_slot(j), v_turn(j))) {
                unsigned char* Vs = Vring + v_slot(j) * KV_BYTES;
                const int r0 = k_end - kt;                        // first row beyond the keys
                for (int e = lane; e < (BN - r0) * NSUB * 8; e += 32) {
                    const int r = r0 + e / (NSUB * 8), c = e % (NSUB * 8);
                    *reinterpret_cast<uint4*>(Vs + (c >> 3) * KV_SUB + r * 128 + (((c & 7) ^ (r & 7)) << 4)) = make_uint4(0, 0, 0, 0);
                }
                asm volatile("fence.proxy.async.shared::cta;" ::: "memory");   // the zeroed rows before the tensor core reads them
                __syncwarp();
                if (lane == 0) mbar_arrive(v_clean);
            }
        }
    } else if (warp < FIRST_SOFTMAX_WARP) {
        // ------------------------------------------------------------ products
        // The whole warp walks the tiles and looks at the barriers; one lane issues.
        constexpr uint32_t idesc_s = umma_idesc(BN);
        constexpr uint32_t idesc_o = umma_idesc(D) | UMMA_B_MN_MAJOR;
        const bool clean_last = tile_k0(n_tiles - 1) + BN > k_end;
        // descriptor addresses count 16 bytes; every tile lies below 256 KB, so the sums stay inside the field
        const uint64_t desc_q0 = umma_desc(Qs), desc_q1 = umma_desc(Qs1), desc_k0 = umma_desc(Kring), desc_v0 = umma_desc_mn_major(Vring, KV_SUB);
        // the first tile, where stream 1 passes it over: once it has landed it is free as far as stream 1 goes
        auto pass_over = [&](uint64_t* full, uint64_t* empty) -> bool {
            if (!passes) return true;
            if (!warp_wait(full, 0)) return false;
            if (lane == 0) mbar_arrive(empty);
            __syncwarp();
            return true;
        };
        // S = Q K(j)^T of a stream's i-th tile
        auto score_product = [&](int stream, int i) -> bool {
            const int j = tile_of(stream, i), s = j % K_STAGES;
            if (!warp_wait(k_full + s, (j / K_STAGES) & 1)) return false;
            tcgen05_fence_after();
            const uint64_t k_desc = desc_k0 + s * (KV_BYTES >> 4), q_desc = shared || !stream ? desc_q0 : desc_q1;
#pragma unroll
            for (int kd = 0; kd < D / 16; ++kd)                   // 16 of the head's dimensions per step
                umma_bf16_elect(tmem_base + (uint32_t)(stream * BN), q_desc + (kd >> 2) * (SUB_BYTES >> 4) + 2 * (kd & 3),
                                k_desc + (kd >> 2) * (KV_SUB >> 4) + 2 * (kd & 3), idesc_s, kd != 0);
            umma_commit_elect(s_full + stream);
            umma_commit_elect(k_empty + s);
            return true;
        };
        // O += P V(j), half a tile's keys at a time, as their P arrives
        auto output_product = [&](int stream, int i) -> bool {
            const int j = tile_of(stream, i), s = v_slot(j);
            if (!warp_wait(v_full + s, v_turn(j))) return false;
            if (clean_last && j == n_tiles - 1 && !warp_wait(v_clean, 0)) return false;
            const uint64_t v_desc = desc_v0 + s * (KV_BYTES >> 4);
            const uint32_t tmem_p = OWN_P ? tmem_base + TMEM_P + (uint32_t)(stream * 64) : tmem_base + (uint32_t)(stream * BN);
#pragma unroll
            for (int half = 0; half < 2; ++half) {
                if (!warp_wait(p_full + 2 * stream + half, i & 1)) return false;
                tcgen05_fence_after();
#pragma unroll
                for (int ks = half * 4; ks < half * 4 + 4; ++ks)  // 16 keys per step: 8 columns of P, V two 8-row groups down
                    umma_bf16_ts_elect(tmem_base + TMEM_O + (uint32_t)(stream * D), tmem_p + 8 * ks, v_desc + ks * (16 * 128 >> 4), idesc_o, (i | ks) != 0);
            }
            umma_commit_elect(v_empty + s);
            if (OWN_P || i == (stream ? count1 : count0) - 1) umma_commit_elect(o_done + stream);
            return true;
        };
        if (OWN_P) {
            // a warp per stream
            const int stream = warp >> 1, count = stream ? count1 : count0;
            bool ok = count > 0 && warp_wait(q_full + (shared ? 0 : stream), 0);
            if (stream) ok = ok && pass_over(k_full, k_empty);
            ok = ok && score_product(stream, 0);
            if (stream) ok = ok && pass_over(v_full, v_empty);
            for (int i = 0; i < count && ok; ++i) {
                if (i + 1 < count) ok = warp_wait(s_free + stream, i & 1) && score_product(stream, i + 1);
                ok = ok && output_product(stream, i);
            }
        } else if (warp == 1) {
            // One warp for both streams, in turn, which keeps one stream's exponentials beside the other's products (with a
            // warp each the streams fell into step: 188 us against 164 for 4096 queries of 32 heads).  Products run in the
            // order they are issued, so a stream's next scores are written over its P after it was read.
            bool ok = warp_wait(q_full, 0) && score_product(0, 0);
            if (ok && count1 > 0) ok = (shared || warp_wait(q_full + 1, 0)) && pass_over(k_full, k_empty) && score_product(1, 0) && pass_over(v_full, v_empty);
            for (int i = 0; i < max(count0, count1) && ok; ++i)
                for (int stream = 0; stream < 2 && ok; ++stream) {
                    const int count = stream ? count1 : count0;
                    if (i < count) ok = output_product(stream, i);
                    if (ok && i + 1 < count) ok = score_product(stream, i + 1);
                }
        }
    } else {
        // ------------------------------------------------------------ softmax and output
        const int quarter = warp & 3;                              // the 32 tensor-memory lanes this warp may touch
        const int stream = (warp - FIRST_SOFTMAX_WARP) >> 2;
        const int row = quarter * 32 + lane;
        const int qbase = qpos0 + (shared ? 0 : stream * BM);      // the stream's first query
        const int qpos = qbase + row;
        const int count = stream ? count1 : count0;
        const uint32_t lane_base = (uint32_t)(quarter * 32) << 16;
        const uint32_t tmem_own = tmem_base + TMEM_O + lane_base + (uint32_t)(stream * D);     // this thread's row of its accumulator
        const uint32_t s_addr = tmem_base + lane_base + (uint32_t)(stream * BN);
        const uint32_t p_addr = OWN_P ? tmem_base + TMEM_P + lane_base + (uint32_t)(stream * 64) : s_addr;
        const float scale2 = SOFTCAP ? 1.f : scale * LOG2E;        // bent scores come in base-2 units
        // bent scores lie in (-cap, cap): where 2^(cap log2 e) is far from a float's range they need no running max, and
        // every exponential is taken against 0
        const bool bounded = SOFTCAP && softcap * LOG2E <= 60.f;
        float m_used = bounded ? 0.f : -INFINITY, l = 0.f;
        bool ok = true;
        for (int i = 0; i < count; ++i) {
            const int kt = tile_k0(tile_of(stream, i));             // the tile's first key
            ok = warp_wait(s_full + stream, i & 1);
            if (!ok) break;
            tcgen05_fence_after();
            // tiles on the diagonal, at the window's start and at the end of the keys need the per-element mask
            const bool edge = kt + BN - 1 > qbase || kt + BN > k_end || (window > 0 && kt <= qbase + BM - 1 - window);
            const int last = min(qpos, k_end - 1) - kt;             // the last key in sight, counted inside the tile
            const int first = window > 0 ? qpos - window + 1 - kt : 0, kept = window > 0 ? keep_first - kt : 0;
            // columns c0 .. c0 + N - 1 of the scores, bent and masked
            auto prepare = [&](auto width, int c0, uint32_t* v) {
                constexpr int N = decltype(width)::value;
                if (SOFTCAP) {
                    const Bend bend(scale, softcap);
#pragma unroll
                    for (int c = 0; c < N; c += 4) {
                        float x[4];
#pragma unroll
                        for (int e = 0; e < 4; ++e) x[e] = __uint_as_float(v[c + e]);
                        bend.four(x[0], x[1], x[2], x[3]);
#pragma unroll
                        for (int e = 0; e < 4; ++e) v[c + e] = __float_as_uint(x[e]);
                    }
                }
                if (edge) {
                    const int l0 = last - c0, f0 = first - c0, p0 = kept - c0;
#pragma unroll
                    for (int c = 0; c < N; ++c)
                        if (c > l0 || (c < f0 && c >= p0)) v[c] = __float_as_uint(-INFINITY);
                }
            };
            float mx[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
            auto take_max = [&](auto width, const uint32_t* v) {
                constexpr int N = decltype(width)::value;
#pragma unroll
                for (int c = 0; c < N; c += 8)
#pragma unroll
                    for (int e = 0; e < 4; ++e) mx[e] = max_nan(mx[e], __uint_as_float(v[c + 2 * e]), __uint_as_float(v[c + 2 * e + 1]));
            };
            auto scores_taken = [&]() {                             // the stream's next scores may be written (OWN_P)
                if (!OWN_P) return;
                tcgen05_fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive(s_free + stream);
            };
            const std::integral_constant<int, 32> part;
            const std::integral_constant<int, BN> whole;
            uint32_t raw[TWO_PASSES ? 64 : BN];
            if (TWO_PASSES) {
                if (!bounded) {
                    tmem_load32_nowait(s_addr, raw);
#pragma unroll 1
                    for (int c0 = 0; c0 < BN; c0 += 64) {
                        tmem_load_wait();
                        tmem_load32_nowait(s_addr + c0 + 32, raw + 32);
                        prepare(part, c0, raw);
                        take_max(part, raw);
                        tmem_load_wait();
                        if (c0 + 64 < BN) tmem_load32_nowait(s_addr + c0 + 64, raw);
                        prepare(part, c0 + 32, raw + 32);
                        take_max(part, raw + 32);
                    }
                }
                tmem_load32_nowait(s_addr, raw);
            } else {
#pragma unroll
                for (int c0 = 0; c0 < BN; c0 += 32) tmem_load32_nowait(s_addr + c0, raw + c0);
                tmem_load_wait();
                scores_taken();
                prepare(whole, 0, raw);
                if (!bounded) take_max(whole, raw);
            }
            float alpha = 1.f;
            if (!bounded) {
                const float m_tile = max_nan(max_nan(mx[0], mx[1], mx[2]), mx[3], mx[3]) * scale2;     // the scale is positive: the max of the raw scores, scaled
                // the max in use moves only when it lags by more than RESCALE_STEP; the first finite max is taken as it is;
                // a NaN is taken too, and its row's sums are NaN from then on
                if (!(m_tile <= m_used + RESCALE_STEP) || (m_used == -INFINITY && m_tile > -INFINITY)) {
                    alpha = m_used == -INFINITY ? 0.f : fast_exp2(m_used - m_tile);
                    m_used = m_tile;
                }
            }
            if (OWN_P && i > 0) {                                   // P of the tile before has been read, and O is this thread's
                ok = warp_wait(o_done + stream, (i - 1) & 1);
                if (!ok) break;
                tcgen05_fence_after();
            }
            if (i > 0 && __any_sync(0xffffffffu, alpha != 1.f)) {
                // (not OWN_P: the output product of the tile before ran before the scores at hand were multiplied.)
                // Tensor-memory access is warp-wide: most lanes go with alpha 1
                if (TWO_PASSES) tmem_load_wait();
#pragma unroll 1
                for (int c0 = 0; c0 < D; c0 += 32) {
                    uint32_t acc[32];
                    tmem_load32(tmem_own + c0, acc);
#pragma unroll
                    for (int c = 0; c < 32; ++c) acc[c] = __float_as_uint(__uint_as_float(acc[c]) * alpha);
                    tmem_store32(tmem_own + c0, acc);
                }
            }
            const float m_ref = m_used == -INFINITY ? 0.f : m_used;
            const uint64_t scale_pair = pack2(scale2, scale2), minus_m = pack2(-m_ref, -m_ref);
            uint64_t sums[2] = {0, 0};
            // P = 2^(s - m) of 32 columns, rounded to bfloat16 for the product; the sum keeps the unrounded values
            auto powers = [&](int c0, uint32_t* v) {
#pragma unroll
                for (int c = 0; c < 32; c += 2) {
                    float p0, p1;
                    unpack2(fma2(pack2(__uint_as_float(v[c]), __uint_as_float(v[c + 1])), scale_pair, minus_m), p0, p1);
                    p0 = fast_exp2(p0);                             // -inf (masked) gives 0
                    p1 = fast_exp2(p1);
                    sums[(c >> 1) & 1] = add2(sums[(c >> 1) & 1], pack2(p0, p1));
                    __nv_bfloat162 pair = __floats2bfloat162_rn(p0, p1);
                    v[c >> 1] = *reinterpret_cast<uint32_t*>(&pair);
                }
                tmem_store16_nowait(p_addr + (c0 >> 1), v);
            };
            auto half_done = [&](int half) {                        // the output product of these 64 keys may run
                tmem_store_wait();
                tcgen05_fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive(p_full + 2 * stream + half);
            };
            if (TWO_PASSES) {
                // P goes over scores that have been taken: its columns c0 / 2 ... lie in the 32 columns at hand or before them
#pragma unroll 1
                for (int half = 0; half < 2; ++half) {
                    tmem_load_wait();
                    tmem_load32_nowait(s_addr + 64 * half + 32, raw + 32);
                    prepare(part, 64 * half, raw);
                    powers(64 * half, raw);
                    tmem_load_wait();
                    if (half == 0) tmem_load32_nowait(s_addr + 64, raw);
                    else scores_taken();
                    prepare(part, 64 * half + 32, raw + 32);
                    powers(64 * half + 32, raw + 32);
                    half_done(half);
                }
            } else {
#pragma unroll
                for (int c0 = 0; c0 < BN; c0 += 32) {
                    powers(c0, raw + c0);
                    if (c0 & 32) half_done(c0 >> 6);
                }
            }
            float s0, s1;
            unpack2(add2(sums[0], sums[1]), s0, s1);
            l = l * alpha + (s0 + s1);
        }
        if (ok && count > 0) ok = wait(o_done + stream, OWN_P ? (count - 1) & 1 : 0);
        const bool all_ok = __all_sync(0xffffffffu, ok);
        if (!all_ok) *(volatile int*)abort_flag = 1;
        const float sink = sink_heads ? sink_heads[head] : sink_all;     // one per head where given
        tcgen05_fence_after();
        if (!shared) {
            const int mine = stream * BM + row;
            if (all_ok) {
                float total = l;
                if (total > 0.f && sink > -INFINITY) total += exp2f(sink * LOG2E - m_used);   // the sink: one more term of the denominator, no value
                const bool some = m_used != -INFINITY;             // a key in sight (NaN and infinite scores pass through)
                const float inv = fabsf(m_used) < INFINITY ? 1.f / total : NAN;
                bf16* dst = out + ((size_t)(tok0 + mine) * hq + head) * D;
#pragma unroll 1
                for (int c0 = 0; c0 < D; c0 += 32) {
                    uint32_t acc[32];
                    tmem_load32(tmem_own + c0, acc);               // warp-wide, also for rows beyond the portion
                    if (mine < rows) {
#pragma unroll
                        for (int q = 0; q < 4; ++q) {
                            uint32_t w[4];
#pragma unroll
                            for (int e = 0; e < 4; ++e) {
                                const int c = 8 * q + 2 * e;
                                __nv_bfloat162 pair = __floats2bfloat162_rn(some ? __uint_as_float(acc[c]) * inv : 0.f, some ? __uint_as_float(acc[c + 1]) * inv : 0.f);
                                w[e] = *reinterpret_cast<uint32_t*>(&pair);
                            }
                            *reinterpret_cast<uint4*>(dst + c0 + 8 * q) = make_uint4(w[0], w[1], w[2], w[3]);
                        }
                    }
                }
            }
        } else {
            // The two streams of a row meet: with m the larger of their maxima, out = (O_0 2^(m_0 - m) + O_1 2^(m_1 - m)) /
            // (l_0 2^(m_0 - m) + l_1 2^(m_1 - m)); each stream writes half of the output columns.
            asm volatile("bar.sync 1, %0;" ::"n"(SOFTMAX_THREADS) : "memory");       // both streams' products are done
            exchange[stream * BM + row] = count > 0 ? m_used : -INFINITY;
            exchange[(2 + stream) * BM + row] = l;
            tcgen05_fence_before();
            asm volatile("bar.sync 1, %0;" ::"n"(SOFTMAX_THREADS) : "memory");
            if (all_ok && !*(volatile int*)abort_flag) {
                tcgen05_fence_after();
                const float m0 = exchange[row], m1 = exchange[BM + row], m = fmaxf(m0, m1);
                const float w0 = m0 == -INFINITY ? 0.f : fast_exp2(m0 - m), w1 = m1 == -INFINITY ? 0.f : fast_exp2(m1 - m);
                float total = exchange[2 * BM + row] * w0 + exchange[3 * BM + row] * w1;
                if (total > 0.f && sink > -INFINITY) total += exp2f(sink * LOG2E - m);
                const float inv = total > 0.f ? 1.f / total : 0.f;
                const float f0 = w0 * inv, f1 = w1 * inv;
                const uint32_t tmem_o = tmem_base + TMEM_O + lane_base;
                bf16* dst = out + ((size_t)(tok0 + row) * hq + head) * D;
#pragma unroll 1
                for (int c0 = stream * (D / 2); c0 < (stream + 1) * (D / 2); c0 += 32) {
                    uint32_t a0[32], a1[32];
                    tmem_load32_nowait(tmem_o + c0, a0);            // warp-wide, also for rows beyond the portion
                    tmem_load32_nowait(tmem_o + D + c0, a1);
                    tmem_load_wait();
                    if (row < rows) {
#pragma unroll
                        for (int q = 0; q < 4; ++q) {
                            uint32_t w[4];
#pragma unroll
                            for (int e = 0; e < 4; ++e) {
                                const int c = 8 * q + 2 * e;
                                // a stream without keys for this row weighs nothing, whatever its accumulator holds; NaN passes through
                                const float x0 = (w0 != 0.f ? __uint_as_float(a0[c]) * f0 : 0.f) + (w1 != 0.f ? __uint_as_float(a1[c]) * f1 : 0.f);
                                const float x1 = (w0 != 0.f ? __uint_as_float(a0[c + 1]) * f0 : 0.f) + (w1 != 0.f ? __uint_as_float(a1[c + 1]) * f1 : 0.f);
                                __nv_bfloat162 pair = __floats2bfloat162_rn(x0, x1);
                                w[e] = *reinterpret_cast<uint32_t*>(&pair);
                            }
                            *reinterpret_cast<uint4*>(dst + c0 + 8 * q) = make_uint4(w[0], w[1], w[2], w[3]);
                        }
                    }
                }
            }
        }
    }
    tcgen05_fence_before();
    __syncthreads();
    if (*(volatile int*)abort_flag) {
        if (warp == 0) {
            mbar_wait(q_full, 0);
            if (!shared && requested) mbar_wait(q_full + 1, 0);
            wait_for_copies(k_full, requested, K_STAGES);
        }
        if (warp == 2) wait_for_copies(v_full, requested, value_slots(shared));
        if (warp == 1 || (OWN_P && warp == 3)) wait_for_products_elect(done + (warp >> 1));
        __syncthreads();
    }
    if (warp == 1) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(512) : "memory");
}
}  // namespace

CISR_EXPORT int cisr_attn_tcgen05_head_dim() { return D; }
CISR_EXPORT int cisr_attn_tcgen05_tile() { return BM; }
// The slots of the key ring, or of the value ring for a tile whose streams share their queries or not, and how many warps issue
// products (one per stream, or one for both): what a check of the rings' turns needs to know.
CISR_EXPORT int cisr_attn_tcgen05_slots(int values, int shared) { return values ? value_slots(shared != 0) : K_STAGES; }
CISR_EXPORT int cisr_attn_tcgen05_product_warps() { return OWN_P ? 2 : 1; }
CISR_EXPORT void cisr_attn_tcgen05_set_pdl(int on) { g_pdl = on != 0; }

// `error_flag`: one zeroed int in device memory that the kernel sets (to 5) when one of its waits ran out.
CISR_EXPORT int cisr_attn_tcgen05_init(int* error_flag) {
    if (int status = tma_load_encoder()) return status;
    g_error = error_flag;
    return 0;
}

// 1 when the kernel takes this page size.
CISR_EXPORT int cisr_attn_tcgen05_ok(int page_size) {
    return page_size > 0 && page_size % 8 == 0 && (BN % page_size == 0 || page_size % BN == 0);
}

// Attention of portions: q, out [n_tokens, hq, D]; tiles of `span` (128 or 256) queries given as (request, first query) pairs.
CISR_EXPORT int cisr_attn_prefill_tcgen05(const void* q, void* out, int n_tokens, const void* k_cache, const void* v_cache,
                                          int n_pages, const int* req_slot, const int* block_table, int table_width,
                                          const int* tile_req, const int* tile_q0, int n_tiles, int span, const int* q_start,
                                          const int* q_len, const int* ctx_len, int hq, int hkv, int page_size, float scale, float softcap,
                                          int window, int keep_first, float sink, const float* sink_heads, void* stream) {
    if (n_tiles <= 0) return 0;
    if (!g_encode || !g_error) return -13;
    if (hq % hkv || (span != BM && span != 2 * BM) || !cisr_attn_tcgen05_ok(page_size) || (SOFTCAP ? !(softcap > 0.f) : softcap != 0.f)) return -2;
    const long long cache_rows = (long long)n_pages * hkv * page_size;
    if (cache_rows <= 0 || cache_rows >= (1ll << 31) || (((uintptr_t)k_cache | (uintptr_t)v_cache | (uintptr_t)q | (uintptr_t)out) & 15)) return -2;
    const int box_rows = page_size < BN ? page_size : BN;
    CUtensorMap map_q, map_k, map_v;
    int status = cached_map(&map_q, q, n_tokens, hq * D, BM, 64);
    if (status) return status;
    if ((status = cached_map(&map_k, k_cache, cache_rows, D, box_rows, 64))) return status;
    if ((status = cached_map(&map_v, v_cache, cache_rows, D, box_rows, 64))) return status;
    const size_t smem = SMEM_FIXED;
    static_assert(SMEM_FIXED <= 227 * 1024, "a CTA has 227 KB of shared memory");
    static size_t configured = 0;
    if (smem > configured) {
        cudaError_t e = cudaFuncSetAttribute(attn_prefill_tcgen05_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        if (e != cudaSuccess) return (int)e;
        configured = smem;
    }
    return launch_kernel(attn_prefill_tcgen05_kernel, dim3((unsigned)n_tiles * hq), dim3(THREADS), smem, (cudaStream_t)stream, g_pdl, map_q,
                         map_k, map_v, (bf16*)out, (int)cache_rows, req_slot, block_table, table_width, tile_req, tile_q0, span,
                         q_start, q_len, ctx_len, hq, hkv, page_size, scale, softcap, window, keep_first, sink, sink_heads, g_error);
}
