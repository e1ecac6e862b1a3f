// Backward of the absorbed-latent causal MLA forward
// (mla_compressed_attention_backward_cuda) on the sm_100a tensor cores.
//
// The interface gives no scratch memory, the gradients of the shared latent /
// rotary key sum over every head and every later query, and the operands are wide
// (576 score columns, 512 value columns), so the work is split the way the
// reference splits it (kernels/attention/mla/sm89.cu:295 query side, :356 key
// side): one kernel owns the key-side gradients, one owns the query-side
// gradients, and each recomputes P from the saved LSE.  Both are tcgen05 kernels whose score tiles are S^T = K Q^T, keys on
// the tensor-memory lanes and (token, head) rows on the columns, so that one thread owns one key and the per-row constants
// (LSE, delta, token index) are read from shared memory.
//
// One call launches, on the caller's stream:
//   1. absorbed_delta_kernel: delta[row] = sum_c dO[row,c] O[row,c], kept in the
//      first four bytes of each dquery_rope row (an output the last kernel
//      overwrites, so no scratch is needed);
//   2. absorbed_backward_key_kernel: cluster of two CTAs = (128-key tile, one part of the rows).  The keys stay in shared
//      memory; the 96-row tiles at or after the diagonal stream by and stay there from the score products to the gradient
//      products dlatent += dS^T query_latent + P^T dO and dkey_rope += dS^T query_rope.  Single writer per output element,
//      no atomics; with several parts absorbed_backward_reduce_kernel adds them in order;
//   3. absorbed_backward_query_kernel: CTA = 64 (token, head) rows, resident as the
//      B operands query_latent | query_rope | dO (136 KB); every 128-key tile up
//      to the diagonal streams by twice: for S^T / dP^T, and again as the
//      MN-major A operand of dQ^T += K^T dS^T (output columns on the lanes, rows on
//      the columns; dS^T goes through shared memory as the B operand).
//
// Warps 0-7: softmax; warp 8: MMA issue (whole warp, one elected lane executes); warp 9: TMA loads.  Every wait is bounded.
#include "mla.h"
#include "cuda_common.h"
#include "attention_internal.h"
#include "sm100_primitives.cuh"
#include "../common/launch.h"
#include "../common/tensor_map.h"

#include <algorithm>
#include <cstddef>
#include <cstdint>
#include <stdexcept>

namespace dscuda {
namespace {

using namespace sm100;

constexpr int RANK = MLA_KV_RANK;             // 512
constexpr int ROPE = MLA_ROPE_SIZE;           // 64
constexpr int CHUNKS = (RANK + ROPE) / 64;    // 9 column chunks of 64; chunk 8 is the rotary part
constexpr int LATENT_CHUNKS = RANK / 64;      // 8
constexpr int KEYS = 128;                     // keys per tile = MMA M = tensor-memory lanes
constexpr int ROWS = 64;                      // (token, head) rows per tile = MMA N
constexpr int KEY_CHUNK = KEYS * 128;         // 16 KB: [128 keys x 64 bf16]
constexpr int ROW_CHUNK = ROWS * 128;         //  8 KB: [64 rows x 64 bf16]
constexpr int THREADS = 320;
constexpr int MMA_WARP = 8;
constexpr int LOAD_WARP = 9;
constexpr int TMEM_COLUMNS = 512;
constexpr int MISC_BYTES = 2048;
constexpr float LOG2E = 1.4426950408889634F;

__device__ int absorbed_backward_status = 0;

struct AbsorbedBackwardParams {
    CUtensorMap q_lat;      // [B*T*H, 512] box 64 x 64
    CUtensorMap q_rope;     // [B*T*H, 64]  box 64 x 64
    CUtensorMap d_out;      // [B*T*H, 512] box 64 x 64
    CUtensorMap k_lat;      // [B*T, 512]   box 128 x 64
    CUtensorMap k_rope;     // [B*T, 64]    box 128 x 64
    // key side; batch entries apart, so rows and keys past the end of one read as zero
    CUtensorMap key_lat8;   // kv_latent, box 64 keys x 8 chunks
    CUtensorMap key_rope1;  // key_rope, box 64 keys
    CUtensorMap row_q8;     // query_latent, box 48 rows x 8 chunks
    CUtensorMap row_q2;     // ... x 2 chunks
    CUtensorMap row_do8;    // dO likewise
    CUtensorMap row_do2;
    CUtensorMap row_rope;   // query_rope, box 48 rows
    CUtensorMap dlatent_out;    // stores of 32 keys: 64 bf16 columns of dlatent, 32 fp32 columns of a partial sum
    CUtensorMap partials;
    __nv_bfloat16* dq_lat;  // [B,T,H,512]
    __nv_bfloat16* dq_rope; // [B,T,H,64]; the first float of each row holds delta until the query kernel overwrites it
    __nv_bfloat16* dlatent; // [B,T,512]
    __nv_bfloat16* dk_rope; // [B,T,64]
    const float* lse;       // [B,H,T]
    int batch;
    int sequence;
    int heads;
    int key_chunk;          // key side: at most this many 96-row tiles per cluster
    int key_direct;         // key side: 1 when every key tile has a single part (results go straight to the outputs)
    float scale;
    float scale_log2;
};

// Key side work split.  Key tile kt meets the rows of its own first token (row kt*128*H) and all later ones, in tiles of 96;
// they are cut into ceil(count / key_chunk) parts of equal size, one cluster each, so that the first key tiles (which meet
// every row) do not set the kernel's duration.  With more than one part the clusters write fp32 partial sums, part p of key
// row (b, key) at scratch[((p*B + b)*T + key)*576 ..], and absorbed_backward_reduce_kernel adds them in part order.  The
// scratch is the dquery_latent output, which the query-side kernel overwrites last.
constexpr int KEY_SIDE_ROWS = 96;

__device__ __forceinline__ int key_tile_row_tiles(const AbsorbedBackwardParams& p, int key_tile) {
    return (p.sequence * p.heads - key_tile * KEYS * p.heads + KEY_SIDE_ROWS - 1) / KEY_SIDE_ROWS;
}

__device__ __forceinline__ int key_tile_parts(const AbsorbedBackwardParams& p, int key_tile) {
    return (key_tile_row_tiles(p, key_tile) + p.key_chunk - 1) / p.key_chunk;
}

// Per-row constants of a 64-row tile, written by the load warp, read by every softmax thread.
struct RowConstants {
    alignas(16) float lse2[ROWS];     // LSE * log2 e
    alignas(16) float delta[ROWS];
    alignas(16) int token[ROWS];      // token index of the row, -1 for rows past the end of the sequence
};

__device__ __forceinline__ float stored_delta(const AbsorbedBackwardParams& p, size_t global_row) {
    return *reinterpret_cast<const float*>(p.dq_rope + global_row * ROPE);
}

// Lanes of one warp fill the constants of rows [row0, row0 + 64) of sequence `b`.
__device__ __forceinline__ void fill_row_constants(const AbsorbedBackwardParams& p, RowConstants& rc, int b, int row0, int lane) {
    const int rows_per_sequence = p.sequence * p.heads;
#pragma unroll
    for (int e = 0; e < ROWS / 32; ++e) {
        const int n = e * 32 + lane;
        const int row = row0 + n;
        float lse_value = 0.0F, delta_value = 0.0F;
        int token = -1;
        if (row < rows_per_sequence) {
            token = row / p.heads;
            const int head = row - token * p.heads;
            lse_value = p.lse[(static_cast<size_t>(b) * p.heads + head) * p.sequence + token] * LOG2E;
            delta_value = stored_delta(p, static_cast<size_t>(b) * rows_per_sequence + row);
        }
        rc.lse2[n] = lse_value;
        rc.delta[n] = delta_value;
        rc.token[n] = token;
    }
}

// One thread's share of a score tile: key `key_pos` (its tensor-memory lane) against 32 of the
// tile's 64 rows.  Reads S^T and dP^T (fp32) from tensor memory and returns P^T and
// dS^T = P^T (dP^T - delta) scale as packed bf16 pairs.  A key is visible to a row when
// key_pos <= token(row); rows past the end have token -1.
__device__ __forceinline__ void score_tile_share(const AbsorbedBackwardParams& p, uint32_t st_tmem, uint32_t dpt_tmem, const RowConstants& rc,
                                                 int group, int key_pos, bool masked, uint32_t (&p_packed)[16], uint32_t (&ds_packed)[16]) {
    uint32_t sb[32];
    float prob[32];
    tmem_ld_x32(st_tmem, sb);
    tmem_wait_ld();
    const float4* lse4 = reinterpret_cast<const float4*>(rc.lse2 + group * 32);
    const float4* delta4 = reinterpret_cast<const float4*>(rc.delta + group * 32);
    const int4* token4 = reinterpret_cast<const int4*>(rc.token + group * 32);
#pragma unroll
    for (int n = 0; n < 32; n += 4) {
        const float4 l = lse4[n / 4];
        prob[n] = exp2_approx(fmaf(__uint_as_float(sb[n]), p.scale_log2, -l.x));
        prob[n + 1] = exp2_approx(fmaf(__uint_as_float(sb[n + 1]), p.scale_log2, -l.y));
        prob[n + 2] = exp2_approx(fmaf(__uint_as_float(sb[n + 2]), p.scale_log2, -l.z));
        prob[n + 3] = exp2_approx(fmaf(__uint_as_float(sb[n + 3]), p.scale_log2, -l.w));
    }
    if (masked) {
#pragma unroll
        for (int n = 0; n < 32; n += 4) {
            const int4 t = token4[n / 4];
            prob[n] = key_pos <= t.x ? prob[n] : 0.0F;
            prob[n + 1] = key_pos <= t.y ? prob[n + 1] : 0.0F;
            prob[n + 2] = key_pos <= t.z ? prob[n + 2] : 0.0F;
            prob[n + 3] = key_pos <= t.w ? prob[n + 3] : 0.0F;
        }
    }
#pragma unroll
    for (int n = 0; n < 32; n += 2) {
        p_packed[n / 2] = pack_bf16x2(prob[n], prob[n + 1]);
    }
    tmem_ld_x32(dpt_tmem, sb);
    tmem_wait_ld();
#pragma unroll
    for (int n = 0; n < 32; n += 4) {
        const float4 d = delta4[n / 4];
        ds_packed[n / 2] = pack_bf16x2(prob[n] * (__uint_as_float(sb[n]) - d.x) * p.scale, prob[n + 1] * (__uint_as_float(sb[n + 1]) - d.y) * p.scale);
        ds_packed[n / 2 + 1] =
            pack_bf16x2(prob[n + 2] * (__uint_as_float(sb[n + 2]) - d.z) * p.scale, prob[n + 3] * (__uint_as_float(sb[n + 3]) - d.w) * p.scale);
    }
}

__device__ __forceinline__ void store_bf16x32(__nv_bfloat16* dst, const uint32_t* values) {
#pragma unroll
    for (int e = 0; e < 32; e += 8) {
        uint4 vec;
        vec.x = pack_bf16x2(__uint_as_float(values[e]), __uint_as_float(values[e + 1]));
        vec.y = pack_bf16x2(__uint_as_float(values[e + 2]), __uint_as_float(values[e + 3]));
        vec.z = pack_bf16x2(__uint_as_float(values[e + 4]), __uint_as_float(values[e + 5]));
        vec.w = pack_bf16x2(__uint_as_float(values[e + 6]), __uint_as_float(values[e + 7]));
        *reinterpret_cast<uint4*>(dst + e) = vec;
    }
}

__device__ __forceinline__ void store_f32x32(float* dst, const uint32_t* values) {
#pragma unroll
    for (int e = 0; e < 32; e += 4) {
        *reinterpret_cast<uint4*>(dst + e) = make_uint4(values[e], values[e + 1], values[e + 2], values[e + 3]);
    }
}

// ---------------------------------------------------------------------------
// delta[row] = sum_c dO[row,c] * O[row,c]; one warp per (token, head) row.  The result is parked
// in the first four bytes of the row's dquery_rope output.
// ---------------------------------------------------------------------------
__global__ void __launch_bounds__(256) absorbed_delta_kernel(__nv_bfloat16* dq_rope, const __nv_bfloat16* dout, const __nv_bfloat16* out,
                                                             size_t rows) {
    const int lane = threadIdx.x % 32;
    const size_t warp_stride = static_cast<size_t>(gridDim.x) * (blockDim.x / 32);
    grid_dependency_wait();
    for (size_t row = static_cast<size_t>(blockIdx.x) * (blockDim.x / 32) + threadIdx.x / 32; row < rows; row += warp_stride) {
        float sum = 0.0F;
#pragma unroll
        for (int part = 0; part < 2; ++part) {
            const uint4 a = __ldg(reinterpret_cast<const uint4*>(dout + row * RANK) + part * 32 + lane);
            const uint4 b = __ldg(reinterpret_cast<const uint4*>(out + row * RANK) + part * 32 + lane);
            const __nv_bfloat162* a2 = reinterpret_cast<const __nv_bfloat162*>(&a);
            const __nv_bfloat162* b2 = reinterpret_cast<const __nv_bfloat162*>(&b);
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                const float2 x = __bfloat1622float2(a2[e]), y = __bfloat1622float2(b2[e]);
                sum += x.x * y.x + x.y * y.y;
            }
        }
#pragma unroll
        for (int offset = 16; offset > 0; offset >>= 1) {
            sum += __shfl_xor_sync(0xffffffffU, sum, offset);
        }
        if (lane == 0) {
            *reinterpret_cast<float*>(dq_rope + row * ROPE) = sum;
        }
    }
}

// ---------------------------------------------------------------------------
// Key side.  A cluster of two CTAs takes 128 keys and a part of the rows; CTA r owns keys 64r..64r+63 of the tile (the A
// rows of every product, tcgen05.mma.cta_group::2 with M = 128) and supplies half of each B operand.  Per 96-row tile:
//
//   S^T = K Q^T, dP^T = latent dO^T  (N = 96, CTA r supplies its own 48 rows of the tile, all columns);
//   dlatent += dS^T Q + P^T dO       (N = 256 twice; K = 96 rows, CTA r supplies columns 128r..128r+127 of each half);
//   dkey_rope += dS^T Q_rope         (N = 128: both CTAs supply all 64 columns, so the result is there twice).
//
// The eight 64-column chunks of a CTA's own 48 rows sit in slots 0..7.  Chunks {2r, 2r+1, 4+2r, 4+2r+1} are in place as
// columns of the gradient products; the other four slots are refilled with the other CTA's rows of those columns as soon as
// the score MMAs have read them (the same scheme as in absorbed_attention.cu), and the rotary columns of all 96 rows are
// loaded once more into a place of their own.  So the scores are computed once per (key, row) pair and a CTA reads 168 KB
// from L2 for 64 x 96 pairs.
//
// What bounds it: shared memory.  The resident keys (72 KB), P and dS (32 KB) and one tile of rows (114 KB) fill it, so the
// chain scores -> softmax -> gradients of a tile is overlapped only by the loads of the next one: query_latent is loaded
// again while P^T dO runs.  96 rows and not 128 because 128 do not fit.  One CTA per (128 keys, half of dlatent), which this
// replaces, computed the scores twice, at the N = 64 rate: 1305 us at B=4 T=2048 H=16 against
// 592 us now, 46 against 11 us at B=2 T=33 H=32 (where a part also had at least 1024 rows).
//
// Tensor memory: dlatent 2 x 128 columns (lanes 0-63: columns 256a + 0..127, lanes 64-127: 256a + 128..255 of the same 64
// keys), dkey_rope 64, S^T 48 (lanes 64-127: rows 48..95), dP^T 48.
// Warps 0-7: softmax (thread = key x 24 rows) and results; 8: MMA issue in the leader, relay of "loaded" events in the other
// CTA; 9: TMA loads; 10: the rows' constants.
// ---------------------------------------------------------------------------
namespace ks {
constexpr int TILE_ROWS = KEY_SIDE_ROWS;
constexpr int HALF_ROWS = 48;                       // rows a CTA supplies
constexpr int SHARE_ROWS = 24;                      // rows of a softmax thread
constexpr int CTA_KEYS = 64;
constexpr int KEY_SLOT = CTA_KEYS * 128;            // 8 KB: [64 keys x 64 bf16]
constexpr int ROW_SLOT = HALF_ROWS * 128;           // 6 KB: [48 rows x 64 bf16]
constexpr int K_BYTES = CHUNKS * KEY_SLOT;
constexpr int P_OFFSET = K_BYTES;                   // P^T, then dS^T: [64 keys x 96 rows] as two 64-row chunks
constexpr int DS_OFFSET = P_OFFSET + 2 * KEY_SLOT;
constexpr int Q_OFFSET = DS_OFFSET + 2 * KEY_SLOT;
constexpr int DO_OFFSET = Q_OFFSET + LATENT_CHUNKS * ROW_SLOT;
constexpr int ROPE_OFFSET = DO_OFFSET + LATENT_CHUNKS * ROW_SLOT;       // own rows, for the scores
constexpr int ROPE_ALL_OFFSET = ROPE_OFFSET + ROW_SLOT;                 // all 96 rows, for dkey_rope
constexpr int MISC_OFFSET = ROPE_ALL_OFFSET + 2 * ROW_SLOT;
constexpr int SMEM_BYTES = MISC_OFFSET + 3072;
constexpr int KEY_THREADS = 352;
constexpr int CONSTANTS_WARP = 10;
constexpr int SLAB_BYTES = 32 * 128;
constexpr uint32_t TMEM_DLAT = 0;
constexpr uint32_t TMEM_DROPE = 256;
constexpr uint32_t TMEM_S = 320;
constexpr uint32_t TMEM_DP = 368;
static_assert(SMEM_BYTES <= 232448, "key-side shared memory");
static_assert(8 * 5 * SLAB_BYTES <= MISC_OFFSET, "result slabs lie in the operands' memory");

struct Rows {
    alignas(16) float lse2[TILE_ROWS];     // LSE * log2 e
    alignas(16) float delta[TILE_ROWS];
    alignas(16) int token[TILE_ROWS];      // -1 for rows past the end of the sequence
};

struct Shared {
    Rows rows[2];
    // completed by TMA transactions of this CTA, one phase per tile
    uint64_t k_full;
    uint64_t q_full;            // own rows: query_latent and the rotary chunk
    uint64_t do_full;           // own rows: dO
    uint64_t q_refilled;        // the other CTA's rows, and the rotary columns of all rows
    uint64_t do_refilled;
    // leader only: the same events of the other CTA, forwarded by its relay (one arrival)
    uint64_t peer_k_full;
    uint64_t peer_q_full;
    uint64_t peer_do_full;
    uint64_t peer_q_refilled;
    uint64_t peer_do_refilled;
    // completed by tcgen05.commit of the leader
    uint64_t q_refill_free;     // S has read the four slots only it needs
    uint64_t do_refill_free;
    uint64_t s_full;
    uint64_t dp_full;
    uint64_t q_free;            // dS^T Q has read everything of query_latent and query_rope
    uint64_t do_free;           // P^T dO too; P, dS and the accumulators are quiescent
    // leader only: one arrival per softmax warp of either CTA, P^T and dS^T are stored
    uint64_t p_full;
    uint64_t rows_ready[2];     // the constants of a tile, by tile parity
    uint64_t rows_done[2];      // eight softmax warps have read them
    uint32_t tmem_base;
    int abort_flag;
};
static_assert(sizeof(Shared) <= SMEM_BYTES - MISC_OFFSET, "key-side barrier block too large");
}  // namespace ks

__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(ks::KEY_THREADS, 1) absorbed_backward_key_kernel(const __grid_constant__ AbsorbedBackwardParams p) {
    using namespace ks;
    extern __shared__ uint8_t smem_raw[];
    // No early exit on a status left by an earlier launch: both CTAs have to take the same path to the cluster barriers.
    const int warp = threadIdx.x / 32;
    const int lane = threadIdx.x % 32;
    const uint32_t rank = cluster_cta_rank();
    const int b = blockIdx.z;
    // blockIdx.x / 2 counts (key tile, part) pairs, key tile 0 first
    int key_tile = 0, part = static_cast<int>(blockIdx.x >> 1), parts = key_tile_parts(p, 0);
    while (part >= parts) {
        part -= parts;
        ++key_tile;
        parts = key_tile_parts(p, key_tile);
    }
    const int key_start = key_tile * KEYS;
    const int rows_per_sequence = p.sequence * p.heads;
    const int tiles_of_key_tile = key_tile_row_tiles(p, key_tile);
    const int first_tile = static_cast<int>(static_cast<long long>(part) * tiles_of_key_tile / parts);
    const int tile_count = static_cast<int>(static_cast<long long>(part + 1) * tiles_of_key_tile / parts) - first_tile;
    const int first_row = key_start * p.heads + first_tile * TILE_ROWS;        // of the batch entry

    const uint32_t smem_base = smem_u32(smem_raw);
    Shared* sh = reinterpret_cast<Shared*>(smem_raw + MISC_OFFSET);
    volatile int* abort_flag = &sh->abort_flag;
    if ((smem_base & 1023U) != 0U) {            // a property of the kernel image: the same in both CTAs
        grid_dependency_wait();
        if (threadIdx.x == 0) {
            atomicExch(&absorbed_backward_status, STATUS_SMEM_MISALIGNED);
        }
        return;
    }

    if (threadIdx.x == 0) {
        for (uint64_t* bar = &sh->k_full; bar <= &sh->do_free; ++bar) {
            mbar_init(smem_u32(bar), 1);
        }
        mbar_init(smem_u32(&sh->p_full), 16);
        for (int i = 0; i < 2; ++i) {
            mbar_init(smem_u32(&sh->rows_ready[i]), 1);
            mbar_init(smem_u32(&sh->rows_done[i]), 8);
        }
        sh->abort_flag = 0;
        mbar_init_fence();
    }
    if (warp == MMA_WARP) {
        tmem_alloc_pair(smem_u32(&sh->tmem_base), TMEM_COLUMNS);
        tmem_relinquish_pair();
    }
    if (warp == LOAD_WARP && lane == 0) {
        tma_prefetch_descriptor(&p.key_lat8);
        tma_prefetch_descriptor(&p.key_rope1);
        tma_prefetch_descriptor(&p.row_q8);
        tma_prefetch_descriptor(&p.row_q2);
        tma_prefetch_descriptor(&p.row_do8);
        tma_prefetch_descriptor(&p.row_do2);
        tma_prefetch_descriptor(&p.row_rope);
    }
    tc_fence_before_sync();
    __syncthreads();
    cluster_sync_all();
    tc_fence_after_sync();
    grid_dependency_wait();
    const uint32_t tmem_base = *reinterpret_cast<volatile uint32_t*>(&sh->tmem_base);
    auto wait = [&](uint64_t& bar, int phase) { return mbar_wait(smem_u32(&bar), phase & 1, abort_flag, &absorbed_backward_status); };

    if (warp == LOAD_WARP) {
        // =================== TMA producer ===================================
        if (lane == 0) {
            const int own = static_cast<int>(rank) * HALF_ROWS, other = HALF_ROWS - own;
            const int own_chunk = 2 * static_cast<int>(rank), other_slot = 2 - own_chunk;
            uint32_t bar = smem_u32(&sh->k_full);
            mbar_arrive_expect_tx(bar, K_BYTES);
            tma_load_4d(smem_base, &p.key_lat8, bar, 0, key_start + static_cast<int>(rank) * CTA_KEYS, 0, b);
            tma_load_4d(smem_base + LATENT_CHUNKS * KEY_SLOT, &p.key_rope1, bar, 0, key_start + static_cast<int>(rank) * CTA_KEYS, 0, b);
            for (int t = 0; t < tile_count; ++t) {
                const int row0 = first_row + t * TILE_ROWS;
                if (t > 0 && !wait(sh->q_free, t - 1)) {
                    break;
                }
                bar = smem_u32(&sh->q_full);
                mbar_arrive_expect_tx(bar, CHUNKS * ROW_SLOT);
                tma_load_4d(smem_base + ROPE_OFFSET, &p.row_rope, bar, 0, row0 + own, 0, b);
                tma_load_4d(smem_base + Q_OFFSET, &p.row_q8, bar, 0, row0 + own, 0, b);
                if (t > 0 && !wait(sh->do_free, t - 1)) {
                    break;
                }
                bar = smem_u32(&sh->do_full);
                mbar_arrive_expect_tx(bar, LATENT_CHUNKS * ROW_SLOT);
                tma_load_4d(smem_base + DO_OFFSET, &p.row_do8, bar, 0, row0 + own, 0, b);
                if (!wait(sh->q_refill_free, t)) {
                    break;
                }
                bar = smem_u32(&sh->q_refilled);
                mbar_arrive_expect_tx(bar, 6 * ROW_SLOT);
                for (int a = 0; a < 2; ++a) {
                    tma_load_4d(smem_base + Q_OFFSET + (4 * a + other_slot) * ROW_SLOT, &p.row_q2, bar, 0, row0 + other, 4 * a + own_chunk, b);
                    tma_load_4d(smem_base + ROPE_ALL_OFFSET + a * ROW_SLOT, &p.row_rope, bar, 0, row0 + a * HALF_ROWS, 0, b);
                }
                if (!wait(sh->do_refill_free, t)) {
                    break;
                }
                bar = smem_u32(&sh->do_refilled);
                mbar_arrive_expect_tx(bar, 4 * ROW_SLOT);
                for (int a = 0; a < 2; ++a) {
                    tma_load_4d(smem_base + DO_OFFSET + (4 * a + other_slot) * ROW_SLOT, &p.row_do2, bar, 0, row0 + other, 4 * a + own_chunk, b);
                }
            }
        }
    } else if (warp == CONSTANTS_WARP) {
        for (int t = 0; t < tile_count; ++t) {
            if (t >= 2 && !__all_sync(0xffffffffU, wait(sh->rows_done[t & 1], (t >> 1) - 1))) {
                break;
            }
            Rows& rows = sh->rows[t & 1];
#pragma unroll
            for (int e = 0; e < TILE_ROWS / 32; ++e) {
                const int n = e * 32 + lane;
                const int row = first_row + t * TILE_ROWS + n;
                float lse_value = 0.0F, delta_value = 0.0F;
                int token = -1;
                if (row < rows_per_sequence) {
                    token = row / p.heads;
                    const int head = row - token * p.heads;
                    lse_value = p.lse[(static_cast<size_t>(b) * p.heads + head) * p.sequence + token] * LOG2E;
                    delta_value = stored_delta(p, static_cast<size_t>(b) * rows_per_sequence + row);
                }
                rows.lse2[n] = lse_value;
                rows.delta[n] = delta_value;
                rows.token[n] = token;
            }
            __syncwarp();
            if (lane == 0) {
                mbar_arrive(smem_u32(&sh->rows_ready[t & 1]));
            }
        }
    } else if (warp == MMA_WARP && rank != 0) {
        // =================== relay: this CTA's "loaded" events -> the leader =========
        if (lane == 0) {
            bool alive = wait(sh->k_full, 0);
            if (alive) {
                mbar_arrive_remote(map_to_cta(smem_u32(&sh->peer_k_full), 0));
            }
            for (int t = 0; t < tile_count && alive; ++t) {
                // in the order in which they are loaded
                uint64_t* const mine[4] = {&sh->q_full, &sh->do_full, &sh->q_refilled, &sh->do_refilled};
                uint64_t* const leaders[4] = {&sh->peer_q_full, &sh->peer_do_full, &sh->peer_q_refilled, &sh->peer_do_refilled};
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    alive = alive && wait(*mine[i], t);
                    if (alive) {
                        mbar_arrive_remote(map_to_cta(smem_u32(leaders[i]), 0));
                    }
                }
            }
        }
    } else if (warp == MMA_WARP) {
        // =================== MMA issuer (leader CTA; whole warp, elected lane executes) ==
        const uint32_t leader = elect_one();
        constexpr uint32_t IDESC_SCORE = make_idesc_bf16(KEYS, TILE_ROWS, false, false);
        constexpr uint32_t IDESC_GRAD = make_idesc_bf16(KEYS, 256, false, true);
        constexpr uint32_t IDESC_ROPE = make_idesc_bf16(KEYS, 128, false, true);
        constexpr uint32_t HI = smem_desc_hi(1024);
        const uint32_t k_lo = smem_desc_lo(smem_base, 16);
        const uint32_t rope_lo = smem_desc_lo(smem_base + ROPE_OFFSET, 16);
        const uint32_t p_lo = smem_desc_lo(smem_base + P_OFFSET, 16);
        const uint32_t ds_lo = smem_desc_lo(smem_base + DS_OFFSET, 16);
        const uint32_t rope_all_lo = smem_desc_lo(smem_base + ROPE_ALL_OFFSET, ROW_SLOT);
        auto both = [&](uint64_t* bar) {        // one commit for this CTA's barrier, one for the other CTA's
            commit_pair(smem_u32(bar), leader);
            commit_pair(map_to_cta(smem_u32(bar), 1), leader);
        };
        // K (chunks of all columns) times the own rows in slots at `operand`; slots {2,3,6,7} (refilled in the leader) first,
        // then {0,1,4,5} (refilled in the other CTA)
        auto issue_scores = [&](uint32_t acc, uint32_t operand, bool fresh, uint64_t* refill_free) {
            const uint32_t row_lo = smem_desc_lo(operand, 16);
#pragma unroll
            for (int group = 0; group < 2; ++group) {
#pragma unroll
                for (int n = 0; n < 4; ++n) {
                    const int c = (group == 0 ? 2 : 0) + (n & 1) + (n >> 1) * 4;
#pragma unroll
                    for (int k = 0; k < 4; ++k) {
                        mma_pair_ss_split(acc, k_lo + c * (KEY_SLOT >> 4) + 2 * k, HI, row_lo + c * (ROW_SLOT >> 4) + 2 * k, HI, IDESC_SCORE,
                                          (fresh && group == 0 && n == 0 && k == 0) ? 0U : 1U, leader);
                    }
                }
                commit_pair(group == 0 ? smem_u32(refill_free) : map_to_cta(smem_u32(refill_free), 1), leader);
            }
        };
        // dlatent += A (P^T or dS^T at a_lo) times the columns in slots at `operand`: rows 48g.. of half a in slots 4a + 2g, + 1
        auto issue_gradients = [&](uint32_t a_lo, uint32_t operand, bool fresh) {
            const uint32_t column_lo = smem_desc_lo(operand, ROW_SLOT);
#pragma unroll
            for (int a = 0; a < 2; ++a) {
#pragma unroll
                for (int kk = 0; kk < 6; ++kk) {
                    mma_pair_ss_split(tmem_base + TMEM_DLAT + a * 128, a_lo + (kk >> 2) * (KEY_SLOT >> 4) + 2 * (kk & 3), HI,
                                      column_lo + (4 * a + 2 * (kk / 3)) * (ROW_SLOT >> 4) + (kk % 3) * (2048 >> 4), HI, IDESC_GRAD,
                                      (fresh && kk == 0) ? 0U : 1U, leader);
                }
            }
        };
        auto wait_both = [&](uint64_t& mine, uint64_t& others, int phase) {
            const bool alive = __all_sync(0xffffffffU, wait(mine, phase) && wait(others, phase));
            tc_fence_after_sync();
            return alive;
        };
        bool alive = wait_both(sh->k_full, sh->peer_k_full, 0);
        for (int t = 0; t < tile_count && alive; ++t) {
            alive = wait_both(sh->q_full, sh->peer_q_full, t);
            if (!alive) {
                break;
            }
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                mma_pair_ss_split(tmem_base + TMEM_S, k_lo + LATENT_CHUNKS * (KEY_SLOT >> 4) + 2 * k, HI, rope_lo + 2 * k, HI, IDESC_SCORE, k != 0 ? 1U : 0U,
                                  leader);
            }
            issue_scores(tmem_base + TMEM_S, smem_base + Q_OFFSET, false, &sh->q_refill_free);
            both(&sh->s_full);
            alive = wait_both(sh->do_full, sh->peer_do_full, t);
            if (!alive) {
                break;
            }
            issue_scores(tmem_base + TMEM_DP, smem_base + DO_OFFSET, true, &sh->do_refill_free);
            both(&sh->dp_full);
            alive = __all_sync(0xffffffffU, wait(sh->p_full, t)) && wait_both(sh->q_refilled, sh->peer_q_refilled, t);
            if (!alive) {
                break;
            }
            issue_gradients(ds_lo, smem_base + Q_OFFSET, t == 0);
#pragma unroll
            for (int kk = 0; kk < 6; ++kk) {
                mma_pair_ss_split(tmem_base + TMEM_DROPE, ds_lo + (kk >> 2) * (KEY_SLOT >> 4) + 2 * (kk & 3), HI,
                                  rope_all_lo + (kk / 3) * (ROW_SLOT >> 4) + (kk % 3) * (2048 >> 4), HI, IDESC_ROPE, (t | kk) != 0 ? 1U : 0U, leader);
            }
            both(&sh->q_free);
            alive = wait_both(sh->do_refilled, sh->peer_do_refilled, t);
            if (!alive) {
                break;
            }
            issue_gradients(p_lo, smem_base + DO_OFFSET, false);
            both(&sh->do_free);
        }
    } else {
        // =================== softmax: thread = (key, 24 of the 96 rows) ======
        const int tmem_lane = (warp % 4) * 32 + lane;
        const int key_in_cta = tmem_lane & 63;
        const int row_half = tmem_lane >> 6;
        const int share = warp / 4;
        const int n0 = row_half * HALF_ROWS + share * SHARE_ROWS;           // first row of this thread
        const uint32_t lane_base = tmem_base + (static_cast<uint32_t>((warp % 4) * 32) << 16);
        const int key_pos = key_start + static_cast<int>(rank) * CTA_KEYS + key_in_cta;
        const uint32_t p_full_bar = map_to_cta(smem_u32(&sh->p_full), 0);
        bool alive = true;
        for (int t = 0; t < tile_count; ++t) {
            alive = __all_sync(0xffffffffU, wait(sh->rows_ready[t & 1], t >> 1) && wait(sh->s_full, t));
            if (!alive) {
                break;
            }
            tc_fence_after_sync();
            const Rows& rows = sh->rows[t & 1];
            const int row0 = first_row + t * TILE_ROWS;
            const bool masked = row0 / p.heads < key_start + KEYS - 1 || row0 + TILE_ROWS > rows_per_sequence;
            uint32_t x[SHARE_ROWS];
            float prob[SHARE_ROWS];
#pragma unroll
            for (int n = 0; n < SHARE_ROWS; n += 8) {
                tmem_ld_x8(lane_base + TMEM_S + share * SHARE_ROWS + n, x + n);
            }
            tmem_wait_ld();
#pragma unroll
            for (int n = 0; n < SHARE_ROWS; n += 4) {
                const float4 l = *reinterpret_cast<const float4*>(rows.lse2 + n0 + n);
                prob[n] = exp2_approx(fmaf(__uint_as_float(x[n]), p.scale_log2, -l.x));
                prob[n + 1] = exp2_approx(fmaf(__uint_as_float(x[n + 1]), p.scale_log2, -l.y));
                prob[n + 2] = exp2_approx(fmaf(__uint_as_float(x[n + 2]), p.scale_log2, -l.z));
                prob[n + 3] = exp2_approx(fmaf(__uint_as_float(x[n + 3]), p.scale_log2, -l.w));
            }
            if (masked) {
#pragma unroll
                for (int n = 0; n < SHARE_ROWS; n += 4) {
                    const int4 token = *reinterpret_cast<const int4*>(rows.token + n0 + n);
                    prob[n] = key_pos <= token.x ? prob[n] : 0.0F;
                    prob[n + 1] = key_pos <= token.y ? prob[n + 1] : 0.0F;
                    prob[n + 2] = key_pos <= token.z ? prob[n + 2] : 0.0F;
                    prob[n + 3] = key_pos <= token.w ? prob[n + 3] : 0.0F;
                }
            }
            // P^T and dS^T of the previous tile have been read; this thread's three 16-byte units, swizzled by the key
            if (t > 0) {
                alive = __all_sync(0xffffffffU, wait(sh->do_free, t - 1));
                if (!alive) {
                    break;
                }
            }
            auto unit_address = [&](int offset, int unit) {
                const int u = n0 / 8 + unit;
                return reinterpret_cast<uint4*>(smem_raw + offset + (u >> 3) * KEY_SLOT + key_in_cta * 128 + (((u & 7) ^ (key_in_cta & 7)) * 16));
            };
#pragma unroll
            for (int unit = 0; unit < SHARE_ROWS / 8; ++unit) {
                const float* v = prob + 8 * unit;
                *unit_address(P_OFFSET, unit) =
                    make_uint4(pack_bf16x2(v[0], v[1]), pack_bf16x2(v[2], v[3]), pack_bf16x2(v[4], v[5]), pack_bf16x2(v[6], v[7]));
            }
            alive = __all_sync(0xffffffffU, wait(sh->dp_full, t));
            if (!alive) {
                break;
            }
            tc_fence_after_sync();
#pragma unroll
            for (int n = 0; n < SHARE_ROWS; n += 8) {
                tmem_ld_x8(lane_base + TMEM_DP + share * SHARE_ROWS + n, x + n);
            }
            tmem_wait_ld();
#pragma unroll
            for (int unit = 0; unit < SHARE_ROWS / 8; ++unit) {
                const float4 d0 = *reinterpret_cast<const float4*>(rows.delta + n0 + 8 * unit);
                const float4 d1 = *reinterpret_cast<const float4*>(rows.delta + n0 + 8 * unit + 4);
                const float* v = prob + 8 * unit;
                const uint32_t* y = x + 8 * unit;
                *unit_address(DS_OFFSET, unit) =
                    make_uint4(pack_bf16x2(v[0] * (__uint_as_float(y[0]) - d0.x) * p.scale, v[1] * (__uint_as_float(y[1]) - d0.y) * p.scale),
                               pack_bf16x2(v[2] * (__uint_as_float(y[2]) - d0.z) * p.scale, v[3] * (__uint_as_float(y[3]) - d0.w) * p.scale),
                               pack_bf16x2(v[4] * (__uint_as_float(y[4]) - d1.x) * p.scale, v[5] * (__uint_as_float(y[5]) - d1.y) * p.scale),
                               pack_bf16x2(v[6] * (__uint_as_float(y[6]) - d1.z) * p.scale, v[7] * (__uint_as_float(y[7]) - d1.w) * p.scale));
            }
            fence_proxy_async_smem();
            tc_fence_before_sync();
            __syncwarp();
            if (lane == 0) {
                mbar_arrive_remote(p_full_bar);
                mbar_arrive(smem_u32(&sh->rows_done[t & 1]));
            }
        }
        alive = __all_sync(0xffffffffU, alive && wait(sh->do_free, tile_count - 1));
        if (alive) {
            tc_fence_after_sync();
            // Every MMA has finished, so the operands' memory is idle: a warp lays out 32 keys x 128 bytes at a time in a 4 KB
            // slab (swizzled) from where a TMA store writes whole lines; keys past the end of the sequence are clipped.
            const uint32_t slabs = static_cast<uint32_t>(warp) * 5 * SLAB_BYTES;
            uint8_t* slab_row = smem_raw + slabs + lane * 128;
            const int store_key = key_start + static_cast<int>(rank) * CTA_KEYS + (warp & 1) * 32;
            const int column = share * 256 + row_half * 128;
            const bool has_rope = row_half == 0;                // lanes 64-127 hold the same sums
#pragma unroll
            for (int c = 0; c < 5; ++c) {
                uint32_t v[32];
                if (c == 4 && !has_rope) {
                    break;
                }
                tmem_ld_x32(lane_base + (c < 4 ? TMEM_DLAT + share * 128 + c * 32 : TMEM_DROPE + share * 32), v);
                tmem_wait_ld();
                if (p.key_direct == 0) {
#pragma unroll
                    for (int u = 0; u < 8; ++u) {
                        *reinterpret_cast<uint4*>(slab_row + c * SLAB_BYTES + ((u ^ (lane & 7)) * 16)) = make_uint4(v[4 * u], v[4 * u + 1], v[4 * u + 2], v[4 * u + 3]);
                    }
                } else if (c < 4) {
#pragma unroll
                    for (int u = 0; u < 4; ++u) {
                        const uint32_t* y = v + 8 * u;
                        *reinterpret_cast<uint4*>(slab_row + (c / 2) * SLAB_BYTES + ((((c & 1) * 4 + u) ^ (lane & 7)) * 16)) =
                            make_uint4(pack_bf16x2(__uint_as_float(y[0]), __uint_as_float(y[1])), pack_bf16x2(__uint_as_float(y[2]), __uint_as_float(y[3])),
                                       pack_bf16x2(__uint_as_float(y[4]), __uint_as_float(y[5])), pack_bf16x2(__uint_as_float(y[6]), __uint_as_float(y[7])));
                    }
                } else if (key_pos < p.sequence) {
                    store_bf16x32(p.dk_rope + (static_cast<size_t>(b) * p.sequence + key_pos) * ROPE + share * 32, v);
                }
            }
            fence_proxy_async_smem();
            __syncwarp();
            if (lane == 0 && store_key < p.sequence) {
                if (p.key_direct == 0) {
                    for (int c = 0; c < (has_rope ? 5 : 4); ++c) {
                        tma_store_4d(&p.partials, smem_base + slabs + c * SLAB_BYTES, c < 4 ? column + c * 32 : RANK + share * 32, 0, store_key, part * p.batch + b);
                    }
                } else {
                    for (int c = 0; c < 2; ++c) {
                        tma_store_3d(&p.dlatent_out, smem_base + slabs + c * SLAB_BYTES, column + c * 64, store_key, b);
                    }
                }
                tma_store_commit();
                tma_store_wait_read();
            }
        }
    }

    // ---- teardown -----------------------------------------------------------
    __syncwarp();
    tc_fence_before_sync();
    __syncthreads();
    if (*abort_flag != 0) {
        for (int k = 0; k < 64; ++k) {
            __nanosleep(1000);
        }
    }
    cluster_sync_all();                 // neither CTA frees tensor memory or exits while the other may still signal it
    if (warp == MMA_WARP) {
        tc_fence_after_sync();
        tmem_dealloc_pair(tmem_base, TMEM_COLUMNS);
    }
}

// ---------------------------------------------------------------------------
// Adds the key side's fp32 partial sums of one key row, in part order (so the result does not
// depend on scheduling), and writes bf16 dlatent / dkey_rope.  One CTA of 144 threads per key
// row, four columns per thread.
// ---------------------------------------------------------------------------
__global__ void __launch_bounds__(144) absorbed_backward_reduce_kernel(const __grid_constant__ AbsorbedBackwardParams p) {
    const int key = blockIdx.x;
    const int b = blockIdx.y;
    const int parts = key_tile_parts(p, key / KEYS);
    const float* scratch = reinterpret_cast<const float*>(p.dq_lat);
    const int column = threadIdx.x * 4;
    grid_dependency_wait();
    float4 sum = make_float4(0.0F, 0.0F, 0.0F, 0.0F);
    for (int part = 0; part < parts; ++part) {
        const float4 v = *reinterpret_cast<const float4*>(scratch + ((static_cast<size_t>(part) * p.batch + b) * p.sequence + key) * (RANK + ROPE) + column);
        sum.x += v.x;
        sum.y += v.y;
        sum.z += v.z;
        sum.w += v.w;
    }
    uint2 packed;
    packed.x = pack_bf16x2(sum.x, sum.y);
    packed.y = pack_bf16x2(sum.z, sum.w);
    const size_t key_row = static_cast<size_t>(b) * p.sequence + key;
    if (column < RANK) {
        *reinterpret_cast<uint2*>(p.dlatent + key_row * RANK + column) = packed;
    } else {
        *reinterpret_cast<uint2*>(p.dk_rope + key_row * ROPE + (column - RANK)) = packed;
    }
}

// ---------------------------------------------------------------------------
// Query side.  Tensor memory: dQ^T as five 64-column blocks at 0..319 (block m holds output
// columns 128m..128m+127 on the lanes and the 64 rows on the columns; block 4 is the rotary part
// on lanes 0..63), S^T 320..383, dP^T 384..447.  Shared memory: the 64 rows' query_latent (8
// chunks), query_rope (1) and dO (8) as 8 KB K-major chunks, a 16 KB dS^T tile (the MN-major B
// operand of dQ^T += K^T dS^T), a ring of two 32 KB units (pairs of 16 KB key chunks), constants.
// Per key tile: 5 units (chunk pairs 0-1 .. 6-7, then the rotary chunk alone) for S^T and dP^T,
// the softmax, and the same 5 units again as the MN-major A operand of the gradient product.
// The rotary unit's second half is whatever the slot held before: its products land on lanes
// 64..127 of block 4, which nothing reads.
// ---------------------------------------------------------------------------
namespace qs {
constexpr int RING_SLOTS = 2;
constexpr int SLOT_BYTES = 2 * KEY_CHUNK;
constexpr int Q_BYTES = CHUNKS * ROW_CHUNK;
constexpr int DO_BYTES = LATENT_CHUNKS * ROW_CHUNK;
constexpr int DS_BYTES = KEYS * 128;
constexpr int SMEM_BYTES = Q_BYTES + DO_BYTES + DS_BYTES + RING_SLOTS * SLOT_BYTES + MISC_BYTES + 1024;
constexpr int UNITS_PER_TILE = 10;
constexpr uint32_t TMEM_DQT = 0;
constexpr uint32_t TMEM_X0 = 320;
constexpr uint32_t TMEM_X1 = 384;
static_assert(SMEM_BYTES <= 232448, "query-side shared memory");

struct Shared {
    uint64_t resident_full;
    uint64_t unit_full[RING_SLOTS];
    uint64_t unit_empty[RING_SLOTS];
    uint64_t rows_ready;
    uint64_t s_ready;
    uint64_t ds_ready;          // 256 softmax threads: dS^T is in shared memory
    uint64_t final_full;
    uint32_t tmem_base;
    int abort_flag;
    RowConstants rows;
};
static_assert(sizeof(Shared) <= MISC_BYTES, "query-side barrier block too large");
}  // namespace qs

__global__ void __launch_bounds__(THREADS, 1) absorbed_backward_query_kernel(const __grid_constant__ AbsorbedBackwardParams p) {
    using namespace qs;
    extern __shared__ uint8_t smem_raw[];
    if (*reinterpret_cast<volatile int*>(&absorbed_backward_status) == STATUS_WAIT_TIMEOUT) {
        grid_dependency_wait();
        return;
    }
    const int warp = threadIdx.x / 32;
    const int lane = threadIdx.x % 32;
    const int b = blockIdx.z;
    const int rows_per_sequence = p.sequence * p.heads;
    const int row0 = static_cast<int>(gridDim.x - 1 - blockIdx.x) * ROWS;       // late rows see the most keys: longest first
    const int last_row = min(row0 + ROWS, rows_per_sequence) - 1;
    const int first_token = row0 / p.heads;
    const int tile_count = (last_row / p.heads) / KEYS + 1;

    const uint32_t smem_base = (smem_u32(smem_raw) + 1023U) & ~1023U;
    uint8_t* smem_aligned = smem_raw + (smem_base - smem_u32(smem_raw));
    const uint32_t q_smem = smem_base;
    const uint32_t do_smem = q_smem + Q_BYTES;
    const uint32_t ds_smem = do_smem + DO_BYTES;
    uint8_t* ds_ptr = smem_aligned + Q_BYTES + DO_BYTES;
    const uint32_t ring = ds_smem + DS_BYTES;
    Shared* sh = reinterpret_cast<Shared*>(smem_aligned + Q_BYTES + DO_BYTES + DS_BYTES + RING_SLOTS * SLOT_BYTES);
    volatile int* abort_flag = &sh->abort_flag;

    if (threadIdx.x == 0) {
        mbar_init(smem_u32(&sh->resident_full), 1);
        for (int i = 0; i < RING_SLOTS; ++i) {
            mbar_init(smem_u32(&sh->unit_full[i]), 1);
            mbar_init(smem_u32(&sh->unit_empty[i]), 1);
        }
        mbar_init(smem_u32(&sh->rows_ready), 1);
        mbar_init(smem_u32(&sh->s_ready), 1);
        mbar_init(smem_u32(&sh->ds_ready), 256);
        mbar_init(smem_u32(&sh->final_full), 1);
        sh->abort_flag = 0;
        mbar_init_fence();
    }
    if (warp == MMA_WARP) {
        tmem_alloc(smem_u32(&sh->tmem_base), TMEM_COLUMNS);
        tmem_relinquish();
    }
    if (warp == LOAD_WARP && lane == 0) {
        tma_prefetch_descriptor(&p.q_lat);
        tma_prefetch_descriptor(&p.q_rope);
        tma_prefetch_descriptor(&p.d_out);
        tma_prefetch_descriptor(&p.k_lat);
        tma_prefetch_descriptor(&p.k_rope);
    }
    tc_fence_before_sync();
    __syncthreads();
    tc_fence_after_sync();
    grid_dependency_wait();
    const uint32_t tmem_base = *reinterpret_cast<volatile uint32_t*>(&sh->tmem_base);

    if (warp == LOAD_WARP) {
        // =================== TMA producer ===================================
        fill_row_constants(p, sh->rows, b, row0, lane);
        __syncwarp();
        if (lane == 0) {
            mbar_arrive(smem_u32(&sh->rows_ready));
            const uint32_t bar = smem_u32(&sh->resident_full);
            mbar_arrive_expect_tx(bar, Q_BYTES + DO_BYTES);
            const int y = b * rows_per_sequence + row0;
            for (int c = 0; c < LATENT_CHUNKS; ++c) {
                tma_load_2d(q_smem + c * ROW_CHUNK, &p.q_lat, bar, c * 64, y);
                tma_load_2d(do_smem + c * ROW_CHUNK, &p.d_out, bar, c * 64, y);
            }
            tma_load_2d(q_smem + LATENT_CHUNKS * ROW_CHUNK, &p.q_rope, bar, 0, y);
            bool alive = true;
            int unit = 0;
            for (int j = 0; j < tile_count && alive; ++j) {
                const int ky = b * p.sequence + j * KEYS;
                for (int u = 0; u < UNITS_PER_TILE && alive; ++u, ++unit) {
                    const int slot = unit % RING_SLOTS;
                    if (unit >= RING_SLOTS) {
                        alive = mbar_wait(smem_u32(&sh->unit_empty[slot]), (unit / RING_SLOTS - 1) & 1, abort_flag, &absorbed_backward_status);
                        if (!alive) {
                            break;
                        }
                    }
                    const uint32_t full = smem_u32(&sh->unit_full[slot]);
                    const uint32_t dst = ring + slot * SLOT_BYTES;
                    const int pair = u % 5;
                    if (pair == 4) {
                        mbar_arrive_expect_tx(full, KEY_CHUNK);
                        tma_load_2d(dst, &p.k_rope, full, 0, ky);
                    } else {
                        mbar_arrive_expect_tx(full, 2 * KEY_CHUNK);
                        tma_load_2d(dst, &p.k_lat, full, pair * 128, ky);
                        tma_load_2d(dst + KEY_CHUNK, &p.k_lat, full, pair * 128 + 64, ky);
                    }
                }
            }
        }
    } else if (warp == MMA_WARP) {
        // =================== MMA issuer (whole warp, elected lane executes) ==
        const uint32_t leader = elect_one();
        constexpr uint32_t IDESC_SCORE = make_idesc_bf16(KEYS, ROWS, false, false);
        constexpr uint32_t IDESC_DQT = make_idesc_bf16(128, ROWS, true, true);        // A = key chunks MN-major, B = dS^T MN-major
        bool alive = __all_sync(0xffffffffU, mbar_wait(smem_u32(&sh->resident_full), 0, abort_flag, &absorbed_backward_status));
        int unit = 0;
        auto wait_unit = [&]() -> uint32_t {
            const int slot = unit % RING_SLOTS;
            alive = __all_sync(0xffffffffU, mbar_wait(smem_u32(&sh->unit_full[slot]), (unit / RING_SLOTS) & 1, abort_flag, &absorbed_backward_status));
            tc_fence_after_sync();
            return ring + slot * SLOT_BYTES;
        };
        auto release_unit = [&]() {
            mma_commit_elect(smem_u32(&sh->unit_empty[unit % RING_SLOTS]), leader);
            ++unit;
        };
        for (int j = 0; j < tile_count && alive; ++j) {
            // ---- S^T = K Q^T, dP^T = latent dO^T ----
            for (int u = 0; u < 5 && alive; ++u) {
                const uint32_t src = wait_unit();
                if (!alive) {
                    break;
                }
                const int chunks_here = u == 4 ? 1 : 2;
                for (int cc = 0; cc < chunks_here; ++cc) {
                    const int chunk = 2 * u + cc;
#pragma unroll
                    for (int k = 0; k < 4; ++k) {
                        mma_ss_elect(tmem_base + TMEM_X0, make_kmajor_desc(src + cc * KEY_CHUNK + k * 32), make_kmajor_desc(q_smem + chunk * ROW_CHUNK + k * 32),
                                     IDESC_SCORE, (chunk | k) != 0 ? 1U : 0U, leader);
                    }
                    if (chunk < LATENT_CHUNKS) {
#pragma unroll
                        for (int k = 0; k < 4; ++k) {
                            mma_ss_elect(tmem_base + TMEM_X1, make_kmajor_desc(src + cc * KEY_CHUNK + k * 32),
                                         make_kmajor_desc(do_smem + chunk * ROW_CHUNK + k * 32), IDESC_SCORE, (chunk | k) != 0 ? 1U : 0U, leader);
                        }
                    }
                }
                release_unit();
            }
            if (!alive) {
                break;
            }
            // this commit also covers the gradient products of the previous tile, the last readers of the dS^T tile
            mma_commit_elect(smem_u32(&sh->s_ready), leader);
            alive = __all_sync(0xffffffffU, mbar_wait(smem_u32(&sh->ds_ready), j & 1, abort_flag, &absorbed_backward_status));
            if (!alive) {
                break;
            }
            tc_fence_after_sync();
            // ---- dQ^T block m += (key chunks 2m, 2m+1)^T dS^T ----
            for (int m = 0; m < 5 && alive; ++m) {
                const uint32_t src = wait_unit();
                if (!alive) {
                    break;
                }
#pragma unroll
                for (int k = 0; k < 8; ++k) {
                    mma_ss_elect(tmem_base + TMEM_DQT + m * ROWS, make_smem_desc(src + k * 2048, KEY_CHUNK, 1024), make_smem_desc(ds_smem + k * 2048, 16, 1024),
                                 IDESC_DQT, (j | k) != 0 ? 1U : 0U, leader);
                }
                release_unit();
            }
        }
        if (alive) {
            mma_commit_elect(smem_u32(&sh->final_full), leader);
        }
    } else {
        // =================== softmax: thread = (key, 32 of the 64 rows) ======
        const int group = warp / 4;
        const int r = threadIdx.x % KEYS;
        const uint32_t lane_base = static_cast<uint32_t>((warp % 4) * 32) << 16;
        const uint32_t st_tmem = tmem_base + lane_base + TMEM_X0 + group * 32;
        const uint32_t dpt_tmem = tmem_base + lane_base + TMEM_X1 + group * 32;
        const bool ragged = row0 + ROWS > rows_per_sequence;
        bool alive = __all_sync(0xffffffffU, mbar_wait(smem_u32(&sh->rows_ready), 0, abort_flag, &absorbed_backward_status));
        for (int j = 0; j < tile_count && alive; ++j) {
            alive = __all_sync(0xffffffffU, mbar_wait(smem_u32(&sh->s_ready), j & 1, abort_flag, &absorbed_backward_status));
            if (!alive) {
                break;
            }
            tc_fence_after_sync();
            const int key_pos = j * KEYS + r;
            const bool masked = ragged || j * KEYS + KEYS - 1 > first_token;
            uint32_t p_packed[16], ds_packed[16];
            score_tile_share(p, st_tmem, dpt_tmem, sh->rows, group, key_pos, masked, p_packed, ds_packed);
            // row r of the MN-major tile: 64 rows = eight 16-byte units, swizzled by the key index
            uint8_t* row = ds_ptr + r * 128;
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const int unit16 = group * 4 + i;
                *reinterpret_cast<uint4*>(row + ((unit16 ^ (r & 7)) * 16)) =
                    make_uint4(ds_packed[4 * i], ds_packed[4 * i + 1], ds_packed[4 * i + 2], ds_packed[4 * i + 3]);
            }
            fence_proxy_async_smem();
            tc_fence_before_sync();
            mbar_arrive(smem_u32(&sh->ds_ready));
        }
        if (alive) {
            alive = __all_sync(0xffffffffU, mbar_wait(smem_u32(&sh->final_full), 0, abort_flag, &absorbed_backward_status));
        }
        if (alive) {
            tc_fence_after_sync();
            // thread = output column (lane r of block m), values = rows 32*group .. 32*group+31
            const size_t first_global_row = static_cast<size_t>(b) * rows_per_sequence + row0 + group * 32;
            const int rows_here = min(32, rows_per_sequence - (row0 + group * 32));
#pragma unroll
            for (int m = 0; m < 5; ++m) {
                uint32_t values[32];
                tmem_ld_x32(tmem_base + lane_base + TMEM_DQT + m * ROWS + group * 32, values);
                tmem_wait_ld();
                if (m < 4) {
                    __nv_bfloat16* dst = p.dq_lat + first_global_row * RANK + m * 128 + r;
#pragma unroll
                    for (int e = 0; e < 32; ++e) {
                        if (e < rows_here) {
                            dst[static_cast<size_t>(e) * RANK] = __float2bfloat16(__uint_as_float(values[e]));
                        }
                    }
                } else if (r < ROPE) {
                    __nv_bfloat16* dst = p.dq_rope + first_global_row * ROPE + r;
#pragma unroll
                    for (int e = 0; e < 32; ++e) {
                        if (e < rows_here) {
                            dst[static_cast<size_t>(e) * ROPE] = __float2bfloat16(__uint_as_float(values[e]));
                        }
                    }
                }
            }
        }
    }

    __syncwarp();
    tc_fence_before_sync();
    __syncthreads();
    if (*abort_flag != 0) {
        for (int k = 0; k < 64; ++k) {
            __nanosleep(1000);
        }
    }
    if (warp == MMA_WARP) {
        tc_fence_after_sync();
        tmem_dealloc(tmem_base, TMEM_COLUMNS);
    }
}

int multiprocessors() {
    static int cached[64] = {};
    int device = 0;
    CUDA_CHECK(cudaGetDevice(&device));
    if (device >= 0 && device < 64 && cached[device] > 0) {
        return cached[device];
    }
    int count = 0;
    CUDA_CHECK(cudaDeviceGetAttribute(&count, cudaDevAttrMultiProcessorCount, device));
    if (device >= 0 && device < 64) {
        cached[device] = count;
    }
    return count > 0 ? count : 148;
}

void configure_kernels() {
    static bool done[16] = {};
    int device = 0;
    CUDA_CHECK(cudaGetDevice(&device));
    if (device < 16 && done[device]) {
        return;
    }
    CUDA_CHECK(cudaFuncSetAttribute(absorbed_backward_key_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, ks::SMEM_BYTES));
    CUDA_CHECK(cudaFuncSetAttribute(absorbed_backward_query_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, qs::SMEM_BYTES));
    if (device < 16) {
        done[device] = true;
    }
}

}  // namespace

namespace internal {

int absorbed_backward_device_status(bool reset) {
    int status = 0;
    CUDA_CHECK(cudaDeviceSynchronize());
    CUDA_CHECK(cudaMemcpyFromSymbol(&status, absorbed_backward_status, sizeof(int)));
    if (reset && status != 0) {
        const int zero = 0;
        CUDA_CHECK(cudaMemcpyToSymbol(absorbed_backward_status, &zero, sizeof(int)));
    }
    return status;
}

}  // namespace internal

void mla_compressed_attention_backward_cuda(__nv_bfloat16* dquery_latent, __nv_bfloat16* dquery_rope, __nv_bfloat16* dkv_latent,
                                            __nv_bfloat16* dkey_rope, const __nv_bfloat16* output_gradient, const __nv_bfloat16* output,
                                            const float* logsumexp, const __nv_bfloat16* query_latent, const __nv_bfloat16* query_rope,
                                            const __nv_bfloat16* kv_latent, const __nv_bfloat16* key_rope, int batch_size, int sequence_length,
                                            int heads, int kv_rank, int rope_size, float scale, cudaStream_t stream) {
    // kernels/attention/mla/sm89.cu:20-24 of the reference: same condition, same message.
    if (kv_rank != MLA_KV_RANK || rope_size != MLA_ROPE_SIZE) {
        throw std::invalid_argument("MLA requires C=512 and RoPE=64");
    }
    if (batch_size <= 0 || sequence_length <= 0 || heads <= 0) {
        throw std::invalid_argument("MLA backward requires positive batch, sequence length and heads");
    }
    if (!(scale > 0.0F)) {
        throw std::invalid_argument("MLA backward requires a positive softmax scale");
    }
    const long long rows_per_sequence = static_cast<long long>(sequence_length) * heads;
    if (rows_per_sequence * batch_size > 0x7fffffffLL || batch_size > 65535) {
        throw std::invalid_argument("MLA backward shape exceeds the supported index range");
    }
    for (const void* pointer : {static_cast<const void*>(dquery_latent), static_cast<const void*>(dquery_rope), static_cast<const void*>(dkv_latent),
                                static_cast<const void*>(dkey_rope), static_cast<const void*>(output_gradient), static_cast<const void*>(output),
                                static_cast<const void*>(logsumexp), static_cast<const void*>(query_latent), static_cast<const void*>(query_rope),
                                static_cast<const void*>(kv_latent), static_cast<const void*>(key_rope)}) {
        if (pointer == nullptr) {
            throw std::invalid_argument("null tensor pointer");
        }
        if ((reinterpret_cast<std::uintptr_t>(pointer) & 15U) != 0) {
            throw std::invalid_argument("tensor pointers must be 16-byte aligned");
        }
    }
    AbsorbedBackwardParams params{};
    const std::uint64_t q_rows = static_cast<std::uint64_t>(rows_per_sequence) * batch_size;
    const std::uint64_t k_rows = static_cast<std::uint64_t>(sequence_length) * batch_size;
    params.q_lat = make_bf16_tile_map(query_latent, q_rows, RANK, RANK, ROWS);
    params.q_rope = make_bf16_tile_map(query_rope, q_rows, ROPE, ROPE, ROWS);
    params.d_out = make_bf16_tile_map(output_gradient, q_rows, RANK, RANK, ROWS);
    params.k_lat = make_bf16_tile_map(kv_latent, k_rows, RANK, RANK, KEYS);
    params.k_rope = make_bf16_tile_map(key_rope, k_rows, ROPE, ROPE, KEYS);
    params.dq_lat = dquery_latent;
    params.dq_rope = dquery_rope;
    params.dlatent = dkv_latent;
    params.dk_rope = dkey_rope;
    params.lse = logsumexp;
    params.batch = batch_size;
    params.sequence = sequence_length;
    params.heads = heads;
    params.scale = scale;
    params.scale_log2 = scale * LOG2E;
    configure_kernels();

    const std::size_t rows = static_cast<std::size_t>(q_rows);
    const unsigned delta_blocks = static_cast<unsigned>(rows / 8 + 1 < 148 * 16 ? rows / 8 + 1 : 148 * 16);
    launch_chained(absorbed_delta_kernel, dim3(delta_blocks), dim3(256), 0, stream, dquery_rope, output_gradient, output, rows);
    // Key side split (see key_tile_parts): about four waves of clusters of equal length, parts of fewer than four tiles only
    // while all of them run at once, never more parts per key tile than fp32 partial rows fit into the dquery_latent buffer.
    const int key_tiles = (sequence_length + KEYS - 1) / KEYS;
    auto tiles_of = [&](int key_tile) { return (rows_per_sequence - static_cast<long long>(key_tile) * KEYS * heads + KEY_SIDE_ROWS - 1) / KEY_SIDE_ROWS; };
    long long tile_units = 0;
    for (int kt = 0; kt < key_tiles; ++kt) {
        tile_units += tiles_of(kt);
    }
    tile_units *= batch_size;
    const long long clusters = std::max(1, multiprocessors() / 2);
    const long long max_parts = std::max<long long>(1, std::min<long long>(64, static_cast<long long>(heads) * RANK * 2 / ((RANK + ROPE) * 4)));
    long long chunk = std::max(std::min<long long>(4, (tile_units + clusters - 1) / clusters), (tile_units + 4 * clusters - 1) / (4 * clusters));
    chunk = std::max(chunk, (tiles_of(0) + max_parts - 1) / max_parts);
    long long part_count = 0;
    for (int kt = 0; kt < key_tiles; ++kt) {
        part_count += (tiles_of(kt) + chunk - 1) / chunk;
    }
    params.key_chunk = static_cast<int>(std::min<long long>(chunk, 0x7fffffffLL));
    params.key_direct = part_count == key_tiles ? 1 : 0;
    params.key_lat8 = make_bf16_batched_chunked_map(kv_latent, batch_size, sequence_length, LATENT_CHUNKS, ks::CTA_KEYS, LATENT_CHUNKS);
    params.key_rope1 = make_bf16_batched_chunked_map(key_rope, batch_size, sequence_length, 1, ks::CTA_KEYS, 1);
    params.row_q8 = make_bf16_batched_chunked_map(query_latent, batch_size, rows_per_sequence, LATENT_CHUNKS, ks::HALF_ROWS, LATENT_CHUNKS);
    params.row_q2 = make_bf16_batched_chunked_map(query_latent, batch_size, rows_per_sequence, LATENT_CHUNKS, ks::HALF_ROWS, 2);
    params.row_do8 = make_bf16_batched_chunked_map(output_gradient, batch_size, rows_per_sequence, LATENT_CHUNKS, ks::HALF_ROWS, LATENT_CHUNKS);
    params.row_do2 = make_bf16_batched_chunked_map(output_gradient, batch_size, rows_per_sequence, LATENT_CHUNKS, ks::HALF_ROWS, 2);
    params.row_rope = make_bf16_batched_chunked_map(query_rope, batch_size, rows_per_sequence, 1, ks::HALF_ROWS, 1);
    params.dlatent_out = make_bf16_batched_rows_map(dkv_latent, batch_size, sequence_length, RANK, 32);
    params.partials = make_f32_records_map(dquery_latent, params.key_direct != 0 ? 1 : static_cast<std::uint64_t>(max_parts) * batch_size,
                                           params.key_direct != 0 ? 1 : sequence_length, 1, RANK + ROPE, 32);
    const dim3 key_grid(static_cast<unsigned>(2 * part_count), 1, batch_size);
    launch_chained(absorbed_backward_key_kernel, key_grid, dim3(ks::KEY_THREADS), ks::SMEM_BYTES, stream, params);
    if (params.key_direct == 0) {
        launch_chained(absorbed_backward_reduce_kernel, dim3(sequence_length, batch_size), dim3(144), 0, stream, params);
    }
    const dim3 query_grid(static_cast<unsigned>((rows_per_sequence + ROWS - 1) / ROWS), 1, batch_size);
    launch_chained(absorbed_backward_query_kernel, query_grid, dim3(THREADS), qs::SMEM_BYTES, stream, params);
}

}  // namespace dscuda
