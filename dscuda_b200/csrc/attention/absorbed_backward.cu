// Backward of the absorbed-latent causal MLA forward
// (mla_compressed_attention_backward_cuda) on the sm_100a tensor cores.
//
// The interface gives no scratch memory, the gradients of the shared latent /
// rotary key sum over every head and every later query, and the operands are wide
// (576 score columns, 512 value columns), so the work is split the way the
// reference splits it (kernels/attention/mla/sm89.cu:295 query side, :356 key
// side): one kernel owns the key-side gradients, one owns the query-side
// gradients, and each recomputes P from the saved LSE.  Both are tcgen05 kernels on
// clusters of two CTAs, with the operands' roles exchanged.
//
// One call launches, on the caller's stream:
//   1. absorbed_delta_kernel: delta[row] = sum_c dO[row,c] O[row,c], kept in the
//      first four bytes of each dquery_rope row (an output the last kernel
//      overwrites, so no scratch is needed);
//   2. absorbed_backward_key_kernel: cluster of two CTAs = (128-key tile, one part of the rows).  The keys stay in shared
//      memory; the 96-row tiles at or after the diagonal stream by and stay there from the score products to the gradient
//      products dlatent += dS^T query_latent + P^T dO and dkey_rope += dS^T query_rope.  Single writer per output element,
//      no atomics; with several parts absorbed_backward_reduce_kernel adds them in order;
//   3. absorbed_backward_query_kernel: cluster = 128 (token, head) rows; query and dO stay in shared memory, every 96-key
//      tile up to the diagonal streams by and stays there from S / dP to dquery += dS K.
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
constexpr int KEYS = 128;                     // key side: keys per cluster
constexpr int THREADS = 320;
constexpr int MMA_WARP = 8;
constexpr int LOAD_WARP = 9;
constexpr int TMEM_COLUMNS = 512;
constexpr float LOG2E = 1.4426950408889634F;

__device__ int absorbed_backward_status = 0;

struct AbsorbedBackwardParams {
    // key side; batch entries are a dimension of their own, so rows and keys past the end of one read as zero
    CUtensorMap key_lat8;   // kv_latent, box 64 keys x 8 chunks
    CUtensorMap key_rope1;  // key_rope, box 64 keys
    CUtensorMap row_q4;     // query_latent, box 48 rows x 4 chunks
    CUtensorMap row_q2;     // ... x 2 chunks
    CUtensorMap row_do4;    // dO likewise
    CUtensorMap row_do2;
    CUtensorMap row_rope;   // query_rope, box 48 rows
    CUtensorMap dlatent_out;    // stores of 32 keys: 64 bf16 columns of dlatent, 32 fp32 columns of a partial sum
    CUtensorMap partials;
    // query side, likewise
    CUtensorMap own_q8;     // query_latent, box 64 rows x 8 chunks
    CUtensorMap own_rope;   // query_rope, box 64 rows
    CUtensorMap own_do8;    // dO, box 64 rows x 8 chunks
    CUtensorMap stream_k4;  // kv_latent, box 48 keys x 4 chunks
    CUtensorMap stream_k2;  // ... x 2 chunks
    CUtensorMap stream_rope;    // key_rope, box 48 keys
    CUtensorMap dq_out;     // stores of 32 rows x 64 columns
    CUtensorMap dq_rope_out;
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

__device__ __forceinline__ float stored_delta(const AbsorbedBackwardParams& p, size_t global_row) {
    return *reinterpret_cast<const float*>(p.dq_rope + global_row * ROPE);
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
            const uint4 a = reinterpret_cast<const uint4*>(dout + row * RANK)[part * 32 + lane];
            const uint4 b = reinterpret_cast<const uint4*>(out + row * RANK)[part * 32 + lane];
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
// loaded once more into a place of their own.  So the scores are computed once per (key, row) pair and a CTA reads 162 KB
// from L2 for 64 x 96 pairs.
//
// What bounds it: shared memory.  The resident keys (72 KB), P and dS (32 KB) and one tile of rows (114 KB) fill it, so the
// chain scores -> softmax -> gradients of a tile is overlapped only by the loads of the next one: a column half of an operand
// is loaded again as soon as its gradient product has read it.  96 rows and not 128 because 128 do not fit.  One CTA per (128 keys, half of dlatent), which this
// replaces, computed the scores twice, at the N = 64 rate: 1305 us at B=4 T=2048 H=16 against
// 532 us now, 46 against 11 us at B=2 T=33 H=32 (where a part also had at least 1024 rows).
//
// Tensor memory: dlatent 2 x 128 columns (lanes 0-63: columns 256a + 0..127, lanes 64-127: 256a + 128..255 of the same 64
// keys), dkey_rope 64, S^T 48 (lanes 64-127: rows 48..95), dP^T 48.
// Warps 0-7: softmax (thread = key x 24 rows) and results; 8: MMA issue in the leader; 9: TMA loads (the other CTA's signal the
// leader's barriers); 10: the rows' constants.
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
    // leader only: completed by the TMA transactions of both CTAs, one phase per tile
    uint64_t k_full;
    uint64_t q_full[2];         // own rows of query_latent, by column half; the rotary chunk with half 0
    uint64_t do_full[2];        // own rows of dO
    uint64_t q_refilled[2];     // the other CTA's rows; the rotary columns of all rows with half 0
    uint64_t do_refilled[2];
    // completed by tcgen05.commit of the leader
    uint64_t q_refill_free[2];  // S has read the half; half 1: S is complete
    uint64_t do_refill_free[2]; // dP^T likewise
    uint64_t q_free[2];         // dS^T Q has read the half
    uint64_t do_free[2];        // P^T dO has read the half; half 1: P, dS and the accumulators are quiescent
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
        for (uint64_t* bar = &sh->k_full; bar < &sh->p_full; ++bar) {
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
        tma_prefetch_descriptor(&p.row_q4);
        tma_prefetch_descriptor(&p.row_q2);
        tma_prefetch_descriptor(&p.row_do4);
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
            // the bytes of both CTAs are counted by the leader's barrier
            auto expect = [&](uint64_t* leaders, uint32_t bytes) {
                if (rank == 0) {
                    mbar_arrive_expect_tx(smem_u32(leaders), 2 * bytes);
                }
                return map_to_cta(smem_u32(leaders), 0);
            };
            const int own = static_cast<int>(rank) * HALF_ROWS, other = HALF_ROWS - own;
            const int own_chunk = 2 * static_cast<int>(rank), other_slot = 2 - own_chunk;
            uint32_t bar = expect(&sh->k_full, K_BYTES);
            tma_load_4d_pair(smem_base, &p.key_lat8, bar, 0, key_start + static_cast<int>(rank) * CTA_KEYS, 0, b);
            tma_load_4d_pair(smem_base + LATENT_CHUNKS * KEY_SLOT, &p.key_rope1, bar, 0, key_start + static_cast<int>(rank) * CTA_KEYS, 0, b);
            bool alive = true;
            for (int t = 0; t < tile_count && alive; ++t) {
                const int row0 = first_row + t * TILE_ROWS;
                // i: query_latent halves 0 and 1, dO halves 0 and 1
                for (int i = 0; i < 4 && alive; ++i) {
                    const int a = i & 1;
                    alive = t == 0 || wait(i < 2 ? sh->q_free[a] : sh->do_free[a], t - 1);
                    if (alive) {
                        bar = expect(i < 2 ? &sh->q_full[a] : &sh->do_full[a], (i == 0 ? 5 : 4) * ROW_SLOT);
                        if (i == 0) {
                            tma_load_4d_pair(smem_base + ROPE_OFFSET, &p.row_rope, bar, 0, row0 + own, 0, b);
                        }
                        tma_load_4d_pair(smem_base + (i < 2 ? Q_OFFSET : DO_OFFSET) + 4 * a * ROW_SLOT, i < 2 ? &p.row_q4 : &p.row_do4, bar, 0, row0 + own, 4 * a, b);
                    }
                }
                for (int i = 0; i < 4 && alive; ++i) {
                    const int a = i & 1;
                    alive = wait(i < 2 ? sh->q_refill_free[a] : sh->do_refill_free[a], t);
                    if (alive) {
                        bar = expect(i < 2 ? &sh->q_refilled[a] : &sh->do_refilled[a], (i == 0 ? 4 : 2) * ROW_SLOT);
                        tma_load_4d_pair(smem_base + (i < 2 ? Q_OFFSET : DO_OFFSET) + (4 * a + other_slot) * ROW_SLOT, i < 2 ? &p.row_q2 : &p.row_do2, bar, 0, row0 + other,
                                    4 * a + own_chunk, b);
                        if (i == 0) {
                            tma_load_4d_pair(smem_base + ROPE_ALL_OFFSET, &p.row_rope, bar, 0, row0, 0, b);
                            tma_load_4d_pair(smem_base + ROPE_ALL_OFFSET + ROW_SLOT, &p.row_rope, bar, 0, row0 + HALF_ROWS, 0, b);
                        }
                    }
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
    } else if (warp == MMA_WARP && rank == 0) {
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
        // K times the own rows in the four slots of column half `half` of the operand at `operand`
        auto issue_scores = [&](uint32_t acc, uint32_t operand, int half, bool fresh) {
            const uint32_t row_lo = smem_desc_lo(operand, 16);
#pragma unroll
            for (int n = 0; n < 4; ++n) {
#pragma unroll
                for (int k = 0; k < 4; ++k) {
                    mma_pair_ss_split(acc, k_lo + (4 * half + n) * (KEY_SLOT >> 4) + 2 * k, HI, row_lo + (4 * half + n) * (ROW_SLOT >> 4) + 2 * k, HI, IDESC_SCORE,
                                      (fresh && n == 0 && k == 0) ? 0U : 1U, leader);
                }
            }
        };
        // columns of half a of dlatent += A (P^T or dS^T at a_lo) times the operand: its rows 48g.. are in slots 4a + 2g, + 1
        auto issue_gradients = [&](uint32_t a_lo, uint32_t operand, int a, bool fresh) {
            const uint32_t column_lo = smem_desc_lo(operand, ROW_SLOT);
#pragma unroll
            for (int kk = 0; kk < 6; ++kk) {
                mma_pair_ss_split(tmem_base + TMEM_DLAT + a * 128, a_lo + (kk >> 2) * (KEY_SLOT >> 4) + 2 * (kk & 3), HI,
                                  column_lo + (4 * a + 2 * (kk / 3)) * (ROW_SLOT >> 4) + (kk % 3) * (2048 >> 4), HI, IDESC_GRAD, (fresh && kk == 0) ? 0U : 1U,
                                  leader);
            }
        };
        auto wait_loaded = [&](uint64_t& bar, int phase) {
            const bool alive = __all_sync(0xffffffffU, wait(bar, phase));
            tc_fence_after_sync();
            return alive;
        };
        bool alive = wait_loaded(sh->k_full, 0);
        for (int t = 0; t < tile_count && alive; ++t) {
            for (int a = 0; a < 2 && alive; ++a) {
                alive = wait_loaded(sh->q_full[a], t);
                if (!alive) {
                    break;
                }
                if (a == 0) {
#pragma unroll
                    for (int k = 0; k < 4; ++k) {
                        mma_pair_ss_split(tmem_base + TMEM_S, k_lo + LATENT_CHUNKS * (KEY_SLOT >> 4) + 2 * k, HI, rope_lo + 2 * k, HI, IDESC_SCORE,
                                          k != 0 ? 1U : 0U, leader);
                    }
                }
                issue_scores(tmem_base + TMEM_S, smem_base + Q_OFFSET, a, false);
                both(&sh->q_refill_free[a]);
            }
            for (int a = 0; a < 2 && alive; ++a) {
                alive = wait_loaded(sh->do_full[a], t);
                if (!alive) {
                    break;
                }
                issue_scores(tmem_base + TMEM_DP, smem_base + DO_OFFSET, a, a == 0);
                both(&sh->do_refill_free[a]);
            }
            alive = alive && __all_sync(0xffffffffU, wait(sh->p_full, t));
            for (int a = 0; a < 2 && alive; ++a) {
                alive = wait_loaded(sh->q_refilled[a], t);
                if (!alive) {
                    break;
                }
                issue_gradients(ds_lo, smem_base + Q_OFFSET, a, t == 0);
                both(&sh->q_free[a]);           // before dkey_rope: the next tile's scores wait for this load
            }
            if (!alive) {
                break;
            }
#pragma unroll
            for (int kk = 0; kk < 6; ++kk) {
                mma_pair_ss_split(tmem_base + TMEM_DROPE, ds_lo + (kk >> 2) * (KEY_SLOT >> 4) + 2 * (kk & 3), HI,
                                  rope_all_lo + (kk / 3) * (ROW_SLOT >> 4) + (kk % 3) * (2048 >> 4), HI, IDESC_ROPE, (t | kk) != 0 ? 1U : 0U, leader);
            }
            for (int a = 0; a < 2 && alive; ++a) {
                alive = wait_loaded(sh->do_refilled[a], t);
                if (!alive) {
                    break;
                }
                issue_gradients(p_lo, smem_base + DO_OFFSET, a, false);
                both(&sh->do_free[a]);
            }
        }
    } else if (warp < MMA_WARP) {
        // =================== softmax: thread = (key, 24 of the 96 rows) ======
        const int tmem_lane = (warp % 4) * 32 + lane;
        const int key_in_cta = tmem_lane & 63;
        const int row_half = tmem_lane >> 6;
        const int share = warp / 4;
        const int n0 = row_half * HALF_ROWS + share * SHARE_ROWS;           // first row of this thread
        const uint32_t lane_base = tmem_base + (static_cast<uint32_t>((warp % 4) * 32) << 16);
        const int key_pos = key_start + static_cast<int>(rank) * CTA_KEYS + key_in_cta;
        const uint32_t p_full_bar = map_to_cta(smem_u32(&sh->p_full), 0);
        bool alive = !gave_up_before(&absorbed_backward_status, abort_flag);
        for (int t = 0; t < tile_count && alive; ++t) {
            alive = __all_sync(0xffffffffU, wait(sh->rows_ready[t & 1], t >> 1) && wait(sh->q_refill_free[1], t));
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
                alive = __all_sync(0xffffffffU, wait(sh->do_free[1], t - 1));
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
            alive = __all_sync(0xffffffffU, wait(sh->do_refill_free[1], t));
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
        alive = __all_sync(0xffffffffU, alive && wait(sh->do_free[1], tile_count - 1));
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
// Query side: the key side with the operands exchanged.  A cluster of two CTAs takes 128 (token, head) rows; CTA r owns rows
// 64r..64r+63, which stay in shared memory as A operands (query 72 KB, dO 64 KB), and every 96-key tile up to the diagonal
// streams by, CTA r supplying 48 of its keys:
//
//   S = Q K^T, dP = dO latent^T     (N = 96), both from the same eight latent chunks of the own keys;
//   dquery_latent += dS latent      (N = 256 twice), dquery_rope += dS K_rope (N = 128, there twice).
//
// The slots of column half a (chunks 4a..4a+3) go round on their own: loaded, read by both score products, two of the four
// refilled with the other CTA's keys, read by the gradient product, loaded again for the next tile; so the loads of one half
// run under the MMAs of the other.
//
// What bounds it: the chain of a tile, as on the key side.  64 rows of one CTA with 128-key tiles, which this replaces, ran
// at the N = 64 rate and streamed every key tile twice (288 KB for 64 x 128 pairs, L2 latency over two 32 KB slots; here
// 90 KB for 64 x 96): 680 us at B=4 T=2048 H=16 against
// 483 us now.
//
// Tensor memory and warps as on the key side; a softmax thread owns 24 keys of one row, so LSE, delta and token are its own.
// ---------------------------------------------------------------------------
namespace qs {
constexpr int TILE_ROWS = 128;                      // rows of a cluster
constexpr int CTA_ROWS = 64;
constexpr int TILE_KEYS = 96;
constexpr int HALF_KEYS = 48;                       // keys a CTA supplies
constexpr int SHARE_KEYS = 24;                      // keys of a softmax thread
constexpr int ROW_SLOT = CTA_ROWS * 128;            // 8 KB: [64 rows x 64 bf16]
constexpr int KEY_SLOT = HALF_KEYS * 128;           // 6 KB: [48 keys x 64 bf16]
constexpr int Q_BYTES = CHUNKS * ROW_SLOT;
constexpr int DO_OFFSET = Q_BYTES;
constexpr int DO_BYTES = LATENT_CHUNKS * ROW_SLOT;
constexpr int DS_OFFSET = DO_OFFSET + DO_BYTES;     // dS: [64 rows x 96 keys] as two 64-key chunks
constexpr int K_OFFSET = DS_OFFSET + 2 * ROW_SLOT;
constexpr int ROPE_OFFSET = K_OFFSET + LATENT_CHUNKS * KEY_SLOT;        // own keys, for the scores
constexpr int ROPE_ALL_OFFSET = ROPE_OFFSET + KEY_SLOT;                 // all 96 keys, for dquery_rope
constexpr int MISC_OFFSET = ROPE_ALL_OFFSET + 2 * KEY_SLOT;
constexpr int SMEM_BYTES = MISC_OFFSET + 1024;
constexpr int SLAB_BYTES = 32 * 128;
constexpr uint32_t TMEM_DQ = 0;
constexpr uint32_t TMEM_DROPE = 256;
constexpr uint32_t TMEM_S = 320;
constexpr uint32_t TMEM_DP = 368;
static_assert(SMEM_BYTES <= 232448, "query-side shared memory");
static_assert(8 * 3 * SLAB_BYTES <= MISC_OFFSET, "result slabs lie in the operands' memory");

struct Shared {
    // leader only: completed by the TMA transactions of both CTAs; the arrays by column half
    uint64_t rows_full;
    uint64_t k_full[2];             // own keys (the rotary chunk with half 0)
    uint64_t refilled[2];           // the other CTA's keys (the rotary columns of all keys with half 0)
    // completed by tcgen05.commit of the leader
    uint64_t refill_free[2];        // both score products have read the half; half 1: dP is complete
    uint64_t s_full;
    uint64_t k_free[2];             // the gradient products have read the half; half 1: dS and the accumulators are quiescent
    // leader only: one arrival per softmax warp of either CTA, dS is stored
    uint64_t ds_full;
    uint32_t tmem_base;
    int abort_flag;
};
static_assert(sizeof(Shared) <= SMEM_BYTES - MISC_OFFSET, "query-side barrier block too large");
}  // namespace qs

__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(THREADS, 1) absorbed_backward_query_kernel(const __grid_constant__ AbsorbedBackwardParams p) {
    using namespace qs;
    extern __shared__ uint8_t smem_raw[];
    const int warp = threadIdx.x / 32;
    const int lane = threadIdx.x % 32;
    const uint32_t rank = cluster_cta_rank();
    const int b = blockIdx.z;
    const int rows_per_sequence = p.sequence * p.heads;
    const int row0 = static_cast<int>((gridDim.x >> 1) - 1 - (blockIdx.x >> 1)) * TILE_ROWS;       // late rows see the most keys: longest first
    const int own_row0 = row0 + static_cast<int>(rank) * CTA_ROWS;
    const int last_token = (min(row0 + TILE_ROWS, rows_per_sequence) - 1) / p.heads;
    const int tile_count = last_token / TILE_KEYS + 1;

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
        for (uint64_t* bar = &sh->rows_full; bar < &sh->ds_full; ++bar) {
            mbar_init(smem_u32(bar), 1);
        }
        mbar_init(smem_u32(&sh->ds_full), 16);
        sh->abort_flag = 0;
        mbar_init_fence();
    }
    if (warp == MMA_WARP) {
        tmem_alloc_pair(smem_u32(&sh->tmem_base), TMEM_COLUMNS);
        tmem_relinquish_pair();
    }
    if (warp == LOAD_WARP && lane == 0) {
        tma_prefetch_descriptor(&p.own_q8);
        tma_prefetch_descriptor(&p.own_rope);
        tma_prefetch_descriptor(&p.own_do8);
        tma_prefetch_descriptor(&p.stream_k4);
        tma_prefetch_descriptor(&p.stream_k2);
        tma_prefetch_descriptor(&p.stream_rope);
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
            // the bytes of both CTAs are counted by the leader's barrier
            auto expect = [&](uint64_t* leaders, uint32_t bytes) {
                if (rank == 0) {
                    mbar_arrive_expect_tx(smem_u32(leaders), 2 * bytes);
                }
                return map_to_cta(smem_u32(leaders), 0);
            };
            const int own = static_cast<int>(rank) * HALF_KEYS, other = HALF_KEYS - own;
            const int own_chunk = 2 * static_cast<int>(rank), other_slot = 2 - own_chunk;
            uint32_t bar = expect(&sh->rows_full, Q_BYTES + DO_BYTES);
            tma_load_4d_pair(smem_base, &p.own_q8, bar, 0, own_row0, 0, b);
            tma_load_4d_pair(smem_base + LATENT_CHUNKS * ROW_SLOT, &p.own_rope, bar, 0, own_row0, 0, b);
            tma_load_4d_pair(smem_base + DO_OFFSET, &p.own_do8, bar, 0, own_row0, 0, b);
            bool alive = true;
            for (int j = 0; j < tile_count && alive; ++j) {
                const int key0 = j * TILE_KEYS;
                for (int a = 0; a < 2 && alive; ++a) {
                    alive = j == 0 || wait(sh->k_free[a], j - 1);
                    if (alive) {
                        bar = expect(&sh->k_full[a], (a == 0 ? 5 : 4) * KEY_SLOT);
                        if (a == 0) {
                            tma_load_4d_pair(smem_base + ROPE_OFFSET, &p.stream_rope, bar, 0, key0 + own, 0, b);
                        }
                        tma_load_4d_pair(smem_base + K_OFFSET + 4 * a * KEY_SLOT, &p.stream_k4, bar, 0, key0 + own, 4 * a, b);
                    }
                }
                for (int a = 0; a < 2 && alive; ++a) {
                    alive = wait(sh->refill_free[a], j);
                    if (alive) {
                        bar = expect(&sh->refilled[a], (a == 0 ? 4 : 2) * KEY_SLOT);
                        tma_load_4d_pair(smem_base + K_OFFSET + (4 * a + other_slot) * KEY_SLOT, &p.stream_k2, bar, 0, key0 + other, 4 * a + own_chunk, b);
                        if (a == 0) {
                            tma_load_4d_pair(smem_base + ROPE_ALL_OFFSET, &p.stream_rope, bar, 0, key0, 0, b);
                            tma_load_4d_pair(smem_base + ROPE_ALL_OFFSET + KEY_SLOT, &p.stream_rope, bar, 0, key0 + HALF_KEYS, 0, b);
                        }
                    }
                }
            }
        }
    } else if (warp == MMA_WARP && rank == 0) {
        // =================== MMA issuer (leader CTA; whole warp, elected lane executes) ==
        const uint32_t leader = elect_one();
        constexpr uint32_t IDESC_SCORE = make_idesc_bf16(TILE_ROWS, TILE_KEYS, false, false);
        constexpr uint32_t IDESC_GRAD = make_idesc_bf16(TILE_ROWS, 256, false, true);
        constexpr uint32_t IDESC_ROPE = make_idesc_bf16(TILE_ROWS, 128, false, true);
        constexpr uint32_t HI = smem_desc_hi(1024);
        const uint32_t q_lo = smem_desc_lo(smem_base, 16);
        const uint32_t do_lo = smem_desc_lo(smem_base + DO_OFFSET, 16);
        const uint32_t ds_lo = smem_desc_lo(smem_base + DS_OFFSET, 16);
        const uint32_t k_lo = smem_desc_lo(smem_base + K_OFFSET, 16);
        const uint32_t rope_lo = smem_desc_lo(smem_base + ROPE_OFFSET, 16);
        const uint32_t column_lo = smem_desc_lo(smem_base + K_OFFSET, KEY_SLOT);
        const uint32_t rope_all_lo = smem_desc_lo(smem_base + ROPE_ALL_OFFSET, KEY_SLOT);
        auto both = [&](uint64_t* bar) {        // one commit for this CTA's barrier, one for the other CTA's
            commit_pair(smem_u32(bar), leader);
            commit_pair(map_to_cta(smem_u32(bar), 1), leader);
        };
        auto issue_scores = [&](uint32_t acc, uint32_t a_lo, int half, bool fresh) {
#pragma unroll
            for (int n = 0; n < 4; ++n) {
#pragma unroll
                for (int k = 0; k < 4; ++k) {
                    mma_pair_ss_split(acc, a_lo + (4 * half + n) * (ROW_SLOT >> 4) + 2 * k, HI, k_lo + (4 * half + n) * (KEY_SLOT >> 4) + 2 * k, HI, IDESC_SCORE,
                                      (fresh && n == 0 && k == 0) ? 0U : 1U, leader);
                }
            }
        };
        auto wait_loaded = [&](uint64_t& bar, int phase) {
            const bool alive = __all_sync(0xffffffffU, wait(bar, phase));
            tc_fence_after_sync();
            return alive;
        };
        bool alive = wait_loaded(sh->rows_full, 0);
        for (int j = 0; j < tile_count && alive; ++j) {
            alive = wait_loaded(sh->k_full[0], j);
            if (!alive) {
                break;
            }
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                mma_pair_ss_split(tmem_base + TMEM_S, q_lo + LATENT_CHUNKS * (ROW_SLOT >> 4) + 2 * k, HI, rope_lo + 2 * k, HI, IDESC_SCORE, k != 0 ? 1U : 0U,
                                  leader);
            }
            issue_scores(tmem_base + TMEM_S, q_lo, 0, false);
            issue_scores(tmem_base + TMEM_DP, do_lo, 0, true);
            both(&sh->refill_free[0]);
            alive = wait_loaded(sh->k_full[1], j);
            if (!alive) {
                break;
            }
            issue_scores(tmem_base + TMEM_S, q_lo, 1, false);
            both(&sh->s_full);
            issue_scores(tmem_base + TMEM_DP, do_lo, 1, false);
            both(&sh->refill_free[1]);
            alive = __all_sync(0xffffffffU, wait(sh->ds_full, j));
            for (int a = 0; a < 2 && alive; ++a) {
                alive = wait_loaded(sh->refilled[a], j);
                if (!alive) {
                    break;
                }
                // keys 48g.. of column half a are in slots 4a + 2g, + 1
#pragma unroll
                for (int kk = 0; kk < 6; ++kk) {
                    mma_pair_ss_split(tmem_base + TMEM_DQ + a * 128, ds_lo + (kk >> 2) * (ROW_SLOT >> 4) + 2 * (kk & 3), HI,
                                      column_lo + (4 * a + 2 * (kk / 3)) * (KEY_SLOT >> 4) + (kk % 3) * (2048 >> 4), HI, IDESC_GRAD, (j | kk) != 0 ? 1U : 0U,
                                      leader);
                }
                both(&sh->k_free[a]);           // before dquery_rope: the next tile's scores wait for this load
                if (a == 0) {
#pragma unroll
                    for (int kk = 0; kk < 6; ++kk) {
                        mma_pair_ss_split(tmem_base + TMEM_DROPE, ds_lo + (kk >> 2) * (ROW_SLOT >> 4) + 2 * (kk & 3), HI,
                                          rope_all_lo + (kk / 3) * (KEY_SLOT >> 4) + (kk % 3) * (2048 >> 4), HI, IDESC_ROPE, (j | kk) != 0 ? 1U : 0U, leader);
                    }
                }
            }
        }
    } else if (warp < MMA_WARP) {
        // =================== softmax: thread = (row, 24 of the 96 keys) ======
        const int tmem_lane = (warp % 4) * 32 + lane;
        const int row_in_cta = tmem_lane & 63;
        const int key_half = tmem_lane >> 6;
        const int share = warp / 4;
        const int n0 = key_half * HALF_KEYS + share * SHARE_KEYS;           // first key of this thread
        const uint32_t lane_base = tmem_base + (static_cast<uint32_t>((warp % 4) * 32) << 16);
        const uint32_t ds_full_bar = map_to_cta(smem_u32(&sh->ds_full), 0);
        const int row = own_row0 + row_in_cta;
        float lse2 = 0.0F, delta = 0.0F;
        int token = -1;                                                     // rows past the end see no key
        if (row < rows_per_sequence) {
            token = row / p.heads;
            lse2 = p.lse[(static_cast<size_t>(b) * p.heads + (row - token * p.heads)) * p.sequence + token] * LOG2E;
            delta = stored_delta(p, static_cast<size_t>(b) * rows_per_sequence + row);
        }
        bool alive = !gave_up_before(&absorbed_backward_status, abort_flag);
        for (int j = 0; j < tile_count && alive; ++j) {
            alive = __all_sync(0xffffffffU, wait(sh->s_full, j));
            if (!alive) {
                break;
            }
            tc_fence_after_sync();
            const int visible = token + 1 - (j * TILE_KEYS + n0);          // keys n < visible count
            uint32_t x[SHARE_KEYS];
            float prob[SHARE_KEYS];
#pragma unroll
            for (int n = 0; n < SHARE_KEYS; n += 8) {
                tmem_ld_x8(lane_base + TMEM_S + share * SHARE_KEYS + n, x + n);
            }
            tmem_wait_ld();
#pragma unroll
            for (int n = 0; n < SHARE_KEYS; ++n) {
                prob[n] = exp2_approx(fmaf(__uint_as_float(x[n]), p.scale_log2, -lse2));
            }
            if (visible < SHARE_KEYS) {
#pragma unroll
                for (int n = 0; n < SHARE_KEYS; ++n) {
                    prob[n] = n < visible ? prob[n] : 0.0F;
                }
            }
            // dP is complete, and dS of the previous tile has been read
            alive = __all_sync(0xffffffffU, wait(sh->refill_free[1], j) && (j == 0 || wait(sh->k_free[1], j - 1)));
            if (!alive) {
                break;
            }
            tc_fence_after_sync();
            __syncwarp();
#pragma unroll
            for (int n = 0; n < SHARE_KEYS; n += 8) {
                tmem_ld_x8(lane_base + TMEM_DP + share * SHARE_KEYS + n, x + n);
            }
            tmem_wait_ld();
#pragma unroll
            for (int unit = 0; unit < SHARE_KEYS / 8; ++unit) {
                const float* v = prob + 8 * unit;
                const uint32_t* y = x + 8 * unit;
                uint32_t packed[4];
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                    packed[e] = pack_bf16x2(v[2 * e] * (__uint_as_float(y[2 * e]) - delta) * p.scale, v[2 * e + 1] * (__uint_as_float(y[2 * e + 1]) - delta) * p.scale);
                }
                const int u = n0 / 8 + unit;        // 16-byte unit of the row, swizzled by the row
                *reinterpret_cast<uint4*>(smem_raw + DS_OFFSET + (u >> 3) * ROW_SLOT + row_in_cta * 128 + (((u & 7) ^ (row_in_cta & 7)) * 16)) =
                    make_uint4(packed[0], packed[1], packed[2], packed[3]);
            }
            fence_proxy_async_smem();
            tc_fence_before_sync();
            __syncwarp();
            if (lane == 0) {
                mbar_arrive_remote(ds_full_bar);
            }
        }
        alive = __all_sync(0xffffffffU, alive && wait(sh->k_free[1], tile_count - 1));
        if (alive) {
            tc_fence_after_sync();
            // Every MMA has finished, so the operands' memory is idle: 32 rows x 128 bytes at a time go through 4 KB slabs
            // (swizzled), from where TMA stores write whole lines; rows past the end of the sequence are clipped.
            const uint32_t slabs = static_cast<uint32_t>(warp) * 3 * SLAB_BYTES;
            uint8_t* slab_row = smem_raw + slabs + lane * 128;
            const int store_row = own_row0 + (warp & 1) * 32;
            const int column = share * 256 + key_half * 128;
            const int parts = warp < 2 ? 6 : 4;                 // warps 0 and 1 also store the rotary columns (lanes 64-127 hold the same sums)
#pragma unroll
            for (int c = 0; c < 6; ++c) {
                if (c >= parts) {
                    break;
                }
                uint32_t v[32];
                tmem_ld_x32(lane_base + (c < 4 ? TMEM_DQ + share * 128 + c * 32 : TMEM_DROPE + (c - 4) * 32), v);
                tmem_wait_ld();
#pragma unroll
                for (int u = 0; u < 4; ++u) {
                    const uint32_t* y = v + 8 * u;
                    *reinterpret_cast<uint4*>(slab_row + (c / 2) * SLAB_BYTES + ((((c & 1) * 4 + u) ^ (lane & 7)) * 16)) =
                        make_uint4(pack_bf16x2(__uint_as_float(y[0]), __uint_as_float(y[1])), pack_bf16x2(__uint_as_float(y[2]), __uint_as_float(y[3])),
                                   pack_bf16x2(__uint_as_float(y[4]), __uint_as_float(y[5])), pack_bf16x2(__uint_as_float(y[6]), __uint_as_float(y[7])));
                }
            }
            fence_proxy_async_smem();
            __syncwarp();
            if (lane == 0 && store_row < rows_per_sequence) {
                for (int c = 0; c < 2; ++c) {
                    tma_store_3d(&p.dq_out, smem_base + slabs + c * SLAB_BYTES, column + c * 64, store_row, b);
                }
                if (parts == 6) {
                    tma_store_3d(&p.dq_rope_out, smem_base + slabs + 2 * SLAB_BYTES, 0, store_row, b);
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
    params.row_q4 = make_bf16_batched_chunked_map(query_latent, batch_size, rows_per_sequence, LATENT_CHUNKS, ks::HALF_ROWS, 4);
    params.row_q2 = make_bf16_batched_chunked_map(query_latent, batch_size, rows_per_sequence, LATENT_CHUNKS, ks::HALF_ROWS, 2);
    params.row_do4 = make_bf16_batched_chunked_map(output_gradient, batch_size, rows_per_sequence, LATENT_CHUNKS, ks::HALF_ROWS, 4);
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
    params.own_q8 = make_bf16_batched_chunked_map(query_latent, batch_size, rows_per_sequence, LATENT_CHUNKS, qs::CTA_ROWS, LATENT_CHUNKS);
    params.own_rope = make_bf16_batched_chunked_map(query_rope, batch_size, rows_per_sequence, 1, qs::CTA_ROWS, 1);
    params.own_do8 = make_bf16_batched_chunked_map(output_gradient, batch_size, rows_per_sequence, LATENT_CHUNKS, qs::CTA_ROWS, LATENT_CHUNKS);
    params.stream_k4 = make_bf16_batched_chunked_map(kv_latent, batch_size, sequence_length, LATENT_CHUNKS, qs::HALF_KEYS, 4);
    params.stream_k2 = make_bf16_batched_chunked_map(kv_latent, batch_size, sequence_length, LATENT_CHUNKS, qs::HALF_KEYS, 2);
    params.stream_rope = make_bf16_batched_chunked_map(key_rope, batch_size, sequence_length, 1, qs::HALF_KEYS, 1);
    params.dq_out = make_bf16_batched_rows_map(dquery_latent, batch_size, rows_per_sequence, RANK, 32);
    params.dq_rope_out = make_bf16_batched_rows_map(dquery_rope, batch_size, rows_per_sequence, ROPE, 32);
    const dim3 query_grid(static_cast<unsigned>(2 * ((rows_per_sequence + qs::TILE_ROWS - 1) / qs::TILE_ROWS)), 1, batch_size);
    launch_chained(absorbed_backward_query_kernel, query_grid, dim3(THREADS), qs::SMEM_BYTES, stream, params);
}

}  // namespace dscuda
