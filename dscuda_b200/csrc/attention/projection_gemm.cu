// The dense projections either side of the attention kernels, on the sm_100a tensor cores:
//
//   * up-projection of the cached latent to per-head keys and values for the training / prefill path:
//       k_nope [rows, H*128] = kv_latent [rows, 512] W_UK^T,   v [rows, H*128] = kv_latent W_UV^T
//     with W_UK, W_UV stored [H*128, 512];
//   * absorption for the decode path: W_UK folded into the query,
//       q_latent [rows, h, 512] = q_nope [rows, h, 128] W_UK[h]          (W_UK[h] is [128, 512])
//     and W_UV applied to the latent output,
//       out [rows, h, 128] = o_latent [rows, h, 512] W_UV[h]^T.
//
// All four are one operation: a batched bf16 GEMM  C_b [M, N] = A_b [M, K] op(B_b)  with fp32 accumulation
// in tensor memory, where a batch entry (a head) is a column offset into A and C and a row offset into
// B, and op(B) is either B^T (B stored [N, K], K-major) or B itself (B stored [K, N], N contiguous: the
// MN-major operand form, no transpose pass).  The reference has none of these (its inputs are drawn
// already projected), so there is no reference kernel to cite.
//
// Two kernels, picked by the number of rows (launch_gemm):
//
//   projection_pair_kernel (many tiles): two CTAs of a cluster work on one 256 x 256 tile with
//   cta_group::2 MMAs.  K is at most 512, so the weights of a column tile (the B operand) stay in shared memory
//   for as long as the cluster walks down the rows, half of them in each CTA, and only A streams: 32 bytes per
//   clock and SM where single-CTA 128 x 128 tiles asked L2 for 128, three times what it gives.
//   projection_gemm_kernel (a decode step, short prompts, and W_UV at any size): persistent CTAs with one 128 x 128
//   tile at a time; less to set up, and at a few rows per head the weights, read once, are what bounds it.
//
// In both the accumulator is double-buffered in tensor memory, so the MMA warp starts the next tile while the epilogue
// warps convert the previous one to bf16 in shared memory, from where TMA stores write whole 128-byte lines; rows past M
// are clipped by the TMA unit.  Warp 4 issues MMAs (whole warp, elected lane), warp 5 loads.  Every mbarrier wait is bounded.
#include "mla.h"
#include "cuda_common.h"
#include "attention_internal.h"
#include "sm100_primitives.cuh"
#include "../common/launch.h"
#include "../common/tensor_map.h"

#include <algorithm>
#include <cstdint>
#include <stdexcept>

namespace dscuda {
namespace {

using namespace sm100;

constexpr int TILE_M = 128;
constexpr int TILE_N = 128;
constexpr int TILE_K = 64;
constexpr int A_BYTES = TILE_M * 128;           // 16 KB: [128 rows x 64 bf16]
constexpr int B_BYTES = TILE_N * 128;           // 16 KB: [128 n x 64 k] (K-major) or two [64 k x 64 n] chunks (MN-major)
constexpr int STAGE_BYTES = A_BYTES + B_BYTES;
constexpr int STAGES = 5;
constexpr int OUT_BYTES = TILE_M * TILE_N * 2;   // 32 KB: two [128 rows x 64 bf16] swizzled chunks
constexpr int MISC_BYTES = 1024;
constexpr int SMEM_BYTES = STAGES * STAGE_BYTES + 2 * OUT_BYTES + MISC_BYTES + 1024;
constexpr int THREADS = 192;
constexpr int MMA_WARP = 4;
constexpr int LOAD_WARP = 5;
constexpr int TMEM_COLUMNS = 256;               // two accumulators of 128 columns

__device__ int projection_status = 0;

struct GemmParams {
    CUtensorMap a;          // [M rows, all A columns], box a_rows x 64
    CUtensorMap b[2];       // K-major: [all B rows, K], box = rows of a CTA's tile x 64; MN-major: [all B rows, N], box 64 x 64
    CUtensorMap c[2];       // [M rows, all C columns], box = rows of one store x 64
    int m, n, k;
    int batch;
    int map_by_batch;       // 1: batch entries are different weights and outputs of the same A (maps b[entry], c[entry])
    int a_rows;             // rows of an A load: 128, or fewer when M is smaller
    int a_batch_cols;       // batch entry b reads A columns [b * a_batch_cols, +K)
    int b_batch_rows;       // ... B rows from b * b_batch_rows
    int c_batch_cols;       // ... writes C columns [b * c_batch_cols, +N)
    int b_mn_major;         // 0: B is [N, K]; 1: B is [K, N]
};

struct Shared {
    uint64_t full[STAGES];
    uint64_t empty[STAGES];
    uint64_t acc_full[2];       // tensor core -> epilogue
    uint64_t acc_empty[2];      // 128 epilogue threads -> tensor core
    uint64_t out_written[2];    // 128 epilogue threads: the tile is in the output buffer
    uint64_t out_free[2];       // the storing thread: the TMA store has read the buffer
    uint32_t tmem_base;
    int abort_flag;
};
static_assert(sizeof(Shared) <= MISC_BYTES, "barrier block too large");

__global__ void __launch_bounds__(THREADS, 1) projection_gemm_kernel(const __grid_constant__ GemmParams p) {
    extern __shared__ uint8_t smem_raw[];
    if (*reinterpret_cast<volatile int*>(&projection_status) == STATUS_WAIT_TIMEOUT) {
        grid_dependency_wait();
        return;
    }
    const int warp = threadIdx.x / 32;
    const int lane = threadIdx.x % 32;
    const uint32_t smem_base = (smem_u32(smem_raw) + 1023U) & ~1023U;
    uint8_t* smem_aligned = smem_raw + (smem_base - smem_u32(smem_raw));
    Shared* sh = reinterpret_cast<Shared*>(smem_aligned + STAGES * STAGE_BYTES + 2 * OUT_BYTES);
    volatile int* abort_flag = &sh->abort_flag;

    if (threadIdx.x == 0) {
        for (int i = 0; i < STAGES; ++i) {
            mbar_init(smem_u32(&sh->full[i]), 1);
            mbar_init(smem_u32(&sh->empty[i]), 1);
        }
        for (int i = 0; i < 2; ++i) {
            mbar_init(smem_u32(&sh->acc_full[i]), 1);
            mbar_init(smem_u32(&sh->acc_empty[i]), TILE_M);
            mbar_init(smem_u32(&sh->out_written[i]), TILE_M);
            mbar_init(smem_u32(&sh->out_free[i]), 1);
        }
        sh->abort_flag = 0;
        mbar_init_fence();
    }
    if (warp == MMA_WARP) {
        tmem_alloc(smem_u32(&sh->tmem_base), TMEM_COLUMNS);
        tmem_relinquish();
    }
    if (warp == LOAD_WARP && lane == 0) {
        tma_prefetch_descriptor(&p.a);
        tma_prefetch_descriptor(&p.b[0]);
        tma_prefetch_descriptor(&p.c[0]);
    }
    tc_fence_before_sync();
    __syncthreads();
    tc_fence_after_sync();
    grid_dependency_wait();
    const uint32_t tmem_base = *reinterpret_cast<volatile uint32_t*>(&sh->tmem_base);

    const int tiles_m = (p.m + TILE_M - 1) / TILE_M;
    const int tiles_n = p.n / TILE_N;
    const long long tiles = static_cast<long long>(tiles_m) * tiles_n * p.batch;
    const int k_chunks = p.k / TILE_K;
    // tile order: M fastest, so that CTAs running at the same time share the B tile (the weights) in L2
    auto locate = [&](long long tile, int& batch, int& tile_n, int& tile_m) {
        tile_m = static_cast<int>(tile % tiles_m);
        const long long rest = tile / tiles_m;
        tile_n = static_cast<int>(rest % tiles_n);
        batch = static_cast<int>(rest / tiles_n);
    };

    if (warp == LOAD_WARP) {
        if (lane == 0) {
            bool alive = true;
            long long chunk = 0;
            for (long long tile = blockIdx.x; tile < tiles && alive; tile += gridDim.x) {
                int batch, tile_n, tile_m;
                locate(tile, batch, tile_n, tile_m);
                const CUtensorMap* b_map = &p.b[p.map_by_batch * batch];
                for (int kc = 0; kc < k_chunks && alive; ++kc, ++chunk) {
                    const int stage = static_cast<int>(chunk % STAGES);
                    if (chunk >= STAGES) {
                        alive = mbar_wait(smem_u32(&sh->empty[stage]), static_cast<uint32_t>((chunk / STAGES - 1) & 1), abort_flag, &projection_status);
                        if (!alive) {
                            break;
                        }
                    }
                    const uint32_t bar = smem_u32(&sh->full[stage]);
                    const uint32_t a_dst = smem_base + stage * STAGE_BYTES;
                    const uint32_t b_dst = a_dst + A_BYTES;
                    // the rows of the tile past a_rows hold whatever they held: their products are rows of C past M
                    mbar_arrive_expect_tx(bar, p.a_rows * 128 + B_BYTES);
                    tma_load_2d(a_dst, &p.a, bar, batch * p.a_batch_cols + kc * TILE_K, tile_m * TILE_M);
                    if (p.b_mn_major == 0) {
                        tma_load_2d(b_dst, b_map, bar, kc * TILE_K, batch * p.b_batch_rows + tile_n * TILE_N);
                    } else {
                        // two [64 k x 64 n] chunks side by side
                        tma_load_2d(b_dst, b_map, bar, tile_n * TILE_N, batch * p.b_batch_rows + kc * TILE_K);
                        tma_load_2d(b_dst + B_BYTES / 2, b_map, bar, tile_n * TILE_N + 64, batch * p.b_batch_rows + kc * TILE_K);
                    }
                }
            }
        }
    } else if (warp == MMA_WARP) {
        const uint32_t leader = elect_one();
        const uint32_t idesc = make_idesc_bf16(TILE_M, TILE_N, false, p.b_mn_major != 0);
        bool alive = true;
        long long chunk = 0;
        int local_tile = 0;
        for (long long tile = blockIdx.x; tile < tiles && alive; tile += gridDim.x, ++local_tile) {
            const int buffer = local_tile & 1;
            if (local_tile >= 2) {
                alive = __all_sync(0xffffffffU, mbar_wait(smem_u32(&sh->acc_empty[buffer]), static_cast<uint32_t>((local_tile / 2 - 1) & 1), abort_flag,
                                                          &projection_status));
                if (!alive) {
                    break;
                }
            }
            tc_fence_after_sync();
            const uint32_t acc = tmem_base + buffer * TILE_N;
            for (int kc = 0; kc < k_chunks && alive; ++kc, ++chunk) {
                const int stage = static_cast<int>(chunk % STAGES);
                alive = __all_sync(0xffffffffU, mbar_wait(smem_u32(&sh->full[stage]), static_cast<uint32_t>((chunk / STAGES) & 1), abort_flag, &projection_status));
                if (!alive) {
                    break;
                }
                tc_fence_after_sync();
                const uint32_t a_smem = smem_base + stage * STAGE_BYTES;
                const uint32_t b_smem = a_smem + A_BYTES;
#pragma unroll
                for (int k = 0; k < 4; ++k) {
                    const uint64_t b_desc = p.b_mn_major == 0 ? make_kmajor_desc(b_smem + k * 32) : make_smem_desc(b_smem + k * 2048, B_BYTES / 2, 1024);
                    mma_ss_elect(acc, make_kmajor_desc(a_smem + k * 32), b_desc, idesc, (kc | k) != 0 ? 1U : 0U, leader);
                }
                mma_commit_elect(smem_u32(&sh->empty[stage]), leader);
            }
            if (alive) {
                mma_commit_elect(smem_u32(&sh->acc_full[buffer]), leader);
            }
        }
    } else {
        // =================== epilogue: thread = row of the tile ==================
        const int r = threadIdx.x;
        const uint32_t lane_base = static_cast<uint32_t>(warp * 32) << 16;
        bool alive = true;
        int local_tile = 0;
        for (long long tile = blockIdx.x; tile < tiles && alive; tile += gridDim.x, ++local_tile) {
            int batch, tile_n, tile_m;
            locate(tile, batch, tile_n, tile_m);
            const int buffer = local_tile & 1;
            alive = __all_sync(0xffffffffU, mbar_wait(smem_u32(&sh->acc_full[buffer]), static_cast<uint32_t>((local_tile / 2) & 1), abort_flag, &projection_status));
            if (!alive) {
                break;
            }
            tc_fence_after_sync();
            // the output buffer was last used two tiles ago; its store must have read it
            if (local_tile >= 2) {
                alive = __all_sync(0xffffffffU, mbar_wait(smem_u32(&sh->out_free[buffer]), static_cast<uint32_t>((local_tile / 2 - 1) & 1), abort_flag,
                                                          &projection_status));
                if (!alive) {
                    break;
                }
            }
            uint8_t* out_row = smem_aligned + STAGES * STAGE_BYTES + buffer * OUT_BYTES + r * 128;
#pragma unroll
            for (int c = 0; c < TILE_N / 32; ++c) {
                uint32_t values[32];
                tmem_ld_x32(tmem_base + lane_base + buffer * TILE_N + c * 32, values);
                tmem_wait_ld();
                // columns 32c..32c+31 = 16-byte units 4(c&1)..4(c&1)+3 of row r in chunk c/2, swizzled by the row
#pragma unroll
                for (int u = 0; u < 4; ++u) {
                    uint4 vec;
                    vec.x = pack_bf16x2(__uint_as_float(values[8 * u]), __uint_as_float(values[8 * u + 1]));
                    vec.y = pack_bf16x2(__uint_as_float(values[8 * u + 2]), __uint_as_float(values[8 * u + 3]));
                    vec.z = pack_bf16x2(__uint_as_float(values[8 * u + 4]), __uint_as_float(values[8 * u + 5]));
                    vec.w = pack_bf16x2(__uint_as_float(values[8 * u + 6]), __uint_as_float(values[8 * u + 7]));
                    const int unit = (c & 1) * 4 + u;
                    *reinterpret_cast<uint4*>(out_row + (c >> 1) * (OUT_BYTES / 2) + ((unit ^ (r & 7)) * 16)) = vec;
                }
            }
            tc_fence_before_sync();
            mbar_arrive(smem_u32(&sh->acc_empty[buffer]));         // the accumulator is free as soon as it is in registers / shared memory
            fence_proxy_async_smem();
            mbar_arrive(smem_u32(&sh->out_written[buffer]));
            if (r == 0) {
                const bool written = mbar_wait(smem_u32(&sh->out_written[buffer]), static_cast<uint32_t>((local_tile / 2) & 1), abort_flag, &projection_status);
                if (written) {
                    const uint32_t src = smem_base + STAGES * STAGE_BYTES + buffer * OUT_BYTES;
                    const int x = batch * p.c_batch_cols + tile_n * TILE_N;
                    const CUtensorMap* c_map = &p.c[p.map_by_batch * batch];
                    tma_store_2d(c_map, src, x, tile_m * TILE_M);
                    tma_store_2d(c_map, src + OUT_BYTES / 2, x + 64, tile_m * TILE_M);
                    tma_store_commit();
                    tma_store_wait_read();
                    mbar_arrive(smem_u32(&sh->out_free[buffer]));
                }
            }
        }
        if (r == 0) {
            tma_store_wait_all();       // the last stores have been written before the CTA exits
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

// ---------------------------------------------------------------------------
// Pair kernel: 256 x 256 tiles by two CTAs.  CTA r holds rows [128 r, +128) of the A tile and of the accumulator and
// half of the B tile (128 of its columns, all of K).  Clusters take contiguous ranges of the tile list (rows
// fastest), so B is loaded once or twice per cluster; its chunks have a barrier each and the first tile starts on the
// first of them.  Tensor memory: two accumulators of 256 columns.  Shared memory: B 128 KB, four 16 KB stages of A,
// two 4 KB output slabs for each epilogue warp (32 rows x 64 columns, one TMA store).
// Up-projection of 16384 rows to 128 heads (k and v): 579 us in two launches of the single-CTA kernel, 483 us here
// (1139 TFLOP/s at the power cap); of 2048 rows 88.5 -> 60.1 us.
// ---------------------------------------------------------------------------
namespace pk {
constexpr int PAIR_M = 256;
constexpr int CTA_M = 128;
constexpr int MAX_K_CHUNKS = 8;
constexpr int A_STAGES = 4;
constexpr int SLAB = 32 * 128;
constexpr int SLABS_BYTES = 4 * 2 * SLAB;

constexpr int N_TILE = 256;
constexpr int HALF_N = N_TILE / 2;
constexpr int B_CHUNK = HALF_N * 128;             // K-major: [128 rows x 64 k]; MN-major: two [64 k x 64 n] blocks side by side
constexpr int PAIR_SMEM_BYTES = MAX_K_CHUNKS * B_CHUNK + A_STAGES * A_BYTES + SLABS_BYTES + MISC_BYTES + 1024;
static_assert(PAIR_SMEM_BYTES <= 232448, "pair kernel shared memory");

struct PairShared {
    uint64_t full[A_STAGES];                // this CTA's A chunk has landed
    uint64_t b_full[MAX_K_CHUNKS];          // this CTA's half of a B chunk has landed
    uint64_t peer_full[A_STAGES];           // leader: the same events of the other CTA, forwarded by its relay warp
    uint64_t peer_b_full[MAX_K_CHUNKS];
    uint64_t empty[A_STAGES];               // tcgen05.commit of the leader, one for each CTA
    uint64_t b_empty;
    uint64_t acc_full[2];
    uint64_t acc_empty[2];                  // leader: one arrival per epilogue warp of either CTA
    uint32_t tmem_base;
    int abort_flag;
};
static_assert(sizeof(PairShared) <= MISC_BYTES, "barrier block too large");
}  // namespace pk

__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(THREADS, 1) projection_pair_kernel(const __grid_constant__ GemmParams p) {
    using namespace pk;
    extern __shared__ uint8_t smem_raw[];
    const int warp = threadIdx.x / 32;
    const int lane = threadIdx.x % 32;
    const uint32_t rank = cluster_cta_rank();
    const int cluster = blockIdx.x >> 1;
    const int clusters = gridDim.x >> 1;
    const uint32_t smem_base = (smem_u32(smem_raw) + 1023U) & ~1023U;
    uint8_t* smem_aligned = smem_raw + (smem_base - smem_u32(smem_raw));
    const uint32_t b_smem = smem_base;
    const uint32_t a_smem = b_smem + MAX_K_CHUNKS * B_CHUNK;
    constexpr int SLABS_OFFSET = MAX_K_CHUNKS * B_CHUNK + A_STAGES * A_BYTES;
    PairShared* sh = reinterpret_cast<PairShared*>(smem_aligned + SLABS_OFFSET + SLABS_BYTES);
    volatile int* abort_flag = &sh->abort_flag;

    if (threadIdx.x == 0) {
        for (int i = 0; i < A_STAGES; ++i) {
            mbar_init(smem_u32(&sh->full[i]), 1);
            mbar_init(smem_u32(&sh->peer_full[i]), 1);
            mbar_init(smem_u32(&sh->empty[i]), 1);
        }
        for (int i = 0; i < MAX_K_CHUNKS; ++i) {
            mbar_init(smem_u32(&sh->b_full[i]), 1);
            mbar_init(smem_u32(&sh->peer_b_full[i]), 1);
        }
        mbar_init(smem_u32(&sh->b_empty), 1);
        for (int i = 0; i < 2; ++i) {
            mbar_init(smem_u32(&sh->acc_full[i]), 1);
            mbar_init(smem_u32(&sh->acc_empty[i]), 8);
        }
        sh->abort_flag = 0;
        mbar_init_fence();
    }
    if (warp == MMA_WARP) {
        tmem_alloc_pair(smem_u32(&sh->tmem_base), 2 * N_TILE);
        tmem_relinquish_pair();
    }
    if (warp == LOAD_WARP && lane == 0) {
        tma_prefetch_descriptor(&p.a);
        tma_prefetch_descriptor(&p.b[0]);
        tma_prefetch_descriptor(&p.c[0]);
    }
    tc_fence_before_sync();
    __syncthreads();
    cluster_sync_all();
    tc_fence_after_sync();
    grid_dependency_wait();
    const uint32_t tmem_base = *reinterpret_cast<volatile uint32_t*>(&sh->tmem_base);

    const int tiles_m = (p.m + PAIR_M - 1) / PAIR_M;
    const int tiles_n = (p.n + N_TILE - 1) / N_TILE;
    const long long tiles = static_cast<long long>(tiles_m) * tiles_n * p.batch;
    const long long tile_begin = tiles * cluster / clusters;
    const long long tile_end = tiles * (cluster + 1) / clusters;
    const int k_chunks = p.k / TILE_K;
    // a column of tiles (batch entry, n) shares its B tile
    auto column_of = [&](long long tile) { return static_cast<int>(tile / tiles_m); };

    if (warp == LOAD_WARP) {
        if (lane == 0) {
            bool alive = true;
            long long chunk = 0;
            int column = -1, b_tiles = 0;
            for (long long tile = tile_begin; tile < tile_end && alive; ++tile) {
                const int tile_m = static_cast<int>(tile % tiles_m);
                const bool new_b = column_of(tile) != column;
                column = column_of(tile);
                const int batch = column / tiles_n, tile_n = column % tiles_n;
                const CUtensorMap* b_map = &p.b[p.map_by_batch * batch];
                if (new_b && b_tiles > 0) {
                    alive = mbar_wait(smem_u32(&sh->b_empty), (b_tiles - 1) & 1, abort_flag, &projection_status);
                }
                for (int kc = 0; kc < k_chunks && alive; ++kc, ++chunk) {
                    if (new_b) {
                        const uint32_t bar = smem_u32(&sh->b_full[kc]);
                        const uint32_t dst = b_smem + kc * B_CHUNK;
                        const int n0 = tile_n * N_TILE + static_cast<int>(rank) * HALF_N;
                        mbar_arrive_expect_tx(bar, B_CHUNK);
                        if (p.b_mn_major == 0) {
                            tma_load_2d(dst, b_map, bar, kc * TILE_K, batch * p.b_batch_rows + n0);
                        } else {
                            for (int block = 0; block < HALF_N / 64; ++block) {
                                tma_load_2d(dst + block * 8192, b_map, bar, n0 + block * 64, batch * p.b_batch_rows + kc * TILE_K);
                            }
                        }
                    }
                    const int stage = static_cast<int>(chunk % A_STAGES);
                    if (chunk >= A_STAGES) {
                        alive = mbar_wait(smem_u32(&sh->empty[stage]), static_cast<uint32_t>((chunk / A_STAGES - 1) & 1), abort_flag, &projection_status);
                        if (!alive) {
                            break;
                        }
                    }
                    const uint32_t bar = smem_u32(&sh->full[stage]);
                    mbar_arrive_expect_tx(bar, A_BYTES);
                    tma_load_2d(a_smem + stage * A_BYTES, &p.a, bar, batch * p.a_batch_cols + kc * TILE_K,
                                tile_m * PAIR_M + static_cast<int>(rank) * CTA_M);
                }
                b_tiles += new_b ? 1 : 0;
            }
        }
    } else if (warp == MMA_WARP && rank != 0) {
        // relay: every load of this CTA, in the order they were issued -> the leader
        if (lane == 0) {
            bool alive = true;
            long long chunk = 0;
            int column = -1, b_tiles = 0;
            for (long long tile = tile_begin; tile < tile_end && alive; ++tile) {
                const bool new_b = column_of(tile) != column;
                column = column_of(tile);
                for (int kc = 0; kc < k_chunks && alive; ++kc, ++chunk) {
                    if (new_b) {
                        alive = mbar_wait(smem_u32(&sh->b_full[kc]), b_tiles & 1, abort_flag, &projection_status);
                        if (!alive) {
                            break;
                        }
                        mbar_arrive_remote(map_to_cta(smem_u32(&sh->peer_b_full[kc]), 0));
                    }
                    const int stage = static_cast<int>(chunk % A_STAGES);
                    alive = mbar_wait(smem_u32(&sh->full[stage]), static_cast<uint32_t>((chunk / A_STAGES) & 1), abort_flag, &projection_status);
                    if (alive) {
                        mbar_arrive_remote(map_to_cta(smem_u32(&sh->peer_full[stage]), 0));
                    }
                }
                b_tiles += new_b ? 1 : 0;
            }
        }
    } else if (warp == MMA_WARP) {
        const uint32_t leader = elect_one();
        const uint32_t idesc = make_idesc_bf16(PAIR_M, N_TILE, false, p.b_mn_major != 0);
        constexpr uint32_t HI = smem_desc_hi(1024);
        auto both = [&](uint64_t* bar) {
            commit_pair(smem_u32(bar), leader);
            commit_pair(map_to_cta(smem_u32(bar), 1), leader);
        };
        bool alive = true;
        long long chunk = 0;
        int column = -1, b_tiles = 0, local_tile = 0;
        auto wait = [&](uint64_t* bar, uint32_t parity) {
            return __all_sync(0xffffffffU, mbar_wait(smem_u32(bar), parity, abort_flag, &projection_status));
        };
        for (long long tile = tile_begin; tile < tile_end && alive; ++tile, ++local_tile) {
            const bool new_b = column_of(tile) != column;
            column = column_of(tile);
            const int buffer = local_tile & 1;
            if (local_tile >= 2) {
                alive = wait(&sh->acc_empty[buffer], static_cast<uint32_t>((local_tile / 2 - 1) & 1));
            }
            const uint32_t acc = tmem_base + buffer * N_TILE;
            for (int kc = 0; kc < k_chunks && alive; ++kc, ++chunk) {
                if (new_b) {
                    alive = wait(&sh->b_full[kc], b_tiles & 1) && wait(&sh->peer_b_full[kc], b_tiles & 1);
                }
                const int stage = static_cast<int>(chunk % A_STAGES);
                const uint32_t parity = static_cast<uint32_t>((chunk / A_STAGES) & 1);
                alive = alive && wait(&sh->full[stage], parity) && wait(&sh->peer_full[stage], parity);
                if (!alive) {
                    break;
                }
                tc_fence_after_sync();
                const uint32_t a_lo = smem_desc_lo(a_smem + stage * A_BYTES, 16);
                if (p.b_mn_major == 0) {
                    const uint32_t b_lo = smem_desc_lo(b_smem + kc * B_CHUNK, 16);
#pragma unroll
                    for (int k = 0; k < 4; ++k) {
                        mma_pair_ss_split(acc, a_lo + 2 * k, HI, b_lo + 2 * k, HI, idesc, (kc | k) != 0 ? 1U : 0U, leader);
                    }
                } else {
                    const uint32_t b_lo = smem_desc_lo(b_smem + kc * B_CHUNK, 8192);
#pragma unroll
                    for (int k = 0; k < 4; ++k) {
                        mma_pair_ss_split(acc, a_lo + 2 * k, HI, b_lo + (k * 2048 >> 4), HI, idesc, (kc | k) != 0 ? 1U : 0U, leader);
                    }
                }
                both(&sh->empty[stage]);
            }
            b_tiles += new_b ? 1 : 0;
            if (alive) {
                both(&sh->acc_full[buffer]);
                if (tile + 1 < tile_end && column_of(tile + 1) != column) {
                    both(&sh->b_empty);
                }
            }
        }
    } else {
        // =================== epilogue: warp = 32 rows of this CTA's half of the tile, thread = row ==================
        const uint32_t lane_base = static_cast<uint32_t>(warp * 32) << 16;
        bool alive = !gave_up_before(&projection_status, abort_flag);
        int local_tile = 0;
        for (long long tile = tile_begin; tile < tile_end && alive; ++tile, ++local_tile) {
            const int column = column_of(tile);
            const int batch = column / tiles_n, tile_n = column % tiles_n;
            const CUtensorMap* c_map = &p.c[p.map_by_batch * batch];
            const int row = static_cast<int>(tile % tiles_m) * PAIR_M + static_cast<int>(rank) * CTA_M + warp * 32;
            const int buffer = local_tile & 1;
            alive = __all_sync(0xffffffffU, mbar_wait(smem_u32(&sh->acc_full[buffer]), static_cast<uint32_t>((local_tile / 2) & 1), abort_flag, &projection_status));
            if (!alive) {
                break;
            }
            tc_fence_after_sync();
#pragma unroll
            for (int c = 0; c < N_TILE / 64; ++c) {
                uint32_t values[64];
                const uint32_t src = tmem_base + lane_base + buffer * N_TILE + c * 64;
                tmem_ld_x32(src, values);
                tmem_ld_x32(src + 32, values + 32);
                tmem_wait_ld();
                if (c + 1 == N_TILE / 64) {             // the accumulator is in registers: the next but one tile may have it
                    tc_fence_before_sync();
                    __syncwarp();
                    if (lane == 0) {
                        if (rank == 0) {
                            mbar_arrive(smem_u32(&sh->acc_empty[buffer]));
                        } else {
                            mbar_arrive_remote(map_to_cta(smem_u32(&sh->acc_empty[buffer]), 0));
                        }
                    }
                }
                if (lane == 0) {
                    tma_store_wait_read_but_one();      // the slab's last store, two stores ago
                }
                __syncwarp();
                const int slab = SLABS_OFFSET + (warp * 2 + (c & 1)) * SLAB;
                uint8_t* row_ptr = smem_aligned + slab + lane * 128;
#pragma unroll
                for (int u = 0; u < 8; ++u) {
                    const uint32_t* x = values + 8 * u;
                    *reinterpret_cast<uint4*>(row_ptr + ((u ^ (lane & 7)) * 16)) =
                        make_uint4(pack_bf16x2(__uint_as_float(x[0]), __uint_as_float(x[1])), pack_bf16x2(__uint_as_float(x[2]), __uint_as_float(x[3])),
                                   pack_bf16x2(__uint_as_float(x[4]), __uint_as_float(x[5])), pack_bf16x2(__uint_as_float(x[6]), __uint_as_float(x[7])));
                }
                fence_proxy_async_smem();
                __syncwarp();
                const int n0 = tile_n * N_TILE + c * 64;
                if (lane == 0) {
                    if (row < p.m && n0 < p.n) {
                        tma_store_2d(c_map, smem_base + slab, batch * p.c_batch_cols + n0, row);
                    }
                    tma_store_commit();
                }
            }
        }
        if (lane == 0) {
            tma_store_wait_all();       // the last stores have been written before the CTA exits
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
    cluster_sync_all();                 // neither CTA frees tensor memory or exits while the other may still signal it
    if (warp == MMA_WARP) {
        tc_fence_after_sync();
        tmem_dealloc_pair(tmem_base, 2 * N_TILE);
    }
}

int sm_count() {
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

void configure_kernel() {
    static bool done[16] = {};
    int device = 0;
    CUDA_CHECK(cudaGetDevice(&device));
    if (device < 16 && done[device]) {
        return;
    }
    CUDA_CHECK(cudaFuncSetAttribute(projection_gemm_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM_BYTES));
    CUDA_CHECK(cudaFuncSetAttribute(projection_pair_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, pk::PAIR_SMEM_BYTES));
    if (device < 16) {
        done[device] = true;
    }
}

// Up to this many (128 x 128 tile, 64-column chunk of K) steps the single-CTA kernel runs: it takes about 5 us + 0.39 us for
// each step of an SM (32 KB from L2), the pair kernel about 8 us + 0.25 us for the same work, so they meet at 20 steps per SM.
// That is for K = 512.  At K = 128 (W_UK into the query), where writing C is the bound, they meet earlier, near 8 steps per SM:
// 16 heads of 1024 rows 8.4 and 8.6 us, of 1536 rows 11.0 and 10.1, of 2048 rows 12.4 and 11.6 (single-CTA, pair).  Beyond L2 the
// place of C in memory decides between them: 128 heads of 4096 rows 152 and 158 us with nothing else allocated, 172 and 163 in a
// program that holds 2 GB more; 64 heads of 16384 rows 299 and 305, 350 and 316.
constexpr long long SMALL_STEPS = 20 * 148;

// C_b [m, n] = A_b [m, k] op(B_b) for b in [0, batch): see GemmParams for the batch offsets.  With `b2` the entries of a
// batch of two are two weights and two outputs of the same A.
void launch_gemm(__nv_bfloat16* c, const __nv_bfloat16* a, const __nv_bfloat16* b, long long m, int n, int k, long long a_cols, long long b_rows,
                 long long b_cols, long long ldc, int batch, int a_batch_cols, int b_batch_rows, int c_batch_cols, bool b_mn_major,
                 cudaStream_t stream, __nv_bfloat16* c2 = nullptr, const __nv_bfloat16* b2 = nullptr) {
    if (m <= 0 || n <= 0 || k <= 0 || batch <= 0) {
        throw std::invalid_argument("MLA projection requires positive sizes");
    }
    if (n % TILE_N != 0 || k % TILE_K != 0 || k > pk::MAX_K_CHUNKS * TILE_K) {
        throw std::invalid_argument("MLA projection requires N to be a multiple of 128 and K a multiple of 64 up to 512");
    }
    if (m > 0x7fffffffLL - pk::PAIR_M) {
        throw std::invalid_argument("MLA projection shape exceeds the supported index range");
    }
    for (const void* pointer : {static_cast<const void*>(c), static_cast<const void*>(a), static_cast<const void*>(b),
                                static_cast<const void*>(b2 != nullptr ? b2 : b), static_cast<const void*>(b2 != nullptr ? c2 : c)}) {
        if (pointer == nullptr) {
            throw std::invalid_argument("null tensor pointer");
        }
        if ((reinterpret_cast<std::uintptr_t>(pointer) & 15U) != 0) {
            throw std::invalid_argument("tensor pointers must be 16-byte aligned");
        }
    }
    const long long small_tiles = ((m + TILE_M - 1) / TILE_M) * (n / TILE_N) * batch;
    // a head's own 128 columns (W_UV) make no 256-wide tile; there the kernel is bound by reading the latent rows anyway
    const bool wide = n % pk::N_TILE == 0 || batch == 1 || b2 != nullptr;
    const bool small = !wide || small_tiles * (k / TILE_K) <= SMALL_STEPS;
    GemmParams params{};
    const std::uint64_t rows = static_cast<std::uint64_t>(m);
    auto columns = [](long long value) { return static_cast<std::uint64_t>(value); };
    // A decode step has a few rows per head: loads of as many (whole groups of 8, the swizzle's period) instead of 128
    params.a_rows = small ? static_cast<int>(std::min<long long>(TILE_M, (m + 7) / 8 * 8)) : TILE_M;
    params.a = make_bf16_tile_map(a, rows, columns(a_cols), columns(a_cols), params.a_rows);
    const std::uint32_t b_box = b_mn_major ? TILE_K : (small ? TILE_N : pk::HALF_N);
    const std::uint32_t c_box = small ? TILE_M : 32;
    params.b[0] = make_bf16_tile_map(b, columns(b_rows), columns(b_cols), columns(b_cols), b_box);
    params.c[0] = make_bf16_tile_map(c, rows, columns(ldc), columns(ldc), c_box);
    if (b2 != nullptr) {
        params.b[1] = make_bf16_tile_map(b2, columns(b_rows), columns(b_cols), columns(b_cols), b_box);
        params.c[1] = make_bf16_tile_map(c2, rows, columns(ldc), columns(ldc), c_box);
        params.map_by_batch = 1;
    }
    params.m = static_cast<int>(m);
    params.n = n;
    params.k = k;
    params.batch = batch;
    params.a_batch_cols = a_batch_cols;
    params.b_batch_rows = b_batch_rows;
    params.c_batch_cols = c_batch_cols;
    params.b_mn_major = b_mn_major ? 1 : 0;
    configure_kernel();
    if (small) {
        const unsigned grid = static_cast<unsigned>(std::min<long long>(small_tiles, sm_count()));
        launch_chained(projection_gemm_kernel, dim3(grid), dim3(THREADS), SMEM_BYTES, stream, params);
        return;
    }
    const long long tiles = ((m + pk::PAIR_M - 1) / pk::PAIR_M) * ((n + pk::N_TILE - 1) / pk::N_TILE) * batch;
    const unsigned grid = 2 * static_cast<unsigned>(std::min<long long>(tiles, sm_count() / 2));
    launch_chained(projection_pair_kernel, dim3(grid), dim3(THREADS), pk::PAIR_SMEM_BYTES, stream, params);
}

void check_heads(long long rows, int heads) {
    if (rows <= 0 || heads <= 0) {
        throw std::invalid_argument("MLA projection requires positive rows and heads");
    }
    if (static_cast<long long>(heads) * MLA_KV_RANK > 0x7fffffffLL) {
        throw std::invalid_argument("MLA projection shape exceeds the supported index range");
    }
}

}  // namespace

namespace internal {

int projection_device_status(bool reset) {
    int status = 0;
    CUDA_CHECK(cudaDeviceSynchronize());
    CUDA_CHECK(cudaMemcpyFromSymbol(&status, projection_status, sizeof(int)));
    if (reset && status != 0) {
        const int zero = 0;
        CUDA_CHECK(cudaMemcpyToSymbol(projection_status, &zero, sizeof(int)));
    }
    return status;
}

}  // namespace internal

void mla_up_project_cuda(__nv_bfloat16* k_nope, __nv_bfloat16* v, const __nv_bfloat16* kv_latent, const __nv_bfloat16* w_uk,
                         const __nv_bfloat16* w_uv, long long rows, int heads, cudaStream_t stream) {
    check_heads(rows, heads);
    const int n = heads * MLA_NOPE_SIZE;
    if (k_nope == nullptr && v == nullptr) {
        throw std::invalid_argument("MLA up-projection needs at least one output");
    }
    if (k_nope != nullptr && v != nullptr) {
        launch_gemm(k_nope, kv_latent, w_uk, rows, n, MLA_KV_RANK, MLA_KV_RANK, n, MLA_KV_RANK, n, 2, 0, 0, 0, false, stream, v, w_uv);
    } else {
        launch_gemm(k_nope != nullptr ? k_nope : v, kv_latent, k_nope != nullptr ? w_uk : w_uv, rows, n, MLA_KV_RANK, MLA_KV_RANK, n, MLA_KV_RANK, n, 1,
                    0, 0, 0, false, stream);
    }
}

void mla_absorb_query_cuda(__nv_bfloat16* q_latent, const __nv_bfloat16* q_nope, const __nv_bfloat16* w_uk, long long rows, int heads,
                           cudaStream_t stream) {
    check_heads(rows, heads);
    // per head: [rows, 128] x W_UK[h] ([128, 512], used as stored: K rows, N contiguous)
    launch_gemm(q_latent, q_nope, w_uk, rows, MLA_KV_RANK, MLA_NOPE_SIZE, static_cast<long long>(heads) * MLA_NOPE_SIZE,
                static_cast<long long>(heads) * MLA_NOPE_SIZE, MLA_KV_RANK, static_cast<long long>(heads) * MLA_KV_RANK, heads, MLA_NOPE_SIZE,
                MLA_NOPE_SIZE, MLA_KV_RANK, true, stream);
}

void mla_unabsorb_output_cuda(__nv_bfloat16* output, const __nv_bfloat16* output_latent, const __nv_bfloat16* w_uv, long long rows, int heads,
                              cudaStream_t stream) {
    check_heads(rows, heads);
    // per head: [rows, 512] x W_UV[h]^T (W_UV[h] is [128, 512]: N rows, K contiguous)
    launch_gemm(output, output_latent, w_uv, rows, MLA_VALUE_SIZE, MLA_KV_RANK, static_cast<long long>(heads) * MLA_KV_RANK,
                static_cast<long long>(heads) * MLA_VALUE_SIZE, MLA_KV_RANK, static_cast<long long>(heads) * MLA_VALUE_SIZE, heads, MLA_KV_RANK,
                MLA_VALUE_SIZE, MLA_VALUE_SIZE, false, stream);
}

}  // namespace dscuda
