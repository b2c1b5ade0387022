// Matrix products over unquantised 16-bit weights for many rows (prefill), dense or grouped by expert, on tcgen05 kind::f16.
//
// Persistent pairs of CTAs (clusters of two, one CTA per SM; cta_group::2).  A tile is 256 weight rows (the MMA's M, 128 in each CTA, one
// tensor-memory lane each) times up to 256 activation rows (its N, each CTA brings half of them).  With gating it is 128 outputs: each CTA
// holds 64 gate rows and the 64 up rows of the same outputs, and two warps of the epilogue exchange halves of what they read through shared
// memory.  Warp 0 of both CTAs streams by TMA through a ring of six stages (64 elements of the contraction, 32 KB in each CTA, 128-byte
// swizzle), warp 1 of the first issues the MMAs of both into one of two 256-column accumulators, warps 2-9 of both drain the other
// one: tcgen05.ld, activation or gating, rounding, a store of 64 bytes per warp and activation row.
// A CTA on its own takes in 48 KB per 128 x 256 x 64 of the product, 96 bytes per clock at the 16-bit rate, where an SM gets about 64 from L2; a pair's CTA takes
// 32: 2048 rows x 16384 x 4096 201 -> 176 us (1.57 PFLOP/s, the rate under the power cap), x 4096 x 4096 56 -> 49, 500 x 2048 x 4096 29 -> 21; eight experts of 2 x
// 7168 x 4096 over 4040 rows 403 -> 376.  Activation rows are the N side because N has any multiple of 32: a tile is as wide as its rows, where 128-row tiles padded the last
// one of each expert.
// Grouped products take their tiles from the list the router's ordering left (MoeRoute::tile_e / tile_row: kMoeTileRows places that do not
// cross experts).  Rows of other experts that a tile's copies bring along are computed and not stored.
// All waits are bounded and report through the caller's status word.
#include "block_ops.cuh"
#include "common.cuh"
#include "i8_gemm.cuh"
#include "tcgen05.cuh"

#include <algorithm>
#include <type_traits>

namespace mynn {

MYNN_DEFINE_WAIT_BUDGET_SETTER(dense_gemm_tc)

constexpr int kDgRows = 128;           // weight rows of one CTA of a pair (half of UMMA M)
constexpr int kDgCols = 256;           // most activation rows per tile (UMMA N)
static_assert(kMoeTileRows == kDgCols, "a tile of the router's list is one tile here");
constexpr int kDgK = 64;               // elements per stage: 128 bytes
constexpr int kDgStages = 6;
constexpr int kDgEpiWarps = 8;
constexpr int kDgThreads = 64 + 32 * kDgEpiWarps;
constexpr uint32_t kDgWBytes = kDgRows * kDgK * 2, kDgABytes = kDgCols / 2 * kDgK * 2, kDgStageBytes = kDgWBytes + kDgABytes;
constexpr int kDgXRows = 16;           // activation rows of a chunk that a warp leaves to its partner (gating)
constexpr uint32_t kDgXBytes = 2 * kDgEpiWarps * kDgXRows * 32 * 4;  // two buffers per epilogue warp

struct DgParams {
    void *out;
    int M, N, K;
    int n_tiles;                                  // weight tiles
    int cols, box;                                // activation rows per tile, a multiple of 32; rows of one copy of them
    const int32_t *off, *tile_e, *tile_row, *m_tiles_dev;  // grouped: see MoeRoute; null: dense
    int row_block;                                // so many row tiles share the weight tiles that are in flight (see locate)
    int ldo, n_main, act_fn, out_block;           // see DenseGemm; out_block 0: none
    long long out_block_stride;
    float *out_f32;
    int groups, group_tiles;                      // dense: groups of rows and row tiles of each; 0: one group
    long long group_rows;                         // distance of the groups' first rows
    int *status;
};

template <typename T, typename O, bool GLU>
__global__ void __launch_bounds__(kDgThreads, 1)
dense_gemm_tc_kernel(const __grid_constant__ CUtensorMap map_a, const __grid_constant__ CUtensorMap map_w, const DgParams p) {
    extern __shared__ uint8_t smem_raw[];
    uint8_t *smem = (uint8_t *)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
    __shared__ uint64_t full_bar[kDgStages], empty_bar[kDgStages], acc_full[2], acc_empty[2];
    __shared__ uint32_t tmem_slot;
    __shared__ int abort_flag, sh_go[2];
    constexpr int NT = GLU ? kDgRows : 2 * kDgRows;  // outputs per tile

    const int warp = __shfl_sync(0xffffffffu, (int)threadIdx.x >> 5, 0), lane = threadIdx.x & 31;
    const uint32_t rank = cluster_ctarank();
    const int first_tile = blockIdx.x >> 1, tile_stride = gridDim.x >> 1;
    const int kblocks = (p.K + kDgK - 1) / kDgK;
    if (threadIdx.x == 0) {
        for (int s = 0; s < kDgStages; s++) {
            mbar_init(&full_bar[s], 1);
            mbar_init(&empty_bar[s], 1);
        }
        for (int b = 0; b < 2; b++) {
            mbar_init(&acc_full[b], 1);
            mbar_init(&acc_empty[b], 2 * kDgEpiWarps);  // one arrival per epilogue warp of both CTAs (used in the first CTA)
        }
        abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 1) tmem_alloc_pair(&tmem_slot, 512);
    tc_fence_before();
    __syncthreads();
    cluster_sync_all();  // the barriers of both CTAs are set up
    tc_fence_after();
    const uint32_t tmem_base = tmem_slot;
    pdl_wait();  // activations and the tile list come from the preceding kernels
    const int m_tiles = p.m_tiles_dev ? *p.m_tiles_dev : p.group_tiles ? p.group_tiles * p.groups : (p.M + p.cols - 1) / p.cols;
    const int total = m_tiles * p.n_tiles;
    auto give_up = [&](int code) {
        atomicExch(&abort_flag, 1);
        atomicExch(p.status, code);
    };
    auto group_base = [&](int mt) { return p.group_tiles ? (int)((mt / p.group_tiles) * p.group_rows) : 0; };
    // first activation row of a row tile, and how many it has
    auto rows_of = [&](int mt, int &row0, int &live) {
        if (p.tile_e) {
            row0 = p.tile_row[mt];
            live = min(p.cols, p.off[p.tile_e[mt] + 1] - row0);
        } else {
            const int base = group_base(mt), in = (p.group_tiles ? mt % p.group_tiles : mt) * p.cols;
            row0 = base + in;
            live = min(p.cols, p.M - in);
        }
    };
    // N of the MMA: the first CTA holds the first half of these rows, the second the other
    auto mma_cols = [](int live) { return ((live + 31) >> 5) << 5; };
    // Blocks of row tiles, in each block the weight tiles, in each weight tile the block's row tiles: what the CTAs read at one time is a
    // few weight tiles and one block of rows, and a weight tile comes from DRAM once per block.
    const int row_block = min(p.row_block, m_tiles), block_tiles = row_block * p.n_tiles;
    auto locate = [&](int tile, int &mt, int &nt) {
        const int block = tile / block_tiles, rest = tile - block * block_tiles, first = block * row_block, here = min(row_block, m_tiles - first);
        nt = rest / here;
        mt = first + rest - nt * here;
    };

    if (warp == 0) {
        // ---------------- TMA producer ----------------
        if (elect_one()) {
            asm volatile("prefetch.tensormap [%0];" ::"l"(&map_a) : "memory");
            asm volatile("prefetch.tensormap [%0];" ::"l"(&map_w) : "memory");
        }
        int s = 0, use = 0;
        bool ok = true;
        for (int tile = first_tile; tile < total && ok; tile += tile_stride) {
            int mt, nt, row0, live;
            locate(tile, mt, nt);
            rows_of(mt, row0, live);
            const int e = p.tile_e ? p.tile_e[mt] : 0, half = mma_cols(live) >> 1, boxes = (half + p.box - 1) / p.box, row = row0 + (int)rank * half;
            const int wrow = e * (GLU ? 2 * p.N : p.N) + nt * NT + (int)rank * (NT / 2);
            const uint32_t bytes = 2 * (kDgWBytes + (uint32_t)(boxes * p.box) * (kDgK * 2));  // what both CTAs bring into a stage
            for (int kb = 0; kb < kblocks; kb++) {
                if (use > 0 && !__all_sync(0xffffffffu, mbar_wait_spin(&empty_bar[s], (use - 1) & 1, &abort_flag))) {
                    ok = false;
                    break;
                }
                uint8_t *st = smem + s * kDgStageBytes;
                const uint32_t bar = map_rank(smem_u32(&full_bar[s]), 0);
                if (elect_one()) {
                    if (rank == 0) mbar_expect_tx(&full_bar[s], bytes);
                    tma_load_2d_pair(st, &map_w, kb * 128, wrow, bar);  // byte maps: x counts bytes
                    if constexpr (GLU) tma_load_2d_pair(st + kDgWBytes / 2, &map_w, kb * 128, wrow + p.N, bar);
                    for (int i = 0; i < boxes; i++) tma_load_2d_pair(st + kDgWBytes + i * p.box * 128, &map_a, kb * 128, row + i * p.box, bar);
                }
                __syncwarp();
                if (++s == kDgStages) s = 0, use++;
            }
        }
        // The commits that give the last stages back arrive in both CTAs: neither is left before its own have.
        for (int i = 0; i < kDgStages && ok; i++) {
            if (use > 0) ok = __all_sync(0xffffffffu, mbar_wait_spin(&empty_bar[s], (use - 1) & 1, &abort_flag));
            if (++s == kDgStages) s = 0, use++;
        }
        if (!ok && lane == 0) give_up(41);
        __syncwarp();
    } else if (warp == 1) {
        // ---------------- MMA issuer of the pair ----------------
        if (rank == 0) {
            constexpr uint32_t ab = std::is_same<T, __nv_bfloat16>::value ? 1u : 0u;  // operand format: 0 = f16, 1 = bf16
            int s = 0, phase = 0, it = 0;
            bool ok = true;
            for (int tile = first_tile; tile < total && ok; tile += tile_stride, it++) {
                const int buf = it & 1, use = it >> 1;
                int mt, nt, row0, live;
                locate(tile, mt, nt);
                rows_of(mt, row0, live);
                const uint32_t idesc = (1u << 4) | (ab << 7) | (ab << 10) | ((uint32_t)(mma_cols(live) >> 3) << 17) | ((uint32_t)(2 * kDgRows >> 4) << 24);
                if (use > 0 && !__all_sync(0xffffffffu, mbar_wait_spin(&acc_empty[buf], (use - 1) & 1, &abort_flag))) {  // the epilogue has drained it
                    if (lane == 0) give_up(42);
                    break;
                }
                tc_fence_after();
                const uint32_t d_tmem = tmem_base + (uint32_t)(buf * kDgCols);
                for (int kb = 0; kb < kblocks; kb++) {
                    if (!__all_sync(0xffffffffu, mbar_wait_spin(&full_bar[s], phase, &abort_flag))) {
                        if (lane == 0) give_up(43);
                        ok = false;
                        break;
                    }
                    tc_fence_after();
                    const uint32_t w_addr = smem_u32(smem + s * kDgStageBytes);
                    const uint64_t wdesc = make_kmajor_sw128_desc(w_addr), adesc = make_kmajor_sw128_desc(w_addr + kDgWBytes);
                    if (elect_one()) {
#pragma unroll
                        for (int k = 0; k < kDgK / 16; k++)
                            umma_f16_pair(d_tmem, wdesc + (uint64_t)(k * 2), adesc + (uint64_t)(k * 2), idesc, (kb | k) ? 1u : 0u);
                        umma_commit_pair(&empty_bar[s]);
                        if (kb == kblocks - 1) umma_commit_pair(&acc_full[buf]);
                    }
                    __syncwarp();
                    if (++s == kDgStages) s = 0, phase ^= 1;
                }
            }
        }
        __syncwarp();
    } else {
        // ---------------- epilogue warps 2..9: lane quadrant = warp & 3, one weight row per thread; two warps per quadrant take its chunks of 32
        // activation rows in turn ----------------
        const int quad = warp & 3, half = (warp - 2) >> 2, r_local = quad * 32 + lane, et = threadIdx.x - 64;
        float *xchg = reinterpret_cast<float *>(smem + kDgStages * kDgStageBytes);  // [warp][buffer][activation row][lane]
        const int pair_bar = 2 + half * 2 + (quad & 1);                              // named barrier of a gate warp and its up warp
        float *x_mine = xchg + (half * 4 + quad) * 2 * kDgXRows * 32 + lane, *x_other = xchg + (half * 4 + (quad ^ 2)) * 2 * kDgXRows * 32 + lane;
        int it = 0, turn = 0;
        for (int tile = first_tile; tile < total; tile += tile_stride, it++) {
            const int buf = it & 1, use = it >> 1;
            int mt, nt, row0, live;
            locate(tile, mt, nt);
            rows_of(mt, row0, live);
            if (et == 0) {  // one thread waits and publishes the outcome, so that all epilogue warps take the same branch
                const bool ok = mbar_wait_spin(&acc_full[buf], use & 1, &abort_flag);
                if (!ok) give_up(44);
                sh_go[buf] = ok ? 1 : 0;
            }
            asm volatile("bar.sync 1, %0;" ::"n"(32 * kDgEpiWarps) : "memory");
            if (!sh_go[buf]) break;
            tc_fence_after();
            const uint32_t t_lane = tmem_base + ((uint32_t)(quad * 32) << 16) + (uint32_t)(buf * kDgCols);
            const int n = nt * NT + (int)rank * (NT / 2) + (GLU ? r_local & 63 : r_local);
            // where this thread's column lies
            const bool f32_col = !GLU && n >= p.n_main;
            O *out = reinterpret_cast<O *>(p.out) + (p.out_block ? (size_t)(n / p.out_block) * p.out_block_stride + n % p.out_block : (size_t)n);
            float *out_f32 = p.out_f32 + (n - p.n_main);  // not read without out_f32
#pragma unroll 1
            for (int c = 32 * half; c < live; c += 64) {
                float v[32];
                tmem_ld32(t_lane + c, reinterpret_cast<uint32_t *>(v));
                tmem_ld_wait();
                if constexpr (GLU) {
                    // a gate warp (quadrants 0 and 1) finishes the first 16 activation rows of the chunk, its up warp the others
                    const bool gate = quad < 2;
                    float *give = x_mine + (turn & 1) * kDgXRows * 32, *take = x_other + (turn & 1) * kDgXRows * 32;
                    turn++;
                    float mine[kDgXRows];
#pragma unroll
                    for (int i = 0; i < kDgXRows; i++) {
                        mine[i] = gate ? v[i] : v[kDgXRows + i];
                        give[i * 32] = gate ? v[kDgXRows + i] : v[i];
                    }
                    asm volatile("bar.sync %0, 64;" ::"r"(pair_bar) : "memory");
                    const int c1 = c + (gate ? 0 : kDgXRows), rows = min(kDgXRows, live - c1);
                    O o[kDgXRows];
#pragma unroll
                    for (int i = 0; i < kDgXRows; i++) {
                        const float other = take[i * 32], g = gate ? mine[i] : other, u = gate ? other : mine[i];
                        o[i] = from_f32<O>(__fdividef(g, 1.0f + __expf(-g)) * u);
                    }
                    if (n < p.N) {
                        O *dst = out + (size_t)(row0 + c1) * p.ldo;
#pragma unroll
                        for (int i = 0; i < kDgXRows; i++)
                            if (i < rows) dst[(size_t)i * p.ldo] = o[i];
                    }
                } else if (n < p.N) {
                    const int rows = min(32, live - c);
                    if (f32_col) {
                        float *dst = out_f32 + (size_t)(row0 + c) * (p.N - p.n_main);
#pragma unroll
                        for (int i = 0; i < 32; i++)
                            if (i < rows) dst[(size_t)i * (p.N - p.n_main)] = v[i];
                    } else {
                        O *dst = out + (size_t)(row0 + c) * p.ldo, o[32];
                        if (p.act_fn) {
#pragma unroll
                            for (int i = 0; i < 32; i++) v[i] = dense_act(v[i], p.act_fn);
                        }
#pragma unroll
                        for (int i = 0; i < 32; i++) o[i] = from_f32<O>(v[i]);
                        if (rows == 32) {
#pragma unroll
                            for (int i = 0; i < 32; i++) dst[(size_t)i * p.ldo] = o[i];
                        } else {
#pragma unroll
                            for (int i = 0; i < 32; i++)
                                if (i < rows) dst[(size_t)i * p.ldo] = o[i];
                        }
                    }
                }
                __syncwarp();
            }
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive_pair(map_rank(smem_u32(&acc_empty[buf]), 0));
        }
    }
    tc_fence_before();
    __syncthreads();
    cluster_sync_all();  // neither CTA leaves while the other's arrivals, copies or MMAs may still reach it
    if (warp == 1) tmem_dealloc_pair(tmem_base, 512);
}

// activation rows in expert order: one 16-byte piece per thread
__global__ void __launch_bounds__(256) gather_places_kernel(uint4 *out, const uint4 *act, const int32_t *tok_of, long long pieces, int per_row) {
    pdl_trigger();
    pdl_wait();
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= pieces) return;
    const int r = (int)(i / per_row), c = (int)(i - (long long)r * per_row);
    out[i] = act[(size_t)tok_of[r] * per_row + c];
}

bool dense_gemm_tc_supported(int dtype, const DenseGemm &g) {
    if (dtype == MYNN_F32 || !g.status || !tensor_map_api_available() || g.K % 8 || g.batch > 1 || (g.lda && g.lda != g.K) || (((uintptr_t)g.act | (uintptr_t)g.w) % 16)) return false;
    const long long wrows = (long long)g.experts * g.N * (g.glu ? 2 : 1), arows = g.route ? (long long)g.M * g.top : g.M;
    if (wrows >= (1ll << 31) || arows >= (1ll << 31) || g.row_groups * g.group_rows >= (1ll << 31)) return false;
    if (!g.route) return g.M > 32;
    if (g.gather && (!g.gather_ws || (uintptr_t)g.gather_ws % 16)) return false;
    return arows >= 16ll * g.experts && g.M > 32;  // enough rows per expert for a tile to beat passes over its weights
}

template <typename T, typename O, bool GLU>
static int launch_dg(cudaStream_t st, const CUtensorMap &ma, const CUtensorMap &mw, const DgParams &p, long long tiles_bound) {
    constexpr size_t smem = (size_t)kDgStages * kDgStageBytes + (GLU ? kDgXBytes : 0) + 1024;
    auto kern = dense_gemm_tc_kernel<T, O, GLU>;
    static SmemLimit limit;
    MYNN_CUDA_OK(limit.raise((const void *)kern, smem));
    const int pairs = sm_count() / 2;
    MYNN_CUDA_OK(launch_ex(true, 2, kern, dim3((unsigned)(2 * (tiles_bound < pairs ? tiles_bound : pairs))), dim3(kDgThreads), smem, st, ma, mw, p));
    MYNN_LAUNCH_OK("dense_gemm_tc_kernel");
    return MYNN_OK;
}

int launch_dense_gemm_tc(cudaStream_t st, int dtype, const DenseGemm &g) {
    const long long arows = g.route ? (long long)g.M * g.top : g.M, wrows = (long long)g.experts * g.N * (g.glu ? 2 : 1);
    const void *act = g.act;
    if (g.route && g.gather) {
        const int per_row = g.K / 8;
        const long long pieces = arows * per_row;
        MYNN_CUDA_OK(launch_dependent(gather_places_kernel, dim3((unsigned)((pieces + 255) / 256)), dim3(256), 0, st, (uint4 *)g.gather_ws, (const uint4 *)g.act,
                                      (const int32_t *)g.route->tok_of, pieces, per_row));
        MYNN_LAUNCH_OK("gather_places_kernel");
        act = g.gather_ws;
    }
    DgParams p = {};
    p.out = g.out;
    p.M = g.M, p.N = g.N, p.K = g.K;
    const int nt = g.glu ? kDgRows : 2 * kDgRows;
    p.n_tiles = (g.N + nt - 1) / nt;
    // Dense: one copy per stage brings a tile's rows.  Grouped: an expert's last tile may have few of its kMoeTileRows rows, so they come 32 at a time.
    p.cols = g.route ? kDgCols : pair_tile_columns(1, g.M, std::max(1, g.row_groups), p.n_tiles, sm_count() / 2);
    p.box = g.route ? 32 : p.cols / 2;
    CUtensorMap ma, mw;
    const uint64_t row_bytes = (uint64_t)g.K * 2;
    const uint64_t map_rows = g.row_groups > 1 ? (uint64_t)((g.row_groups - 1) * g.group_rows + g.M) : (uint64_t)arows;
    if (int rc = make_map(&ma, act, map_rows, row_bytes, row_bytes, (uint32_t)p.box)) return rc;
    if (int rc = make_map(&mw, g.w, (uint64_t)wrows, row_bytes, row_bytes, g.glu ? kDgRows / 2 : kDgRows)) return rc;
    p.status = g.status;
    p.n_main = g.out_f32 ? g.n_main : g.N;
    p.ldo = g.ldo ? g.ldo : p.n_main;
    p.act_fn = g.act_fn;
    p.out_block = g.out_block;
    p.out_block_stride = g.out_block_stride;
    p.out_f32 = g.out_f32;
    long long m_bound = (g.M + p.cols - 1) / p.cols;
    if (g.row_groups > 1) {
        p.groups = g.row_groups;
        p.group_tiles = (int)m_bound;
        p.group_rows = g.group_rows;
        m_bound *= g.row_groups;
    }
    if (g.route) {
        p.off = g.route->off;
        p.tile_e = g.route->tile_e;
        p.tile_row = g.route->tile_row;
        p.m_tiles_dev = g.route->n_tiles;
        m_bound = arows / kMoeTileRows + (g.experts < arows ? g.experts : arows);
    }
    // A block of rows that stays in L2 beside the weights passing through.  (The grouped products walked the weight tiles fastest: each of an
    // expert's row tiles then read all of its weights again, 4 x 0.94 GB for 4040 rows on eight experts of 2 x 7168 x 4096: 461 -> 401 us.)
    constexpr long long kBlockBytes = 48ll << 20;
    p.row_block = (int)std::max(1ll, kBlockBytes / ((long long)p.cols * g.K * 2));
    const long long bound = m_bound * p.n_tiles;
    const bool f32 = g.out_dtype == MYNN_F32;
    if (dtype == MYNN_BF16) {
        using T = __nv_bfloat16;
        if (g.glu) return f32 ? launch_dg<T, float, true>(st, ma, mw, p, bound) : launch_dg<T, T, true>(st, ma, mw, p, bound);
        return f32 ? launch_dg<T, float, false>(st, ma, mw, p, bound) : launch_dg<T, T, false>(st, ma, mw, p, bound);
    }
    using T = __half;
    if (g.glu) return f32 ? launch_dg<T, float, true>(st, ma, mw, p, bound) : launch_dg<T, T, true>(st, ma, mw, p, bound);
    return f32 ? launch_dg<T, float, false>(st, ma, mw, p, bound) : launch_dg<T, T, false>(st, ma, mw, p, bound);
}

}  // namespace mynn
