// Lean DequantMatMul for one to five activation rows (the products of a decode step of a few sequences).
//
//   out[m,n] = scale[n] * sum_k act[m,k] * wq[n,k],   M <= 5, wq [N,K] int8
//
// A matrix of 10-30 MB streams from HBM in 2-5 us, so everything that is fixed cost in the tcgen05 kernel (tensor-memory
// allocation, tensor maps, mbarrier ring, a separate limb pre-pass launch, 128-row tiles that leave SMs idle) would dominate.
// This kernel has none of it (the engine's counterpart is dequant_gemv, src/codegen/cuda/cpp/dequant_gemv.cuh:11-59: one
// warp per row, one 16-byte load in flight per lane):
//   * one CTA per SM with an equal share of the rows, so the grid is a single balanced wave.  Its rows are tiles of 16; the sixteen warps
//     deal out the contraction, so that every warp has the same piece of every row, and each lane issues all its loads (up to 320 bytes)
//     before it touches anything else and, where the weights are settled (i8_gemm.cuh), before the programmatic-dependent-launch wait: they
//     are in flight while the preceding kernel drains;
//   * the activation row(s) are the same three signed 8-bit limbs of a 23-bit fixed-point value the tensor-core kernel uses, either read
//     from the workspace, where a fused producer left them, or computed here in shared memory (no extra launch).  Three limbs of up to
//     five rows are the columns of mma.m16n8k32 (int8, exact int32 sums).  The contraction index is permuted so that each 16 bytes of a
//     lane are its fragments of two MMAs, for weights and limbs alike; a warp needs its own piece of the limbs only;
//   * the warps' int32 sums meet in shared memory once, limbs recombined in int64, the same two roundings as the tensor-core kernel:
//     the outputs are bit-identical to that kernel's, whichever of the two a shape is dispatched to.
// The legacy tensor path is enough here: 156 KB of weights per SM (gate/up of a 1B model) are 312 MMAs per eight columns, 0.3 us.  With
// dp4a instead (12 per 16 weights and row, plus a warp reduction per output) the arithmetic took longer than the loads from two
// rows on.
// Measured against it and dropped: staging the weights through shared memory with untiled bulk copies (cp.async.bulk) so that
// the next kernel's CTA fits beside this one (6.5 us against 4.3 us per launch on a 5632 x 2048 matrix), and 256-thread CTAs
// two per SM (4.7 us).
#include "common.cuh"
#include "i8_gemm.cuh"
#include "limbs.cuh"

namespace mynn {

constexpr int kLeanThreads = 512;
constexpr int kLeanMaxRows = 5;
constexpr int kLeanWarps = kLeanThreads / 32;
constexpr int kLeanTiles = 8;                       // row tiles whose partial sums are kept at a time
constexpr int kLeanFreeSms = 8;
constexpr int kLeanPitch = 16 * kLeanTiles + 4;     // int32 per (warp, column): no two lanes of a store in one bank
// Limb rows in shared memory are this far apart.  A phase of a fragment load is eight lanes, four chunks of 16 bytes in each of two rows: 32 bytes apart
// with pairs, where the second row fills the gaps, side by side without, where it takes the other half of the banks.
__host__ __device__ constexpr int lean_limb_pitch(int K, bool pairs) { return (K + 127) / 128 * 128 + (pairs ? 16 : 64); }
constexpr bool lean_phase_has_all_banks(int K, bool pairs) {
    unsigned banks = 0;  // in groups of four: the 16 bytes of a lane
    for (int row = 0; row < 2; row++)
        for (int t = 0; t < 4; t++) banks |= 1u << (row * lean_limb_pitch(K, pairs) + (pairs ? 32 : 16) * t) / 16 % 8;
    return banks == 0xffu;
}
static_assert(lean_phase_has_all_banks(1024, false) && lean_phase_has_all_banks(2064, false) && lean_phase_has_all_banks(2080, true) && lean_phase_has_all_banks(4096, true),
              "two lanes of a phase in one bank");

struct LeanParams {
    void *out;
    const void *act;        // [M,K] or null (then limbs_g / ascale_g hold the activations)
    const int8_t *wq;
    const void *scale, *resid;
    int8_t *limbs_g;        // workspace limb matrix [(3m + l)][K]; read when act == null, written by CTA 0 otherwise
    float *ascale_g;        // [M] row scales
    int N, K, act_dtype, rows_per_cta;
    int settled;            // wq and scale may be read while the kernels in front still run
};

// not ld.global.nc: weights that are not settled may have been written during the lifetime of this grid
__device__ __forceinline__ uint4 ldg_stream_16(const void *p) {
    uint4 v;
    asm volatile("ld.global.L1::no_allocate.v4.u32 {%0,%1,%2,%3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(p));
    return v;
}

__device__ __forceinline__ void ldg_stream_32(uint4 &a, uint4 &b, const void *p) {
    asm volatile("ld.global.L1::no_allocate.v8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
                 : "=r"(a.x), "=r"(a.y), "=r"(a.z), "=r"(a.w), "=r"(b.x), "=r"(b.y), "=r"(b.z), "=r"(b.w)
                 : "l"(p));
}

template <typename T>
__device__ __forceinline__ void lean_unpack(const uint4 &raw, float (&v)[8]) {
    const T *e = reinterpret_cast<const T *>(&raw);
#pragma unroll
    for (int j = 0; j < 8; j++) v[j] = to_f32<T>(e[j]);
}

// The activation rows as limbs in shared memory (and from CTA 0 in the workspace), with the arithmetic of the limb pre-pass of
// the tensor-core kernel: |a| * 2^(22-e) rounded to an integer below 2^22, split into three signed bytes.  Every CTA does this for
// itself: all rows at once, eight elements per thread and round, two barriers and no launch in between.  (The norm or the SiLU product in
// front taken inside as well cost as much as the launch it saved at one row and more at three: 10.2 us for norm and gate/up against 3.0 + 6.0.
// The SiLU product belongs behind the product that makes its operands: see GATED below.)
template <typename ActT, int M, int NB>
__device__ __forceinline__ void lean_rows_to_limbs(const LeanParams &p, int pitch, int8_t *sm_limbs, float *sm_ascale, unsigned (*sm_max)[kLeanWarps]) {
    static_assert(M <= 2, "rows of a warp's chunks");
    constexpr int ROUNDS = (M * NB * 128 + kLeanThreads - 1) / kLeanThreads;
    constexpr bool HALF = sizeof(ActT) == 2;  // 16-bit rows stay in registers between the passes
    const int per = p.K >> 3, total = M * per, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const ActT *act = reinterpret_cast<const ActT *>(p.act);
    const bool vec = (uintptr_t)act % 16 == 0;
    auto fetch = [&](int i, uint4 &raw) {  // eight 16-bit elements
        const ActT *src = act + 8 * (size_t)i;
        if (vec) {
            raw = __ldcg(reinterpret_cast<const uint4 *>(src));
        } else {
            __align__(16) ActT e[8];
#pragma unroll
            for (int j = 0; j < 8; j++) e[j] = src[j];
            raw = *reinterpret_cast<const uint4 *>(e);
        }
    };
    auto values = [&](int i, const uint4 &raw, float (&v)[8]) {
        if constexpr (HALF) {
            lean_unpack<ActT>(raw, v);
        } else {
#pragma unroll
            for (int j = 0; j < 8; j++) v[j] = to_f32<ActT>(act[8 * (size_t)i + j]);
        }
    };
    uint4 keep[ROUNDS];
#pragma unroll
    for (int k = 0; k < ROUNDS; k++) {  // all loads first
        const int i = threadIdx.x + k * kLeanThreads;
        keep[k] = make_uint4(0u, 0u, 0u, 0u);
        if (HALF && i < total) fetch(i, keep[k]);
    }
    unsigned mx[M] = {};
#pragma unroll
    for (int k = 0; k < ROUNDS; k++) {
        const int i = threadIdx.x + k * kLeanThreads;
        if (i >= total) continue;
        float v[8];
        values(i, keep[k], v);
        const unsigned top = max_bits8(v);
        if (M == 1 || i < per) mx[0] = max(mx[0], top);
        else mx[M - 1] = max(mx[M - 1], top);
    }
#pragma unroll
    for (int m = 0; m < M; m++) {
        mx[m] = __reduce_max_sync(0xffffffffu, mx[m]);
        if (lane == 0) sm_max[m][warp] = mx[m];
    }
    __syncthreads();
    float sc[M];
#pragma unroll
    for (int m = 0; m < M; m++) {
        sc[m] = limb_scale(__reduce_max_sync(0xffffffffu, sm_max[m][lane & (kLeanWarps - 1)]));
        if (threadIdx.x == m) {
            const float as = limb_unscale(sc[m]);
            sm_ascale[m] = as;
            if (blockIdx.x == 0) p.ascale_g[m] = as;
        }
    }
#pragma unroll
    for (int k = 0; k < ROUNDS; k++) {
        const int i = threadIdx.x + k * kLeanThreads, m = M > 1 && i >= per ? 1 : 0, c = i - m * per;
        if (i >= total) break;
        float v[8];
        values(i, keep[k], v);
        uint32_t l[3][2];
#pragma unroll
        for (int h = 0; h < 2; h++) limbs_of_4(v + 4 * h, M > 1 && m ? sc[M - 1] : sc[0], l[0][h], l[1][h], l[2][h]);
#pragma unroll
        for (int x = 0; x < 3; x++) {
            *reinterpret_cast<uint2 *>(sm_limbs + (size_t)(3 * m + x) * pitch + 8 * c) = make_uint2(l[x][0], l[x][1]);
            if (blockIdx.x == 0) *reinterpret_cast<uint2 *>(p.limbs_g + (size_t)(3 * m + x) * p.K + 8 * c) = make_uint2(l[x][0], l[x][1]);
        }
    }
}

__device__ __forceinline__ void mma_i8(int (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
    asm volatile("mma.sync.aligned.m16n8k32.row.col.s32.s8.s8.s32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
                 : "+r"(c[0]), "+r"(c[1]), "+r"(c[2]), "+r"(c[3])
                 : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}

// One CTA per SM owns a contiguous range of weight rows, so that the whole grid is one balanced wave.  A warp owns NB blocks of 64 along K
// (K <= 1024 NB) of all of them; TG tiles of 16 rows are in flight (2 NB TG <= 20 loads per lane, issued before anything else happens).
// K % 16 == 0; wq and limbs 16-byte aligned.  Dynamic shared memory: limbs [3 M][pitch] (ACT), partial sums [warp][3 M][kLeanPitch].
// PAIRS (rows of weights that begin on 32 bytes): a lane's chunks come in pairs, so that the four lanes of a row read a whole line of 128 bytes with one
// load; with loads of 16 bytes the two halves of a line are two requests.  Steps over 700 rows, 1 / 2 / 3 / 4 sequences: Llama-3-8B shapes 1997 -> 1861,
// 2004 -> 1875, 1916 -> 1914, 1929 -> 1922 us, TinyLlama shapes 563 -> 558, 575 -> 553, 598 -> 587, 609 -> 597.  (A choice at every load instead of a form of the
// kernel lost it at one row of TinyLlama, 573 us: code that runs once per launch; loads of 32 bytes for the limbs, too.)
// GATED: wq holds 2 N rows, N gate rows and behind them the N up rows of the same outputs, and out[m,n] = round(swish(gate) * up) of the two sums,
// each rounded first.  A tile is eight gate rows and their eight up rows, so both sums of an output lie in one column of the partial sums.
// TinyLlama shapes, us per layer at 1 / 3 rows: gate/up, SiLU product to limbs, down 3.1 + 3.1 + 2.0 / 4.8 + 3.6 + 2.8; gated, row to limbs, down
// 2.9 + 1.6 + 2.4 / 4.8 + 1.7 + 2.8.
template <typename OutT, int M, int NB, int TG, bool ACT, bool GATED, bool PAIRS>
__global__ void __launch_bounds__(kLeanThreads, 1) gemv_lean_kernel(const LeanParams p) {
    extern __shared__ __align__(16) int8_t sm_dyn[];
    __shared__ float sm_ascale[8];
    __shared__ unsigned sm_max[2][kLeanWarps];
    constexpr int C = 3 * M, NT = (C + 7) / 8;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, gq = lane >> 2, t = lane & 3;
    const int K = p.K, chunks = K >> 4, pitch = lean_limb_pitch(K, PAIRS);
    constexpr int kTileOut = GATED ? 8 : 16;  // outputs per tile of 16 rows
    const int row0 = blockIdx.x * p.rows_per_cta, rows = min(p.rows_per_cta, p.N - row0), tiles = (rows + kTileOut - 1) / kTileOut;  // in outputs
    int8_t *sm_limbs = sm_dyn;
    int *sm_sum = reinterpret_cast<int *>(sm_dyn + (ACT ? (size_t)C * pitch : 0));
    const OutT *scale_p = reinterpret_cast<const OutT *>(p.scale);
    const OutT *resid_p = reinterpret_cast<const OutT *>(p.resid);
    OutT *out_p = reinterpret_cast<OutT *>(p.out);

    // this lane's 16-byte chunks of a row
    auto chunk = [&](int j) { return warp * 4 * NB + (PAIRS ? 8 * (j / 2) + 2 * t + j % 2 : 4 * j + t); };
    uint4 w[TG][NB][2];
    auto load_tile = [&](uint4 (&x)[NB][2], int tile) {
#pragma unroll
        for (int h = 0; h < 2; h++) {
            const int row = kTileOut * tile + gq + (GATED ? 0 : 8 * h);
            const int8_t *wr = p.wq + (size_t)(row0 + (row < rows ? row : 0) + (GATED && h ? p.N : 0)) * K;
#pragma unroll
            for (int j = 0; j < NB; j += PAIRS ? 2 : 1) {
                const int c = chunk(j);
                if constexpr (PAIRS) {
                    x[j][h] = x[j + 1][h] = make_uint4(0u, 0u, 0u, 0u);
                    if (row < rows && c < chunks) ldg_stream_32(x[j][h], x[j + 1][h], wr + 16 * (size_t)c);
                } else {
                    x[j][h] = row < rows && c < chunks ? ldg_stream_16(wr + 16 * (size_t)c) : make_uint4(0u, 0u, 0u, 0u);
                }
            }
        }
    };
    // settled: the first tiles of weights and the row scale of this thread's output depend on nothing an earlier kernel writes; else the
    // weights only travel to L2 ahead of the wait
    if (!GATED && !p.settled) {
        const int8_t *w0 = p.wq + (size_t)row0 * K;
#pragma unroll 1
        for (int i = 128 * threadIdx.x; i < min(rows, 16 * TG) * K; i += 128 * kLeanThreads) prefetch_l2(w0 + i);
        pdl_wait();
    }
#pragma unroll
    for (int i = 0; i < TG; i++)
        if (i < tiles) load_tile(w[i], i);
    // outputs of the first pass: thread -> (row, activation row)
    const int pass_rows = min(rows, kTileOut * kLeanTiles), my_m = threadIdx.x / pass_rows, my_r = threadIdx.x - my_m * pass_rows;
    float wscale_first = 0.f, resv_first = 0.f;  // GATED: the gate's and the up row's scale
    if (my_m < M) wscale_first = to_f32<OutT>(scale_p[row0 + my_r]);
    if (GATED && my_m < M) resv_first = to_f32<OutT>(scale_p[p.N + row0 + my_r]);
    pdl_trigger();
    pdl_wait();
    if (!GATED && my_m < M && resid_p) resv_first = to_f32<OutT>(resid_p[(size_t)my_m * p.N + row0 + my_r]);
    // limbs of this warp's piece of K: column gq (and gq + 8) of the MMAs is limb row gq (gq + 8) = 3 m + l
    uint4 b[NT][NB];
    if constexpr (ACT) {
        if (p.act_dtype == MYNN_F32) lean_rows_to_limbs<float, M, NB>(p, pitch, sm_limbs, sm_ascale, sm_max);
        else if (p.act_dtype == MYNN_BF16) lean_rows_to_limbs<__nv_bfloat16, M, NB>(p, pitch, sm_limbs, sm_ascale, sm_max);
        else lean_rows_to_limbs<__half, M, NB>(p, pitch, sm_limbs, sm_ascale, sm_max);
        __syncthreads();
#pragma unroll
        for (int n = 0; n < NT; n++)
#pragma unroll
            for (int j = 0; j < NB; j++) {
                const int c = chunk(j), col = 8 * n + gq;
                b[n][j] = col < C && c < chunks ? *reinterpret_cast<const uint4 *>(sm_limbs + (size_t)col * pitch + 16 * c) : make_uint4(0u, 0u, 0u, 0u);
            }
    } else {
#pragma unroll
        for (int n = 0; n < NT; n++)
#pragma unroll
            for (int j = 0; j < NB; j++) {
                const int c = chunk(j), col = 8 * n + gq;
                b[n][j] = col < C && c < chunks ? __ldcg(reinterpret_cast<const uint4 *>(p.limbs_g + (size_t)col * K + 16 * (size_t)c)) : make_uint4(0u, 0u, 0u, 0u);
            }
        if (threadIdx.x < M) sm_ascale[threadIdx.x] = __ldcg(p.ascale_g + threadIdx.x);
    }

    for (int first = 0; first < tiles; first += kLeanTiles) {
        const int last = min(first + kLeanTiles, tiles);
        // kLeanTiles is not a multiple of TG: the register slot of a tile is its number modulo TG, walked slot by slot
        for (int base = first / TG * TG; base < last; base += TG) {
#pragma unroll
            for (int i = 0; i < TG; i++) {
                const int tile = base + i;
                if (tile < first || tile >= last) continue;
                int acc[NT][4];
#pragma unroll
                for (int n = 0; n < NT; n++) {
                    acc[n][0] = acc[n][1] = acc[n][2] = acc[n][3] = 0;
#pragma unroll
                    for (int j = 0; j < NB; j++) {
                        mma_i8(acc[n], w[i][j][0].x, w[i][j][1].x, w[i][j][0].y, w[i][j][1].y, b[n][j].x, b[n][j].y);
                        mma_i8(acc[n], w[i][j][0].z, w[i][j][1].z, w[i][j][0].w, w[i][j][1].w, b[n][j].z, b[n][j].w);
                    }
                }
                if (tile + TG < tiles) load_tile(w[i], tile + TG);
                // registers: (row gq, columns 2t, 2t + 1), (row gq + 8, the same columns)
                const int r = 16 * (tile - first) + gq;
#pragma unroll
                for (int n = 0; n < NT; n++)
#pragma unroll
                    for (int e = 0; e < 2; e++) {
                        const int col = 8 * n + 2 * t + e;
                        if (col < C) {
                            int *at = sm_sum + (warp * C + col) * kLeanPitch + r;
                            at[0] = acc[n][e];
                            at[8] = acc[n][2 + e];
                        }
                    }
            }
        }
        __syncthreads();
        const int beg = kTileOut * first, n_rows = min(rows, kTileOut * last) - beg;
        for (int i = threadIdx.x; i < n_rows * M; i += kLeanThreads) {
            const int m = i / n_rows, r = i - m * n_rows, row = row0 + beg + r;
            const bool known = first == 0 && i == (int)threadIdx.x;  // requested at the top of the kernel
            const float wscale = known ? wscale_first : to_f32<OutT>(scale_p[row]);
            // the sum of one row of the tiles, times both scales
            auto row_value = [&](int at, float ws) {
                int v[3] = {0, 0, 0};
#pragma unroll
                for (int x = 0; x < kLeanWarps; x++)
#pragma unroll
                    for (int l = 0; l < 3; l++) v[l] += sm_sum[(x * C + 3 * m + l) * kLeanPitch + at];
                const long long sum = (long long)v[2] * 65536 + (long long)v[1] * 256 + (long long)v[0];
                return __fmul_rn(__fmul_rn((float)sum, sm_ascale[m]), ws);
            };
            float y;
            if constexpr (GATED) {
                const float uscale = known ? resv_first : to_f32<OutT>(scale_p[p.N + row]);
                const int at = 16 * (r >> 3) + (r & 7);
                const float g = round_store<OutT>(row_value(at, wscale)), u = round_store<OutT>(row_value(at + 8, uscale));
                y = (g / (1.0f + expf(-g))) * u;
            } else {
                const float resv = known ? resv_first : resid_p ? to_f32<OutT>(resid_p[(size_t)m * p.N + row]) : 0.f;
                y = row_value(r, wscale);
                if (resid_p) y = __fadd_rn(round_store<OutT>(y), resv);
            }
            out_p[(size_t)m * p.N + row] = from_f32<OutT>(y);
        }
        if (last < tiles) __syncthreads();  // the sums are read before the next tiles' replace them
    }
}

constexpr int kLeanMaxSmem = 226 * 1024;
static size_t lean_smem(bool act, bool pairs, int M, int K) { return (act ? (size_t)3 * M * lean_limb_pitch(K, pairs) : 0) + (size_t)kLeanWarps * 3 * M * kLeanPitch * sizeof(int); }

// Up to two rows all matrices of a layer (28672 x 4096, 112 MB, as an operator at one row: 20.5 us against 23.5 us with the tcgen05 kernel and
// its pre-pass; Llama-3-8B steps of one and two sequences over 1000 rows 2356 -> 2232 and 2342 -> 2265 us).  The line at 160 MB lies above the
// largest of them.  What lies beyond are heads of large vocabularies: 128256 x 4096, 501 MB, by itself 79 against 85 us, but nothing in the
// same two steps (2229 and 2267 us), so it stays where the pre-pass and the tiles are the smaller part.
// Three to five rows fill two column tiles and the finish has that much more to do: up to 32 MB (Llama-3-8B at five rows: norm and qkv 10.4 ->
// 8.8 us), above that the tcgen05 kernel (a step of five sequences 2577 us, 3324 us with gate/up and head here; gate/up 19 and 36 us).
bool gemv_lean_supported(int M, int N, int K, const void *wq) {
    return M >= 1 && M <= kLeanMaxRows && K >= 16 && K % 16 == 0 && K <= 6144 && (size_t)N * K <= ((size_t)(M <= 2 ? 160 : 32) << 20) && ((uintptr_t)wq % 16) == 0;
}

template <typename OutT, int M, int NB, int TG, bool ACT, bool GATED, bool PAIRS>
static int launch_lean(cudaStream_t st, LeanParams p) {
    const size_t smem = lean_smem(ACT, PAIRS, M, p.K);
    auto kern = gemv_lean_kernel<OutT, M, NB, TG, ACT, GATED, PAIRS>;
    static SmemLimit limit;
    MYNN_CUDA_OK(limit.raise((const void *)kern, kLeanMaxSmem));
    static int sms = 0;
    if (sms == 0) {
        int dev = 0;
        cudaGetDevice(&dev);
        if (cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || sms <= 0) sms = 148;
    }
    // One CTA per SM, each with an equal share of the rows; a few SMs stay free, where the CTAs of the row kernel behind this one (launched
    // as its dependent) are resident by the time it ends.
    const int ctas = sms > 4 * kLeanFreeSms ? sms - kLeanFreeSms : sms;
    int rpc = (p.N + ctas - 1) / ctas;
    // Whole tiles where half of the free SMs pay for them: 11264 rows are 139 x 81, the last row of each share a tile of its own that is
    // loaded behind the others, or 141 x 80.
    const int tile = GATED ? 8 : 16, whole = rpc / tile * tile;
    if (whole > 0 && (p.N + whole - 1) / whole <= ctas + kLeanFreeSms / 2) rpc = whole;
    p.rows_per_cta = rpc;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((p.N + rpc - 1) / rpc);
    cfg.blockDim = dim3(kLeanThreads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;  // may start (and load weights) while its predecessor drains
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    MYNN_CUDA_OK(cudaLaunchKernelEx(&cfg, kern, p));
    MYNN_LAUNCH_OK("gemv_lean_kernel");
    return MYNN_OK;
}

// blocks of 64 per warp (K <= 1024 / 2048 / 4096 / 6144) and row tiles in flight
template <typename OutT, int M, bool ACT, bool GATED = false>
static int launch_by_k(cudaStream_t st, const LeanParams &p) {
    const bool pairs = p.K % 32 == 0 && (uintptr_t)p.wq % 32 == 0;
    if (p.K <= 1024) return launch_lean<OutT, M, 1, 8, ACT, GATED, false>(st, p);
    if (p.K <= 2048) return pairs ? launch_lean<OutT, M, 2, 5, ACT, GATED, true>(st, p) : launch_lean<OutT, M, 2, 5, ACT, GATED, false>(st, p);
    if (p.K <= 4096) return pairs ? launch_lean<OutT, M, 4, 2, ACT, GATED, true>(st, p) : launch_lean<OutT, M, 4, 2, ACT, GATED, false>(st, p);
    return pairs ? launch_lean<OutT, M, 6, 1, ACT, GATED, true>(st, p) : launch_lean<OutT, M, 6, 1, ACT, GATED, false>(st, p);
}
template <typename OutT>
static int launch_by_rows(cudaStream_t st, const LeanParams &p, int M) {
    switch (M) {
        case 1: return p.act ? launch_by_k<OutT, 1, true>(st, p) : launch_by_k<OutT, 1, false>(st, p);
        case 2: return p.act ? launch_by_k<OutT, 2, true>(st, p) : launch_by_k<OutT, 2, false>(st, p);
        case 3: return launch_by_k<OutT, 3, false>(st, p);
        case 4: return launch_by_k<OutT, 4, false>(st, p);
        default: return launch_by_k<OutT, 5, false>(st, p);
    }
}
template <typename OutT>
static int launch_gated_by_rows(cudaStream_t st, const LeanParams &p, int M) {
    switch (M) {
        case 1: return launch_by_k<OutT, 1, false, true>(st, p);
        case 2: return launch_by_k<OutT, 2, false, true>(st, p);
        case 3: return launch_by_k<OutT, 3, false, true>(st, p);
        case 4: return launch_by_k<OutT, 4, false, true>(st, p);
        default: return launch_by_k<OutT, 5, false, true>(st, p);
    }
}

int gemv_lean_gated_launch(cudaStream_t st, void *out, const int8_t *wq, const void *scale, int M, int F, int K, int dtype, void *workspace, size_t workspace_bytes) {
    const size_t need = i8_gemm_workspace_bytes(M, K);
    if (!workspace || workspace_bytes < need || (uintptr_t)workspace % 256)
        return fail(MYNN_E_ARG, "gated product: workspace of %zu bytes (256-byte aligned) needed", need);
    LeanParams p = {};
    p.out = out;
    p.wq = wq;
    p.scale = scale;
    p.ascale_g = (float *)((char *)workspace + 256);
    p.limbs_g = (int8_t *)workspace + 512;
    p.N = F;
    p.K = K;
    p.act_dtype = dtype;
    p.settled = 1;
    MYNN_DISPATCH_DTYPE(dtype, T, return launch_gated_by_rows<T>(st, p, M));
    return MYNN_OK;
}

// Same contract as i8_gemm_launch: `workspace` holds status word, row scales and the limb matrix; act == nullptr means a fused
// producer (or the previous call) left the limbs there.
int gemv_lean_launch(cudaStream_t st, void *out, const void *act, const int8_t *wq, const void *scale, const void *resid, int M, int N,
                     int K, int act_dtype, int out_dtype, void *workspace, size_t workspace_bytes, bool settled) {
    const size_t need = i8_gemm_workspace_bytes(M, K);
    if (!workspace || workspace_bytes < need || (uintptr_t)workspace % 256)
        return fail(MYNN_E_ARG, "dequant_matmul: workspace of %zu bytes (256-byte aligned) needed", need);
    // In a step the limbs are made by a row kernel in front, which is resident when the kernel before it ends (1.6 us; inside, a row of 2048 takes 0.5 to
    // 0.9 us more than without and a row of 5632 2.7).  Operators come one by one and make those of one or two rows inside (5632 x 2048, one row: 4.4 us
    // against 4.9; 4096 x 4096 5.4 against 5.9), of more in front (three rows of 2048: 5.0 us inside, 2.2 + 2.3 so).
    if (act && (M > 2 || settled)) {
        if (int rc = launch_act_limbs(st, act, M, K, act_dtype, (int8_t *)workspace + 512, (float *)((char *)workspace + 256))) return rc;
        act = nullptr;
    }
    LeanParams p = {};
    p.out = out;
    p.act = act;
    p.wq = wq;
    p.scale = scale;
    p.resid = resid;
    p.ascale_g = (float *)((char *)workspace + 256);
    p.limbs_g = (int8_t *)workspace + 512;
    p.N = N;
    p.K = K;
    p.act_dtype = act_dtype;
    p.settled = settled;
    if (out_dtype == MYNN_BF16) return launch_by_rows<__nv_bfloat16>(st, p, M);
    if (out_dtype == MYNN_F16) return launch_by_rows<__half>(st, p, M);
    return launch_by_rows<float>(st, p, M);
}

}  // namespace mynn
