// Prefill DequantMatMul (many activation rows) on tcgen05 kind::i8:  out[m,n] = scale[n] * sum_k act[m,k] * wq[n,k].
//
// This is a dense contraction, judged by tensor-pipe utilisation.  Like the decode kernel it never converts a weight:
// the activations are rewritten once as fixed point with a per-row power-of-two scale and split into TWO signed
// int8 limbs (15 significant bits relative to the row maximum: every bf16 element within 2^-7 of its row maximum is
// exact, the rest carry an absolute error below 2^-15 of the maximum -- finer than the bf16 rounding of the
// dequantised weights in the engine's own tensor-core prefill kernel).  The product is then an int8 GEMM with exact
// int32 accumulation, [N weight rows] x [2 x tokens] x K, and the int8 pipe runs at twice the bf16 rate, so two limbs
// cost the same tensor time as one bf16 product.
//
// Kernel: persistent pairs of CTAs (clusters of two, one CTA per SM), tile = 256 weight rows x up to 128 tokens (256 limb columns), UMMA
// cta_group::2 M=256 N<=256 K=32.  Each CTA of a pair owns 128 of the weight rows, and brings them and half of the limb rows to its
// shared memory: 32 KB per 128 of K, 64 bytes per clock at the int8 rate of 128 x 256 x 32 per 128 clocks, where a CTA on its own needs 48 KB and 96.
// An SM gets about 60 from L2 (ncu): full tiles keep the tensor pipe 95 % busy and run at the power cap, narrower ones wait for their copies (160
// columns ask for 83 bytes per clock: 57 arrive, the pipe is 69 % busy).
// 2048 rows: 28672 x 4096 325 -> 272 us (3.54 POP/s), 4096 x 14336 198 -> 166, 6144 x 4096 76 -> 69, 4096 x 4096 52 -> 48; one limb,
// 777 rows of 14336 x 4096, 48 -> 36.  About half of it came from walking the two issuing loops with whole warps (see elect_one).
// Warp 0 of both CTAs streams by TMA through a ring of six to nine mbarrier stages, warp 1 of the first issues the MMAs of both into one
// of two 256-column TMEM accumulators, warps 2-9 of both drain the other accumulator (tcgen05.ld), recombine
// the limbs, scale, add the optional residual and store -- so the epilogue of one tile overlaps the main loop of the
// next.  Tiles are walked with the token tile fastest, so concurrently running CTAs share weight tiles in L2.
// All waits are bounded and report through the workspace status word.
#include <algorithm>
#include <type_traits>

#include "common.cuh"
#include "i8_gemm.cuh"
#include "tcgen05.cuh"

namespace mynn {

MYNN_DEFINE_WAIT_BUDGET_SETTER(i8_gemm_prefill)

constexpr int kPfRows = 128;      // weight rows of one CTA of a pair (half of UMMA M)
constexpr int kPfCols = 256;      // most accumulator columns per tile (UMMA N): LIMBS columns per activation row
constexpr int kPfBlockK = 128;
constexpr int kPfMaxStages = 9;
constexpr int kPfEpiWarps = 8;    // two per TMEM lane quadrant
constexpr int kPfThreads = 64 + 32 * kPfEpiWarps;
constexpr uint32_t kPfWBytes = kPfRows * kPfBlockK;
constexpr uint32_t kPfRingBytes = 216 * 1024;  // six stages of 256 columns (32 KB in each CTA), nine of up to 128

// ---- pre-pass: rows -> two int8 limbs + power-of-two row scale ----------------------------------------------------
// limbs [(2m + l)][K]; with max |row| < 2^e the row is scaled by 2^(14-e), so |A| <= 2^14 and the high limb is within
// [-64, 64]; ascale[m] = 2^(e-14).
// One CTA of 256 threads per row (several rows are resident per SM, which hides the two block-wide reductions); VEC: 16-bit
// activations read 8 at a time (rows 16-byte aligned); the limbs are always written 8 bytes at a time (K is a multiple of 16).
constexpr int kLimbThreads = 256;

// The producers below are bound by instructions, not by memory: 2048 rows of 14336 SiLU products took 57 us for 176 MB.  So 16-bit values
// are kept two to a register wherever nothing needs them as f32: the row maximum is taken over magnitudes as 16-bit integers
// (ordered like the numbers, infinities and NaN above all of them), and the limbs are cut out of the mantissa of x * scale + 1.5 * 2^23, whose low
// bits are the rounded integer, with byte permutes: 3.5 instructions per element instead of 12.
template <typename T>
__device__ __forceinline__ uint32_t pack_pair(float lo, float hi);
template <>
__device__ __forceinline__ uint32_t pack_pair<__nv_bfloat16>(float lo, float hi) {
    const __nv_bfloat162 v = __floats2bfloat162_rn(lo, hi);
    return reinterpret_cast<const uint32_t &>(v);
}
template <>
__device__ __forceinline__ uint32_t pack_pair<__half>(float lo, float hi) {
    const __half2 v = __floats2half2_rn(lo, hi);
    return reinterpret_cast<const uint32_t &>(v);
}
template <typename T>
__device__ __forceinline__ void unpack8(const uint4 &raw, float (&v)[8]) {
    const T *e = reinterpret_cast<const T *>(&raw);
#pragma unroll
    for (int i = 0; i < 8; i++) v[i] = to_f32<T>(e[i]);
}
// larger magnitudes of both halves
__device__ __forceinline__ uint32_t max_abs2(uint32_t m, uint32_t pair) {
    uint32_t r;
    asm("max.u16x2 %0, %1, %2;" : "=r"(r) : "r"(m), "r"(pair & 0x7fff7fffu));
    return r;
}
__device__ __forceinline__ uint32_t max_abs8(uint32_t m, const uint4 &raw) { return max_abs2(max_abs2(max_abs2(max_abs2(m, raw.x), raw.y), raw.z), raw.w); }
// largest magnitude that has a scale: 3.0e38 in bf16, every finite f16
template <typename T>
constexpr uint32_t kMagnitudeLimit = std::is_same<T, __nv_bfloat16>::value ? 0x7f61u : 0x7bffu;

// Row maximum (two magnitudes per thread) -> scale of the limbs, 0 for a row that holds something non-finite; writes the row scale.
template <typename T>
__device__ __forceinline__ float limb2_scale(uint32_t mx, float *ascale_m, uint32_t *red /* kLimbThreads / 32 */) {
    mx = __reduce_max_sync(0xffffffffu, max(mx & 0xffffu, mx >> 16));
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = mx;
    __syncthreads();
#pragma unroll
    for (int i = 0; i < kLimbThreads / 32; i++) mx = max(mx, red[i]);
    const unsigned short bits = (unsigned short)mx;
    const float t = to_f32<T>(reinterpret_cast<const T &>(bits));
    const bool bad = mx > kMagnitudeLimit<T>;
    int e = 0;
    if (t > 0.f && !bad) frexpf(t, &e);
    const float sc = t > 0.f && !bad ? ldexpf(1.0f, 14 - e) : 1.0f;
    if (threadIdx.x == 0) *ascale_m = bad ? __int_as_float(0x7fc00000) : 1.0f / sc;
    return bad ? 0.f : sc;
}

// A row in shared memory in its storage type -> both limb rows (K % 8 == 0).
template <typename T>
__device__ __forceinline__ void smem_row_to_limbs2(const T *row_s, int K, int8_t *limb_row0, float sc) {
    uint2 *l0 = reinterpret_cast<uint2 *>(limb_row0);
    uint2 *l1 = reinterpret_cast<uint2 *>(limb_row0 + K);
    for (int gi = threadIdx.x; gi < (K >> 3); gi += kLimbThreads) {
        float x[8];
        unpack8<T>(reinterpret_cast<const uint4 *>(row_s)[gi], x);
        uint32_t w0[2] = {0u, 0u}, w1[2] = {0u, 0u};
        if (sc != 0.f) {
#pragma unroll
            for (int h = 0; h < 2; h++) {
                uint32_t a[4], r[4];  // A in the low 16 bits; the high limb of A, rounded to the nearest, is byte 1 of A + 128
#pragma unroll
                for (int i = 0; i < 4; i++) {
                    a[i] = __float_as_uint(fmaf(x[4 * h + i], sc, 12582912.0f));
                    r[i] = a[i] + 128u;
                }
                w0[h] = __byte_perm(__byte_perm(a[0], a[1], 0x0040u), __byte_perm(a[2], a[3], 0x0040u), 0x5410u);
                w1[h] = __byte_perm(__byte_perm(r[0], r[1], 0x0051u), __byte_perm(r[2], r[3], 0x0051u), 0x5410u);
            }
        }
        l0[gi] = make_uint2(w0[0], w0[1]);
        l1[gi] = make_uint2(w1[0], w1[1]);
    }
}

template <typename T, bool VEC>
__global__ void __launch_bounds__(kLimbThreads) act_to_limbs2_kernel(int8_t *limbs, float *ascale, const T *act, int K) {
    extern __shared__ __align__(16) uint8_t row_raw[];
    T *row_s = reinterpret_cast<T *>(row_raw);
    __shared__ uint32_t red[kLimbThreads / 32];
    pdl_trigger();
    pdl_wait();
    const int m = blockIdx.x;
    const T *src = act + (size_t)m * K;
    uint32_t mx = 0u;
    if constexpr (VEC) {
        for (int i = 8 * threadIdx.x; i < K; i += 8 * kLimbThreads) {
            const uint4 raw = *reinterpret_cast<const uint4 *>(src + i);
            *reinterpret_cast<uint4 *>(row_s + i) = raw;
            mx = max_abs8(mx, raw);
        }
    } else {
        for (int i = threadIdx.x; i < K; i += kLimbThreads) {
            const T v = src[i];
            row_s[i] = v;
            mx = max_abs2(mx, reinterpret_cast<const unsigned short &>(v));
        }
    }
    const float sc = limb2_scale<T>(mx, ascale + m, red);  // its barrier also publishes row_s
    smem_row_to_limbs2<T>(row_s, K, limbs + (size_t)(2 * m) * K, sc);
}

// ---- fused producers: the operator that makes a DequantMatMul's activations writes the two limbs itself -------------------
// (the prefill counterpart of rms_norm_limbs_kernel / swiglu_limbs_kernel of the decode step: no activation tensor is written
// and read back, and no separate pre-pass runs).  One CTA of 256 threads per row; D, F multiples of 8, rows 16-byte aligned.

// y = round(x * rsqrt(mean x^2 + eps) * w) -> two limbs per element; with `add` first x = round(x + add), stored back (a pass over
// the rows less than an addition of its own: 9.7 + 13.5 us for 2048 rows of 4096)
template <typename T>
__global__ void __launch_bounds__(kLimbThreads)
rms_norm_limbs2_kernel(int8_t *limbs, float *ascale, T *x, const T *add, const T *w, float eps, int D) {
    extern __shared__ __align__(16) uint8_t row_raw[];
    T *row_s = reinterpret_cast<T *>(row_raw);
    __shared__ float red[kLimbThreads / 32];
    __shared__ uint32_t red_m[kLimbThreads / 32];
    pdl_trigger();
    pdl_wait();
    const int m = blockIdx.x;
    const size_t base = (size_t)m * D;
    float ss = 0.f;
    for (int i = 8 * threadIdx.x; i < D; i += 8 * kLimbThreads) {
        uint4 raw = *reinterpret_cast<const uint4 *>(x + base + i);
        float v[8];
        unpack8<T>(raw, v);
        if (add != nullptr) {
            float a[8];
            unpack8<T>(*reinterpret_cast<const uint4 *>(add + base + i), a);
#pragma unroll
            for (int j = 0; j < 8; j++) v[j] += a[j];
            raw = make_uint4(pack_pair<T>(v[0], v[1]), pack_pair<T>(v[2], v[3]), pack_pair<T>(v[4], v[5]), pack_pair<T>(v[6], v[7]));
            unpack8<T>(raw, v);
            *reinterpret_cast<uint4 *>(x + base + i) = raw;
        }
        *reinterpret_cast<uint4 *>(row_s + i) = raw;
#pragma unroll
        for (int j = 0; j < 8; j++) ss += v[j] * v[j];
    }
    ss = warp_sum(ss);
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = ss;
    __syncthreads();
    float tot = 0.f;
#pragma unroll
    for (int i = 0; i < kLimbThreads / 32; i++) tot += red[i];
    const float inv = 1.0f / sqrtf(tot / (float)D + eps);
    uint32_t mx = 0u;
    for (int i = 8 * threadIdx.x; i < D; i += 8 * kLimbThreads) {  // each thread revisits the elements it wrote
        float xv[8], wv[8];
        unpack8<T>(*reinterpret_cast<const uint4 *>(row_s + i), xv);
        unpack8<T>(*reinterpret_cast<const uint4 *>(w + i), wv);
#pragma unroll
        for (int j = 0; j < 8; j++) xv[j] = xv[j] * inv * wv[j];
        const uint4 y = make_uint4(pack_pair<T>(xv[0], xv[1]), pack_pair<T>(xv[2], xv[3]), pack_pair<T>(xv[4], xv[5]), pack_pair<T>(xv[6], xv[7]));
        mx = max_abs8(mx, y);
        *reinterpret_cast<uint4 *>(row_s + i) = y;
    }
    const float sc = limb2_scale<T>(mx, ascale + m, red_m);  // its barrier also publishes row_s
    smem_row_to_limbs2<T>(row_s, D, limbs + (size_t)(2 * m) * D, sc);
}

// h = round(swish(gate) * up) -> two limbs per element; gate / up rows are in_stride elements apart
template <typename T>
__global__ void __launch_bounds__(kLimbThreads)
swiglu_limbs2_kernel(int8_t *limbs, float *ascale, const T *gate, const T *up, int F, long long in_stride) {
    extern __shared__ __align__(16) uint8_t row_raw[];
    T *row_s = reinterpret_cast<T *>(row_raw);
    __shared__ uint32_t red[kLimbThreads / 32];
    pdl_trigger();
    pdl_wait();
    const int m = blockIdx.x;
    uint32_t mx = 0u;
    for (int i = 8 * threadIdx.x; i < F; i += 8 * kLimbThreads) {
        float g[8], u[8];
        unpack8<T>(*reinterpret_cast<const uint4 *>(gate + (size_t)m * in_stride + i), g);
        unpack8<T>(*reinterpret_cast<const uint4 *>(up + (size_t)m * in_stride + i), u);
#pragma unroll
        for (int j = 0; j < 8; j++) g[j] = (g[j] / (1.0f + expf(-g[j]))) * u[j];
        const uint4 h = make_uint4(pack_pair<T>(g[0], g[1]), pack_pair<T>(g[2], g[3]), pack_pair<T>(g[4], g[5]), pack_pair<T>(g[6], g[7]));
        mx = max_abs8(mx, h);
        *reinterpret_cast<uint4 *>(row_s + i) = h;
    }
    const float sc = limb2_scale<T>(mx, ascale + m, red);
    smem_row_to_limbs2<T>(row_s, F, limbs + (size_t)(2 * m) * F, sc);
}

struct PfParams {
    void *out;
    const void *scale, *resid;
    const float *ascale;    // f32 row scales (DequantMatMul pre-pass), or null when ascale_t is used
    const void *ascale_t;   // QuantizedMatMul: lhs scales in the output dtype, element m * ascale_stride
    int ascale_stride;      // 1 = one scale per row, 0 = one scale for the whole tensor
    int M, N, K;
    int stages;           // of the ring
    int cols;             // accumulator columns per tile, a multiple of 32
    int w_tiles, t_tiles, t_full;  // weight tiles (of a pair), token tiles, token tiles that have all their rows
    int *status;
};

// Tiles in the order they are walked: the full ones with the token tile fastest, behind them the ragged ones of the last token tile, so
// that a CTA's share of either kind is the same however the grid's size and the number of token tiles divide one another.
__device__ __forceinline__ void pf_place(const PfParams &p, int tile, int &wt, int &tt) {
    const int full = p.w_tiles * p.t_full;
    if (tile < full) {
        wt = tile / p.t_full;
        tt = tile - wt * p.t_full;
    } else {
        wt = tile - full;
        tt = p.t_full;
    }
}

// min(#SMs / 2, #tiles) persistent pairs of CTAs that walk the tiles with stride gridDim.x / 2.
// LIMBS = 2: DequantMatMul, limb rows (2m + l), up to 128 activation rows per tile.
// LIMBS = 1: QuantizedMatMul (W8A8), the int8 lhs matrix itself is the operand, up to 256 activation rows per tile.
template <typename OutT, int LIMBS>
__global__ void __launch_bounds__(kPfThreads, 1)
i8_prefill_gemm_kernel(const __grid_constant__ CUtensorMap map_w, const __grid_constant__ CUtensorMap map_a, const PfParams p) {
    extern __shared__ uint8_t smem_raw[];
    uint8_t *smem = (uint8_t *)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
    __shared__ uint64_t full_bar[kPfMaxStages], empty_bar[kPfMaxStages], acc_full[2], acc_empty[2];
    __shared__ uint32_t tmem_slot;
    __shared__ int abort_flag;
    __shared__ __align__(16) float sh_ascale[2][kPfCols / LIMBS];
    __shared__ int sh_go[2];

    const int warp = __shfl_sync(0xffffffffu, (int)threadIdx.x >> 5, 0), lane = threadIdx.x & 31;
    const uint32_t rank = cluster_ctarank();
    const int first_tile = blockIdx.x >> 1, tile_stride = gridDim.x >> 1;
    const int n_tiles = p.w_tiles * p.t_tiles, tok = p.cols / LIMBS;  // tok: activation rows per tile
    // N of a tile's MMA = the accumulator columns the tile really has (rows past M are zero-filled by TMA and need no tensor time), rounded
    // up to the instruction's granularity of 32; the first CTA holds the first half of them as B's rows, the second the other
    const uint32_t stage_bytes = kPfWBytes + (uint32_t)p.cols * (kPfBlockK / 2);
    auto tile_cols = [&](int tt) { return min(p.cols, (((p.M - tt * tok) * LIMBS + 31) >> 5) << 5); };
    const int kblocks = (p.K + kPfBlockK - 1) / kPfBlockK;

    if (threadIdx.x == 0) {
        for (int s = 0; s < p.stages; s++) {
            mbar_init(&full_bar[s], 1);
            mbar_init(&empty_bar[s], 1);
        }
        for (int b = 0; b < 2; b++) {
            mbar_init(&acc_full[b], 1);
            mbar_init(&acc_empty[b], 2 * kPfEpiWarps);  // one arrival per epilogue warp of both CTAs (used in the first CTA)
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
    pdl_wait();  // limbs and row scales come from the pre-pass

    if (warp == 0) {
        // ---------------- TMA producer ----------------
        if (elect_one()) {
            asm volatile("prefetch.tensormap [%0];" ::"l"(&map_w) : "memory");
            asm volatile("prefetch.tensormap [%0];" ::"l"(&map_a) : "memory");
        }
        int s = 0, use = 0;
        bool ok = true;
        for (int tile = first_tile; tile < n_tiles && ok; tile += tile_stride) {
            int wt, tt;
            pf_place(p, tile, wt, tt);
            const int w_row = (2 * wt + (int)rank) * kPfRows, a_row = tt * p.cols + (int)rank * (tile_cols(tt) >> 1);
            for (int kb = 0; kb < kblocks; kb++) {
                if (use > 0 && !__all_sync(0xffffffffu, mbar_wait_spin(&empty_bar[s], (use - 1) & 1, &abort_flag))) {
                    ok = false;
                    break;
                }
                uint8_t *st = smem + s * stage_bytes;
                const uint32_t bar = map_rank(smem_u32(&full_bar[s]), 0);
                if (elect_one()) {
                    if (rank == 0) mbar_expect_tx(&full_bar[s], 2 * stage_bytes);  // what both CTAs bring into a stage
                    tma_load_2d_pair(st, &map_w, kb * kPfBlockK, w_row, bar);
                    tma_load_2d_pair(st + kPfWBytes, &map_a, kb * kPfBlockK, a_row, bar);
                }
                __syncwarp();
                if (++s == p.stages) s = 0, use++;
            }
        }
        // The commits that give the last stages back arrive in both CTAs: neither is left before its own have.
        for (int i = 0; i < p.stages && ok; i++) {
            if (use > 0) ok = __all_sync(0xffffffffu, mbar_wait_spin(&empty_bar[s], (use - 1) & 1, &abort_flag));
            if (++s == p.stages) s = 0, use++;
        }
        if (!ok && lane == 0) {
            atomicExch(&abort_flag, 1);
            atomicExch(p.status, 11);
        }
        __syncwarp();
    } else if (warp == 1) {
        // ---------------- MMA issuer of the pair ----------------
        if (rank == 0) {
            int s = 0, phase = 0, it = 0;
            bool ok = true;
            for (int tile = first_tile; tile < n_tiles && ok; tile += tile_stride, it++) {
                const int buf = it & 1, use = it >> 1;
                int wt_, tt_;
                pf_place(p, tile, wt_, tt_);
                const int cols = tile_cols(tt_);
                const uint32_t idesc = (2u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(cols >> 3) << 17) | ((uint32_t)(2 * kPfRows >> 4) << 24);
                if (use > 0 && !__all_sync(0xffffffffu, mbar_wait_spin(&acc_empty[buf], (use - 1) & 1, &abort_flag))) {  // epilogue has drained it
                    if (lane == 0) {
                        atomicExch(&abort_flag, 1);
                        atomicExch(p.status, 12);
                    }
                    break;
                }
                tc_fence_after();
                const uint32_t d_tmem = tmem_base + (uint32_t)(buf * kPfCols);
                for (int kb = 0; kb < kblocks; kb++) {
                    if (!__all_sync(0xffffffffu, mbar_wait_spin(&full_bar[s], phase, &abort_flag))) {
                        if (lane == 0) {
                            atomicExch(&abort_flag, 1);
                            atomicExch(p.status, 13);
                        }
                        ok = false;
                        break;
                    }
                    tc_fence_after();
                    const uint32_t a_addr = smem_u32(smem + s * stage_bytes);
                    const uint64_t adesc = make_kmajor_sw128_desc(a_addr), bdesc = make_kmajor_sw128_desc(a_addr + kPfWBytes);
                    if (elect_one()) {
#pragma unroll
                        for (int k = 0; k < kPfBlockK / 32; k++)
                            umma_i8_pair(d_tmem, adesc + (uint64_t)(k * 2), bdesc + (uint64_t)(k * 2), idesc, (kb | k) ? 1u : 0u);
                        umma_commit_pair(&empty_bar[s]);
                        if (kb == kblocks - 1) umma_commit_pair(&acc_full[buf]);
                    }
                    __syncwarp();
                    if (++s == p.stages) s = 0, phase ^= 1;
                }
            }
        }
        __syncwarp();
    } else {
        // ---------------- epilogue warps 2..9: TMEM lane quadrant = warp & 3, one weight row per thread ----------------
        // The epilogue has to keep up with the main loop, an output per thread every 45 ns (LIMBS = 2, K = 4096).  One output after the
        // other (row scale from shared memory, 64-bit conversion, two products, rounding, store) took 100 ns and set the pace of
        // every shape with K up to 4096.  So two warps share a quadrant and take its chunks of 32 columns in turn, and a chunk goes
        // through each stage as a whole: all scales, all values, then all stores (a store through the generic `out` pointer holds back
        // every load behind it).
        const int quad = warp & 3, half = (warp - 2) >> 2, r_local = quad * 32 + lane, et = threadIdx.x - 64;
        const OutT *scale_p = reinterpret_cast<const OutT *>(p.scale);
        const OutT *resid_p = reinterpret_cast<const OutT *>(p.resid);
        OutT *out_p = reinterpret_cast<OutT *>(p.out);
        int it = 0;
        for (int tile = first_tile; tile < n_tiles; tile += tile_stride, it++) {
            int wt, tt;
            pf_place(p, tile, wt, tt);
            const int buf = it & 1, use = it >> 1;
            const int n = (2 * wt + (int)rank) * kPfRows + r_local, tok0 = tt * tok, live = min(tok, p.M - tok0);
            const float wscale = n < p.N ? to_f32<OutT>(scale_p[n]) : 0.f;
            for (int i = et; i < tok; i += 32 * kPfEpiWarps) {
                float a = 0.f;
                if (i < live)
                    a = p.ascale ? p.ascale[tok0 + i]
                                 : to_f32<OutT>(reinterpret_cast<const OutT *>(p.ascale_t)[(size_t)(tok0 + i) * p.ascale_stride]);
                sh_ascale[buf][i] = a;
            }
            constexpr int R = 32 / LIMBS;  // activation rows per chunk
            // `out` may alias `resid` (x += ...): the residuals of a warp's next chunk are loaded in front of this one's stores
            float res[R];
            auto load_res = [&](int r0, float (&dst)[R]) {
                if (LIMBS == 2 && resid_p && n < p.N) {
#pragma unroll
                    for (int j = 0; j < R; j++) dst[j] = r0 + j < live ? to_f32<OutT>(resid_p[(size_t)(tok0 + r0 + j) * p.N + n]) : 0.f;
                }
            };
            load_res(half * R, res);
            // one thread waits for the accumulator and publishes the outcome, so that all epilogue warps take the same
            // branch (a warp leaving alone would strand the others at the named barrier)
            if (et == 0) {
                const bool ok = mbar_wait_spin(&acc_full[buf], use & 1, &abort_flag);
                if (!ok) {
                    atomicExch(&abort_flag, 1);
                    atomicExch(p.status, 14);
                }
                sh_go[buf] = ok ? 1 : 0;
            }
            asm volatile("bar.sync 1, %0;" ::"n"(32 * kPfEpiWarps) : "memory");  // the epilogue warps: sh_ascale[buf], sh_go[buf] are set
            if (!sh_go[buf]) break;
            tc_fence_after();
#pragma unroll 1
            for (int r0 = half * R; r0 < live; r0 += 2 * R) {
                uint32_t v[32];
                tmem_ld32(tmem_base + ((uint32_t)(quad * 32) << 16) + (uint32_t)(buf * kPfCols + r0 * LIMBS), v);
                float as[R], y[R], nres[R];
#pragma unroll
                for (int j = 0; j < R; j += 4) {
                    const float4 a4 = *reinterpret_cast<const float4 *>(&sh_ascale[buf][r0 + j]);
                    as[j] = a4.x, as[j + 1] = a4.y, as[j + 2] = a4.z, as[j + 3] = a4.w;
                }
                load_res(r0 + 2 * R, nres);
                tmem_ld_wait();
                if constexpr (LIMBS == 2) {
                    // 256 high + low: in 32 bits wherever every high limb sum of the chunk is below 2^22 (the low ones are below 2^30), the
                    // same number
                    unsigned wide = 0u;
#pragma unroll
                    for (int j = 0; j < R; j++) wide |= (v[2 * j + 1] + (1u << 22)) >> 23;
                    if (!__any_sync(0xffffffffu, wide)) {
#pragma unroll
                        for (int j = 0; j < R; j++) y[j] = (float)((int)v[2 * j + 1] * 256 + (int)v[2 * j]);
                    } else {
#pragma unroll
                        for (int j = 0; j < R; j++) y[j] = (float)((long long)(int)v[2 * j + 1] * 256 + (long long)(int)v[2 * j]);
                    }
                } else {
#pragma unroll
                    for (int j = 0; j < R; j++) y[j] = (float)(int)v[j];
                }
                OutT o[R];
#pragma unroll
                for (int j = 0; j < R; j++) {
                    // (acc * lhs scale) * weight scale with separate roundings, as the CPU kernels compute it
                    float r = __fmul_rn(__fmul_rn(y[j], as[j]), wscale);
                    if (LIMBS == 2 && resid_p) r = __fadd_rn(round_store<OutT>(r), res[j]);
                    o[j] = from_f32<OutT>(r);
                }
                if (n < p.N) {
                    OutT *dst = out_p + (size_t)(tok0 + r0) * p.N + n;
                    if (r0 + R <= live) {
#pragma unroll
                        for (int j = 0; j < R; j++) dst[(size_t)j * p.N] = o[j];
                    } else {
#pragma unroll
                        for (int j = 0; j < R; j++)
                            if (r0 + j < live) dst[(size_t)j * p.N] = o[j];
                    }
                }
#pragma unroll
                for (int j = 0; j < R; j++) res[j] = nres[j];
            }
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive_pair(map_rank(smem_u32(&acc_empty[buf]), 0));  // this warp has drained its share of the accumulator
        }
    }

    tc_fence_before();
    __syncthreads();
    cluster_sync_all();  // neither CTA leaves while the other's arrivals, copies or MMAs may still reach it
    if (warp == 1) tmem_dealloc_pair(tmem_base, 512);
}

// ---- host side ---------------------------------------------------------------------------------------------------
static size_t pf_scale_bytes(int M) { return ((size_t)M * sizeof(float) + 255) / 256 * 256; }

size_t i8_prefill_workspace_bytes(int M, int K) {
    if (M <= 0 || K <= 0) return 0;
    return 256 + pf_scale_bytes(M) + ((size_t)2 * M * K + 255) / 256 * 256;
}

bool i8_prefill_supported(int M, int N, int K, const void *wq, int act_dtype, int out_dtype) {
    (void)out_dtype;
    // two limbs carry 15 bits: right for 16-bit activations, not for f32 graphs (those keep the f32-accurate kernels)
    return act_dtype != MYNN_F32 && M > kI8MaxRows && N >= 1 && K >= 16 && K % 16 == 0 && (size_t)K * 4 <= 200 * 1024 && ((uintptr_t)wq % 16) == 0 &&
           tensor_map_api_available();
}

int sm_count() {
    int dev = 0, sms = 148;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    return sms;
}

// The width whose slowest pair has the least to do.  A stage brings 128 weight rows and half of the columns into each SM at about 64 bytes per
// clock, so a tile costs its columns plus 256 (the tensor core, at two clocks per column, is not slower up to 256 columns); full tiles are
// dealt out first, ragged ones behind them.
int pair_tile_columns(int limbs, int M, int groups, int w_tiles, int pairs) {
    int best = kPfCols;
    long long best_cost = -1;
    for (int cols = kPfCols; cols >= 96; cols -= 32) {
        const int tok = cols / limbs, full_t = M / tok, rest = M - full_t * tok;
        const long long full = (long long)w_tiles * groups * full_t, all = full + (rest ? (long long)w_tiles * groups : 0), r = full % pairs;
        const int unit = cols + 256, rest_unit = (rest * limbs + 31) / 32 * 32 + 256;
        const long long f0 = (full + pairs - 1) / pairs, c0 = f0 * unit + ((all + pairs - 1) / pairs - f0) * rest_unit;  // the first pair
        const long long f1 = full / pairs, c1 = f1 * unit + (all > r ? (all - r + pairs - 1) / pairs - f1 : 0) * rest_unit;  // the first with one full tile less
        const long long cost = c0 > c1 ? c0 : c1;
        if (best_cost < 0 || cost < best_cost) best_cost = cost, best = cols;
    }
    return best;
}
static void pf_tiles(PfParams &p, int limbs) {
    p.w_tiles = (p.N + 2 * kPfRows - 1) / (2 * kPfRows);
    p.cols = pair_tile_columns(limbs, p.M, 1, p.w_tiles, sm_count() / 2);
    const int tok = p.cols / limbs;
    p.stages = std::min<int>(kPfMaxStages, kPfRingBytes / (kPfWBytes + p.cols * (kPfBlockK / 2)));
    p.t_full = p.M / tok;
    p.t_tiles = (p.M + tok - 1) / tok;
}

template <typename OutT, int LIMBS>
static int launch_pf(cudaStream_t st, const CUtensorMap &mw, const CUtensorMap &ma, const PfParams &p) {
    const size_t smem = (size_t)kPfRingBytes + 1024;
    auto kern = i8_prefill_gemm_kernel<OutT, LIMBS>;
    static SmemLimit limit;
    MYNN_CUDA_OK(limit.raise((const void *)kern, smem));
    const int tiles = p.w_tiles * p.t_tiles, pairs = sm_count() / 2;
    MYNN_CUDA_OK(launch_ex(true, 2, kern, dim3(2 * (tiles < pairs ? tiles : pairs)), dim3(kPfThreads), smem, st, mw, ma, p));
    MYNN_LAUNCH_OK("i8_prefill_gemm_kernel");
    return MYNN_OK;
}

int i8_prefill_launch(cudaStream_t st, void *out, const void *act, const int8_t *wq, const void *scale, const void *resid,
                      int M, int N, int K, int act_dtype, int out_dtype, void *workspace, size_t workspace_bytes) {
    const size_t need = i8_prefill_workspace_bytes(M, K);
    if (!workspace || workspace_bytes < need)
        return fail(MYNN_E_ARG, "dequant_matmul: workspace of %zu bytes needed, %zu given", need, workspace ? workspace_bytes : (size_t)0);
    if ((uintptr_t)workspace % 256) return fail(MYNN_E_ARG, "dequant_matmul: workspace must be 256-byte aligned");
    int *status = (int *)workspace;
    float *ascale = (float *)((char *)workspace + 256);
    int8_t *limbs = (int8_t *)workspace + 256 + pf_scale_bytes(M);
    const size_t smem = (size_t)K * 2;
    if (act != nullptr) {  // act == nullptr: a fused producer has left limbs and row scales in the workspace
    const bool vec = K % 8 == 0 && ((uintptr_t)act % 16) == 0;
#define PREP(T)                                                                                                          \
    {                                                                                                                    \
        auto kern = vec ? act_to_limbs2_kernel<T, true> : act_to_limbs2_kernel<T, false>;                      \
        if (smem > 48 * 1024) MYNN_CUDA_OK(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem)); \
        MYNN_CUDA_OK(launch_dependent(kern, dim3(M), dim3(kLimbThreads), smem, st, limbs, ascale, (const T *)act, K));         \
    }
    switch (act_dtype) {
        case MYNN_BF16: PREP(__nv_bfloat16) break;
        case MYNN_F16: PREP(__half) break;
        default: return fail(MYNN_E_ARG, "dequant_matmul: bad activation dtype %d", act_dtype);
    }
#undef PREP
    MYNN_LAUNCH_OK("act_to_limbs2_kernel");
    }
    PfParams p;
    p.out = out;
    p.scale = scale;
    p.resid = resid;
    p.ascale = ascale;
    p.ascale_t = nullptr;
    p.ascale_stride = 1;
    p.M = M;
    p.N = N;
    p.K = K;
    p.status = status;
    pf_tiles(p, 2);
    CUtensorMap mw, ma;
    int rc = make_map(&mw, wq, (uint64_t)N, (uint64_t)K, (uint64_t)K, kPfRows);
    if (rc) return rc;
    rc = make_map(&ma, limbs, (uint64_t)2 * M, (uint64_t)K, (uint64_t)K, (uint32_t)p.cols / 2);
    if (rc) return rc;
    if (out_dtype == MYNN_BF16) return launch_pf<__nv_bfloat16, 2>(st, mw, ma, p);
    if (out_dtype == MYNN_F16) return launch_pf<__half, 2>(st, mw, ma, p);
    return launch_pf<float, 2>(st, mw, ma, p);
}

// QuantizedMatMul (W8A8): out[m,n] = (sum_k lhs[m,k] * rhs[n,k]) * lhs_scale[m] * rhs_scale[n].  The int8 lhs matrix is
// the TMA source as it is (no pre-pass, one accumulator column per row), so the int8 pipe does a quarter of the work
// per output that a bf16 product would need.  workspace: 256 bytes (status word), zeroed once.
// Fused producers of the prefill DequantMatMul (rows > 32): limbs and row scales go to the layout i8_prefill_launch reads.
static int pf_fused_ws(void *workspace, size_t workspace_bytes, int rows, int K, int8_t **limbs, float **ascale) {
    const size_t need = i8_prefill_workspace_bytes(rows, K);
    if (!workspace || workspace_bytes < need)
        return fail(MYNN_E_ARG, "fused limb producer: workspace of %zu bytes needed, %zu given", need, workspace ? workspace_bytes : (size_t)0);
    if ((uintptr_t)workspace % 256) return fail(MYNN_E_ARG, "fused limb producer: workspace must be 256-byte aligned");
    *ascale = (float *)((char *)workspace + 256);
    *limbs = (int8_t *)workspace + 256 + pf_scale_bytes(rows);
    return MYNN_OK;
}

bool prefill_fused_supported(int dtype, int K, const void *a, const void *b) {
    return dtype != MYNN_F32 && K % 16 == 0 && (size_t)K * 4 <= 200 * 1024 && (((uintptr_t)a | (uintptr_t)b) % 16) == 0;
}

int launch_rms_norm_limbs2(cudaStream_t st, int dtype, void *workspace, size_t workspace_bytes, void *x, const void *add, const void *w, float eps,
                           int rows, int D) {
    int8_t *limbs;
    float *ascale;
    if (int rc = pf_fused_ws(workspace, workspace_bytes, rows, D, &limbs, &ascale)) return rc;
    const size_t smem = (size_t)D * 2;
#define RUN(T)                                                                                                                \
    {                                                                                                                         \
        auto kern = rms_norm_limbs2_kernel<T>;                                                                                \
        if (smem > 48 * 1024) MYNN_CUDA_OK(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem)); \
        MYNN_CUDA_OK(launch_dependent(kern, dim3(rows), dim3(kLimbThreads), smem, st, limbs, ascale, (T *)x, (const T *)add, (const T *)w, eps, D)); \
    }
    if (dtype == MYNN_BF16) RUN(__nv_bfloat16) else if (dtype == MYNN_F16) RUN(__half) else return fail(MYNN_E_ARG, "rms_norm_limbs2: bad dtype %d", dtype);
#undef RUN
    MYNN_LAUNCH_OK("rms_norm_limbs2_kernel");
    return MYNN_OK;
}

int launch_swiglu_limbs2(cudaStream_t st, int dtype, void *workspace, size_t workspace_bytes, const void *gate, const void *up, int rows,
                         int F, long long in_stride) {
    int8_t *limbs;
    float *ascale;
    if (int rc = pf_fused_ws(workspace, workspace_bytes, rows, F, &limbs, &ascale)) return rc;
    const size_t smem = (size_t)F * 2;
#define RUN(T)                                                                                                                \
    {                                                                                                                         \
        auto kern = swiglu_limbs2_kernel<T>;                                                                                  \
        if (smem > 48 * 1024) MYNN_CUDA_OK(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem)); \
        MYNN_CUDA_OK(launch_dependent(kern, dim3(rows), dim3(kLimbThreads), smem, st, limbs, ascale, (const T *)gate, (const T *)up, F, in_stride)); \
    }
    if (dtype == MYNN_BF16) RUN(__nv_bfloat16) else if (dtype == MYNN_F16) RUN(__half) else return fail(MYNN_E_ARG, "swiglu_limbs2: bad dtype %d", dtype);
#undef RUN
    MYNN_LAUNCH_OK("swiglu_limbs2_kernel");
    return MYNN_OK;
}

bool i8_w8a8_supported(int M, int N, int K, const void *lhs, const void *rhs) {
    return M >= 1 && N >= 1 && K >= 16 && K % 16 == 0 && (((uintptr_t)lhs | (uintptr_t)rhs) % 16) == 0 && tensor_map_api_available();
}

int i8_w8a8_launch(cudaStream_t st, void *out, const int8_t *lhs, const void *lhs_scale, int lhs_scale_per_row, const int8_t *rhs,
                   const void *rhs_scale, int M, int N, int K, int dtype, void *workspace, size_t workspace_bytes) {
    if (!workspace || workspace_bytes < 256 || (uintptr_t)workspace % 256)
        return fail(MYNN_E_ARG, "quantized_matmul: a 256-byte aligned workspace of at least 256 bytes is needed");
    PfParams p;
    p.out = out;
    p.scale = rhs_scale;
    p.resid = nullptr;
    p.ascale = nullptr;
    p.ascale_t = lhs_scale;
    p.ascale_stride = lhs_scale_per_row ? 1 : 0;
    p.M = M;
    p.N = N;
    p.K = K;
    p.status = (int *)workspace;
    pf_tiles(p, 1);
    CUtensorMap mw, ma;
    int rc = make_map(&mw, rhs, (uint64_t)N, (uint64_t)K, (uint64_t)K, kPfRows);
    if (rc) return rc;
    rc = make_map(&ma, lhs, (uint64_t)M, (uint64_t)K, (uint64_t)K, (uint32_t)p.cols / 2);
    if (rc) return rc;
    if (dtype == MYNN_BF16) return launch_pf<__nv_bfloat16, 1>(st, mw, ma, p);
    if (dtype == MYNN_F16) return launch_pf<__half, 1>(st, mw, ma, p);
    return launch_pf<float, 1>(st, mw, ma, p);
}

}  // namespace mynn
