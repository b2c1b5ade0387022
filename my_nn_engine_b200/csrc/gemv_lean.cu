// Lean DequantMatMul for one to four activation rows over small weight matrices (the GEMV of batch-1 decode).
//
//   out[m,n] = scale[n] * sum_k act[m,k] * wq[n,k],   M <= 4, wq [N,K] int8 of at most a few tens of MB
//
// A matrix of 10-30 MB streams from HBM in 2-5 us, so everything that is fixed cost in the tcgen05 kernel (tensor-memory
// allocation, tensor maps, mbarrier ring, a separate limb pre-pass launch, 128-row tiles that leave SMs idle) would dominate.
// This kernel has none of it (the engine's counterpart is dequant_gemv, src/codegen/cuda/cpp/dequant_gemv.cuh:11-59: one
// warp per row, one 16-byte load in flight per lane):
//   * one CTA per SM with an equal share of the rows, so the grid is a single balanced wave.  Its rows are tiles of 16; the sixteen warps
//     deal out the contraction, so that every warp has the same piece of every row, and each lane issues all its 128-bit loads (up to 20)
//     before it touches anything else, and before the programmatic-dependent-launch wait: the weights are in flight while
//     the preceding kernel drains;
//   * the activation row(s) are the same three signed 8-bit limbs of a 23-bit fixed-point value the tensor-core kernel uses, either read
//     from the workspace, where a fused producer left them, or computed here in shared memory (no extra launch).  Three limbs of up to
//     four rows are the columns of mma.m16n8k32 (int8, exact int32 sums).  The contraction index is permuted so that the 16 bytes a lane
//     loads are its fragments of two MMAs, for weights and limbs alike; a warp needs its own piece of the limbs only;
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

namespace mynn {

constexpr int kLeanThreads = 512;
constexpr int kLeanWarps = kLeanThreads / 32;
constexpr int kLeanTiles = 8;                       // row tiles whose partial sums are kept at a time
constexpr int kLeanFreeSms = 8;
constexpr int kLeanPitch = 16 * kLeanTiles + 4;     // int32 per (warp, column): no two lanes of a store in one bank
// limb rows in shared memory are this far apart: eight rows of a fragment load fall into different banks
__host__ __device__ __forceinline__ int lean_limb_pitch(int K) { return (K + 127) / 128 * 128 + 64; }

struct LeanParams {
    void *out;
    const void *act;        // [M,K] or null (then limbs_g / ascale_g hold the activations)
    const int8_t *wq;
    const void *scale, *resid;
    int8_t *limbs_g;        // workspace limb matrix [(3m + l)][K]; read when act == null, written by CTA 0 otherwise
    float *ascale_g;        // [M] row scales
    int N, K, act_dtype, rows_per_cta;
};

__device__ __forceinline__ uint4 ldg_stream_16(const void *p) {
    uint4 v;
    asm volatile("ld.global.nc.L1::no_allocate.v4.u32 {%0,%1,%2,%3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(p));
    return v;
}

// One activation row -> limbs in shared memory (and, from CTA 0, in the workspace), with the arithmetic of the limb pre-pass
// of the tensor-core kernel: |a| * 2^(22-e) rounded to an integer below 2^22, split into three signed bytes.  Rows of up to
// 8 elements per thread stay in registers between the two passes.
template <typename ActT>
__device__ __forceinline__ void row_to_limbs(const ActT *row, int K, int pitch, int8_t *l_s, int8_t *l_g, float *ascale_s, float *ascale_g,
                                             float *red) {
    constexpr int kKeep = 8;
    float keep[kKeep];
    float mx = 0.f;
    bool bad = false;
#pragma unroll
    for (int u = 0; u < kKeep; u++) {
        const int i = threadIdx.x + u * kLeanThreads;
        keep[u] = i < K ? to_f32<ActT>(row[i]) : 0.f;
        bad |= !(fabsf(keep[u]) <= 3.0e38f);
        mx = fmaxf(mx, fabsf(keep[u]));
    }
    for (int i = threadIdx.x + kKeep * kLeanThreads; i < K; i += kLeanThreads) {
        const float a = to_f32<ActT>(row[i]);
        bad |= !(fabsf(a) <= 3.0e38f);
        mx = fmaxf(mx, fabsf(a));
    }
    mx = warp_max(mx);
    const unsigned anybad = __syncthreads_or(bad);
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = mx;
    __syncthreads();
    float t = red[0];
#pragma unroll
    for (int w = 1; w < kLeanThreads / 32; w++) t = fmaxf(t, red[w]);
    int e = 0;
    if (t > 0.f) frexpf(t, &e);
    const float sc1 = t > 0.f ? ldexpf(1.0f, 22 - e) : 1.0f;
    const float sc = anybad ? 0.f : sc1;
    if (threadIdx.x == 0) {
        const float as = anybad ? __int_as_float(0x7fc00000) : 1.0f / sc1;  // a non-finite input row gives NaN outputs
        *ascale_s = as;
        if (ascale_g) *ascale_g = as;
    }
    auto emit = [&](float a, int i) {
        int A = sc == 0.f ? 0 : __float2int_rn(a * sc);
        const int d0 = (int)(int8_t)(A & 0xFF);
        A = (A - d0) >> 8;
        const int d1 = (int)(int8_t)(A & 0xFF);
        A = (A - d1) >> 8;
        l_s[i] = (int8_t)d0;
        l_s[pitch + i] = (int8_t)d1;
        l_s[2 * pitch + i] = (int8_t)A;
        if (l_g) {
            l_g[i] = (int8_t)d0;
            l_g[K + i] = (int8_t)d1;
            l_g[2 * (size_t)K + i] = (int8_t)A;
        }
    };
#pragma unroll
    for (int u = 0; u < kKeep; u++) {
        const int i = threadIdx.x + u * kLeanThreads;
        if (i < K) emit(keep[u], i);
    }
    for (int i = threadIdx.x + kKeep * kLeanThreads; i < K; i += kLeanThreads) emit(to_f32<ActT>(row[i]), i);
    __syncthreads();  // red is reused by the next row
}

__device__ __forceinline__ void mma_i8(int (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
    asm volatile("mma.sync.aligned.m16n8k32.row.col.s32.s8.s8.s32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
                 : "+r"(c[0]), "+r"(c[1]), "+r"(c[2]), "+r"(c[3])
                 : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}

// One CTA per SM owns a contiguous range of weight rows, so that the whole grid is one balanced wave.  A warp owns NB blocks of 64 along K
// (K <= 1024 NB) of all of them; TG tiles of 16 rows are in flight (2 NB TG <= 20 loads per lane, issued before anything else happens).
// K % 16 == 0; wq and limbs 16-byte aligned.  Dynamic shared memory: limbs [3 M][pitch] (only with act), partial sums [warp][3 M][kLeanPitch].
template <typename OutT, int M, int NB, int TG>
__global__ void __launch_bounds__(kLeanThreads, 1) gemv_lean_kernel(const LeanParams p) {
    extern __shared__ __align__(16) int8_t sm_dyn[];
    __shared__ float sm_ascale[4];
    __shared__ float red[kLeanWarps];
    constexpr int C = 3 * M, NT = (C + 7) / 8;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, gq = lane >> 2, t = lane & 3;
    const int K = p.K, chunks = K >> 4, pitch = lean_limb_pitch(K);
    const int row0 = blockIdx.x * p.rows_per_cta, rows = min(p.rows_per_cta, p.N - row0), tiles = (rows + 15) >> 4;
    int8_t *sm_limbs = sm_dyn;
    int *sm_sum = reinterpret_cast<int *>(sm_dyn + (p.act ? (size_t)C * pitch : 0));
    const OutT *scale_p = reinterpret_cast<const OutT *>(p.scale);
    const OutT *resid_p = reinterpret_cast<const OutT *>(p.resid);
    OutT *out_p = reinterpret_cast<OutT *>(p.out);

    const int c0 = warp * 4 * NB + t;  // this lane's 16-byte chunks of a row: c0 + 4 j
    uint4 w[TG][NB][2];
    auto load_tile = [&](uint4 (&x)[NB][2], int tile) {
#pragma unroll
        for (int h = 0; h < 2; h++) {
            const int row = 16 * tile + gq + 8 * h;
            const int8_t *wr = p.wq + (size_t)(row0 + (row < rows ? row : 0)) * K;
#pragma unroll
            for (int j = 0; j < NB; j++) {
                const int c = c0 + 4 * j;
                x[j][h] = row < rows && c < chunks ? ldg_stream_16(wr + 16 * (size_t)c) : make_uint4(0u, 0u, 0u, 0u);
            }
        }
    };
    // the first tiles of weights and the row scale of this thread's output depend on nothing an earlier kernel writes
#pragma unroll
    for (int i = 0; i < TG; i++)
        if (i < tiles) load_tile(w[i], i);
    // outputs of the first pass: thread -> (row, activation row)
    const int pass_rows = min(rows, 16 * kLeanTiles), my_m = threadIdx.x / pass_rows, my_r = threadIdx.x - my_m * pass_rows;
    float wscale_first = 0.f, resv_first = 0.f;
    if (my_m < M) wscale_first = to_f32<OutT>(scale_p[row0 + my_r]);
    pdl_trigger();
    pdl_wait();
    if (my_m < M && resid_p) resv_first = to_f32<OutT>(resid_p[(size_t)my_m * p.N + row0 + my_r]);
    // limbs of this warp's piece of K: column gq (and gq + 8) of the MMAs is limb row gq (gq + 8) = 3 m + l
    uint4 b[NT][NB];
    if (p.act != nullptr) {
        int8_t *lg = blockIdx.x == 0 ? p.limbs_g : nullptr;
        float *ag = blockIdx.x == 0 ? p.ascale_g : nullptr;
#pragma unroll 1
        for (int m = 0; m < M; m++) {
            int8_t *ls = sm_limbs + (size_t)m * 3 * pitch;
            if (p.act_dtype == MYNN_F32)
                row_to_limbs<float>((const float *)p.act + (size_t)m * K, K, pitch, ls, lg ? lg + (size_t)m * 3 * K : nullptr, &sm_ascale[m], ag ? ag + m : nullptr, red);
            else if (p.act_dtype == MYNN_BF16)
                row_to_limbs<__nv_bfloat16>((const __nv_bfloat16 *)p.act + (size_t)m * K, K, pitch, ls, lg ? lg + (size_t)m * 3 * K : nullptr, &sm_ascale[m], ag ? ag + m : nullptr, red);
            else
                row_to_limbs<__half>((const __half *)p.act + (size_t)m * K, K, pitch, ls, lg ? lg + (size_t)m * 3 * K : nullptr, &sm_ascale[m], ag ? ag + m : nullptr, red);
        }
        __syncthreads();
#pragma unroll
        for (int n = 0; n < NT; n++)
#pragma unroll
            for (int j = 0; j < NB; j++) {
                const int c = c0 + 4 * j, col = 8 * n + gq;
                b[n][j] = col < C && c < chunks ? *reinterpret_cast<const uint4 *>(sm_limbs + (size_t)col * pitch + 16 * c) : make_uint4(0u, 0u, 0u, 0u);
            }
    } else {
#pragma unroll
        for (int n = 0; n < NT; n++)
#pragma unroll
            for (int j = 0; j < NB; j++) {
                const int c = c0 + 4 * j, col = 8 * n + gq;
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
        const int beg = 16 * first, n_rows = min(rows, 16 * last) - beg;
        for (int i = threadIdx.x; i < n_rows * M; i += kLeanThreads) {
            const int m = i / n_rows, r = i - m * n_rows, row = row0 + beg + r;
            const bool known = first == 0 && i == (int)threadIdx.x;  // requested at the top of the kernel
            const float wscale = known ? wscale_first : to_f32<OutT>(scale_p[row]);
            const float resv = known ? resv_first : resid_p ? to_f32<OutT>(resid_p[(size_t)m * p.N + row]) : 0.f;
            int v[3] = {0, 0, 0};
#pragma unroll
            for (int x = 0; x < kLeanWarps; x++)
#pragma unroll
                for (int l = 0; l < 3; l++) v[l] += sm_sum[(x * C + 3 * m + l) * kLeanPitch + r];
            const long long sum = (long long)v[2] * 65536 + (long long)v[1] * 256 + (long long)v[0];
            float y = __fmul_rn(__fmul_rn((float)sum, sm_ascale[m]), wscale);
            if (resid_p) y = __fadd_rn(round_store<OutT>(y), resv);
            out_p[(size_t)m * p.N + row] = from_f32<OutT>(y);
        }
        if (last < tiles) __syncthreads();  // the sums are read before the next tiles' replace them
    }
}

bool gemv_lean_supported(int M, int N, int K, const void *wq) {
    // small matrices only: larger ones amortise the tensor-core kernel's set-up and stream faster there
    return M >= 1 && M <= 4 && K >= 16 && K % 16 == 0 && K <= 6144 && (size_t)3 * M * K <= 96 * 1024 && (size_t)N * K <= ((size_t)32 << 20) &&
           ((uintptr_t)wq % 16) == 0;
}

template <typename OutT, int M, int NB, int TG>
static int launch_lean(cudaStream_t st, LeanParams p) {
    const size_t smem = (p.act ? (size_t)3 * M * lean_limb_pitch(p.K) : 0) + (size_t)kLeanWarps * 3 * M * kLeanPitch * sizeof(int);
    auto kern = gemv_lean_kernel<OutT, M, NB, TG>;
    static bool attr_set = false;
    if (!attr_set) {  // the most this form can need
        constexpr int most = 3 * M * (1024 * NB + 64) + kLeanWarps * 3 * M * kLeanPitch * (int)sizeof(int);
        static_assert(most <= 227 * 1024, "shared memory of a CTA");
        MYNN_CUDA_OK(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, most));
        attr_set = true;
    }
    static int sms = 0;
    if (sms == 0) {
        int dev = 0;
        cudaGetDevice(&dev);
        if (cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || sms <= 0) sms = 148;
    }
    // One CTA per SM, each with an equal share of the rows; a few SMs stay free, where the CTAs of the row kernel behind this one (launched
    // as its dependent) are resident by the time it ends.
    const int ctas = sms > 4 * kLeanFreeSms ? sms - kLeanFreeSms : sms, rpc = (p.N + ctas - 1) / ctas;
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

// Same contract as i8_gemm_launch: `workspace` holds status word, row scales and the limb matrix; act == nullptr means a fused
// producer (or the previous call) left the limbs there.
int gemv_lean_launch(cudaStream_t st, void *out, const void *act, const int8_t *wq, const void *scale, const void *resid, int M, int N,
                     int K, int act_dtype, int out_dtype, void *workspace, size_t workspace_bytes) {
    const size_t need = i8_gemm_workspace_bytes(M, K);
    if (!workspace || workspace_bytes < need || (uintptr_t)workspace % 256)
        return fail(MYNN_E_ARG, "dequant_matmul: workspace of %zu bytes (256-byte aligned) needed", need);
    LeanParams p;
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
    p.rows_per_cta = 0;
    // blocks of 64 per warp (K <= 1024 / 2048 / 4096 / 6144) and row tiles in flight
#define BY_K(OT, MV)                                        \
    if (K <= 1024) return launch_lean<OT, MV, 1, 8>(st, p); \
    if (K <= 2048) return launch_lean<OT, MV, 2, 5>(st, p); \
    if (K <= 4096) return launch_lean<OT, MV, 4, 2>(st, p); \
    return launch_lean<OT, MV, 6, 1>(st, p);
#define GO(OT)               \
    switch (M) {             \
        case 1: BY_K(OT, 1)  \
        case 2: BY_K(OT, 2)  \
        case 3: BY_K(OT, 3)  \
        default: BY_K(OT, 4) \
    }
    if (out_dtype == MYNN_BF16) GO(__nv_bfloat16)
    if (out_dtype == MYNN_F16) GO(__half)
    GO(float)
#undef GO
#undef BY_K
}

}  // namespace mynn
