// Layer norms (and norms by root mean square) of the block decoder, fused with the residual step in front of them.
//
// A sandwich-normed layer does x += mult * LN(sublayer output) and then feeds LN(x) to the next sublayer.  Both norms, the
// residual sum, the combination of routed experts and the addition of the embedding output at the start of a repeated pass
// are row operations, so one kernel does them with one read of the sublayer output and one read and write of x.
// The row stays in registers, so the deviations are taken around its mean in a second pass, which stays accurate when the mean is
// large against them.  (Merged moments, one block reduction in place of two, were slower: a division per merge in a chain of 13.)
#include "block_ops.cuh"
#include "common.cuh"

namespace mynn {

// Sums of two numbers over the block; every thread gets them.  sm holds two numbers per warp (32 pairs) and must not be the buffer of the
// call before (calls take turns between two), so one barrier per call is enough.
__device__ __forceinline__ float2 block_sum2(float a, float b, float2 *sm) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        a += __shfl_xor_sync(0xffffffffu, a, o);
        b += __shfl_xor_sync(0xffffffffu, b, o);
    }
    const int warps = blockDim.x >> 5, lane = threadIdx.x & 31;
    if (lane == 0) sm[threadIdx.x >> 5] = make_float2(a, b);
    __syncthreads();
    float2 t = lane < warps ? sm[lane] : make_float2(0.f, 0.f);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        if (o >= warps) continue;  // the warps past the last one hold zeros
        t.x += __shfl_xor_sync(0xffffffffu, t.x, o);
        t.y += __shfl_xor_sync(0xffffffffu, t.y, o);
    }
    return make_float2(__shfl_sync(0xffffffffu, t.x, 0), __shfl_sync(0xffffffffu, t.y, 0));
}

template <typename T, int V>
__device__ __forceinline__ void load_vec(const T *p, float (&v)[V]) {
    if constexpr (V == 4 && sizeof(T) == 2) {
        const uint2 r = *reinterpret_cast<const uint2 *>(p);
        const T *e = reinterpret_cast<const T *>(&r);
#pragma unroll
        for (int i = 0; i < 4; i++) v[i] = to_f32<T>(e[i]);
    } else if constexpr (V == 4) {
        const float4 r = *reinterpret_cast<const float4 *>(p);
        v[0] = r.x, v[1] = r.y, v[2] = r.z, v[3] = r.w;
    } else {
#pragma unroll
        for (int i = 0; i < V; i++) v[i] = to_f32<T>(p[i]);
    }
}
// the same without the conversion
template <typename T, int V>
__device__ __forceinline__ void raw_vec(const T *p, T (&v)[V]) {
    if constexpr (V == 4 && sizeof(T) == 2) {
        const uint2 r = *reinterpret_cast<const uint2 *>(p);
        const T *e = reinterpret_cast<const T *>(&r);
#pragma unroll
        for (int i = 0; i < 4; i++) v[i] = e[i];
    } else if constexpr (V == 4) {
        const float4 r = *reinterpret_cast<const float4 *>(p);
        const T *e = reinterpret_cast<const T *>(&r);
#pragma unroll
        for (int i = 0; i < 4; i++) v[i] = e[i];
    } else {
#pragma unroll
        for (int i = 0; i < V; i++) v[i] = p[i];
    }
}
template <typename T, int V>
__device__ __forceinline__ void store_vec(T *p, const float (&v)[V]) {
    if constexpr (V == 4 && sizeof(T) == 2) {
        uint2 r;
        T *e = reinterpret_cast<T *>(&r);
#pragma unroll
        for (int i = 0; i < 4; i++) e[i] = from_f32<T>(v[i]);
        *reinterpret_cast<uint2 *>(p) = r;
    } else if constexpr (V == 4) {
        *reinterpret_cast<float4 *>(p) = make_float4(v[0], v[1], v[2], v[3]);
    } else {
#pragma unroll
        for (int i = 0; i < V; i++) p[i] = from_f32<T>(v[i]);
    }
}

// grid = rows.  NV groups of V elements per thread live in registers between the passes (NV * V * blockDim.x >= W).
// FEW: a decode step, whose time is the chain of dependent steps: the weights are requested in front of the wait for the preceding kernel
// when they are known not to come from it, and all expert rows together.  Many rows are bound by how many of them an SM has on their
// way: 256 threads per row of up to 4096 elements and at most 64 registers, four rows per SM (two of 512 threads before).
template <typename T, int V, int NV, bool FEW, int THREADS>
__global__ void __launch_bounds__(THREADS, !FEW && THREADS == 256 && V == 4 ? 4 : 1) norm_step_kernel(const NormStep p) {
    __shared__ float2 sm[2][32];
    const int row = blockIdx.x, W = p.W;
    const int step = blockDim.x * V, i0 = threadIdx.x * V;
    constexpr bool EARLY = FEW;  // weights of both norms in registers
    float we[EARLY ? 4 : 1][NV][V];
    auto get_weights = [&]() {
        const float *src[4] = {p.w1, p.rms ? nullptr : p.b1, p.w2, p.rms ? nullptr : p.b2};
#pragma unroll
        for (int q = 0; q < 4; q++)
#pragma unroll
            for (int j = 0; j < NV; j++) {
#pragma unroll
                for (int k = 0; k < V; k++) we[q][j][k] = q & 1 ? 0.f : 1.f;
                if (src[q] && i0 + j * step < W) load_vec<float, V>(src[q] + i0 + j * step, we[q][j]);
            }
    };
    // Few rows: the product behind starts fetching its weights when it becomes resident, and this kernel's loads would queue behind them; it
    // is let go once they are here (combining norm of a step of one row 12 -> 6 us, the product behind unchanged).
    if (!FEW) pdl_trigger();
    if (!p.fixed_weights) pdl_wait();
    if constexpr (EARLY) get_weights();
    pdl_wait();
    const int src = p.row_map ? p.row_map[row] : row;
    float xv[NV][V];
    int turn = 0;
    // mean (0 for a norm by root mean square) and reciprocal deviation of the row.  The deviations are taken around the mean of the whole
    // row, and what rounding left of their own mean corrects both.
    auto norm_of = [&](const float (&v)[NV][V]) {
        float s = 0.f, q = 0.f, mean = 0.f;
#pragma unroll
        for (int pass = 0; pass < 2; pass++) {
            if (pass == 0 && p.rms) continue;
            s = q = 0.f;
#pragma unroll
            for (int j = 0; j < NV; j++)
                if (i0 + j * step < W) {
#pragma unroll
                    for (int e = 0; e < V; e++) {
                        const float d = v[j][e] - mean;
                        s += d;
                        if (pass) q += d * d;
                    }
                }
            const float2 t = block_sum2(s, q, sm[turn]);
            turn ^= 1;
            s = t.x / (float)W;
            q = t.y / (float)W;
            if (pass == 0) mean = s;
        }
        if (!p.rms) {
            mean += s;
            q = fmaxf(q - s * s, 0.f);
        }
        return make_float2(mean, 1.0f / sqrtf(q + p.eps));
    };
    if (p.embed) {
        const long long id = min(max((long long)p.ids[row], 0ll), (long long)p.vocab - 1);
        const T *e = reinterpret_cast<const T *>(p.embed) + (size_t)id * W;
#pragma unroll
        for (int j = 0; j < NV; j++) {
            const int i = i0 + j * step;
            if (i < W) {
                load_vec<T, V>(e + i, xv[j]);
#pragma unroll
                for (int k = 0; k < V; k++) xv[j][k] *= p.embed_scale;
                store_vec<float, V>(p.x + (size_t)row * W + i, xv[j]);
                if (p.x0) store_vec<float, V>(p.x0 + (size_t)row * W + i, xv[j]);
            }
        }
    } else {
#pragma unroll
        for (int j = 0; j < NV; j++) {
            const int i = i0 + j * step;
            if (i < W) load_vec<float, V>(p.x + (size_t)src * W + i, xv[j]);
        }
        if (p.sub) {
            float sv[NV][V];
            const T *sub = reinterpret_cast<const T *>(p.sub);
            if (p.pair_row) {
#pragma unroll
                for (int j = 0; j < NV; j++)
#pragma unroll
                    for (int k = 0; k < V; k++) sv[j][k] = 0.f;
                // rows in flight together: one after the other each would cost a trip to L2
                constexpr int U = FEW ? 8 : NV <= 4 ? 2 : 1;
                for (int s0 = 0; s0 < p.top; s0 += U) {
                    T t[U][NV][V];
                    float g[U];
                    int at[U];
#pragma unroll
                    for (int u = 0; u < U; u++) {
                        const size_t pair = (size_t)row * p.top + min(s0 + u, p.top - 1);
                        at[u] = p.pair_row[pair];
                        g[u] = p.pair_w[pair];
                    }
#pragma unroll
                    for (int u = 0; u < U; u++)
#pragma unroll
                        for (int j = 0; j < NV; j++)
                            if (i0 + j * step < W) raw_vec<T, V>(sub + (size_t)at[u] * W + i0 + j * step, t[u][j]);
#pragma unroll
                    for (int u = 0; u < U; u++)
                        if (s0 + u < p.top) {
#pragma unroll
                            for (int j = 0; j < NV; j++)
                                if (i0 + j * step < W) {
#pragma unroll
                                    for (int k = 0; k < V; k++) sv[j][k] += g[u] * to_f32<T>(t[u][j][k]);
                                }
                        }
                }
            } else {
#pragma unroll
                for (int j = 0; j < NV; j++) {
                    const int i = i0 + j * step;
                    if (i < W) load_vec<T, V>(sub + (size_t)row * W + i, sv[j]);
                }
            }
            if (FEW) pdl_trigger();
            float2 m = make_float2(0.f, 1.f);
            if (p.w1) m = norm_of(sv);
#pragma unroll
            for (int j = 0; j < NV; j++) {
                const int i = i0 + j * step;
                if (i < W) {
                    float w[V], b[V], z[V];
#pragma unroll
                    for (int k = 0; k < V; k++) w[k] = EARLY ? we[0][j][k] : 1.f, b[k] = EARLY ? we[EARLY ? 1 : 0][j][k] : 0.f;
                    if constexpr (!EARLY) {
                        if (p.w1) load_vec<float, V>(p.w1 + i, w);
                        if (p.w1 && !p.rms) load_vec<float, V>(p.b1 + i, b);
                    }
                    if (p.add_x0) load_vec<float, V>(p.x0 + (size_t)row * W + i, z);
#pragma unroll
                    for (int k = 0; k < V; k++) {
                        xv[j][k] += p.mult * ((sv[j][k] - m.x) * m.y * w[k] + b[k]);
                        if (p.add_x0) xv[j][k] += z[k];
                    }
                    store_vec<float, V>(p.x + (size_t)row * W + i, xv[j]);
                }
            }
        }
    }
    if (!p.out) return;
    const float2 m = norm_of(xv);
    T *out = reinterpret_cast<T *>(p.out) + (size_t)row * W;
#pragma unroll
    for (int j = 0; j < NV; j++) {
        const int i = i0 + j * step;
        if (i < W) {
            float w[V], b[V], y[V];
#pragma unroll
            for (int k = 0; k < V; k++) w[k] = EARLY ? we[EARLY ? 2 : 0][j][k] : 1.f, b[k] = EARLY ? we[EARLY ? 3 : 0][j][k] : 0.f;
            if constexpr (!EARLY) {
                load_vec<float, V>(p.w2 + i, w);
                if (!p.rms) load_vec<float, V>(p.b2 + i, b);
            }
#pragma unroll
            for (int k = 0; k < V; k++) y[k] = (xv[j][k] - m.x) * m.y * w[k] + b[k];
            store_vec<T, V>(out + i, y);
        }
    }
}

template <typename T, int V>
static int run_norm(cudaStream_t st, const NormStep &p, int rows) {
    const int groups = (p.W + V - 1) / V;
#define RUN(NV, FEW, THREADS) MYNN_CUDA_OK(launch_dependent(norm_step_kernel<T, V, NV, FEW, THREADS>, dim3(rows), dim3(threads), 0, st, p))
    // one wave of CTAs at most, rows of up to 4096 elements: measured inside a decode step of one row of 2048 (two norms, eight expert rows)
    const bool few = rows <= 148 && V == 4 && groups <= 1024;
    const int nv = few ? (groups <= 256 ? 1 : 2) : V == 4 && groups <= 1024 ? (groups <= 256 ? 1 : groups <= 512 ? 2 : 4)
                   : groups <= 2048 ? 2 : groups <= 4096 ? 4 : groups <= 8192 ? 8 : V == 1 && groups <= 32768 ? 32 : 0;
    if (!nv) return fail(MYNN_E_UNSUPPORTED, "layer_norm: rows of %d elements", p.W);
    const int threads = ((groups + nv - 1) / nv + 31) / 32 * 32;
    if constexpr (V == 4) {
        if (few) {
            if (nv == 1) RUN(1, true, 256);
            else RUN(2, true, 512);
        } else if (groups <= 1024) {
            if (nv == 1) RUN(1, false, 256);
            else if (nv == 2) RUN(2, false, 256);
            else RUN(4, false, 256);
        }
    }
    if (!few && (V != 4 || groups > 1024)) {
        switch (nv) {
            case 2: RUN(2, false, 1024); break;
            case 4: RUN(4, false, 1024); break;
            case 8: RUN(8, false, 1024); break;
            default:
                if constexpr (V == 1) RUN(32, false, 1024);
                break;
        }
    }
#undef RUN
    MYNN_LAUNCH_OK("norm_step_kernel");
    return MYNN_OK;
}

int launch_norm_step(cudaStream_t st, int dtype, const NormStep &p, int rows) {
    if (rows < 0 || p.W <= 0 || !p.x) return fail(MYNN_E_ARG, "layer_norm: bad shape rows=%d W=%d", rows, p.W);
    if (rows == 0) return MYNN_OK;
    uintptr_t a = (uintptr_t)p.embed | (uintptr_t)p.x | (uintptr_t)p.x0 | (uintptr_t)p.sub | (uintptr_t)p.out | (uintptr_t)p.w1 | (uintptr_t)p.b1 |
                  (uintptr_t)p.w2 | (uintptr_t)p.b2;
    const bool vec = p.W % 4 == 0 && a % 16 == 0;
    MYNN_DISPATCH_DTYPE(dtype, T, { return vec ? run_norm<T, 4>(st, p, rows) : run_norm<T, 1>(st, p, rows); });
    return MYNN_OK;
}

}  // namespace mynn

using namespace mynn;

extern "C" int mynn_b200_layer_norm(void *stream, void *out, const float *x, const float *weight, const float *bias, float eps, int rows,
                                    int W, int out_dtype) {
    if (rows < 0 || W <= 0) return fail(MYNN_E_ARG, "layer_norm: bad shape rows=%d W=%d", rows, W);
    if (!dtype_ok(out_dtype)) return fail(MYNN_E_ARG, "layer_norm: bad dtype %d", out_dtype);
    if (rows == 0) return MYNN_OK;
    if (!out || !x || !weight || !bias) return fail(MYNN_E_ARG, "layer_norm: null pointer");
    NormStep p;
    p.x = const_cast<float *>(x);  // without a sublayer output the kernel only reads it
    p.w2 = weight;
    p.b2 = bias;
    p.eps = eps;
    p.out = out;
    p.W = W;
    return launch_norm_step((cudaStream_t)stream, out_dtype, p, rows);
}

extern "C" int mynn_b200_residual_layer_norm(void *stream, float *x, const void *sub, const float *post_weight, const float *post_bias, float mult,
                                             const float *extra, const float *weight, const float *bias, void *out, float eps, int rows, int W,
                                             int dtype) {
    if (rows < 0 || W <= 0) return fail(MYNN_E_ARG, "residual_layer_norm: bad shape rows=%d W=%d", rows, W);
    if (!dtype_ok(dtype)) return fail(MYNN_E_ARG, "residual_layer_norm: bad dtype %d", dtype);
    if (rows == 0) return MYNN_OK;
    if (!x || !sub || !post_weight || !post_bias || (out && (!weight || !bias))) return fail(MYNN_E_ARG, "residual_layer_norm: null pointer");
    NormStep p;
    p.x = x;
    p.x0 = const_cast<float *>(extra);
    p.add_x0 = extra != nullptr;
    p.sub = sub;
    p.w1 = post_weight;
    p.b1 = post_bias;
    p.w2 = weight;
    p.b2 = bias;
    p.mult = mult;
    p.eps = eps;
    p.out = out;
    p.W = W;
    return launch_norm_step((cudaStream_t)stream, dtype, p, rows);
}

extern "C" int mynn_b200_residual_rms_norm(void *stream, float *x, const void *sub, const float *weight, void *out, float eps, int rows, int W, int dtype) {
    if (rows < 0 || W <= 0) return fail(MYNN_E_ARG, "residual_rms_norm: bad shape rows=%d W=%d", rows, W);
    if (!dtype_ok(dtype)) return fail(MYNN_E_ARG, "residual_rms_norm: bad dtype %d", dtype);
    if (rows == 0) return MYNN_OK;
    if (!x || (out && !weight)) return fail(MYNN_E_ARG, "residual_rms_norm: null pointer");
    NormStep p;
    p.x = x;
    p.sub = sub;
    p.w2 = weight;
    p.eps = eps;
    p.rms = 1;
    p.out = out;
    p.W = W;
    return launch_norm_step((cudaStream_t)stream, dtype, p, rows);
}
