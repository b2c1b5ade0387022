// Layer norms (and norms by root mean square) of the block decoder, fused with the residual step in front of them.
//
// A sandwich-normed layer does x += mult * LN(sublayer output) and then feeds LN(x) to the next sublayer.  Both norms, the
// residual sum, the combination of routed experts and the addition of the embedding output at the start of a repeated pass
// are row operations, so one kernel does them with one read of the sublayer output and one read and write of x.
// Two forms of the statistics, both accurate when the mean is large against the deviations.  Many rows: mean and squared deviations are
// gathered per thread around the thread's own mean and merged pairwise (the update of Chan, Golub and LeVeque), one block reduction
// per norm.  Few rows: sums, first for the mean and then for the deviations around it, because the merge's divisions are the longer chain.
#include "block_ops.cuh"
#include "common.cuh"

namespace mynn {

struct Moments {
    float n, mean, m2;
};
__device__ __forceinline__ Moments merge(const Moments &a, const Moments &b) {
    Moments r;
    r.n = a.n + b.n;
    const float d = b.mean - a.mean, f = r.n > 0.f ? b.n / r.n : 0.f;
    r.mean = a.mean + d * f;
    r.m2 = a.m2 + b.m2 + d * d * a.n * f;
    return r;
}

// every thread gets the moments of the whole row; sm holds one entry per warp
__device__ __forceinline__ Moments block_moments(Moments v, Moments *sm) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        Moments u;
        u.n = __shfl_xor_sync(0xffffffffu, v.n, o);
        u.mean = __shfl_xor_sync(0xffffffffu, v.mean, o);
        u.m2 = __shfl_xor_sync(0xffffffffu, v.m2, o);
        v = merge(v, u);
    }
    const int warps = blockDim.x >> 5;
    __syncthreads();  // sm may still be read from the previous call
    if ((threadIdx.x & 31) == 0) sm[threadIdx.x >> 5] = v;
    __syncthreads();
    Moments t = sm[0];
    for (int w = 1; w < warps; w++) t = merge(t, sm[w]);
    return t;
}

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
// when they are known not to come from it, the expert rows are requested together, and the statistics take the shorter chain.
// For many rows that would only cost registers.
template <typename T, int V, int NV, bool FEW>
__global__ void __launch_bounds__(NV == 1 ? 256 : FEW ? 512 : 1024) norm_step_kernel(const NormStep p) {
    __shared__ float2 sm[2][32];
    __shared__ Moments sm_m[32];
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
    pdl_trigger();
    if (!p.fixed_weights) pdl_wait();
    if constexpr (EARLY) get_weights();
    pdl_wait();
    const int src = p.row_map ? p.row_map[row] : row;
    float xv[NV][V];
    int turn = 0;
    // mean (0 for a norm by root mean square) and reciprocal deviation of the row.  The deviations are taken around the mean of the whole
    // row, and what rounding left of their own mean corrects both.
    auto norm_of = [&](const float (&v)[NV][V]) {
        if constexpr (!FEW) {
            Moments m = {0.f, 0.f, 0.f};
            float s = 0.f;
            int n = 0;
#pragma unroll
            for (int j = 0; j < NV; j++)
                if (i0 + j * step < W) {
#pragma unroll
                    for (int e = 0; e < V; e++) s += v[j][e];
                    n += V;
                }
            m.n = (float)n;
            m.mean = n ? s / (float)n : 0.f;
#pragma unroll
            for (int j = 0; j < NV; j++)
                if (i0 + j * step < W) {
#pragma unroll
                    for (int e = 0; e < V; e++) {
                        const float d = v[j][e] - m.mean;
                        m.m2 += d * d;
                    }
                }
            m = block_moments(m, sm_m);
            float q = m.m2 / (float)W;
            if (p.rms) {  // nothing is taken off, and mean(v^2) = var + mean^2
                q += m.mean * m.mean;
                m.mean = 0.f;
            }
            return make_float2(m.mean, 1.0f / sqrtf(q + p.eps));
        }
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
                constexpr int U = FEW ? 8 : 1;
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
    // one wave of CTAs at most, rows of up to 4096 elements: measured inside a decode step of one row of 2048 (two norms, eight expert rows)
    if (rows <= 148 && V == 4 && groups <= 1024) {
        const int nv = groups <= 256 ? 1 : 2, threads = ((groups + nv - 1) / nv + 31) / 32 * 32;
        if (nv == 1) MYNN_CUDA_OK(launch_dependent(norm_step_kernel<T, 4, 1, true>, dim3(rows), dim3(threads), 0, st, p));
        else MYNN_CUDA_OK(launch_dependent(norm_step_kernel<T, 4, 2, true>, dim3(rows), dim3(threads), 0, st, p));
        MYNN_LAUNCH_OK("norm_step_kernel");
        return MYNN_OK;
    }
    const int nv = groups <= 256 ? 1 : groups <= 2048 ? 2 : groups <= 4096 ? 4 : groups <= 8192 ? 8 : V == 1 && groups <= 32768 ? 32 : 0;
    if (!nv) return fail(MYNN_E_UNSUPPORTED, "layer_norm: rows of %d elements", p.W);
    const int threads = ((groups + nv - 1) / nv + 31) / 32 * 32;
    switch (nv) {
        case 1: MYNN_CUDA_OK(launch_dependent(norm_step_kernel<T, V, 1, false>, dim3(rows), dim3(threads), 0, st, p)); break;
        case 2: MYNN_CUDA_OK(launch_dependent(norm_step_kernel<T, V, 2, false>, dim3(rows), dim3(threads), 0, st, p)); break;
        case 4: MYNN_CUDA_OK(launch_dependent(norm_step_kernel<T, V, 4, false>, dim3(rows), dim3(threads), 0, st, p)); break;
        case 8: MYNN_CUDA_OK(launch_dependent(norm_step_kernel<T, V, 8, false>, dim3(rows), dim3(threads), 0, st, p)); break;
        default:
            if constexpr (V == 1) MYNN_CUDA_OK(launch_dependent(norm_step_kernel<T, V, 32, false>, dim3(rows), dim3(threads), 0, st, p));
            break;
    }
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
