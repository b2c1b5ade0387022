// Expert routing: softmax over the router logits, the groups with the best member, the best experts of those groups, and the
// (token, slot) pairs ordered by expert for the grouped matrix products.
//
// One warp per token makes the choice (repeated warp-wide maxima; equal scores go to the lower index).
// A step of a few tokens runs entirely in one CTA; longer ones count in global memory, order in a second kernel and scatter in a
// third.  The order of the pairs of one expert is not fixed, and nothing depends on it: every pair is a row of its own.
#include "block_ops.cuh"
#include "common.cuh"

namespace mynn {

static size_t up16(size_t x) { return (x + 15) / 16 * 16; }

// The counts come first and have a fixed size: layers with different numbers of experts share one workspace, and what has to be
// zero between calls must not move over what another layer has written.
constexpr int kMaxExperts = 1024;
constexpr size_t kCountBytes = kMaxExperts * 4;

static int max_tiles(int M, int experts, int top) {
    const long long pairs = (long long)M * top;
    return (int)(pairs / kMoeTileRows + (experts < pairs ? experts : pairs) + 1);
}

size_t moe_route_bytes(int M, int experts, int top) {
    const size_t pairs = (size_t)M * top;
    return kCountBytes + 4 * up16(pairs * 4) + 2 * up16((size_t)(experts + 1) * 4) + 2 * up16((size_t)max_tiles(M, experts, top) * 4) + 32;
}

MoeRoute moe_route_bind(void *base, int M, int experts, int top) {
    const size_t pairs = (size_t)M * top;
    char *p = (char *)base;
    auto take = [&](size_t n) {
        char *r = p;
        p += up16(n);
        return r;
    };
    MoeRoute r;
    r.count = (int32_t *)take(kCountBytes);
    r.pair_w = (float *)take(pairs * 4);
    r.pair_row = (int32_t *)take(pairs * 4);
    r.pair_e = (int32_t *)take(pairs * 4);
    r.tok_of = (int32_t *)take(pairs * 4);
    r.off = (int32_t *)take((size_t)(experts + 1) * 4);
    r.active = (int32_t *)take((size_t)(experts + 1) * 4);
    r.tile_e = (int32_t *)take((size_t)max_tiles(M, experts, top) * 4);
    r.tile_row = (int32_t *)take((size_t)max_tiles(M, experts, top) * 4);
    r.n_active = (int32_t *)take(4);
    r.n_tiles = (int32_t *)take(4);
    return r;
}

// Floats as integers in the same order (zeros of both signs are one number); 0 is below every number and marks what is out of the race.
__device__ __forceinline__ unsigned order_key(float v) {
    const unsigned b = __float_as_uint(v + 0.0f);
    return b ^ ((b >> 31) ? 0xffffffffu : 0x80000000u);
}
__device__ __forceinline__ float key_value(unsigned k) { return __uint_as_float(k ^ ((k >> 31) ? 0x80000000u : 0xffffffffu)); }

// the largest key of the warp and, of those that have it, the lowest index
__device__ __forceinline__ void warp_argmax(unsigned &key, int &i) {
    const unsigned best = __reduce_max_sync(0xffffffffu, key);
    i = (int)__reduce_min_sync(0xffffffffu, key == best ? (unsigned)i : 0x7fffffffu);
    key = best;
}

// The choice for one token by one warp; z: room for its E logits in shared memory.  Slot s: expert in lane s's `e`, weight in `w`.
// NU: logits per lane (E <= 32 NU), in registers as ordered integers, so that a slot costs two warp reductions: at one token the choice
// is a chain of `keep + top` of them and nothing else (eight of 64 experts out of four of eight groups: 9.1 us for the whole kernel, one after the other in a graph,
// with five shuffle steps of value and index over shared memory, 5.8 us so).
template <int NU>
__device__ __forceinline__ void choose(float *z, const float *src, int E, int top, int groups, int keep, int &e_out, float &w_out) {
    const int lane = threadIdx.x & 31;
    float raw[NU], mx = -INFINITY;
    unsigned key[NU];
#pragma unroll
    for (int u = 0; u < NU; u++) raw[u] = lane + 32 * u < E ? src[lane + 32 * u] : 0.f;
#pragma unroll
    for (int u = 0; u < NU; u++) {
        key[u] = 0u;
        if (lane + 32 * u < E) {
            const float v = fmaxf(raw[u], -3.0e38f);  // also for NaN: every expert stays comparable, and above the excluded ones
            key[u] = order_key(v);
            mx = fmaxf(mx, v);
            if (keep < groups) z[lane + 32 * u] = v;
        }
    }
    mx = warp_max(mx);
    float sum = 0.f;
#pragma unroll
    for (int u = 0; u < NU; u++)
        if (lane + 32 * u < E) sum += expf(raw[u] - mx);  // a NaN logit makes the weights NaN
    sum = warp_sum(sum);
    __syncwarp();
    if (keep < groups) {
        // softmax is monotonic, so group scores may be compared as logits
        const int per = E / groups;
        unsigned gk[2], kept[2] = {0u, 0u};  // this lane's groups lane, lane + 32
#pragma unroll
        for (int u = 0; u < 2; u++) {
            const int g = lane + 32 * u;
            gk[u] = 0u;
            if (g < groups) {
                float v = -INFINITY;
                for (int i = 0; i < per; i++) v = fmaxf(v, z[g * per + i]);
                gk[u] = order_key(v);
            }
        }
        for (int k = 0; k < keep; k++) {
            unsigned v = gk[0];
            int g = lane;
            if (gk[1] > v) v = gk[1], g = lane + 32;
            warp_argmax(v, g);
            if (g == lane) gk[0] = 0u;
            if (g == lane + 32) gk[1] = 0u;
            kept[g >> 5] |= 1u << (g & 31);
        }
#pragma unroll
        for (int u = 0; u < NU; u++) {
            const int i = lane + 32 * u, g = i / per;
            if (i < E && !((g < 32 ? kept[0] : kept[1]) >> (g & 31) & 1u)) key[u] = 0u;
        }
    }
    e_out = 0;
    w_out = 0.f;
    unsigned mine = 0u;
    for (int s = 0; s < top; s++) {
        unsigned v = key[0];
        int e = lane;
#pragma unroll
        for (int u = 1; u < NU; u++)
            if (key[u] > v) v = key[u], e = lane + 32 * u;
        warp_argmax(v, e);
        if (lane == s) e_out = e, mine = v;
#pragma unroll
        for (int u = 0; u < NU; u++)
            if (e == lane + 32 * u) key[u] = 0u;
    }
    if (lane < top) w_out = expf(key_value(mine) - mx) / sum;
}

// counts -> offsets, list of used experts, tiles; one warp.  Counts are cleared on the way.
__device__ __forceinline__ void order_experts(const MoeRoute &r, int32_t *count, int E, int32_t *off_s = nullptr) {
    const int lane = threadIdx.x & 31;
    int off = 0, act = 0, tiles = 0;
    for (int base = 0; base < E; base += 32) {
        const int e = base + lane, c = e < E ? count[e] : 0;
        const int nt = (c + kMoeTileRows - 1) / kMoeTileRows, used = c > 0;
        int so = c, st = nt, su = used;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int a = __shfl_up_sync(0xffffffffu, so, o), b = __shfl_up_sync(0xffffffffu, st, o), d = __shfl_up_sync(0xffffffffu, su, o);
            if (lane >= o) so += a, st += b, su += d;
        }
        const int my_off = off + so - c, my_tile = tiles + st - nt;
        if (e < E) {
            r.off[e] = my_off;
            if (off_s) off_s[e] = my_off;
            if (used) r.active[act + su - 1] = e;
            for (int t = 0; t < nt; t++) {
                r.tile_e[my_tile + t] = e;
                r.tile_row[my_tile + t] = my_off + t * kMoeTileRows;
            }
            count[e] = 0;
        }
        off += __shfl_sync(0xffffffffu, so, 31);
        tiles += __shfl_sync(0xffffffffu, st, 31);
        act += __shfl_sync(0xffffffffu, su, 31);
    }
    if (lane == 0) {
        r.off[E] = off;
        *r.n_active = act;
        *r.n_tiles = tiles;
    }
}

// everything for a few tokens: one CTA; dynamic shared memory: E logits per warp, E counts, E offsets, expert and place of every pair
static size_t route_small_smem(int warps, int M, int E, int top) { return ((size_t)(warps + 2) * E + 2 * (size_t)M * top) * 4; }
template <int NU>
__global__ void __launch_bounds__(1024) moe_route_small_kernel(const MoeRoute r, const float *logits, int M, int E, int top, int groups, int keep) {
    extern __shared__ float sm[];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, warps = blockDim.x >> 5;
    float *z = sm + (size_t)warp * E;
    int32_t *count = reinterpret_cast<int32_t *>(sm + (size_t)warps * E), *off = count + E, *pair_e = off + E, *place = pair_e + M * top;
    for (int i = threadIdx.x; i < E; i += blockDim.x) count[i] = 0;
    pdl_trigger();
    pdl_wait();
    __syncthreads();
    for (int t = warp; t < M; t += warps) {
        int e;
        float w;
        choose<NU>(z, logits + (size_t)t * E, E, top, groups, keep, e, w);
        if (lane < top) {
            const int pair = t * top + lane;
            r.pair_w[pair] = w;
            r.pair_e[pair] = e;
            pair_e[pair] = e;
            place[pair] = atomicAdd(&count[e], 1);
        }
    }
    __syncthreads();
    if (warp == 0) order_experts(r, count, E, off);
    __syncthreads();
    for (int i = threadIdx.x; i < M * top; i += blockDim.x) {
        const int row = off[pair_e[i]] + place[i];
        r.pair_row[i] = row;
        r.tok_of[row] = i / top;
    }
}

template <int NU>
__global__ void __launch_bounds__(256) moe_choose_kernel(const MoeRoute r, const float *logits, int M, int E, int top, int groups, int keep) {
    extern __shared__ float sm[];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, t = blockIdx.x * (blockDim.x >> 5) + warp;
    if (t >= M) return;
    int e;
    float w;
    choose<NU>(sm + (size_t)warp * E, logits + (size_t)t * E, E, top, groups, keep, e, w);
    if (lane < top) {
        const size_t pair = (size_t)t * top + lane;
        r.pair_w[pair] = w;
        r.pair_e[pair] = e;
        r.pair_row[pair] = atomicAdd(&r.count[e], 1);
    }
}
__global__ void moe_order_kernel(const MoeRoute r, int E) { order_experts(r, r.count, E); }
__global__ void __launch_bounds__(256) moe_scatter_kernel(const MoeRoute r, int pairs, int top) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= pairs) return;
    const int row = r.off[r.pair_e[i]] + r.pair_row[i];
    r.pair_row[i] = row;
    r.tok_of[row] = i / top;
}

int launch_moe_route(cudaStream_t st, const MoeRoute &r, const float *logits, int M, int E, int top, int groups, int keep) {
    if (M <= 0 || E <= 0 || top <= 0 || top > 32 || top > E || groups <= 0 || groups > 64 || E % groups || keep <= 0 || keep > groups || E > kMaxExperts ||
        (long long)top > (long long)keep * (E / groups))
        return fail(MYNN_E_ARG, "moe_route: bad routing (%d experts, top %d, %d of %d groups)", E, top, keep, groups);
    if ((long long)M * top > (1ll << 30)) return fail(MYNN_E_UNSUPPORTED, "moe_route: too many tokens");
#define BY_EXPERTS(LAUNCH) \
    if (E <= 64) LAUNCH(2) else if (E <= 256) LAUNCH(8) else LAUNCH(32)
    if (M <= 64) {
        const int warps = M < 32 ? M : 32;
        const size_t smem = route_small_smem(warps, M, E, top);
#define SMALL(NU)                                                                                                                              \
    {                                                                                                                                          \
        auto kern = moe_route_small_kernel<NU>;                                                                                                \
        if (smem > 48 * 1024) MYNN_CUDA_OK(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));                \
        MYNN_CUDA_OK(launch_dependent(kern, dim3(1), dim3(warps * 32), smem, st, r, logits, M, E, top, groups, keep));                         \
    }
        BY_EXPERTS(SMALL)
#undef SMALL
        MYNN_LAUNCH_OK("moe_route_small_kernel");
        return MYNN_OK;
    }
#define CHOOSE(NU) moe_choose_kernel<NU><<<(M + 7) / 8, 256, (size_t)8 * E * 4, st>>>(r, logits, M, E, top, groups, keep);
    BY_EXPERTS(CHOOSE)
#undef CHOOSE
#undef BY_EXPERTS
    MYNN_LAUNCH_OK("moe_choose_kernel");
    moe_order_kernel<<<1, 32, 0, st>>>(r, E);
    MYNN_LAUNCH_OK("moe_order_kernel");
    moe_scatter_kernel<<<(M * top + 255) / 256, 256, 0, st>>>(r, M * top, top);
    MYNN_LAUNCH_OK("moe_scatter_kernel");
    return MYNN_OK;
}

}  // namespace mynn

using namespace mynn;

extern "C" size_t mynn_b200_moe_workspace_bytes(int M, int experts, int top) {
    if (M <= 0 || experts <= 0 || top <= 0) return 0;
    return moe_route_bytes(M, experts, top);
}

extern "C" int mynn_b200_moe_route(void *stream, void *workspace, size_t workspace_bytes, float *weights_out, int32_t *experts_out, const float *logits,
                                   int M, int experts, int top, int groups, int groups_keep) {
    if (M < 0 || experts <= 0 || top <= 0) return fail(MYNN_E_ARG, "moe_route: bad shape");
    if (M == 0) return MYNN_OK;
    if (!workspace || !logits) return fail(MYNN_E_ARG, "moe_route: null pointer");
    if (workspace_bytes < moe_route_bytes(M, experts, top) || (uintptr_t)workspace % 16)
        return fail(MYNN_E_ARG, "moe_route: a 16-byte aligned workspace of %zu bytes is needed, %zu given", moe_route_bytes(M, experts, top), workspace_bytes);
    const MoeRoute r = moe_route_bind(workspace, M, experts, top);
    cudaStream_t st = (cudaStream_t)stream;
    if (int rc = launch_moe_route(st, r, logits, M, experts, top, groups, groups_keep)) return rc;
    const size_t n = (size_t)M * top * 4;
    if (weights_out) MYNN_CUDA_OK(cudaMemcpyAsync(weights_out, r.pair_w, n, cudaMemcpyDeviceToDevice, st));
    if (experts_out) MYNN_CUDA_OK(cudaMemcpyAsync(experts_out, r.pair_e, n, cudaMemcpyDeviceToDevice, st));
    return MYNN_OK;
}
