// The fixed-point form that int8 products give an activation row: scaled by a power of two so that its largest magnitude lies below 2^22,
// rounded to whole numbers A and cut into three signed bytes, A = l0 + 256 l1 + 65536 l2.
#pragma once
#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <stdint.h>

namespace mynn {

// Largest magnitude of a row -> scale 2^(22 - e) with top < 2^e, by its exponent bits; 0 for a row that holds something non-finite (bits of the
// magnitude: infinities and NaN are above all numbers).  Rows below 2^-105 get the largest scale there is.
__device__ __forceinline__ float limb_scale(uint32_t top_bits) {
    if (top_bits > 0x7f61b1e6u) return 0.f;  // 3.0e38
    const uint32_t e = top_bits >> 23;
    return top_bits == 0u ? 1.0f : __uint_as_float((275u - (e < 21u ? 21u : e)) << 23);
}
// what the sums of a row are multiplied with; a non-finite input row gives NaN outputs
__device__ __forceinline__ float limb_unscale(float sc) { return sc == 0.f ? __int_as_float(0x7fc00000) : 1.0f / sc; }

// Four elements -> one word of each limb.  x * sc + 1.5 * 2^23 has the rounded number in its low bits; with 128 (and 128 * 256) added, byte 1 (and
// byte 2) are the limbs that make the lower ones signed.  Five instructions per element; with conversions, masks and shifts it was about twenty.
__device__ __forceinline__ void limbs_of_4(const float *x, float sc, uint32_t &w0, uint32_t &w1, uint32_t &w2) {
    uint32_t a[4], b[4], c[4];
#pragma unroll
    for (int i = 0; i < 4; i++) {
        a[i] = __float_as_uint(fmaf(x[i], sc, 12582912.0f));  // 0x4b400000 + A
        b[i] = a[i] + 0x80u;
        c[i] = a[i] + (0x8080u - 0x400000u);
    }
    w0 = __byte_perm(__byte_perm(a[0], a[1], 0x0040u), __byte_perm(a[2], a[3], 0x0040u), 0x5410u);
    w1 = __byte_perm(__byte_perm(b[0], b[1], 0x0051u), __byte_perm(b[2], b[3], 0x0051u), 0x5410u);
    w2 = __byte_perm(__byte_perm(c[0], c[1], 0x0062u), __byte_perm(c[2], c[3], 0x0062u), 0x5410u);
    if (sc == 0.f) w0 = w1 = w2 = 0u;
}
// Largest magnitude of eight elements, as bits.
__device__ __forceinline__ uint32_t max_bits8(const float (&v)[8]) {
    uint32_t mx = 0u;
#pragma unroll
    for (int j = 0; j < 8; j++) mx = max(mx, __float_as_uint(v[j]) & 0x7fffffffu);
    return mx;
}

}  // namespace mynn
