// The packed roots, reciprocals and quotients of sf_device.cuh against CUDA's
// correctly rounded ones (tests/test_rounding.py).  Every function adds its
// mismatches to a counter.
#include "sf_device.cuh"

using namespace sf;

namespace {

__device__ bool same(F2 got, float want) {
    const float2 g = unpack(got);
    return __float_as_uint(g.x) == __float_as_uint(want) && __float_as_uint(g.y) == __float_as_uint(want);
}
__device__ F2 both(float x) { return f2(x, x); }

// Whether both halves of y are within (1/2 + 2^-20) of a last place of 1 / x (the
// fused residual 1 - x y is exact).
__device__ bool near_reciprocal(F2 got, float x) {
    const float2 g = unpack(got);
    const float ulp = __uint_as_float(__float_as_uint(g.x) + 1u) - g.x;
    return g.x == g.y && fabs((double)fmaf(-x, g.x, 1.f)) <= (double)x * (double)ulp * (0.5 + 0x1p-20);
}

// r^2 of the bit patterns [first, last): miss[0] roots, [1] 1 / r, [2] 1 / r^2
__global__ void k_roots(uint32_t first, uint32_t last, unsigned long long* miss) {
    const uint64_t step = (uint64_t)gridDim.x * blockDim.x;
    for (uint64_t b = first + (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; b < last; b += step) {
        const float r2 = __uint_as_float((uint32_t)b);
        const float y0 = rsqrt_approx(r2);
        const RootRecip o = root_recip(both(-r2), both(y0));
        const float r = __fsqrt_rn(r2);
        if (!same(o.nr, -r)) atomicAdd(miss, 1ull);
        if (!near_reciprocal(o.y, r)) atomicAdd(miss + 1, 1ull);
        if (!near_reciprocal(recip_step(both(-r2), mul2(both(y0), both(y0))), r2)) atomicAdd(miss + 2, 1ull);
    }
}

// The quotient of the numerator `a` by r (square clear) or r^2, scaled by 2^e.
__device__ bool quotient_fails(float a, float den, bool square, int e) {
    const float r2 = square ? den : den * den;
    const float y0 = rsqrt_approx(r2);
    const F2 y = square ? recip_step(both(-r2), mul2(both(y0), both(y0))) : root_recip(both(-r2), both(y0)).y;
    const float num = ldexpf(a, e);
    return !same(quotient2(both(num), both(-den), y), __fdiv_rn(num, den));
}

// Denominators B * 2^scale, 2^23 <= B < 2^24.  Numerators A with
// A / B within |D| / (2 B) of the last place from the middle of two floats, |D| <=
// 8: A 2^(k+1) = (2Q + 1) B + D with k = 23 (A >= B) or 24, Q of 24 bits; and
// `random` others.  miss[0] counts failures, miss[1] the numerators tried.
__global__ void k_quotients(int scale, bool square, int random, unsigned long long* miss) {
    const uint32_t B = (1u << 23) + blockIdx.x * blockDim.x + threadIdx.x;
    const float den = ldexpf((float)B, scale);
    const int t = __ffs((int)B) - 1;
    const uint32_t odd = B >> t;
    uint32_t inverse = odd;  // of odd modulo 2^32: each step doubles the correct bits (3 to begin with)
    for (int i = 0; i < 4; ++i) inverse *= 2u - odd * inverse;
    unsigned long long bad = 0, tried = 0;
    for (int D = -8; D <= 8; ++D) {
        if (D == 0 || __ffs(D < 0 ? -D : D) - 1 != t) continue;
        for (int k = 23; k <= 24; ++k) {
            const uint64_t m = (1ull << (k + 1)) >> t;
            uint64_t mid = (uint64_t)(uint32_t)(-(D >> t) * (int64_t)inverse) % m;
            for (; mid < (1ull << 25); mid += m) {
                if (mid < (1ull << 24)) continue;
                const int64_t scaled = (int64_t)(mid * B) + D;
                const int64_t A = scaled >> (k + 1);
                if ((A << (k + 1)) != scaled || A < (1 << 23) || A >= (1 << 24) || (k == 23) != (A >= (int64_t)B)) continue;
                ++tried;
                bad += quotient_fails((float)A, den, square, 0);
                bad += quotient_fails((float)A, den, square, -123);  // to the smallest numerators, 2^-100
            }
        }
    }
    uint32_t x = B * 2654435761u + (uint32_t)scale;
    for (int i = 0; i < random; ++i) {
        x = mix32(x + 0x9e3779b9u);
        ++tried;
        bad += quotient_fails((float)((1u << 23) | (x >> 9)), den, square, (int)(x & 127u) - 123);
    }
    if (bad) atomicAdd(miss, bad);
    atomicAdd(miss + 1, tried);
}

}  // namespace

extern "C" __attribute__((visibility("default"))) int check_rounding(float r2_min, float r2_max, int random, unsigned long long out[7]) {
    unsigned long long* d = nullptr;
    if (cudaMalloc(&d, 7 * sizeof(*d)) != cudaSuccess) return 1;
    cudaMemset(d, 0, 7 * sizeof(*d));
    uint32_t lo, hi;
    memcpy(&lo, &r2_min, 4);
    memcpy(&hi, &r2_max, 4);
    k_roots<<<4096, 256>>>(lo, hi + 1u, d);
    k_quotients<<<(1 << 23) / 256, 256>>>(-23, false, random, d + 3);  // r in [1, 2)
    k_quotients<<<(1 << 23) / 256, 256>>>(-23, true, random, d + 5);   // r^2 in [1, 2)
    k_quotients<<<(1 << 23) / 256, 256>>>(-22, true, random, d + 5);   // and [2, 4)
    const cudaError_t e = cudaMemcpy(out, d, 7 * sizeof(*d), cudaMemcpyDeviceToHost);
    cudaFree(d);
    return e == cudaSuccess ? 0 : 2;
}
