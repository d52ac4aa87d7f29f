// The corrected reciprocals, quotients and roots of the product's kernels
// against the general operators, bit for bit (test_gpu_exact_arithmetic.py
// compiles this file with the rasters' flags). Counters: mismatches, then the
// operands compared, per check.
#include "fiber_raster.cu"

namespace fiber {

using Count = unsigned long long;
enum Check : int { kRcp = 0, kSqrt, kNear, kRandom, kUnorm, kChecks };

__device__ __forceinline__ bool same(float a, float b) { return __float_as_uint(a) == __float_as_uint(b); }

__device__ __forceinline__ void add_counts(Count* out, int check, Count bad, Count seen) {
    if (bad) atomicAdd(out + 2 * check, bad);
    if (seen) atomicAdd(out + 2 * check + 1, seen);
}

__device__ __forceinline__ uint64_t mix(uint64_t x) {  // splitmix64 (Steele, Lea, Flood 2014)
    x += 0x9E3779B97F4A7C15ull;
    x = (x ^ (x >> 30)) * 0xBF58476D1CE4E5B9ull;
    x = (x ^ (x >> 27)) * 0x94D049BB133111EBull;
    return x ^ (x >> 31);
}

// Every binary32 of magnitude 2^-100 to 2^101: both signs for the reciprocal,
// the root in both lanes of a pair.
__global__ void k_check_unary(Count* out, Mul2 mul2) {
    const uint64_t n = 201ull << 23, stride = (uint64_t)gridDim.x * blockDim.x;
    Count bad_r = 0, bad_s = 0, seen = 0;
    for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += stride) {
        const float x = __uint_as_float((uint32_t)i + (27u << 23)), z = __uint_as_float((uint32_t)(n - 1u - i) + (27u << 23));
        bad_r += !same(rcp_exact(x), __frcp_rn(x));
        bad_r += !same(rcp_exact(-x), __frcp_rn(-x));
        float s0, s1;
        unpack2(sqrt2_exact(mul2, x, z), s0, s1);
        bad_s += !same(s0, __fsqrt_rn(x));
        bad_s += !same(s1, __fsqrt_rn(z));
        seen += 2;
    }
    add_counts(out, kRcp, bad_r, seen);
    add_counts(out, kSqrt, bad_s, seen);
}

__device__ __forceinline__ int quotient_bad(Mul2 mul2, float a, float b) {
    const float want = __fdiv_rn(a, b);
    float q0, q1;
    unpack2(div2_exact(mul2, pack2(a, -a), b, b), q0, q1);
    return !same(div_by_rcp(a, b, rcp_exact(b)), want) + !same(q0, want) + !same(q1, -want);
}

// Quotients nearest to a rounding boundary: 24-bit integers a and odd b with
// 2^k a - b M = r for an odd M of 25 bits (M / 2 is the boundary) and 0 < |r| <= 8.
__global__ void k_check_near(Count* out, Mul2 mul2) {
    const uint32_t stride = gridDim.x * blockDim.x;
    Count bad = 0, seen = 0;
    for (uint32_t t = blockIdx.x * blockDim.x + threadIdx.x; t < (1u << 22); t += stride) {
        const uint32_t b = (1u << 23) + 2u * t + 1u;
        uint32_t inv = b;  // b^-1 mod 2^32 by Newton's iteration
        for (int k = 0; k < 5; ++k) inv *= 2u - b * inv;
        for (int r = -8; r <= 8; ++r) {
            if (r == 0) continue;
            for (uint32_t k = 24u; k <= 25u; ++k) {
                const uint32_t m0 = ((uint32_t)(-r) * inv) & ((1u << k) - 1u);
                for (uint32_t M = m0; M < (1u << 25); M += 1u << k) {
                    if (M < (1u << 24) || !(M & 1u)) continue;
                    const uint64_t p = (uint64_t)b * M + (uint64_t)(int64_t)r;
                    const uint64_t a = p >> k;
                    if (a < (1ull << 23) || a >= (1ull << 24)) continue;
                    const uint64_t h = mix(((uint64_t)b << 32) ^ M);
                    const float fa = scalbnf((float)a, (int)(h % 140u) - 90), fb = scalbnf((float)b, (int)((h >> 32) % 60u) - 60);
                    bad += quotient_bad(mul2, (float)a, (float)b) + quotient_bad(mul2, fa, fb);
                    seen += 6;
                }
            }
        }
    }
    add_counts(out, kNear, bad, seen);
}

// 2^29 seeded quotients: |a| of 2^-79 to 2^80, b of 2^-40 to 2^40.
__global__ void k_check_random(Count* out, Mul2 mul2) {
    const uint32_t stride = gridDim.x * blockDim.x;
    Count bad = 0, seen = 0;
    for (uint32_t t = blockIdx.x * blockDim.x + threadIdx.x; t < (1u << 29); t += stride) {
        const uint64_t h = mix(t), g = mix(h);
        const uint32_t ea = 127u - 79u + (uint32_t)(g % 159u), eb = 127u - 40u + (uint32_t)((g >> 32) % 80u);
        const float a = __uint_as_float((ea << 23) | ((uint32_t)h & 0x7FFFFFu));
        const float b = __uint_as_float((eb << 23) | ((uint32_t)(h >> 32) & 0x7FFFFFu));
        bad += quotient_bad(mul2, a, b);
        seen += 3;
    }
    add_counts(out, kRandom, bad, seen);
}

// The 16-bit and 24-bit unpackings, every value.
__global__ void k_check_unorm(Count* out) {
    const uint32_t stride = gridDim.x * blockDim.x;
    Count bad = 0, seen = 0;
    for (uint32_t q = blockIdx.x * blockDim.x + threadIdx.x; q < (1u << 24); q += stride) {
        bad += !same(dequantize_depth01(q), u2f(q) / 16777215.0f);
        const float2 v = unpack2x16unorm((q << 16) | (q & 0xFFFFu));
        bad += !same(v.x, u2f(q & 0xFFFFu) / 65535.0f) + !same(v.y, u2f(q & 0xFFFFu) / 65535.0f);
        seen += 3;
    }
    add_counts(out, kUnorm, bad, seen);
}

}  // namespace fiber

extern "C" int exact_arithmetic(unsigned long long* host /* [2 kChecks] */) {
    using namespace fiber;
    unsigned long long* d = nullptr;
    const size_t bytes = 2 * kChecks * sizeof(*d);
    if (cudaMalloc(&d, bytes) != cudaSuccess || cudaMemset(d, 0, bytes) != cudaSuccess) return 1;
    const Mul2 mul2{0x8000000080000000ull};
    k_check_unary<<<148 * 8, 256>>>(d, mul2);
    k_check_near<<<148 * 8, 256>>>(d, mul2);
    k_check_random<<<148 * 8, 256>>>(d, mul2);
    k_check_unorm<<<148 * 8, 256>>>(d);
    const int rc = cudaGetLastError() == cudaSuccess && cudaMemcpy(host, d, bytes, cudaMemcpyDeviceToHost) == cudaSuccess ? 0 : 2;
    cudaFree(d);
    return rc;
}
