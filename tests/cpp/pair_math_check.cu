// Checks the packed pair arithmetic of physica_b200/csrc/pbf_math.cuh against the IEEE intrinsics.
// Built and called by tests/test_gpu_pair_math.py; every entry returns the number of mismatches.
#include <cstdint>

#include "sph_math.cuh"

namespace {

using namespace pbf;

// Calls visit(a) for every 24-bit a in [1, 2) whose quotient a / b lies within `limit` units of
// 1 / (2^25 b) (2^24 b for quotients of at least 1) of the midpoint of two floats; b = B / 2^23.
// With numerator units N = A 2^25 - M B (M odd: the midpoint M / 2^25), the solutions of
// M B = -N (mod 2^25) are the numerators nearest a rounding boundary.  Any other quotient lies
// further from a boundary than the residual correction's error.
template <class Visit>
__device__ void nearest_boundaries(const uint32_t B, const int limit, Visit visit) {
    const int v = __ffs(static_cast<int>(B)) - 1;
    const uint32_t odd = B >> v;
    uint32_t inverse = odd;
    for (int k = 0; k < 5; ++k) inverse *= 2u - odd * inverse;
    for (int N = -limit; N <= limit; ++N) {
        if (N == 0 || v > 4 || (N & ((1 << v) - 1))) continue;
        for (int shift = 24; shift <= 25; ++shift) {
            const int bits = shift - v;
            const uint32_t mask = (1u << bits) - 1u;
            for (uint64_t M = static_cast<uint32_t>(-(N >> v)) * inverse & mask; M < (1u << 25); M += 1ull << bits) {
                if (M < (1u << 24) || (M & 1u) == 0u) continue;
                const int64_t numerator = N + static_cast<int64_t>(M) * B;
                if (numerator & ((1ll << shift) - 1)) continue;
                const int64_t A = numerator >> shift;
                if (A < (1 << 23) || A >= (1 << 24) || (shift == 24) != (A >= static_cast<int64_t>(B))) continue;
                visit(static_cast<float>(A) * 0x1p-23F);
            }
        }
    }
}

__device__ uint32_t mix(uint32_t x) {
    x ^= x >> 16; x *= 0x7feb352du; x ^= x >> 15; x *= 0x846ca68bu; x ^= x >> 16;
    return x;
}

__device__ void count(unsigned long long* bad, const bool wrong) {
    if (wrong) atomicAdd(bad, 1ull);
}

__device__ bool differs(const float a, const float b) { return __float_as_uint(a) != __float_as_uint(b); }

// every float r2 in [first, first + n)
__global__ void root_kernel(const uint32_t first, const uint32_t n, unsigned long long* bad) {
    const uint64_t i = static_cast<uint64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const float r2 = __uint_as_float(first + static_cast<uint32_t>(i));
    float2 reciprocal;
    const float2 ns = negated_root_pair(make_float2(-r2, -r2), reciprocal);
    count(bad, differs(-ns.x, __fsqrt_rn(r2)) || differs(ns.x, ns.y));
    const double inverse = 1.0 / sqrt(static_cast<double>(r2)), reciprocal_d = 1.0 / static_cast<double>(r2);
    count(bad, !(fabs(wide_rsqrt(r2) - inverse) <= 0x1p-51 * inverse));
    count(bad, !(fabs(wide_reciprocal(r2) - reciprocal_d) <= 0x1p-52 * reciprocal_d));
}

// quotients by s = sqrt(r2) for every r2 in [1, 4): all significands of s with every approximation
// they come with
__global__ void root_quotient_kernel(const int limit, unsigned long long* bad) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= (1u << 24)) return;
    const float r2 = __uint_as_float(0x3f800000u + i);
    float2 R;
    const float2 ns = negated_root_pair(make_float2(-r2, -r2), R);
    auto check = [&](const float a) { count(bad, differs(quotient_pair(both(a), ns, R).x, __fdiv_rn(a, -ns.x))); };
    if (ns.x > -2.0F) nearest_boundaries(__float_as_uint(-ns.x) & 0x7fffffu | 0x800000u, limit, check);
    for (uint32_t t = 0; t < 16u; ++t) check(__uint_as_float(0x3f800000u | (mix(i * 16u + t) >> 9)));
}

// quotients by every significand b with its correctly rounded reciprocal
__global__ void constant_quotient_kernel(const int limit, unsigned long long* bad) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= (1u << 23)) return;
    const float b = __uint_as_float(0x3f800000u + i);
    const float R = __frcp_rn(b);
    auto check = [&](const float a) { count(bad, differs(quotient_pair(both(a), both(-b), both(R)).x, __fdiv_rn(a, b))); };
    nearest_boundaries(i | 0x800000u, limit, check);
    // a reciprocal that rounds up where 1 / b lies within 2^-18 ulp below the next rounding boundary
    const double above = 1.0 / static_cast<double>(b) * (1.0 + 0x1p-41);
    const float U = static_cast<float>(above);
    if (U != R) nearest_boundaries(i | 0x800000u, limit, [&](const float a) {
        count(bad, differs(quotient_pair(both(a), both(-b), both(U)).x, __fdiv_rn(a, b)));
    });
    for (uint32_t t = 0; t < 32u; ++t) check(__uint_as_float(0x3f800000u | (mix(i * 32u + t) >> 9)));
}

// whether r2 is in the range of the packed arithmetic (0 is: the weight there needs no root)
__device__ __forceinline__ bool fast_pair(const float r2, const KernelConstants& k) {
    return r2 <= k.fast_max && (r2 >= k.fast_min || r2 == 0.0F);
}

// the kernels' values at n squared distances spread over that range
__global__ void kernels_kernel(const float h, const uint32_t n, unsigned long long* bad, unsigned long long* tested) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const KernelConstants k = kernel_constants(h);
    float r2 = k.h2 * (static_cast<float>(mix(i) >> 8) * 0x1p-24F);
    if (i % 4u == 1u) r2 = __uint_as_float(__float_as_uint(k.fast_max) - (mix(i) & 0xffffu));   // the support's edge
    if (i % 4u == 2u) r2 = ldexpf(r2, -static_cast<int>(mix(~i) % 60u));                         // towards zero
    if (i == 3u) r2 = 0.0F;
    if (i == 7u) r2 = k.fast_min;
    if (i == 11u) r2 = k.fast_max;
    if (!fast_pair(r2, k)) return;
    atomicAdd(tested, 1ull);
    const float2 nr2 = make_float2(-r2, -r2);
    count(bad, differs(poly6_pair(nr2, k).y, poly6_inside(r2, k)));
    count(bad, differs(poly6_call(r2, k.h2, k.poly6_denominator), poly6_inside(r2, k)));
    count(bad, differs(poly6_weight(r2, k), poly6_inside(r2, k)));
    const float difference = __fsub_rn(k.h2, r2);
    count(bad, differs(poly6_gradient_scale(r2, k),
                       __fdiv_rn(__fmul_rn(__fmul_rn(-945.0F, difference), difference), k.poly6_grad_denominator)));
    if (r2 == 0.0F) return;
    const float distance = __fsqrt_rn(r2);
    count(bad, !(distance < k.h && distance > 0.0F && r2 < k.h2));
    const float scale_at = spiky_gradient_at(mk(1.0F, 0.0F, 0.0F), distance, k).x;
    count(bad, differs(spiky_scale_pair(nr2, k).y, scale_at));
    count(bad, differs(spiky_scale_call(distance, k.h, k.spiky_coefficient), scale_at));
    const PairDerivatives w = pair_derivatives(r2, k);
    count(bad, differs(w.scale, scale_at));
    const double r = sqrt(static_cast<double>(r2)), gap = k.h - r;
    const double along = k.spiky_coefficient_d * gap * gap / r;
    const double across = k.spiky_coefficient_d * (-2.0 * gap - gap * gap / r) / (static_cast<double>(r2));
    // the distance's rounding (2^-52 h) moves the gap h - r, the other factors a few 2^-53
    const double bound = 0x1p-48 + 0x1p-50 * k.h / gap;
    count(bad, !(fabs(w.along - along) <= bound * fabs(along)) || !(fabs(w.across - across) <= bound * fabs(across)));
}

// the cubic spline's values likewise, to beyond the support
__global__ void cubic_kernel(const float h, const uint32_t n, unsigned long long* bad, unsigned long long* tested) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    sph::SphConstants k{};
    k.h = h;
    k.cubic_coefficient = __fdiv_rn(8.0F, __fmul_rn(__fmul_rn(__fmul_rn(kPi, h), h), h));
    k.cubic_coefficient_2 = __fmul_rn(k.cubic_coefficient, 2.0F);
    k.support_threshold = kernel_constants(h).spiky_threshold;
    k.inverse_h = __frcp_rn(h);
    k.fast_min = __fmul_rn(__fmul_rn(h, h), 0x1p-60F);
    k.fast_max = __fmul_rn(__fmul_rn(h, h), 2.0F);
    float r2 = h * h * 1.3F * (static_cast<float>(mix(i) >> 8) * 0x1p-24F);
    if (i % 4u == 1u) r2 = __uint_as_float(__float_as_uint(k.support_threshold) + 64u - (mix(i) & 0xffffu));
    if (i % 4u == 2u) r2 = ldexpf(r2, -static_cast<int>(mix(~i) % 60u));
    const float2 nr2 = make_float2(-r2, -r2);
    if (!sph::detail::in_range(nr2, k)) return;
    atomicAdd(tested, 1ull);
    const float distance = __fsqrt_rn(r2);
    const float weight = distance < h ? sph::detail::cubic_inside(distance, k) : 0.0F;
    const float slope = distance < h ? sph::detail::cubic_gradient_scale(distance, k) : 0.0F;
    count(bad, differs(sph::detail::any_cubic(r2, &k), weight) || differs(sph::detail::any_cubic_gradient(r2, &k), slope));
    if (!sph::detail::inside(-r2, k)) {
        count(bad, distance < h);
        return;
    }
    count(bad, differs(sph::detail::cubic_pair(nr2, k).y, weight));
    const float packed = sph::detail::cubic_gradient_pair(nr2, k).y;   // a zero's sign may differ
    count(bad, packed != slope);
}

unsigned long long* counter() {
    unsigned long long* bad = nullptr;
    cudaMallocManaged(&bad, 2 * sizeof(unsigned long long));
    bad[0] = bad[1] = 0;
    return bad;
}

long long finish(unsigned long long* bad) {
    const cudaError_t e = cudaDeviceSynchronize();
    const long long wrong = e == cudaSuccess ? static_cast<long long>(bad[0]) : -1;
    cudaFree(bad);
    return wrong;
}

}  // namespace

extern "C" long long check_roots(const uint32_t first, const uint32_t n) {
    unsigned long long* bad = counter();
    root_kernel<<<(n + 255u) / 256u, 256>>>(first, n, bad);
    return finish(bad);
}

extern "C" long long check_root_quotients(const int limit) {
    unsigned long long* bad = counter();
    root_quotient_kernel<<<(1u << 24) / 256u, 256>>>(limit, bad);
    return finish(bad);
}

extern "C" long long check_constant_quotients(const int limit) {
    unsigned long long* bad = counter();
    constant_quotient_kernel<<<(1u << 23) / 256u, 256>>>(limit, bad);
    return finish(bad);
}

// Mismatches of the kernel values at support radius h (n samples); *tested: samples inside the range.
extern "C" long long check_kernels(const float h, const uint32_t n, long long* tested) {
    unsigned long long* bad = counter();
    kernels_kernel<<<(n + 255u) / 256u, 256>>>(h, n, bad, bad + 1);
    cudaDeviceSynchronize();
    *tested = static_cast<long long>(bad[1]);
    return finish(bad);
}

// The same for the cubic spline.
extern "C" long long check_cubic(const float h, const uint32_t n, long long* tested) {
    unsigned long long* bad = counter();
    cubic_kernel<<<(n + 255u) / 256u, 256>>>(h, n, bad, bad + 1);
    cudaDeviceSynchronize();
    *tested = static_cast<long long>(bad[1]);
    return finish(bad);
}
