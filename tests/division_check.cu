// Test program (built and run by tests/test_gpu_division.py): the arithmetic of
// sgx_device.cuh that stands for divisions and square roots, against the
// compiler's own, and one step of the FP32 fixed-step forms with shared
// reciprocals against the same step with compiled divisions, and the precision
// form's error norm from one component.  Prints mismatch counts
// (FP32: bit for bit) and worst errors in units of the last place (FP64).
#include <cmath>
#include <cstdio>

#include "sgx_device.cuh"

using namespace sgxd;

__device__ unsigned long long g_bad[7];
__device__ unsigned long long g_ulp[3];

__device__ __forceinline__ std::uint32_t mix(std::uint32_t x) {
    x ^= x >> 16;
    x *= 0x7feb352dU;
    x ^= x >> 15;
    x *= 0x846ca68bU;
    return x ^ (x >> 16);
}

__device__ __forceinline__ void differ(int k, float a, float b) {
    if (__float_as_uint(a) != __float_as_uint(b)) atomicAdd(&g_bad[k], 1ull);
}

// Every significand m at exponent e: the reciprocal, x / 6, and quotients of
// pseudo-random numerators by it; both signs.
__global__ void single(int e, int enum_lo, int enum_hi) {
    const std::uint32_t m = blockIdx.x * blockDim.x + threadIdx.x;  // < 2^23
    const float b = __uint_as_float((std::uint32_t(127 + e) << 23) | m);
    const RecipF rb(b), rn(-b);
    differ(0, rb.y, 1.0f / b);
    differ(0, rn.y, 1.0f / -b);
    differ(1, sixth(b), b / 6.0f);
    differ(1, sixth(-b), -b / 6.0f);
    for (std::uint32_t i = 0; i < 8u; ++i) {
        const std::uint32_t r = mix(m * 8u + i + std::uint32_t(e + 128) * 0x9e3779b9u);
        const int ea = enum_lo + int(mix(r) % std::uint32_t(enum_hi - enum_lo));
        const float a = __uint_as_float((r & 0x80000000u) | (std::uint32_t(127 + ea) << 23) | (r & 0x7fffffu));
        differ(2, rb(a), a / b);
        differ(2, rn(a), a / -b);
    }
    differ(3, rb(b), 1.0f);  // a zero's sign may differ: +0 for -0, which is all that does
    differ(3, rb(0.0f), 0.0f);
}

__global__ void dbl(int e) {
    const std::uint32_t m = blockIdx.x * blockDim.x + threadIdx.x;
    const unsigned long long bits = ((unsigned long long)(1023 + e) << 52) | ((unsigned long long)m << 29) | mix(m);
    const double x = __longlong_as_double((long long)bits);
    auto ulps = [](double a, double b) {
        const long long d = __double_as_longlong(a) - __double_as_longlong(b);
        return (unsigned long long)(d < 0 ? -d : d);
    };
    atomicMax(&g_ulp[0], ulps(rcp_newton(x), 1.0 / x));
    atomicMax(&g_ulp[1], ulps(sqrt_newton(x), sqrt(x)));
}

// States over all the range a step can meet and beyond it: radii from inside the
// horizon to 1e6, either pole, momenta of 1e-9 to 1e12, zeros, infinities, NaN.
__global__ void steps() {
    std::uint32_t s = mix(blockIdx.x * blockDim.x + threadIdx.x + 1u);
    auto uni = [&]() {
        s = mix(s + 0x9e3779b9u);
        return float(s >> 8) * 0x1p-24f;
    };
    auto wide = [&](float lo, float hi) {  // either sign, log-uniform; now and then a special value
        const float u = uni();
        if (u < 0.002f) return 0.0f;
        if (u < 0.003f) return INFINITY;
        if (u < 0.004f) return NAN;
        const float x = lo * exp2f(uni() * log2f(hi / lo));
        return uni() < 0.5f ? -x : x;
    };
    const bool far = uni() < 0.2f;
    auto num = [&](float lo, float hi) { return far ? wide(1e-9f, 1e12f) : wide(lo, hi); };
    View<float> v;
    v.M = uni() < 0.5f ? 1.0f : exp2f(16.0f * uni() - 8.0f);
    v.a = v.M * uni();
    v.a2 = v.a * v.a;
    v.twoM = 2.0f * v.M;
    v.rs = 2.0f * v.M;
    v.shared_div = 1u;
    const float r = v.M * (far ? fabsf(wide(1e-3f, 1e6f)) : 1.0f + 60.0f * uni());
    const float th = uni() < 0.1f ? wide(1e-9f, 1e-2f) : 3.2f * uni();
    const float h = exp2f(8.0f * uni() - 6.0f) * v.M;
    auto same = [](float a, float b) { return __float_as_uint(a) == __float_as_uint(b) || (isnan(a) && isnan(b)) || a == b; };
    KS<float> y{r, th, 6.0f * uni(), num(1e-4f, 10.0f), num(1e-4f, 10.0f * v.M)}, z = y;
    const KC<float> c = make_kc<float>(v, 0.8f + 0.4f * uni(), num(1e-3f, 10.0f * v.M));
    kerr_step_ref(y, h, v, c);
    kerr_rk4_ref_div(z, h, v, c);
    if (!(same(y.r, z.r) && same(y.th, z.th) && same(y.ph, z.ph) && same(y.pr, z.pr) && same(y.pth, z.pth)))
        atomicAdd(&g_bad[4], 1ull);
    SS<float> p{r, th, 6.0f * uni(), num(0.5f, 2.0f), num(1e-4f, 1.0f), num(1e-6f, 0.1f) / v.M, num(1e-6f, 0.1f) / v.M}, q = p;
    schw_step(p, h, v);
    schw_rk4_div(q, h, v.rs);
    if (!(same(p.r, q.r) && same(p.th, q.th) && same(p.ph, q.ph) && same(p.ut, q.ut) && same(p.ur, q.ur) &&
          same(p.uth, q.uth) && same(p.uph, q.uph)))
        atomicAdd(&g_bad[5], 1ull);
}

// The precision form's error norm from one FP64 component against the norm over
// all of them: random attempts, with ties, near ties, zeros and NaN among the
// components.
__global__ void norms() {
    std::uint32_t s = mix(blockIdx.x * blockDim.x + threadIdx.x + 77u);
    auto uni = [&]() {
        s = mix(s + 0x9e3779b9u);
        return float(s >> 8) * 0x1p-24f;
    };
    float y[6], y4[6], k4[6], k5[6];
    const float tie = uni(), d0 = exp2f(-30.0f * uni());
    for (int i = 0; i < 6; ++i) {
        y[i] = exp2f(10.0f * uni() - 8.0f) * (uni() < 0.5f ? -1.0f : 1.0f);
        y4[i] = y[i] * (1.0f + 0.01f * uni());
        k4[i] = uni() - 0.5f;
        float d = exp2f(-30.0f * uni());
        if (tie < 0.3f) {  // ratios equal to a few ulp
            y[i] = y[0];
            y4[i] = y4[0];
            d = d0 * (1.0f + 0x1p-22f * float(int(8.0f * uni())));
            k4[i] = 1.0f;
        }
        k5[i] = k4[i] - d;
        if (tie > 0.95f && uni() < 0.3f) k5[i] = k4[i];
        if (tie > 0.99f && uni() < 0.3f) k5[i] = NAN;
    }
    auto six = [](const float* v) { return KSC<float>{v[0], v[1], v[2], v[3], v[4], v[5]}; };
    const KSC<float> Y = six(y);
    const KAttempt<float> A{six(y4), six(k4), six(k5), exp2f(-8.0f * uni())};
    const double one = error_norm_zone(Y, A, 1e-6f), all = error_norm_fp64_1div(Y, A, 1e-6f);
    if (__double_as_longlong(one) != __double_as_longlong(all)) atomicAdd(&g_bad[6], 1ull);
}

// The FP64 norm against the definition evaluated with divisions, in units of
// the last place: three products, a reciprocal and two sums, each rounded once.
__global__ void norms64() {
    std::uint32_t s = mix(blockIdx.x * blockDim.x + threadIdx.x + 991u);
    auto uni = [&]() {
        s = mix(s + 0x9e3779b9u);
        return double(s >> 8) * 0x1p-24 + double(mix(s)) * 0x1p-56;
    };
    double y[6], y4[6], k4[6], k5[6];
    const double tie = uni(), d0 = exp2(-40.0 * uni());
    for (int i = 0; i < 6; ++i) {
        y[i] = exp2(10.0 * uni() - 8.0) * (uni() < 0.5 ? -1.0 : 1.0);
        y4[i] = y[i] * (1.0 + 0.01 * uni());
        k4[i] = 2.0 * uni() - 1.0;
        double d = exp2(-40.0 * uni());
        if (tie < 0.3) {  // ratios equal, or nearly
            y[i] = y[0];
            y4[i] = y4[0];
            d = d0 * (1.0 + 0x1p-18 * int(8.0 * uni()));
            k4[i] = 0.0;
        }
        k5[i] = k4[i] - d;
        if (tie > 0.95 && uni() < 0.3) k5[i] = k4[i];
    }
    auto six = [](const double* v) { return KSC<double>{v[0], v[1], v[2], v[3], v[4], v[5]}; };
    const KAttempt<double> A{six(y4), six(k4), six(k5), exp2(-8.0 * uni())};
    double want = 0.0;
    for (int i = 0; i < 6; ++i)
        want = fmax(want, fabs(A.h6 * (k4[i] - k5[i])) / (double(1e-6f) * (1.0 + fmax(fabs(y[i]), fabs(y4[i])))));
    want = fmin(want, 1e30);
    const long long d = __double_as_longlong(error_norm_pos(six(y), A, 1e-6f)) - __double_as_longlong(want);
    atomicMax(&g_ulp[2], (unsigned long long)(d < 0 ? -d : d));
}

int main() {
    for (int e : {-60, -20, -3, -1, 0, 1, 2, 9, 28, 60}) single<<<(1 << 23) / 256, 256>>>(e, -30, 30);
    for (int e : {-67, -20, -1, 0, 1, 7, 16, 40}) dbl<<<(1 << 23) / 256, 256>>>(e);
    steps<<<(1 << 22) / 256, 256>>>();
    norms<<<(1 << 22) / 256, 256>>>();
    norms64<<<(1 << 22) / 256, 256>>>();
    unsigned long long bad[7], ulp[3];
    cudaMemcpyFromSymbol(bad, g_bad, sizeof(bad));
    cudaMemcpyFromSymbol(ulp, g_ulp, sizeof(ulp));
    if (cudaDeviceSynchronize() != cudaSuccess) return 1;
    std::printf("%llu %llu %llu %llu %llu %llu %llu %llu %llu %llu\n", bad[0], bad[1], bad[2], bad[3], bad[4], bad[5], bad[6], ulp[0],
                ulp[1], ulp[2]);
    return 0;
}
