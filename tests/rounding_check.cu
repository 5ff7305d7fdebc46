// Test program (built and run by tests/test_gpu_rounding.py): tests/division_check.cu
// with its launches and copies checked, and the same arithmetic where it is
// hardest or leaves the ordinary: quotients nearest to a rounding boundary,
// the ends of the exponent range, x / 6 in FP64, momenta and angular momenta down
// to the subnormals, roots of subnormals, differences that are not finite.  Every
// kernel counts what it compared.  Prints division_check's line, then mismatches,
// comparisons and worst errors (in thousandths of a unit in the last place).
#define main division_main
#include "division_check.cu"
#undef main

enum { HARD, SIXTH_F, SIXTH_D, TINY_KERR, TINY_SCHW, ROOT, NORM, N_CHECKS };
__device__ unsigned long long g_miss[N_CHECKS], g_done[N_CHECKS], g_milli[2];

__device__ __forceinline__ void count(int k, bool ok) {
    atomicAdd(&g_done[k], 1ull);
    if (!ok) atomicAdd(&g_miss[k], 1ull);
}
__device__ __forceinline__ bool bits_equal(float a, float b) { return __float_as_uint(a) == __float_as_uint(b); }
__device__ __forceinline__ bool bits_equal(double a, double b) {
    return __double_as_longlong(a) == __double_as_longlong(b) || (isnan(a) && isnan(b));
}

// For every divisor significand B the numerators A with A 2^k = B M + r, M odd of
// 25 bits and |r| <= 7: quotients r / (B M) from the midpoint of two floats.
// B = 2^t B', B' odd, leaves r = 2^t r', so t <= 2, and 2^t solutions M of
// M = -r' / B' mod 2^(k - t).  Exponents ea, eb of numerator and divisor.
__global__ void hard(int ea, int eb) {
    const std::uint32_t B = 0x800000u + blockIdx.x * blockDim.x + threadIdx.x;  // 2^23 of them
    const int t = __ffs(int(B)) - 1;
    if (t > 2) return;
    const std::uint32_t odd = B >> t;
    std::uint32_t inv = odd;  // 1 / B' mod 2^32 by Newton's iteration (3 bits to begin with)
    for (int i = 0; i < 4; ++i) inv *= 2u - odd * inv;
    const float b = __uint_as_float((std::uint32_t(127 + eb) << 23) | (B & 0x7fffffu));
    const RecipF rb(b);
    for (int r = -7; r <= 7; r += 2) {
        if ((r < 0 ? -r : r) << t > 7) continue;
        for (int k = 24; k <= 25; ++k)
            for (std::uint32_t j = 0; j < (1u << t); ++j) {
                const std::uint32_t low = (std::uint32_t(-r) * inv) & ((1u << (k - t)) - 1u);
                std::uint32_t M = low + (j << (k - t));
                if (k == 24) M |= 1u << 24;
                if (M < (1u << 24)) continue;
                const unsigned long long num = (unsigned long long)B * M + (unsigned long long)((long long)r * (1 << t));
                const std::uint32_t A = std::uint32_t(num >> k);
                if (A < 0x800000u || A > 0xffffffu) continue;
                const float a = __uint_as_float((std::uint32_t(127 + ea) << 23) | (A & 0x7fffffu));
                count(HARD, bits_equal(rb(a), a / b));
                count(HARD, bits_equal(rb(-a), -a / b));
            }
    }
}

__global__ void sixths(int e) {
    const std::uint32_t m = blockIdx.x * blockDim.x + threadIdx.x;  // < 2^23
    const float x = __uint_as_float((std::uint32_t(127 + e) << 23) | m);
    count(SIXTH_F, bits_equal(sixth(x), x / 6.0f));
    // FP64: exponents over -968 .. 1023
    const std::uint32_t h = mix(m + 0x51ed270bu * std::uint32_t(e + 200));
    const int ed = -968 + int(mix(h) % 1992u);
    const double y = __longlong_as_double((long long)(((unsigned long long)(1023 + ed) << 52) |
                                                      ((unsigned long long)(h & 0xfffffu) << 32) | mix(h + 1u)));
    count(SIXTH_D, bits_equal(sixth(y), y / 6.0) && bits_equal(sixth(-y), -y / 6.0));
}

// Errors of the Newton reciprocal and root by their exact residuals.
__global__ void newton(int e) {
    const std::uint32_t m = blockIdx.x * blockDim.x + threadIdx.x;
    const double x = __longlong_as_double((long long)(((unsigned long long)(1023 + e) << 52) |
                                                      ((unsigned long long)m << 29) | (mix(m) & 0x1fffffffu)));
    auto ulp = [](double v) { return ldexp(1.0, ilogb(v) - 52); };
    const double y = rcp_newton(x), s = sqrt_newton(x);
    atomicMax(&g_milli[0], (unsigned long long)ceil(1000.0 * fabs(fma(-x, y, 1.0) / x) / ulp(y)));
    atomicMax(&g_milli[1], (unsigned long long)ceil(1000.0 * fabs(fma(-s, s, x) / (2.0 * s)) / ulp(s)));
}

// Steps of states whose momenta, or whose constant L, go down to the subnormals.
__global__ void tiny() {
    std::uint32_t s = mix(blockIdx.x * blockDim.x + threadIdx.x + 4242u);
    auto uni = [&]() {
        s = mix(s + 0x9e3779b9u);
        return float(s >> 8) * 0x1p-24f;
    };
    auto small = [&](float top) {
        const float u = uni(), x = u < 0.3f ? top * uni() : top * exp2f(-126.0f * uni());
        return u > 0.97f ? 0.0f : (uni() < 0.5f ? -x : x);
    };
    View<float> v;
    v.M = 1.0f;
    v.a = uni() < 0.5f ? 0.0f : uni();
    v.a2 = v.a * v.a;
    v.twoM = v.rs = 2.0f;
    v.shared_div = 1u;
    const float r = 2.1f + 58.0f * uni(), th = 0.05f + 3.04f * uni(), h = 0.05f + 0.45f * uni(), E = 0.8f + 0.4f * uni();
    auto near = [](float a, float b) { return a == b || fabsf(a - b) <= 0x1p-100f; };
    KS<float> y{r, th, 0.1f + 6.0f * uni(), small(1.0f), small(1.0f)}, z = y;
    const KC<float> c = make_kc<float>(v, E, small(4.0f));
    kerr_step_ref(y, h, v, c);
    kerr_rk4_ref_div(z, h, v, c);
    count(TINY_KERR, y.r == z.r && y.th == z.th && y.ph == z.ph && near(y.pr, z.pr) && near(y.pth, z.pth));
    SS<float> p{r, th, 0.1f + 6.0f * uni(), 1.0f + uni(), small(0.5f), small(0.05f), small(0.05f)}, q = p;
    schw_step(p, h, v);
    schw_rk4_div(q, h, v.rs);
    count(TINY_SCHW, p.r == q.r && p.th == q.th && p.ph == q.ph && p.ut == q.ut && near(p.ur, q.ur) &&
                         near(p.uth, q.uth) && near(p.uph, q.uph));
}

// p_theta on the Carter constant (Theta = Q with cos theta = 0) for Theta of every kind.
__global__ void roots() {
    const int i = threadIdx.x;
    const double kinds[] = {0.0, -0.0, -1.0, 5e-324, 1e-310, 2.2250738585072009e-308, 2.2250738585072014e-308, 1e-300, 0.25,
                            4.0, 1e300, 1.7976931348623157e308, __longlong_as_double(0x7ff0000000000000ll),
                            __longlong_as_double((long long)0xfff0000000000000ull)};
    if (i >= int(sizeof(kinds) / sizeof(kinds[0]))) return;
    KC<double> k{};
    const double th = kinds[i], got = project_pth(-3.0, 1.0, 0.0, th, k), want = copysign(th > 0.0 ? sqrt(th) : 0.0, -3.0);
    const long long d = __double_as_longlong(got) - __double_as_longlong(want);
    count(ROOT, d >= -1 && d <= 1);
}

// The FP64 norm with one difference, or its scale, not finite or too large: 1e30 where a
// difference is NaN or infinite or its quotient beyond 1e30, the other components'
// norm where only a scale is infinite.
__global__ void odd_norms() {
    std::uint32_t s = mix(blockIdx.x * blockDim.x + threadIdx.x + 31337u);
    auto uni = [&]() {
        s = mix(s + 0x9e3779b9u);
        return double(s >> 8) * 0x1p-24;
    };
    const int which = int(uni() * 6.0), kind = int(uni() * 8.0);
    const long long specials[] = {0x7ff8000000000000ll, (long long)0xfff8000000000000ull, 0x7ff0000000000001ll,
                                  0x7fffffffffffffffll, 0x7ff0000000000000ll, (long long)0xfff0000000000000ull};
    double y[6], y4[6], k4[6], k5[6];
    for (int i = 0; i < 6; ++i) {
        y[i] = 4.0 * uni() - 2.0;
        y4[i] = y[i] * (1.0 + 0.01 * uni());
        k4[i] = 2.0 * uni() - 1.0;
        k5[i] = k4[i] - exp2(-40.0 * uni());
    }
    if (kind < 6) (uni() < 0.5 ? k4 : k5)[which] = __longlong_as_double(specials[kind]);
    else if (kind == 6) k4[which] = 1e200;
    else y4[which] = __longlong_as_double(0x7ff0000000000000ll);
    auto six = [](const double* v) { return KSC<double>{v[0], v[1], v[2], v[3], v[4], v[5]}; };
    const KAttempt<double> A{six(y4), six(k4), six(k5), 0.015625};
    double want = 0.0;
    for (int i = 0; i < 6; ++i)
        want = fmax(want, fabs(A.h6 * (k4[i] - k5[i])) / (double(1e-6f) * (1.0 + fmax(fabs(y[i]), fabs(y4[i])))));
    if (kind < 7) want = 1e30;
    const long long d = __double_as_longlong(error_norm_pos(six(y), A, 1e-6f)) - __double_as_longlong(want);
    count(NORM, kind < 7 ? d == 0 : d >= -8 && d <= 8);
}

#define CHECK(call)                                                                              \
    do {                                                                                         \
        const cudaError_t e_ = (call);                                                           \
        if (e_ != cudaSuccess) {                                                                 \
            std::fprintf(stderr, "%s:%d %s\n", __FILE__, __LINE__, cudaGetErrorString(e_));      \
            return 1;                                                                            \
        }                                                                                        \
    } while (0)

int main() {
    if (division_main() != 0) return 1;
    CHECK(cudaGetLastError());  // any launch or copy of it that was refused
    for (int ea : {-102, -30, 0, 60})
        for (int eb : {-60, -1, 0, 20}) {
            hard<<<(1 << 23) / 256, 256>>>(ea, eb);
            CHECK(cudaGetLastError());
        }
    for (int e : {-102, -80, 0, 100, 127}) {
        sixths<<<(1 << 23) / 256, 256>>>(e);
        CHECK(cudaGetLastError());
    }
    for (int e : {-300, -67, -1, 0, 1, 16, 300}) {
        newton<<<(1 << 23) / 256, 256>>>(e);
        CHECK(cudaGetLastError());
    }
    tiny<<<(1 << 22) / 256, 256>>>();
    CHECK(cudaGetLastError());
    roots<<<1, 32>>>();
    CHECK(cudaGetLastError());
    odd_norms<<<(1 << 20) / 256, 256>>>();
    CHECK(cudaGetLastError());
    CHECK(cudaDeviceSynchronize());
    unsigned long long miss[N_CHECKS], done[N_CHECKS], milli[2];
    CHECK(cudaMemcpyFromSymbol(miss, g_miss, sizeof(miss)));
    CHECK(cudaMemcpyFromSymbol(done, g_done, sizeof(done)));
    CHECK(cudaMemcpyFromSymbol(milli, g_milli, sizeof(milli)));
    for (int k = 0; k < N_CHECKS; ++k) std::printf("%llu %llu ", miss[k], done[k]);
    std::printf("%llu %llu\n", milli[0], milli[1]);
    return 0;
}
