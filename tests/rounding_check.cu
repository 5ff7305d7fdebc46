// Test program (built and run by tests/test_gpu_rounding.py): tests/division_check.cu
// with its launches and copies checked, x / 6 in FP64 and at the ends of
// the exponent range, and the exact errors of the FP64 reciprocal and root.  Every kernel counts what it compared.  Prints division_check's line, then mismatches,
// comparisons and worst errors (in thousandths of a unit in the last place).
#define main division_main
#include "division_check.cu"
#undef main

enum { SIXTH_F, SIXTH_D, N_CHECKS };
__device__ unsigned long long g_miss[N_CHECKS], g_done[N_CHECKS], g_milli[2];

__device__ __forceinline__ void count(int k, bool ok) {
    atomicAdd(&g_done[k], 1ull);
    if (!ok) atomicAdd(&g_miss[k], 1ull);
}
__device__ __forceinline__ bool bits_equal(float a, float b) { return __float_as_uint(a) == __float_as_uint(b); }
__device__ __forceinline__ bool bits_equal(double a, double b) {
    return __double_as_longlong(a) == __double_as_longlong(b);
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
    for (int e : {-102, -80, 0, 100, 127}) {
        sixths<<<(1 << 23) / 256, 256>>>(e);
        CHECK(cudaGetLastError());
    }
    for (int e : {-300, -67, -1, 0, 1, 16, 300}) {
        newton<<<(1 << 23) / 256, 256>>>(e);
        CHECK(cudaGetLastError());
    }
    CHECK(cudaDeviceSynchronize());
    unsigned long long miss[N_CHECKS], done[N_CHECKS], milli[2];
    CHECK(cudaMemcpyFromSymbol(miss, g_miss, sizeof(miss)));
    CHECK(cudaMemcpyFromSymbol(done, g_done, sizeof(done)));
    CHECK(cudaMemcpyFromSymbol(milli, g_milli, sizeof(milli)));
    for (int k = 0; k < N_CHECKS; ++k) std::printf("%llu %llu ", miss[k], done[k]);
    std::printf("%llu %llu\n", milli[0], milli[1]);
    return 0;
}
