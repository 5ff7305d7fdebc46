// singularity_gb300/csrc/sgx_diff_impl.cuh
//
// Kernels and launch helpers of the differentiable form and its adjoint,
// shared by sgx_diff.cu (the C ABI and the FP32 instantiations) and
// sgx_diff64.cu (the FP64 instantiations) so the two compile in parallel.
// Everything here has internal linkage; each translation unit instantiates
// only the precision it launches.  The method is described in sgx_diff.cu.
#pragma once

#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstdint>
#include <cstring>
#include <string>
#include <type_traits>

#include "sgx.h"
#include "sgx_context.hpp"
#include "sgx_adjoint.cuh"
#include "sgx_dual.cuh"

namespace {

using namespace sgxd;

// Steps between checkpoints.  Sparse (64): the adjoint recomputes each
// segment into thread-local memory (65 states, 2.3 KB a thread, which streams
// through L2 and DRAM).  Dense (10): the 11 states of a segment fit in shared
// memory for 16 resident warps per SM (11 x 9 values x 4 B x 128 threads =
// 50.7 KB a block, four blocks), at 6.4x the checkpoint bytes.  FP32 with the
// hand-derived reverse pass takes the dense form when its records fit the
// form's memory budget, everything else the sparse one.
constexpr int kCkSparse = 64;
constexpr int kCkDense = 10;
// Threads a block of the one-ray-a-thread kernels.  Blocks of 128 leave SMs
// idle when there are few rays: 24,576 rays are 192 of them on 152 SMs, and an
// SM with two runs twice as long as one with one.  One-warp blocks spread such
// a launch evenly.  Where the line lies (128 against 32 threads, ms on one
// GB300): forward FP32 65,536 rays 0.53 / 0.46, 131,072 rays 0.72 / 0.66,
// 262,144 1.05 / 1.04, 524,288 1.73 / 1.73; FP64 65,536 rays 18.2 / 13.9, 131,072
// 27.4 / 27.5; backward FP64 8,192 rays 13.1 / 12.4, 32,768 21.1 / 18.6, 65,536
// 32.1 / 33.3; FP32 64-step checkpoints 262,144 rays 1.97 / 2.01, 1,048,576
// crossings 5.27 / 5.31.  The FP32 backward over 10-step checkpoints runs one-warp
// blocks at every size, since the next block need not wait for the slowest of
// four warps: slab 65,536 rays 0.75 / 0.58, 1,048,576 6.06 / 5.75, 2,097,152 14.1 /
// 13.4, crossings 1,048,576 5.01 / 4.84.
constexpr int kThreads = 128, kSmallThreads = 32;
constexpr std::uint64_t kSmallForward = 1u << 18, kSmallBackward = 1u << 16;  // fewer rays: one-warp blocks
// Warps an SM has to hold in the backward kernels (their comment says why).
template <class T, bool SLAB, bool DUALJ, int CK>
constexpr int kBackwardWarps = sizeof(T) == 8 || DUALJ ? 8 : CK == kCkDense ? 10 : SLAB ? 12 : 16;
constexpr std::uint64_t kOneWaveRaysPerSm = 8 * 32;  // rays that 8 warps hold at once
constexpr int kMaxCross = 8;  // crossings recorded per ray (crossing model)
constexpr int NS = 8;         // state: r, theta, phi, p_r, p_theta, psi (swept angle), sin(theta), cos(theta)
constexpr int NC = NS + 1;    // checkpoint: state and transmittance

template <class T> struct DiffConst {
    T M, dcam, aspect, tanh_, width_f, height_f;
    T r_out, peak_T, escape_r, h, exposure, turbulence, time_sec;
    T eps, fade_start, fade_width, H, kappa;
    std::uint32_t width, height, spp, max_steps, flags, fade;
};

template <class T> struct DiffParamsT {
    T spin, incl, r_in, t_scale;
};

// SoA views of the per-ray buffers.
template <class T> struct DiffBufs {
    std::uint64_t n;  // rays
    std::uint32_t slots;
    T* ckpt;          // [slots][NC][n]
    T* hdr;           // [3][n]
    std::uint32_t* nsteps;
    std::uint32_t* ncross;  // crossings (crossing model) or emitting steps (slab)
    std::uint32_t* xk;  // [kMaxCross][n]: crossing steps; slab: [0] = last emitting step
    T* xw;              // [kMaxCross][n]
    T* xc;              // [kMaxCross][3][n]
    T* xs;              // [kMaxCross][7][n]: r, theta, psi before and r, theta, phi, psi after the crossing step
                        // (nullptr: not kept, the sweep forms a crossing's seeds from the states it rebuilds)
    double* grads;      // [4][n]
    const T* ox;        // [spp] sub-pixel offsets
    const T* oy;
    unsigned long long* overflow;  // [0] dropped crossings, [1] steps of all rays
};

template <class S> __device__ __forceinline__ S selv(bool c, const S& a, const S& b) { return c ? a : b; }

// 1/x of the right-hand side: the SFU reciprocal in FP32, rcp_newton in FP64
// (sgxa::hrcp alike), a division for dual numbers.
template <class S> __device__ __forceinline__ S rcp_g(const S& x) {
    if constexpr (std::is_same_v<S, float>) return DM<float>::rcp_fast(x);
    else if constexpr (std::is_same_v<S, double>) return rcp_newton(x);
    else {
        using T = decltype(value_of(x));
        return S(T(1)) / x;
    }
}

template <class S> __device__ __forceinline__ S smooth01(const S& x) {
    using T = decltype(value_of(x));
    if (value_of(x) <= T(0)) return S(T(0));
    if (value_of(x) >= T(1)) return S(T(1));
    return x * x * (S(T(3)) - S(T(2)) * x);
}

// Kerr Hamiltonian right-hand side (kerr_hamilton.h:97-155) in Carter's
// separated form, generic in the scalar, with sin(theta), cos(theta) read from
// the state (y[6], y[7]); d[0..6] = dr, dtheta, dphi, dp_r, dp_theta, ds, dc.
// Operation for operation sgxa::rhs7 (sgx_adjoint.cuh), which states the
// equations.
template <class S, class T>
__device__ __forceinline__ void rhs_g7(const S* y, const S& E, const S& L, const S& a, T M, S* d) {
    if constexpr (std::is_same_v<S, double>) return sgxa::rhs7<double>(y, E, L, a, M, d);
    const S& st = y[6];
    const S& ct = y[7];
    const S r = y[0];
    const S a2 = a * a;
    const S s2 = st * st;
    const S safe_s2 = selv(value_of(s2) < T(1e-10), S(T(1e-10)), s2);
    const S r2 = r * r;
    const S r2a2 = r2 + a2;
    const S Sigma = r2 + a2 * (ct * ct);
    const S Delta = r2a2 - S(T(2) * M) * r;
    const S aE = a * E;
    const S P = r2a2 * E - a * L;
    const S W = L - aE * s2;
    const S iS = rcp_g(Sigma);
    const S iD = rcp_g(Delta);
    const S is2 = rcp_g(safe_s2);
    const S Q = P * iD, U = W * is2;
    d[0] = Delta * y[3] * iS;
    d[1] = y[4] * iS;
    d[2] = (a * Q + U) * iS;
    const S pr2 = y[3] * y[3];
    const S N = ((Delta * pr2 + y[4] * y[4]) - P * Q) + W * U;
    const S NiS = N * iS;
    d[3] = (r * NiS + ((S(M) - r) * (Q * Q + pr2) + (S(T(2)) * E * r) * Q)) * iS;
    d[4] = -(iS * (st * ct)) * (a2 * NiS - U * (S(T(2)) * aE + U));
    d[5] = ct * d[1];
    d[6] = -(st * d[1]);
}

// One fixed RK4 step with the reference's pole damping, plus the swept angle;
// (sin theta, cos theta) integrated with the state and put back on the unit
// circle by n = 3/2 - (s^2 + c^2)/2.  Operation for operation sgxa::step.
template <class S, class T>
__device__ __forceinline__ void step_g(const S* y, const S& E, const S& L, const S& a, T M, T h, bool fade, S* o) {
    const S st0 = y[6];
    S ps = selv(value_of(st0) < T(0), -st0, st0) * S(T(5));
    ps = selv(value_of(ps) > T(1), S(T(1)), selv(value_of(ps) < T(0.05), S(T(0.05)), ps));
    const S he = S(h) * ps;
    const S hh = S(T(0.5)) * he;
    S k1[7], k2[7], k3[7], k4[7], t[NS];
    t[5] = y[5];
    if constexpr (std::is_same_v<S, float>) {
        // FP32: the same fused multiply-adds on pairs of state slots (0, 1),
        // (2, 3), (6, 7) (derivative slots (0, 1), (2, 3), (5, 6)), slot 4 alone
        auto axpy = [&](const float* k, float f) {
            const F2 ff = f2(f, f);
            unf2(fma2(f2(k[0], k[1]), ff, f2(y[0], y[1])), t[0], t[1]);
            unf2(fma2(f2(k[2], k[3]), ff, f2(y[2], y[3])), t[2], t[3]);
            unf2(fma2(f2(k[5], k[6]), ff, f2(y[6], y[7])), t[6], t[7]);
            t[4] = fmaf(k[4], f, y[4]);
        };
        rhs_g7(y, E, L, a, M, k1);
        axpy(k1, hh);
        rhs_g7(t, E, L, a, M, k2);
        axpy(k2, hh);
        rhs_g7(t, E, L, a, M, k3);
        axpy(k3, he);
        rhs_g7(t, E, L, a, M, k4);
        const float h6 = sixth(he);
        const F2 two = f2(2.0f, 2.0f), hp = f2(h6, h6);
        auto comb = [&](int i, int j, int si, int sj) {
            const F2 sum = add2(fma2(f2(k2[i], k2[j]), two, f2(k1[i], k1[j])),
                                fma2(f2(k3[i], k3[j]), two, f2(k4[i], k4[j])));
            unf2(fma2(sum, hp, f2(y[si], y[sj])), o[si], o[sj]);
        };
        comb(0, 1, 0, 1);
        comb(2, 3, 2, 3);
        comb(5, 6, 6, 7);
        o[4] = fmaf(fmaf(k2[4], 2.0f, k1[4]) + fmaf(k3[4], 2.0f, k4[4]), h6, y[4]);
    } else {
        rhs_g7(y, E, L, a, M, k1);
#pragma unroll
        for (int i = 0; i < 7; ++i) t[sgxa::sidx(i)] = y[sgxa::sidx(i)] + k1[i] * hh;
        rhs_g7(t, E, L, a, M, k2);
#pragma unroll
        for (int i = 0; i < 7; ++i) t[sgxa::sidx(i)] = y[sgxa::sidx(i)] + k2[i] * hh;
        rhs_g7(t, E, L, a, M, k3);
#pragma unroll
        for (int i = 0; i < 7; ++i) t[sgxa::sidx(i)] = y[sgxa::sidx(i)] + k3[i] * he;
        rhs_g7(t, E, L, a, M, k4);
        if constexpr (std::is_same_v<S, double>) {
            S ks[7];
            const S h6 = sixth(he);
            sgxa::ksum7(k1, k2, k3, k4, ks);
#pragma unroll
            for (int i = 0; i < 7; ++i) o[sgxa::sidx(i)] = y[sgxa::sidx(i)] + ks[i] * h6;
        } else {
            const S h6 = he / S(T(6));
#pragma unroll
            for (int i = 0; i < 7; ++i)
                o[sgxa::sidx(i)] = y[sgxa::sidx(i)] + ((k1[i] + k2[i] * S(T(2))) + (k3[i] * S(T(2)) + k4[i])) * h6;
        }
    }
    const S n = S(T(1.5)) - S(T(0.5)) * (o[6] * o[6] + o[7] * o[7]);
    o[6] = o[6] * n;
    o[7] = o[7] * n;
    if (fade) {
        const S dth = o[1] - y[1], dph = o[2] - y[2], st = o[6];
        o[5] = y[5] + DM<S>::sqrt_(dth * dth + st * st * dph * dph);
    } else {
        o[5] = y[5];
    }
}

// Blackbody colour continuous at 6600 K (the fit of geodesic_kernel.cu:77-104
// jumps there when it switches branch): the low (t <= 66) and high branch,
// t = temperature / 100 K, blended by S((t - 65) / 2); identical outside.
template <class S> __device__ __forceinline__ V3<S> blackbody_c0(const S& temp) {
    using T = decltype(value_of(temp));
    const S t = clampv(temp, S(T(1000)), S(T(40000))) * S(DM<T>::lit(0.01f, 0.01));
    const T tv = value_of(t);
    V3<S> lo, hi;
    const bool need_lo = tv < T(67), need_hi = tv > T(65);
    if (need_lo) {
        lo.x = S(T(1));
        lo.y = clampv(S(DM<T>::lit(0.39008157876901960784f, 0.39008157876901960784)) * DM<S>::log_(t) -
                          S(DM<T>::lit(0.63184144378862745098f, 0.63184144378862745098)),
                      S(T(0)), S(T(1)));
        lo.z = tv <= T(19) ? S(T(0))
                           : clampv(S(DM<T>::lit(0.54320678911019607843f, 0.54320678911019607843)) *
                                            DM<S>::log_(t - S(T(10))) -
                                        S(DM<T>::lit(1.19625408914f, 1.19625408914)),
                                    S(T(0)), S(T(1)));
    }
    if (need_hi) {
        const S t1 = t - S(T(60));
        hi.x = clampv(S(DM<T>::lit(1.29293618606274509804f, 1.29293618606274509804)) *
                          DM<S>::pow_(t1, S(DM<T>::lit(-0.1332047592f, -0.1332047592))),
                      S(T(0)), S(T(1)));
        hi.y = clampv(S(DM<T>::lit(1.12989086089529411765f, 1.12989086089529411765)) *
                          DM<S>::pow_(t1, S(DM<T>::lit(-0.0755148492f, -0.0755148492))),
                      S(T(0)), S(T(1)));
        hi.z = S(T(1));
    }
    if (!need_hi) return lo;
    if (!need_lo) return hi;
    const S sb = smooth01((t - S(T(65))) * S(T(0.5)));
    return mk3(lo.x + sb * (hi.x - lo.x), lo.y + sb * (hi.y - lo.y), lo.z + sb * (hi.z - lo.z));
}

// Disc colour at a crossing (geodesic_kernel.cu:368-393 with blackbody_c0),
// generic in the scalar.
template <class S, class T>
__device__ __forceinline__ void disc_colour_g(const S& r_c, const S& ph, const S& L, const S& a, const S& r_in,
                                              const S& T_local, const DiffConst<T>& k, S* col) {
    const T M = k.M;
    const S f_emit = S(T(1)) - S(T(2) * M) / r_c;
    const T f_obs = T(1) - T(2) * M / k.dcam;
    S g_grav = S(T(1));
    if (k.flags & SGX_FLAG_REDSHIFT_ON)
        g_grav = DM<S>::sqrt_(DM<S>::fmax_(f_emit, S(T(1e-6))) / S(f_obs > T(1e-6) ? f_obs : T(1e-6)));
    S g_dop = S(T(1));
    if (k.flags & SGX_FLAG_DOPPLER_ON) {
        const S om0 = DM<S>::sqrt_(S(M) / (r_c * r_c * r_c));
        const S omega_K = om0 / (S(T(1)) + a * om0);
        const S vel = r_c * omega_K / DM<S>::sqrt_(DM<S>::fmax_(f_emit, S(T(1e-6))));
        const S cos_psi = clampv(L / r_c, S(T(-1)), S(T(1)));
        g_dop = DM<S>::sqrt_(DM<S>::fmax_(S(T(1)) - vel * vel, S(T(0)))) /
                DM<S>::fmax_(S(T(1)) - vel * cos_psi, S(T(1e-4)));
    }
    const S g = g_grav * g_dop;
    const V3<S> bb = blackbody_c0(g * T_local);
    const S flux = clampv(DM<S>::pow_(r_in / r_c, S(T(3))), S(T(0.05)), S(T(1.5)));
    const S bands = disc_band_mask(r_c, ph, r_in, S(k.turbulence), S(k.time_sec));
    const S g2 = g * g;
    const S kk = flux * bands * g2 * g2;
    col[0] = bb.x * kk;
    col[1] = bb.y * kk;
    col[2] = bb.z * kk;
}

// Crossing between states y0 (step k-1) and y1 (step k): weight and colour.
template <class S, class T>
__device__ __forceinline__ void crossing_g(const S& r0, const S& th0, const S& psi0, const S& r1, const S& th1,
                                           const S& ph1, const S& psi1, const S& L, const S& a, const S& r_in,
                                           const S& t_scale, const DiffConst<T>& k, S* col, S& w) {
    const S mid = S(T(1.5707963267948966));
    const S frac = (mid - th0) / (th1 - th0);
    const S r_c = r0 + frac * (r1 - r0);
    w = smooth01((r_c - r_in) / S(k.eps)) * smooth01((S(k.r_out) - r_c) / S(k.eps));
    if (k.fade) {
        const S psi_c = psi0 + frac * (psi1 - psi0);
        w = w * (S(T(1)) - smooth01((psi_c - S(k.fade_start)) / S(k.fade_width)));
    }
    const S T_local = disc_temperature(r_c, r_in, S(k.peak_T) * t_scale);
    if (value_of(T_local) > T(0)) {
        disc_colour_g(r_c, ph1, L, a, r_in, T_local, k, col);
    } else {
        col[0] = col[1] = col[2] = S(T(0));
    }
}

// Camera ray and canonical initial state at pixel (gx, gy) with offset (ox, oy).
template <class S, class T>
__device__ __forceinline__ bool init_g(const S& a, const S& incl, const DiffConst<T>& k, std::uint32_t gx,
                                       std::uint32_t gy, T ox, T oy, S* y, S& E, S& L) {
    S si, ci;
    DM<S>::sincos_(incl, &si, &ci);
    const T fx = T(float(gx)) + ox, fy = T(float(gy)) + oy;
    const T u_ndc = (T(2) * fx / k.width_f - T(1)) * k.aspect * k.tanh_;
    const T v_ndc = -(T(2) * fy / k.height_f - T(1)) * k.tanh_;
    // forward (-sin i, 0, -cos i) + right (0, 1, 0) u + up (cos i, 0, -sin i) v
    S dx = -si + ci * S(v_ndc);
    S dy = S(u_ndc);
    S dz = -ci - si * S(v_ndc);
    const S len = DM<S>::fmax_(DM<S>::sqrt_(dx * dx + dy * dy + dz * dz), S(T(1e-20)));
    const S ik = S(T(1)) / len;
    dx = dx * ik;
    dy = dy * ik;
    dz = dz * ik;
    const S ur = dx * si + dz * ci;
    const S uth = (dx * ci - dz * si) / S(k.dcam);
    const S uph = dy / (S(k.dcam) * DM<S>::fmax_(si, S(T(1e-6))));
    const S r = S(k.dcam);
    const S M = S(k.M);
    const S s2 = si * si;
    const S Sigma = r * r + a * a * ci * ci;
    const S Delta = r * r - S(T(2)) * M * r + a * a;
    const S g_tt = -(S(T(1)) - S(T(2)) * M * r / Sigma);
    const S g_tp = S(T(-2)) * M * r * a * s2 / Sigma;
    const S g_rr = Sigma / Delta;
    const S g_pp = s2 * ((r * r + a * a) * (r * r + a * a) - a * a * Delta * s2) / Sigma;
    const S B = S(T(2)) * g_tp * uph;
    const S C = g_rr * ur * ur + Sigma * uth * uth + g_pp * uph * uph;
    const S disc = B * B - S(T(4)) * g_tt * C;
    if (value_of(disc) < T(0)) return false;
    const S ut = (-B - DM<S>::sqrt_(disc)) / (S(T(2)) * g_tt);
    E = -(g_tt * ut + g_tp * uph);
    L = g_tp * ut + g_pp * uph;
    y[0] = r;
    y[1] = incl;
    y[2] = S(T(0));
    y[3] = g_rr * ur;
    y[4] = Sigma * uth;
    y[5] = S(T(0));
    y[6] = si;
    y[7] = ci;
    return true;
}

// Height z certainly outside the emitting layer: |z| beyond H by more than the
// rounding of (z / H)^2 < 1, so the test's division is left to the few steps in
// and at the layer.
template <class T> __device__ __forceinline__ bool outside_layer(T z, const DiffConst<T>& k) {
    return absv(z) > k.H * T(1.001);
}

// Slab emission of the step y0 -> y1, evaluated at y1, in two parts: the
// absorption alpha (false, alpha = 0, outside the layer, the annulus or past
// the fade) and the colour.  The colour depends on (r1, ph1, L, a, r_in,
// t_scale) only, so the adjoint differentiates the parts over their own
// inputs (10 and 6 dual lanes instead of 13).
template <class S, class T>
__device__ __forceinline__ bool slab_alpha_g(const S& r0, const S& th0, const S& ph0, const S& r1, const S& th1,
                                             const S& ph1, const S& psi1, const S& s1, const S& c1, const S& r_in,
                                             const DiffConst<T>& k, S& alpha) {
    const S z = r1 * c1;
    if (outside_layer(value_of(z), k)) return false;
    const S q = z / S(k.H);
    if (!(value_of(q) * value_of(q) < T(1))) return false;
    S w = smooth01((r1 - r_in) / S(k.eps)) * smooth01((S(k.r_out) - r1) / S(k.eps));
    if (k.fade) w = w * (S(T(1)) - smooth01((psi1 - S(k.fade_start)) / S(k.fade_width)));
    if (!(value_of(w) > T(0))) return false;
    const S b = S(T(1)) - q * q;
    const S rho = b * b;
    const S dr = r1 - r0, dth = th1 - th0, dph = ph1 - ph0;
    const S ds = DM<S>::sqrt_(dr * dr + r1 * r1 * (dth * dth + s1 * s1 * dph * dph));
    alpha = w * (S(T(1)) - DM<S>::exp_(-(S(k.kappa) * rho * ds)));
    return true;
}

template <class S, class T>
__device__ __forceinline__ void slab_colour_g(const S& r1, const S& ph1, const S& L, const S& a, const S& r_in,
                                              const S& t_scale, const DiffConst<T>& k, S* col) {
    const S T_local = disc_temperature(r1, r_in, S(k.peak_T) * t_scale);
    if (value_of(T_local) > T(0)) {
        disc_colour_g(r1, ph1, L, a, r_in, T_local, k, col);
    } else {
        col[0] = col[1] = col[2] = S(T(0));
    }
}

template <class S, class T>
__device__ __forceinline__ bool slab_g(const S& r0, const S& th0, const S& ph0, const S& r1, const S& th1,
                                       const S& ph1, const S& psi1, const S& s1, const S& c1, const S& L,
                                       const S& a, const S& r_in, const S& t_scale, const DiffConst<T>& k, S* col,
                                       S& alpha) {
    if (!slab_alpha_g(r0, th0, ph0, r1, th1, ph1, psi1, s1, c1, r_in, k, alpha)) return false;
    slab_colour_g(r1, ph1, L, a, r_in, t_scale, k, col);
    return true;
}

// Reverse passes of the emission, derived by hand: values and gradients from
// one evaluation.  (On dual numbers the colour carries six derivative lanes and
// the absorption ten through every operation, next to a separate evaluation of
// the values; that form stays as the cross-check.)  At the ends of a clamped
// range the derivative is the inner one, as for the duals.  With the regrouped
// rhs_vjp7_at, backward pass of 1,048,576 rays: slab FP32 6.7 -> 6.0 ms; crossing
// model, whose seeds also leave the divergent sweep, 255 x 193 forward and
// backward 2.15 -> 1.53 ms.

// S(x) = 3x^2 - 2x^3 and S'(x) of x clamped to [0, 1].
template <class T> __device__ __forceinline__ T smooth01_d(T x, T& dS) {
    if (x <= T(0) || x >= T(1)) {
        dS = T(0);
        return x <= T(0) ? T(0) : T(1);
    }
    dS = T(6) * x * (T(1) - x);
    return x * x * (T(3) - T(2) * x);
}

template <class T> __device__ __forceinline__ T clamp_d(T x, T lo, T hi, T& dx) {
    dx = (x < lo || x > hi) ? T(0) : T(1);
    return clampv(x, lo, hi);
}

// blackbody_c0 and its derivative by temperature.
template <class T> __device__ __forceinline__ void blackbody_c0_d(T temp, T* c, T* dc) {
    T in;
    const T t = clamp_d(temp, T(1000), T(40000), in) * DM<T>::lit(0.01f, 0.01);
    in *= DM<T>::lit(0.01f, 0.01);
    const bool need_lo = t < T(67), need_hi = t > T(65);
    T lo[3], dlo[3], hi[3], dhi[3], u;
    if (need_lo) {
        const T kg = DM<T>::lit(0.39008157876901960784f, 0.39008157876901960784);
        const T kb = DM<T>::lit(0.54320678911019607843f, 0.54320678911019607843);
        lo[0] = T(1);
        dlo[0] = T(0);
        lo[1] = clamp_d(kg * DM<T>::log_(t) - DM<T>::lit(0.63184144378862745098f, 0.63184144378862745098), T(0), T(1), u);
        dlo[1] = u * kg / t;
        lo[2] = dlo[2] = T(0);
        if (t > T(19)) {
            lo[2] = clamp_d(kb * DM<T>::log_(t - T(10)) - DM<T>::lit(1.19625408914f, 1.19625408914), T(0), T(1), u);
            dlo[2] = u * kb / (t - T(10));
        }
    }
    if (need_hi) {
        const T t1 = t - T(60), er = DM<T>::lit(-0.1332047592f, -0.1332047592), eg = DM<T>::lit(-0.0755148492f, -0.0755148492);
        const T pr = DM<T>::lit(1.29293618606274509804f, 1.29293618606274509804) * DM<T>::pow_(t1, er);
        const T pg = DM<T>::lit(1.12989086089529411765f, 1.12989086089529411765) * DM<T>::pow_(t1, eg);
        hi[0] = clamp_d(pr, T(0), T(1), u);
        dhi[0] = u * er * pr / t1;
        hi[1] = clamp_d(pg, T(0), T(1), u);
        dhi[1] = u * eg * pg / t1;
        hi[2] = T(1);
        dhi[2] = T(0);
    }
    T dS = T(0);
    const T S = need_lo ? (need_hi ? smooth01_d((t - T(65)) * T(0.5), dS) : T(0)) : T(1);
    dS *= T(0.5);
#pragma unroll
    for (int i = 0; i < 3; ++i) {
        if (!need_hi) {
            c[i] = lo[i];
            dc[i] = in * dlo[i];
        } else if (!need_lo) {
            c[i] = hi[i];
            dc[i] = in * dhi[i];
        } else {
            c[i] = lo[i] + S * (hi[i] - lo[i]);
            dc[i] = in * (dlo[i] + S * (dhi[i] - dlo[i]) + dS * (hi[i] - lo[i]));
        }
    }
}

// Disc colour at radius r, azimuth ph (disc_temperature and disc_colour_g):
// col[3], and grad[0..5] = w . d col / d(r, ph, L, a, r_in, t_scale).
template <class T>
__device__ __forceinline__ void colour_vjp(T r, T ph, T L, T a, T r_in, T t_scale, const DiffConst<T>& k, const T* w,
                                           T* col, T* grad) {
#pragma unroll
    for (int i = 0; i < 6; ++i) grad[i] = T(0);
    const T peak = k.peak_T * t_scale;
    const T T_local = disc_temperature(r, r_in, peak);
    if (!(T_local > T(0))) {
        col[0] = col[1] = col[2] = T(0);
        return;
    }
    T r_b = T(0), rin_b = T(0), L_b = T(0), a_b = T(0), x_b = T(0);
    const T x = r_in / r, rx = r / r_in;
    // redshift and Doppler
    const T f_emit = T(1) - T(2) * k.M / r, f_obs = T(1) - T(2) * k.M / k.dcam;
    const T fe = DM<T>::fmax_(f_emit, T(1e-6)), fo = f_obs > T(1e-6) ? f_obs : T(1e-6);
    const bool red = (k.flags & SGX_FLAG_REDSHIFT_ON) != 0u, dop = (k.flags & SGX_FLAG_DOPPLER_ON) != 0u;
    const T gg = red ? DM<T>::sqrt_(fe / fo) : T(1);
    T gd = T(1), om0, den1, omK, se, vel, cp, dcp, g1, sg, dn, dnin;
    if (dop) {
        om0 = DM<T>::sqrt_(k.M / (r * r * r));
        den1 = T(1) + a * om0;
        omK = om0 / den1;
        se = DM<T>::sqrt_(fe);
        vel = r * omK / se;
        cp = clamp_d(L / r, T(-1), T(1), dcp);
        g1 = T(1) - vel * vel;
        sg = DM<T>::sqrt_(DM<T>::fmax_(g1, T(0)));
        dn = clamp_d(T(1) - vel * cp, T(1e-4), T(1e30), dnin);
        gd = sg / dn;
    }
    const T g = gg * gd;
    T bb[3], dbb[3];
    blackbody_c0_d(g * T_local, bb, dbb);
    // flux and bands
    const T fl0 = DM<T>::pow_(x, T(3));
    T dfl;
    const T fl = clamp_d(fl0, T(0.05), T(1.5), dfl);
    T drm;
    const T rm = clamp_d(rx, T(0.1), T(1e30), drm);
    const T rho = DM<T>::log_(rm), p15 = DM<T>::pow_(rx, T(1.5)), om = DM<T>::pow_(rm, T(-1.5));
    T dsh;
    const T shd = clamp_d(p15, T(0.25), T(1e30), dsh);
    const T kt = T(0.8) * k.time_sec;
    const T pa = ph - kt * om;
    T s1, c1, s2, c2;
    DM<T>::sincos_(T(10) * rho + T(3) * pa + T(4) / shd, &s1, &c1);
    DM<T>::sincos_(T(22) * rho - DM<T>::lit(1.7f, 1.7) * pa, &s2, &c2);
    const T b1 = T(0.5) + T(0.5) * c1, b2 = T(0.5) + T(0.5) * c2;
    const T comb = DM<T>::lit(0.8f, 0.8) + k.turbulence * (b1 * b1 * b2 - DM<T>::lit(0.8f, 0.8));
    T dbd;
    const T bd = clamp_d(DM<T>::lit(0.65f, 0.65) + DM<T>::lit(0.55f, 0.55) * comb, T(0), DM<T>::lit(1.3f, 1.3), dbd);
    const T g2 = g * g, g4 = g2 * g2, kk = fl * bd * g4;
    T kk_b = T(0), tc_b = T(0);
#pragma unroll
    for (int i = 0; i < 3; ++i) {
        col[i] = bb[i] * kk;
        kk_b += w[i] * bb[i];
        tc_b += w[i] * kk * dbb[i];
    }
    // reverse: kk = fl bd g^4, colour temperature g T
    const T g_b = kk_b * fl * bd * (T(4) * g2 * g) + tc_b * T_local;
    const T T_b = tc_b * g;
    // T = peak q edge / 0.186, q = x^(3/4), edge = 1 - sqrt(x) (> 0 here)
    const T sx = DM<T>::sqrt_(x);
    x_b += T_b * T_local * (T(0.75) / x - T(0.5) / (sx * (T(1) - sx)));
    x_b += dfl * kk_b * bd * g4 * (T(3) * fl0 / x);
    // bands
    const T comb_b = kk_b * fl * g4 * dbd * DM<T>::lit(0.55f, 0.55) * k.turbulence;
    const T A1_b = -(comb_b * b1 * b2) * s1, A2_b = -(T(0.5) * comb_b * b1 * b1) * s2;
    const T pa_b = T(3) * A1_b - DM<T>::lit(1.7f, 1.7) * A2_b;
    const T rx_b = drm * ((T(10) * A1_b + T(22) * A2_b) / rm + pa_b * kt * (T(1.5) * om / rm)) -
                   dsh * A1_b * T(4) / (shd * shd) * (T(1.5) * p15 / rx);
    // Doppler and redshift
    T fe_b = T(0);
    if (dop) {
        const T gd_b = g_b * gg;
        const T dn_b = -dnin * gd_b * gd / dn;
        T vel_b = -dn_b * cp;
        const T cp_b = -dcp * dn_b * vel;
        if (sg > T(0)) vel_b -= gd_b / dn * vel / sg;
        L_b += cp_b / r;
        r_b -= cp_b * L / (r * r);
        const T omK_b = vel_b * r / se;
        const T om0_b = omK_b / (den1 * den1);
        a_b -= omK_b * omK * omK;
        r_b += vel_b * omK / se - om0_b * T(1.5) * om0 / r;
        fe_b -= vel_b * vel * T(0.5) / fe;
    }
    if (red) fe_b += g_b * gd * T(0.5) * gg / fe;
    if (!(f_emit < T(1e-6))) r_b += fe_b * T(2) * k.M / (r * r);
    r_b += rx_b / r_in - x_b * x / r;
    rin_b += x_b / r - rx_b * rx / r_in;
    grad[0] = r_b;
    grad[1] = pa_b;
    grad[2] = L_b;
    grad[3] = a_b;
    grad[4] = rin_b;
    grad[5] = T_b * T_local / t_scale;
}

// Absorption alpha of the slab step (slab_alpha_g) and grad[0..9] = d alpha /
// d(r0, th0, ph0, r1, th1, ph1, psi1, s1, c1, r_in); false outside the layer.
template <class T>
__device__ __forceinline__ bool slab_alpha_d(T r0, T th0, T ph0, T r1, T th1, T ph1, T psi1, T s1, T c1, T r_in,
                                             const DiffConst<T>& k, T& alpha, T* grad) {
    const T z = r1 * c1;
    if (outside_layer(z, k)) return false;
    const T q = z / k.H;
    if (!(q * q < T(1))) return false;
    T dA, dB, dF = T(0), F = T(1);
    const T A = smooth01_d((r1 - r_in) / k.eps, dA), B = smooth01_d((k.r_out - r1) / k.eps, dB);
    if (k.fade) F = T(1) - smooth01_d((psi1 - k.fade_start) / k.fade_width, dF);
    const T w = A * B * F;
    if (!(w > T(0))) return false;
    const T b = T(1) - q * q, rho = b * b;
    const T dr = r1 - r0, dth = th1 - th0, dph = ph1 - ph0;
    const T an2 = dth * dth + s1 * s1 * dph * dph;
    const T ds = DM<T>::sqrt_(dr * dr + r1 * r1 * an2);
    const T ex = DM<T>::exp_(-(k.kappa * rho * ds));
    alpha = w * (T(1) - ex);
    const T t = w * k.kappa * ex;           // d alpha / d(rho ds)
    const T q_b = t * ds * T(-4) * q * b;   // by q = r1 c1 / H
    const T i_b = ds > T(0) ? t * rho / ds : T(0);
    const T m = T(1) - ex;
    const T rr = r1 * r1 * i_b;
    grad[0] = -dr * i_b;
    grad[1] = -rr * dth;
    grad[2] = -rr * s1 * s1 * dph;
    grad[3] = m * F * (dA * B - A * dB) / k.eps + q_b * c1 / k.H + (dr + r1 * an2) * i_b;
    grad[4] = rr * dth;
    grad[5] = rr * s1 * s1 * dph;
    grad[6] = k.fade ? -m * A * B * dF / k.fade_width : T(0);
    grad[7] = rr * s1 * dph * dph;
    grad[8] = q_b * r1 / k.H;
    grad[9] = -m * F * dA * B / k.eps;
    return true;
}

// Crossing (crossing_g): its gradient q[0..10] = (xcs g . d colour + xgw d w) /
// d(r0, th0, psi0, r1, th1, ph1, psi1, L, a, r_in, t_scale).
template <class T>
__device__ __forceinline__ void crossing_vjp(T r0, T th0, T psi0, T r1, T th1, T ph1, T psi1, T L, T a, T r_in,
                                             T t_scale, const DiffConst<T>& k, const T* g, T xcs, T xgw, T* q) {
    const T mid = T(1.5707963267948966);
    const T id = T(1) / (th1 - th0);
    const T frac = (mid - th0) * id;
    const T r_c = r0 + frac * (r1 - r0);
    T dA, dB, dF = T(0), F = T(1);
    const T A = smooth01_d((r_c - r_in) / k.eps, dA), B = smooth01_d((k.r_out - r_c) / k.eps, dB);
    if (k.fade) F = T(1) - smooth01_d((psi0 + frac * (psi1 - psi0) - k.fade_start) / k.fade_width, dF);
    T col[3], gr[6];
    const T w[3] = {xcs * g[0], xcs * g[1], xcs * g[2]};
    colour_vjp(r_c, ph1, L, a, r_in, t_scale, k, w, col, gr);
    const T rc_b = gr[0] + xgw * F * (dA * B - A * dB) / k.eps;
    const T pc_b = k.fade ? -xgw * A * B * dF / k.fade_width : T(0);
    const T fr_b = rc_b * (r1 - r0) + pc_b * (psi1 - psi0);
    q[0] = rc_b * (T(1) - frac);
    q[1] = fr_b * (frac - T(1)) * id;
    q[2] = pc_b * (T(1) - frac);
    q[3] = rc_b * frac;
    q[4] = -fr_b * frac * id;
    q[5] = gr[1];
    q[6] = pc_b * frac;
    q[7] = gr[2];
    q[8] = gr[3];
    q[9] = gr[4] - xgw * F * dA * B / k.eps;
    q[10] = gr[5];
}

// Capture radius of the form: the prograde equatorial photon orbit radius
// (the smallest photon orbit: an ingoing ray from outside that gets inside it
// falls in) less 0.05 M, at least the reference's 1.02 r_+.  Closer to the
// horizon the fixed-step RK4 turns unstable (p_r ~ 1/Delta) and a blown-up
// state could emit.
template <class T> __device__ __forceinline__ T capture_radius(T M, T a) {
    const T r_pro = T(2) * M * (T(1) + DM<T>::cos_(T(2) / T(3) * DM<T>::acos_(-a / M)));
    const T hcut = DM<T>::lit(1.02f, 1.02) * (M + DM<T>::sqrt_(DM<T>::fmax_(M * M - a * a, T(0))));
    return DM<T>::fmax_(r_pro - DM<T>::lit(0.05f, 0.05) * M, hcut);
}

template <class T>
__device__ __forceinline__ void ray_pixel(const DiffConst<T>& k, std::uint64_t id, std::uint32_t& gx, std::uint32_t& gy,
                                          std::uint32_t& s) {
    const std::uint64_t pix = id / k.spp;
    s = std::uint32_t(id - pix * k.spp);
    gy = std::uint32_t(pix / k.width);
    gx = std::uint32_t(pix - std::uint64_t(gy) * k.width);
}

template <class T, int CK>
__device__ __forceinline__ void store_ckpt(const DiffBufs<T>& b, std::uint64_t id, std::uint32_t n, const T* y, T tau) {
    const std::uint64_t base = std::uint64_t(n / CK) * NC * b.n + id;
#pragma unroll
    for (int i = 0; i < NS; ++i) b.ckpt[base + std::uint64_t(i) * b.n] = y[i];
    b.ckpt[base + std::uint64_t(NS) * b.n] = tau;
}

// Forward: one thread per ray.  SLAB: emission and absorption every step in
// the layer; otherwise soft crossings of the equatorial plane.
template <class T, bool SLAB, int CK>
__global__ void __launch_bounds__(128) diff_forward_kernel(DiffConst<T> k, DiffParamsT<T> p, DiffBufs<T> b) {
    const std::uint64_t id = std::uint64_t(blockIdx.x) * blockDim.x + threadIdx.x;
    std::uint32_t n = 0;
    if (id < b.n) {
        std::uint32_t gx, gy, s;
        ray_pixel(k, id, gx, gy, s);
        const T a = p.spin * k.M;
        const T r_in = p.r_in * k.M;
        T y[NS], prev[NS], E, L;
        T hdr[3] = {T(0), T(0), T(0)};
        std::uint32_t nc = 0, last = 0;
        if (init_g<T, T>(a, p.incl, k, gx, gy, b.ox[s], b.oy[s], y, E, L)) {
            const T hcut = capture_radius(k.M, a);
            const bool disc = (k.flags & SGX_FLAG_DISC_ON) != 0u;
            T tau = T(1);
#pragma unroll
            for (int i = 0; i < NS; ++i) prev[i] = y[i];
            for (; n < k.max_steps; ++n) {
                if (!SLAB && n % CK == 0) store_ckpt<T, CK>(b, id, n, y, tau);
                if (!isfinite(y[0]) || y[0] < hcut) break;
                if (y[0] > k.escape_r) break;
                if constexpr (SLAB) {
                    T col[3], alpha;
                    if (disc && n > 0 &&
                        slab_g<T, T>(prev[0], prev[1], prev[2], y[0], y[1], y[2], y[5], y[6], y[7], L, a, r_in,
                                     p.t_scale, k, col, alpha)) {
#pragma unroll
                        for (int c = 0; c < 3; ++c) hdr[c] = hdr[c] + tau * alpha * col[c];
                        tau = tau * (T(1) - alpha);
                        ++nc;
                        last = n;
                    }
                    if (n % CK == 0) store_ckpt<T, CK>(b, id, n, y, tau);
                } else {
                    const T mid = T(1.5707963267948966);
                    if (disc && n > 0 && ((prev[1] - mid) * (y[1] - mid) < T(0))) {
                        T col[3], w;
                        crossing_g<T, T>(prev[0], prev[1], prev[5], y[0], y[1], y[2], y[5], L, a, r_in, p.t_scale,
                                         k, col, w);
                        if (w > T(0)) {
                            if (nc < kMaxCross) {
                                b.xk[std::uint64_t(nc) * b.n + id] = n;
                                b.xw[std::uint64_t(nc) * b.n + id] = w;
#pragma unroll
                                for (int c = 0; c < 3; ++c) b.xc[(std::uint64_t(nc) * 3 + c) * b.n + id] = col[c];
                                if (b.xs != nullptr) {
                                    const T xs[7] = {prev[0], prev[1], prev[5], y[0], y[1], y[2], y[5]};
#pragma unroll
                                    for (int c = 0; c < 7; ++c) b.xs[(std::uint64_t(nc) * 7 + c) * b.n + id] = xs[c];
                                }
                            } else {
                                atomicAdd(b.overflow, 1ull);
                            }
                            ++nc;
#pragma unroll
                            for (int c = 0; c < 3; ++c) hdr[c] = hdr[c] + tau * w * col[c];
                            tau = tau * (T(1) - w);
                            if (!(tau > T(0))) break;
                        }
                    }
                }
                // outgoing beyond the disc, after this step's emission or crossing: a
                // photon outside the photon region moving out has no turning point
                // left, and nothing emits there (starfield off)
                if (y[3] > T(0) && y[0] > k.r_out) break;
#pragma unroll
                for (int i = 0; i < NS; ++i) prev[i] = y[i];
                step_g<T, T>(prev, E, L, a, k.M, k.h, k.fade != 0u, y);
            }
        }
#pragma unroll
        for (int c = 0; c < 3; ++c) b.hdr[std::uint64_t(c) * b.n + id] = hdr[c];
        b.nsteps[id] = n;
        if constexpr (SLAB) {
            b.ncross[id] = nc;
            b.xk[id] = last;
        } else {
            b.ncross[id] = nc < kMaxCross ? nc : kMaxCross;
        }
    }
    // steps of the launch, one atomic per warp
    unsigned long long v = n;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
    if ((threadIdx.x & 31u) == 0u) atomicAdd(b.overflow + 1, v);
}

// Per pixel: mean over samples of ACES(hdr * exposure) (geodesic_kernel.cu:482-503).
template <class T>
__global__ void diff_image_kernel(DiffConst<T> k, DiffBufs<T> b, float* img) {
    const std::uint64_t pix = std::uint64_t(blockIdx.x) * blockDim.x + threadIdx.x;
    if (pix >= std::uint64_t(k.width) * k.height) return;
    T sum[3] = {T(0), T(0), T(0)};
    for (std::uint32_t s = 0; s < k.spp; ++s) {
        const std::uint64_t id = pix * k.spp + s;
#pragma unroll
        for (int c = 0; c < 3; ++c) sum[c] = sum[c] + aces1(b.hdr[std::uint64_t(c) * b.n + id] * k.exposure);
    }
    const T sc = T(1) / T(float(k.spp));
#pragma unroll
    for (int c = 0; c < 3; ++c) img[pix * 3 + c] = float(sum[c] * sc);
}

// d ACES(x) / dx of the Narkowicz fit, 0 where it clamps.
template <class T> __device__ __forceinline__ T aces_d(T x) {
    const T a = T(2.51), bb = T(0.03), c = T(2.43), d = T(0.59), e = T(0.14);
    const T N = x * (a * x + bb), D = x * (c * x + d) + e;
    const T f = N / D;
    if (f <= T(0) || f >= T(1)) return T(0);
    return ((T(2) * a * x + bb) * D - N * (T(2) * c * x + d)) / (D * D);
}

// lam <- J^T lam + pend for the step y_{k-1} -> y_k (J over the 6 state
// components), and the step's terms of dLoss/d(E, L, a).  DUALJ: J built
// column by column with dual numbers (the cross-check); otherwise the
// hand-derived reverse pass of sgx_adjoint.cuh.
template <class T, bool DUALJ>
__device__ __forceinline__ void step_adjoint(const T* yp, T E, T L, T a, const DiffConst<T>& k, bool fade, T* lam,
                                             const T* pend, T& muE, T& muL, T& mua) {
    if constexpr (!DUALJ) {
        T gc[3] = {T(0), T(0), T(0)};
        sgxa::step_vjp<T>(yp, E, L, a, k.M, k.h, fade, lam, gc);
        muE += gc[0];
        muL += gc[1];
        mua += gc[2];
#pragma unroll
        for (int i = 0; i < NS; ++i) lam[i] += pend[i];
        return;
    }
    using DJ = Dual<T, NS + 3>;
    DJ yd[NS], od[NS];
#pragma unroll
    for (int i = 0; i < NS; ++i) yd[i] = DJ::var(yp[i], i);
    step_g<DJ, T>(yd, DJ::var(E, NS), DJ::var(L, NS + 1), DJ::var(a, NS + 2), k.M, k.h, fade, od);
    T nl[NS];
#pragma unroll
    for (int i = 0; i < NS; ++i) {
        T acc = T(0);
#pragma unroll
        for (int j = 0; j < NS; ++j) acc += lam[j] * od[j].d[i];
        nl[i] = acc;
    }
#pragma unroll
    for (int j = 0; j < NS; ++j) {
        muE += lam[j] * od[j].d[NS];
        muL += lam[j] * od[j].d[NS + 1];
        mua += lam[j] * od[j].d[NS + 2];
    }
#pragma unroll
    for (int i = 0; i < NS; ++i) lam[i] = nl[i] + pend[i];
}

// Adjoint: one thread per ray, a reverse sweep from the ray's last emitting
// step to the camera, one checkpoint segment at a time.  CK = kCkDense keeps
// the recomputed segment in dynamic shared memory, (CK + 1) * NC values a
// thread laid out [slot][value][thread] (consecutive threads, consecutive
// words); CK = kCkSparse in a thread-local array.  Launched with at most TH
// threads a block, exactly TH where the segment is shared.
//
// W is the number of warps that an SM has to hold, which caps the registers at
// 65,536 / (32 W).  The FP32 sweep's arithmetic has independent chains, so
// registers for more of them in flight are worth more than warps.  Backward call
// on one GB300, ms, at W = 16 (128 registers) / W = 10 (168, 12 warps resident):
// one-warp blocks 160 x 96 x 4 spp 0.80 / 0.59, 255 x 193 crossings 0.57 / 0.50;
// 128-thread blocks 512 x 512 x 4 6.38 / 6.05.  Up to 256 rays an SM (38,912
// on its 152) 8 warps hold them all at once, and 224 registers take 64 x 64 x 4 from 0.34 to 0.32;
// above that line they need a second wave (160 x 96 x 4: 0.71).  In the sparse
// form W = 12 takes the slab from 6.61 to 6.48, but the crossings, whose segment
// is their main traffic, from 1.63 to 1.65: they stay at 16.  The dual numbers
// spill 3 KB a thread at 128 registers and 0.9 KB at 255: 80 / 47.
//
// XS: the forward stored the crossing states.  Without them (records at the
// memory limit) the crossing model's seeds are formed in the sweep.
template <class T, bool SLAB, bool DUALJ, int CK, int TH, int W = kBackwardWarps<T, SLAB, DUALJ, CK>,
          bool XS = !SLAB && !DUALJ>
__global__ void __launch_bounds__(TH, W * 32 / TH)
    diff_backward_kernel(DiffConst<T> k, DiffParamsT<T> p, DiffBufs<T> b, const float* __restrict__ gimg) {
    constexpr bool SHARED = CK == kCkDense;
    extern __shared__ __align__(16) unsigned char diff_seg_raw[];
    // value v of slot j of this thread's segment (shared form)
    T* const seg = reinterpret_cast<T*>(diff_seg_raw) + threadIdx.x;
    auto at = [](int j, int v) { return (j * NC + v) * TH; };
    const std::uint64_t id = std::uint64_t(blockIdx.x) * blockDim.x + threadIdx.x;
    if (id >= b.n) return;
    double* gout = b.grads;
    const std::uint32_t nc = b.ncross[id];
    // the last step whose state the image depends on
    const std::uint32_t klast = nc == 0 ? 0u : (SLAB ? b.xk[id] : b.xk[std::uint64_t(nc - 1) * b.n + id]);
    if (klast == 0) {
#pragma unroll
        for (int q = 0; q < 4; ++q) gout[std::uint64_t(q) * b.n + id] = 0.0;
        return;
    }
    std::uint32_t gx, gy, s;
    ray_pixel(k, id, gx, gy, s);
    const std::uint64_t pix = id / k.spp;
    T g[3];
    const T inv_spp = T(1) / T(float(k.spp));
#pragma unroll
    for (int c = 0; c < 3; ++c) {
        const T x = b.hdr[std::uint64_t(c) * b.n + id] * k.exposure;
        g[c] = T(gimg[pix * 3 + c]) * inv_spp * aces_d(x) * k.exposure;
    }
    const T a = p.spin * k.M;
    const T r_in = p.r_in * k.M;
    T E, L, y0[NS];
    init_g<T, T>(a, p.incl, k, gx, gy, b.ox[s], b.oy[s], y0, E, L);

    T lam[NS] = {};
    T muE = T(0), muL = T(0), mua = T(0), g_a = T(0), g_rin = T(0), g_ts = T(0);
    const bool fade = k.fade != 0u;
    [[maybe_unused]] T Y[SHARED ? 1 : CK + 1][NS];

    // Crossing model: seeds of the transmittance chain
    //   colour = sum_j tau_j w_j c_j,  tau_{j+1} = tau_j (1 - w_j):
    //   dcolour/dc_j = tau_j w_j,  dcolour/dw_j = tau_j (c_j - R_{j+1}),
    //   R_j = w_j c_j + (1 - w_j) R_{j+1}.
    // The reverse pass's seeds (xq: adjoints of the states before and after the
    // crossing step) are formed here, all lanes at their j-th crossing
    // together, from the states the forward stored: inside the sweep the lanes
    // of a warp meet their crossings at different steps and would evaluate the
    // colour one after another.
    T xcs[kMaxCross], xgw[kMaxCross];
    std::uint32_t xkk[kMaxCross];
    [[maybe_unused]] T xq[XS ? kMaxCross : 1][7];
    if constexpr (!SLAB) {
        T w[kMaxCross], c3[kMaxCross][3], tau_j[kMaxCross];
        T tau = T(1);
        for (std::uint32_t j = 0; j < nc; ++j) {
            xkk[j] = b.xk[std::uint64_t(j) * b.n + id];
            w[j] = b.xw[std::uint64_t(j) * b.n + id];
#pragma unroll
            for (int c = 0; c < 3; ++c) c3[j][c] = b.xc[(std::uint64_t(j) * 3 + c) * b.n + id];
            tau_j[j] = tau;
            tau = tau * (T(1) - w[j]);
        }
        T R[3] = {T(0), T(0), T(0)};
        for (int j = int(nc) - 1; j >= 0; --j) {
            xcs[j] = tau_j[j] * w[j];
            xgw[j] = tau_j[j] * (g[0] * (c3[j][0] - R[0]) + g[1] * (c3[j][1] - R[1]) + g[2] * (c3[j][2] - R[2]));
#pragma unroll
            for (int c = 0; c < 3; ++c) R[c] = w[j] * c3[j][c] + (T(1) - w[j]) * R[c];
        }
        if constexpr (XS) {
            for (std::uint32_t j = 0; j < nc; ++j) {
                T x[7], q[11];
#pragma unroll
                for (int c = 0; c < 7; ++c) x[c] = b.xs[(std::uint64_t(j) * 7 + c) * b.n + id];
                crossing_vjp<T>(x[0], x[1], x[2], x[3], x[4], x[5], x[6], L, a, r_in, p.t_scale, k, g, xcs[j], xgw[j], q);
#pragma unroll
                for (int c = 0; c < 7; ++c) xq[j][c] = q[c];
                muL += q[7];
                g_a += q[8] * k.M;
                g_rin += q[9] * k.M;
                g_ts += q[10];
            }
        }
    }
    [[maybe_unused]] int jx = int(nc) - 1;  // crossing model: the next crossing of the sweep
    // Slab model: the same chain over every emitting step, R carried through the sweep.
    T R[3] = {T(0), T(0), T(0)};
    [[maybe_unused]] T tb[SHARED ? 1 : CK + 1];

    const int mlast = int((klast - 1) / CK);
    for (int m = mlast; m >= 0; --m) {
        const std::uint32_t kbeg = std::uint32_t(m) * CK;
        const std::uint32_t kend = (kbeg + CK < klast) ? kbeg + CK : klast;
        const std::uint64_t cb = std::uint64_t(m) * NC * b.n + id;
        T tau = b.ckpt[cb + std::uint64_t(NS) * b.n];
        if constexpr (SHARED) {
            // the running state in registers, each state stored once
            T yc[NS];
#pragma unroll
            for (int i = 0; i < NS; ++i) {
                yc[i] = b.ckpt[cb + std::uint64_t(i) * b.n];
                seg[at(0, i)] = yc[i];
            }
            for (std::uint32_t kk = kbeg + 1; kk <= kend; ++kk) {
                const int j = int(kk - kbeg);
                T yn[NS];
                step_g<T, T>(yc, E, L, a, k.M, k.h, fade, yn);
                if constexpr (SLAB) {
                    seg[at(j, NS)] = tau;  // transmittance before step kk's emission
                    T alpha;
                    if (slab_alpha_g<T, T>(yc[0], yc[1], yc[2], yn[0], yn[1], yn[2], yn[5], yn[6], yn[7], r_in, k, alpha))
                        tau = tau * (T(1) - alpha);
                }
#pragma unroll
                for (int i = 0; i < NS; ++i) {
                    seg[at(j, i)] = yn[i];
                    yc[i] = yn[i];
                }
            }
        } else {
#pragma unroll
            for (int i = 0; i < NS; ++i) Y[0][i] = b.ckpt[cb + std::uint64_t(i) * b.n];
            for (std::uint32_t kk = kbeg + 1; kk <= kend; ++kk) {
                const T* yp = Y[kk - 1 - kbeg];
                T* yc = Y[kk - kbeg];
                step_g<T, T>(yp, E, L, a, k.M, k.h, fade, yc);
                if constexpr (SLAB) {
                    tb[kk - kbeg] = tau;  // transmittance before step kk's emission
                    T alpha;
                    if (slab_alpha_g<T, T>(yp[0], yp[1], yp[2], yc[0], yc[1], yc[2], yc[5], yc[6], yc[7], r_in, k, alpha))
                        tau = tau * (T(1) - alpha);
                }
            }
        }
        for (std::uint32_t kk = kend; kk > kbeg; --kk) {
            const int j = int(kk - kbeg);
            [[maybe_unused]] T ypr[NS], ycr[NS];
            const T* yp;
            const T* yc;
            if constexpr (SHARED) {
#pragma unroll
                for (int i = 0; i < NS; ++i) {
                    ypr[i] = seg[at(j - 1, i)];
                    ycr[i] = seg[at(j, i)];
                }
                yp = ypr;
                yc = ycr;
            } else {
                yp = Y[j - 1];
                yc = Y[j];
            }
            T pend[NS] = {};
            using D = Dual<T, 11>;
            using DA = Dual<T, 10>;
            using DC = Dual<T, 6>;
            if constexpr (SLAB) {
                T qa[10], qc[6], colv[3], alv, tj;
                bool emits = (k.flags & SGX_FLAG_DISC_ON) != 0u;
                if constexpr (SHARED) tj = seg[at(j, NS)];
                else tj = tb[j];
                if constexpr (DUALJ) {
                    emits = emits && slab_g<T, T>(yp[0], yp[1], yp[2], yc[0], yc[1], yc[2], yc[5], yc[6], yc[7], L, a,
                                                  r_in, p.t_scale, k, colv, alv);
                    if (emits) {
                        // d alpha / d(r0, th0, ph0, r1, th1, ph1, psi1, s1, c1, r_in)
                        DA ald;
                        slab_alpha_g<DA, T>(DA::var(yp[0], 0), DA::var(yp[1], 1), DA::var(yp[2], 2),
                                            DA::var(yc[0], 3), DA::var(yc[1], 4), DA::var(yc[2], 5),
                                            DA::var(yc[5], 6), DA::var(yc[6], 7), DA::var(yc[7], 8),
                                            DA::var(r_in, 9), k, ald);
                        // d colour / d(r1, ph1, L, a, r_in, t_scale)
                        DC col[3];
                        slab_colour_g<DC, T>(DC::var(yc[0], 0), DC::var(yc[2], 1), DC::var(L, 2), DC::var(a, 3),
                                             DC::var(r_in, 4), DC::var(p.t_scale, 5), k, col);
#pragma unroll
                        for (int x = 0; x < 10; ++x) qa[x] = ald.d[x];
#pragma unroll
                        for (int x = 0; x < 6; ++x)
                            qc[x] = tj * alv * (g[0] * col[0].d[x] + g[1] * col[1].d[x] + g[2] * col[2].d[x]);
                    }
                } else {
                    emits = emits && slab_alpha_d<T>(yp[0], yp[1], yp[2], yc[0], yc[1], yc[2], yc[5], yc[6], yc[7],
                                                     r_in, k, alv, qa);
                    if (emits) {
                        const T w[3] = {tj * alv * g[0], tj * alv * g[1], tj * alv * g[2]};
                        colour_vjp<T>(yc[0], yc[2], L, a, r_in, p.t_scale, k, w, colv, qc);
                    }
                }
                if (emits) {
                    const T gal = tj * (g[0] * (colv[0] - R[0]) + g[1] * (colv[1] - R[1]) + g[2] * (colv[2] - R[2]));
#pragma unroll
                    for (int c = 0; c < 3; ++c) R[c] = alv * colv[c] + (T(1) - alv) * R[c];
                    pend[0] += gal * qa[0];
                    pend[1] += gal * qa[1];
                    pend[2] += gal * qa[2];
                    lam[0] += gal * qa[3] + qc[0];
                    lam[1] += gal * qa[4];
                    lam[2] += gal * qa[5] + qc[1];
                    lam[5] += gal * qa[6];
                    lam[6] += gal * qa[7];
                    lam[7] += gal * qa[8];
                    muL += qc[2];
                    g_a += qc[3] * k.M;
                    g_rin += (gal * qa[9] + qc[4]) * k.M;
                    g_ts += qc[5];
                }
            } else if constexpr (!DUALJ) {
                if (jx >= 0 && kk == xkk[jx]) {
                    const T* q;
                    [[maybe_unused]] T qv[11];
                    if constexpr (XS) {
                        q = xq[jx];
                    } else {
                        crossing_vjp<T>(yp[0], yp[1], yp[5], yc[0], yc[1], yc[2], yc[5], L, a, r_in, p.t_scale, k, g,
                                        xcs[jx], xgw[jx], qv);
                        q = qv;
                        muL += qv[7];
                        g_a += qv[8] * k.M;
                        g_rin += qv[9] * k.M;
                        g_ts += qv[10];
                    }
                    --jx;
                    pend[0] += q[0];
                    pend[1] += q[1];
                    pend[5] += q[2];
                    lam[0] += q[3];
                    lam[1] += q[4];
                    lam[2] += q[5];
                    lam[5] += q[6];
                }
            } else {
                for (std::uint32_t j = 0; j < nc; ++j) {
                    if (xkk[j] != kk) continue;
                    // d(colour, weight)/d(r0, th0, psi0, r1, th1, ph1, psi1, L, a, r_in, t_scale)
                    D col[3], wd;
                    crossing_g<D, T>(D::var(yp[0], 0), D::var(yp[1], 1), D::var(yp[5], 2), D::var(yc[0], 3),
                                     D::var(yc[1], 4), D::var(yc[2], 5), D::var(yc[5], 6), D::var(L, 7),
                                     D::var(a, 8), D::var(r_in, 9), D::var(p.t_scale, 10), k, col, wd);
                    T qv[11];
#pragma unroll
                    for (int x = 0; x < 11; ++x)
                        qv[x] = xcs[j] * (g[0] * col[0].d[x] + g[1] * col[1].d[x] + g[2] * col[2].d[x]) +
                                xgw[j] * wd.d[x];
                    pend[0] += qv[0];
                    pend[1] += qv[1];
                    pend[5] += qv[2];
                    lam[0] += qv[3];
                    lam[1] += qv[4];
                    lam[2] += qv[5];
                    lam[5] += qv[6];
                    muL += qv[7];
                    g_a += qv[8] * k.M;
                    g_rin += qv[9] * k.M;
                    g_ts += qv[10];
                }
            }
            step_adjoint<T, DUALJ>(yp, E, L, a, k, fade, lam, pend, muE, muL, mua);
        }
    }
    // Chain through the camera set-up: y0, E, L as functions of (a, incl).
    using D2 = Dual<T, 2>;
    D2 yd0[NS], Ed, Ld;
    init_g<D2, T>(D2::var(a, 0), D2::var(p.incl, 1), k, gx, gy, b.ox[s], b.oy[s], yd0, Ed, Ld);
    T grad_a = g_a + mua * k.M, grad_i = T(0);
#pragma unroll
    for (int i = 0; i < NS; ++i) {
        grad_a += lam[i] * yd0[i].d[0] * k.M;
        grad_i += lam[i] * yd0[i].d[1];
    }
    grad_a += (muE * Ed.d[0] + muL * Ld.d[0]) * k.M;
    grad_i += muE * Ed.d[1] + muL * Ld.d[1];
    gout[id] = double(grad_a);
    gout[b.n + id] = double(grad_i);
    gout[2 * b.n + id] = double(g_rin);
    gout[3 * b.n + id] = double(g_ts);
}

// Fixed-order sum of the per-ray gradients: block-level tree over 1024-ray
// chunks, then one block over the chunk sums.
__global__ void reduce_chunks(const double* __restrict__ in, std::uint64_t n, double* __restrict__ part,
                              std::uint32_t nchunks) {
    __shared__ double sh[256];
    const std::uint32_t chunk = blockIdx.x, q = blockIdx.y;
    const std::uint64_t beg = std::uint64_t(chunk) * 1024;
    double acc = 0.0;
    for (int i = 0; i < 4; ++i) {
        const std::uint64_t j = beg + threadIdx.x + i * 256;
        if (j < n) acc += in[std::uint64_t(q) * n + j];
    }
    sh[threadIdx.x] = acc;
    __syncthreads();
    for (int st = 128; st > 0; st >>= 1) {
        if (int(threadIdx.x) < st) sh[threadIdx.x] += sh[threadIdx.x + st];
        __syncthreads();
    }
    if (threadIdx.x == 0) part[std::uint64_t(q) * nchunks + chunk] = sh[0];
}

__global__ void reduce_final(const double* __restrict__ part, std::uint32_t nchunks, double* __restrict__ out) {
    __shared__ double sh[256];
    const std::uint32_t q = blockIdx.x;
    double acc = 0.0;
    for (std::uint32_t i = threadIdx.x; i < nchunks; i += 256) acc += part[std::uint64_t(q) * nchunks + i];
    sh[threadIdx.x] = acc;
    __syncthreads();
    for (int st = 128; st > 0; st >>= 1) {
        if (int(threadIdx.x) < st) sh[threadIdx.x] += sh[threadIdx.x + st];
        __syncthreads();
    }
    if (threadIdx.x == 0) out[q] = sh[0];
}

template <class T> __global__ void offsets_kernel(std::uint32_t spp, T* ox, T* oy) {
    const std::uint32_t s = blockIdx.x * blockDim.x + threadIdx.x;
    if (s < spp) sample_offset<T>(spp, s, ox[s], oy[s]);
}

template <class T>
DiffConst<T> make_const(const sgx_uniforms& u, const sgx_diff_opts& o) {
    DiffConst<T> k{};
    k.M = T(u.mass_M);
    {  // |cam_pos| formed in T from the float components
        const T x = T(u.cam_pos.x), y = T(u.cam_pos.y), z = T(u.cam_pos.z);
        k.dcam = T(std::sqrt(x * x + y * y + z * z));
    }
    k.aspect = T(u.aspect);
    k.tanh_ = T(u.tan_half_fov);
    k.width_f = T(float(u.width));
    k.height_f = T(float(u.height));
    k.r_out = T(u.disc_r_outer);
    k.peak_T = T(u.disc_peak_T);
    k.escape_r = T(u.escape_r);
    k.h = T(u.h_step);
    k.exposure = T(u.exposure);
    k.turbulence = T(u.disc_turbulence);
    k.time_sec = T(u.time_sec);
    k.eps = T(o.edge_width) * T(u.mass_M);
    k.fade_start = T(o.fade_start);
    k.fade_width = T(o.fade_width);
    k.fade = o.fade_start > 0.0f ? 1u : 0u;
    k.H = T(o.half_thickness) * T(u.mass_M);
    k.kappa = T(o.tau_perp) / (T(16) / T(15) * k.H);
    k.width = u.width;
    k.height = u.height;
    k.spp = u.supersample < 1u ? 1u : (u.supersample > 1024u ? 1024u : u.supersample);
    k.max_steps = u.max_steps;
    k.flags = u.flags;
    return k;
}

}  // namespace

// Per-context state of the differentiable form (the forward's records).
struct sgx_diff_state {
    void* mem = nullptr;
    std::size_t cap = 0;
    std::uint64_t n = 0;
    std::uint32_t slots = 0;
    std::uint32_t ck = kCkSparse;  // steps between checkpoints (kCkSparse or kCkDense)
    std::uint32_t precision = SGX_PRECISION_FP32;
    std::uint32_t nx = kMaxCross;  // crossing records per ray (1 for the slab model)
    bool xs = false;               // crossing states kept behind the records
    sgx_uniforms u{};
    sgx_diff_params p{};
    sgx_diff_opts o{};
    bool valid = false;
    float* img = nullptr;  // internal image when the caller passes none
    std::size_t img_cap = 0;
};

namespace {

template <class T>
std::size_t state_bytes(std::uint64_t n, std::uint32_t slots, std::uint32_t spp, std::size_t nx) {
    auto r = [](std::size_t x) { return (x + 255) / 256 * 256; };
    return r(std::size_t(slots) * NC * n * sizeof(T)) + r(3 * n * sizeof(T)) + 2 * r(n * 4) + r(nx * n * 4) +
           (nx > 1 ? r(nx * n * sizeof(T)) + r(nx * 3 * n * sizeof(T)) : 0) + r(4 * n * 8) +
           r(2 * std::size_t(spp) * sizeof(T)) + 256 +
           // reduction scratch: 4 x chunk sums + 4 results
           r(4 * ((n + 1023) / 1024) * 8) + 256;
}

// Bytes of the crossing states (after state_bytes).
template <class T> std::size_t crossing_bytes(std::uint64_t n, std::size_t nx) { return nx * 7 * n * sizeof(T); }

template <class T>
DiffBufs<T> carve_bufs(sgx_diff_state& st, std::uint32_t spp) {
    DiffBufs<T> b{};
    const std::uint64_t n = st.n;
    unsigned char* p = static_cast<unsigned char*>(st.mem);
    auto take = [&](std::size_t bytes) {
        unsigned char* r = p;
        p += (bytes + 255) / 256 * 256;
        return r;
    };
    b.n = n;
    b.slots = st.slots;
    const std::size_t nx = st.nx;
    b.ckpt = reinterpret_cast<T*>(take(std::size_t(st.slots) * NC * n * sizeof(T)));
    b.hdr = reinterpret_cast<T*>(take(3 * n * sizeof(T)));
    b.nsteps = reinterpret_cast<std::uint32_t*>(take(n * 4));
    b.ncross = reinterpret_cast<std::uint32_t*>(take(n * 4));
    b.xk = reinterpret_cast<std::uint32_t*>(take(nx * n * 4));
    b.xw = nx > 1 ? reinterpret_cast<T*>(take(nx * n * sizeof(T))) : nullptr;
    b.xc = nx > 1 ? reinterpret_cast<T*>(take(nx * 3 * n * sizeof(T))) : nullptr;
    b.grads = reinterpret_cast<double*>(take(4 * n * 8));
    T* off = reinterpret_cast<T*>(take(2 * std::size_t(spp) * sizeof(T)));
    b.ox = off;
    b.oy = off + spp;
    b.overflow = reinterpret_cast<unsigned long long*>(take(64));
    b.xs = st.xs ? reinterpret_cast<T*>(static_cast<unsigned char*>(st.mem) + state_bytes<T>(n, st.slots, spp, nx))
                 : nullptr;
    return b;
}

template <class T>
cudaError_t run_forward(sgx_diff_state& st, float* img, cudaStream_t s) {
    const DiffConst<T> k = make_const<T>(st.u, st.o);
    const DiffParamsT<T> p{T(st.p.spin), T(st.p.incl), T(st.p.r_in), T(st.p.t_scale)};
    DiffBufs<T> b = carve_bufs<T>(st, k.spp);
    cudaError_t e = cudaMemsetAsync(b.overflow, 0, 16, s);
    if (e != cudaSuccess) return e;
    offsets_kernel<T><<<(k.spp + 127) / 128, 128, 0, s>>>(k.spp, const_cast<T*>(b.ox), const_cast<T*>(b.oy));
    const int th = st.n < kSmallForward ? kSmallThreads : kThreads;
    const unsigned grid = unsigned((st.n + th - 1) / th);
    const bool slab = st.o.model == SGX_DIFF_MODEL_SLAB;
    bool dense = false;
    if constexpr (sizeof(T) == 4) dense = st.ck == std::uint32_t(kCkDense);
    if constexpr (sizeof(T) == 4) {
        if (dense && slab) diff_forward_kernel<T, true, kCkDense><<<grid, th, 0, s>>>(k, p, b);
        else if (dense) diff_forward_kernel<T, false, kCkDense><<<grid, th, 0, s>>>(k, p, b);
    }
    if (!dense && slab) diff_forward_kernel<T, true, kCkSparse><<<grid, th, 0, s>>>(k, p, b);
    else if (!dense) diff_forward_kernel<T, false, kCkSparse><<<grid, th, 0, s>>>(k, p, b);
    const std::uint64_t npix = std::uint64_t(k.width) * k.height;
    diff_image_kernel<T><<<unsigned((npix + 255) / 256), 256, 0, s>>>(k, b, img);
    return cudaGetLastError();
}

template <class T>
cudaError_t run_backward(sgx_diff_state& st, const float* gimg, double* d_out4, cudaStream_t s) {
    const DiffConst<T> k = make_const<T>(st.u, st.o);
    const DiffParamsT<T> p{T(st.p.spin), T(st.p.incl), T(st.p.r_in), T(st.p.t_scale)};
    DiffBufs<T> b = carve_bufs<T>(st, k.spp);
    const bool slab = st.o.model == SGX_DIFF_MODEL_SLAB, dual = st.o.adjoint_form == SGX_DIFF_ADJOINT_DUAL;
    bool dense = false;
    if constexpr (sizeof(T) == 4) dense = st.ck == std::uint32_t(kCkDense);
    const int th = dense || st.n < kSmallBackward ? kSmallThreads : kThreads;
    const unsigned grid = unsigned((st.n + th - 1) / th);
    if constexpr (sizeof(T) == 4) {
        // the dense checkpoints pair with the hand-derived reverse pass only;
        // their segments are laid out for the block size
        if (dense) {
            const int smem = (kCkDense + 1) * NC * th * int(sizeof(T));
            constexpr int kW = kBackwardWarps<T, false, false, kCkDense>;
            int dev = 0, sms = 0;
            cudaError_t e = cudaGetDevice(&dev);
            if (e == cudaSuccess) e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
            if (e != cudaSuccess) return e;
            auto* kern = !slab && !st.xs ? diff_backward_kernel<T, false, false, kCkDense, kSmallThreads, kW, false>
                         : st.n > kOneWaveRaysPerSm * std::uint64_t(sms)
                             ? (slab ? diff_backward_kernel<T, true, false, kCkDense, kSmallThreads>
                                     : diff_backward_kernel<T, false, false, kCkDense, kSmallThreads>)
                             : (slab ? diff_backward_kernel<T, true, false, kCkDense, kSmallThreads, 8>
                                     : diff_backward_kernel<T, false, false, kCkDense, kSmallThreads, 8>);
            e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
            if (e != cudaSuccess) return e;
            kern<<<grid, th, smem, s>>>(k, p, b, gimg);
        }
    }
    if (!dense) {
        if (slab && !dual) diff_backward_kernel<T, true, false, kCkSparse, kThreads><<<grid, th, 0, s>>>(k, p, b, gimg);
        else if (slab) diff_backward_kernel<T, true, true, kCkSparse, kThreads><<<grid, th, 0, s>>>(k, p, b, gimg);
        else if (!dual && st.xs) diff_backward_kernel<T, false, false, kCkSparse, kThreads><<<grid, th, 0, s>>>(k, p, b, gimg);
        else if (!dual)
            diff_backward_kernel<T, false, false, kCkSparse, kThreads, kBackwardWarps<T, false, false, kCkSparse>, false>
                <<<grid, th, 0, s>>>(k, p, b, gimg);
        else diff_backward_kernel<T, false, true, kCkSparse, kThreads><<<grid, th, 0, s>>>(k, p, b, gimg);
    }
    const std::uint32_t nchunks = std::uint32_t((st.n + 1023) / 1024);
    double* part = reinterpret_cast<double*>(reinterpret_cast<unsigned char*>(b.overflow) + 256);
    reduce_chunks<<<dim3(nchunks, 4), 256, 0, s>>>(b.grads, st.n, part, nchunks);
    reduce_final<<<4, 256, 0, s>>>(part, nchunks, d_out4);
    return cudaGetLastError();
}

}  // namespace


// Entry points of the two translation units (defined in sgx_diff.cu for
// float and in sgx_diff64.cu for double).
cudaError_t sgx_diff_run_forward_f32(sgx_diff_state& st, float* img, cudaStream_t s);
cudaError_t sgx_diff_run_backward_f32(sgx_diff_state& st, const float* gimg, double* d_out4, cudaStream_t s);
cudaError_t sgx_diff_run_forward_f64(sgx_diff_state& st, float* img, cudaStream_t s);
cudaError_t sgx_diff_run_backward_f64(sgx_diff_state& st, const float* gimg, double* d_out4, cudaStream_t s);
