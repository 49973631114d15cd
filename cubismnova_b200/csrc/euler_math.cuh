// euler_math.cuh -- pointwise math of the compressible Euler RHS (device).
//
// WENO5-JS reconstruction (Jiang & Shu, J. Comput. Phys. 126, 1996) of the
// primitive variables (rho, u, v, w, p) and the Rusanov (local Lax-Friedrichs)
// flux, gamma-law gas.  The reference library only promises these operators
// (README.rst:28-31); this is an implementation of the published method.
//
// Floating-point contract.  The file is compiled with FMA contraction on
// (nvcc's default --fmad=true): beyond the fma() calls written out below, the
// compiler fuses any multiply feeding an add.  Reciprocals and square roots
// are not IEEE-rounded: FP64 uses the hardware approximations refined by one
// third-order step (rcp_pos / rsqrt_pos below, within a few ulp), FP32 calls
// CUDA's fast intrinsics (__fdividef, rsqrtf: about 2 ulp).  The CPU oracle
// computes the same formulas with IEEE division and square root and no
// contraction; FP64 results agree with it within 1e-13 relative, FP32 results
// are judged by their error against FP64.
//
// Nonlinear weights: with s_k = eps + beta_k and t_k = s_k^2 the JS weights
// alpha_k = d_k / t_k normalise to omega_k = d_k*prod_{j!=k} t_j / D with
// D = sum_k d_k*prod_{j!=k} t_j, so one division per reconstruction suffices.
// The indicators beta_k and the products t_i t_j belong to the cell, not to
// the face: a cell's left-biased state (at its upper face) and right-biased
// state (at its lower face) share them, and neighbouring cells share the
// differences they are made of (weno5_run).
//
// Range.  The sums are formed as 4 s_k.  A jump J in the data gives 4 s ~ 13
// J^2 and products of two squares ~ 5e3 J^8, which leaves the FP32 range
// above J ~ 2e4 (a pressure jump of a fifth of a bar in SI units).  So in FP32
// the sums are formed as s_k (4 s_k would leave the range at half the jump) and
// t_k is formed from s_k * 2^-e, with e the mean of the binary exponents of
// the largest and the middle s_k (rounded down).  Scaling by a power of two is
// exact and cancels in every ratio below.  With it the dominant product
// t_max t_mid lies in [1, 64) and every FP32 denominator in [1, 640]; the only
// products that can underflow are those of negligible weights.  FP64 needs no
// scaling: its denominators lie in [2e-21, ~2e4 J^8].
// Since the factor is an exact power of two, the scaled and unscaled forms
// give the same values wherever the unscaled one stays in range; a tile whose
// primitives are all within kUnscaledMax in magnitude (then the products stay
// below 4e32 and the numerators below 4e36, and eps keeps the products above
// 2e-22) skips the scaling.
#pragma once

#include <cuda_runtime.h>

namespace cn {
namespace euler {

// largest primitive magnitude of a tile for the unscaled FP32 WENO5 weights
constexpr float kUnscaledMax = 1000.0f;

template <typename T> struct K {
    static constexpr T c133 = T(13.0 / 3.0), c1312 = T(13.0 / 12.0);
    static constexpr T eps4 = T(4e-6), eps = T(1e-6);
    static constexpr T third = T(1.0 / 3.0);
    static constexpr T half = T(0.5);
};

__device__ __forceinline__ double dfma(double a, double b, double c) { return fma(a, b, c); }
__device__ __forceinline__ float dfma(float a, float b, float c) { return fmaf(a, b, c); }
__device__ __forceinline__ double dabs(double a) { return fabs(a); }
__device__ __forceinline__ float dabs(float a) { return fabsf(a); }
__device__ __forceinline__ double dmax(double a, double b) { return fmax(a, b); }
__device__ __forceinline__ float dmax(float a, float b) { return fmaxf(a, b); }

// 1/x for a positive normal x (denominators of the face states, densities).
// FP64: the PTX approximation rcp.approx.ftz.f64 refined by one step of the
// third-order iteration that truncates the series 1/x = r / (1 - e) =
// r (1 + e + e^2 + ...), e = 1 - x r:  r' = r + r (e + e^2), relative error
// e^3 plus rounding.  FP32: CUDA's __fdividef (valid for x < 2^126).
__device__ __forceinline__ double rcp_pos(double x)
{
    double r;
    asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(r) : "d"(x));
    const double e = fma(-x, r, 1.0);
    return fma(r, fma(e, e, e), r);
}
__device__ __forceinline__ float rcp_pos(float x) { return __fdividef(1.0f, x); }

// 1/sqrt(x) for a positive normal x.  FP64: rsqrt.approx.ftz.f64 refined by one
// step of the third-order iteration from the series (1 - h)^(-1/2) =
// 1 + h/2 + 3h^2/8 + ..., h = 1 - x y^2:  y' = y + y h (1/2 + 3/8 h).
// FP32: CUDA's rsqrtf.
__device__ __forceinline__ double rsqrt_pos(double x)
{
    double y;
    asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
    const double h = fma(-x * y, y, 1.0);
    return fma(y * h, fma(0.375, h, 0.5), y);
}
__device__ __forceinline__ float rsqrt_pos(float x) { return rsqrtf(x); }

// The FP32 factor 2^-e of the range note above for s0, s1, s2 >= eps: e =
// floor((E_max + E_mid) / 2) - 127 from the biased exponents of the largest
// and the middle of the three (E_max + E_mid = E0 + E1 + E2 - E_min).  The
// exponents come from the bit patterns (integer instructions only).  A NaN
// or infinite s gives NaN states, and so do two sums above 2^127 (~1.7e38,
// jumps ~1e19: the factor leaves the normal range there).
__device__ __forceinline__ float weno5_scale(float s0, float s1, float s2)
{
    const int e0 = __float_as_int(s0) >> 23, e1 = __float_as_int(s1) >> 23, e2 = __float_as_int(s2) >> 23;
    const int emin = min(min(e0, e1), e2);
    return __int_as_float(int(unsigned(254 - ((e0 + e1 + e2 - emin) >> 1)) << 23));
}

// ---------------------------------------------------------------------------
// Reconstruction of a run of three faces.  The value type V is double, float,
// or float2: Blackwell executes FP32 add, multiply and fused multiply-add on a
// pair of values per thread (PTX add/mul/fma .rn.f32x2, CUDA's __fadd2_rn /
// __fmul2_rn / __ffma2_rn), so the FP32 kernel reconstructs two primitive
// variables per instruction, lane x holding one and lane y the other.  (The
// Rusanov flux stays scalar: packing its left and right states measured
// slower, 11.9 against 12.5 Gcell-updates/s at 1024^3, from the moves that
// regroup the lanes.)
// ---------------------------------------------------------------------------
template <typename V> struct Scalar { using type = V; };
template <> struct Scalar<float2> { using type = float; };
template <typename V> __device__ __forceinline__ V vset(typename Scalar<V>::type a) { return a; }
template <> __device__ __forceinline__ float2 vset<float2>(float a) { return make_float2(a, a); }
template <typename V> __device__ __forceinline__ V vadd(V a, V b) { return a + b; }
template <> __device__ __forceinline__ float2 vadd<float2>(float2 a, float2 b) { return __fadd2_rn(a, b); }
template <typename V> __device__ __forceinline__ V vmul(V a, V b) { return a * b; }
template <> __device__ __forceinline__ float2 vmul<float2>(float2 a, float2 b) { return __fmul2_rn(a, b); }
template <typename V> __device__ __forceinline__ V vfma(V a, V b, V c) { return dfma(a, b, c); }
template <> __device__ __forceinline__ float2 vfma<float2>(float2 a, float2 b, float2 c) { return __ffma2_rn(a, b, c); }
template <typename V> __device__ __forceinline__ V vsub(V a, V b) { return a - b; }
template <> __device__ __forceinline__ float2 vsub<float2>(float2 a, float2 b)
{
    return __ffma2_rn(b, make_float2(-1.0f, -1.0f), a);
}
template <typename V> __device__ __forceinline__ V vrcp(V a) { return rcp_pos(a); }
template <> __device__ __forceinline__ float2 vrcp<float2>(float2 a) { return make_float2(rcp_pos(a.x), rcp_pos(a.y)); }

__device__ __forceinline__ float range_scale(float s0, float s1, float s2) { return weno5_scale(s0, s1, s2); }
// weno5_scale for both lanes of a pair at once, from the top 7 bits of each
// biased exponent (byte 3 of a positive float, E >> 1) packed as two 16-bit
// halves: m = (E_max >> 1) + (E_mid >> 1) differs from (E_max + E_mid) / 2
// by at most 1, so the dominant product t_max t_mid lies in [1/4, 256) and
// the range note's bounds widen by a factor 4 at most.  The halves never
// carry into each other (each stays below 2^9).
__device__ __forceinline__ float2 range_scale(float2 s0, float2 s1, float2 s2)
{
    // bytes [x.b3, 0, y.b3, 0]: selector nibbles 3, 7 pick byte 3 of each
    // word, 0xB / 0xF replicate its sign bit (0 for s > 0)
    const unsigned e0 = __byte_perm(__float_as_uint(s0.x), __float_as_uint(s0.y), 0xF7B3);
    const unsigned e1 = __byte_perm(__float_as_uint(s1.x), __float_as_uint(s1.y), 0xF7B3);
    const unsigned e2 = __byte_perm(__float_as_uint(s2.x), __float_as_uint(s2.y), 0xF7B3);
    const unsigned mn = __vmins2(__vmins2(e0, e1), e2);
    const unsigned b = 0x00FE00FEu - (e0 + e1 + e2 - mn); // biased exponents of the factors
    return make_float2(__uint_as_float(b << 23), __uint_as_float((b >> 16) << 23));
}

// States at three consecutive faces of a line from its 8 cells around them,
// u[0..7]; face i lies between cells u[i+2] and u[i+3].  wl[i]: the
// left-biased state (of cell u[i+2]), wr[i]: the right-biased one (of cell
// u[i+3]).
//
// Everything is written in differences along the line, each formed once and
// shared by the cells that use it: first differences d, second differences
// a_k = d_k - d_(k-1), third differences b.  With a0, a1, a2 the second
// differences at cells j-1, j, j+1, d12 = u_j - u_(j-1), d23 = u_(j+1) - u_j
// the smoothness sums are
//   4 s0 = 13/3 a0^2 + (a0 + 2 d12)^2 + 4 eps,   4 s1 = 13/3 a1^2 + (d12 + d23)^2 + 4 eps,
//   4 s2 = 13/3 a2^2 + (a2 - 2 d23)^2 + 4 eps
// (the factor 4 cancels in the weights, the rescaled FP32 form goes without it), so the term q = 13/3 a^2 + 4 eps of
// a second difference serves the three cells around it.  The candidates
// differ from the middle one by third differences only,
//   6 q0 - 6 q1 = -2 b01,  6 q2 - 6 q1 = -b12,  b01 = a1 - a0, b12 = a2 - a1,
// so with p12 = t1 t2 and so on, A = p12 b01 and B = p01 b12:
//   left  = u_j + [ d12/2 + a1/3 - (A/3 + B/2) / (S + 2 p01) ],
//   right = u_j + [-d23/2 + a1/3 + (A/2 + B/3) / (S + 2 p12) ],
//   S = p12 + 6 p02 + p01.
// The bracket is summed before u_j is added, so a state carries one rounding
// at the cell value's magnitude.  Per variable and run 152 operations in
// FP64 (reciprocals included), against 205 with each cell's differences,
// indicators and candidates formed on their own; with the fluxes' fused sums
// (rusanov) a step of 512^3 cells went from 54.1 to 46.6 ms in FP64, of 384^3
// cells from 13.4 to 12.4 ms in FP32.
template <bool SCALED, typename V>
__device__ __forceinline__ void weno5_run(const V (&u)[8], V (&wl)[3], V (&wr)[3])
{
    using T = typename Scalar<V>::type;
    using C = K<T>;
    V d[7], a[6], q[6], b[5];
#pragma unroll
    for (int k = 0; k < 7; ++k)
        d[k] = vsub(u[k + 1], u[k]);
#pragma unroll
    for (int k = 0; k < 6; ++k) {
        a[k] = vsub(d[k + 1], d[k]);
        q[k] = vfma(vmul(vset<V>(SCALED ? C::c1312 : C::c133), a[k]), a[k], vset<V>(SCALED ? C::eps : C::eps4));
    }
#pragma unroll
    for (int k = 0; k < 5; ++k)
        b[k] = vsub(a[k + 1], a[k]);
#pragma unroll
    for (int j = 0; j < 4; ++j) { // cell u[j + 2]
        V h0, h1, h2;
        if constexpr (SCALED) { // half of the others, to the bit
            h0 = vfma(vset<V>(C::half), a[j], d[j + 1]);
            h1 = vmul(vset<V>(C::half), vadd(d[j + 1], d[j + 2]));
            h2 = vfma(vset<V>(-C::half), a[j + 2], d[j + 2]);
        } else {
            h0 = vfma(vset<V>(T(2)), d[j + 1], a[j]);
            h1 = vadd(d[j + 1], d[j + 2]);
            h2 = vfma(vset<V>(T(-2)), d[j + 2], a[j + 2]);
        }
        V s0 = vfma(h0, h0, q[j]), s1 = vfma(h1, h1, q[j + 1]), s2 = vfma(h2, h2, q[j + 2]);
        if constexpr (SCALED) { // FP32: exact power-of-two rescaling
            const V sc = range_scale(s0, s1, s2);
            s0 = vmul(s0, sc);
            s1 = vmul(s1, sc);
            s2 = vmul(s2, sc);
        }
        const V t0 = vmul(s0, s0), t1 = vmul(s1, s1), t2 = vmul(s2, s2);
        const V p12 = vmul(t1, t2), p02 = vmul(t0, t2), p01 = vmul(t0, t1);
        const V A = vmul(p12, b[j]), B = vmul(p01, b[j + 1]);
        const V S = vfma(vset<V>(T(6)), p02, vadd(p12, p01));
        const V m = vmul(vset<V>(C::third), a[j + 1]);
        if (j < 3) {
            const V den = vfma(vset<V>(T(2)), p01, S);
            const V num = vfma(vset<V>(-C::third), A, vmul(vset<V>(-C::half), B));
            wl[j] = vadd(u[j + 2], vfma(num, vrcp(den), vfma(vset<V>(C::half), d[j + 1], m)));
        }
        if (j > 0) {
            const V den = vfma(vset<V>(T(2)), p12, S);
            const V num = vfma(vset<V>(C::third), B, vmul(vset<V>(C::half), A));
            wr[j - 1] = vadd(u[j + 2], vfma(num, vrcp(den), vfma(vset<V>(-C::half), d[j + 2], m)));
        }
    }
}

// Twice the Rusanov flux through a face with normal direction `d` (0,1,2)
// from the reconstructed primitive states WL, WR = (rho, u, v, w, p):
// F = (f(UL) + f(UR)) - a (UR - UL), a = max(|u_n| + c) of both sides.  The
// factor 1/2 of the flux is exact and is taken with 1/h by the flux
// differences.
template <typename T>
__device__ __forceinline__ void rusanov(const T (&WL)[5], const T (&WR)[5], int d, T gamma,
                                        T igm1, T (&F)[5])
{
    using C = K<T>;
    const T rl = WL[0], rr = WR[0];
    // normal velocities (selects, not an index: d is a runtime value)
    const T unl = d == 0 ? WL[1] : (d == 1 ? WL[2] : WL[3]);
    const T unr = d == 0 ? WR[1] : (d == 1 ? WR[2] : WR[3]);
    const T pl = WL[4], pr = WR[4];
    // sound speeds c = sqrt(gamma p / rho) = (gamma p) / sqrt(gamma p rho)
    const T gpl = gamma * pl, gpr = gamma * pr;
    const T cl = gpl * rsqrt_pos(gpl * rl);
    const T cr = gpr * rsqrt_pos(gpr * rr);
    const T a = dmax(dabs(unl) + cl, dabs(unr) + cr);
    // per variable (fL + fR) - a (UR - UL), products of one side fused onto
    // those of the other
    const T fl0 = rl * unl, fr0 = rr * unr;
    F[0] = dfma(-a, rr - rl, fl0 + fr0);
    // momentum: flux = mass flux * velocity (+ p along the normal)
#pragma unroll
    for (int k = 1; k <= 3; ++k) {
        const T f = dfma(fl0, WL[k], k - 1 == d ? pl : T(0)) + dfma(fr0, WR[k], k - 1 == d ? pr : T(0));
        F[k] = dfma(-a, dfma(rr, WR[k], -(rl * WL[k])), f);
    }
    // energy
    const T kel = dfma(WL[1], WL[1], dfma(WL[2], WL[2], WL[3] * WL[3]));
    const T ker = dfma(WR[1], WR[1], dfma(WR[2], WR[2], WR[3] * WR[3]));
    const T El = dfma(C::half * rl, kel, pl * igm1);
    const T Er = dfma(C::half * rr, ker, pr * igm1);
    F[4] = dfma(-a, Er - El, dfma(El + pl, unl, (Er + pr) * unr));
}

// Conservative -> primitive (rho, u, v, w, p).
template <typename T>
__device__ __forceinline__ void to_primitive(T r, T m0, T m1, T m2, T E, T gm1, T (&W)[5])
{
    const T inv = rcp_pos(r);
    const T u = m0 * inv, v = m1 * inv, w = m2 * inv;
    const T ke = K<T>::half * dfma(m0, u, dfma(m1, v, m2 * w));
    W[0] = r;
    W[1] = u;
    W[2] = v;
    W[3] = w;
    W[4] = gm1 * (E - ke);
}

} // namespace euler
} // namespace cn
