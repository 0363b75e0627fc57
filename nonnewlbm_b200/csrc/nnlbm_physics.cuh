// nnlbm_physics.cuh -- per-cell D3Q27 physics for the sm_100a step kernels.
//
// Direction q = 9*(cx+1) + 3*(cy+1) + (cz+1) (the reference enum, solver/lbm3d/defs.h:215-247),
// opposite direction 26-q.  CT is the arithmetic type: float for F32/F16/BF16 storage and
// double for F64 storage.
#pragma once

#include <cuda_runtime.h>
#include <math.h>
#include <stdint.h>

#include <type_traits>

namespace nnlbm {

__host__ __device__ constexpr int cxq(int q) { return q / 9 - 1; }
__host__ __device__ constexpr int cyq(int q) { return (q / 3) % 3 - 1; }
__host__ __device__ constexpr int czq(int q) { return q % 3 - 1; }
__host__ __device__ constexpr int oppq(int q) { return 26 - q; }
__host__ __device__ constexpr int nnzq(int q) { return (cxq(q) != 0) + (cyq(q) != 0) + (czq(q) != 0); }

// lattice weights 8/27, 2/27, 1/54, 1/216 by the number of non-zero velocity components
template <class CT>
__host__ __device__ constexpr CT weight(int q)
{
    return nnzq(q) == 0 ? CT(8.0 / 27.0) : nnzq(q) == 1 ? CT(2.0 / 27.0) : nnzq(q) == 2 ? CT(1.0 / 54.0) : CT(1.0 / 216.0);
}

enum : int { EQ_INV_CUM_REF = 0, EQ_INV_CUM = 1, EQ_DEFAULT = 2, EQ_ENTROPIC = 3 };
enum : int { COL_CUM = 0, COL_KBC_N1 = 1, COL_KBC_N2, COL_KBC_N3, COL_KBC_N4, COL_KBC_C1, COL_KBC_C2,
             COL_KBC_C3, COL_KBC_C4, COL_MRT = 9, COL_BGK = 10 };

template <class CT> __device__ __forceinline__ CT dsqrt(CT v);
template <> __device__ __forceinline__ float dsqrt<float>(float v) { return sqrtf(v); }
template <> __device__ __forceinline__ double dsqrt<double>(double v) { return sqrt(v); }
template <class CT> __device__ __forceinline__ CT dpow(CT b, CT e);
template <> __device__ __forceinline__ float dpow<float>(float b, float e) { return powf(b, e); }
template <> __device__ __forceinline__ double dpow<double>(double b, double e) { return pow(b, e); }

// ---------------------------------------------------------------------------------------
// f2: one quantity of two cells at once on the packed FP32 pipe of sm_100 (FADD2, FMUL2,
// FFMA2), so that the step of two cells issues the arithmetic instructions of one.  Each
// half is rounded exactly as the scalar float operation; division is per half.
// ---------------------------------------------------------------------------------------
struct f2 {
    float2 v;
    __device__ __forceinline__ f2() {}
    __device__ __forceinline__ f2(float2 a) : v(a) {}
    __device__ __forceinline__ f2(float a, float b) : v(make_float2(a, b)) {}
    __device__ __forceinline__ explicit f2(double s) : v(make_float2((float)s, (float)s)) {}
};
__device__ __forceinline__ f2 operator+(f2 a, f2 b) { return __fadd2_rn(a.v, b.v); }
__device__ __forceinline__ f2 operator*(f2 a, f2 b) { return __fmul2_rn(a.v, b.v); }
__device__ __forceinline__ f2 operator-(f2 a, f2 b) { return __ffma2_rn(b.v, make_float2(-1.f, -1.f), a.v); }
__device__ __forceinline__ f2 operator-(f2 a) { return __fmul2_rn(a.v, make_float2(-1.f, -1.f)); }
__device__ __forceinline__ f2 operator/(f2 a, f2 b) { return f2(a.v.x / b.v.x, a.v.y / b.v.y); }
__device__ __forceinline__ f2& operator+=(f2& a, f2 b) { return a = a + b; }
__device__ __forceinline__ f2& operator-=(f2& a, f2 b) { return a = a - b; }
template <> __device__ __forceinline__ f2 dsqrt<f2>(f2 v) { return f2(sqrtf(v.v.x), sqrtf(v.v.y)); }

// a b + c: one rounding for f2 (FFMA2); for float the compiler contracts it under
// --use_fast_math; for double (built with -fmad=false) it is the product, then the sum,
// so an expression rewritten with mad keeps its FP64 rounding
template <class CT>
__device__ __forceinline__ CT mad(CT a, CT b, CT c) { return a * b + c; }
template <>
__device__ __forceinline__ f2 mad<f2>(f2 a, f2 b, f2 c) { return __ffma2_rn(a.v, b.v, c.v); }

// ---------------------------------------------------------------------------------------
// density and velocity with the F/2 shift, in the pairwise order of Geier 2015 Appendix J
// (the order of LBM_COMMON::computeDensityAndVelocity, solver/lbm3d/lbm_common.h:31-38)
// ---------------------------------------------------------------------------------------
template <class CT>
__device__ __forceinline__ void density_velocity(const CT* f, CT fx, CT fy, CT fz, CT& rho, CT& ux, CT& uy, CT& uz)
{
    enum { mmm = 0, mmz, mmp, mzm, mzz, mzp, mpm, mpz, mpp, zmm, zmz, zmp, zzm, zzz, zzp, zpm, zpz, zpp,
           pmm, pmz, pmp, pzm, pzz, pzp, ppm, ppz, ppp };
    rho = ((((f[ppp] + f[mmm]) + (f[pmp] + f[mpm])) + ((f[ppm] + f[mmp]) + (f[mpp] + f[pmm])))
           + (((f[zpp] + f[zmm]) + (f[zpm] + f[zmp])) + ((f[pzp] + f[mzm]) + (f[pzm] + f[mzp]))
              + ((f[ppz] + f[mmz]) + (f[pmz] + f[mpz])))
           + ((f[pzz] + f[mzz]) + (f[zpz] + f[zmz]) + (f[zzp] + f[zzm]))) + f[zzz];
    const CT ir = CT(1) / rho;
    uz = ((((f[ppp] - f[mmm]) + (f[mpp] - f[pmm])) + ((f[pmp] - f[mpm]) + (f[mmp] - f[ppm])))
          + (((f[zpp] - f[zmm]) + (f[zmp] - f[zpm])) + ((f[pzp] - f[mzm]) + (f[mzp] - f[pzm])))
          + (f[zzp] - f[zzm]) + fz * CT(0.5)) * ir;
    ux = ((((f[ppp] - f[mmm]) + (f[pmp] - f[mpm])) + ((f[ppm] - f[mmp]) + (f[pmm] - f[mpp])))
          + (((f[pzp] - f[mzm]) + (f[pzm] - f[mzp])) + ((f[ppz] - f[mmz]) + (f[pmz] - f[mpz])))
          + (f[pzz] - f[mzz]) + fx * CT(0.5)) * ir;
    uy = ((((f[ppp] - f[mmm]) + (f[ppm] - f[mmp])) + ((f[mpp] - f[pmm]) + (f[mpm] - f[pmp])))
          + (((f[ppz] - f[mmz]) + (f[mpz] - f[pmz])) + ((f[zpp] - f[zmm]) + (f[zpm] - f[zmp])))
          + (f[zpz] - f[zmz]) + fy * CT(0.5)) * ir;
}

template <class CT>
__device__ __forceinline__ CT density(const CT* f)
{
    CT r, a, b, c;
    density_velocity<CT>(f, CT(0), CT(0), CT(0), r, a, b, c);
    return r;
}

// ---------------------------------------------------------------------------------------
// equilibria for boundary nodes and initial states
// ---------------------------------------------------------------------------------------
template <class CT>
__device__ __forceinline__ CT inv_cum_factor(int c, CT v)
{
    return c == 0 ? CT(3) * v * v - CT(2) : (c > 0 ? CT(3) * v * v + CT(3) * v + CT(1) : CT(3) * v * v - CT(3) * v + CT(1));
}

// population q of the equilibrium of kind `eq` (q and eq may be runtime values; equilibrium()
// below evaluates the same expression for every q)
template <class CT>
__device__ __forceinline__ CT feq_one(int eq, int q, CT rho, CT ux, CT uy, CT uz)
{
    const int cx = cxq(q), cy = cyq(q), cz = czq(q);
    if (eq == EQ_DEFAULT) {
        // LBM_EQ_DEFAULT, lbm_eq.h:12-47
        const CT u2 = ux * ux + uy * uy + uz * uz;
        const CT cu = CT(cx) * ux + CT(cy) * uy + CT(cz) * uz;
        return weight<CT>(q) * rho * (CT(1) - CT(1.5) * u2 + CT(3) * cu + CT(4.5) * cu * cu);
    }
    if (eq == EQ_ENTROPIC) {
        // LBM_EQ_ENTROPIC, lbm_eq_entropic.h:12-38: per axis weight (2/3 or 1/6) times
        // (2 - sqrt(1+3v^2)) times B^c with B = (2v + sqrt(1+3v^2)) / (1 - v)
        const CT sx = dsqrt<CT>(CT(1) + CT(3) * ux * ux), sy = dsqrt<CT>(CT(1) + CT(3) * uy * uy);
        const CT sz = dsqrt<CT>(CT(1) + CT(3) * uz * uz);
        const CT bx = (CT(2) * ux + sx) / (CT(1) - ux), by = (CT(2) * uy + sy) / (CT(1) - uy), bz = (CT(2) * uz + sz) / (CT(1) - uz);
        const CT base = (CT(2) - sx) * (CT(2) - sy) * (CT(2) - sz);
        CT v = (cx ? CT(1.0 / 6.0) : CT(2.0 / 3.0)) * (cy ? CT(1.0 / 6.0) : CT(2.0 / 3.0)) * (cz ? CT(1.0 / 6.0) : CT(2.0 / 3.0)) * base;
        if (cx > 0) v *= bx; else if (cx < 0) v *= CT(1) / bx;
        if (cy > 0) v *= by; else if (cy < 0) v *= CT(1) / by;
        if (cz > 0) v *= bz; else if (cz < 0) v *= CT(1) / bz;
        return rho * v;
    }
    // factorised equilibrium of LBM_EQ_INV_CUM (lbm_eq_inv_cum.h:71-101): prefactor by the
    // number of zero components 3: -1/27, 2: 1/54, 1: -1/108, 0: 1/216
    const int nz0 = nnzq(q);
    const CT pre = nz0 == 0 ? CT(-1.0 / 27.0) : nz0 == 1 ? CT(1.0 / 54.0) : nz0 == 2 ? CT(-1.0 / 108.0) : CT(1.0 / 216.0);
    CT v = pre * rho * (inv_cum_factor<CT>(cx, ux) * inv_cum_factor<CT>(cy, uy) * inv_cum_factor<CT>(cz, uz));
    // the shipped feq_pmm multiplies by rho twice (lbm_eq_inv_cum.h:49)
    if (eq == EQ_INV_CUM_REF && q == 18) v *= rho;
    return v;
}

// feq of kind `eq` (runtime-uniform switch) into f[27]
template <class CT>
__device__ __forceinline__ void equilibrium(int eq, CT rho, CT ux, CT uy, CT uz, CT* f)
{
#pragma unroll
    for (int q = 0; q < 27; ++q) f[q] = feq_one<CT>(eq, q, rho, ux, uy, uz);
}

// ---------------------------------------------------------------------------------------
// Carreau-Yasuda local viscosity from the non-equilibrium second moments:
// Pi = sum f (c-u)(c-u) - rho/3 I, S = -3/(2 rho tau) Pi, gamma_dot = sqrt(2 S:S),
// nu = nu_inf + (nu0-nu_inf)(1 + (lambda gamma_dot)^a)^((n-1)/a), tau = 3 nu + 1/2, solved by
// three Newton steps on g(tau) = tau - 3 nu_CY(K/tau) - 1/2 from tau = 3 nu0 + 1/2.
// The viscosity law is the reference's (solver/lbm3d/core.h:763-766).
// ---------------------------------------------------------------------------------------
template <class CT>
struct CYParams { CT nu_inf, nu0, lam, a, n; };

// from the central second moments, those on the diagonal reduced by rho/3 (Pxx ..)
template <class CT>
__device__ __forceinline__ CT cy_nu_from_central(CT Pxx, CT Pyy, CT Pzz, CT Cxy, CT Cxz, CT Cyz, CT rho, const CYParams<CT>& p,
                                                 CT* S)
{
    const CT pn = dsqrt<CT>(Pxx * Pxx + Pyy * Pyy + Pzz * Pzz + CT(2) * (Cxy * Cxy + Cxz * Cxz + Cyz * Cyz));
    const CT K = CT(3) * CT(1.4142135623730951) * pn / (CT(2) * rho);
    CT tau = CT(3) * p.nu0 + CT(0.5);
    if (K > CT(0)) {
        const CT e = (p.n - CT(1)) / p.a;
#pragma unroll
        for (int it = 0; it < 3; ++it) {
            const CT g = K / tau;
            // (lambda gamma)^a; in single precision the usual a = 2 is a product
            CT s;
            if constexpr (sizeof(CT) == 4) s = p.a == CT(2) ? (p.lam * g) * (p.lam * g) : dpow<CT>(p.lam * g, p.a);
            else s = dpow<CT>(p.lam * g, p.a);
            const CT pw = dpow<CT>(CT(1) + s, e);
            const CT nuc = p.nu_inf + (p.nu0 - p.nu_inf) * pw;
            const CT G = tau - CT(3) * nuc - CT(0.5);
            const CT gdn = (p.nu0 - p.nu_inf) * (p.n - CT(1)) * s * pw / (CT(1) + s);
            const CT Gp = CT(1) + CT(3) * gdn / tau;
            tau = tau - G / Gp;
        }
    }
    const CT sc = CT(-3) / (CT(2) * rho * tau);
    S[0] = sc * Pxx; S[1] = sc * Cxy; S[2] = sc * Cxz; S[3] = sc * Pyy; S[4] = sc * Cyz; S[5] = sc * Pzz;
    return (tau - CT(0.5)) * CT(1.0 / 3.0);
}

// two cells at once: the same Newton solve in packed arithmetic; the powers, square roots
// and divisions run per half, and a half whose strain is zero keeps tau = 3 nu0 + 1/2
__device__ __forceinline__ f2 cy_nu_from_central(f2 Pxx, f2 Pyy, f2 Pzz, f2 Cxy, f2 Cxz, f2 Cyz, f2 rho,
                                                 const CYParams<float>& p, f2* S)
{
    const f2 third(1.0 / 3.0), half(0.5), three(3.0), one(1.0);
    const f2 pn = dsqrt<f2>(Pxx * Pxx + Pyy * Pyy + Pzz * Pzz + f2(2.0) * (Cxy * Cxy + Cxz * Cxz + Cyz * Cyz));
    const f2 K = three * f2(1.4142135623730951) * pn / (f2(2.0) * rho);
    const f2 tau0 = three * f2(p.nu0) + half;
    f2 tau = tau0;
    const bool ka = K.v.x > 0.f, kb = K.v.y > 0.f;
    if (ka || kb) {
        const float e = (p.n - 1.f) / p.a;
        const f2 dn(p.nu0 - p.nu_inf), ninf(p.nu_inf), lam(p.lam), nm1(p.n - 1.f);
#pragma unroll
        for (int it = 0; it < 3; ++it) {
            const f2 g = K / tau;
            const f2 lg = lam * g;
            // (lambda gamma)^a; the usual a = 2 is a product
            const f2 s = p.a == 2.f ? lg * lg : f2(dpow<float>(lg.v.x, p.a), dpow<float>(lg.v.y, p.a));
            const f2 s1 = one + s;
            const f2 pw(dpow<float>(s1.v.x, e), dpow<float>(s1.v.y, e));
            const f2 nuc = ninf + dn * pw;
            const f2 G = tau - three * nuc - half;
            const f2 gdn = dn * nm1 * s * pw / s1;
            const f2 Gp = one + three * gdn / tau;
            tau = tau - G / Gp;
        }
        tau = f2(ka ? tau.v.x : tau0.v.x, kb ? tau.v.y : tau0.v.y);
    }
    const f2 sc = f2(-3.0) / (f2(2.0) * rho * tau);
    S[0] = sc * Pxx; S[1] = sc * Cxy; S[2] = sc * Cxz; S[3] = sc * Pyy; S[4] = sc * Cyz; S[5] = sc * Pzz;
    return (tau - half) * third;
}

// ---------------------------------------------------------------------------------------
// The collisions of FP32 and FP64 storage work on the stored values themselves: g_q = f_q - w_q
// for FP32 (DT = 1), f_q for FP64 (DT = 0).  (Those of the 16-bit types: nnlbm_physics16.cuh.)
// Every moment is linear in them, so the weights meet a handful of moments (or the factors of
// the equilibrium) instead of each of the 27 populations on the way in and out, and a moment
// of g carries no rounding of the rest state.
//
// PLANES (one cell in single precision): the planes x = -1 and x = 0 run as f2 pairs on the
// packed FP32 pipe, the plane x = +1 scalar.
// ---------------------------------------------------------------------------------------
// the moments of order <= 2 in (y, z), and 21, 12, of the 9 populations 3 iy + iz of one x
// plane: 17 additions (19 with the third order)
template <class V>
struct PlaneMom { V a00, a10, a01, a20, a02, a11, a21, a12; };
template <class V>
__device__ __forceinline__ PlaneMom<V> plane_moments(const V* g)
{
    V s[3], d[3], c[3];
#pragma unroll
    for (int i = 0; i < 3; ++i) {
        s[i] = g[3 * i + 2] + g[3 * i];
        d[i] = g[3 * i + 2] - g[3 * i];
        c[i] = s[i] + g[3 * i + 1];
    }
    PlaneMom<V> p;
    p.a20 = c[2] + c[0];
    p.a00 = p.a20 + c[1];
    p.a10 = c[2] - c[0];
    p.a21 = d[2] + d[0];
    p.a01 = p.a21 + d[1];
    p.a11 = d[2] - d[0];
    p.a02 = (s[2] + s[0]) + s[1];
    p.a12 = s[2] - s[0];
    return p;
}
__device__ __forceinline__ PlaneMom<float> plane_half(const PlaneMom<f2>& p, int h)
{
    auto v = [h](f2 a) { return h ? a.v.y : a.v.x; };
    return {v(p.a00), v(p.a10), v(p.a01), v(p.a20), v(p.a02), v(p.a11), v(p.a21), v(p.a12)};
}

// raw moments of the stored values: r = sum g, j = sum c g, second order, and the third order
// that KBC reads
template <class CT>
struct Moments {
    CT r, jx, jy, jz, xx, yy, zz, xy, xz, yz, xxy, xxz, xyy, yyz, xzz, yzz, xyz;
};
template <class CT>
__device__ __forceinline__ Moments<CT> moments_of_planes(const PlaneMom<CT>& m, const PlaneMom<CT>& z, const PlaneMom<CT>& p)
{
    Moments<CT> M;
    M.xx = p.a00 + m.a00;
    M.r = M.xx + z.a00;
    M.jx = p.a00 - m.a00;
    M.xxy = p.a10 + m.a10;
    M.jy = M.xxy + z.a10;
    M.xy = p.a10 - m.a10;
    M.xxz = p.a01 + m.a01;
    M.jz = M.xxz + z.a01;
    M.xz = p.a01 - m.a01;
    M.yy = (p.a20 + m.a20) + z.a20;
    M.xyy = p.a20 - m.a20;
    M.zz = (p.a02 + m.a02) + z.a02;
    M.xzz = p.a02 - m.a02;
    M.yz = (p.a11 + m.a11) + z.a11;
    M.xyz = p.a11 - m.a11;
    M.yyz = (p.a21 + m.a21) + z.a21;
    M.yzz = (p.a12 + m.a12) + z.a12;
    return M;
}
template <class CT, bool PLANES>
__device__ __forceinline__ Moments<CT> raw_moments(const CT* g)
{
    if constexpr (PLANES) {
        f2 pair[9];
#pragma unroll
        for (int j = 0; j < 9; ++j) pair[j] = f2(g[j], g[9 + j]);
        const PlaneMom<f2> p01 = plane_moments<f2>(pair);
        return moments_of_planes<float>(plane_half(p01, 0), plane_half(p01, 1), plane_moments<float>(g + 18));
    } else {
        return moments_of_planes<CT>(plane_moments<CT>(g), plane_moments<CT>(g + 9), plane_moments<CT>(g + 18));
    }
}

// what a collision starts from: density (dr = rho - 1 with shifted storage, rho itself with
// FP64), u = (j + F/2) / rho, its momentum m = j + F/2, the raw moments (the second moments on
// the diagonal less their rest value 1/3 with shifted storage)
template <class CT>
struct CellState {
    Moments<CT> M;
    CT dr, rho, ir, mx, my, mz, ux, uy, uz;
};
template <class CT, int DT, bool PLANES>
__device__ __forceinline__ CellState<CT> cell_state(const CT* g, CT fx, CT fy, CT fz)
{
    CellState<CT> c;
    c.M = raw_moments<CT, PLANES>(g);
    c.dr = c.M.r;
    c.rho = DT == 0 ? c.dr : c.dr + CT(1);
    c.ir = CT(1) / c.rho;
    c.mx = mad(CT(0.5), fx, c.M.jx);
    c.my = mad(CT(0.5), fy, c.M.jy);
    c.mz = mad(CT(0.5), fz, c.M.jz);
    c.ux = c.mx * c.ir;
    c.uy = c.my * c.ir;
    c.uz = c.mz * c.ir;
    return c;
}

// central second moments (about u) with rho/3 taken off the diagonal:
// C_ab = M_ab - u_a j_b - u_b j_a + rho u_a u_b with j = rho u - F/2
template <class CT>
struct Central { CT xx, yy, zz, xy, xz, yz; };
template <class CT>
__device__ __forceinline__ Central<CT> central_moments(const CellState<CT>& c, CT fx, CT fy, CT fz)
{
    const CT third = c.dr * CT(1.0 / 3.0);
    Central<CT> C;
    C.xx = mad(-c.ux, c.M.jx - CT(0.5) * fx, c.M.xx - third);
    C.yy = mad(-c.uy, c.M.jy - CT(0.5) * fy, c.M.yy - third);
    C.zz = mad(-c.uz, c.M.jz - CT(0.5) * fz, c.M.zz - third);
    C.xy = mad(-c.uy, c.M.jx, mad(c.ux, CT(0.5) * fy, c.M.xy));
    C.xz = mad(-c.uz, c.M.jx, mad(c.ux, CT(0.5) * fz, c.M.xz));
    C.yz = mad(-c.uz, c.M.jy, mad(c.uy, CT(0.5) * fz, c.M.yz));
    return C;
}

// ---------------------------------------------------------------------------------------
// cumulant collision (Geier et al. 2015) with the reference configuration of
// solver/lbm3d/lbm_col_cum.h:166-282: shear rate omega1 = 1/(3 nu + 1/2), every other rate
// 1, A = B = 0, no limiter.  With those rates all cumulants of order >= 3 are reset to
// zero: the collision reads the moments up to second order only, and the post-collision
// central moments of order 4 and 6 are those of a Gaussian (G2015 Eq 81-84 with the odd
// orders zero; the sixth, collected, is
// s222 = (s200 s020 s002 + 2 (s200 s011^2 + s020 s101^2 + s002 s110^2) + 8 s110 s101 s011) / rho^2).
// The first-order ones are F/2.
//
// The populations are rebuilt axis by axis: central -> raw moments (r1 = k1 + u k0,
// r2 = k2 + u (k1 + r1)), the rest state's raw moments taken off, raw moments -> populations
// (p = (r2 + r1)/2, m = (r2 - r1)/2, z = r0 - r2).  Each moment carries a factor 1/2 per axis
// of non-zero order from the start, so that no halving is left: 3 operations a triple
// and direction.
// ---------------------------------------------------------------------------------------
template <class V>
__device__ __forceinline__ void to_raw(V u, V uh, V k0, V& k1, V& k2)
{
    const V r1 = mad(uh, k0, k1);
    k2 = mad(u, k1 + r1, k2);
    k1 = r1;
}
template <class V>
__device__ __forceinline__ void to_pops(V& a, V& b, V& c)
{
    const V p = c + b, m = c - b;
    b = mad(V(-2.0), c, a);
    a = m;
    c = p;
}

// scaled central moments of a cell after the collision: the halves and quarters of the second
// order (x = s200/2, a = s110/4, ...) and the density
template <class CT>
struct CumPost { CT r, x, y, z, a, b, c; };  // a: 110, b: 101, c: 011

// the raw moments k[i][j][l] of the post-collision state (x pass; the orders that vanish are
// left out of the arithmetic)
template <class CT>
__device__ __forceinline__ void cum_x_raw(const CumPost<CT>& s, CT ir, CT ux, CT fx, CT fy, CT fz, CT (&k)[3][3][3])
{
    const CT uh = CT(0.5) * ux;
    const CT four = CT(4), eight = CT(8);
    // fourth and sixth order from products
    const CT s211 = mad(s.x, s.c, four * (s.a * s.b)) * ir;
    const CT s121 = mad(s.y, s.b, four * (s.a * s.c)) * ir;
    const CT s112 = mad(s.z, s.a, four * (s.b * s.c)) * ir;
    const CT s220 = mad(s.x, s.y, eight * (s.a * s.a)) * ir;
    const CT s202 = mad(s.x, s.z, eight * (s.b * s.b)) * ir;
    const CT s022 = mad(s.y, s.z, eight * (s.c * s.c)) * ir;
    const CT s222 = mad(s.x, s022, eight * mad(s.b, s121, s.a * s112)) * ir;
    // first order F/2 (times 1/2)
    k[0][0][0] = s.r; k[1][0][0] = CT(0.25) * fx; k[2][0][0] = s.x;
    to_raw<CT>(ux, uh, k[0][0][0], k[1][0][0], k[2][0][0]);
    // orders (., 1, 0) and (., 0, 1): no k2
    k[0][1][0] = CT(0.25) * fy;
    k[1][1][0] = mad(uh, k[0][1][0], s.a);
    k[2][1][0] = ux * (s.a + k[1][1][0]);
    k[0][0][1] = CT(0.25) * fz;
    k[1][0][1] = mad(uh, k[0][0][1], s.b);
    k[2][0][1] = ux * (s.b + k[1][0][1]);
    // orders (., 2, 0), (., 0, 2), (., 1, 1), (., 2, 2): no k1
    auto even = [&](int j, int l, CT k0, CT k2) {
        k[0][j][l] = k0;
        k[1][j][l] = uh * k0;
        k[2][j][l] = mad(ux, k[1][j][l], k2);
    };
    even(2, 0, s.y, s220);
    even(0, 2, s.z, s202);
    even(1, 1, s.c, s211);
    even(2, 2, s022, s222);
    // orders (., 2, 1) and (., 1, 2): k1 only
    k[0][2][1] = CT(0); k[1][2][1] = s121; k[2][2][1] = ux * (s121 + s121);
    k[0][1][2] = CT(0); k[1][1][2] = s112; k[2][1][2] = ux * (s112 + s112);
}

template <class CT, int DT, bool PLANES>
__device__ __forceinline__ void collide_cum(CT* g, const CellState<CT>& c, const Central<CT>& C, CT fx, CT fy, CT fz, CT nu)
{
    const CT om = CT(1) / (CT(3) * nu + CT(0.5));
    // relaxation (lbm_col_cum.h:205-235 with omega2 = 1): the shear parts by omega1, the trace
    // to rho
    const CT k = CT(1) - om;
    const CT e1 = k * (C.xx - C.yy), e2 = k * (C.xx - C.zz), kq = CT(0.25) * k;
    CumPost<CT> s;
    s.r = c.rho;
    s.x = CT(1.0 / 6.0) * ((e1 + e2) + s.r);
    s.y = mad(CT(-0.5), e1, s.x);
    s.z = mad(CT(-0.5), e2, s.x);
    s.a = kq * C.xy;
    s.b = kq * C.xz;
    s.c = kq * C.yz;
    CT m[3][3][3];
    cum_x_raw<CT>(s, c.ir, c.ux, fx, fy, fz, m);
    const CT w1 = CT(1.0 / 6.0);
    const CT w2 = w1 * CT(1.0 / 6.0), w3 = w2 * CT(1.0 / 6.0);
    // the rest state's raw moments (times 1/2 per axis of order 2) off plane m[i] (order i in x)
    const CT r0 = c.dr;
    if constexpr (PLANES) {
        // orders i = 0, 1 in x as pairs, i = 2 scalar
        f2 P[3][3];
        float Q[3][3];
#pragma unroll
        for (int j = 0; j < 3; ++j)
#pragma unroll
            for (int l = 0; l < 3; ++l) { P[j][l] = f2(m[0][j][l], m[1][j][l]); Q[j][l] = m[2][j][l]; }
        const f2 uy2(c.uy, c.uy), uyh2(0.5f * c.uy, 0.5f * c.uy), uz2(c.uz, c.uz), uzh2(0.5f * c.uz, 0.5f * c.uz);
#pragma unroll
        for (int l = 0; l < 3; ++l) {
            to_raw<f2>(uy2, uyh2, P[0][l], P[1][l], P[2][l]);
            to_raw<float>(uy2.v.x, uyh2.v.x, Q[0][l], Q[1][l], Q[2][l]);
        }
#pragma unroll
        for (int j = 0; j < 3; ++j) {
            to_raw<f2>(uz2, uzh2, P[j][0], P[j][1], P[j][2]);
            to_raw<float>(uz2.v.x, uzh2.v.x, Q[j][0], Q[j][1], Q[j][2]);
        }
        P[0][0].v.x = r0;
        P[2][0].v.x -= w1; P[0][2].v.x -= w1; Q[0][0] -= w1;
        P[2][2].v.x -= w2; Q[2][0] -= w2; Q[0][2] -= w2;
        Q[2][2] -= w3;
#pragma unroll
        for (int l = 0; l < 3; ++l) {
            to_pops<f2>(P[0][l], P[1][l], P[2][l]);
            to_pops<float>(Q[0][l], Q[1][l], Q[2][l]);
        }
#pragma unroll
        for (int j = 0; j < 3; ++j) {
            to_pops<f2>(P[j][0], P[j][1], P[j][2]);
            to_pops<float>(Q[j][0], Q[j][1], Q[j][2]);
#pragma unroll
            for (int l = 0; l < 3; ++l) {
                float a = P[j][l].v.x, b = P[j][l].v.y, d = Q[j][l];
                to_pops<float>(a, b, d);
                g[3 * j + l] = a; g[9 + 3 * j + l] = b; g[18 + 3 * j + l] = d;
            }
        }
    } else {
        const CT uyh = CT(0.5) * c.uy, uzh = CT(0.5) * c.uz;
#pragma unroll
        for (int i = 0; i < 3; ++i) {
#pragma unroll
            for (int l = 0; l < 3; ++l) to_raw<CT>(c.uy, uyh, m[i][0][l], m[i][1][l], m[i][2][l]);
#pragma unroll
            for (int j = 0; j < 3; ++j) to_raw<CT>(c.uz, uzh, m[i][j][0], m[i][j][1], m[i][j][2]);
        }
        if constexpr (DT != 0) {
            m[0][0][0] = r0;
            m[2][0][0] -= w1; m[0][2][0] -= w1; m[0][0][2] -= w1;
            m[2][2][0] -= w2; m[2][0][2] -= w2; m[0][2][2] -= w2;
            m[2][2][2] -= w3;
        }
#pragma unroll
        for (int i = 0; i < 3; ++i) {
#pragma unroll
            for (int l = 0; l < 3; ++l) to_pops<CT>(m[i][0][l], m[i][1][l], m[i][2][l]);
#pragma unroll
            for (int j = 0; j < 3; ++j) to_pops<CT>(m[i][j][0], m[i][j][1], m[i][j][2]);
        }
#pragma unroll
        for (int j = 0; j < 3; ++j)
#pragma unroll
            for (int l = 0; l < 3; ++l) {
                to_pops<CT>(m[0][j][l], m[1][j][l], m[2][j][l]);
                g[3 * j + l] = m[0][j][l]; g[9 + 3 * j + l] = m[1][j][l]; g[18 + 3 * j + l] = m[2][j][l];
            }
    }
}

// ---------------------------------------------------------------------------------------
// factorised equilibrium of the BGK / KBC schemes (lbm_col_bgk.h:43-53, 85-111):
// feq_q = -rho X_cx Y_cy Z_cz with Xz = u^2 - 2/3, Xp = -(u^2 + u + 1/3)/2, Xm = Xp + u
// ---------------------------------------------------------------------------------------
template <class CT>
struct FactEq {
    CT X[3], Y[3], Z[3];
    __device__ __forceinline__ FactEq(CT ux, CT uy, CT uz)
    {
        X[1] = mad(ux, ux, CT(1.0 / 3.0) - CT(1)); X[2] = CT(-0.5) * (X[1] + CT(1) + ux); X[0] = X[2] + ux;
        Y[1] = mad(uy, uy, CT(1.0 / 3.0) - CT(1)); Y[2] = CT(-0.5) * (Y[1] + CT(1) + uy); Y[0] = Y[2] + uy;
        Z[1] = mad(uz, uz, CT(1.0 / 3.0) - CT(1)); Z[2] = CT(-0.5) * (Z[1] + CT(1) + uz); Z[0] = Z[2] + uz;
    }
};

// forcing source S_q of lbm_col_bgk.h:57-83
template <class CT>
__device__ __forceinline__ CT force_src(int q, CT ir, CT ux, CT uy, CT uz, CT fx, CT fy, CT fz)
{
    return (CT(3) * ((CT(cxq(q)) - ux) * fx + (CT(cyq(q)) - uy) * fy + (CT(czq(q)) - uz) * fz)) * ir;
}
// whether a cell carries a body force (the source terms of BGK and KBC vanish without one)
__device__ __forceinline__ bool any_force(float fx, float fy, float fz) { return fx != 0.f || fy != 0.f || fz != 0.f; }
__device__ __forceinline__ bool any_force(double fx, double fy, double fz) { return fx != 0.0 || fy != 0.0 || fz != 0.0; }
__device__ __forceinline__ bool any_force(f2 fx, f2 fy, f2 fz)
{
    return any_force(fx.v.x, fy.v.x, fz.v.x) || any_force(fx.v.y, fy.v.y, fz.v.y);
}
// g_q += k S_q feq_q for every direction, out of line on a copy, so that the
// path without a force keeps its populations in registers
template <class CT>
__device__ __noinline__ void add_force_all(CT* g, CT k, CT rho, CT ir, CT ux, CT uy, CT uz, CT fx, CT fy, CT fz)
{
    const FactEq<CT> E(ux, uy, uz);
#pragma unroll
    for (int q = 0; q < 27; ++q) {
        const CT feq = -rho * E.X[q / 9] * E.Y[(q / 3) % 3] * E.Z[q % 3];
        g[q] += k * force_src<CT>(q, ir, ux, uy, uz, fx, fy, fz) * feq;
    }
}
template <class CT>
__device__ __forceinline__ void add_force(CT* g, CT k, CT rho, CT ir, CT ux, CT uy, CT uz, CT fx, CT fy, CT fz)
{
    CT t[27];
#pragma unroll
    for (int q = 0; q < 27; ++q) t[q] = g[q];
    add_force_all<CT>(t, k, rho, ir, ux, uy, uz, fx, fy, fz);
#pragma unroll
    for (int q = 0; q < 27; ++q) g[q] = t[q];
}

// The equilibrium of BGK and KBC in the units of the stored values, geq_q = (feq_q - w_q) s
// (feq_q s with FP64 storage).  Per axis the factor F is its weight W (1/6, 2/3, 1/6) plus a
// deviation A ((u^2 - u)/2, -u^2, (u^2 + u)/2); the product less w_q is collected as
//   F_i b_jl + T_i,n,   b_jl = B_j F_l + W_j B_l,  B = s rho A,
//   T_i,n = (B_i + s (rho - 1) W_i) W_j W_l
// so that nothing of the size of w_q is ever rounded and taken off again (a population's
// error would then be a bias of the density, the same in every step).
//
// The rounded constants would be such a bias too: the sums over an axis have to be exact, sum F = 1,
// F_+ - F_- = u, sum W = 1, T_0 + 4 T_1 + 4 T_2 = B_i + s (rho - 1) W_i.  So W and the products of
// two W are floats that add up (each within 1.2 units of its value), and with FP64 the outer F come from
// the middle one.  And so would rho u in place of the momentum m, since 1/rho just above 1 rounds up
// more often than down: B = s (m u - m)/2, -s m u, s (m u + m)/2.  Change per step on a periodic lattice
// (24x20x16 cells, 3000 steps), with constants and rho u rounded by themselves -> now: FP64 mass
// 3.3e-16 -> 4e-20 a cell, FP32 momentum (BGK, KBC_N4) 1.3e-7 -> 1.4e-9, 1.2e-9 of it
template <class CT, int DT>
struct GridEq {
    CT X[3], T[3][3], b[3][3];
    // 1/6 and 2/3 as floats with 2 W0 + W1 = 1
    static constexpr double W0 = 11184810.0 / 67108864.0, W1 = 11184811.0 / 16777216.0;
    // p = s m / 2
    __device__ static __forceinline__ void axis(CT u, CT p, CT* B, CT* F)
    {
        B[1] = CT(-2) * p * u;
        B[2] = mad(p, u, p);
        B[0] = mad(p, u, -p);
        const CT uu = u * u;
        F[1] = CT(2.0 / 3.0) - uu;
        if constexpr (DT == 0) {
            F[2] = CT(0.5) * ((CT(1) - F[1]) + u);
            F[0] = F[2] - u;
        } else {
            const CT e = mad(CT(0.5), uu, CT(W0));
            F[2] = mad(CT(0.5), u, e);
            F[0] = mad(CT(-0.5), u, e);
        }
    }
    __device__ __forceinline__ GridEq(const CellState<CT>& c, CT s, CT* Fx, CT* Fy, CT* Fz)
    {
        const CT h = CT(0.5) * s;
        CT Bx[3], By[3], Bz[3];
        axis(c.ux, h * c.mx, Bx, Fx);
        axis(c.uy, h * c.my, By, Fy);
        axis(c.uz, h * c.mz, Bz, Fz);
        const CT W[3] = {CT(W0), CT(W1), CT(W0)};
        const CT sr = s * c.rho, sd = s * c.dr;
#pragma unroll
        for (int i = 0; i < 3; ++i) {
            X[i] = DT == 0 ? sr * Fx[i] : Fx[i];
            if constexpr (DT != 0) {
                const CT t = mad(sd, W[i], Bx[i]);
                // 4/9, 1/9, 1/36 as floats with K_0 + 4 K_1 + 4 K_2 = 1
                T[i][0] = t * CT(14913082.0 / 33554432.0);
                T[i][1] = t * CT(14913080.0 / 134217728.0);
                T[i][2] = t * CT(14913080.0 / 536870912.0);
            }
        }
#pragma unroll
        for (int j = 0; j < 3; ++j)
#pragma unroll
            for (int l = 0; l < 3; ++l) b[j][l] = DT == 0 ? Fy[j] * Fz[l] : mad(By[j], Fz[l], W[j] * Bz[l]);
    }
    __device__ __forceinline__ CT operator()(int i, int j, int l) const
    {
        return DT == 0 ? X[i] * b[j][l] : mad(X[i], b[j][l], T[i][(j != 1) + (l != 1)]);
    }
    // the planes i = 0, 1 as a pair
    __device__ __forceinline__ f2 pair(int j, int l) const
    {
        const int n = (j != 1) + (l != 1);
        return mad(f2(X[0], X[1]), f2(b[j][l], b[j][l]), f2(T[0][n], T[1][n]));
    }
};

// BGK, solver/lbm3d/lbm_col_bgk.h:14-140: g' = (1 - om) g + om geq, the factor om inside geq:
// two operations a direction
template <class CT, int DT, bool PLANES>
__device__ __forceinline__ void collide_bgk(CT* g, const CellState<CT>& c, CT fx, CT fy, CT fz, CT nu)
{
    const CT om = CT(1) / (CT(3) * nu + CT(0.5));
    CT Fx[3], Fy[3], Fz[3];
    const GridEq<CT, DT> E(c, om, Fx, Fy, Fz);
    const CT k = CT(1) - om;
#pragma unroll
    for (int j = 0; j < 3; ++j)
#pragma unroll
        for (int l = 0; l < 3; ++l) {
            const int q = 3 * j + l;
            if constexpr (PLANES) {
                const f2 v = mad(f2(k, k), f2(g[q], g[9 + q]), E.pair(j, l));
                g[q] = v.v.x;
                g[9 + q] = v.v.y;
            } else {
                g[q] = mad(k, g[q], E(0, j, l));
                g[9 + q] = mad(k, g[9 + q], E(1, j, l));
            }
            g[18 + q] = mad(k, g[18 + q], E(2, j, l));
        }
    if (any_force(fx, fy, fz)) add_force<CT>(g, CT(1) - CT(0.5) * om, c.rho, c.ir, c.ux, c.uy, c.uz, fx, fy, fz);
}

// ---------------------------------------------------------------------------------------
// MRT_LES, solver/lbm3d/lbm_col_mrt.h:12-78: second moments relaxed with a Smagorinsky rate,
// everything rebuilt as w_q [rho (1 + 3 c.u) + 9/2 (c c - I/3) : (P - rho I/3)] form.  With P
// and rho less their rest values the brackets give (f - w) directly; opposite directions
// share their even part and differ by the sign of the odd one (3 rho c.u).
// ---------------------------------------------------------------------------------------
template <class CT, int DT>
__device__ __forceinline__ void collide_mrt(CT* g, const CellState<CT>& c, CT nu)
{
    const Moments<CT>& M = c.M;
    const CT third = c.dr * CT(1.0 / 3.0);
    const CT nxx = mad(-c.mx, c.ux, M.xx - third), nyy = mad(-c.my, c.uy, M.yy - third), nzz = mad(-c.mz, c.uz, M.zz - third);
    const CT nxy = mad(-c.mx, c.uy, M.xy), nxz = mad(-c.mx, c.uz, M.xz), nyz = mad(-c.my, c.uz, M.yz);
    const CT Qs = CT(2) * (nxx * nxx + nyy * nyy + nzz * nzz + CT(2) * (nxy * nxy + nxz * nxz + nyz * nyz));
    const CT tau = CT(3) * nu + CT(0.5);
    const CT om = CT(2) / (dsqrt<CT>(tau * tau + CT(2) * CT(0.0342) * CT(9) * dsqrt<CT>(Qs) * c.ir) + tau);
    const CT Pxx = mad(-om, nxx, M.xx), Pyy = mad(-om, nyy, M.yy), Pzz = mad(-om, nzz, M.zz);
    const CT sn = CT(9);
    const CT xy = sn * mad(-om, nxy, M.xy), xz = sn * mad(-om, nxz, M.xz), yz = sn * mad(-om, nyz, M.yz);
    // even part: A + B_a per axis with c_a != 0 + 9 c_a c_b P_ab; odd part: 3 rho c.u
    const CT h = CT(1.5);
    const CT A = mad(CT(-1.5), (Pxx + Pyy) + Pzz, CT(2.5) * c.dr);
    const CT bx = h * mad(CT(3), Pxx, -c.dr), by = h * mad(CT(3), Pyy, -c.dr), bz = h * mad(CT(3), Pzz, -c.dr);
    const CT s3 = CT(3);
    const CT jx = s3 * c.mx, jy = s3 * c.my, jz = s3 * c.mz;
    // direction q and its opposite from the even and odd parts
    auto put = [&](int q, CT e, CT o) {
        const CT w = CT(weight<double>(q));
        g[q] = w * (e + o);
        g[26 - q] = w * (e - o);
    };
    const CT ax = A + bx, ay = A + by, az = A + bz;
    // The rounded weights all carry the same factor 1 + 7.6e-9 (FP32), which would be a bias of what is
    // conserved: along an axis the odd part is what the others leave of the momentum,
    // m/2 - 4 (w_25 + w_26) j, and the rest population what they leave of the density
    auto axis = [&](int q, CT e, CT m, CT j) {
        const CT o = mad(CT(-5), CT(weight<double>(25)) * j, CT(0.5) * m);
        const CT w = CT(weight<double>(q));
        g[q] = mad(w, e, o);
        g[26 - q] = mad(w, e, -o);
    };
    axis(22, ax, c.mx, jx); axis(16, ay, c.my, jy); axis(14, az, c.mz, jz);
    const CT axy = ax + by, axz = ax + bz, ayz = ay + bz, all = axy + bz;
    g[13] = mad(-CT(weight<double>(22)), mad(CT(2), (ax + ay) + az, mad(CT(0.5), all, (axy + axz) + ayz)), c.dr);
    put(25, axy + xy, jx + jy); put(19, axy - xy, jx - jy);
    put(23, axz + xz, jx + jz); put(21, axz - xz, jx - jz);
    put(17, ayz + yz, jy + jz); put(15, ayz - yz, jy - jz);
    put(26, (all + xy) + (xz + yz), (jx + jy) + jz);
    put(24, (all + xy) - (xz + yz), (jx + jy) - jz);
    put(20, (all - xy) + (xz - yz), (jx - jy) + jz);
    put(18, (all - xy) - (xz - yz), (jx - jy) - jz);
}

// ---------------------------------------------------------------------------------------
// KBC (Karlin, Boesch, Chikatamarla 2015), lbm_col_kbc_n.h / lbm_col_kbc_c.h: shear part
// s = D [+T] [+Q] of raw (N) or central (C) moments, entropic stabiliser gamma,
// f -= beta (2 ds + gamma dh) - (1-beta) S feq.  The shear part is linear in the moments:
// ds = s(m) - s(m_eq) = s(m - m_eq).  The 27 ds are formed once (opposite directions share
// their even part) and serve both passes: the products of the stabiliser, whose 1/feq is
// the product of the inverse factors, and the relaxation
// g' = g - beta gamma (g - geq) - beta (2 - gamma) ds, geq = feq - w.
// ---------------------------------------------------------------------------------------
// the entropic stabiliser gamma = 1/beta - (2 - 1/beta) num/den; the reference divides 0/0
// when dh vanishes identically, where gamma*dh is zero for any finite gamma and the
// regularised limit 1/beta is taken
template <class CT>
__device__ __forceinline__ CT kbc_gamma(CT num, CT den, CT beta)
{
    return den != CT(0) ? CT(1) / beta - (CT(2) - CT(1) / beta) * num / den : CT(1) / beta;
}

// ds_q of the moment differences: trace T, normal differences Nxz, Nyz, shears P, third order
// (its order: xxy xxz xyy yyz xzz yzz xyz)
template <class CT, bool USE_T, bool USE_Q>
__device__ __forceinline__ void kbc_shear(CT T, CT Nxz, CT Nyz, CT Pxy, CT Pxz, CT Pyz, const CT* Q, CT* ds)
{
    const CT sixth = CT(1.0 / 6.0), q = CT(0.25), h = CT(0.5);
    CT dx = sixth * (CT(2) * Nxz - Nyz), dy = sixth * (CT(2) * Nyz - Nxz), dz = -(sixth * (Nxz + Nyz));
    if constexpr (USE_T) {
        const CT t = sixth * T;
        dx += t; dy += t; dz += t;
    }
    const CT pxy = q * Pxy, pxz = q * Pxz, pyz = q * Pyz;
    ds[13] = USE_T ? -T : CT(0);
    if constexpr (USE_Q) {
        // the odd part of direction q (an opposite one has its negative)
        auto put = [&](int a, CT e, CT o) { ds[a] = e + o; ds[26 - a] = e - o; };
        put(22, dx, -(h * (Q[2] + Q[4])));
        put(16, dy, -(h * (Q[0] + Q[5])));
        put(14, dz, -(h * (Q[1] + Q[3])));
        put(25, pxy, q * (Q[2] + Q[0])); put(19, -pxy, q * (Q[2] - Q[0]));
        put(23, pxz, q * (Q[4] + Q[1])); put(21, -pxz, q * (Q[4] - Q[1]));
        put(17, pyz, q * (Q[5] + Q[3])); put(15, -pyz, q * (Q[5] - Q[3]));
        const CT e = CT(0.125) * Q[6];
        ds[26] = e; ds[24] = -e; ds[20] = -e; ds[18] = e; ds[0] = -e; ds[2] = e; ds[6] = e; ds[8] = -e;
    } else {
        ds[22] = dx; ds[4] = dx; ds[16] = dy; ds[10] = dy; ds[14] = dz; ds[12] = dz;
        ds[25] = pxy; ds[1] = pxy; ds[19] = -pxy; ds[7] = -pxy;
        ds[23] = pxz; ds[3] = pxz; ds[21] = -pxz; ds[5] = -pxz;
        ds[17] = pyz; ds[9] = pyz; ds[15] = -pyz; ds[11] = -pyz;
        ds[0] = ds[2] = ds[6] = ds[8] = ds[18] = ds[20] = ds[24] = ds[26] = CT(0);
    }
}

template <class CT, int DT, bool CENTRAL, bool USE_T, bool USE_Q>
__device__ __forceinline__ void collide_kbc(CT* g, const CellState<CT>& c, CT fx, CT fy, CT fz, CT nu)
{
    const Moments<CT>& M = c.M;
    const CT rho = c.rho, ux = c.ux, uy = c.uy, uz = c.uz;
    const CT xx = ux * ux, yy = uy * uy, zz = uz * uz;
    const CT cs2 = CT(1.0 / 3.0);
    CT T, Nxz, Nyz, Pxy, Pxz, Pyz, Q[7];
    // m - m_eq; the trace of g lacks the rest state's 1, so rho goes in as dr there
    if constexpr (!CENTRAL) {
        T = (M.xx + M.yy + M.zz) - c.dr - rho * (xx + yy + zz);
        Nxz = (M.xx - M.zz) - rho * (xx - zz);
        Nyz = (M.yy - M.zz) - rho * (yy - zz);
        Pxy = M.xy - rho * ux * uy; Pxz = M.xz - rho * ux * uz; Pyz = M.yz - rho * uy * uz;
        Q[0] = M.xxy - rho * uy * (cs2 + xx); Q[1] = M.xxz - rho * uz * (cs2 + xx);
        Q[2] = M.xyy - rho * ux * (cs2 + yy); Q[3] = M.yyz - rho * uz * (cs2 + yy);
        Q[4] = M.xzz - rho * ux * (cs2 + zz); Q[5] = M.yzz - rho * uy * (cs2 + zz);
        Q[6] = M.xyz - rho * ux * uy * uz;
    } else {
        T = (M.xx + M.yy + M.zz) - c.dr - rho * (xx + yy + zz);
        const CT cT = T + rho; // the central trace itself
        Nxz = (M.xx - M.zz) + rho * (zz - xx);
        Nyz = (M.yy - M.zz) + rho * (zz - yy);
        Pxy = M.xy - rho * ux * uy; Pxz = M.xz - rho * ux * uz; Pyz = M.yz - rho * uy * uz;
        const CT s = CT(6), three = CT(3);
        Q[0] = M.xxy - cs2 * (s * ux * Pxy + uy * (three * xx + CT(2) * Nxz - Nyz + cT));
        Q[1] = M.xxz - cs2 * (s * ux * Pxz + uz * (three * xx + CT(2) * Nxz - Nyz + cT));
        Q[2] = M.xyy - cs2 * (s * uy * Pxy + ux * (three * yy + CT(2) * Nyz - Nxz + cT));
        Q[3] = M.yyz - cs2 * (s * uy * Pyz + uz * (three * yy + CT(2) * Nyz - Nxz + cT));
        Q[4] = M.xzz - cs2 * (s * uz * Pxz + ux * (three * zz - Nyz - Nxz + cT));
        Q[5] = M.yzz - cs2 * (s * uz * Pyz + uy * (three * zz - Nyz - Nxz + cT));
        Q[6] = M.xyz - ux * Pyz - uy * Pxz - uz * Pxy - ux * uy * uz;
    }
    CT ds[27];
    kbc_shear<CT, USE_T, USE_Q>(T, Nxz, Nyz, Pxy, Pxz, Pyz, Q, ds);
    const CT beta = CT(1) / (CT(6) * nu + CT(1));
    CT Fx[3], Fy[3], Fz[3];
    const GridEq<CT, DT> E(c, CT(1), Fx, Fy, Fz);
    CT num = CT(0), den = CT(0);
    {
        // 1/feq, less the factor rho with FP32 storage (gamma takes the ratio of the sums)
        const CT iZ[3] = {CT(1) / Fz[0], CT(1) / Fz[1], CT(1) / Fz[2]};
#pragma unroll
        for (int i = 0; i < 3; ++i)
#pragma unroll
            for (int j = 0; j < 3; ++j) {
                const CT ixy = CT(1) / (E.X[i] * Fy[j]);
#pragma unroll
                for (int l = 0; l < 3; ++l) {
                    const int q = 9 * i + 3 * j + l;
                    const CT dh = (g[q] - E(i, j, l)) - ds[q];
                    const CT t = dh * (ixy * iZ[l]);
                    num = mad(ds[q], t, num);
                    den = mad(dh, t, den);
                }
            }
    }
    const CT gamma = kbc_gamma(num, den, beta);
    const CT bg = beta * gamma, b2 = beta * (CT(2) - gamma);
#pragma unroll
    for (int i = 0; i < 3; ++i)
#pragma unroll
        for (int j = 0; j < 3; ++j)
#pragma unroll
            for (int l = 0; l < 3; ++l) {
                const int q = 9 * i + 3 * j + l;
                g[q] = mad(-b2, ds[q], mad(-bg, g[q] - E(i, j, l), g[q]));
            }
    if (any_force(fx, fy, fz)) add_force<CT>(g, CT(1) - beta, rho, c.ir, ux, uy, uz, fx, fy, fz);
}

// density, velocity and collision of one cell's stored values (or of two cells', CT = f2) with FP32 or
// FP64 storage; see step_cell in nnlbm_physics16.cuh
template <class CT, int COL, int DT, bool PLANES, class PT, class Out>
__device__ __forceinline__ void step_cell_stored(CT* g, CT fx, CT fy, CT fz, CT nu, const CYParams<PT>* cy, Out&& out)
{
    const CellState<CT> c = cell_state<CT, DT, PLANES>(g, fx, fy, fz);
    Central<CT> C;
    if (COL == COL_CUM || cy) C = central_moments<CT>(c, fx, fy, fz);
    if (cy) {
        CT S[6];
        nu = cy_nu_from_central(C.xx, C.yy, C.zz, C.xy, C.xz, C.yz, c.rho, *cy, S);
        out(c.rho, c.ux, c.uy, c.uz, (const CT*)S);
    } else {
        out(c.rho, c.ux, c.uy, c.uz, (const CT*)nullptr);
    }
    if constexpr (COL == COL_CUM) {
        collide_cum<CT, DT, PLANES>(g, c, C, fx, fy, fz, nu);
    } else if constexpr (COL == COL_MRT) {
        collide_mrt<CT, DT>(g, c, nu);
    } else if constexpr (COL == COL_BGK) {
        collide_bgk<CT, DT, PLANES>(g, c, fx, fy, fz, nu);
    } else {
        constexpr bool central = COL >= COL_KBC_C1;
        constexpr int v = central ? COL - COL_KBC_C1 + 1 : COL - COL_KBC_N1 + 1;
        collide_kbc<CT, DT, central, (v == 2 || v == 4), (v == 3 || v == 4)>(g, c, fx, fy, fz, nu);
    }
}

} // namespace nnlbm
