// nnlbm_physics16.cuh -- the collisions of a cell with 16-bit storage, and the choice between them
// and those of nnlbm_physics.cuh.
//
// FP16 and BF16 hold (f - w) sc.  The cell is widened to its populations f in single precision, collided
// there and rounded once, to the stored type.  A value next to a rounding boundary of the 16-bit type
// is stored one unit (FP16 4.9e-4, BF16 3.9e-3 of itself) away by any other order of the same FP32
// operations, and later steps carry that on; on lattices of a million cells, where the rounding noise
// of the cells averages out, a systematic part of the order shows in the sums.  Working on the
// stored values, as FP32 and FP64 storage do, changed the sums of a KBC_N4 junction (x0.75, FP16) that
// way: their error against 64 bits went from 1.1e-6 to 2.0e-6.  So this order is kept.
//
// CT = float is one cell a thread, with the planes x = -1 and x = 0 as f2 pairs; CT = f2 is two
// cells a thread.
#pragma once

#include "nnlbm_physics.cuh"

namespace nnlbm {
namespace pops {

// ---------------------------------------------------------------------------------------
// cumulant collision, the rates of nnlbm_physics.cuh's: only the central moments up to second order are
// needed from the forward transform; the backward transform rebuilds orders 4..6 from products of
// second order ones (G2015 Eq 81-84).
// ---------------------------------------------------------------------------------------
template <class CT>
__device__ __forceinline__ void fwd3(CT m, CT z, CT p, CT u, CT& k0, CT& k1, CT& k2)
{
    // k0 = (p+m)+z, k1 = (p-m) - u k0, k2 = (p+m) - 2u (p-m) + u^2 k0
    const CT s = p + m, d = p - m;
    k0 = s + z;
    k1 = mad(-u, k0, d);
    k2 = mad(u * u, k0, mad(-(CT(2) * u), d, s));
}

// Products of the one-cell cumulant that meet an addition.  Where such a product has other uses, or two
// products meet, the compiler's choice of what to fuse changes with the code around it: the same
// source stored other values after a change elsewhere in the kernel (one population in 10^7, one
// unit of the 16-bit type).  So these are written out.  Fuse: whether the coefficients of a
// backward pass take u^2 unrounded; the values are those that runs have had in each form
// of the step, the one-cell form's even and odd step and the one-cell chunks of the paired form
template <bool ODD, bool IN_PAIR>
struct Fuse {
    static constexpr bool x = IN_PAIR, y = IN_PAIR || ODD, z = IN_PAIR;
};
// a b + c d, the second product unrounded, and a b rounded; two cells at once as the expressions stand
template <class CT>
__device__ __forceinline__ CT mul2(CT a, CT b, CT c, CT d) { return a * b + c * d; }
template <>
__device__ __forceinline__ float mul2<float>(float a, float b, float c, float d) { return __fmaf_rn(c, d, __fmul_rn(a, b)); }
template <class CT>
__device__ __forceinline__ CT mul(CT a, CT b) { return a * b; }
template <>
__device__ __forceinline__ float mul<float>(float a, float b) { return __fmul_rn(a, b); }

// the coefficients of one axis of the backward transform:
// z = k0 (1-u^2) - 2u k1 - k2, m = k0 (u^2-u)/2 + k1 (u - 1/2) + k2/2,
// p = k0 (u^2+u)/2 + k1 (u + 1/2) + k2/2
template <class CT>
struct Bwd {
    CT a, b, c, d, e, ntu;
    __device__ __forceinline__ explicit Bwd(CT u)
    {
        const CT uu = u * u;
        a = CT(1) - uu; b = CT(0.5) * (uu - u); c = u - CT(0.5); d = CT(0.5) * (uu + u); e = u + CT(0.5); ntu = CT(-2) * u;
    }
};
template <>
struct Bwd<float> {
    float a, b, c, d, e, ntu;
    __device__ __forceinline__ Bwd(float u, bool fuse)
    {
        const float uu = mul(u, u);
        a = fuse ? __fmaf_rn(-u, u, 1.f) : 1.f - uu;
        b = 0.5f * (fuse ? __fmaf_rn(u, u, -u) : uu - u);
        d = 0.5f * (fuse ? __fmaf_rn(u, u, u) : uu + u);
        c = u - 0.5f; e = u + 0.5f; ntu = -2.f * u;
    }
};

template <class CT>
__device__ __forceinline__ void bwd3(CT k0, CT k1, CT k2, const Bwd<CT>& w, CT& m, CT& z, CT& p)
{
    const CT h = CT(0.5) * k2;
    z = mad(k0, w.a, mad(w.ntu, k1, -k2));
    m = mad(k0, w.b, mad(k1, w.c, h));
    p = mad(k0, w.d, mad(k1, w.e, h));
}
__device__ __forceinline__ void bwd2(float k0, float k1, const Bwd<float>& w, float& m, float& z, float& p)
{
    z = mul2(k0, w.a, w.ntu, k1);
    m = mul2(k1, w.c, k0, w.b);
    p = mul2(k1, w.e, k0, w.d);
}

// the Carreau-Yasuda viscosity from the central second moments, not yet reduced by rho/3 on the diagonal
template <class CT, class PT>
__device__ __forceinline__ CT cy_nu(CT Cxx, CT Cyy, CT Czz, CT Cxy, CT Cxz, CT Cyz, CT rho, const CYParams<PT>& p, CT* S)
{
    const CT Pxx = Cxx - rho * CT(1.0 / 3.0), Pyy = Cyy - rho * CT(1.0 / 3.0), Pzz = Czz - rho * CT(1.0 / 3.0);
    return cy_nu_from_central(Pxx, Pyy, Pzz, Cxy, Cxz, Cyz, rho, p, S);
}

// the first half of the forward z pass, which needs no velocity: per (x, y) column of
// populations (m, z, p) at f[9 ix + 3 iy + 0..2], its sum k0 = (p + m) + z, d = p - m and
// s = p + m, in place
template <class CT>
__device__ __forceinline__ void cum_columns(CT* f)
{
#pragma unroll
    for (int c = 0; c < 9; ++c) {
        const CT m = f[3 * c], z = f[3 * c + 1], p = f[3 * c + 2];
        const CT sp = p + m, d = p - m;
        f[3 * c] = sp + z;
        f[3 * c + 1] = d;
        f[3 * c + 2] = sp;
    }
}

// density and velocity u = (j + F/2) / rho from the columns of cum_columns: rho sums the
// column sums, j_z their d, j_y and j_x the column sums' differences across y and x
template <class CT>
__device__ __forceinline__ void cum_density_velocity(const CT* k, CT fx, CT fy, CT fz, CT& rho, CT& ux, CT& uy, CT& uz)
{
    auto k0 = [&](int ix, int iy) { return k[9 * ix + 3 * iy]; };
    auto d = [&](int ix, int iy) { return k[9 * ix + 3 * iy + 1]; };
    const CT rx0 = (k0(0, 0) + k0(0, 2)) + k0(0, 1), rx1 = (k0(1, 0) + k0(1, 2)) + k0(1, 1), rx2 = (k0(2, 0) + k0(2, 2)) + k0(2, 1);
    rho = (rx0 + rx2) + rx1;
    const CT ir = CT(1) / rho;
    ux = mul<CT>((rx2 - rx0) + fx * CT(0.5), ir);
    uy = mul<CT>(((k0(0, 2) - k0(0, 0)) + (k0(2, 2) - k0(2, 0))) + (k0(1, 2) - k0(1, 0)) + fy * CT(0.5), ir);
    uz = mul<CT>((((d(0, 0) + d(0, 2)) + (d(2, 0) + d(2, 2))) + ((d(0, 1) + d(2, 1)) + (d(1, 0) + d(1, 2)))) + d(1, 1) + fz * CT(0.5), ir);
}

// the relaxation of the cumulant (lbm_col_cum.h:205-235 with omega2 = 1 and no anti-aliasing
// terms) from the central moments k of total order <= 2: s receives the post-collision
// cumulants as central moments (orders 3 and 5 zero).  `cy` non-null: the shear viscosity
// comes from the Carreau-Yasuda law on k's second moments, S receives the strain rate
template <class CT, class PT>
__device__ __forceinline__ void cum_relax(const CT (&k)[3][3][3], CT rho, CT nu, const CYParams<PT>* cy, CT* S, CT (&s)[3][3][3])
{
    const CT ir = CT(1) / rho;
    if (cy) nu = cy_nu<CT>(k[2][0][0], k[0][2][0], k[0][0][2], k[1][1][0], k[1][0][1], k[0][1][1], rho, *cy, S);
    const CT om = CT(1) / (CT(3) * nu + CT(0.5));
    const CT k000 = k[0][0][0];
    // relaxation (lbm_col_cum.h:205-235 with omega2 = 1 and no anti-aliasing terms)
    const CT s110 = (CT(1) - om) * k[1][1][0];
    const CT s101 = (CT(1) - om) * k[1][0][1];
    const CT s011 = (CT(1) - om) * k[0][1][1];
    const CT e33 = mul<CT>(CT(1) - om, k[2][0][0] - k[0][2][0]);
    const CT e34 = mul<CT>(CT(1) - om, k[2][0][0] - k[0][0][2]);
    const CT s200 = CT(1.0 / 3.0) * (e33 + e34 + k000);
    const CT s020 = CT(1.0 / 3.0) * (CT(-2) * e33 + e34 + k000);
    const CT s002 = CT(1.0 / 3.0) * (e33 - CT(2) * e34 + k000);
    // fourth order from products (Eq 81-82); third and fifth order vanish
    const CT s211 = mul2<CT>(s200, s011, CT(2) * s101, s110) * ir;
    const CT s121 = mul2<CT>(s020, s101, CT(2) * s110, s011) * ir;
    const CT s112 = mul2<CT>(s002, s110, CT(2) * s011, s101) * ir;
    const CT s220 = mul2<CT>(s020, s200, CT(2) * s110, s110) * ir;
    const CT s022 = mul2<CT>(s002, s020, CT(2) * s011, s011) * ir;
    const CT s202 = mul2<CT>(s200, s002, CT(2) * s101, s101) * ir;
    // sixth order (Eq 84 with the odd orders at zero)
    CT s222;
    if constexpr (std::is_same<CT, float>::value) {
        const float p = __fmaf_rn(4.f, mad(s110, s112, mul2(s101, s121, s011, s211)), mad(s002, s220, mul2(s020, s202, s200, s022)));
        const float r = __fmaf_rn(mul(16.f * s110, s101), s011,
                                  4.f * mad(mul(s110, s110), s002, mul2(mul(s011, s011), s200, mul(s101, s101), s020)));
        s222 = mul2(-mul(mad(mul(2.f * s200, s020), s002, r), ir), ir, p, ir);
    } else {
        s222 = (s200 * s022 + s020 * s202 + s002 * s220 + CT(4) * (s011 * s211 + s101 * s121 + s110 * s112)) * ir
               - (CT(16) * s110 * s101 * s011 + CT(4) * (s101 * s101 * s020 + s011 * s011 * s200 + s110 * s110 * s002)
                  + CT(2) * s200 * s020 * s002) * ir * ir;
    }

#pragma unroll
    for (int i = 0; i < 3; ++i)
#pragma unroll
        for (int j = 0; j < 3; ++j)
#pragma unroll
            for (int l = 0; l < 3; ++l) s[i][j][l] = CT(0);
    s[0][0][0] = k000;
    s[1][0][0] = -k[1][0][0]; s[0][1][0] = -k[0][1][0]; s[0][0][1] = -k[0][0][1];
    s[1][1][0] = s110; s[1][0][1] = s101; s[0][1][1] = s011;
    s[2][0][0] = s200; s[0][2][0] = s020; s[0][0][2] = s002;
    s[2][1][1] = s211; s[1][2][1] = s121; s[1][1][2] = s112;
    s[2][2][0] = s220; s[0][2][2] = s022; s[2][0][2] = s202;
    s[2][2][2] = s222;
}

// `f`: the columns of cum_columns; the post-collision populations replace them
template <class CT, class PT>
__device__ __forceinline__ void collide_cum_columns(CT* f, CT rho, CT ux, CT uy, CT uz, CT nu, const CYParams<PT>* cy, CT* S)
{
    // forward: the z pass's second half over the 9 (x,y) columns (fwd3 from k0, d, s)
    CT a[3][3][3];
    const CT uzz = uz * uz, m2uz = CT(-2) * uz;
#pragma unroll
    for (int ix = 0; ix < 3; ++ix)
#pragma unroll
        for (int iy = 0; iy < 3; ++iy) {
            const CT c0 = f[9 * ix + 3 * iy], d = f[9 * ix + 3 * iy + 1], sp = f[9 * ix + 3 * iy + 2];
            a[ix][iy][0] = c0;
            a[ix][iy][1] = mad(-uz, c0, d);
            a[ix][iy][2] = mad(uzz, c0, mad(m2uz, d, sp));
        }
    // y pass
    CT b[3][3][3];
#pragma unroll
    for (int ix = 0; ix < 3; ++ix)
#pragma unroll
        for (int kz = 0; kz < 3; ++kz)
            fwd3<CT>(a[ix][0][kz], a[ix][1][kz], a[ix][2][kz], uy, b[ix][0][kz], b[ix][1][kz], b[ix][2][kz]);
    // x pass, only the moments of total order <= 2 are used below
    CT k[3][3][3];
#pragma unroll
    for (int ky = 0; ky < 3; ++ky)
#pragma unroll
        for (int kz = 0; kz < 3; ++kz)
            if (ky + kz <= 2) fwd3<CT>(b[0][ky][kz], b[1][ky][kz], b[2][ky][kz], ux, k[0][ky][kz], k[1][ky][kz], k[2][ky][kz]);

    CT s[3][3][3];
    cum_relax<CT, PT>(k, rho, nu, cy, S, s);
    // backward: x, y, z (G2015 Eq 88-96), each axis's coefficients made just before its pass
    {
        const Bwd<CT> wx(ux);
#pragma unroll
        for (int ky = 0; ky < 3; ++ky)
#pragma unroll
            for (int kz = 0; kz < 3; ++kz)
                bwd3<CT>(s[0][ky][kz], s[1][ky][kz], s[2][ky][kz], wx, b[0][ky][kz], b[1][ky][kz], b[2][ky][kz]);
    }
    {
        const Bwd<CT> wy(uy);
#pragma unroll
        for (int ix = 0; ix < 3; ++ix)
#pragma unroll
            for (int kz = 0; kz < 3; ++kz)
                bwd3<CT>(b[ix][0][kz], b[ix][1][kz], b[ix][2][kz], wy, a[ix][0][kz], a[ix][1][kz], a[ix][2][kz]);
    }
    {
        const Bwd<CT> wz(uz);
#pragma unroll
        for (int ix = 0; ix < 3; ++ix)
#pragma unroll
            for (int iy = 0; iy < 3; ++iy)
                bwd3<CT>(a[ix][iy][0], a[ix][iy][1], a[ix][iy][2], wz, f[9 * ix + 3 * iy], f[9 * ix + 3 * iy + 1],
                         f[9 * ix + 3 * iy + 2]);
    }
}

// The cumulant step of one cell in single precision with the columns of x = -1 and x = 0
// packed into f2 (the packed FP32 pipe runs both at once): the z and y passes of both
// transforms treat the 18 populations of those two x planes as 9 pairs, the x passes (which
// combine the planes) and the relaxation run scalar.  The operations and their order are
// those of cum_columns / collide_cum_columns, so the results are bitwise the same.
template <class FUSE>
__device__ __forceinline__ void step_cell_cum_packed(float* f, float fx, float fy, float fz, float nu, const CYParams<float>* cy,
                                                     float* S, float& rho, float& ux, float& uy, float& uz)
{
    // z pass, first half: per column (iy) of the planes ix = 0, 1 (P) and ix = 2 (Q)
    f2 c0P[3], dP[3], spP[3];
    float c0Q[3], dQ[3], spQ[3];
#pragma unroll
    for (int iy = 0; iy < 3; ++iy) {
        const f2 m(f[3 * iy], f[9 + 3 * iy]), z(f[3 * iy + 1], f[9 + 3 * iy + 1]), p(f[3 * iy + 2], f[9 + 3 * iy + 2]);
        spP[iy] = p + m;
        dP[iy] = p - m;
        c0P[iy] = spP[iy] + z;
        const float mq = f[18 + 3 * iy], zq = f[18 + 3 * iy + 1], pq = f[18 + 3 * iy + 2];
        spQ[iy] = pq + mq;
        dQ[iy] = pq - mq;
        c0Q[iy] = spQ[iy] + zq;
    }
    {
        float k[27];
#pragma unroll
        for (int iy = 0; iy < 3; ++iy) {
            k[3 * iy] = c0P[iy].v.x; k[9 + 3 * iy] = c0P[iy].v.y; k[18 + 3 * iy] = c0Q[iy];
            k[3 * iy + 1] = dP[iy].v.x; k[9 + 3 * iy + 1] = dP[iy].v.y; k[18 + 3 * iy + 1] = dQ[iy];
        }
        cum_density_velocity<float>(k, fx, fy, fz, rho, ux, uy, uz);
    }
    // z pass, second half
    f2 aP[3][3];
    float aQ[3][3];
    {
        const f2 nuz(-uz), uzz(uz * uz), m2uz(-2.f * uz);
#pragma unroll
        for (int iy = 0; iy < 3; ++iy) {
            aP[iy][0] = c0P[iy];
            aP[iy][1] = mad(nuz, c0P[iy], dP[iy]);
            aP[iy][2] = mad(uzz, c0P[iy], mad(m2uz, dP[iy], spP[iy]));
            aQ[iy][0] = c0Q[iy];
            aQ[iy][1] = mad(-uz, c0Q[iy], dQ[iy]);
            aQ[iy][2] = mad(uz * uz, c0Q[iy], mad(-2.f * uz, dQ[iy], spQ[iy]));
        }
    }
    // y pass
    f2 bP[3][3];
    float bQ[3][3];
#pragma unroll
    for (int kz = 0; kz < 3; ++kz) {
        fwd3<f2>(aP[0][kz], aP[1][kz], aP[2][kz], f2(uy), bP[0][kz], bP[1][kz], bP[2][kz]);
        fwd3<float>(aQ[0][kz], aQ[1][kz], aQ[2][kz], uy, bQ[0][kz], bQ[1][kz], bQ[2][kz]);
    }
    // x pass (scalar), orders <= 2
    float k[3][3][3];
#pragma unroll
    for (int ky = 0; ky < 3; ++ky)
#pragma unroll
        for (int kz = 0; kz < 3; ++kz)
            if (ky + kz <= 2) fwd3<float>(bP[ky][kz].v.x, bP[ky][kz].v.y, bQ[ky][kz], ux, k[0][ky][kz], k[1][ky][kz], k[2][ky][kz]);
    float s[3][3][3];
    cum_relax<float, float>(k, rho, nu, cy, S, s);
    // backward x (scalar): the planes ix = 0, 1 of each (ky, kz) land as one pair
    {
        const Bwd<float> wx(ux, FUSE::x);
#pragma unroll
        for (int ky = 0; ky < 3; ++ky)
#pragma unroll
            for (int kz = 0; kz < 3; ++kz) {
                float m, z, p;
                // (no second order in x beside a first order in y or z)
                if (ky + kz == 1) bwd2(s[0][ky][kz], s[1][ky][kz], wx, m, z, p);
                else bwd3<float>(s[0][ky][kz], s[1][ky][kz], s[2][ky][kz], wx, m, z, p);
                bP[ky][kz] = f2(m, z);
                bQ[ky][kz] = p;
            }
    }
    // backward y
    {
        const Bwd<f2> wy2{f2(uy)};
        const Bwd<float> wy(uy, FUSE::y);
#pragma unroll
        for (int kz = 0; kz < 3; ++kz) {
            bwd3<f2>(bP[0][kz], bP[1][kz], bP[2][kz], wy2, aP[0][kz], aP[1][kz], aP[2][kz]);
            bwd3<float>(bQ[0][kz], bQ[1][kz], bQ[2][kz], wy, aQ[0][kz], aQ[1][kz], aQ[2][kz]);
        }
    }
    // backward z, into the populations
    {
        const Bwd<f2> wz2{f2(uz)};
        const Bwd<float> wz(uz, FUSE::z);
#pragma unroll
        for (int iy = 0; iy < 3; ++iy) {
            f2 m, z, p;
            bwd3<f2>(aP[iy][0], aP[iy][1], aP[iy][2], wz2, m, z, p);
            f[3 * iy] = m.v.x; f[9 + 3 * iy] = m.v.y;
            f[3 * iy + 1] = z.v.x; f[9 + 3 * iy + 1] = z.v.y;
            f[3 * iy + 2] = p.v.x; f[9 + 3 * iy + 2] = p.v.y;
            bwd3<float>(aQ[iy][0], aQ[iy][1], aQ[iy][2], wz, f[18 + 3 * iy], f[18 + 3 * iy + 1], f[18 + 3 * iy + 2]);
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
        X[1] = CT(1.0 / 3.0) - CT(1) + ux * ux; X[2] = CT(-0.5) * (X[1] + CT(1) + ux); X[0] = X[2] + ux;
        Y[1] = CT(1.0 / 3.0) - CT(1) + uy * uy; Y[2] = CT(-0.5) * (Y[1] + CT(1) + uy); Y[0] = Y[2] + uy;
        Z[1] = CT(1.0 / 3.0) - CT(1) + uz * uz; Z[2] = CT(-0.5) * (Z[1] + CT(1) + uz); Z[0] = Z[2] + uz;
    }
    __device__ __forceinline__ CT operator()(int q, CT rho) const { return -rho * X[q / 9] * Y[(q / 3) % 3] * Z[q % 3]; }
};

// BGK, solver/lbm3d/lbm_col_bgk.h:14-140
template <class CT>
__device__ __forceinline__ void collide_bgk(CT* f, CT rho, CT ux, CT uy, CT uz, CT fx, CT fy, CT fz, CT nu)
{
    const CT om = CT(1) / (CT(3) * nu + CT(0.5));
    const CT ir = CT(1) / rho;
    const FactEq<CT> E(ux, uy, uz);
#pragma unroll
    for (int q = 0; q < 27; ++q) {
        const CT feq = E(q, rho);
        f[q] += (feq - f[q]) * om + (CT(1) - CT(0.5) * om) * force_src<CT>(q, ir, ux, uy, uz, fx, fy, fz) * feq;
    }
}

// density and velocity of one cell in single precision from its column sums (the z pass's
// first half, cum_columns, with the columns of the planes x = -1, 0 as packed pairs), f
// unchanged
__device__ __forceinline__ void packed_density_velocity(const float* f, float fx, float fy, float fz, float& rho, float& ux,
                                                        float& uy, float& uz)
{
    float k[27];
#pragma unroll
    for (int iy = 0; iy < 3; ++iy) {
        const f2 m(f[3 * iy], f[9 + 3 * iy]), z(f[3 * iy + 1], f[9 + 3 * iy + 1]), p(f[3 * iy + 2], f[9 + 3 * iy + 2]);
        const f2 d = p - m, c0 = (p + m) + z;
        const float mq = f[18 + 3 * iy], zq = f[18 + 3 * iy + 1], pq = f[18 + 3 * iy + 2];
        k[3 * iy] = c0.v.x; k[9 + 3 * iy] = c0.v.y; k[18 + 3 * iy] = (pq + mq) + zq;
        k[3 * iy + 1] = d.v.x; k[9 + 3 * iy + 1] = d.v.y; k[18 + 3 * iy + 1] = pq - mq;
    }
    cum_density_velocity<float>(k, fx, fy, fz, rho, ux, uy, uz);
}

// BGK of one cell in single precision with the populations of the planes x = -1 and x = 0
// packed into f2 pairs (the same operations in the same order as collide_bgk; the x = +1
// plane runs scalar)
__device__ __forceinline__ void collide_bgk_packed(float* f, float rho, float ux, float uy, float uz, float fx, float fy,
                                                   float fz, float nu)
{
    const float om = 1.f / (3.f * nu + 0.5f);
    const float ir = 1.f / rho;
    const float k = 1.f - 0.5f * om;
    const FactEq<float> E(ux, uy, uz);
    const f2 rX(-rho * E.X[0], -rho * E.X[1]);
    const float rX2 = -rho * E.X[2];
    const f2 A((-1.f - ux) * fx, (0.f - ux) * fx);
    const float A2 = (1.f - ux) * fx;
    const f2 om2(om), k2(k), three(3.0), ir2(ir);
#pragma unroll
    for (int iy = 0; iy < 3; ++iy)
#pragma unroll
        for (int iz = 0; iz < 3; ++iz) {
            const int j = 3 * iy + iz;
            const float Y = E.Y[iy], Z = E.Z[iz];
            const float B = ((float)(iy - 1) - uy) * fy, C = ((float)(iz - 1) - uz) * fz;
            const f2 feq = (rX * f2(Y, Y)) * f2(Z, Z);
            const f2 src = (three * ((A + f2(B, B)) + f2(C, C))) * ir2;
            const f2 fv(f[j], f[9 + j]);
            const f2 nv = fv + mad(feq - fv, om2, (k2 * src) * feq);
            f[j] = nv.v.x;
            f[9 + j] = nv.v.y;
            const float feq1 = (rX2 * Y) * Z;
            const float src1 = (3.f * ((A2 + B) + C)) * ir;
            f[18 + j] += (feq1 - f[18 + j]) * om + (k * src1) * feq1;
        }
}

// MRT_LES, solver/lbm3d/lbm_col_mrt.h:12-78: second moments relaxed with a Smagorinsky rate,
// everything rebuilt as w_q [rho (1 + 3 c.u) + 9/2 (c c - I/3) : (P - rho I/3)] form
// the relaxed second moments of MRT_LES (P, and tr = trace P) from the populations
template <class CT>
__device__ __forceinline__ void mrt_moments(const CT* f, CT rho, CT ux, CT uy, CT uz, CT nu, CT& Pxx, CT& Pyy, CT& Pzz, CT& Pxy,
                                            CT& Pxz, CT& Pyz, CT& tr)
{
    Pxx = CT(0); Pyy = CT(0); Pzz = CT(0); Pxy = CT(0); Pxz = CT(0); Pyz = CT(0);
#pragma unroll
    for (int q = 0; q < 27; ++q) {
        const int cx = cxq(q), cy = cyq(q), cz = czq(q);
        if (cx) Pxx += f[q];
        if (cy) Pyy += f[q];
        if (cz) Pzz += f[q];
        if (cx * cy > 0) Pxy += f[q]; else if (cx * cy < 0) Pxy -= f[q];
        if (cx * cz > 0) Pxz += f[q]; else if (cx * cz < 0) Pxz -= f[q];
        if (cy * cz > 0) Pyz += f[q]; else if (cy * cz < 0) Pyz -= f[q];
    }
    const CT Pnxx = Pxx - rho * (CT(1.0 / 3.0) + ux * ux);
    const CT Pnyy = Pyy - rho * (CT(1.0 / 3.0) + uy * uy);
    const CT Pnzz = Pzz - rho * (CT(1.0 / 3.0) + uz * uz);
    const CT Pnxz = Pxz - rho * ux * uz;
    const CT Pnxy = Pxy - rho * ux * uy;
    const CT Pnyz = Pyz - rho * uy * uz;
    const CT Qs = CT(2) * (Pnxx * Pnxx + Pnyy * Pnyy + Pnzz * Pnzz + CT(2) * (Pnxy * Pnxy + Pnxz * Pnxz + Pnyz * Pnyz));
    const CT tau = CT(3) * nu + CT(0.5);
    const CT om = CT(2) / (dsqrt<CT>(tau * tau + CT(2) * CT(0.0342) * CT(9) * dsqrt<CT>(Qs) / rho) + tau);
    Pxx -= om * Pnxx; Pyy -= om * Pnyy; Pzz -= om * Pnzz;
    Pxy -= om * Pnxy; Pxz -= om * Pnxz; Pyz -= om * Pnyz;
    tr = Pxx + Pyy + Pzz;
}

template <class CT>
__device__ __forceinline__ void collide_mrt(CT* f, CT rho, CT ux, CT uy, CT uz, CT nu)
{
    CT Pxx, Pyy, Pzz, Pxy, Pxz, Pyz, tr;
    mrt_moments<CT>(f, rho, ux, uy, uz, nu, Pxx, Pyy, Pzz, Pxy, Pxz, Pyz, tr);
#pragma unroll
    for (int q = 0; q < 27; ++q) {
        const int cx = cxq(q), cy = cyq(q), cz = czq(q);
        const int c2 = cx * cx + cy * cy + cz * cz;
        const CT cu = CT(cx) * ux + CT(cy) * uy + CT(cz) * uz;
        const CT pp = CT(cx * cx) * Pxx + CT(cy * cy) * Pyy + CT(cz * cz) * Pzz
                      + CT(2) * (CT(cx * cy) * Pxy + CT(cx * cz) * Pxz + CT(cy * cz) * Pyz);
        f[q] = weight<CT>(q) * (rho * (CT(2.5) - CT(1.5) * CT(c2) + CT(3) * cu) + CT(4.5) * pp - CT(1.5) * tr);
    }
}

// MRT_LES of one cell in single precision, its rebuild with the planes x = -1 and x = 0 as
// packed f2 pairs (the terms without c_x are shared by the pair; the x = +1 plane runs
// scalar)
__device__ __forceinline__ void collide_mrt_packed(float* f, float rho, float ux, float uy, float uz, float nu)
{
    float Pxx, Pyy, Pzz, Pxy, Pxz, Pyz, tr;
    mrt_moments<float>(f, rho, ux, uy, uz, nu, Pxx, Pyy, Pzz, Pxy, Pxz, Pyz, tr);
    const f2 rho2(rho, rho), ux0(-ux, 0.f), three(3.0), p45(4.5), tr15(1.5f * tr, 1.5f * tr);
#pragma unroll
    for (int iy = 0; iy < 3; ++iy)
#pragma unroll
        for (int iz = 0; iz < 3; ++iz) {
            const int cy = iy - 1, cz = iz - 1, j = 3 * iy + iz;
            const float s_cu = (float)cy * uy + (float)cz * uz;
            const float s_pp = (float)(cy * cy) * Pyy + (float)(cz * cz) * Pzz + 2.f * (float)(cy * cz) * Pyz;
            const float x_pp = 2.f * ((float)cy * Pxy + (float)cz * Pxz);
            const int s_c2 = cy * cy + cz * cz;
            // x = -1 (c_x^2 = 1) and x = 0
            const f2 cu = ux0 + f2(s_cu, s_cu);
            const f2 pp = f2(Pxx - x_pp, 0.f) + f2(s_pp, s_pp);
            const f2 k(2.5f - 1.5f * (float)(1 + s_c2), 2.5f - 1.5f * (float)s_c2);
            const f2 w(weight<float>(j), weight<float>(9 + j));
            const f2 v = w * (mad(rho2, mad(three, cu, k), p45 * pp) - tr15);
            f[j] = v.v.x;
            f[9 + j] = v.v.y;
            // x = +1
            const float cu1 = ux + s_cu, pp1 = Pxx + x_pp + s_pp;
            f[18 + j] = weight<float>(18 + j) * (rho * (2.5f - 1.5f * (float)(1 + s_c2) + 3.f * cu1) + 4.5f * pp1 - 1.5f * tr);
        }
}

// ---------------------------------------------------------------------------------------
// KBC (Karlin, Boesch, Chikatamarla 2015), lbm_col_kbc_n.h / lbm_col_kbc_c.h: shear part
// s = D [+T] [+Q] of raw (N) or central (C) moments, entropic stabiliser gamma,
// f -= beta (2 ds + gamma dh) - (1-beta) S feq.  Two passes over q keep the per-direction
// temporaries out of registers.
// ---------------------------------------------------------------------------------------
template <class CT>
struct KbcMom { CT T, Nxz, Nyz, Pxy, Pxz, Pyz, Qxxy, Qxxz, Qxyy, Qyyz, Qxzz, Qyzz, Qxyz; };

template <class CT, bool USE_T, bool USE_Q>
__device__ __forceinline__ CT kbc_shear(int q, const KbcMom<CT>& m)
{
    const int cx = cxq(q), cy = cyq(q), cz = czq(q), nz0 = nnzq(q);
    CT D = CT(0), T = CT(0), Qv = CT(0);
    if (nz0 == 1) {
        if (cx) D = (CT(2) * m.Nxz - m.Nyz) * CT(1.0 / 6.0);
        if (cy) D = (-m.Nxz + CT(2) * m.Nyz) * CT(1.0 / 6.0);
        if (cz) D = (-m.Nxz - m.Nyz) * CT(1.0 / 6.0);
        T = m.T * CT(1.0 / 6.0);
        if (cx) Qv = CT(-cx) * (m.Qxyy + m.Qxzz) * CT(0.5);
        if (cy) Qv = CT(-cy) * (m.Qxxy + m.Qyzz) * CT(0.5);
        if (cz) Qv = CT(-cz) * (m.Qxxz + m.Qyyz) * CT(0.5);
    } else if (nz0 == 2) {
        if (!cz) { D = CT(cx * cy) * m.Pxy * CT(0.25); Qv = (CT(cx) * m.Qxyy + CT(cy) * m.Qxxy) * CT(0.25); }
        if (!cy) { D = CT(cx * cz) * m.Pxz * CT(0.25); Qv = (CT(cx) * m.Qxzz + CT(cz) * m.Qxxz) * CT(0.25); }
        if (!cx) { D = CT(cy * cz) * m.Pyz * CT(0.25); Qv = (CT(cy) * m.Qyzz + CT(cz) * m.Qyyz) * CT(0.25); }
    } else if (nz0 == 3) {
        Qv = CT(cx * cy * cz) * m.Qxyz * CT(0.125);
    } else {
        T = -m.T;
    }
    return D + (USE_T ? T : CT(0)) + (USE_Q ? Qv : CT(0));
}

template <class CT, bool CENTRAL, bool USE_T, bool USE_Q>
__device__ __forceinline__ void collide_kbc(CT* f, CT rho, CT ux, CT uy, CT uz, CT fx, CT fy, CT fz, CT nu)
{
    CT M200 = CT(0), M020 = CT(0), M002 = CT(0), M110 = CT(0), M101 = CT(0), M011 = CT(0), M111 = CT(0);
    CT M201 = CT(0), M102 = CT(0), M210 = CT(0), M120 = CT(0), M021 = CT(0), M012 = CT(0);
#pragma unroll
    for (int q = 0; q < 27; ++q) {
        const int cx = cxq(q), cy = cyq(q), cz = czq(q);
        const CT v = f[q];
        if (cx) { M200 += v; if (cz) M201 += CT(cz) * v; if (cy) M210 += CT(cy) * v; }
        if (cy) { M020 += v; if (cz) M021 += CT(cz) * v; if (cx) M120 += CT(cx) * v; }
        if (cz) { M002 += v; if (cx) M102 += CT(cx) * v; if (cy) M012 += CT(cy) * v; }
        if (cx && cy) M110 += CT(cx * cy) * v;
        if (cx && cz) M101 += CT(cx * cz) * v;
        if (cy && cz) M011 += CT(cy * cz) * v;
        if (cx && cy && cz) M111 += CT(cx * cy * cz) * v;
    }
    const CT cs2 = CT(1.0 / 3.0);
    KbcMom<CT> m, e;
    const CT rT = M200 + M020 + M002, rNxz = M200 - M002, rNyz = M020 - M002;
    if (!CENTRAL) {
        m = {rT, rNxz, rNyz, M110, M101, M011, M210, M201, M120, M021, M102, M012, M111};
        e.T = rho * (CT(3) * cs2 + ux * ux + uy * uy + uz * uz);
        e.Nxz = rho * (ux * ux - uz * uz); e.Nyz = rho * (uy * uy - uz * uz);
        e.Pxy = rho * ux * uy; e.Pxz = rho * ux * uz; e.Pyz = rho * uy * uz;
        e.Qxxy = rho * uy * (cs2 + ux * ux); e.Qxxz = rho * uz * (cs2 + ux * ux);
        e.Qxyy = rho * ux * (cs2 + uy * uy); e.Qyyz = rho * uz * (cs2 + uy * uy);
        e.Qxzz = rho * ux * (cs2 + uz * uz); e.Qyzz = rho * uy * (cs2 + uz * uz);
        e.Qxyz = rho * ux * uy * uz;
    } else {
        const CT cT = rT - rho * (ux * ux + uy * uy + uz * uz);
        const CT cNxz = rNxz + rho * (uz * uz - ux * ux), cNyz = rNyz + rho * (uz * uz - uy * uy);
        const CT cPxy = M110 - rho * ux * uy, cPxz = M101 - rho * ux * uz, cPyz = M011 - rho * uy * uz;
        m.T = cT; m.Nxz = cNxz; m.Nyz = cNyz; m.Pxy = cPxy; m.Pxz = cPxz; m.Pyz = cPyz;
        m.Qxxy = M210 - CT(1.0 / 3.0) * (CT(6) * ux * cPxy + uy * (CT(3) * ux * ux + CT(2) * cNxz - cNyz + cT));
        m.Qxxz = M201 - CT(1.0 / 3.0) * (CT(6) * ux * cPxz + uz * (CT(3) * ux * ux + CT(2) * cNxz - cNyz + cT));
        m.Qxyy = M120 - CT(1.0 / 3.0) * (CT(6) * uy * cPxy + ux * (CT(3) * uy * uy + CT(2) * cNyz - cNxz + cT));
        m.Qyyz = M021 - CT(1.0 / 3.0) * (CT(6) * uy * cPyz + uz * (CT(3) * uy * uy + CT(2) * cNyz - cNxz + cT));
        m.Qxzz = M102 - CT(1.0 / 3.0) * (CT(6) * uz * cPxz + ux * (CT(3) * uz * uz - cNyz - cNxz + cT));
        m.Qyzz = M012 - CT(1.0 / 3.0) * (CT(6) * uz * cPyz + uy * (CT(3) * uz * uz - cNyz - cNxz + cT));
        m.Qxyz = M111 - ux * cPyz - uy * cPxz - uz * cPxy - ux * uy * uz;
        const CT z = CT(0);
        e = {rho * CT(3) * cs2, z, z, z, z, z, z, z, z, z, z, z, z};
    }
    const FactEq<CT> E(ux, uy, uz);
    const CT beta = CT(1) / (CT(2) * nu / cs2 + CT(1));
    // the shear part is linear in the moments: Delta s_q = s_q(m) - s_q(m_eq) = s_q(m - m_eq)
    const KbcMom<CT> dm = {m.T - e.T, m.Nxz - e.Nxz, m.Nyz - e.Nyz, m.Pxy - e.Pxy, m.Pxz - e.Pxz, m.Pyz - e.Pyz,
                           m.Qxxy - e.Qxxy, m.Qxxz - e.Qxxz, m.Qxyy - e.Qxyy, m.Qyyz - e.Qyyz, m.Qxzz - e.Qxzz,
                           m.Qyzz - e.Qyzz, m.Qxyz - e.Qxyz};
    CT num = CT(0), den = CT(0);
#pragma unroll
    for (int q = 0; q < 27; ++q) {
        const CT feq = E(q, rho);
        const CT ds = kbc_shear<CT, USE_T, USE_Q>(q, dm);
        const CT dh = f[q] - feq - ds;
        const CT ifeq = CT(1) / feq;
        num += ds * dh * ifeq;
        den += dh * dh * ifeq;
    }
    const CT gamma = kbc_gamma(num, den, beta);
    const CT ir = CT(1) / rho;
#pragma unroll
    for (int q = 0; q < 27; ++q) {
        const CT feq = E(q, rho);
        const CT ds = kbc_shear<CT, USE_T, USE_Q>(q, dm);
        const CT dh = f[q] - feq - ds;
        f[q] -= beta * (CT(2) * ds + gamma * dh) - (CT(1) - beta) * force_src<CT>(q, ir, ux, uy, uz, fx, fy, fz) * feq;
    }
}

// the same from the populations: raw second moments by additions only (c in {-1,0,1}),
// shifted to central ones with the raw momentum j: C_ab = M_ab - u_a j_b - u_b j_a + rho u_a u_b
template <class CT, class PT>
__device__ __forceinline__ CT local_nu(const CT* f, CT rho, CT ux, CT uy, CT uz, const CYParams<PT>& p, CT* S)
{
    CT Mxx = CT(0), Myy = CT(0), Mzz = CT(0), Mxy = CT(0), Mxz = CT(0), Myz = CT(0), jx = CT(0), jy = CT(0), jz = CT(0);
#pragma unroll
    for (int q = 0; q < 27; ++q) {
        const int cx = cxq(q), cy = cyq(q), cz = czq(q);
        const CT v = f[q];
        if (cx) { Mxx += v; if (cx > 0) jx += v; else jx -= v; }
        if (cy) { Myy += v; if (cy > 0) jy += v; else jy -= v; }
        if (cz) { Mzz += v; if (cz > 0) jz += v; else jz -= v; }
        if (cx * cy > 0) Mxy += v; else if (cx * cy < 0) Mxy -= v;
        if (cx * cz > 0) Mxz += v; else if (cx * cz < 0) Mxz -= v;
        if (cy * cz > 0) Myz += v; else if (cy * cz < 0) Myz -= v;
    }
    const CT Cxx = Mxx - CT(2) * ux * jx + rho * ux * ux;
    const CT Cyy = Myy - CT(2) * uy * jy + rho * uy * uy;
    const CT Czz = Mzz - CT(2) * uz * jz + rho * uz * uz;
    const CT Cxy = Mxy - ux * jy - uy * jx + rho * ux * uy;
    const CT Cxz = Mxz - ux * jz - uz * jx + rho * ux * uz;
    const CT Cyz = Myz - uy * jz - uz * jy + rho * uy * uz;
    return cy_nu<CT>(Cxx, Cyy, Czz, Cxy, Cxz, Cyz, rho, p, S);
}

} // namespace pops

// step_cell_stored (nnlbm_physics.cuh) for 16-bit storage: g holds the stored values as float (or those of
// two cells, CT = f2), before and after; sc, isc: the storage scale and its inverse
template <class CT, int COL, class FUSE, class PT, class Out>
__device__ __forceinline__ void step_cell_16(CT* g, CT fx, CT fy, CT fz, CT nu, const CYParams<PT>* cy, CT sc, CT isc, Out&& out)
{
    // one cell with BGK or MRT_LES: the planes x = -1 and x = 0 scale and shift as packed pairs on
    // the way in and out (measured +2 % each; the cumulant measured 3 % slower)
    constexpr bool ONE = std::is_same<CT, float>::value;
    constexpr bool PAIR_IO = ONE && (COL == COL_BGK || COL == COL_MRT);
    CT f[27];
    if constexpr (PAIR_IO) {
#pragma unroll
        for (int j = 0; j < 9; ++j) {
            const f2 v = mad(f2(g[j], g[9 + j]), f2(isc, isc), f2(weight<float>(j), weight<float>(9 + j)));
            f[j] = v.v.x;
            f[9 + j] = v.v.y;
        }
    }
#pragma unroll
    for (int q = PAIR_IO ? 18 : 0; q < 27; ++q) f[q] = mad(g[q], isc, CT(weight<float>(q)));
    CT rho, ux, uy, uz, S[6];
    if constexpr (COL == COL_CUM) {
        if constexpr (ONE) {
            pops::step_cell_cum_packed<FUSE>(f, fx, fy, fz, nu, cy, S, rho, ux, uy, uz);
        } else {
            pops::cum_columns<CT>(f);
            pops::cum_density_velocity<CT>(f, fx, fy, fz, rho, ux, uy, uz);
            pops::collide_cum_columns<CT, PT>(f, rho, ux, uy, uz, nu, cy, S);
        }
    } else {
        if constexpr (PAIR_IO) pops::packed_density_velocity(f, fx, fy, fz, rho, ux, uy, uz);
        else density_velocity<CT>(f, fx, fy, fz, rho, ux, uy, uz);
        if (cy) nu = pops::local_nu<CT, PT>(f, rho, ux, uy, uz, *cy, S);
        if constexpr (COL == COL_MRT && ONE) pops::collide_mrt_packed(f, rho, ux, uy, uz, nu);
        else if constexpr (COL == COL_MRT) pops::collide_mrt<CT>(f, rho, ux, uy, uz, nu);
        else if constexpr (COL == COL_BGK && ONE) pops::collide_bgk_packed(f, rho, ux, uy, uz, fx, fy, fz, nu);
        else if constexpr (COL == COL_BGK) pops::collide_bgk<CT>(f, rho, ux, uy, uz, fx, fy, fz, nu);
        else {
            constexpr bool central = COL >= COL_KBC_C1;
            constexpr int v = central ? COL - COL_KBC_C1 + 1 : COL - COL_KBC_N1 + 1;
            pops::collide_kbc<CT, central, (v == 2 || v == 4), (v == 3 || v == 4)>(f, rho, ux, uy, uz, fx, fy, fz, nu);
        }
    }
    // (v - w) sc as one fused v sc - w sc
    if constexpr (PAIR_IO) {
#pragma unroll
        for (int j = 0; j < 9; ++j) {
            const f2 v = mad(f2(f[j], f[9 + j]), f2(sc, sc), f2(-(weight<float>(j) * sc), -(weight<float>(9 + j) * sc)));
            g[j] = v.v.x;
            g[9 + j] = v.v.y;
        }
    }
#pragma unroll
    for (int q = PAIR_IO ? 18 : 0; q < 27; ++q) g[q] = mad(f[q], sc, -(CT(weight<float>(q)) * sc));
    out(rho, ux, uy, uz, cy ? (const CT*)S : (const CT*)nullptr);
}

// density, velocity (u = (j + F/2) / rho) and the collision of one cell's stored values g (or of
// two cells', CT = f2).  With `cy` the shear viscosity is the local Carreau-Yasuda one.  PT: the
// type of the viscosity-law parameters.  out(rho, ux, uy, uz, S) is called once they are known
// (S: the strain rate with `cy`, else null): with FP32 and FP64 storage before the populations are
// rebuilt, so that nothing of it is held in registers meanwhile
template <class CT, int COL, int DT, bool PLANES, bool ODD, bool IN_PAIR, class PT, class Out>
__device__ __forceinline__ void step_cell(CT* g, CT fx, CT fy, CT fz, CT nu, const CYParams<PT>* cy, CT sc, CT isc, Out&& out)
{
    if constexpr (DT >= 2) step_cell_16<CT, COL, pops::Fuse<ODD, IN_PAIR>, PT>(g, fx, fy, fz, nu, cy, sc, isc, out);
    else step_cell_stored<CT, COL, DT, PLANES, PT>(g, fx, fy, fz, nu, cy, out);
}

} // namespace nnlbm
