// sfwi_cell.cuh — the per-cell arithmetic of a time step, on single cells
// (T = float) or on two lanes as FP32x2 (T = float2).  Every kernel that
// advances a field calls these functions, so a cell takes the same operations
// in the same order whichever kernel, tile or strip holds it.  Every
// multiply-add is written out as one operation: the compiler fuses a packed
// product into a following packed add where the product has no other use, also with
// -fmad=false, so a product that is only added must not be left to it.
#pragma once
#include "sfwi_common.cuh"

namespace sfwi {

// 8th-order staggered first-derivative weights, sfwi-stage1/FD2DGPU.cuh:16
constexpr float K1 = (float)(1225.0 / 1024.0);
constexpr float K2 = (float)(-245.0 / 3072.0);
constexpr float K3 = (float)(49.0 / 5120.0);
constexpr float K4 = (float)(-5.0 / 7168.0);

__device__ __forceinline__ float2 B2(float x) { return make_float2(x, x); }
template <class T>
__device__ __forceinline__ T all(float x) {
    if constexpr (sizeof(T) == 8)
        return make_float2(x, x);
    else
        return x;
}
__device__ __forceinline__ float add2(float a, float b) { return __fadd_rn(a, b); }
__device__ __forceinline__ float mul2(float a, float b) { return __fmul_rn(a, b); }
__device__ __forceinline__ float fma2(float a, float b, float c) { return __fmaf_rn(a, b, c); }
__device__ __forceinline__ float2 add2(float2 a, float2 b) { return __fadd2_rn(a, b); }
__device__ __forceinline__ float2 mul2(float2 a, float2 b) { return __fmul2_rn(a, b); }
__device__ __forceinline__ float2 fma2(float2 a, float2 b, float2 c) { return __ffma2_rn(a, b, c); }
// k*(p - q) + a; p - q is formed as fma(q, -1, p), which rounds exactly like
// a subtraction
__device__ __forceinline__ float2 kdiff2(float k, float2 p, float2 q, float2 a) {
    const float2 d = __ffma2_rn(q, make_float2(-1.f, -1.f), p);
    return __ffma2_rn(make_float2(k, k), d, a);
}
__device__ __forceinline__ float kdiff2(float k, float p, float q, float a) {
    return __fmaf_rn(k, __fsub_rn(p, q), a);
}

// PML factors of a damped cell: the split update (d1*m + c*D)/d2 is evaluated
// as (d1*m + c*D) * (1/d2) with a correctly rounded reciprocal, one rounding
// more than a division
template <class T>
struct DampT {
    T d1, r2, d3, r4;
};
using Damp2 = DampT<float2>;
// 1 -+ (dt d)/2: halving is exact, so one fused step rounds once
__device__ __forceinline__ float damp_minus(float dt, float d) { return fmaf(dt * d, -0.5f, 1.f); }
__device__ __forceinline__ float damp_plus_rcp(float dt, float d) { return __frcp_rn(fmaf(dt * d, 0.5f, 1.f)); }
__device__ __forceinline__ Damp2 make_damp2(float dt, float2 x, float2 z) {
    Damp2 d;
    d.d1 = make_float2(damp_minus(dt, x.x), damp_minus(dt, x.y));
    d.r2 = make_float2(damp_plus_rcp(dt, x.x), damp_plus_rcp(dt, x.y));
    d.d3 = make_float2(damp_minus(dt, z.x), damp_minus(dt, z.y));
    d.r4 = make_float2(damp_plus_rcp(dt, z.x), damp_plus_rcp(dt, z.y));
    return d;
}

// Velocity update, one component: v += dir*ib*(dtdx*Dx + dtdz*Dz) with cx =
// ib*dir*dtdx, cz = ib*dir*dtdz (vx: Dx = D+x txx, Dz = D-z txz; vz: Dx = D-x
// txz, Dz = D+z tzz).
template <class T>
__device__ __forceinline__ T v_plain1(T v, T cx, T cz, T dx, T dz) {
    return add2(v, fma2(cx, dx, mul2(cz, dz)));
}
// the split update of the reference in damped cells,
//   v_x = (d1 v_x + c_x D_x) r2,  v_z = (d3 v_z + c_z D_z) r4,  v = v_x + v_z,
// with the x-part kept in m and the z-part = v - m; returns the new total and
// sets m to the new x-part
template <class T>
__device__ __forceinline__ T v_split1(T v, T &m, const DampT<T> &d, T cx, T cz, T dx, T dz) {
    const T x = mul2(fma2(d.d1, m, mul2(cx, dx)), d.r2);
    const T z = fma2(d.d3, fma2(m, all<T>(-1.f), v), mul2(cz, dz));
    m = x;
    return fma2(z, d.r4, x);
}
template <class T>
struct VT {
    T x, z;
};
using V2 = VT<float2>;
template <class T>
__device__ __forceinline__ VT<T> v_plain2(VT<T> v, T cx, T cz, T ax, T bz, T dx, T dz) {
    return VT<T>{v_plain1(v.x, cx, cz, ax, bz), v_plain1(v.z, cx, cz, dx, dz)};
}
template <class T>
__device__ __forceinline__ VT<T> v_split2(VT<T> v, VT<T> &m, const DampT<T> &d, T cx, T cz, T ax, T bz, T dx, T dz) {
    return VT<T>{v_split1(v.x, m.x, d, cx, cz, ax, bz), v_split1(v.z, m.z, d, cx, cz, dx, dz)};
}

// Stress update from a = D-x vx, b = D-z vz (the normal stresses), c = D+z vx,
// d = D+x vz (the shear stress).
template <class T>
struct ST {
    T xx, zz, xz;
};
using S2 = ST<float2>;
// Born increments of txx, tzz, txz: t times xx_x, zz_x, xz_x those of the
// x-parts (formed where they are added), xx_z, zz_z, xz_z those of the z-parts
// and xx, zz, xz the sums of both
template <class T>
struct BornT {
    T t, xx_x, xx_z, zz_x, zz_z, xz_x, xz_z, xx, zz, xz;
};
using Born2 = BornT<float2>;
// Born virtual source from the background strains (add_born_source_components,
// sfwi-stage2/born.cu:788-798); bp/bs are zero outside the Born region
template <class T>
__device__ __forceinline__ void born_norm2(BornT<T> &q, T bp, T bs, float idx, float idz, float dt, T a, T b) {
    const T mix = fma2(bs, all<T>(-2.f), bp);
    const T ax = mul2(a, all<T>(idx)), bz = mul2(b, all<T>(idz));
    q.t = all<T>(dt);
    q.xx_x = mul2(bp, ax), q.xx_z = mul2(q.t, mul2(mix, bz));
    q.zz_x = mul2(mix, ax), q.zz_z = mul2(q.t, mul2(bp, bz));
    q.xx = fma2(q.t, q.xx_x, q.xx_z);
    q.zz = fma2(q.t, q.zz_x, q.zz_z);
}
template <class T>
__device__ __forceinline__ void born_shear2(BornT<T> &q, T bs, float idx, float idz, float dt, T c, T d) {
    const T dx = mul2(d, all<T>(idx)), cz = mul2(c, all<T>(idz));
    q.t = all<T>(dt);
    q.xz_x = mul2(bs, dx), q.xz_z = mul2(q.t, mul2(bs, cz));
    q.xz = fma2(q.t, q.xz_x, q.xz_z);
}
template <class T>
__device__ __forceinline__ BornT<T> born2(T bp, T bs, float idx, float idz, float dt, T a, T b, T c, T d) {
    BornT<T> q;
    born_norm2(q, bp, bs, idx, idz, dt, a, b);
    born_shear2(q, bs, idx, idz, dt, c, d);
    return q;
}
template <class T>
__device__ __forceinline__ void s_norm_plain(T &xx, T &zz, T tx, T tz, T l, T u, T a, T b) {
    const T l2m = fma2(u, all<T>(2.f), l);
    const T ax = mul2(tx, a), bz = mul2(tz, b);
    xx = add2(xx, fma2(l2m, ax, mul2(l, bz)));
    zz = add2(zz, fma2(l, ax, mul2(l2m, bz)));
}
template <class T>
__device__ __forceinline__ T s_shear_plain(T xz, T tx, T tz, T u, T c, T d) {
    return fma2(u, fma2(tz, c, mul2(tx, d)), xz);
}
// the split updates in damped cells, from the x-parts m and the z-parts z
// (total - x-part), both with their Born increments; return the new totals and
// set m to the new x-parts
template <class T>
__device__ __forceinline__ void s_norm_split(T &mxx, T &mzz, T &zxx, T &zzz, const DampT<T> &k, T tx, T tz, T l, T u,
                                             T a, T b) {
    const T l2m = fma2(u, all<T>(2.f), l);
    const T ax = mul2(tx, a), bz = mul2(tz, b);
    const T xx_z = fma2(k.d3, zxx, mul2(l, bz)), zz_z = fma2(k.d3, zzz, mul2(l2m, bz));
    mxx = mul2(fma2(k.d1, mxx, mul2(l2m, ax)), k.r2);
    mzz = mul2(fma2(k.d1, mzz, mul2(l, ax)), k.r2);
    zxx = fma2(xx_z, k.r4, mxx);
    zzz = fma2(zz_z, k.r4, mzz);
}
template <class T>
__device__ __forceinline__ T s_shear_split(T &mxz, T zxz, const DampT<T> &k, T tx, T tz, T u, T c, T d) {
    const T xz_z = fma2(k.d3, zxz, mul2(u, mul2(tz, c)));
    mxz = mul2(fma2(k.d1, mxz, mul2(u, mul2(tx, d))), k.r2);
    return fma2(xz_z, k.r4, mxz);
}
template <class T>
__device__ __forceinline__ T zpart(T total, T m) {
    return fma2(m, all<T>(-1.f), total);
}
template <bool BORN, class T>
__device__ __forceinline__ ST<T> s_plain2(ST<T> s, T tx, T tz, T l, T u, T a, T b, T c, T d, const BornT<T> &q) {
    if (BORN) {
        s.xx = add2(s.xx, q.xx);
        s.zz = add2(s.zz, q.zz);
        s.xz = add2(s.xz, q.xz);
    }
    s_norm_plain(s.xx, s.zz, tx, tz, l, u, a, b);
    s.xz = s_shear_plain(s.xz, tx, tz, u, c, d);
    return s;
}
template <bool BORN, class T>
__device__ __forceinline__ ST<T> s_split2(ST<T> s, ST<T> &m, const DampT<T> &k, T tx, T tz, T l, T u, T a, T b, T c,
                                          T d, const BornT<T> &q) {
    ST<T> z{zpart(s.xx, m.xx), zpart(s.zz, m.zz), zpart(s.xz, m.xz)};
    if (BORN) {
        m.xx = fma2(q.t, q.xx_x, m.xx), z.xx = add2(z.xx, q.xx_z);
        m.zz = fma2(q.t, q.zz_x, m.zz), z.zz = add2(z.zz, q.zz_z);
        m.xz = fma2(q.t, q.xz_x, m.xz), z.xz = add2(z.xz, q.xz_z);
    }
    s_norm_split(m.xx, m.zz, z.xx, z.zz, k, tx, tz, l, u, a, b);
    z.xz = s_shear_split(m.xz, z.xz, k, tx, tz, u, c, d);
    return z;
}

// Adjoint stresses: txx' keeps only an x-part and tzz' only a z-part; txz' is
// split, its x-part in m.
template <class T>
__device__ __forceinline__ ST<T> as_plain2(ST<T> s, T tx, T tz, T a, T b, T c, T d) {
    return ST<T>{fma2(tx, a, s.xx), fma2(tz, b, s.zz), add2(s.xz, fma2(tx, d, mul2(tz, c)))};
}
template <class T>
__device__ __forceinline__ ST<T> as_split2(ST<T> s, T &m, const DampT<T> &k, T tx, T tz, T a, T b, T c, T d) {
    const T neg = all<T>(-1.f);
    const T nxx = mul2(fma2(k.d1, s.xx, mul2(tx, a)), k.r2);
    const T nzz = mul2(fma2(k.d3, s.zz, mul2(tz, b)), k.r4);
    const T nx = mul2(fma2(k.d1, m, mul2(tx, d)), k.r2);
    const T nz = fma2(k.d3, fma2(m, neg, s.xz), mul2(tz, c));
    m = nx;
    return ST<T>{nxx, nzz, fma2(nz, k.r4, nx)};
}
// Lame-weighted adjoint stresses: P = (l+2m) txx + l tzz, Q = l txx + (l+2m) tzz, R = m txz
template <class T>
__device__ __forceinline__ ST<T> lame2(ST<T> s, T l, T u) {
    const T l2m = fma2(all<T>(2.f), u, l);
    return ST<T>{fma2(l2m, s.xx, mul2(l, s.zz)), fma2(l, s.xx, mul2(l2m, s.zz)), mul2(u, s.xz)};
}

// Zero-lag imaging terms of the lambda and mu kernels (doimage_gradient,
// sfwi-stage1/FD2DGPU.cu:3350-3382), from the forward strains and the adjoint
// stresses; the increments are -lg and -mg:
//   lg = (gxx + gzz)(txx' + tzz'),  mg = 2 (gxx txx' + gzz tzz') + (gxz + gzx) txz'
// with gxx = a/dx, gzz = b/dz, gxz = c/dz, gzx = d/dx
template <class T>
struct ImgT {
    T lg, mg;
};
using Img2 = ImgT<float2>;
template <class T>
__device__ __forceinline__ ImgT<T> image2(float idx, float idz, T a, T b, T c, T d, ST<T> s) {
    const T gxx = mul2(a, all<T>(idx)), gzz = mul2(b, all<T>(idz));
    const T gxz_gzx = fma2(c, all<T>(idz), mul2(d, all<T>(idx)));
    return ImgT<T>{mul2(add2(gxx, gzz), add2(s.xx, s.zz)),
                   fma2(all<T>(2.f), fma2(gxx, s.xx, mul2(gzz, s.zz)), mul2(gxz_gzx, s.xz))};
}

}  // namespace sfwi
