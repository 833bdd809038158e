// The link update with its products, quotients and square roots on the integer pipes.
//
// Bound: GB300's FP64 pipe.  A warp's FP64 addition occupies it for about 80 cycles of an SM
// quarter (see Add) whatever its active lanes, and a link took about 400 of them while the integer pipes
// issued in one cycle of ten.  Here the FP64 pipe keeps the additions (and the libm calls);
// multiplications, divisions, roots and conversions are the exact integer forms of
// fp64_int.cuh, so every stored value has the bits of the plain form (link_orient and
// link_finish in kernels.cuh).  Those forms hold for operands in their exponent band; a link
// with any other operand (zeros in a body's first steps, exact symmetries, overflow) is found
// by the `rare` word at the end and taken again by the plain form, on which it then stays (LF_PLAIN).  In-place state is therefore
// written only after that check; the direction slots, which are outputs alone, before it.
//
// k_links on 128 settled creatures (371 k links): 329 -> 218 us, 4.98 -> 2.35 M FP64 warp
// instructions beside 64 M integer ones (issue slots 11 -> 31 % used); with elements grouped by form, 337 -> 208
// us over another 128 (375 k links).  Leaving any group of the
// products (orientation, damping, a rotation) on the FP64 pipe measured 1.5-6 % slower passes.
//
// The terms that the two angle modes make exactly zero (see beam_forces) are left out: their
// partners are checked to be nonzero by the products they enter.
#pragma once
#include "physics.cuh"

namespace gvx {
namespace GVX_KNS {

// A double whose sums and differences, with F set, are formed as x * 1 + y by DFMA, with the 1 in a
// register that the compiler cannot see through.  Exactly x + y, and faster where the whole chip is
// busy: with all four quarters of an SM at it a DFMA of three registers takes 17.0 cycles of the SM, a
// DADD or DMUL (or a DFMA with a constant or uniform operand) 20.1, 80 of a quarter's.  A quarter alone takes 69 for either,
// and the register and the negations cost small batches 1-2 %, so those take F clear.
template <bool F>
struct Add {
    double v, one;
    __device__ __forceinline__ operator double() const { return v; }
    __device__ __forceinline__ Add plus(double y) const { return {F ? __fma_rn(v, one, y) : v + y, one}; }
};
template <bool F> __device__ __forceinline__ Add<F> operator+(const Add<F>& x, const Add<F>& y) { return x.plus(y.v); }
template <bool F> __device__ __forceinline__ Add<F> operator+(const Add<F>& x, double y) { return x.plus(y); }
template <bool F> __device__ __forceinline__ Add<F> operator+(double x, const Add<F>& y) { return y.plus(x); }
template <bool F> __device__ __forceinline__ Add<F> operator-(const Add<F>& x) { return {-x.v, x.one}; }
template <bool F> __device__ __forceinline__ Add<F> operator-(const Add<F>& x, const Add<F>& y) { return x.plus(-y.v); }
template <bool F> __device__ __forceinline__ Add<F> operator-(const Add<F>& x, double y) { return x.plus(-y); }
template <bool F> __device__ __forceinline__ Add<F> operator-(double x, const Add<F>& y) { return Add<F>{x, y.one}.plus(-y.v); }

template <bool F>
struct IntPipes {
    double one;               // 1.0 (see Add)
    uint32_t rare = 0;
    __device__ __forceinline__ explicit IntPipes(double one_ = 1.0) : one(one_) {}
    __device__ __forceinline__ Add<F> add(double x) const { return {x, one}; }   // x as a term of a sum
    __device__ __forceinline__ Add<F> mul(double x, double y) { return {fp64i::mul_band(x, y, rare), one}; }
    // a product that may have an exact zero for a factor
    __device__ __forceinline__ Add<F> mul0(double x, double y) {
        const bool z = fp64i::eq0(x) | fp64i::eq0(y);
        const double p = mul(z ? 1.0 : x, z ? 1.0 : y);
        return {z ? times_zero(x, y) : p, one};
    }
    __device__ __forceinline__ Add<F> div(double x, double y) { return {fp64i::div_band(x, y, rare), one}; }
    __device__ __forceinline__ Add<F> root(double x) { return {fp64i::sqrt_band(x, rare), one}; }
    __device__ __forceinline__ Add<F> wide(float x) { return {fp64i::f2d_band(x, rare), one}; }
    __device__ __forceinline__ float narrow(double x) { return fp64i::d2f_band(x, rare); }
    __device__ __forceinline__ float cut(double x) { return fp64i::cut_band(x, rare); }
    __device__ __forceinline__ void flag(bool b) { rare = b ? fp64i::kOutOfBand : rare; }
    __device__ __forceinline__ void check(const d3& v) { rare |= fp64i::band(fp64i::hi32(v.x)) | fp64i::band(fp64i::hi32(v.y)) | fp64i::band(fp64i::hi32(v.z)); }
    __device__ __forceinline__ bool ok() const { return (rare & fp64i::kOutOfBand) == 0; }
};
using fp64i::half_band;
using fp64i::mul2_band;

// Quat3D::RotateVec3D, operator* and RotateVec3DInv (qrot, qmul, qrotinv and their x = 0 forms in
// physics.cuh): the same terms in the same order.
template <class Pipes>
__device__ __forceinline__ d3 qrot_int(Pipes& a, const q4& q, const d3& f) {
    const double tw = a.mul(f.x, q.x) + a.mul(f.y, q.y) + a.mul(f.z, q.z);
    const double tx = a.mul(f.x, q.w) - a.mul(f.y, q.z) + a.mul(f.z, q.y);
    const double ty = a.mul(f.x, q.z) + a.mul(f.y, q.w) - a.mul(f.z, q.x);
    const double tz = a.mul(f.y, q.x) - a.mul(f.x, q.y) + a.mul(f.z, q.w);
    return D3(a.mul(q.w, tx) + a.mul(q.x, tw) + a.mul(q.y, tz) - a.mul(q.z, ty),
              a.mul(q.w, ty) - a.mul(q.x, tz) + a.mul(q.y, tw) + a.mul(q.z, tx),
              a.mul(q.w, tz) + a.mul(q.x, ty) - a.mul(q.y, tx) + a.mul(q.z, tw));
}
template <class Pipes>
__device__ __forceinline__ q4 qmul_int(Pipes& a, const q4& p, const q4& f) {
    return Q4(a.mul(p.w, f.w) - a.mul(p.x, f.x) - a.mul(p.y, f.y) - a.mul(p.z, f.z),
              a.mul(p.w, f.x) + a.mul(p.x, f.w) + a.mul(p.y, f.z) - a.mul(p.z, f.y),
              a.mul(p.w, f.y) - a.mul(p.x, f.z) + a.mul(p.y, f.w) + a.mul(p.z, f.x),
              a.mul(p.w, f.z) + a.mul(p.x, f.y) - a.mul(p.y, f.x) + a.mul(p.z, f.w));
}
template <class Pipes>
__device__ __forceinline__ d3 qrotinv_int(Pipes& a, const q4& q, const d3& f) {
    const double tw = a.mul(q.x, f.x) + a.mul(q.y, f.y) + a.mul(q.z, f.z);
    const double tx = a.mul(q.w, f.x) - a.mul(q.y, f.z) + a.mul(q.z, f.y);
    const double ty = a.mul(q.w, f.y) + a.mul(q.x, f.z) - a.mul(q.z, f.x);
    const double tz = a.mul(q.w, f.z) - a.mul(q.x, f.y) + a.mul(q.y, f.x);
    return D3(a.mul(tw, q.x) + a.mul(tx, q.w) + a.mul(ty, q.z) - a.mul(tz, q.y),
              a.mul(tw, q.y) - a.mul(tx, q.z) + a.mul(ty, q.w) + a.mul(tz, q.x),
              a.mul(tw, q.z) + a.mul(tx, q.y) - a.mul(ty, q.x) + a.mul(tz, q.w));
}
template <class Pipes>
__device__ __forceinline__ q4 qmul_x0_int(Pipes& a, const q4& p, const q4& f) {
    return Q4(a.mul(p.w, f.w) - a.mul(p.y, f.y) - a.mul(p.z, f.z), a.mul(p.w, f.x) + a.mul(p.y, f.z) - a.mul(p.z, f.y),
              a.mul(p.w, f.y) + a.mul(p.y, f.w) + a.mul(p.z, f.x), a.mul(p.w, f.z) - a.mul(p.y, f.x) + a.mul(p.z, f.w));
}
template <class Pipes>
__device__ __forceinline__ d3 qrotinv_x0_int(Pipes& a, const q4& q, const d3& f) {
    const double tw = a.mul(q.y, f.y) + a.mul(q.z, f.z);
    const double tx = a.mul(q.w, f.x) - a.mul(q.y, f.z) + a.mul(q.z, f.y);
    const double ty = a.mul(q.w, f.y) - a.mul(q.z, f.x);
    const double tz = a.mul(q.w, f.z) + a.mul(q.y, f.x);
    return D3(a.mul(tx, q.w) + a.mul(ty, q.z) - a.mul(tz, q.y), a.mul(tw, q.y) - a.mul(tx, q.z) + a.mul(ty, q.w),
              a.mul(tw, q.z) + a.mul(tx, q.y) + a.mul(tz, q.w));
}

// Quat3D::ToRotationVector (q_to_rotvec); kX0: q.x is exactly zero and so is the result's x.
template <bool kX0, class Pipes>
__device__ __forceinline__ d3 q_to_rotvec_int(Pipes& a, const q4& q, bool* wide) {
    a.flag((fp64i::hi32(q.w) & 0x7FFFFFFFu) >= 0x3FF00000u);   // |w| >= 1
    const double sl = a.one - a.mul(q.w, q.w);
    d3 v;
    if (fp64i::lt_pos(sl, 2.4e-3)) {
        const double s = a.root(a.div(mul2_band(a.one - a.add(q.w)), sl))   /* 2 - 2w */;
        v = D3(kX0 ? 0.0 : a.mul(mul2_band(q.x), s), a.mul(mul2_band(q.y), s), a.mul(mul2_band(q.z), s));
    } else {
        *wide = true;
        const double t = acos(q.w);
        const double inv = a.div(1.0, a.root(sl));
        v = D3(kX0 ? 0.0 : a.mul(a.mul(mul2_band(q.x), t), inv), a.mul(a.mul(mul2_band(q.y), t), inv), a.mul(a.mul(mul2_band(q.z), t), inv));
    }
    return v;
}

// Quat3D::FromAngleToPosX (q_from_angle_to_posx) for a vector whose y and z are not zero; the x
// component of the result is zero.  The small-angle test compares cut floats with a margin of
// 2^-16; a quotient that close to the threshold is left to the plain form.
template <class Pipes>
__device__ __forceinline__ q4 q_from_angle_to_posx_int(Pipes& a, const d3& r, double len, bool* wide) {
    const float x = 1.732e-2f * fabsf(a.cut(r.x)), y = fabsf(a.cut(r.y)), z = fabsf(a.cut(r.z));
    const float lo = x * (1.0f - 0x1p-16f), hi = x * (1.0f + 0x1p-16f);
    const bool small_turn = y < lo && z < lo;
    a.flag(!small_turn && !(y > hi || z > hi));
    if (small_turn) {
        const double qy = half_band(a.div(r.z, r.x)), qz = -half_band(a.div(r.y, r.x));
        return Q4(a.one - a.add(half_band(a.mul(qy, qy) + a.mul(qz, qz))), 0, qy, qz);
    }
    *wide = true;
    const double li = a.div(1.0, len);
    const double nx = a.mul(r.x, li), ny = a.mul(r.y, li), nz = a.mul(r.z, li);
    const double theta = acos(nx);
    a.flag(!fp64i::lt_pos(theta, 3.14159265358979 - 1e-7));
    const double ami = a.div(1.0, a.root(a.mul(nz, nz) + a.mul(ny, ny)));
    double sn, cs;
    sincos(half_band(theta), &sn, &cs);
    return Q4(cs, 0, a.mul(a.mul(nz, ami), sn), -a.mul(a.mul(ny, ami), sn));
}

// CVX_Voxel::transverseArea (voxel_tarea)
template <class Pipes>
__device__ __forceinline__ float voxel_tarea_int(Pipes& a, const VMat& m, float psa, float psb) {
    const float size = m.sizef;
    if (m.nu == 0) return size * size;
    return a.narrow(a.mul(a.mul(a.wide(size * size), a.wide(psa) + a.one), a.wide(psb) + a.one));
}

// link_orient of kernels.cuh.  SmallTurn and ExtendPerc are compared on cut floats with a margin
// of 2^-16 (their relative error is below 2^-21); closer ones are left to the plain form.
template <class Pipes>
__device__ __forceinline__ void link_orient_int(Pipes& a, const Sim& S, int l, uint8_t fl, LinkOrient* out) {
    const int ng = __ldg(S.lneg + l), pv = __ldg(S.lpos + l);
    const int axis = __ldg(S.lax + l);
    const VMat& vN = S.vm[__ldg(S.vmat + ng)];
    const VMat& vP = S.vm[__ldg(S.vmat + pv)];
    const float tN = S.temp[ng], tP = S.temp[pv];
    const double restLen = half_band(a.mul(vN.nom, a.wide(1 + tN * vN.cte)) + a.mul(vP.nom, a.wide(1 + tP * vP.cte)));
    const bool was = fl & LF_SMALL;
    const d3 d = to_axis_x(axis, D3(a.add(S.px[pv]) - S.px[ng], a.add(S.py[pv]) - S.py[ng], a.add(S.pz[pv]) - S.pz[ng]));
    const q4 q1 = q_to_axis_x(axis, Q4(S.qw[ng], S.qx[ng], S.qy[ng], S.qz[ng]));
    const q4 q2 = q_to_axis_x(axis, Q4(S.qw[pv], S.qx[pv], S.qy[pv], S.qz[pv]));
    const q4 tr = Q4(q1.w, -q1.x, -q1.y, -q1.z);
    const d3 pos2 = qrot_int(a, tr, d);
    out->angle2 = qmul_int(a, tr, q2);
    const float n = a.cut(a.add(fabs(pos2.z)) + fabs(pos2.y)), x = a.cut(pos2.x), r = a.cut(restLen);
    const float T = (was ? HB_TURN : 0.05f) * x, X = was ? HB_EXT : 0.50f;
    const float in = (1.0f - X) * r, ex = (1.0f + X) * r;
    constexpr float kUp = 1.0f + 0x1p-16f, kDown = 1.0f - 0x1p-16f;
    const bool yes = n < T * kDown && x > in * kUp && x < ex * kDown;
    const bool no = n > T * kUp || x < in * kDown || x > ex * kUp;
    a.flag(!(x > 0) || yes == no);
    out->pos2 = pos2; out->restLen = restLen; out->small = yes;
    out->switched = yes != was;
    out->lvv = (fl & LF_LVV) && yes == was;
}

// What the second half of a link's update takes from the first.
struct LinkPose {
    d3 pos2, a2v;
    double a1y, a1z;          // large-angle mode: angle1's rotation vector (its x is zero)
    double a1w, q1y, q1z;     // and angle1 (its x is zero)
    q4 angle2;
    float strain, maxStrain, strainOffset, fx;
    uint8_t fl;               // the new link flags
    bool small, lvv;
};

// link_finish of kernels.cuh for a link oriented by link_orient_int, first half: the end angles and
// the axial stress.  False: the link is left to the plain form.
template <class Pipes>
__device__ __forceinline__ bool link_pose_int(Pipes& a, const Sim& S, int l, const LinkOrient& lo, LinkPose* out) {
    const int ng = __ldg(S.lneg + l), pv = __ldg(S.lpos + l);
    const int axis = __ldg(S.lax + l);
    const LMat& m = S.lm[__ldg(S.lmt + l)];
    const VMat& vN = S.vm[__ldg(S.vmat + ng)];
    const VMat& vP = S.vm[__ldg(S.vmat + pv)];
    const double restLen = lo.restLen;
    const int nl = S.nl, nv = S.nv;
    const bool small = lo.small;
    d3 pos2 = lo.pos2;
    q4 angle2 = lo.angle2, angle1 = Q4(1, 0, 0, 0);
    double a1y = 0, a1z = 0;
    bool wide1 = false, acos1 = false, wide2 = false;
    if (small) {
        pos2.x = a.add(pos2.x) - restLen;
    } else {
        const double len = a.root(a.mul(pos2.x, pos2.x) + a.mul(pos2.y, pos2.y) + a.mul(pos2.z, pos2.z));
        angle1 = q_from_angle_to_posx_int(a, pos2, len, &wide1);
        angle2 = qmul_x0_int(a, angle1, angle2);
        pos2 = D3(a.add(len) - restLen, 0, 0);
        const d3 v = q_to_rotvec_int<true>(a, angle1, &acos1);
        a1y = v.y; a1z = v.z;
    }
    const d3 a2v = q_to_rotvec_int<false>(a, angle2, &wide2);

    // updateTransverseInfo
    float A, tss;
    if (m.nu != 0.0f) {
        const int ta = axis == 0 ? nv : 0, tb = axis == 2 ? nv : 2 * nv;
        const float na = S.ps[ta + ng], nb = S.ps[tb + ng], pa = S.ps[ta + pv], pb = S.ps[tb + pv];
        A = 0.5f * (voxel_tarea_int(a, vN, na, nb) + voxel_tarea_int(a, vP, pa, pb));
        tss = 0.5f * (voxel_tss(vN, na, nb) + voxel_tss(vP, pa, pb));
    } else {
        A = 0.5f * (vN.sizef * vN.sizef + vP.sizef * vP.sizef);
        tss = 0.0f;
    }
    // updateStrain
    float maxStrain = S.lsf[nl + l], strainOffset = S.lsf[2 * nl + l];
    const float strain = a.narrow(a.div(pos2.x, restLen));
    float stress;
    if (m.linear) {
        if (strain > maxStrain) maxStrain = strain;
        stress = mat_stress(m, strain, tss, false);
    } else if (strain > maxStrain) {
        maxStrain = strain;
        stress = mat_stress(m, strain, tss, false);
        if (m.nu != 0.0f) strainOffset = maxStrain - mat_stress(m, strain, 0.0f, false) / (m.eHat * (1 - m.nu));
        else strainOffset = maxStrain - stress / m.E;
    } else {
        const float rel = strain - strainOffset;
        stress = (m.nu != 0.0f) ? mat_stress(m, rel, tss, true) : m.E * rel;
    }
    a.flag(m.epsFail != -1.0f && maxStrain > m.epsFail);
    if (S.lnew) a.flag(S.lnew[l] > 0);
    out->pos2 = pos2; out->a2v = a2v; out->a1y = a1y; out->a1z = a1z;
    out->a1w = angle1.w; out->q1y = angle1.y; out->q1z = angle1.z; out->angle2 = angle2;
    out->strain = strain; out->maxStrain = maxStrain; out->strainOffset = strainOffset; out->fx = stress * A;
    out->fl = (uint8_t)((small ? LF_SMALL : 0) | LF_LVV | (wide1 ? LF_WIDE1 : 0) | (wide2 ? LF_WIDE2 : 0) | (acos1 ? LF_ACOS1 : 0));
    out->small = small; out->lvv = lo.lvv;
    return a.ok();
}

// Second half: the beam forces with their damping, rotated into the world, and the link's state.
// False: an operand was out of band, and no state was written.
template <class Pipes>
__device__ __forceinline__ bool link_forces_int(Pipes& a, const Sim& S, int l, float dt, const LinkPose& p, bool* diverged) {
    const int ng = __ldg(S.lneg + l), pv = __ldg(S.lpos + l);
    const int axis = __ldg(S.lax + l);
    const LMat& m = S.lm[__ldg(S.lmt + l)];
    const VMat& vN = S.vm[__ldg(S.vmat + ng)];
    const VMat& vP = S.vm[__ldg(S.vmat + pv)];
    const int nl = S.nl, nv = S.nv;
    double* st = S.lst;
    const bool small = p.small, lvv = p.lvv;
    const d3 pos2 = p.pos2, a2v = p.a2v;
    const double a1y = p.a1y, a1z = p.a1z;
    const q4 angle1 = Q4(p.a1w, 0, p.q1y, p.q1z), angle2 = p.angle2;
    const float strain = p.strain;
    // beam_forces, the zero terms left out and common products shared: b3*(2y) is 2(b3*y)
    const double fx = a.wide(p.fx);
    const double dmN = a.wide(vN.dampNum / dt), dmP = a.wide(vP.dampNum / dt);   // CVX_Voxel::dampingMultiplier
    d3 fN, fP, mN, mP;
    if (small) {
        const auto uz = a.mul(m.b2D, pos2.z), uy = a.mul(m.b2D, pos2.y), ty = a.mul(m.b3D, a2v.y), tz = a.mul(m.b3D, a2v.z);
        const double tx = a.mul(m.a2D, a2v.x);
        fN = D3(fx, a.mul(m.b1D, pos2.y) - a.mul(m.b2D, a2v.z), a.mul(m.b1D, pos2.z) + a.mul(m.b2D, a2v.y));
        mN = D3(tx, -uz - ty, uy - tz);
        mP = D3(-tx, -uz - mul2_band(ty), uy - mul2_band(tz));
    } else {
        const double tx = a.mul(m.a2D, a2v.x);
        fN = D3(fx, -a.mul(m.b2D, a.add(a1z) + a2v.z), a.mul(m.b2D, a.add(a1y) + a2v.y));
        mN = D3(tx, -a.mul(m.b3D, a.add(mul2_band(a1y)) + a2v.y), -a.mul(m.b3D, a.add(mul2_band(a1z)) + a2v.z));
        mP = D3(-tx, -a.mul(m.b3D, a.add(a1y) + mul2_band(a2v.y)), -a.mul(m.b3D, a.add(a1z) + mul2_band(a2v.z)));
    }
    fP = D3(-fN.x, -fN.y, -fN.z);
    if (lvv && vN.dampNum == 0 && vP.dampNum == 0) {
        // no bond damping: the plain form adds zeros, which change nothing but a zero's sign
        a.check(fN); a.check(mN); a.check(mP);
    } else if (lvv) {
        const d3 d2 = D3(half_band(a.add(a2v.x) - st[6 * nl + l]), half_band(a.add(a2v.y) - st[7 * nl + l]), half_band(a.add(a2v.z) - st[8 * nl + l]));
        const double dPx = half_band(a.add(pos2.x) - st[l]);
        d3 pc, tN, tP;
        const double wx = a.mul(m.sqA2xIpD, d2.x);
        if (small) {
            const double dPy = half_band(a.add(pos2.y) - st[nl + l]), dPz = half_band(a.add(pos2.z) - st[2 * nl + l]);
            const auto uz = a.mul(m.sqB2xFMpD, dPz), uy = a.mul(m.sqB2xFMpD, dPy), ty = a.mul(m.sqB3xIpD, d2.y), tz = a.mul(m.sqB3xIpD, d2.z);
            pc = D3(a.mul(m.sqA1D, dPx), a.mul(m.sqB1D, dPy) - a.mul(m.sqB2xFMpD, d2.z), a.mul(m.sqB1D, dPz) + a.mul(m.sqB2xFMpD, d2.y));
            tN = D3(-wx, uz + ty, tz - uy);
            tP = D3(wx, uz + mul2_band(ty), mul2_band(tz) - uy);
        } else {
            const double d1y = half_band(a.add(a1y) - st[4 * nl + l]), d1z = half_band(a.add(a1z) - st[5 * nl + l]);
            pc = D3(a.mul(m.sqA1D, dPx), -a.mul(m.sqB2xFMpD, a.add(d1z) + d2.z), a.mul(m.sqB2xFMpD, a.add(d1y) + d2.y));
            tN = D3(-wx, a.mul(m.sqB3xIpD, a.add(mul2_band(d1y)) + d2.y), a.mul(m.sqB3xIpD, a.add(mul2_band(d1z)) + d2.z));
            tP = D3(wx, a.mul(m.sqB3xIpD, a.add(d1y) + mul2_band(d2.y)), a.mul(m.sqB3xIpD, a.add(d1z) + mul2_band(d2.z)));
        }
        fN = D3(fN.x + a.mul(dmN, pc.x), fN.y + a.mul(dmN, pc.y), fN.z + a.mul(dmN, pc.z));
        fP = D3(fP.x - a.mul(dmP, pc.x), fP.y - a.mul(dmP, pc.y), fP.z - a.mul(dmP, pc.z));
        const double hN = half_band(dmN), hP = half_band(dmP);
        mN = D3(mN.x - a.mul(hN, tN.x), mN.y - a.mul(hN, tN.y), mN.z - a.mul(hN, tN.z));
        mP = D3(mP.x - a.mul(hP, tP.x), mP.y - a.mul(hP, tP.y), mP.z - a.mul(hP, tP.z));
    }
    const int dn = 2 * axis, dp = 2 * axis + 1;
    double* sf = S.sf;
    double* sm = S.sm;
    if (!small) {
        // one copy of the rotation for the two vectors: the instruction cache is the tighter limit
        d3 u = fN;
#pragma unroll 1
        for (int k = 0; k < 2; k++) {
            const d3 r = qrotinv_x0_int(a, angle1, u);
            if (k == 0) { fN = r; u = mN; } else mN = r;
        }
    }
    fN = to_axis_orig(axis, fN);
    mN = to_axis_orig(axis, mN);
    sf[(dn * 3 + 0) * nv + ng] = fN.x; sf[(dn * 3 + 1) * nv + ng] = fN.y; sf[(dn * 3 + 2) * nv + ng] = fN.z;
    sm[(dn * 3 + 0) * nv + ng] = mN.x; sm[(dn * 3 + 1) * nv + ng] = mN.y; sm[(dn * 3 + 2) * nv + ng] = mN.z;
    double* slot = sf;
    d3 u = fP;
#pragma unroll 1
    for (int k = 0; k < 2; k++) {
        const d3 r = to_axis_orig(axis, qrotinv_int(a, angle2, u));
        slot[(dp * 3 + 0) * nv + pv] = r.x; slot[(dp * 3 + 1) * nv + pv] = r.y; slot[(dp * 3 + 2) * nv + pv] = r.z;
        slot = sm;
        u = mP;
    }
    const float ratio = vP.E / vN.E;
    S.ss[dn * nv + ng] = 2.0f * strain / (1.0f + ratio);
    S.ss[dp * nv + pv] = 2.0f * strain * ratio / (1.0f + ratio);
    if (!a.ok()) return false;

    if (strain > 100) *diverged = true;
    st[l] = pos2.x; st[nl + l] = pos2.y; st[2 * nl + l] = pos2.z;
    st[3 * nl + l] = 0.0; st[4 * nl + l] = a1y; st[5 * nl + l] = a1z;
    st[6 * nl + l] = a2v.x; st[7 * nl + l] = a2v.y; st[8 * nl + l] = a2v.z;
    S.lsf[l] = strain; S.lsf[nl + l] = p.maxStrain; S.lsf[2 * nl + l] = p.strainOffset;
    S.lfl[l] = p.fl;
    return true;
}

}  // namespace GVX_KNS
}  // namespace gvx
