// The voxel update with its products, quotients and roots on the integer pipes, as links_int.cuh
// does for the links and for the same reason: of about 230 FP64 instructions a voxel about 100
// are additions, and those (with the temperature's sine) stay on the FP64 pipe.  The stored values
// have the bits of the plain form (voxel_update in kernels.cuh).  k_voxels on 128 settled creatures
// (203 k voxels): 119 -> 80 us, 1.66 -> 0.86 M FP64 warp instructions; one 10^3 creature 28 -> 20 us.
//
// It takes voxels without an external in simulations without the VX3 extras that act on voxels;
// others go to the plain form at once.  A voxel with an operand out of band is left to the plain
// form before anything is stored; VF_PLAIN keeps it there until it is voxel_ready.  The horizontal
// momentum of a voxel held by static friction is exactly zero: its products stand in with 1 and
// are not used.
#pragma once
#include "links_int.cuh"

namespace gvx {
namespace GVX_KNS {

template <class Pipes>
__device__ __forceinline__ q4 q_from_rotvec_int(Pipes& a, const d3& v, bool* wide) {
    const double tx = half_band(v.x), ty = half_band(v.y), tz = half_band(v.z);
    const double m2 = a.mul(tx, tx) + a.mul(ty, ty) + a.mul(tz, tz);
    double w, s;
    if (fp64i::lt_pos(a.mul(m2, m2), 5.328e-15)) {
        w = a.one - a.add(half_band(m2));
        s = a.one - a.div(m2, 6.0);
    } else {
        *wide = true;
        const double m = a.root(m2);
        double sn;
        sincos(m, &sn, &w);
        s = a.div(sn, m);
    }
    return Q4(w, a.mul(tx, s), a.mul(ty, s), a.mul(tz, s));
}

// False: the voxel is left to the plain form, and nothing was stored.
template <bool kFma>
__device__ __forceinline__ bool voxel_update_int(const Sim& S, int v, uint32_t fl, float dt, const StepTimes& st, int flags, double one, int* hash_next_table,
                                                 int* watch_moved) {
    IntPipes<kFma> a(one);
    const int nv = S.nv;
    const VMat& m = S.vm[__ldg(S.vmat + v)];
    d3 pos = D3(S.px[v], S.py[v], S.pz[v]);
    d3 lm = D3(S.mx[v], S.my[v], S.mz[v]);
    q4 q = Q4(S.qw[v], S.qx[v], S.qy[v], S.qz[v]);
    d3 am = D3(S.ax[v], S.ay[v], S.az[v]);
    const float temp = S.temp[v];
    const double dtd = a.wide(dt);

    // moment() and the new orientation
    const double* sm = S.sm;
    d3 M = (fl & 1u) ? D3(sm[v], sm[nv + v], sm[2 * nv + v]) : D3(0, 0, 0);
#pragma unroll
    for (int d = 1; d < 6; d++)
        if (fl & (1u << d)) M = D3(a.add(M.x) + sm[(d * 3) * nv + v], a.add(M.y) + sm[(d * 3 + 1) * nv + v], a.add(M.z) + sm[(d * 3 + 2) * nv + v]);
    const double* sf = S.sf;
    d3 F = (fl & 1u) ? D3(sf[v], sf[nv + v], sf[2 * nv + v]) : D3(0, 0, 0);
#pragma unroll
    for (int d = 1; d < 6; d++)
        if (fl & (1u << d)) F = D3(a.add(F.x) + sf[(d * 3) * nv + v], a.add(F.y) + sf[(d * 3 + 1) * nv + v], a.add(F.z) + sf[(d * 3 + 2) * nv + v]);
    // one copy of the rotation for the two vectors, as in link_forces_int
    {
        d3 u = M;
#pragma unroll 1
        for (int k = 0; k < 2; k++) {
            const d3 r = qrot_int(a, q, u);
            if (k == 0) { M = r; u = F; } else F = r;
        }
    }
    if (m.gDampRD != 0) {
        const double wx = a.mul(m.IinvD, am.x), wy = a.mul(m.IinvD, am.y), wz = a.mul(m.IinvD, am.z);
        M = D3(M.x - a.mul(m.gDampRD, wx), M.y - a.mul(m.gDampRD, wy), M.z - a.mul(m.gDampRD, wz));
    }
    am = D3(am.x + a.mul(dtd, M.x), am.y + a.mul(dtd, M.y), am.z + a.mul(dtd, M.z));
    const double sI = a.wide(dt * m.Iinv);
    bool wrot = false;
    q = qmul_int(a, q_from_rotvec_int(a, D3(a.mul(sI, am.x), a.mul(sI, am.y), a.mul(sI, am.z)), &wrot), q);
    fl = wrot ? (fl | VF_WROT) : (fl & ~VF_WROT);

    // force()
    const bool held = fl & VF_STATIC;
    const double vx = a.mul(m.massInvD, held ? 1.0 : lm.x), vy = a.mul(m.massInvD, held ? 1.0 : lm.y), vz = a.mul(m.massInvD, lm.z);
    if (held) a.flag(!(fp64i::eq0(lm.x) && fp64i::eq0(lm.y)));   // so only before the first step
    if (m.gDampTD != 0) {
        const double gx = a.mul(m.gDampTD, vx), gy = a.mul(m.gDampTD, vy);
        F = D3(a.add(F.x) - (held ? 0.0 : gx), a.add(F.y) - (held ? 0.0 : gy), F.z - a.mul(m.gDampTD, vz));
    }
    F.z = a.add(F.z) + m.gravForceD;
    if (flags & SF_COLLIDE) {
        const int nc = S.ccount[v];
        const float* cf = nc <= S.contact_inline ? S.cforce + (size_t)v * 3 * kContactInline : S.spill_f + 3 * (size_t)S.cspill[v];
        for (int k = 0; k < nc; k++) { F.x -= cf[3 * k]; F.y -= cf[3 * k + 1]; F.z -= cf[3 * k + 2]; }
    }
    // floorForce()
    const d3 F0 = F;
    bool contact = false;
    if (flags & SF_FLOOR) {
        const double b = a.mul(m.nom, a.wide(1 + temp * m.cte));
        const float pen = a.narrow(a.add(half_band(a.div(a.add(mul2_band(b)) + b, 3.0f))) - m.halfNom - pos.z);
        contact = pen >= 0;
        if (contact) {
            const float normal = m.penStiff * pen;
            F.z = a.add(F.z) + (a.wide(normal) - (m.cDampTD != 0 ? (double)a.mul(m.cDampTD, vz) : 0.0));
            if (held) {
                const float surf = d2f(a.mul(F.x, F.x) + a.mul(F.y, F.y)), fr = (m.mus * normal) * (m.mus * normal);
                if (surf > fr) fl &= ~VF_STATIC;
            } else if (m.muk != 0) {
                const double inv = a.div(1.0, a.root(a.mul(vx, vx) + a.mul(vy, vy)));
                const double k = a.wide(m.muk * normal);
                F.x = F.x - a.mul(k, a.mul(inv, vx));
                F.y = F.y - a.mul(k, a.mul(inv, vy));
            }
        }
        fl = contact ? (fl | VF_FLOORC) : (fl & ~VF_FLOORC);
    }
    if (!contact) fl &= ~VF_STATIC;
    lm = D3(lm.x + a.mul(dtd, F.x), lm.y + a.mul(dtd, F.y), lm.z + a.mul(dtd, F.z));
    const double sdt = a.wide(dt * m.massInv);
    d3 tr = D3(a.mul(sdt, lm.x), a.mul(sdt, lm.y), a.mul(sdt, lm.z));
    if (contact) {
        // the friction's work (none on a held voxel) against the kinetic energy
        const double hKe = a.mul(m.halfMassInv, a.mul(lm.x, lm.x) + a.mul(lm.y, lm.y));
        if (!held && fp64i::le(hKe + ((F.x - F0.x) * tr.x + (F.y - F0.y) * tr.y), 0.0)) fl |= VF_STATIC;
        if (fl & VF_STATIC) { lm.x = lm.y = 0; tr.x = tr.y = 0; }
    }
    if (!a.ok()) return false;

    pos = D3(a.add(pos.x) + tr.x, a.add(pos.y) + tr.y, a.add(pos.z) + tr.z);
    S.px[v] = pos.x; S.py[v] = pos.y; S.pz[v] = pos.z;
    S.mx[v] = lm.x; S.my[v] = lm.y; S.mz[v] = lm.z;
    S.qw[v] = q.w; S.qx[v] = q.x; S.qy[v] = q.y; S.qz[v] = q.z;
    S.ax[v] = am.x; S.ay[v] = am.y; S.az[v] = am.z;
    S.vfl[v] = fl & ~VF_PLAIN;
    voxel_after(S, v, m, fl, nullptr, pos, temp, st, flags, hash_next_table, watch_moved);
    return true;
}

}  // namespace GVX_KNS
}  // namespace gvx
