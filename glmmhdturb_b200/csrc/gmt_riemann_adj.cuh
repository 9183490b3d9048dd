// gmt_riemann_adj.cuh -- hand-written reverse sweeps of the step's physics functions: cons2prim and
// prim2cons, the ideal-MHD flux, the fast speed, HLL and the Miyoshi-Kusano HLLD (gmt_phys.cuh;
// glmmhd_turb.jl:68-115, 193-272, 335-354), and of riemann_glm (GLM pair and state floors) in the
// x-normal frame.
//
// Each function re-evaluates the forward expressions it needs and then propagates the adjoint of
// its outputs back to its inputs.  The branch conventions are those of the dual numbers and of
// the oracle's tangent step: max(a, b) passes the derivative of a when a >= b, min(a, b) of a when
// a <= b, |a| takes the sign of a >= 0, sqrt has derivative 0 at 0, and the degenerate star state
// (|denK| < 1e-12) and the fan region follow the branch the values take.  The exact-speed LLF
// paths are not covered here (riemann_x_adj returns false and the caller uses dual numbers).
#pragma once
#include "gmt_phys.cuh"

namespace gmt {

template <class R> GMT_HD R sel_ge(R a, R b) { return a >= b ? R(1) : R(0); }   // d max(a, b) / da
template <class R> GMT_HD R sel_le(R a, R b) { return a <= b ? R(1) : R(0); }   // d min(a, b) / da

// qb[0,4,5,6,7], bnb += adjoint of fast_speed(q, gamma, bn) for output adjoint cb
template <class R> GMT_HD void fast_speed_adj(const Q9<R>& q, R gamma, R bn, R cb, Q9<R>& qb, R& bnb) {
    const R rho = q.v[0];
    const R c2 = gamma * q.v[4] / rho;
    const R bsq = q.v[5] * q.v[5] + q.v[6] * q.v[6] + q.v[7] * q.v[7];
    const R b2 = bsq / rho;
    const R d2 = R(0.5) * (b2 + c2);
    const R disc = d2 * d2 - c2 * bn * bn / rho;
    const R dm = rmax(disc, R(0));
    const R sd = sqrt_r(dm);
    const R cf = sqrt_r(d2 + sd);
    const R t_b = cf > R(0) ? cb * (R(0.5) / cf) : R(0);
    R d2_b = t_b;
    const R dm_b = sd > R(0) ? t_b * (R(0.5) / sd) : R(0);
    const R disc_b = dm_b * sel_ge(disc, R(0));
    d2_b += disc_b * R(2) * d2;
    const R ir = R(1) / rho, w = bn * bn * ir;
    R c2_b = -disc_b * w;
    bnb += -disc_b * c2 * R(2) * bn * ir;
    R rho_b = disc_b * c2 * w * ir;
    const R b2_b = R(0.5) * d2_b;
    c2_b += R(0.5) * d2_b;
    const R bsq_b = b2_b * ir;
    rho_b += -b2_b * b2 * ir;
    qb.v[5] += bsq_b * R(2) * q.v[5];
    qb.v[6] += bsq_b * R(2) * q.v[6];
    qb.v[7] += bsq_b * R(2) * q.v[7];
    qb.v[4] += c2_b * gamma * ir;
    rho_b += -c2_b * c2 * ir;
    qb.v[0] += rho_b;
}

// qb += adjoint of phys_flux_x(q, gamma) (F[Bx] = F[psi] = 0) for output adjoint fb
template <class R> GMT_HD void phys_flux_x_adj(const Q9<R>& q, R gamma, const Q9<R>& fb, Q9<R>& qb) {
    const R rho = q.v[0], vx = q.v[1], vy = q.v[2], vz = q.v[3], p = q.v[4];
    const R bx = q.v[5], by = q.v[6], bz = q.v[7];
    const R b2 = bx * bx + by * by + bz * bz;
    const R ptot = p + R(0.5) * b2;
    const R vsq = vx * vx + vy * vy + vz * vz;
    const R igm1 = R(1) / (gamma - R(1));
    const R E = p * igm1 + R(0.5) * rho * vsq + R(0.5) * b2;
    const R vdotb = vx * bx + vy * by + vz * bz;
    const R f0 = fb.v[0], f1 = fb.v[1], f2 = fb.v[2], f3 = fb.v[3], f4 = fb.v[4], f6 = fb.v[6], f7 = fb.v[7];
    R rho_b = f0 * vx + f1 * vx * vx + f2 * vx * vy + f3 * vx * vz;
    R vx_b = f0 * rho + f1 * R(2) * rho * vx + f2 * rho * vy + f3 * rho * vz + f4 * (E + ptot) + f6 * by + f7 * bz;
    R vy_b = f2 * rho * vx - f6 * bx;
    R vz_b = f3 * rho * vx - f7 * bx;
    const R ptot_b = f1 + f4 * vx;
    const R E_b = f4 * vx;
    const R vdotb_b = -f4 * bx;
    R bx_b = -R(2) * f1 * bx - f2 * by - f3 * bz - f4 * vdotb - f6 * vy - f7 * vz;
    R by_b = -f2 * bx + f6 * vx;
    R bz_b = -f3 * bx + f7 * vx;
    vx_b += vdotb_b * bx; vy_b += vdotb_b * by; vz_b += vdotb_b * bz;
    bx_b += vdotb_b * vx; by_b += vdotb_b * vy; bz_b += vdotb_b * vz;
    R p_b = E_b * igm1 + ptot_b;
    rho_b += E_b * R(0.5) * vsq;
    vx_b += E_b * rho * vx; vy_b += E_b * rho * vy; vz_b += E_b * rho * vz;
    const R b2_b = R(0.5) * E_b + R(0.5) * ptot_b;
    bx_b += b2_b * R(2) * bx; by_b += b2_b * R(2) * by; bz_b += b2_b * R(2) * bz;
    qb.v[0] += rho_b; qb.v[1] += vx_b; qb.v[2] += vy_b; qb.v[3] += vz_b; qb.v[4] += p_b;
    qb.v[5] += bx_b; qb.v[6] += by_b; qb.v[7] += bz_b;
}

// cb += adjoint of cons2prim(c, gamma, smallr, pf) for output adjoint qb
template <class R>
GMT_HD void cons2prim_adj(const Q9<R>& c, R gamma, R smallr, R pf, const Q9<R>& qb, Q9<R>& cb) {
    const R rho = rmax(c.v[0], smallr);
    const R ir = R(1) / rho;
    const R msq = c.v[1] * c.v[1] + c.v[2] * c.v[2] + c.v[3] * c.v[3];
    const R ekin = R(0.5) * msq * ir;
    const R emag = R(0.5) * (c.v[5] * c.v[5] + c.v[6] * c.v[6] + c.v[7] * c.v[7]);
    const R pr = (gamma - R(1)) * (c.v[4] - ekin - emag);
    const R pr_b = qb.v[4] * sel_ge(pr, pf);
    const R g1 = pr_b * (gamma - R(1));
    const R ekin_b = -g1, emag_b = -g1;
    cb.v[4] += g1;
    cb.v[5] += qb.v[5] + emag_b * c.v[5];
    cb.v[6] += qb.v[6] + emag_b * c.v[6];
    cb.v[7] += qb.v[7] + emag_b * c.v[7];
    cb.v[8] += qb.v[8];
    cb.v[1] += qb.v[1] * ir + ekin_b * c.v[1] * ir;
    cb.v[2] += qb.v[2] * ir + ekin_b * c.v[2] * ir;
    cb.v[3] += qb.v[3] * ir + ekin_b * c.v[3] * ir;
    const R ir_b = qb.v[1] * c.v[1] + qb.v[2] * c.v[2] + qb.v[3] * c.v[3] + ekin_b * R(0.5) * msq;
    const R rho_b = qb.v[0] - ir_b * ir * ir;
    cb.v[0] += rho_b * sel_ge(c.v[0], smallr);
}

// qb += adjoint of prim2cons(q, gamma) for output adjoint ub (the psi slot passes through)
template <class R> GMT_HD void prim2cons_adj(const Q9<R>& q, R gamma, const Q9<R>& ub, Q9<R>& qb) {
    const R rho = q.v[0], vx = q.v[1], vy = q.v[2], vz = q.v[3];
    const R vsq = vx * vx + vy * vy + vz * vz;
    const R E_b = ub.v[4];
    qb.v[0] += ub.v[0] + ub.v[1] * vx + ub.v[2] * vy + ub.v[3] * vz + E_b * R(0.5) * vsq;
    qb.v[1] += ub.v[1] * rho + E_b * rho * vx;
    qb.v[2] += ub.v[2] * rho + E_b * rho * vy;
    qb.v[3] += ub.v[3] * rho + E_b * rho * vz;
    qb.v[4] += E_b / (gamma - R(1));
    qb.v[5] += ub.v[5] + E_b * q.v[5];
    qb.v[6] += ub.v[6] + E_b * q.v[6];
    qb.v[7] += ub.v[7] + E_b * q.v[7];
    qb.v[8] += ub.v[8];
}

// HLL (hll_x): Lb, Rb, bnb += adjoint for flux adjoint fb; f[5], f[8] are the GLM fluxes set by the
// caller, so fb[5], fb[8] do not enter
template <class R>
GMT_HD void hll_x_adj(const Q9<R>& L, const Q9<R>& Rr, R gamma, R bn, const Q9<R>& fb, Q9<R>& Lb, Q9<R>& Rb, R& bnb) {
    const R cfL = fast_speed(L, gamma, bn), cfR = fast_speed(Rr, gamma, bn);
    const R aL = L.v[1] - cfL, aR = Rr.v[1] - cfR;
    const R m = rmin(aL, aR);
    const R SL = rmin(m, R(0));
    const R bL = L.v[1] + cfL, bR = Rr.v[1] + cfR;
    const R M = rmax(bL, bR);
    const R SR = rmax(M, R(0));
    const Q9<R> fL = phys_flux_x(L, gamma), fR = phys_flux_x(Rr, gamma);
    const Q9<R> uL = prim2cons(L, gamma), uR = prim2cons(Rr, gamma);
    const R ihd = R(1) / (SR - SL);
    Q9<R> fLb, fRb, uLb, uRb;
    R SL_b = R(0), SR_b = R(0), ihd_b = R(0);
#pragma unroll
    for (int i = 0; i < 9; ++i) {
        const R g = (i == 5 || i == 8) ? R(0) : fb.v[i];
        const R num = SR * fL.v[i] - SL * fR.v[i] + SL * SR * (uR.v[i] - uL.v[i]);
        ihd_b += g * num;
        const R nb = g * ihd;
        SR_b += nb * fL.v[i] + nb * SL * (uR.v[i] - uL.v[i]);
        SL_b += -nb * fR.v[i] + nb * SR * (uR.v[i] - uL.v[i]);
        fLb.v[i] = nb * SR;
        fRb.v[i] = -nb * SL;
        uRb.v[i] = nb * SL * SR;
        uLb.v[i] = -nb * SL * SR;
    }
    // ihd = 1 / (SR - SL)
    const R dd_b = -ihd_b * ihd * ihd;
    SR_b += dd_b;
    SL_b -= dd_b;
    phys_flux_x_adj(L, gamma, fLb, Lb);
    phys_flux_x_adj(Rr, gamma, fRb, Rb);
    prim2cons_adj(L, gamma, uLb, Lb);
    prim2cons_adj(Rr, gamma, uRb, Rb);
    // SL = min(min(aL, aR), 0), SR = max(max(bL, bR), 0)
    const R m_b = SL_b * sel_le(m, R(0));
    const R aL_b = m_b * sel_le(aL, aR), aR_b = m_b - aL_b;
    const R M_b = SR_b * sel_ge(M, R(0));
    const R bL_b = M_b * sel_ge(bL, bR), bR_b = M_b - bL_b;
    Lb.v[1] += aL_b + bL_b;
    Rb.v[1] += aR_b + bR_b;
    fast_speed_adj(L, gamma, bn, -aL_b + bL_b, Lb, bnb);
    fast_speed_adj(Rr, gamma, bn, -aR_b + bR_b, Rb, bnb);
}

// HLLD star state of one side (hlld_star) and its reverse; `ik` is 1 / denK, `degen` the branch taken
template <class R> struct HStar {
    R vy, vz, by, bz, ik;
    bool degen;
};
template <class R> GMT_HD HStar<R> hstar(R d, R u, R v, R w, R by, R bz, R S, R SM, R bn) {
    HStar<R> s;
    const R denK = d * (S - u) * (S - SM) - bn * bn;
    s.degen = rabs(denK) < R(1e-12);
    s.vy = v; s.vz = w; s.by = by; s.bz = bz; s.ik = R(0);
    if (!s.degen) {
        s.ik = R(1) / denK;
        const R fac = bn * (SM - u) * s.ik, t = (d * (S - u) * (S - u) - bn * bn) * s.ik;
        s.vy = v - by * fac;
        s.vz = w - bz * fac;
        s.by = by * t;
        s.bz = bz * t;
    }
    return s;
}
template <class R>
GMT_HD void hstar_adj(R d, R u, R by, R bz, R S, R SM, R bn, const HStar<R>& s, R vy_b, R vz_b, R byS_b, R bzS_b,
                      R& d_b, R& u_b, R& v_b, R& w_b, R& by_b, R& bz_b, R& S_b, R& SM_b, R& bn_b) {
    v_b += vy_b;
    w_b += vz_b;
    if (s.degen) {
        by_b += byS_b; bz_b += bzS_b;
        return;
    }
    const R a = S - u, b = S - SM, ik = s.ik;
    const R fac = bn * (SM - u) * ik, t = (d * a * a - bn * bn) * ik;
    by_b += -vy_b * fac + byS_b * t;
    bz_b += -vz_b * fac + bzS_b * t;
    const R fac_b = -(vy_b * by + vz_b * bz) * ik;        // of the numerators
    const R num_b = (byS_b * by + bzS_b * bz) * ik;
    const R denK_b = -(num_b * t + fac_b * fac);
    bn_b += fac_b * (SM - u) - R(2) * bn * (num_b + denK_b);
    d_b += (num_b * a + denK_b * b) * a;
    const R a_b = num_b * R(2) * d * a + denK_b * d * b;
    const R b_b = denK_b * d * a;
    SM_b += fac_b * bn - b_b;
    u_b += -fac_b * bn - a_b;
    S_b += a_b + b_b;
}

// HLLD (hlld_x): Lb, Rb, bnb += adjoint for flux adjoint fb (fb[5], fb[8] do not enter).
//
// The fan is swept in the frame of its sampled side s (the left one when SM >= 0, which every region
// implies: SL* >= 0 has SM >= 0, SR* < 0 has SM < 0) and the other side o.  SM, pT* and the averages
// are the same functions of (s, o) as of (L, R): exchanging the sides changes the sign of numerator
// and denominator alike, and of the double-star differences, which sgn(bn) absorbs.  So one body
// serves the four regions, F = F_s + S_s (U*_s - U_s), plus S*_s (U**_s - U*_s) in the double-star
// ones, instead of a copy per region: a warp whose faces lie in different regions no longer runs
// several of them in turn, and the code fits the instruction cache better (in FP64 the pass spent
// most of its issue slots waiting for instructions: 64^3 FP64 513 us).  Only s has an energy and a
// flux of its own in the result, so those of o are not formed, and one fast speed carries the whole
// adjoint of max(cL, cR).  The branches are decided by the forward step's own expressions; quotients
// that only enter the adjoint are formed with one reciprocal per divisor.
template <class R>
GMT_HD void hlld_x_adj(const Q9<R>& L, const Q9<R>& Rr, R gamma, R bn, const Q9<R>& fb, Q9<R>& Lb, Q9<R>& Rb, R& bnb) {
    const R tiny = R(1e-12), igm1 = R(1) / (gamma - R(1));
    bool left;
    R S, oS, SM, pts, cfL, cfR, xL, xR;
    {
        const R dL = L.v[0], uL = L.v[1], dR = Rr.v[0], uR = Rr.v[1];
        const R ptL = L.v[4] + R(0.5) * (bn * bn + L.v[6] * L.v[6] + L.v[7] * L.v[7]);
        const R ptR = Rr.v[4] + R(0.5) * (bn * bn + Rr.v[6] * Rr.v[6] + Rr.v[7] * Rr.v[7]);
        cfL = fast_speed(L, gamma, bn);
        cfR = fast_speed(Rr, gamma, bn);
        xL = rmin(uL, uR) - rmax(cfL, cfR);
        xR = rmax(uL, uR) + rmax(cfL, cfR);
        const R SL = rmin(xL, R(0)), SR = rmax(xR, R(0));
        const R aL = SL - uL, aR = SR - uR;
        const R den = aR * dR - aL * dL;
        SM = (aR * dR * uR - aL * dL * uL - ptR + ptL) / den;
        pts = (aR * dR * ptL - aL * dL * ptR + dL * dR * aR * aL * (uR - uL)) / den;
        left = SM >= R(0);
        S = left ? SL : SR;
        oS = left ? SR : SL;
    }
    const R sig = left ? R(1) : R(-1);
    // (value by value: a reference chosen at run time would put the states in local memory)
    const R d = left ? L.v[0] : Rr.v[0], u = left ? L.v[1] : Rr.v[1], v = left ? L.v[2] : Rr.v[2];
    const R w = left ? L.v[3] : Rr.v[3], p = left ? L.v[4] : Rr.v[4];
    const R by = left ? L.v[6] : Rr.v[6], bz = left ? L.v[7] : Rr.v[7];
    const R od = left ? Rr.v[0] : L.v[0], ou = left ? Rr.v[1] : L.v[1], ov = left ? Rr.v[2] : L.v[2];
    const R ow = left ? Rr.v[3] : L.v[3], op = left ? Rr.v[4] : L.v[4];
    const R oby = left ? Rr.v[6] : L.v[6], obz = left ? Rr.v[7] : L.v[7];
    const R b2 = bn * bn + by * by + bz * bz, pt = p + R(0.5) * b2;
    const R vsq = u * u + v * v + w * w, E = p * igm1 + R(0.5) * d * vsq + R(0.5) * b2;
    const R opt = op + R(0.5) * (bn * bn + oby * oby + obz * obz);
    const R a = S - u, oa = oS - ou, l = S - SM, ol = oS - SM;
    const R il = R(1) / l;
    const R q = d * a / l, oq = od * oa / ol;
    const R ds = rmax(q, tiny), ods = rmax(oq, tiny);
    const R sq = sqrt_r(ds), osq = sqrt_r(ods);
    const R abn = rabs(bn);
    const R Ss = SM - sig * (abn / sq);                       // S*_L or S*_R
    const bool inner = left ? Ss < R(0) : Ss >= R(0);

    // forward: the star state of s
    const HStar<R> st = hstar(d, u, v, w, by, bz, S, SM, bn);
    const R vdotb = u * bn + v * by + w * bz, vdotbs = SM * bn + st.vy * st.by + st.vz * st.bz;
    const R Es = (a * E - pt * u + pts * SM + bn * (vdotb - vdotbs)) * il;

    const R g0 = fb.v[0], g1 = fb.v[1], g2 = fb.v[2], g3 = fb.v[3], g4 = fb.v[4], g6 = fb.v[6], g7 = fb.v[7];
    // F_s + S (U* - U): adjoints of U* (gs), of U (-S g) and of S
    R SM_b = g1 * S * ds, bn_b = R(0);
    R S_b = g0 * (ds - d) + g1 * (ds * SM - d * u) + g2 * (ds * st.vy - d * v) + g3 * (ds * st.vz - d * w) +
            g4 * (Es - E) + g6 * (st.by - by) + g7 * (st.bz - bz);
    R f = S;                                                    // U*'s weight: S, less S* in the double star
    R sq_b = R(0), osq_b = R(0), Ss_b = R(0), oS_b = R(0);
    R vy_b = R(0), vz_b = R(0), bys_b = R(0), bzs_b = R(0), vdotbs_b = R(0), Es_b = R(0), ds_b = R(0);
    R d_b = R(0), u_b = R(0), v_b = R(0), w_b = R(0), by_b = R(0), bz_b = R(0), E_b, pt_b;
    R od_b = R(0), ou_b = R(0), ov_b = R(0), ow_b = R(0), oby_b = R(0), obz_b = R(0), opt_b;
    if (inner) {
        const HStar<R> ot = hstar(od, ou, ov, ow, oby, obz, oS, SM, bn);
        const R sg = bn >= R(0) ? sig : -sig, invsum = R(1) / (sq + osq), sqq = sq * osq;
        const R vyss = (sq * st.vy + osq * ot.vy + (ot.by - st.by) * sg) * invsum;
        const R vzss = (sq * st.vz + osq * ot.vz + (ot.bz - st.bz) * sg) * invsum;
        const R byss = (sq * ot.by + osq * st.by + sqq * (ot.vy - st.vy) * sg) * invsum;
        const R bzss = (sq * ot.bz + osq * st.bz + sqq * (ot.vz - st.vz) * sg) * invsum;
        const R vdotbss = SM * bn + vyss * byss + vzss * bzss;
        const R dv = vdotbs - vdotbss;
        // F += S* (U** - U*), U**'s energy Es - sq (v.B* - v.B**) sgn
        Ss_b = g2 * ds * (vyss - st.vy) + g3 * ds * (vzss - st.vz) - g4 * sq * dv * sg + g6 * (byss - st.by) +
               g7 * (bzss - st.bz);
        f = S - Ss;
        const R e = g4 * Ss * sg;
        sq_b = -e * dv;
        vdotbs_b = -e * sq;
        const R vdotbss_b = e * sq;
        ds_b = Ss * (g0 + g1 * SM + g2 * vyss + g3 * vzss);
        SM_b += g1 * Ss * ds + vdotbss_b * bn;
        bn_b += vdotbss_b * SM;
        Es_b = g4 * Ss;
        // the averages (divided by the sum of roots)
        const R tvy = (g2 * Ss * ds + vdotbss_b * byss) * invsum, tvz = (g3 * Ss * ds + vdotbss_b * bzss) * invsum;
        const R tby = (g6 * Ss + vdotbss_b * vyss) * invsum, tbz = (g7 * Ss + vdotbss_b * vzss) * invsum;
        const R sum_b = -(tvy * vyss + tvz * vzss + tby * byss + tbz * bzss);
        const R cross = (tby * (ot.vy - st.vy) + tbz * (ot.vz - st.vz)) * sg;
        sq_b += tvy * st.vy + tvz * st.vz + tby * ot.by + tbz * ot.bz + osq * cross + sum_b;
        osq_b = tvy * ot.vy + tvz * ot.vz + tby * st.by + tbz * st.bz + sq * cross + sum_b;
        vy_b = tvy * sq - tby * sqq * sg;
        vz_b = tvz * sq - tbz * sqq * sg;
        bys_b = -tvy * sg + tby * osq;
        bzs_b = -tvz * sg + tbz * osq;
        hstar_adj(od, ou, oby, obz, oS, SM, bn, ot, tvy * osq + tby * sqq * sg, tvz * osq + tbz * sqq * sg,
                  tvy * sg + tby * sq, tvz * sg + tbz * sq, od_b, ou_b, ov_b, ow_b, oby_b, obz_b, oS_b, SM_b, bn_b);
        // S* = SM - sig |bn| / sq
        const R isq = R(1) / sq, h = sig * Ss_b * isq;
        SM_b += Ss_b;
        bn_b += bn >= R(0) ? -h : h;
        sq_b += h * abn * isq;
    }
    // U* = (ds, ds SM, ds vy*, ds vz*, Es, bn, by*, bz*) with weight f; U with weight -S
    ds_b += f * (g0 + g1 * SM + g2 * st.vy + g3 * st.vz);
    if (inner) SM_b -= g1 * Ss * ds;                            // (f - S) g1 ds
    vy_b += f * g2 * ds;
    vz_b += f * g3 * ds;
    bys_b += f * g6;
    bzs_b += f * g7;
    Es_b += f * g4;
    d_b -= S * (g0 + g1 * u + g2 * v + g3 * w);
    u_b -= S * g1 * d; v_b -= S * g2 * d; w_b -= S * g3 * d;
    E_b = -S * g4;
    by_b -= S * g6; bz_b -= S * g7;
    // Es = (a E - pt u + pts SM + bn (v.B - v.B*)) / l
    const R n_b = Es_b * il, l_b0 = -n_b * Es;
    R pts_b = n_b * SM;
    S_b += l_b0 + n_b * E;
    SM_b += n_b * pts - l_b0;
    u_b -= n_b * (E + pt);
    E_b += n_b * a;
    pt_b = -n_b * u;
    const R vdotb_b = n_b * bn;
    vdotbs_b -= vdotb_b;
    bn_b += n_b * (vdotb - vdotbs) + vdotbs_b * SM + vdotb_b * u;
    SM_b += vdotbs_b * bn;
    vy_b += vdotbs_b * st.by; bys_b += vdotbs_b * st.vy;
    vz_b += vdotbs_b * st.bz; bzs_b += vdotbs_b * st.vz;
    u_b += vdotb_b * bn;
    v_b += vdotb_b * by; by_b += vdotb_b * v;
    w_b += vdotb_b * bz; bz_b += vdotb_b * w;
    hstar_adj(d, u, by, bz, S, SM, bn, st, vy_b, vz_b, bys_b, bzs_b, d_b, u_b, v_b, w_b, by_b, bz_b, S_b, SM_b, bn_b);
    // roots and floors, then rho* = d a / l of either side
    ds_b += sq > R(0) ? sq_b * (R(0.5) / sq) : R(0);
    const R q_b = ds_b * sel_ge(q, tiny) * il;
    R a_b = q_b * d;
    d_b += q_b * a;
    S_b -= q_b * q;
    SM_b += q_b * q;
    R oa_b = R(0);
    if (inner) {
        const R oq_b = (osq > R(0) ? osq_b * (R(0.5) / osq) : R(0)) * sel_ge(oq, tiny) / ol;
        oa_b = oq_b * od;
        od_b += oq_b * oa;
        oS_b -= oq_b * oq;
        SM_b += oq_b * oq;
    }
    {
        // pts and SM over den = oa od - a d (with s in the place of L)
        const R m = a * d, om = oa * od, iden = R(1) / (om - m), du = ou - u;
        const R tn = pts_b * iden, sn = SM_b * iden, den_b = -(tn * pts + sn * SM);
        const R om_b = tn * (pt + m * du) + sn * ou + den_b, m_b = tn * (om * du - opt) - sn * u - den_b;
        oa_b += om_b * od;
        od_b += om_b * oa;
        a_b += m_b * d;
        d_b += m_b * a;
        pt_b += tn * om + sn;
        opt_b = -tn * m - sn;
        const R du_b = tn * m * om;
        ou_b += du_b + sn * om - oa_b;
        u_b += -du_b - sn * m - a_b;
        S_b += a_b;
        oS_b += oa_b;
    }
    // F_s = phys_flux_x of (d, u, v, w, p, bn, by, bz)
    R p_b = R(0);
    {
        const Q9<R> qf{{d, u, v, w, p, bn, by, bz, R(0)}};
        const Q9<R> gf{{g0, g1, g2, g3, g4, R(0), g6, g7, R(0)}};
        Q9<R> qb;
#pragma unroll
        for (int i = 0; i < 9; ++i) qb.v[i] = R(0);
        phys_flux_x_adj(qf, gamma, gf, qb);
        d_b += qb.v[0]; u_b += qb.v[1]; v_b += qb.v[2]; w_b += qb.v[3]; p_b += qb.v[4];
        bn_b += qb.v[5]; by_b += qb.v[6]; bz_b += qb.v[7];
    }
    // E = p/(gamma-1) + d|v|^2/2 + b2/2, pt = p + b2/2 (of o only pt)
    const R b2_b = E_b + pt_b;                                  // twice the adjoint of b2
    p_b += E_b * igm1 + pt_b;
    d_b += E_b * R(0.5) * vsq;
    u_b += E_b * d * u; v_b += E_b * d * v; w_b += E_b * d * w;
    by_b += b2_b * by; bz_b += b2_b * bz;
    oby_b += opt_b * oby; obz_b += opt_b * obz;
    bn_b += (b2_b + opt_b) * bn;
    // back to L and R
    const R SL_b = left ? S_b : oS_b, SR_b = left ? oS_b : S_b;
    const R xL_b = SL_b * sel_le(xL, R(0)), xR_b = SR_b * sel_ge(xR, R(0));
    const R ul_min = sel_le(L.v[1], Rr.v[1]), ul_max = sel_ge(L.v[1], Rr.v[1]);
    const R uLx = xL_b * ul_min + xR_b * ul_max, uRx = xL_b + xR_b - uLx;
    Lb.v[0] += left ? d_b : od_b;   Rb.v[0] += left ? od_b : d_b;
    Lb.v[1] += (left ? u_b : ou_b) + uLx;
    Rb.v[1] += (left ? ou_b : u_b) + uRx;
    Lb.v[2] += left ? v_b : ov_b;   Rb.v[2] += left ? ov_b : v_b;
    Lb.v[3] += left ? w_b : ow_b;   Rb.v[3] += left ? ow_b : w_b;
    Lb.v[4] += left ? p_b : opt_b;  Rb.v[4] += left ? opt_b : p_b;
    Lb.v[6] += left ? by_b : oby_b; Rb.v[6] += left ? oby_b : by_b;
    Lb.v[7] += left ? bz_b : obz_b; Rb.v[7] += left ? obz_b : bz_b;
    // max(cL, cR) takes the side of the larger speed
    {
        const bool cl = cfL >= cfR;
        Q9<R> c, cb;
#pragma unroll
        for (int i = 0; i < 9; ++i) {
            c.v[i] = cl ? L.v[i] : Rr.v[i];
            cb.v[i] = R(0);
        }
        fast_speed_adj(c, gamma, bn, xR_b - xL_b, cb, bn_b);
        const R m = cl ? R(1) : R(0), om = R(1) - m;
        Lb.v[0] += cb.v[0] * m; Rb.v[0] += cb.v[0] * om;
        Lb.v[4] += cb.v[4] * m; Rb.v[4] += cb.v[4] * om;
        Lb.v[5] += cb.v[5] * m; Rb.v[5] += cb.v[5] * om;
        Lb.v[6] += cb.v[6] * m; Rb.v[6] += cb.v[6] * om;
        Lb.v[7] += cb.v[7] * m; Rb.v[7] += cb.v[7] * om;
    }
    bnb += bn_b;
}

// Reverse of riemann_glm<0, RIEM> (floors, GLM pair, solver; glmmhd_turb.jl:275-292): Lqb, Rqb =
// J^T fb.  Returns false for the exact-speed LLF paths, which the caller differentiates otherwise.
template <int RIEM, class R>
GMT_HD bool riemann_x_adj(const Q9<R>& Lq, const Q9<R>& Rq, const Q9<R>& fb, const Consts<R>& K, R ch, bool use_llf,
                          Q9<R>& Lqb, Q9<R>& Rqb) {
    if (RIEM != RIEM_HLLD && RIEM != RIEM_HLL) return false;
    Q9<R> L = Lq, Rr = Rq;
    L.v[0] = rmax(L.v[0], K.smallr); L.v[4] = rmax(L.v[4], K.pfl);
    Rr.v[0] = rmax(Rr.v[0], K.smallr); Rr.v[4] = rmax(Rr.v[4], K.pfl);
    if (RIEM == RIEM_HLLD) {
        const bool uself = (K.llf_dmin > R(0) && rmin(L.v[0], Rr.v[0]) < K.llf_dmin) ||
                           (K.llf_pmin > R(0) && rmin(L.v[4], Rr.v[4]) < K.llf_pmin) || use_llf;
        if (uself) return false;
    }
    R bns, psis;
    glm_pair(L.v[5], Rr.v[5], L.v[8], Rr.v[8], ch, bns, psis);
    L.v[5] = bns;
    Rr.v[5] = bns;
    Q9<R> Lb, Rb;
#pragma unroll
    for (int i = 0; i < 9; ++i) { Lb.v[i] = R(0); Rb.v[i] = R(0); }
    R bnb = R(0);
    if (RIEM == RIEM_HLLD) hlld_x_adj(L, Rr, K.gamma, bns, fb, Lb, Rb, bnb);
    else hll_x_adj(L, Rr, K.gamma, bns, fb, Lb, Rb, bnb);
    // f[5] = psis, f[8] = ch^2 bns; the solver's L[5] = R[5] = bns
    const R bns_b = bnb + Lb.v[5] + Rb.v[5] + fb.v[8] * ch * ch;
    const R psis_b = fb.v[5];
    Lb.v[5] = R(0.5) * bns_b + R(0.5) * ch * psis_b;
    Rb.v[5] = R(0.5) * bns_b - R(0.5) * ch * psis_b;
    Lb.v[8] += R(0.5) * bns_b / ch + R(0.5) * psis_b;
    Rb.v[8] += -R(0.5) * bns_b / ch + R(0.5) * psis_b;
    Lqb = Lb;
    Rqb = Rb;
    Lqb.v[0] = Lb.v[0] * sel_ge(Lq.v[0], K.smallr);
    Lqb.v[4] = Lb.v[4] * sel_ge(Lq.v[4], K.pfl);
    Rqb.v[0] = Rb.v[0] * sel_ge(Rq.v[0], K.smallr);
    Rqb.v[4] = Rb.v[4] * sel_ge(Rq.v[4], K.pfl);
    return true;
}


// Reverse sweep of the update epilogue finish_update (void floor, psi damping, forcing kick;
// glmmhd_turb.jl:450-475): given the output adjoint ob, the adjoint rb of the pre-epilogue state
// r and ab of the three accelerations.  A max(a, b) passes its adjoint to a when a >= b, as the
// dual-number evaluation of the forward does.
template <class R>
GMT_HD void finish_update_adj(const Q9<R>& rin, const Consts<R>& K, R glm_fac, bool turb, R ax, R ay, R az, R dt,
                              const Q9<R>& ob, Q9<R>& rb, R ab[3]) {
    Q9<R> r = rin;
    const bool voidf = r.v[0] < K.smallr;
    if (voidf) {
        r.v[0] = K.smallr; r.v[1] = R(0); r.v[2] = R(0); r.v[3] = R(0);
        r.v[4] = K.pfl / (K.gamma - R(1)) + R(0.5) * (r.v[5] * r.v[5] + r.v[6] * r.v[6] + r.v[7] * r.v[7]);
    }
    Q9<R> b = ob;   // adjoint of the state after the void floor (psi handled below)
    ab[0] = ab[1] = ab[2] = R(0);
    if (turb && r.v[0] >= K.turb_min_rho) {
        const R rho = r.v[0], rhom = rmax(rho, K.smallr), irm = R(1) / rhom;
        const R fl = rho * (K.smallc * K.smallc);
        const R acc[3] = {ax, ay, az};
        // forward values and branch flags of the six floored energy updates
        R e = r.v[4], m[3];
        bool t[6];
#pragma unroll
        for (int i = 0; i < 3; ++i) {
            const R x = e - R(0.5) * r.v[1 + i] * r.v[1 + i] / rhom;
            t[i] = x >= fl;
            e = t[i] ? x : fl;
        }
#pragma unroll
        for (int i = 0; i < 3; ++i) m[i] = r.v[1 + i] + rhom * acc[i] * dt;
#pragma unroll
        for (int i = 0; i < 3; ++i) {
            const R x = e + R(0.5) * m[i] * m[i] / rhom;
            t[3 + i] = x >= fl;
            e = t[3 + i] ? x : fl;
        }
        // reverse
        R eb = ob.v[4], flb = R(0), rhomb = R(0);
        R mb[3] = {ob.v[1], ob.v[2], ob.v[3]};
        R vb[3] = {R(0), R(0), R(0)};
#pragma unroll
        for (int i = 2; i >= 0; --i) {
            if (t[3 + i]) {
                mb[i] += eb * m[i] * irm;
                rhomb -= eb * R(0.5) * m[i] * m[i] * irm * irm;
            } else {
                flb += eb;
                eb = R(0);
            }
        }
#pragma unroll
        for (int i = 0; i < 3; ++i) {
            vb[i] += mb[i];
            rhomb += mb[i] * acc[i] * dt;
            ab[i] = mb[i] * rhom * dt;
        }
#pragma unroll
        for (int i = 2; i >= 0; --i) {
            if (t[i]) {
                vb[i] -= eb * r.v[1 + i] * irm;
                rhomb += eb * R(0.5) * r.v[1 + i] * r.v[1 + i] * irm * irm;
            } else {
                flb += eb;
                eb = R(0);
            }
        }
        b.v[1] = vb[0]; b.v[2] = vb[1]; b.v[3] = vb[2];
        b.v[4] = eb;
        b.v[0] = ob.v[0] + flb * (K.smallc * K.smallc) + (rho >= K.smallr ? rhomb : R(0));
    }
    rb = b;
    rb.v[8] = ob.v[8] * glm_fac;
    if (voidf) {
        // rho, momentum and E were overwritten: only B reaches E through the magnetic energy
        rb.v[5] += b.v[4] * r.v[5];
        rb.v[6] += b.v[4] * r.v[6];
        rb.v[7] += b.v[4] * r.v[7];
        rb.v[0] = rb.v[1] = rb.v[2] = rb.v[3] = rb.v[4] = R(0);
    }
}

}  // namespace gmt
