// box.cuh -- the box algebra of a step by one thread, and the per-atom terms
// of the kinetic moment and of update_therm_avs, shared by the step kernels
// (eam.cu) and the fused runs of steps (run.cu).
#pragma once

#include "engine.h"

namespace moldy {

// kinten's moment M = sum m x1 x1^T over atoms with a species
// (src/thermostat_m.F90:138-157); tk = B0 M / dt^2 in k_finalize_force
__device__ __forceinline__ void kin_moment(double (&v)[6], double m, double ux, double uy, double uz) {
    v[0] += m * ux * ux; v[1] += m * uy * uy; v[2] += m * uz * uz;
    v[3] += m * ux * uy; v[4] += m * ux * uz; v[5] += m * uy * uz;
}

// True in every thread of the block that finishes last of the grid, once the
// partials of all blocks are visible to it; the ticket is left at zero for the
// next launch.
__device__ __forceinline__ bool last_block(int32_t *ticket) {
    __shared__ int last;
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0) {
        last = atomicAdd(ticket, 1) == (int)gridDim.x - 1;
        if (last) *ticket = 0;
    }
    __syncthreads();
    if (last) __threadfence();
    return last != 0;
}

// ---------------------------------------------------------- thermo sums ----
// update_therm_avs (src/dynamics_m.F90:649-734): tg, tgdot (ivol != 1),
// tgid = tg^-1 tgdot, vol, and per-atom s1 = sum |F|^2, s2 = sum |F|^4,
// s3 = sum m |B0 x1|^2.
__device__ __forceinline__ bool therm_box(const Params &p, const double *b0, const double *b1, double *tg,
                                          double *tgdot, double *tginv, double *tgid, double &vol) {
#pragma unroll
    for (int k = 0; k < 9; ++k) { tg[k] = 0.0; tgdot[k] = 0.0; }
#pragma unroll
    for (int i = 1; i <= 3; ++i)
#pragma unroll
        for (int k = 1; k <= 3; ++k)
#pragma unroll
            for (int j = 1; j <= 3; ++j) {
                MAT(tg, i, j) = MAT(tg, i, j) + MAT(b0, k, i) * MAT(b0, k, j);
                if (p.ivol != 1)
                    MAT(tgdot, i, j) = MAT(tgdot, i, j) + MAT(b1, k, i) * MAT(b0, k, j) +
                                       MAT(b0, k, i) * MAT(b1, k, j);
            }
    bool ok = mat_invert(tg, tginv);
    mat_mul(tginv, tgdot, tgid);
    vol = mat_volume(b0);
    return ok;
}

// The box quantities k_therm needs, from the box after the force call:
// tgid = tg^-1 tgdot of the new B1 and cof(B0)/vol (the b0_xxdet ... of
// update_therm_avs); computed once, by one thread, from register copies of
// B0 and B1.
static __device__ void therm_prep(const Params &p, const double *b, const double *b1, BoxState &B) {
    double tg[9], tgdot[9], tginv[9], tgid[9], vol, d[9];   // d row-major as in the reference's names
    therm_box(p, b, b1, tg, tgdot, tginv, tgid, vol);
    d[0] = (MAT(b, 2, 2) * MAT(b, 3, 3) - MAT(b, 2, 3) * MAT(b, 3, 2)) / vol;
    d[1] = (MAT(b, 2, 3) * MAT(b, 3, 1) - MAT(b, 3, 3) * MAT(b, 2, 1)) / vol;
    d[2] = (MAT(b, 2, 1) * MAT(b, 3, 2) - MAT(b, 3, 1) * MAT(b, 2, 2)) / vol;
    d[3] = (MAT(b, 3, 2) * MAT(b, 1, 3) - MAT(b, 1, 2) * MAT(b, 3, 3)) / vol;
    d[4] = (MAT(b, 1, 1) * MAT(b, 3, 3) - MAT(b, 1, 3) * MAT(b, 3, 1)) / vol;
    d[5] = (MAT(b, 3, 1) * MAT(b, 1, 2) - MAT(b, 1, 1) * MAT(b, 3, 2)) / vol;
    d[6] = (MAT(b, 1, 2) * MAT(b, 2, 3) - MAT(b, 2, 2) * MAT(b, 1, 3)) / vol;
    d[7] = (MAT(b, 1, 3) * MAT(b, 2, 1) - MAT(b, 1, 1) * MAT(b, 2, 3)) / vol;
    d[8] = (MAT(b, 1, 1) * MAT(b, 2, 2) - MAT(b, 1, 2) * MAT(b, 2, 1)) / vol;
#pragma unroll
    for (int k = 0; k < 9; ++k) { B.th_tgid[k] = tgid[k]; B.th_cof[k] = d[k]; }
}

// The box algebra of k_finalize_force, by one thread on the block's shared
// copy of the box: sr holds the 15 reduced sums (embedding energy, pair
// count; pair energy, virial moments; kinetic moments).
static __device__ void finalize_box(const Params &p, BoxState &B, const double *sr, int mode, bool prep = true) {
    const double *se = sr, *sf = sr + 2, *sk = sr + 9;
    // the box algebra runs on register copies and is stored once at the end
    double b0[9], b1[9], b2[9], tp[9], tk[9], tc[9], tg[9], tgdot[9], fb[9];
#pragma unroll
    for (int k = 0; k < 9; ++k) { b0[k] = B.b0[k]; b1[k] = B.b1[k]; b2[k] = B.b2[k]; }
    B.pe_emb = se[0];
    B.pe_pair = sf[0];
    B.pe = se[0] + sf[0];
    B.npairs = se[1];
    // symmetric moments (xx, yy, zz, xy, xz, yz) -> full 3x3
    double M[9], D[9];
    M[0] = sk[0]; M[4] = sk[1]; M[8] = sk[2]; M[3] = M[1] = sk[3]; M[6] = M[2] = sk[4]; M[7] = M[5] = sk[5];
    D[0] = sf[1]; D[4] = sf[2]; D[8] = sf[3]; D[3] = D[1] = sf[4]; D[6] = D[2] = sf[5]; D[7] = D[5] = sf[6];
    double dt2 = p.deltat * p.deltat;
    mat_mul(b0, D, tp);                           // tp(a,b) = sum r_a d_b fp, r = B0 d
    mat_mul(b0, M, tk);                           // tk(a,b) = sum m (B0 x1)_a x1_b
#pragma unroll
    for (int k = 0; k < 9; ++k) tk[k] = tk[k] / dt2;
    mat_cofactor(b0, tc);
#pragma unroll
    for (int k = 0; k < 9; ++k) { tgdot[k] = 0.0; tg[k] = 0.0; }
#pragma unroll
    for (int i = 1; i <= 3; ++i)
#pragma unroll
        for (int k = 1; k <= 3; ++k)
#pragma unroll
            for (int j = 1; j <= 3; ++j) {
                MAT(tg, i, j) = MAT(tg, i, j) + MAT(b0, k, i) * MAT(b0, k, j);
                MAT(tgdot, i, j) = MAT(tgdot, i, j) + MAT(b0, k, i) * MAT(b1, k, j) + MAT(b1, k, i) * MAT(b0, k, j);
            }
    const double vol = mat_volume(b0);
#pragma unroll
    for (int k = 0; k < 9; ++k) fb[k] = tk[k] + tp[k] - p.press * tc[k];
#pragma unroll
    for (int k = 0; k < 9; ++k) {
        B.tp[k] = tp[k]; B.tk[k] = tk[k]; B.tc[k] = tc[k]; B.tg[k] = tg[k]; B.tgdot[k] = tgdot[k]; B.fb[k] = fb[k];
    }
    B.vol = vol;
    if (mode == 1) {
        if (p.ivol < 1) {
#pragma unroll
            for (int k = 0; k < 9; ++k) b2[k] = p.bdel2 * fb[k];
#pragma unroll
            for (int k = 0; k < 9; ++k) b1[k] = b1[k] + b2[k];
        }
        if (p.ivol == 4) {
            MAT(b2, 3, 3) = p.bdel2 * MAT(fb, 3, 3);
#pragma unroll
            for (int k = 0; k < 9; ++k) b1[k] = b1[k] + b2[k];
        }
    } else if (mode == 2) {
        double tginv[9], tgid[9];
        if (!mat_invert(tg, tginv)) { B.status = MOLDY_ERR_SINGULAR_BOX; return; }
        mat_mul(tginv, tgdot, tgid);
#pragma unroll
        for (int k = 0; k < 9; ++k) { B.tginv[k] = tginv[k]; B.tgid[k] = tgid[k]; b2[k] = p.bdel2 * fb[k]; }
    }
#pragma unroll
    for (int k = 0; k < 9; ++k) { B.b1[k] = b1[k]; B.b2[k] = b2[k]; }
    if (prep) therm_prep(p, b0, b1, B);       // for the update_therm_avs that follows
}

// update_therm_avs (src/dynamics_m.F90:649-734), one atom's terms: s1 += |F|^2,
// s2 += |F|^4, s3 += m |B0 x1|^2, with F = cof(B0)/vol (2 x2 + tgid x1); t, b, d
// are tgid, B0 and cof(B0)/vol in shared memory, read at every use (volatile)
// rather than held in 54 registers across the atom loop, which would halve the
// resident warps of the streaming kernels that call this.  The caller skips
// atoms without a species.
__device__ __forceinline__ void therm_terms(double (&v)[3], const volatile double *t, const volatile double *b,
                                            const volatile double *d,
                                            double ma, double ux, double uy, double uz, double wx, double wy,
                                            double wz) {
    double sxi = t[0] * ux + t[3] * uy + t[6] * uz;
    double syi = t[1] * ux + t[4] * uy + t[7] * uz;
    double szi = t[2] * ux + t[5] * uy + t[8] * uz;
    double fxp = 2.0 * wx + sxi, fyp = 2.0 * wy + syi, fzp = 2.0 * wz + szi;
    double fx = d[0] * fxp + d[1] * fyp + d[2] * fzp;
    double fy = d[3] * fxp + d[4] * fyp + d[5] * fzp;
    double fz = d[6] * fxp + d[7] * fyp + d[8] * fzp;
    double f2 = fx * fx + fy * fy + fz * fz;
    v[0] += f2;
    v[1] += f2 * f2;
    double rx = b[0] * ux + b[3] * uy + b[6] * uz;
    double ry = b[1] * ux + b[4] * uy + b[7] * uz;
    double rz = b[2] * ux + b[5] * uy + b[8] * uz;
    v[2] += ma * (rx * rx + ry * ry + rz * rz);
}

// The mdloop quantities (src/moldin.F90:760-790) from the three sums of
// update_therm_avs (s3 = s1, s2, s3), by one thread.  The box has not moved
// since the force evaluation that ended the step.
// rec (may be null): the step's thermo record, kThermoRec doubles in the order
// of moldy_thermo (ke, pe, te, h, th, vol, s1, s2, s3, temp, boxke)
static __device__ void therm_store(const Params &p, BoxState &B, const double *s3, double *rec) {
    double b0[9], b1[9], tg[9], tgdot[9], tginv[9], tgid[9], vol;
#pragma unroll
    for (int k = 0; k < 9; ++k) { b0[k] = B.b0[k]; b1[k] = B.b1[k]; }
    if (!therm_box(p, b0, b1, tg, tgdot, tginv, tgid, vol)) B.status = MOLDY_ERR_SINGULAR_BOX;
#pragma unroll
    for (int k = 0; k < 9; ++k) { B.tg[k] = tg[k]; B.tgdot[k] = tgdot[k]; B.tginv[k] = tginv[k]; B.tgid[k] = tgid[k]; }
    B.vol = vol;
    B.s1 = s3[0]; B.s2 = s3[1]; B.s3 = s3[2];
    const double bk = 1.3806504e-23 / 1.602176487e-19;
    B.ke = s3[2] / (p.deltat * p.deltat) / 2.0;
    B.temp = B.ke / (1.5 * bk * (double)p.nm);
    double boxke = 0.0;
    for (int i = 1; i <= 3; ++i)
        for (int j = 1; j <= 3; ++j) boxke = boxke + (MAT(b1, i, j) * MAT(b1, i, j)) / p.bdel2;
    B.boxke = boxke;
    B.te = B.ke + B.pe;
    B.h = B.te + p.press * B.vol;
    B.th = B.h + boxke;
    if (rec) {
        rec[0] = B.ke; rec[1] = B.pe; rec[2] = B.te; rec[3] = B.h; rec[4] = B.th; rec[5] = B.vol;
        rec[6] = B.s1; rec[7] = B.s2; rec[8] = B.s3; rec[9] = B.temp; rec[10] = B.boxke;
    }
}

// The list-rebuild decisions and the box advance of k_mid_decide, by one
// thread on the block's shared copy of the box.
static __device__ void mid_decide_box(const Params &p, BoxState &B, double rmid, double rcut, double rout, int force,
                               int half_build, int apply_box) {
    // register copies; the box is stored back once
    double b0[9], b1[9], b2[9], bb[9];
#pragma unroll
    for (int k = 0; k < 9; ++k) { b0[k] = B.b0[k]; b1[k] = B.b1[k]; b2[k] = B.b2[k]; bb[k] = B.bbuild[k]; }
    if (apply_box) {   // velocityverlet box half (src/quench_m.F90:582-589)
        if (p.ivol == 4) {
            MAT(b1, 3, 3) = MAT(b1, 3, 3) + MAT(b2, 3, 3);
            MAT(b0, 3, 3) = MAT(b0, 3, 3) + MAT(b1, 3, 3);
        }
        if (p.ivol < 1) {
#pragma unroll
            for (int k = 0; k < 9; ++k) b1[k] = b1[k] + b2[k];
#pragma unroll
            for (int k = 0; k < 9; ++k) b0[k] = b0[k] + b1[k];
        }
#pragma unroll
        for (int k = 0; k < 9; ++k) { B.b0[k] = b0[k]; B.b1[k] = b1[k]; }
    }
    // displacements are measured in FP32 from fixed-point positions: the
    // factor and the offset cover their rounding
    double md = sqrt(__longlong_as_double((long long)B.maxdisp2)) * (1.0 + 1.0e-5) + 1.0e-6;
    B.maxdisp2 = 0ull;
    double eps = 2.0e-6 * frob(b0) + 1.0e-4;
    // dmax = rnear |B_build^-1|_F bounds the fractional separation of a listed
    // pair; it is stored with each build (0: none yet, or a singular box)
    double db[9];
#pragma unroll
    for (int k = 0; k < 9; ++k) db[k] = b0[k] - bb[k];
    const double dmax = B.dmax_mid;
    double shrink = 2.0 * md + frob(db) * dmax;
    // A half-list rebuild this step (half_build) keeps the outer and
    // intermediate lists when the outer list needs no pair that its own
    // source half list lacked.  A pair missing from that source was farther
    // than rnear at the source's build; at the outer build it was farther
    // than rnear - eps - shrink_h (shrink_h: twice the largest displacement
    // between the two builds, measured by the outer build, plus the box
    // change times the source's dmax).  When that is beyond r_out + eps the
    // pair was left out of the outer list like any pair beyond r_out, and the
    // outer list's own rule below bounds its approach from then on.
    bool keep_lists = false;
    if (half_build) {
        double dbh[9];
#pragma unroll
        for (int k = 0; k < 9; ++k) dbh[k] = B.bout[k] - B.bhalf_out[k];
        const double dh = sqrt(__longlong_as_double((long long)B.halfdisp2)) * (1.0 + 1.0e-5) + 1.0e-6;
        const double shrink_h = 2.0 * dh + frob(dbh) * B.dmax_half_out;
        keep_lists = B.dmax_half_out > 0.0 && B.dmax_out > 0.0 && B.dmax_mid > 0.0 &&
                     shrink_h < p.rnear - eps - (rout + eps);
        double hinv[9];
        const double dh_new = mat_invert(b0, hinv) ? p.rnear * frob(hinv) : 0.0;
#pragma unroll
        for (int k = 0; k < 9; ++k) B.bhalf[k] = b0[k];
        B.dmax_half = dh_new;
    }
    const int forced = force || (half_build && !keep_lists);
    int need = forced || !(dmax > 0.0) || !(shrink < rmid - eps - (rcut + eps));
    int need_out = 0;
    if (need) {
        // The intermediate list is filtered from the outer list, which must
        // then hold every pair within r_mid: a pair left out of it was farther
        // than r_out - eps at its build, and each atom has moved since then by
        // at most its displacement at the last intermediate build (outdisp2)
        // plus its displacement since (md).
        double dbo[9];
#pragma unroll
        for (int k = 0; k < 9; ++k) dbo[k] = b0[k] - B.bout[k];
        const double dmaxo = B.dmax_out;
        const double dout = sqrt(__longlong_as_double((long long)B.outdisp2)) * (1.0 + 1.0e-5) + 1.0e-6 + md;
        const double shrink_out = 2.0 * dout + frob(dbo) * dmaxo;
        need_out = forced || !(dmaxo > 0.0) || !(shrink_out < rout - eps - (rmid + 2.0 * eps));
        double inv[9];
        const double dnew = mat_invert(b0, inv) ? p.rnear * frob(inv) : 0.0;
#pragma unroll
        for (int k = 0; k < 9; ++k) B.bbuild[k] = b0[k];
        B.dmax_mid = dnew;
        B.mid_builds += 1;
        B.outdisp2 = 0ull;   // measured again by the intermediate build
        if (need_out) {
            // the half list this outer list is filtered from, and the
            // displacement since that half list's build (measured by the build)
#pragma unroll
            for (int k = 0; k < 9; ++k) B.bhalf_out[k] = B.bhalf[k];
            B.dmax_half_out = B.dmax_half;
            B.halfdisp2 = 0ull;
#pragma unroll
            for (int k = 0; k < 9; ++k) B.bout[k] = b0[k];
            B.dmax_out = dnew;
            B.out_builds += 1;
        }
    }
    B.mid_rebuild = need;
    B.out_rebuild = need_out;
}

}  // namespace moldy
