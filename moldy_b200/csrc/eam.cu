// eam.cu -- box algebra, the velocity-Verlet / Parrinello-Rahman update, the
// thermodynamic sums and energy_calc (dynamics_m, thermostat_m::kinten,
// quench_m::velocityverlet).  The pair passes are in pairs.cu.
#include "engine.h"
#include "box.cuh"

namespace moldy {

int stream_blocks(int nm) {
    static const int sms = [] {
        int dev = 0, n = 0;
        cudaGetDevice(&dev);
        cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev);
        return n > 0 ? n : 148;
    }();
    const int nb = grid_blocks(nm, kAtomThreads);
    return nb < 4 * sms ? nb : 4 * sms;
}

// mode 0: force only; 1: velocity Verlet second half (box); 2: md_init
__global__ void __launch_bounds__(256)
k_finalize_force(Params p, BoxState *__restrict__ box, const double *__restrict__ part_embed,
                 int nblk_embed, const double *__restrict__ part_force, int nblk_force,
                 const double *__restrict__ part_kin, int nblk_kin, int mode) {
    grid_dep_wait();   // launched dependent on the step's previous kernel
    // the box in shared memory, loaded while the partials are summed
    __shared__ BoxState sbox;
    box_load(sbox, box);
    // the three sets of block partials in one pass: each thread issues the
    // loads of all three before adding (per set, the same order as
    // reduce_partials)
    __shared__ double sm[8][15], sr[15];
    double acc[15];
#pragma unroll
    for (int k = 0; k < 15; ++k) acc[k] = 0.0;
    const int nmax = max(nblk_embed, max(nblk_force, nblk_kin));
    for (int b = threadIdx.x; b < nmax; b += blockDim.x) {
        double e[15];
#pragma unroll
        for (int k = 0; k < 2; ++k) e[k] = b < nblk_embed ? part_embed[(size_t)b * kPartials + k] : 0.0;
#pragma unroll
        for (int k = 0; k < 7; ++k) e[2 + k] = b < nblk_force ? part_force[(size_t)b * kPartials + k] : 0.0;
#pragma unroll
        for (int k = 0; k < 6; ++k) e[9 + k] = b < nblk_kin ? part_kin[(size_t)b * kPartials + k] : 0.0;
#pragma unroll
        for (int k = 0; k < 15; ++k) acc[k] += e[k];
    }
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
    for (int k = 0; k < 15; ++k) {
        const double w = warp_sum(acc[k]);
        if (lane == 0) sm[warp][k] = w;
    }
    __syncthreads();
    if (warp == 0 && lane < 15) {
        double w = 0.0;
        for (int q = 0; q < (int)(blockDim.x >> 5); ++q) w += sm[q][lane];
        sr[lane] = w;
    }
    __syncthreads();
    __syncthreads();
    if (threadIdx.x == 0) finalize_box(p, sbox, sr, mode);
    __syncthreads();
    box_store(box, sbox);
}

void launch_finalize_force(DeviceState &d, const Params &p, const double *part_embed, int nblk_embed,
                           const double *part_force, int nblk_force, const double *part_kin, int nblk_kin,
                           int mode, cudaStream_t s) {
    launch_pdl(k_finalize_force, 1, 256, 0, s, p, d.box, part_embed, nblk_embed, part_force, nblk_force, part_kin, nblk_kin,
                                        mode);
}

__global__ void __launch_bounds__(256)
k_kinetic(Params p, const double *__restrict__ x1, const double *__restrict__ mass,
          const int32_t *__restrict__ znum, double *__restrict__ partials) {
    double v[6] = {0.0, 0.0, 0.0, 0.0, 0.0, 0.0};
    const int nm = p.nm;
    for (int a = blockIdx.x * blockDim.x + threadIdx.x; a < nm; a += gridDim.x * blockDim.x)
        if (znum[a] != 0) kin_moment(v, mass[a], x1[a], x1[nm + a], x1[2 * nm + a]);
    block_partials<6>(v, partials, 0);
}

int launch_kinetic(DeviceState &d, const Params &p, double *partials, cudaStream_t s) {
    int nb = stream_blocks(p.nm);
    k_kinetic<<<nb, kAtomThreads, 0, s>>>(p, d.x1, d.mass, d.znum, partials);
    return nb;
}

__global__ void k_therm_prep(Params p, BoxState *__restrict__ box) {
    double b0[9], b1[9];
    for (int k = 0; k < 9; ++k) { b0[k] = box->b0[k]; b1[k] = box->b1[k]; }
    therm_prep(p, b0, b1, *box);
}

// ------------------------------------------------ intermediate-list check --
// therm_nblk > 0: first finish the update_therm_avs that the drift kernel
// took for the step that has just ended (its block partials), before the box
// moves.
__global__ void __launch_bounds__(256)
k_mid_decide(Params p, BoxState *__restrict__ box, double rmid, double rcut, double rout, int force,
             int half_build, int apply_box, const double *__restrict__ therm_partials, int therm_nblk,
             double *__restrict__ rec, int rec_indexed) {
    grid_dep_wait();   // launched dependent on the step's previous kernel
    __shared__ BoxState sbox;
    box_load(sbox, box);
    __syncthreads();
    if (therm_nblk > 0) {
        __shared__ double s3[3];
        reduce_partials<3>(therm_partials, therm_nblk, s3);
        if (threadIdx.x == 0) {
            // rec_indexed: rec is the first record, and the box says which one
            // this step writes (a replayed step's launches are all alike)
            double *r = rec;
            if (rec_indexed) {
                if (r) r += (size_t)kThermoRec * (size_t)sbox.rec_step;
                sbox.rec_step += 1;
            }
            therm_store(p, sbox, s3, r);
        }
    }
    if (threadIdx.x == 0) mid_decide_box(p, sbox, rmid, rcut, rout, force, half_build, apply_box);
    __syncthreads();
    box_store(box, sbox);
}

void launch_mid_decide(DeviceState &d, const Params &p, double rmid, double rcut, double rout, int force,
                       int half_build, int apply_box, int therm_nblk, double *rec, cudaStream_t s,
                       int rec_indexed) {
    launch_pdl(k_mid_decide, 1, 256, 0, s, p, d.box, rmid, rcut, rout, force, half_build, apply_box, d.partials,
                                   therm_nblk, rec, rec_indexed);
}

__global__ void k_set_rec_step(BoxState *__restrict__ box, int step) { box->rec_step = step; }

// the record index the next indexed k_mid_decide writes
void launch_set_rec_step(DeviceState &d, int step, cudaStream_t s) { k_set_rec_step<<<1, 1, 0, s>>>(d.box, step); }

// ------------------------------------------------------------- integrator --
// velocityverlet first half (src/quench_m.F90:574-589): x1_dt2 = x1 + x2;
// x0 += x1_dt2.  The box half (b1 += b2; b0 += b1 for ivol < 1, zz only for
// ivol 4) is applied by k_mid_decide, which runs next.
//
// THERM: the update_therm_avs of the previous step is taken here too.  x1 and
// x2 are read unchanged from the force evaluation that ended that step, the
// box has not yet moved, and the grid is k_therm's, so the sums are k_therm's
// to the last bit.  The block partials go to therm_partials; k_mid_decide,
// which runs next, finishes them.
//
// SCALE: the scalev that ended the previous step left its mean and scaling in
// the box; x1 = (x1 - mean) (1 + snhv) of the movable atoms is formed and stored
// here, as k_scalev_scale would have.
template <bool THERM, bool SCALE>
__global__ void __launch_bounds__(256, 4)   // the grid is 4 blocks per SM (stream_blocks): one wave
k_drift(Params p, double4 *__restrict__ pos, int4 *__restrict__ posq,
        double *__restrict__ x1, const double *__restrict__ x2, BoxState *__restrict__ box,
        const int4 *__restrict__ xbuild, const double *__restrict__ mass, const int32_t *__restrict__ znum,
        double *__restrict__ kin_partials, double *__restrict__ therm_partials) {
    grid_dep_wait();   // launched dependent on the step's previous kernel
    // every thread forms the post-drift box exactly as thread 0 stores it
    __shared__ float nbs[9];   // that box per fixed-point unit
    __shared__ double sh[THERM ? 27 : 1];   // tgid, b0, cof(b0)/vol of the previous step
    if (THERM && threadIdx.x < 9) {
        sh[threadIdx.x] = box->th_tgid[threadIdx.x];
        sh[9 + threadIdx.x] = box->b0[threadIdx.x];
        sh[18 + threadIdx.x] = box->th_cof[threadIdx.x];
    }
    __shared__ double scale[SCALE ? 4 : 1];
    if (SCALE && threadIdx.x >= 32 && threadIdx.x < 36)
        scale[threadIdx.x - 32] = threadIdx.x < 35 ? box->sc_mean[threadIdx.x - 32] : 1.0 + box->snhv;
    if (threadIdx.x == 0) {
        const BoxState &B = *box;
        double b1[9], b0[9];
        for (int k = 0; k < 9; ++k) { b1[k] = B.b1[k]; b0[k] = B.b0[k]; }
        if (p.ivol == 4) {
            MAT(b1, 3, 3) = MAT(b1, 3, 3) + MAT(B.b2, 3, 3);
            MAT(b0, 3, 3) = MAT(b0, 3, 3) + MAT(b1, 3, 3);
        }
        if (p.ivol < 1) {
            for (int k = 0; k < 9; ++k) b1[k] = b1[k] + B.b2[k];
            for (int k = 0; k < 9; ++k) b0[k] = b0[k] + b1[k];
        }
        for (int k = 0; k < 9; ++k) nbs[k] = (float)(b0[k] * kFixUnit);
    }
    __syncthreads();
    float d2 = 0.f;
    double v[6] = {0.0, 0.0, 0.0, 0.0, 0.0, 0.0};
    double vt[3] = {0.0, 0.0, 0.0};
    const int nm = p.nm;
    for (int a = blockIdx.x * blockDim.x + threadIdx.x; a < nm; a += gridDim.x * blockDim.x) {
        double ex = x1[a], ey = x1[nm + a], ez = x1[2 * nm + a];
        const double wx = x2[a], wy = x2[nm + a], wz = x2[2 * nm + a];
        double4 q = pos[a];
        if (SCALE && !(znum[a] == 0 || mass[a] < 0.1)) {
            ex = (ex - scale[0]) * scale[3]; ey = (ey - scale[1]) * scale[3]; ez = (ez - scale[2]) * scale[3];
            x1[a] = ex; x1[nm + a] = ey; x1[2 * nm + a] = ez;
        }
        q.x = q.x + (ex + wx);
        q.y = q.y + (ey + wy);
        q.z = q.z + (ez + wz);
        pos[a] = q;
        const int4 qn = make_int4(fix32(q.x), fix32(q.y), fix32(q.z), 0);
        posq[a] = qn;
        d2 = fmaxf(d2, fix_disp2(nbs, qn, xbuild[a]));
        // x1 is not changed by this half of the step: the kinetic moment of
        // the coming force evaluation can be taken here
        if (znum[a] != 0) {
            const double ma = mass[a];
            kin_moment(v, ma, ex, ey, ez);
            if (THERM) therm_terms(vt, sh, sh + 9, sh + 18, ma, ex, ey, ez, wx, wy, wz);
        }
    }
    block_partials<6>(v, kin_partials, 0);
    // block maximum, then one atomic per block (non-negative doubles order as their bits)
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) d2 = fmaxf(d2, __shfl_xor_sync(0xffffffffu, d2, o));
    __shared__ float wmax[8];
    if ((threadIdx.x & 31) == 0) wmax[threadIdx.x >> 5] = d2;
    __syncthreads();
    if (threadIdx.x == 0) {
        float m = 0.f;
        for (int w = 0; w < (int)(blockDim.x >> 5); ++w) m = fmaxf(m, wmax[w]);
        atomicMax(&box->maxdisp2, (unsigned long long)__double_as_longlong((double)m));
    }
    // the sums are finished by k_mid_decide, which runs next
    if (THERM) block_partials<3>(vt, therm_partials, 0);
    // the box itself is advanced afterwards by k_mid_decide, so that no block
    // here can read a box another block has already moved
}

int launch_drift(DeviceState &d, const Params &p, double *kin_partials, bool therm, cudaStream_t s, bool scale) {
    int nb = stream_blocks(p.nm);
    // a step that scalev ended has taken its thermo sums already
    auto k = therm ? k_drift<true, false> : (scale ? k_drift<false, true> : k_drift<false, false>);
    launch_pdl(k, nb, kAtomThreads, 0, s, p, d.pos, d.posq, d.x1, d.x2, d.box, d.xbuild, d.mass, d.znum, kin_partials,
               therm ? d.partials : nullptr);
    return nb;
}

// moldin strain-loop preparation (src/moldin.F90:458-471): every atom with a
// species, x2 = del2 f - tgid x1 / 2
__global__ void k_md_init_x2(Params p, const BoxState *__restrict__ box, const double *__restrict__ f,
                             const double *__restrict__ x1, double *__restrict__ x2,
                             const double *__restrict__ del2) {
    const int a = blockIdx.x * blockDim.x + threadIdx.x;
    if (a >= p.nm) return;
    const double *t = box->tgid;
    const int nm = p.nm;
    double ux = x1[a], uy = x1[nm + a], uz = x1[2 * nm + a];
    double a1 = t[0] * ux + t[3] * uy + t[6] * uz;
    double a2 = t[1] * ux + t[4] * uy + t[7] * uz;
    double a3 = t[2] * ux + t[5] * uy + t[8] * uz;
    double d2 = del2[a];
    x2[a] = d2 * f[a] - 0.5 * a1;
    x2[nm + a] = d2 * f[nm + a] - 0.5 * a2;
    x2[2 * nm + a] = d2 * f[2 * nm + a] - 0.5 * a3;
}

void launch_md_init_x2(DeviceState &d, const Params &p, cudaStream_t s) {
    int nb = (p.nm + kAtomThreads - 1) / kAtomThreads;
    k_md_init_x2<<<nb, kAtomThreads, 0, s>>>(p, d.box, d.f, d.x1, d.x2, d.del2);
}

// update_therm_avs over the atoms with a species, after a force evaluation
// (therm_prep has left tgid and cof(B0)/vol in the box state).  MEAN: also the
// mean of x1 over all atoms, for the scalev that follows.  The last block to
// finish sums the block partials in order and stores what follows from them.
template <bool MEAN>
__global__ void __launch_bounds__(256, 4)
k_therm(Params p, BoxState *__restrict__ box, const double *__restrict__ x1,
        const double *__restrict__ x2, const double *__restrict__ mass,
        const int32_t *__restrict__ znum, double *__restrict__ partials, double *__restrict__ rec,
        int32_t *__restrict__ ticket) {
    grid_dep_wait();   // launched dependent on the step's previous kernel
    __shared__ double sh[9 + 9 + 9];   // tgid, b0, cof(b0)/vol
    if (threadIdx.x < 9) {
        sh[threadIdx.x] = box->th_tgid[threadIdx.x];
        sh[9 + threadIdx.x] = box->b0[threadIdx.x];
        sh[18 + threadIdx.x] = box->th_cof[threadIdx.x];
    }
    __syncthreads();
    double v[3] = {0.0, 0.0, 0.0}, m[3] = {0.0, 0.0, 0.0};
    const int nm = p.nm;
    for (int a = blockIdx.x * blockDim.x + threadIdx.x; a < nm; a += gridDim.x * blockDim.x) {
        // every load issued before the species test, so none waits on it
        const int z = znum[a];
        const double ux = x1[a], uy = x1[nm + a], uz = x1[2 * nm + a];
        const double wx = x2[a], wy = x2[nm + a], wz = x2[2 * nm + a];
        const double ma = mass[a];
        if (MEAN) { m[0] += ux; m[1] += uy; m[2] += uz; }
        if (z == 0) continue;
        therm_terms(v, sh, sh + 9, sh + 18, ma, ux, uy, uz, wx, wy, wz);
    }
    block_partials<3>(v, partials, 0);
    if (MEAN) block_partials<3>(m, partials, 3);
    if (!last_block(ticket)) return;
    __shared__ double s3[MEAN ? 6 : 3];
    reduce_partials<MEAN ? 6 : 3, true>(partials, gridDim.x, s3);
    if (threadIdx.x == 0) {
        therm_store(p, *box, s3, rec);
        if (MEAN)
            for (int k = 0; k < 3; ++k) box->sc_mean[k] = s3[3 + k] / (double)(float)nm;   // float(nm): default REAL
    }
}

// prep: compute the box quantities first (the call does not follow a force
// evaluation that left them); mean: for a scalev that follows
int launch_therm(DeviceState &d, const Params &p, bool prep, double *rec, cudaStream_t s, bool mean) {
    if (prep) k_therm_prep<<<1, 1, 0, s>>>(p, d.box);
    // with the mean, scalev's grouping of the atoms (launch_scalev)
    int nblocks = mean ? grid_blocks(p.nm, kAtomThreads) : stream_blocks(p.nm);
    launch_pdl(mean ? k_therm<true> : k_therm<false>, nblocks, kAtomThreads, 0, s, p, d.box, d.x1, d.x2, d.mass, d.znum,
               d.partials, rec, d.flags + 14);
    return nblocks;
}

// ----------------------------------------------------------------- scalev --
// scalev (src/thermostat_m.F90:317-395), the Nose-Hoover Euler thermostat:
// remove the mean of x1 (over all atoms) from the movable atoms, measure their
// kinetic energy, update snhv -= (ke - rqke) / (nose nm) and scale their x1
// by 1 + snhv.  Atoms with Z = 0 or mass < 0.1 are not movable.
//
// In an MD step the mean comes with the thermo sums (k_therm), k_scalev_ke
// measures the energy without writing x1, its last block updates snhv, and the
// next step's drift, which streams x1 anyway, removes the mean and scales: two
// passes over x1 and three launches fewer than mean, removal, finish and
// scaling one after the other (1,024,000 atoms: 84 us per step with the thermo
// sums, of which 35 us for every block of the removal pass summing 1,184
// blocks' partials).
__global__ void __launch_bounds__(256, 4)
k_scalev_mean(int nm, BoxState *__restrict__ box, const double *__restrict__ x1, double *__restrict__ partials,
              int32_t *__restrict__ ticket) {
    double v[3] = {0.0, 0.0, 0.0};
    for (int a = blockIdx.x * blockDim.x + threadIdx.x; a < nm; a += gridDim.x * blockDim.x) {
        v[0] += x1[a]; v[1] += x1[nm + a]; v[2] += x1[2 * nm + a];
    }
    block_partials<3>(v, partials, 0);
    if (!last_block(ticket)) return;
    __shared__ double s[3];
    reduce_partials<3, true>(partials, gridDim.x, s);
    if (threadIdx.x < 3) box->sc_mean[threadIdx.x] = s[threadIdx.x] / (double)(float)nm;
}

__global__ void __launch_bounds__(256, 4)
k_scalev_ke(Params p, BoxState *__restrict__ box, const double *__restrict__ x1, const double *__restrict__ mass,
            const int32_t *__restrict__ znum, double *__restrict__ partials, double nose, double rqke,
            int32_t *__restrict__ ticket) {
    grid_dep_wait();   // launched dependent on the step's previous kernel
    __shared__ double sh[12];   // B0, the mean
    if (threadIdx.x < 9) sh[threadIdx.x] = box->b0[threadIdx.x];
    else if (threadIdx.x < 12) sh[threadIdx.x] = box->sc_mean[threadIdx.x - 9];
    __syncthreads();
    const int nm = p.nm;
    const double *b = sh;
    const double sx = sh[9], sy = sh[10], sz = sh[11];
    double v[1] = {0.0};
    for (int a = blockIdx.x * blockDim.x + threadIdx.x; a < nm; a += gridDim.x * blockDim.x) {
        const int z = znum[a];
        const double ma = mass[a];
        const double ux = x1[a] - sx, uy = x1[nm + a] - sy, uz = x1[2 * nm + a] - sz;
        if (z == 0 || ma < 0.1) continue;
        const double rx = b[0] * ux + b[3] * uy + b[6] * uz;
        const double ry = b[1] * ux + b[4] * uy + b[7] * uz;
        const double rz = b[2] * ux + b[5] * uy + b[8] * uz;
        v[0] += ma * (rx * rx + ry * ry + rz * rz);
    }
    block_partials<1>(v, partials, 0);
    if (!last_block(ticket)) return;
    __shared__ double s[1];
    reduce_partials<1, true>(partials, gridDim.x, s);
    if (threadIdx.x != 0) return;
    BoxState &B = *box;
    double ke = s[0] / (p.deltat * p.deltat) / 2.0;
    // snhf keeps its previous value when ke is not positive
    if (ke > 0.0) B.snhf = (ke - rqke) / (nose * (double)p.nm);
    B.snhv = B.snhv - B.snhf;
    B.scalev_ke = ke;
}

__global__ void __launch_bounds__(256)
k_scalev_scale(int nm, const BoxState *__restrict__ box, double *__restrict__ x1, const double *__restrict__ mass,
               const int32_t *__restrict__ znum) {
    const double f = 1.0 + box->snhv, sx = box->sc_mean[0], sy = box->sc_mean[1], sz = box->sc_mean[2];
    for (int a = blockIdx.x * blockDim.x + threadIdx.x; a < nm; a += gridDim.x * blockDim.x) {
        if (znum[a] == 0 || mass[a] < 0.1) continue;
        x1[a] = (x1[a] - sx) * f;
        x1[nm + a] = (x1[nm + a] - sy) * f;
        x1[2 * nm + a] = (x1[2 * nm + a] - sz) * f;
    }
}

// mean: the mean is not in the box yet; scale: scale x1 now (else the next
// drift does)
void launch_scalev(DeviceState &d, const Params &p, double nose, double rqke, bool mean, bool scale, cudaStream_t s) {
    // Mean and energy are summed over up to 1,184 blocks, as they were as passes
    // of their own: the scaling factor multiplies every velocity, so another
    // order of these sums (592 blocks, 7 us a step less at 1,024,000 atoms) would
    // move every trajectory of a thermostatted run by its last bits.
    const int nb = grid_blocks(p.nm, kAtomThreads);
    double *part = d.partials + (size_t)kMaxBlocks * kPartials;
    if (mean) k_scalev_mean<<<nb, kAtomThreads, 0, s>>>(p.nm, d.box, d.x1, part, d.flags + 15);
    launch_pdl(k_scalev_ke, nb, kAtomThreads, 0, s, p, d.box, d.x1, d.mass, d.znum, part, nose, rqke, d.flags + 15);
    if (scale) k_scalev_scale<<<nb, kAtomThreads, 0, s>>>(p.nm, d.box, d.x1, d.mass, d.znum);
}

// ------------------------------------------------------------ energy_calc --
// src/dynamics_m.F90:412-483: en_atom = F(rho) + half of each exact pair term
__global__ void __launch_bounds__(256)
k_energy_pairs(Params p, Tables t, const double4 *__restrict__ pos, const BoxState *__restrict__ box,
               const int32_t *__restrict__ nlist, const int32_t *__restrict__ numn,
               double *__restrict__ en) {
    __shared__ double sb[9];
    if (threadIdx.x < 9) sb[threadIdx.x] = box->b0[threadIdx.x];
    __syncthreads();
    const int a = blockIdx.x * blockDim.x + threadIdx.x;
    if (a >= p.nm) return;
    const double4 pa = pos[a];
    const int n = numn[a];
    double own = 0.0;
    for (int k = 0; k < n; ++k) {
        int j = nlist[(size_t)a * p.nnbrs + k];
        double4 pj = pos[j];
        double dx = pa.x - pj.x, dy = pa.y - pj.y, dz = pa.z - pj.z;
        min_image(p.ivol, dx, dy, dz);
        double rx = sb[0] * dx + sb[3] * dy + sb[6] * dz;
        double ry = sb[1] * dx + sb[4] * dy + sb[7] * dz;
        double rz = sb[2] * dx + sb[5] * dy + sb[8] * dz;
        double r = sqrt(rx * rx + ry * ry + rz * rz);
        double pp = fetm_vee(t, r) / 2.0;
        if (pp != 0.0) {
            own += pp;
            atomicAdd(&en[j], pp);
        }
    }
    atomicAdd(&en[a], own);
}

void launch_energy_calc(DeviceState &d, const Params &p, const Tables &t, cudaStream_t s) {
    cudaMemcpyAsync(d.en_atom, d.afrho, sizeof(double) * p.nm, cudaMemcpyDeviceToDevice, s);
    int nb = (p.nm + kAtomThreads - 1) / kAtomThreads;
    k_energy_pairs<<<nb, kAtomThreads, 0, s>>>(p, t, d.pos, d.box, d.nlist, d.numn, d.en_atom);
}

}  // namespace moldy
