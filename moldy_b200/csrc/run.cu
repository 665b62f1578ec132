// run.cu -- runs of velocity-Verlet steps of one small system in one launch.
//
// A step is a chain of small dependent pieces: drift, box and list decision,
// density, forces, box half-kick.  Launched one after the other (seven
// launches) a step of a 2,000-atom system takes 52 us, nearly all of it
// launch, prologue and tail latency.  k_run keeps one resident grid (a
// cooperative launch, at most one block per SM) for a whole run of ordinary
// steps and separates its pieces by grid barriers, two per step:
//
//   A  (positions of step s published)   every block reduces the partial sums
//      of step s - 1 and advances its own shared-memory copy of the box
//      (bit-identical in every block), decides the list builds, builds the
//      rows of its atoms, and takes rho, F and F' of its atoms
//   B  (F' of step s published)          forces, the second half-kick, and the
//      first half-kick and drift of step s + 1
//
// The update_therm_avs of the run's last step is piece A's of the run that
// follows at once, else a launch of its own (k_run_therm).
//
// L lanes of a warp share one atom's rows, so that a row of 14 to 20 entries
// is one or two rounds of independent gathers instead of a serial walk; rows
// are written in the order one lane would write them (a ballot places each
// kept entry).  The lookup tables sit in shared memory: every barrier drops
// what L1 holds, and the tables would be fetched again in each piece.
//
// The partial sums are double buffered by the parity of the step, since a
// block past a barrier may already write the next step's while another still
// reads; positions, F' records and rows are each written in one piece and
// read in the other, or only by their own block.
//
// Sums over an atom's pairs are grouped by lane and partial sums by block, in
// a fixed order, so a run gives the same bits every time.  A run may be cut
// into launches of single pieces (h0..h1), as per-launch profiling does, and
// steps may be cut into runs in any way: the results are the same bit for bit.
// So every sum has one grouping (the atoms of a block, lane 0 of each group),
// the box advances by the same code inside a run and at its end, and
// k_run_therm takes its sums as piece A does.  The steps between that launch
// the passes one by one (half-list builds) are the same steps however a run is
// cut, and their update_therm_avs is taken here, too.
#include <type_traits>

#include "box.cuh"
#include "engine.h"
#include "pairs.cuh"

namespace moldy {
namespace {

constexpr int kRunThreads = 512;              // most threads per block
constexpr int kRunWarps = kRunThreads / 32;
constexpr int kRunBlocks = 148;               // most blocks
constexpr int kRunEmb = 256;                  // emb nodes kept in shared memory
// columns of a block's partial sums
constexpr int kColF = 0, kColK = 7, kColE = 13, kColMax = 15, kColOut = 16, kColHalf = 17, kColT = 18, kCols = 21;
constexpr int kBarStride = 4;                 // 32 bytes between barrier words

struct RunArgs {
    double4 *pos, *pos2;
    int4 *posq, *posq2;
    BoxState *box;
    const int32_t *nlist, *numn, *rlist, *numr;
    int32_t *olist, *out_cnt, *mlist, *mid_cnt, *alist, *pair_cnt;
    int4 *xout, *xbuild;
    const int4 *xhalf;
    const double *mass, *del2;
    const int32_t *znum;
    double *x1, *x2, *f, *rho, *afrho, *dafrho;
    double *part;                             // [2][kCols][gridDim.x]
    unsigned long long *bar;                  // one word per barrier of the launch, kBarStride apart (zero at its start)
    int32_t *flags;
    double *rec;                              // thermo records (null: none)
    int rec0;                                 // index of the record of the step before the run
    double rmid, rcut, rout;
    int m;                                    // steps of the run
    int h0, h1;                               // pieces of this launch (0: first drift, 2s+1: A, 2s+2: B, 2m+1: box)
    int therm;                                // the step before the run awaits its update_therm_avs
    int store;                                // 1: the run's last step also stores rho and the forces
    RunWait wait;                             // how long a barrier waits for the other blocks
};

// What the threads of a block share beside the tables
struct RunShared {
    BoxState box;
    double sum[kCols];                        // reduced columns
    double warp[kRunWarps][16];
    double tmp[27];
    float keep_out, keep_mid, rs2, rin2;
    float disp2;                              // largest squared displacement of the step, over the grid
    float md2_ok;                             // fixed box: squared displacements below this need no build
    int fail;
};

__device__ __forceinline__ unsigned long long load_relaxed(const unsigned long long *p) {
    unsigned long long v;
    asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
    return v;
}

__device__ __forceinline__ unsigned long long global_ns() {
    unsigned long long v;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(v));
    return v;
}

__device__ __forceinline__ void red_max(unsigned *p, unsigned v) {
    asm volatile("red.relaxed.gpu.global.max.u32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}

__device__ __forceinline__ void red_add_release(unsigned *p, unsigned v) {
    asm volatile("red.release.gpu.global.add.u32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}

__device__ __forceinline__ double *column(const RunArgs &a, int buf, int col) {
    return a.part + ((size_t)buf * kCols + col) * gridDim.x;
}

// This warp's sums (or maxima) of v[0..NV) as its local columns col0..
template <int NV>
__device__ __forceinline__ void warp_columns(RunShared &s, int col0, const double *v) {
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
#pragma unroll
    for (int k = 0; k < NV; ++k) {
        const double x = warp_sum(v[k]);
        if (lane == 0) s.warp[w][col0 + k] = x;
    }
}

__device__ __forceinline__ void warp_column_max(RunShared &s, int col, float v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, o));
    if ((threadIdx.x & 31) == 0) s.warp[threadIdx.x >> 5][col] = (double)v;
}

// local columns of the two pieces
constexpr int kA_E = 0, kA_T = 2, kA_Out = 5, kA_Half = 6, kB_F = 0, kB_K = 7, kB_Max = 13;

// Ends a piece: the block's sums of the local columns in mask go to the
// partial sums, and the grid meets.  Each barrier of a launch has its own
// word: arrivals in the high half, the largest displacement (kB_Max in mask;
// non-negative floats order as their bits) in the low half, so one thread per
// block polls both with one load.  No atomic returns a value, so the first
// poll leaves right after the arrival.  (A word per block polled by every
// block was slower: 143 x 143 polls of ten lines, 15.5 against 13.3 us per
// step at 2,000 atoms.)  A cooperative launch's blocks are all resident, so the
// others arrive within microseconds unless the device stands still; a barrier
// gives up after that many polls and, from then on, that much time (a device
// that is only slow, or stopped by a debugger, is waited for).  False in that
// case: flag 13 is set and the kernel ends.
__device__ __forceinline__ bool end_piece(const RunArgs &a, RunShared &s, unsigned &epoch, unsigned mask, bool piece_a,
                                          int buf) {
    __syncthreads();
    if (threadIdx.x < 32) {
        const int lane = threadIdx.x, nw = blockDim.x >> 5;
        float mx = 0.f;
        if ((mask >> lane) & 1u) {
            const bool ismax = piece_a ? lane >= kA_Out : lane == kB_Max;
            double x = s.warp[0][lane];
            for (int q = 1; q < nw; ++q) x = ismax ? fmax(x, s.warp[q][lane]) : x + s.warp[q][lane];
            const int col = piece_a ? (lane < kA_T ? kColE + lane : (lane < kA_Out ? kColT + lane - kA_T
                                                                                   : kColOut + lane - kA_Out))
                                    : (lane < kB_K ? kColF + lane : (lane < kB_Max ? kColK + lane - kB_K : kColMax));
            // what belongs to the next step (kinetic moment, displacement) goes to its buffer
            const int cb = !piece_a && lane >= kB_K ? buf ^ 1 : buf;
            column(a, cb, col)[blockIdx.x] = x;
            mx = (float)x;
        }
        mx = __shfl_sync(0xffffffffu, mx, kB_Max);
        ++epoch;
        __threadfence();
        __syncwarp();
        if (lane == 0) {
            unsigned *w = reinterpret_cast<unsigned *>(a.bar + (size_t)(epoch - 1) * kBarStride);   // little endian
            if ((mask >> kB_Max) & 1u) {
                red_max(w, __float_as_uint(mx));
                __threadfence();
            }
            red_add_release(w + 1, 1u);
            unsigned long long v = load_relaxed(a.bar + (size_t)(epoch - 1) * kBarStride);
            unsigned it = 0;
            for (unsigned long long t0 = 0ull; (unsigned)(v >> 32) != gridDim.x;
                 v = load_relaxed(a.bar + (size_t)(epoch - 1) * kBarStride)) {
                if (it < a.wait.polls) {
                    ++it;
                    continue;
                }
                const unsigned long long now = global_ns();
                if (t0 == 0ull) t0 = now;
                if (now - t0 >= a.wait.ns) {
                    s.fail = 1;
                    atomicExch(&a.flags[13], 1);
                    break;
                }
            }
            __threadfence();
            s.disp2 = __uint_as_float((unsigned)v);
        }
    } else {
        ++epoch;
    }
    __syncthreads();
    return s.fail == 0;
}

// finalize_box at the end of a run, by one thread (out of line: its registers
// do not count against the pieces)
__device__ __noinline__ void end_box(const Params &p, RunShared &s) {
    double sr[15];
    sr[0] = s.sum[kColE]; sr[1] = s.sum[kColE + 1];
    for (int k = 0; k < 7; ++k) sr[2 + k] = s.sum[kColF + k];
    for (int k = 0; k < 6; ++k) sr[9 + k] = s.sum[kColK + k];
    if (s.box.mid_rebuild) s.box.outdisp2 = (unsigned long long)__double_as_longlong(s.sum[kColOut]);
    if (s.box.out_rebuild) s.box.halfdisp2 = (unsigned long long)__double_as_longlong(s.sum[kColHalf]);
    finalize_box(p, s.box, sr, 0, false);
}

// Column col of buffer buf over the blocks, by one warp: the same bits in every block
__device__ __forceinline__ double reduce_col(const RunArgs &a, int buf, int col) {
    const double *c = column(a, buf, col);
    const int lane = threadIdx.x & 31;
    double e[(kRunBlocks + 31) / 32];
#pragma unroll
    for (int q = 0; q < (kRunBlocks + 31) / 32; ++q) {
        const int b = lane + 32 * q;
        e[q] = b < (int)gridDim.x ? __ldcg(&c[b]) : 0.0;
    }
    const bool mx = col == kColMax || col == kColOut || col == kColHalf;
    double x = e[0];
#pragma unroll
    for (int q = 1; q < (kRunBlocks + 31) / 32; ++q) x = mx ? fmax(x, e[q]) : x + e[q];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        const double y = __shfl_xor_sync(0xffffffffu, x, o);
        x = mx ? fmax(x, y) : x + y;
    }
    return x;
}

__device__ __forceinline__ unsigned long long dbits(double v) { return (unsigned long long)__double_as_longlong(v); }

// element (i, j) of the cofactor matrix of b as mat_cofactor forms it (0-based)
__device__ __forceinline__ double cof_at(const double *b, int i, int j) {
    const int i1 = i == 2 ? 0 : i + 1, i2 = i == 0 ? 2 : i - 1, j1 = j == 2 ? 0 : j + 1, j2 = j == 0 ? 2 : j - 1;
    return b[i1 + 3 * j1] * b[i2 + 3 * j2] - b[i2 + 3 * j1] * b[i1 + 3 * j2];
}

// The box half-kick that ends a step (finalize_box), one matrix element per
// lane, by one warp.
__device__ __forceinline__ void warp_half_kick(const Params &p, RunShared &s, int lane) {
    BoxState &B = s.box;
    const int e = lane < 9 ? lane : 0, i = e % 3, j = e / 3;
    const double *D = s.sum + kColF + 1, *M = s.sum + kColK;
    if (p.ivol == 0 || p.ivol == 4) {
        double tp = 0.0, tk = 0.0;
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            const int q = c == j ? c : c + j + 2;     // (c, j) of a symmetric matrix in xx yy zz xy xz yz
            tp += B.b0[i + 3 * c] * D[q];
            tk += B.b0[i + 3 * c] * M[q];
        }
        tk = tk / (p.deltat * p.deltat);
        const double fb = tk + tp - p.press * cof_at(B.b0, i, j);
        double b2 = B.b2[e];
        if (p.ivol == 0 || e == 8) b2 = p.bdel2 * fb;
        const double b1 = B.b1[e] + b2;
        __syncwarp();
        if (lane < 9) { B.b2[e] = b2; B.b1[e] = b1; }
        __syncwarp();
    }
}

// The box quantities of a step's update_therm_avs (therm_prep), likewise.
__device__ __noinline__ void warp_therm_prep(const Params &p, RunShared &s, int lane) {
    BoxState &B = s.box;
    const int e = lane < 9 ? lane : 0, i = e % 3, j = e / 3;
    double tg = 0.0, td = 0.0;
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        tg += B.b0[k + 3 * i] * B.b0[k + 3 * j];
        td = td + B.b1[k + 3 * i] * B.b0[k + 3 * j] + B.b0[k + 3 * i] * B.b1[k + 3 * j];
    }
    if (p.ivol == 1) td = 0.0;                        // the box does not move
    if (lane < 9) { s.tmp[e] = tg; s.tmp[9 + e] = td; }
    __syncwarp();
    double det = 0.0;
#pragma unroll
    for (int k = 0; k < 3; ++k) det += s.tmp[k] * cof_at(s.tmp, k, 0);
    const double inv = cof_at(s.tmp, j, i) / det;
    if (lane < 9) s.tmp[18 + e] = inv;
    if (lane == 0 && fabs(det) == 0.0) B.status = MOLDY_ERR_SINGULAR_BOX;
    __syncwarp();
    double g = 0.0;
#pragma unroll
    for (int k = 0; k < 3; ++k) g += s.tmp[18 + i + 3 * k] * s.tmp[9 + k + 3 * j];
    const double vol = mat_volume(B.b0);
    if (lane < 9) {
        B.th_tgid[e] = g;
        B.th_cof[3 * i + j] = cof_at(B.b0, i, j) / vol;
    }
    __syncwarp();
}

// A step's thermo record (therm_store) from its box b0, b1, the three sums of
// update_therm_avs and its energy, by one thread
__device__ __forceinline__ void step_record(const Params &p, const double *b0, const double *b1, const double *s3, double pe,
                                         double *r) {
    const double bk = 1.3806504e-23 / 1.602176487e-19;
    const double ke = s3[2] / (p.deltat * p.deltat) / 2.0, vol = mat_volume(b0);
    double boxke = 0.0;
    for (int k = 0; k < 9; ++k) boxke = boxke + (b1[k] * b1[k]) / p.bdel2;
    const double te = ke + pe, hh = te + p.press * vol;
    r[0] = ke; r[1] = pe; r[2] = te; r[3] = hh; r[4] = hh + boxke; r[5] = vol;
    r[6] = s3[0]; r[7] = s3[1]; r[8] = s3[2]; r[9] = ke / (1.5 * bk * (double)p.nm); r[10] = boxke;
}

// The box half of velocityverlet's first part, and the list decision of
// k_mid_decide.  disp is the largest displacement since the intermediate
// build, measured in the box before this advance.
__device__ void warp_decide(const Params &p, const RunArgs &a, RunShared &s, float disp2, int lane) {
    BoxState &B = s.box;
    const int e = lane < 9 ? lane : 0;
    double db0 = 0.0;
    if (p.ivol == 0 || (p.ivol == 4 && e == 8)) {
        const double b1 = B.b1[e] + B.b2[e];
        db0 = b1;
        if (lane < 9) { B.b1[e] = b1; B.b0[e] = B.b0[e] + b1; }
    }
    if (lane < 9) s.tmp[lane] = db0;
    __syncwarp();
    // Frobenius norms of B0, of B0 less its value at the build, and of this
    // step's change, by lanes 0..2; in FP32, rounded up (a decision may come
    // early, never late: mid_decide_box decides in FP64 what this asks for)
    float n2 = 0.f;
    if (lane < 3)
        for (int k = 0; k < 9; ++k) {
            const float x = (float)(lane == 0 ? B.b0[k] : (lane == 1 ? B.b0[k] - B.bbuild[k] : s.tmp[k]));
            n2 = fmaf(x, x, n2);
        }
    const float nf = sqrtf(n2) * 1.00001f;
    const float f0 = __shfl_sync(0xffffffffu, nf, 0), fd = __shfl_sync(0xffffffffu, nf, 1),
                fs = __shfl_sync(0xffffffffu, nf, 2);
    const float eps = (float)(2.0e-6) * f0 + 1.0e-4f;
    const float dmax = (float)B.dmax_mid * 1.00001f;
    // |B_new x| <= |B_old x| (1 + |B_new - B_old|_F |B_old^-1|_F), the inverse's norm from the build
    const float grow = 1.00002f + 2.f * fs * dmax / (float)p.rnear;
    const float md = sqrtf(disp2) * grow + 1.0e-6f;
    const bool need = !(dmax > 0.f) || !(1.00001f * (2.f * md + fd * dmax) < (float)(a.rmid - a.rcut) * 0.99999f - 2.f * eps);
    if (lane == 0) {
        B.mid_rebuild = 0;
        B.out_rebuild = 0;
        // with a box that does not move, what a displacement must stay below
        const float ok = ((float)(a.rmid - a.rcut) * 0.99998f - 2.f * eps - fd * dmax) * 0.49999f - 2.0e-6f;
        s.md2_ok = dmax > 0.f && ok > 0.f ? ok * ok * 0.9999f : 0.f;
        if (need) {
            B.maxdisp2 = dbits((double)md * (double)md);
            mid_decide_box(p, B, a.rmid, a.rcut, a.rout, 0, 0, 0);
            s.md2_ok = 0.f;                   // measured anew at the next step
        }
    }
    __syncwarp();
}

// The screening band of the mixed density pass (screen_radius2) in FP32: the
// band may be wider than there, never narrower, and inside it the FP64
// distance decides.
__device__ __forceinline__ void lane_screen(RunShared &s, double rcull2) {
    float b[9], n2 = 0.f;
#pragma unroll
    for (int k = 0; k < 9; ++k) { b[k] = (float)s.box.b0[k]; n2 = fmaf(b[k], b[k], n2); }
    float wmin = 3.0e38f;
    const float rc = sqrtf((float)rcull2);
    const float rs = rc * 1.000001f + 2.01e-6f * sqrtf(n2) + 1.01e-4f;
    for (int k = 0; k < 3; ++k) {
        const int i = 3 * ((k + 1) % 3), j = 3 * ((k + 2) % 3);
        float u[3], w[3], o[3];
        for (int q = 0; q < 3; ++q) {
            u[q] = (float)s.box.b0[i + q]; w[q] = (float)s.box.b0[j + q]; o[q] = (float)s.box.b0[3 * k + q];
        }
        const float cx = u[1] * w[2] - u[2] * w[1], cy = u[2] * w[0] - u[0] * w[2], cz = u[0] * w[1] - u[1] * w[0];
        wmin = fminf(wmin, fabsf(o[0] * cx + o[1] * cy + o[2] * cz) * rsqrtf(cx * cx + cy * cy + cz * cz));
    }
    const bool ok = 0.49f * wmin > rs;       // 2 % below the width: a narrower box sends every pair to FP64
    const float rin = 2.f * rc - rs;
    s.rs2 = ok ? rs * rs : 3.0e38f;
    s.rin2 = !ok || rin <= 0.f ? -1.f : rin * rin;
}

// inside_cut_fp64 on positions that this kernel also writes (in its other piece)
__device__ __noinline__ bool inside_cut(const double4 *pos, int a, int j, const double *b, int ivol, double rcull2) {
    const double2 *pa = reinterpret_cast<const double2 *>(pos + a), *pj = reinterpret_cast<const double2 *>(pos + j);
    const double2 axy = __ldcg(pa), az = __ldcg(pa + 1), jxy = __ldcg(pj), jz = __ldcg(pj + 1);
    double ex = axy.x - jxy.x, ey = axy.y - jxy.y, ez = az.x - jz.x;
    min_image(ivol, ex, ey, ez);
    const double sx = b[0] * ex + b[3] * ey + b[6] * ez;
    const double sy = b[1] * ex + b[4] * ey + b[7] * ez;
    const double sz = b[2] * ex + b[5] * ey + b[8] * ez;
    return (sx * sx + sy * sy + sz * sz) <= rcull2;
}

// ------------------------------------------------- tables in shared memory --
struct TabMixed {
    const float4 *r4;      // per interval: node, difference to the next node
    const float2 *phi;
};
struct TabFp64 {
    const double4 *r4;
    const double2 *phi;
};

__device__ __forceinline__ float4 tab_r4(const TabMixed &m, const Tables &t, float r) {
    const float x = fmaf(r, t.recipstep_f, t.xoff_f);
    float fl;
    const int idx = floor_small(fmaxf(x, 0.f), fl);
    if (idx >= t.nr - 1) return t.tail_f;
    const float dr = x - fl;
    const float4 a = m.r4[2 * idx], b = m.r4[2 * idx + 1];
    return make_float4(fmaf(b.x, dr, a.x), fmaf(b.y, dr, a.y), fmaf(b.z, dr, a.z), fmaf(b.w, dr, a.w));
}

__device__ __forceinline__ float tab_phi(const TabMixed &m, const Tables &t, float r) {
    const float x = fmaf(r, t.recipstep_f, t.xoff_f);
    float fl;
    const int idx = floor_small(fmaxf(x, 0.f), fl);
    if (idx >= t.nr - 1) return t.tail_f.z;
    const float2 v = m.phi[idx];
    return fmaf(v.y, x - fl, v.x);
}

__device__ __forceinline__ double4 tab_r4(const TabFp64 &m, const Tables &t, double r) {
    if (r >= t.vp_rmax) return m.r4[t.nlookup < t.nr ? t.nlookup : t.nr - 1];
    int idx = (int)(((double)t.nlookup * (r - t.vp_rmin)) * t.vp_reciprange);
    if (idx >= t.nr - 1) return make_double4(0.0, 0.0, 0.0, 0.0);
    idx = idx < 0 ? 0 : idx;
    const double rlow = t.vp_rmin + (t.vp_range * (double)idx) * t.vp_recipnlkp;
    const double dr = (r - rlow) * t.vp_recipstep, w = 1.0 - dr;
    const double4 a = m.r4[idx], b = m.r4[idx + 1];
    return make_double4(a.x * w + b.x * dr, a.y * w + b.y * dr, a.z * w + b.z * dr, a.w * w + b.w * dr);
}

__device__ __forceinline__ double tab_phi(const TabFp64 &m, const Tables &t, double r) {
    if (r >= t.vp_rmax) return m.r4[t.nlookup < t.nr ? t.nlookup : t.nr - 1].z;
    int idx = (int)(((double)t.nlookup * (r - t.vp_rmin)) * t.vp_reciprange);
    if (idx >= t.nr - 1) return 0.0;
    idx = idx < 0 ? 0 : idx;
    const double rlow = t.vp_rmin + (t.vp_range * (double)idx) * t.vp_recipnlkp;
    const double dr = (r - rlow) * t.vp_recipstep;
    const double2 v = m.phi[idx];
    return v.x * (1.0 - dr) + v.y * dr;
}

// (emb, demb) with the first kRunEmb nodes in shared memory
__device__ __forceinline__ double2 tab_emb(const double2 *se, int ne, const Tables &t, double rho) {
    if (rho >= t.e_rmax) return __ldg(&t.e2[t.nlookup]);
    int idx = (int)(((double)t.nlookup * (rho - t.e_rmin)) * t.e_reciprange);
    idx = idx < 0 ? 0 : (idx > t.nlookup - 1 ? t.nlookup - 1 : idx);
    const double rlow = t.e_rmin + (t.e_range * (double)idx) * t.e_recipnlkp;
    const double dr = (rho - rlow) * t.e_recipstep, w = 1.0 - dr;
    const bool in = idx + 1 < ne;
    const double2 a = in ? se[idx] : __ldg(&t.e2[idx]), b = in ? se[idx + 1] : __ldg(&t.e2[idx + 1]);
    return make_double2(a.x * w + b.x * dr, a.y * w + b.y * dr);
}

// an element of 8 or 16 bytes from global to shared memory, behind the thread's back
template <typename T>
__device__ __forceinline__ void copy_async(T *dst, const T *src) {
    static_assert(sizeof(T) == 8 || sizeof(T) == 16, "cp.async sizes");
    asm volatile("cp.async.ca.shared.global [%0], [%1], %2;" ::"r"((unsigned)__cvta_generic_to_shared(dst)), "l"(src),
                 "n"(sizeof(T)));
}

// waits for this thread's copies
__device__ __forceinline__ void copies_arrived() { asm volatile("cp.async.wait_all;" ::: "memory"); }

// sum over the L lanes of an atom's group, in every lane of it
template <int L>
__device__ __forceinline__ double group_sum(double v) {
#pragma unroll
    for (int o = L / 2; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

// Appends to row a of dst the entries of a source row whose FP32 distance is
// within keep2, in their order: the L lanes test L entries at a time and a
// ballot places them (filter_row's result).  The whole warp runs every round
// (n = 0 for groups without an atom): a ballot per group mask would split the
// warp into its groups.
template <int L>
__device__ __forceinline__ int group_filter(const Params &p, const int32_t *row, size_t step, int n, int a,
                                            const int4 &qa, const int4 *posq, const float *bs, float keep2,
                                            int32_t own, int32_t *dst, int cap, int cnt, int g, unsigned gmask) {
    const unsigned below = (1u << (threadIdx.x & 31)) - 1u;
    constexpr int U = 4;                      // entries gathered ahead
    const int nmax = __reduce_max_sync(0xffffffffu, n);
    for (int k0 = 0; k0 < nmax; k0 += U * L) {
        int ent[U];
        int4 qq[U];
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const int k = k0 + u * L + g;
            ent[u] = k < n ? row[(size_t)k * step] : -1;
        }
#pragma unroll
        for (int u = 0; u < U; ++u) qq[u] = posq[ent[u] != -1 ? (ent[u] & kIdMask) : a];
#pragma unroll
        for (int u = 0; u < U; ++u) {
            float rx, ry, rz;
            const bool hit = ent[u] != -1 && fix_sep(bs, qa, qq[u], rx, ry, rz) <= keep2;
            const unsigned m = __ballot_sync(0xffffffffu, hit) & gmask;
            if (hit) {
                const int e = cnt + __popc(m & below);
                if (e < cap) dst[(size_t)e * p.nm + a] = ent[u] | own;
            }
            cnt += __popc(m);
        }
    }
    return cnt;
}

// -------------------------------------------------------------- the kernel --
template <bool MIXED, int L>
__global__ void __launch_bounds__(kRunThreads, 1)
k_run(Params p, Tables t, RunArgs a) {
    extern __shared__ __align__(16) unsigned char dsm[];
    __shared__ RunShared s;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, nw = blockDim.x >> 5;
    const int g = tid % L;
    const unsigned gmask = (L == 32 ? 0xffffffffu : ((1u << L) - 1u)) << (lane - g);
    const unsigned below = (1u << lane) - 1u;
    const int nm = p.nm;
    const size_t stride = (size_t)nm;
    const int per_round = gridDim.x * (blockDim.x / L);
    const int first = blockIdx.x * (blockDim.x / L) + tid / L;
    const int rounds = (nm + per_round - 1) / per_round;
    // row entries a lane gathers before it uses any: a row of 14 to 20 entries
    // is then one to three rounds
    constexpr int BD = L >= 8 ? 2 : (!MIXED ? 3 : (L >= 2 ? 5 : 8)), BF = L >= 8 ? 2 : (MIXED ? 4 : 3);
    const bool boxed = p.ivol == 0 || p.ivol == 4;   // the box moves: every step needs its virial

    // the tables, on their way while the first drift runs
    using Tab = typename std::conditional<MIXED, TabMixed, TabFp64>::type;
    Tab tab;
    double2 *se;
    const int ne_emb = t.nlookup + 1 < kRunEmb ? t.nlookup + 1 : kRunEmb;
    if constexpr (MIXED) {
        float4 *r4 = reinterpret_cast<float4 *>(dsm);
        float2 *ph = reinterpret_cast<float2 *>(r4 + 2 * (size_t)t.nr);
        se = reinterpret_cast<double2 *>(ph + ((t.nr + 1) & ~1));
        for (int k = tid; k < 2 * t.nr; k += blockDim.x) copy_async(&r4[k], &t.r4f[k]);
        for (int k = tid; k < t.nr; k += blockDim.x) copy_async(&ph[k], &t.phi2f[k]);
        tab.r4 = r4; tab.phi = ph;
    } else {
        double4 *r4 = reinterpret_cast<double4 *>(dsm);
        double2 *ph = reinterpret_cast<double2 *>(r4 + t.nr);
        se = ph + t.nr;
        for (int k = tid; k < 2 * t.nr; k += blockDim.x)
            copy_async(reinterpret_cast<double2 *>(r4) + k, reinterpret_cast<const double2 *>(t.r4) + k);
        for (int k = tid; k < t.nr; k += blockDim.x) copy_async(&ph[k], &t.phi2[k]);
        tab.r4 = r4; tab.phi = ph;
    }
    for (int k = tid; k < ne_emb; k += blockDim.x) copy_async(&se[k], &t.e2[k]);
    box_load(s.box, a.box);
    if (tid == 0) s.fail = a.flags[13];       // an earlier run of the call gave up: so does this one
    __syncthreads();
    if (s.fail) {
        copies_arrived();                     // no block ends with copies on their way
        return;
    }

    unsigned epoch = 0;
    for (int h = a.h0; h <= a.h1; ++h) {
        if (h == (a.h0 > 0 ? a.h0 : 1)) {     // the first piece that reads them
            copies_arrived();
            __syncthreads();
        }
        if (h == 0) {
            // ---- first half-kick and drift of the run's first step (k_drift),
            // with the sums in piece B's grouping
            double k6[6] = {0.0, 0.0, 0.0, 0.0, 0.0, 0.0};
            float d2 = 0.f, bs[9];
#pragma unroll
            for (int k = 0; k < 9; ++k) bs[k] = (float)(s.box.b0[k] * kFixUnit);
            for (int it = 0; it < rounds; ++it) {
                const int i = first + it * per_round;
                if (i >= nm || g != 0) continue;
                const double ex = a.x1[i], ey = a.x1[nm + i], ez = a.x1[2 * nm + i];
                const double wx = a.x2[i], wy = a.x2[nm + i], wz = a.x2[2 * nm + i];
                double4 q = a.pos[i];
                q.x = q.x + (ex + wx); q.y = q.y + (ey + wy); q.z = q.z + (ez + wz);
                a.pos[i] = q;
                const int4 qn = make_int4(fix32(q.x), fix32(q.y), fix32(q.z), 0);
                a.posq[i] = qn;
                d2 = fmaxf(d2, fix_disp2(bs, qn, a.xbuild[i]));
                if (a.znum[i] != 0) kin_moment(k6, a.mass[i], ex, ey, ez);
            }
            warp_columns<6>(s, kB_K, k6);
            warp_column_max(s, kB_Max, d2);
            if (!end_piece(a, s, epoch, 0x3f80u, false, 1)) {   // step 0's buffer is 0
                copies_arrived();
                return;
            }
            continue;
        }
        if (h == 2 * a.m + 1) {
            // ---- the box at the end of the run, by block 0
            const int pb = (a.m - 1) & 1;
            if (blockIdx.x == 0) {
                for (int c = warp; c < kColT; c += nw)
                    if (c != kColMax) {
                        const double x = reduce_col(a, pb, c);
                        if (lane == 0) s.sum[c] = x;
                    }
                __syncthreads();
                if (tid == 0) {
                    // finalize_box takes embedding energy, pairs; pair energy, virial; kinetic moments;
                    // the half-kick is that of the steps before, and what update_therm_avs
                    // needs is formed where it is taken
                    end_box(p, s);
                }
                __syncwarp();
                if (warp == 0) warp_half_kick(p, s, lane);
            }
            if (!end_piece(a, s, epoch, 0u, false, 0)) return;
            continue;
        }
        const int step = (h - 1) >> 1, buf = step & 1, pbuf = buf ^ 1;
        if (h & 1) {
            // ---- A: box, lists, density of step `step`
            const bool fin = step > 0, therm = (fin || a.therm) && a.rec != nullptr;
            if (h == a.h0) {       // no barrier of this launch brought the largest displacement
                if (warp == 0) {
                    const double x = reduce_col(a, buf, kColMax);
                    if (lane == 0) s.disp2 = (float)x;
                }
                __syncthreads();
            }
            // with a fixed box and no build, before or now, nothing about the box or the lists changes
            const bool quiet = !boxed && h != a.h0 && step > 0 && !s.box.mid_rebuild && s.disp2 < s.md2_ok;
            if (!quiet) {
                if (fin)
                    for (int c = warp; c < kColMax + 3; c += nw) {
                        if (c == kColMax || (!boxed && c < kColOut)) continue;
                        const double x = reduce_col(a, pbuf, c);
                        if (lane == 0) s.sum[c] = x;
                    }
                __syncthreads();
                if (warp == 0) {
                    if (fin) {
                        if (lane == 0) {
                            if (s.box.mid_rebuild) s.box.outdisp2 = dbits(s.sum[kColOut]);
                            if (s.box.out_rebuild) s.box.halfdisp2 = dbits(s.sum[kColHalf]);
                        }
                        warp_half_kick(p, s, lane);
                    }
                    // of a fixed box they are the same at every step
                    if (p.ivol == 1 ? step == 0 || h == a.h0 : fin || a.therm) warp_therm_prep(p, s, lane);
                    if (lane < 9) {
                        s.box.rec_b0[lane] = s.box.b0[lane];
                        s.box.rec_b1[lane] = s.box.b1[lane];
                        if (fin || a.therm) s.box.tgid[lane] = s.box.th_tgid[lane];
                    }
                    __syncwarp();
                    warp_decide(p, a, s, s.disp2, lane);
                    if (MIXED && lane == 0 && (boxed || h == 1 || h == a.h0)) lane_screen(s, t.rcull2);
                    if (lane == 0 && (s.box.mid_rebuild || s.box.out_rebuild)) {
                        s.keep_out = keep_radius2(s.box.b0, a.rout);
                        s.keep_mid = keep_radius2(s.box.b0, a.rmid);
                    }
                }
                __syncthreads();
            }
            const bool need_out = s.box.out_rebuild != 0, need_mid = s.box.mid_rebuild != 0;
            float bs[9];
            double b[9];
#pragma unroll
            for (int k = 0; k < 9; ++k) { b[k] = s.box.b0[k]; bs[k] = (float)(b[k] * kFixUnit); }
            double v2[2] = {0.0, 0.0}, vt[3] = {0.0, 0.0, 0.0};
            float dout = 0.f, dhalf = 0.f;
            int over = 0, over_max = 0, oover = 0;
            for (int it = 0; it < rounds; ++it) {
                const bool live = first + it * per_round < nm;   // the same for all lanes of a group
                const int i = live ? first + it * per_round : 0;
                const int4 qa = a.posq[i];
                int mc = need_mid || !live ? 0 : a.mid_cnt[i];
                if (need_out) {
                    int cnt = group_filter<L>(p, a.nlist + (size_t)i * p.nnbrs, 1, live ? a.numn[i] : 0, i, qa,
                                              a.posq, bs, s.keep_out, kOwnBit, a.olist, p.out_cap, 0, g, gmask);
                    cnt = group_filter<L>(p, a.rlist + i, stride, live ? a.numr[i] : 0, i, qa, a.posq, bs,
                                          s.keep_out, 0, a.olist, p.out_cap, cnt, g, gmask);
                    if (cnt > p.out_cap) oover = max(oover, cnt);
                    if (live && g == 0) {
                        dhalf = fmaxf(dhalf, fix_disp2(bs, qa, a.xhalf[i]));
                        a.out_cnt[i] = cnt;
                        a.xout[i] = qa;
                    }
                    __syncwarp();
                }
                if (need_mid) {
                    const int nt = live ? a.out_cnt[i] : 0;
                    mc = group_filter<L>(p, a.olist + i, stride, nt < p.out_cap ? nt : p.out_cap, i, qa, a.posq, bs,
                                         s.keep_mid, 0, a.mlist, p.mid_cap, 0, g, gmask);
                    if (live && g == 0) {
                        a.mid_cnt[i] = mc;
                        a.xbuild[i] = qa;
                        dout = fmaxf(dout, fix_disp2(bs, qa, a.xout[i]));
                    }
                    __syncwarp();
                }
                const int n = mc < p.mid_cap ? mc : p.mid_cap;
                // update_therm_avs of the step before, by one lane
                if (therm && live && g == 0 && a.znum[i] != 0) {
                    therm_terms(vt, s.box.th_tgid, s.box.rec_b0, s.box.th_cof, a.mass[i], a.x1[i], a.x1[nm + i],
                                a.x1[2 * nm + i], a.x2[i], a.x2[nm + i], a.x2[2 * nm + i]);
                }
                double4 pa = make_double4(0.0, 0.0, 0.0, 0.0);
                if (!MIXED) pa = a.pos[i];
                double rho = 0.0;
                int cnt = 0;
                const int nmax = __reduce_max_sync(0xffffffffu, n);
                for (int k0 = 0; k0 < nmax; k0 += BD * L) {
                    int ee[BD];
#pragma unroll
                    for (int u = 0; u < BD; ++u) {
                        const int k = k0 + u * L + g;
                        ee[u] = k < n ? a.mlist[(size_t)k * stride + i] : -1;
                    }
                    bool hit[BD];
                    if constexpr (MIXED) {
                        int4 qq[BD];
#pragma unroll
                        for (int u = 0; u < BD; ++u) qq[u] = a.posq[ee[u] != -1 ? (ee[u] & kIdMask) : i];
#pragma unroll
                        for (int u = 0; u < BD; ++u) {
                            float rx, ry, rz;
                            const float r2 = fix_sep(bs, qa, qq[u], rx, ry, rz);
                            hit[u] = ee[u] != -1 && !(r2 > s.rs2);
                            if (hit[u] && !(r2 < s.rin2))
                                hit[u] = inside_cut(a.pos, i, ee[u] & kIdMask, s.box.b0, p.ivol, t.rcull2);
                            if (hit[u]) rho += (double)tab_phi(tab, t, r2 * rsqrt_ftz(r2));
                        }
                    } else {
                        double4 qq[BD];
#pragma unroll
                        for (int u = 0; u < BD; ++u) qq[u] = a.pos[ee[u] != -1 ? (ee[u] & kIdMask) : i];
#pragma unroll
                        for (int u = 0; u < BD; ++u) {
                            double dx = pa.x - qq[u].x, dy = pa.y - qq[u].y, dz = pa.z - qq[u].z;
                            min_image(p.ivol, dx, dy, dz);
                            const double rx = b[0] * dx + b[3] * dy + b[6] * dz;
                            const double ry = b[1] * dx + b[4] * dy + b[7] * dz;
                            const double rz = b[2] * dx + b[5] * dy + b[8] * dz;
                            const double r2 = rx * rx + ry * ry + rz * rz;
                            hit[u] = ee[u] != -1 && r2 <= t.rcull2;
                            if (hit[u]) rho += tab_phi(tab, t, sqrt(r2));
                        }
                    }
#pragma unroll
                    for (int u = 0; u < BD; ++u) {
                        const unsigned m = __ballot_sync(0xffffffffu, hit[u]) & gmask;
                        if (hit[u]) {
                            const int e = cnt + __popc(m & below);
                            if (e < p.pair_cap) a.alist[(size_t)e * stride + i] = ee[u];
                        }
                        cnt += __popc(m);
                    }
                }
                rho = group_sum<L>(rho);
                if (cnt > p.pair_cap) { over |= 1; over_max = max(over_max, cnt); }
                if (mc > p.mid_cap) { over |= 2; over_max = max(over_max, mc); }
                if (live && g == 0) {
                    a.pair_cnt[i] = cnt;
                    v2[1] += (double)cnt;
                    double fd;
                    if (rho > 1e-40) {            // src/potential_m.F90:162: else the old values stay
                        const double2 e = tab_emb(se, ne_emb, t, rho);
                        a.afrho[i] = e.x;
                        a.dafrho[i] = e.y;
                        fd = e.y;
                        v2[0] += e.x;
                    } else {
                        fd = a.dafrho[i];
                    }
                    if (a.store && step == a.m - 1) a.rho[i] = rho;
                    if (MIXED) a.posq2[i] = make_int4(qa.x, qa.y, qa.z, __float_as_int((float)fd));
                    else a.pos2[i] = make_double4(pa.x, pa.y, pa.z, fd);
                }
            }
            if (over & 1) { atomicExch(&a.flags[3], 1); atomicMax(&a.flags[4], over_max); }
            if (over & 2) { atomicExch(&a.flags[5], 1); atomicMax(&a.flags[6], over_max); }
            if (oover) { atomicExch(&a.flags[8], 1); atomicMax(&a.flags[9], oover); }
            warp_columns<2>(s, kA_E, v2);
            if (therm) warp_columns<3>(s, kA_T, vt);
            if (need_mid) warp_column_max(s, kA_Out, dout);
            if (need_out) warp_column_max(s, kA_Half, dhalf);
            if (!end_piece(a, s, epoch, 3u | (therm ? 0x1cu : 0u) | (need_mid ? 0x20u : 0u) | (need_out ? 0x40u : 0u),
                           true, buf))
                return;
            continue;
        }
        // ---- B: forces and second half-kick of step `step`, drift of the next
        const bool last = step == a.m - 1, drift = !last;
        const bool vir = boxed || last, kin = boxed || step == a.m - 2;
        // the thermo record of the step before, by the last block
        const bool fin = step > 0;
        if (a.rec && (fin || a.therm) && blockIdx.x == gridDim.x - 1 && warp == nw - 1) {
            double s3[3];
#pragma unroll
            for (int k = 0; k < 3; ++k) s3[k] = reduce_col(a, buf, kColT + k);
            // the energy of that step: of this run, or as the launches before it left it
            const double pe = fin ? reduce_col(a, pbuf, kColE) + reduce_col(a, pbuf, kColF) : s.box.pe;
            if (lane == 0) {
                step_record(p, s.box.rec_b0, s.box.rec_b1, s3, pe, a.rec + (size_t)kThermoRec * (size_t)(a.rec0 + step));
            }
            __syncwarp();
        }
        float bs[9];
        double b[9];
#pragma unroll
        for (int k = 0; k < 9; ++k) { b[k] = s.box.b0[k]; bs[k] = (float)(b[k] * kFixUnit); }
        double v[7] = {0.0, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0}, k6[6] = {0.0, 0.0, 0.0, 0.0, 0.0, 0.0};
        float d2 = 0.f;
        for (int it = 0; it < rounds; ++it) {
            const bool live = first + it * per_round < nm;
            const int i = live ? first + it * per_round : 0;
            // the integrator's loads, ahead of the row
            double u1[3], w2[3], del = 0.0;
            double4 q0 = make_double4(0.0, 0.0, 0.0, 0.0);
            int4 xb = make_int4(0, 0, 0, 0);
            int zn = 0;
            const double ma = a.mass[i];
            if (live && g == 0) {
#pragma unroll
                for (int k = 0; k < 3; ++k) { u1[k] = a.x1[k * nm + i]; w2[k] = a.x2[k * nm + i]; }
                del = a.del2[i];
                zn = a.znum[i];
                if (drift) { q0 = a.pos[i]; xb = a.xbuild[i]; }
            }
            int ne = live ? a.pair_cnt[i] : 0;
            ne = ne < p.pair_cap ? ne : p.pair_cap;
            double fx = 0.0, fy = 0.0, fz = 0.0;
            if constexpr (MIXED) {
                const int4 qa = a.posq2[i];
                const float fa = __int_as_float(qa.w);
                for (int e0 = g; e0 < ne; e0 += BF * L) {
                    int ee[BF];
#pragma unroll
                    for (int u = 0; u < BF; ++u) {
                        const int e = e0 + u * L;
                        ee[u] = e < ne ? a.alist[(size_t)e * stride + i] : -1;
                    }
                    int4 qq[BF];
#pragma unroll
                    for (int u = 0; u < BF; ++u) qq[u] = a.posq2[ee[u] != -1 ? (ee[u] & kIdMask) : i];
#pragma unroll
                    for (int u = 0; u < BF; ++u) {
                        if (ee[u] == -1) continue;
                        const int4 qj = qq[u];
                        const int32_t ex = (int32_t)((uint32_t)qa.x - (uint32_t)qj.x);
                        const int32_t ey = (int32_t)((uint32_t)qa.y - (uint32_t)qj.y);
                        const int32_t ez = (int32_t)((uint32_t)qa.z - (uint32_t)qj.z);
                        const float dx = fix_to_float(ex), dy = fix_to_float(ey), dz = fix_to_float(ez);
                        const float rx = fmaf(bs[6], dz, fmaf(bs[3], dy, bs[0] * dx));
                        const float ry = fmaf(bs[7], dz, fmaf(bs[4], dy, bs[1] * dx));
                        const float rz = fmaf(bs[8], dz, fmaf(bs[5], dy, bs[2] * dx));
                        const float r2 = fmaf(rz, rz, fmaf(ry, ry, rx * rx));
                        const float rr = rsqrt_ftz(r2);
                        const float4 tv = tab_r4(tab, t, r2 * rr);
                        const float fp = -(tv.y + tv.w * (fa + __int_as_float(qj.w))) * rr;
                        const float dfx = dx * fp, dfy = dy * fp, dfz = dz * fp;
                        fx += (double)dfx; fy += (double)dfy; fz += (double)dfz;
                        if (ee[u] & kOwnBit) v[0] += (double)tv.x;
                        if (vir) {
                            // pairs across a periodic boundary, and those the mass filter leaves out (k_forces)
                            const int32_t wx = (qa.x ^ qj.x) & (qa.x ^ ex), wy = (qa.y ^ qj.y) & (qa.y ^ ey),
                                          wz = (qa.z ^ qj.z) & (qa.z ^ ez);
                            const bool excluded = !(ma > 0.1 || ma + a.mass[ee[u] & kIdMask] > 0.1);
                            if ((wx | wy | wz) < 0 || excluded) {
                                double cx = wx < 0 ? (qa.x >= 0 ? kFixScale : -kFixScale) : 0.0;
                                double cy = wy < 0 ? (qa.y >= 0 ? kFixScale : -kFixScale) : 0.0;
                                double cz = wz < 0 ? (qa.z >= 0 ? kFixScale : -kFixScale) : 0.0;
                                if (excluded) { cx += (double)ex; cy += (double)ey; cz += (double)ez; }
                                add_sym(v, cx, cy, cz, (double)dfx, (double)dfy, (double)dfz, -0.5);
                            }
                        }
                    }
                }
                fx = group_sum<L>(fx); fy = group_sum<L>(fy); fz = group_sum<L>(fz);
                if (vir && live && g == 0) add_sym(v, (double)qa.x, (double)qa.y, (double)qa.z, fx, fy, fz, 1.0);
                fx *= kFixUnit; fy *= kFixUnit; fz *= kFixUnit;
            } else {
                const double4 pa = a.pos2[i];
                const bool pxy = p.ivol == 0 || p.ivol == 1 || p.ivol == 4 || p.ivol == 2;
                const bool pz = p.ivol == 0 || p.ivol == 1 || p.ivol == 4 || p.ivol == 5;
                for (int e0 = g; e0 < ne; e0 += BF * L) {
                    int ee[BF];
#pragma unroll
                    for (int u = 0; u < BF; ++u) {
                        const int e = e0 + u * L;
                        ee[u] = e < ne ? a.alist[(size_t)e * stride + i] : -1;
                    }
                    double4 qq[BF];
#pragma unroll
                    for (int u = 0; u < BF; ++u) qq[u] = a.pos2[ee[u] != -1 ? (ee[u] & kIdMask) : i];
#pragma unroll
                    for (int u = 0; u < BF; ++u) {
                        if (ee[u] == -1) continue;
                        const double4 q = qq[u];
                        const double ux = pa.x - q.x, uy = pa.y - q.y, uz = pa.z - q.z;
                        const double mx = pxy ? round(ux) : 0.0, my = pxy ? round(uy) : 0.0,
                                     mz = pz ? round(uz) : 0.0;
                        const double dx = __dsub_rn(ux, mx), dy = __dsub_rn(uy, my), dz = __dsub_rn(uz, mz);
                        const double rx = b[0] * dx + b[3] * dy + b[6] * dz;
                        const double ry = b[1] * dx + b[4] * dy + b[7] * dz;
                        const double rz = b[2] * dx + b[5] * dy + b[8] * dz;
                        const double r = sqrt(rx * rx + ry * ry + rz * rz);
                        const double rr = 1.0 / r;
                        const double4 tv = tab_r4(tab, t, r);
                        const double fp = -tv.y * rr - (tv.w * pa.w + tv.w * q.w) * rr;
                        const double gx = dx * fp, gy = dy * fp, gz = dz * fp;
                        fx += gx; fy += gy; fz += gz;
                        if (ee[u] & kOwnBit) v[0] += tv.x;
                        if (vir) {
                            const bool excluded = !(ma > 0.1 || ma + a.mass[ee[u] & kIdMask] > 0.1);
                            if (mx != 0.0 || my != 0.0 || mz != 0.0 || excluded)
                                add_sym(v, excluded ? ux : mx, excluded ? uy : my, excluded ? uz : mz, gx, gy, gz,
                                        -0.5);
                        }
                    }
                }
                fx = group_sum<L>(fx); fy = group_sum<L>(fy); fz = group_sum<L>(fz);
                if (vir && live && g == 0) add_sym(v, pa.x, pa.y, pa.z, fx, fy, fz, 1.0);
            }
            if (live && g == 0) {
                if (last && a.store) { a.f[i] = fx; a.f[nm + i] = fy; a.f[2 * nm + i] = fz; }
                // velocity Verlet second half (src/quench_m.F90:606-622), previous tgid
                const double *tg = s.box.tgid;
                const double hx = u1[0] + w2[0], hy = u1[1] + w2[1], hz = u1[2] + w2[2];
                if (!(zn == 0 || ma < 0.1)) {
                    double s0 = 0.0, s1 = 0.0, s2 = 0.0;
                    if (p.ivol == 0) {
                        s0 = tg[0] * u1[0] + tg[3] * u1[1] + tg[6] * u1[2];
                        s1 = tg[1] * u1[0] + tg[4] * u1[1] + tg[7] * u1[2];
                        s2 = tg[2] * u1[0] + tg[5] * u1[1] + tg[8] * u1[2];
                    }
                    if (p.ivol == 4) s2 = tg[8] * u1[2];
                    w2[0] = del * fx - 0.5 * s0; w2[1] = del * fy - 0.5 * s1; w2[2] = del * fz - 0.5 * s2;
#pragma unroll
                    for (int k = 0; k < 3; ++k) a.x2[k * nm + i] = w2[k];
                }
                u1[0] = hx + w2[0]; u1[1] = hy + w2[1]; u1[2] = hz + w2[2];
#pragma unroll
                for (int k = 0; k < 3; ++k) a.x1[k * nm + i] = u1[k];
                if (drift) {
                    // the next step's first half (k_drift)
                    q0.x = q0.x + (u1[0] + w2[0]); q0.y = q0.y + (u1[1] + w2[1]); q0.z = q0.z + (u1[2] + w2[2]);
                    a.pos[i] = q0;
                    const int4 qn = make_int4(fix32(q0.x), fix32(q0.y), fix32(q0.z), 0);
                    a.posq[i] = qn;
                    d2 = fmaxf(d2, fix_disp2(bs, qn, xb));
                    if (kin && zn != 0) kin_moment(k6, ma, u1[0], u1[1], u1[2]);
                }
            }
        }
        if (MIXED) {   // the virial moments were summed in fixed-point units^2
#pragma unroll
            for (int k = 1; k < 7; ++k) v[k] *= kFixUnit * kFixUnit;
        }
        if (vir) warp_columns<7>(s, kB_F, v);
        else warp_columns<1>(s, kB_F, v);
        if (drift) {
            if (kin) warp_columns<6>(s, kB_K, k6);
            warp_column_max(s, kB_Max, d2);
        }
        if (!end_piece(a, s, epoch, (vir ? 0x7fu : 1u) | (drift && kin ? 0x1f80u : 0u) | (drift ? 1u << kB_Max : 0u),
                       false, buf))
            return;
    }
    // the box for the launches that follow: every block has read it before the last barrier
    if (blockIdx.x == 0) box_store(a.box, s.box);
}

// update_therm_avs of a step, with piece A's grouping of the atoms (the run's
// blocks, lane 0 of every group of `lanes`); the last block to finish sums the
// blocks and stores what follows (therm_store).  rec may be null.
__global__ void __launch_bounds__(kRunThreads)
k_run_therm(Params p, RunArgs a, int lanes, int32_t *__restrict__ ticket) {
    __shared__ RunShared s;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, nw = blockDim.x >> 5;
    const int g = tid & (lanes - 1), per_block = blockDim.x / lanes, per_round = gridDim.x * per_block;
    box_load(s.box, a.box);
    __syncthreads();
    if (warp == 0) warp_therm_prep(p, s, lane);
    __syncthreads();
    double vt[3] = {0.0, 0.0, 0.0};
    for (int i = blockIdx.x * per_block + tid / lanes; i < p.nm; i += per_round) {
        if (g != 0 || a.znum[i] == 0) continue;
        therm_terms(vt, s.box.th_tgid, s.box.b0, s.box.th_cof, a.mass[i], a.x1[i], a.x1[p.nm + i], a.x1[2 * p.nm + i],
                    a.x2[i], a.x2[p.nm + i], a.x2[2 * p.nm + i]);
    }
    warp_columns<3>(s, kA_T, vt);
    __syncthreads();
    if (tid < 3) {                                    // end_piece's order
        double x = s.warp[0][kA_T + tid];
        for (int q = 1; q < nw; ++q) x = x + s.warp[q][kA_T + tid];
        column(a, 0, kColT + tid)[blockIdx.x] = x;
    }
    if (!last_block(ticket)) return;
    if (warp != 0) return;
    double s3[3];
#pragma unroll
    for (int k = 0; k < 3; ++k) s3[k] = reduce_col(a, 0, kColT + k);
    BoxState &B = *a.box;
    if (lane < 9) {                                   // as warp_therm_prep left them
        B.tg[lane] = s.tmp[lane]; B.tgdot[lane] = s.tmp[9 + lane]; B.tginv[lane] = s.tmp[18 + lane];
        B.tgid[lane] = s.box.th_tgid[lane];
        B.th_tgid[lane] = s.box.th_tgid[lane]; B.th_cof[lane] = s.box.th_cof[lane];
    }
    if (lane != 0) return;
    double r[kThermoRec];
    step_record(p, s.box.b0, s.box.b1, s3, s.box.pe, r);
    if (a.rec)
        for (int k = 0; k < kThermoRec; ++k) a.rec[(size_t)kThermoRec * (size_t)a.rec0 + k] = r[k];
    B.ke = r[0]; B.te = r[2]; B.h = r[3]; B.th = r[4]; B.vol = r[5]; B.s1 = r[6]; B.s2 = r[7]; B.s3 = r[8];
    B.temp = r[9]; B.boxke = r[10];
    if (s.box.status) B.status = s.box.status;
}

using RunKernel = void (*)(Params, Tables, RunArgs);

template <bool MIXED>
RunKernel run_kernel(int lanes) {
    switch (lanes) {
    case 16: return k_run<MIXED, 16>;
    case 8: return k_run<MIXED, 8>;
    case 4: return k_run<MIXED, 4>;
    case 2: return k_run<MIXED, 2>;
    default: return k_run<MIXED, 1>;
    }
}

size_t run_smem(const Tables &t, bool mixed) {
    const size_t emb = (size_t)kRunEmb * sizeof(double2);
    return mixed ? 2 * (size_t)t.nr * sizeof(float4) + (size_t)((t.nr + 1) & ~1) * sizeof(float2) + emb
                 : (size_t)t.nr * (sizeof(double4) + sizeof(double2)) + emb;
}

}  // namespace

// Lanes per atom, threads per block and blocks of a run: the most lanes that
// still give every atom its group at once, and the atoms spread over all SMs.
static void run_shape(int nm, int &lanes, int &threads, int &blocks) {
    lanes = 16;
    while (lanes > 1 && (long long)nm * lanes > (long long)kRunBlocks * kRunThreads) lanes >>= 1;
    const long long want = ((long long)nm * lanes + kRunBlocks - 1) / kRunBlocks;
    threads = (int)((want + 31) / 32 * 32);
    threads = threads < 128 ? 128 : (threads > kRunThreads ? kRunThreads : threads);
    const long long nb = ((long long)nm * lanes + threads - 1) / threads;
    blocks = (int)(nb < kRunBlocks ? nb : kRunBlocks);
}

// A run keeps one block of at most 512 threads per SM (its box algebra, list
// builds and both pair pieces share the registers), the launched passes up to
// 1024.  Against those passes (us per step, NPT, launched / run): mixed 54,000
// atoms 46.2 / 32.8, 71,874 48.4 / 36.1, 78,608 52.6 / 53.9, 85,750 54.9 / 54.7,
// 93,312 55.1 / 55.1, 109,744 54.9 / 55.8, 128,000 68.7 / 56.2, 148,176 70.9 /
// 57.6, 159,014 74.1 / 76.2; FP64 54,000 53.6 / 44.2, 71,874 55.4 / 48.8, 78,608
// 69.0 / 78.2, 101,306 72.2 / 79.8.  So runs are taken while every atom has a
// thread of its own, and in mixed precision, whose pair terms are shorter, up to
// two atoms per thread: just past one the second round is half empty and the
// two forms are equal to 2 %, so the rule has no gap there.
bool run_applies(const Params &p, const Tables &t, bool mixed) {
    // the whole grid has to be resident: a partition of the device takes the launches
    int dev = 0, sms = 0;
    if (cudaGetDevice(&dev) != cudaSuccess ||
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || sms < kRunBlocks)
        return false;
    return p.nm <= (mixed ? 2 : 1) * kRunBlocks * kRunThreads && !t.exact && !p.atomstress && (p.ivol == 0 || p.ivol == 1 || p.ivol == 4) &&
           run_smem(t, mixed) <= 200 * 1024;
}

size_t run_scratch_bytes() { return 2 * (size_t)kCols * kRunBlocks * sizeof(double) +
           (size_t)(2 * kRunMaxSteps + 2) * kBarStride * sizeof(unsigned long long); }

static RunArgs run_args(DeviceState &d, double *rec, int rec0) {
    RunArgs a = {};
    a.pos = d.pos; a.pos2 = d.pos2; a.posq = d.posq; a.posq2 = d.posq2; a.box = d.box;
    a.nlist = d.nlist; a.numn = d.numn; a.rlist = d.rlist; a.numr = d.numr;
    a.olist = d.olist; a.out_cnt = d.out_cnt; a.mlist = d.mlist; a.mid_cnt = d.mid_cnt;
    a.alist = d.alist; a.pair_cnt = d.pair_cnt; a.xout = d.xout; a.xbuild = d.xbuild; a.xhalf = d.xhalf;
    a.mass = d.mass; a.del2 = d.del2; a.znum = d.znum; a.x1 = d.x1; a.x2 = d.x2; a.f = d.f;
    a.rho = d.rho; a.afrho = d.afrho; a.dafrho = d.dafrho;
    a.part = d.run_scratch; a.bar = reinterpret_cast<unsigned long long *>(d.run_scratch + 2 * (size_t)kCols * kRunBlocks);
    a.flags = d.flags; a.rec = rec; a.rec0 = rec0;
    return a;
}

int launch_run(DeviceState &d, const Params &p, const Tables &t, bool mixed, double rmid, double rcut, double rout,
               int m, int h0, int h1, int therm, double *rec, int rec0, int store, RunWait wait, cudaStream_t s) {
    int lanes, threads, blocks;
    run_shape(p.nm, lanes, threads, blocks);
    RunArgs a = run_args(d, rec, rec0);
    a.wait = wait;
    a.rmid = rmid; a.rcut = rcut; a.rout = rout;
    a.m = m; a.h0 = h0; a.h1 = h1; a.therm = therm; a.store = store;
    RunKernel k = mixed ? run_kernel<true>(lanes) : run_kernel<false>(lanes);
    const size_t smem = run_smem(t, mixed);
    cudaError_t e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e == cudaSuccess) e = cudaMemsetAsync(a.bar, 0, (size_t)(h1 - h0 + 1) * kBarStride * sizeof(unsigned long long), s);
    if (e != cudaSuccess) return (int)e;
    Params pp = p;
    Tables tt = t;
    void *args[] = {&pp, &tt, &a};
    return (int)cudaLaunchCooperativeKernel((const void *)k, dim3((unsigned)blocks), dim3((unsigned)threads), args, smem,
                                            s);
}

void launch_run_therm(DeviceState &d, const Params &p, double *rec, int k, cudaStream_t s) {
    int lanes, threads, blocks;
    run_shape(p.nm, lanes, threads, blocks);
    k_run_therm<<<blocks, threads, 0, s>>>(p, run_args(d, rec, k), lanes, d.flags + 14);
}

}  // namespace moldy
