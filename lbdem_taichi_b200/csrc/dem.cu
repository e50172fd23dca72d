// DEM sub-step on the GPU (DEMSolver.run_simulation, demsolver.py:848-862).
//
// Broad phase: the reference hashes cells of size 4*r_max with a Morton code
// into a 2^20..2^22 table and probes each particle's own cell plus the seven
// cells of its octant (bpcd.py:114-152), proposing pairs i < j.  Here the same
// cells are kept in a dense grid (no hash) and probed with the same octant
// rule, which proposes the same pairs whenever distinct cells do not alias in
// the reference's hash (checked on the host).
//
// Cells keep fixed-capacity particle lists filled by the binning atomics, so
// no scan is needed.  A sub-step has a contact phase (eight lanes per particle:
// candidate pairs j > i with contact history owned by i, and the six walls;
// forces go to accumulators) and an integration (accumulated + body + fluid
// force, improved Verlet, quaternion update, contact-list compaction, binning
// of the new positions into the other half of the counts).  Many sub-steps run
// as one launch: k_dem_flow with a workspace (a particle waits for the
// particles it can touch), else one block, one cluster or a cooperative grid;
// otherwise two launches per sub-step, k_contacts and k_integrate.
// FP64 throughout; compiled with -fmad=false, so that every operation rounds as
// it is written.  The integration follows the reference's order; the contact law
// is rearranged (one root for both dampings, the transpose of a rotation for its
// inverse, the spring set by the friction ratio) to the same value within
// roundings.
#include <float.h>
#include <math.h>
#include <stdlib.h>
#include <string.h>

#include <cooperative_groups.h>
#include <mutex>

#include "common.cuh"

namespace cg = cooperative_groups;

namespace lbdem {

struct M3 {
    double m[3][3];
};

// Quotients and square roots without branches: the hardware's approximation of
// the reciprocal or reciprocal root (PTX rcp.approx / rsqrt.approx.ftz.f64,
// about 22 bits), two Newton-Raphson steps, and Markstein's correction of the
// quotient or root by its fused remainder ("Computation of elementary functions
// on the IBM RISC System/6000 processor", 1990).  A contact has half a dozen of
// them, one after another in a chain that nothing hides, and the library forms
// branch for special values, so that not even independent ones overlap.
// Results are those of IEEE division and root for normal arguments whose
// reciprocal and quotient are normal too (but for cases within 1e-8 ulp of a
// tie).  A zero or infinite divisor gives what division gives (a frozen sphere
// may have an infinite mass).
__device__ __forceinline__ double rcp64(double x) {
    double a, r;
    asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(a) : "d"(x));
    const bool normal = fabs(a) <= DBL_MAX && a != 0.0;   // (tested beside the steps, not after them)
    r = fma(a, fma(-x, a, 1.0), a);
    r = fma(r, fma(-x, r, 1.0), r);
    return normal ? r : a;
}
// a / b given r, 1 / b to an ulp or two
__device__ __forceinline__ double div64(double a, double b, double r) {
    const double q = a * r;
    const bool normal = fabs(q) <= DBL_MAX && r != 0.0;
    const double c = fma(fma(-b, q, a), r, q);
    return normal ? c : q;
}
__device__ __forceinline__ double div64(double a, double b) { return div64(a, b, rcp64(b)); }
__device__ __forceinline__ double rsqrt64(double x) {
    double r;
    asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(r) : "d"(x));
    r = fma(0.5 * r, fma(-x * r, r, 1.0), r);
    return fma(0.5 * r, fma(-x * r, r, 1.0), r);
}
// 1 / sqrt(x) to half an ulp: the last step with the rounding error of x r
__device__ __forceinline__ double rsqrt64_round(double x) {
    double r;
    asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(r) : "d"(x));
    r = fma(0.5 * r, fma(-x * r, r, 1.0), r);
    const double s = x * r, e = fma(-fma(x, r, -s), r, fma(-s, r, 1.0));
    return fma(0.5 * r, e, r);
}
// root of x given r = rsqrt64(x); of 0 and of infinity, x
__device__ __forceinline__ double sqrt64(double x, double r) {
    const double s = x * r, c = fma(0.5 * r, fma(-s, s, x), s);
    return r == r || x < 0.0 ? c : x;
}
__device__ __forceinline__ double sqrt64(double x) { return sqrt64(x, rsqrt64(x)); }

__device__ __forceinline__ void cross3(const double *a, const double *b, double *o) {
    const double t0 = a[1] * b[2] - a[2] * b[1], t1 = a[2] * b[0] - a[0] * b[2], t2 = a[0] * b[1] - a[1] * b[0];
    o[0] = t0; o[1] = t1; o[2] = t2;
}
__device__ __forceinline__ double dot3(const double *a, const double *b) { return a[0] * b[0] + a[1] * b[1] + a[2] * b[2]; }
__device__ __forceinline__ void mv(const M3 &M, const double *v, double *o) {
    double t[3];
    for (int r = 0; r < 3; ++r) t[r] = M.m[r][0] * v[0] + M.m[r][1] * v[1] + M.m[r][2] * v[2];
    o[0] = t[0]; o[1] = t[1]; o[2] = t[2];
}
// R^T v: the inverse of a rotation (the reference inverts the matrix)
__device__ __forceinline__ void mtv(const M3 &M, const double *v, double *o) {
    for (int r = 0; r < 3; ++r) o[r] = M.m[0][r] * v[0] + M.m[1][r] * v[1] + M.m[2][r] * v[2];
}
__device__ M3 inv3(const M3 &A) {
    const double(*a)[3] = A.m;
    const double det = a[0][0] * (a[1][1] * a[2][2] - a[2][1] * a[1][2]) -
                       a[1][0] * (a[0][1] * a[2][2] - a[2][1] * a[0][2]) +
                       a[2][0] * (a[0][1] * a[1][2] - a[1][1] * a[0][2]);
    const double id = 1.0 / det;
    M3 o;
    for (int i = 0; i < 3; ++i)
        for (int j = 0; j < 3; ++j)
            o.m[j][i] = id * (a[(i + 1) % 3][(j + 1) % 3] * a[(i + 2) % 3][(j + 2) % 3] -
                              a[(i + 2) % 3][(j + 1) % 3] * a[(i + 1) % 3][(j + 2) % 3]);
    return o;
}

// rotation taking unit vector a onto +x (demsolver.py:686-701, :757-773)
__device__ M3 rot_to_x(const double *a) {
    const double b[3] = {1.0, 0.0, 0.0};
    double v[3];
    cross3(a, b, v);
    const double s2 = dot3(v, v);
    const double c = dot3(a, b);
    M3 R;
    for (int i = 0; i < 3; ++i)
        for (int j = 0; j < 3; ++j) R.m[i][j] = 0.0;
    if (s2 < 1e-24) {
        if (c > 0.0) {
            R.m[0][0] = R.m[1][1] = R.m[2][2] = 1.0;
        } else {
            R.m[0][0] = -1.0; R.m[1][1] = 1.0; R.m[2][2] = -1.0;
        }
    } else {
        const double vx[3][3] = {{0.0, -v[2], v[1]}, {v[2], 0.0, -v[0]}, {-v[1], v[0], 0.0}};
        const double coef = div64(1.0 - c, s2);
        for (int r = 0; r < 3; ++r)
            for (int q = 0; q < 3; ++q) {
                double acc = 0.0;
                for (int t = 0; t < 3; ++t) acc += (coef * vx[r][t]) * vx[t][q];
                R.m[r][q] = ((r == q ? 1.0 : 0.0) + vx[r][q]) + acc;
            }
    }
    return R;
}

constexpr int SLOTS_IN_REGS = 8;    // contact slots whose partners are fetched with the particle state

struct DemArgs {
    lbdem_dem d;
    int ncell;
    int parity;
    // Hertz constants of a contact, [0] particle-particle, [1] particle-wall
    // (hertz.py:45-97, 99-153), computed once per launch on the host: with
    // x = sqrt(Rs delta) and y = sqrt(x ms), stiffnesses kn x and kt x,
    // dampings gn y and gt y
    double hz_kn[2], hz_kt[2], hz_gn[2], hz_gt[2];
};

__device__ __forceinline__ int cell_index(const lbdem_dem &d, int cx_, int cy_, int cz_) {
    // grid covers reference cells -1 .. gdim-2 per axis
    const int gx = cx_ + 1, gy = cy_ + 1, gz = cz_ + 1;
    if (gx < 0 || gy < 0 || gz < 0 || gx >= d.gdim[0] || gy >= d.gdim[1] || gz >= d.gdim[2]) return -1;
    return (gz * d.gdim[1] + gy) * d.gdim[0] + gx;
}

__device__ __forceinline__ void ref_cell(const lbdem_dem &d, const double *p, int *ijk) {
    // bpcd.py:191-194
    for (int a = 0; a < 3; ++a) ijk[a] = (int)floor((p[a] - d.bp_min[a]) / d.cell_size);
}

// Bin particle i into its reference cell: the atomic rank is its slot in the
// cell's fixed-capacity list (no scan needed).
__device__ __forceinline__ void bin_particle(const lbdem_dem &d, int i, int32_t *count) {
    int ijk[3];
    ref_cell(d, d.pos + 3 * i, ijk);
    const int c = cell_index(d, ijk[0], ijk[1], ijk[2]);
    if (c < 0) {
        atomicOr(d.status, (int)LBDEM_ST_GRID_OVERFLOW);
        return;
    }
    const int rank = atomicAdd(count + c, 1);
    if (rank < d.cell_cap) d.cell_list[(size_t)c * d.cell_cap + rank] = i;
    else atomicOr(d.status, (int)LBDEM_ST_CELL_OVERFLOW);
}

__global__ void k_bin(const __grid_constant__ DemArgs A) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= A.d.n) return;
    bin_particle(A.d, i, A.d.cell_count + (size_t)A.parity * A.ncell);
}

// ------------------------------- contact laws ------------------------------
// hertz.py:45-97 / linear.py:43-101 (particle-particle), hertz.py:99-153 /
// linear.py:103-152 (particle-wall).  `wall` selects the wall variant; Rs and
// ms are the effective radius and mass (pair_effective).  The damping factors
// of both directions share one root (DemArgs).
__device__ __forceinline__ void pair_effective(double rad_i, double rad_j, double mass_i, double mass_j, double &Rs,
                                               double &ms) {
    Rs = rcp64(rcp64(rad_i) + rcp64(rad_j));
    ms = rcp64(rcp64(mass_i) + rcp64(mass_j));
}
__device__ __forceinline__ void contact_force(const DemArgs &A, double Rs, double ms, bool wall, double *shear,
                                              double delta_n, const double *vc, double *F) {
    const lbdem_dem &d = A.d;
    const double gap = -1 * delta_n;
    const double dt = d.dt;
    double inc[3] = {vc[0] * dt, vc[1] * dt, vc[2] * dt};
    inc[0] = 0.0;
    double kt, gt, F0, mu;
    const int tj = wall ? 1 : 0;
    mu = wall ? d.mu[1] : d.mu[0];
    if (d.model == 0) {
        const double x = sqrt64(Rs * delta_n), y = sqrt64(x * ms);
        const double kn = A.hz_kn[tj] * x, gn = A.hz_gn[tj] * y;
        kt = A.hz_kt[tj] * x;
        gt = A.hz_gt[tj] * y;
        F0 = -kn * gap - gn * vc[0];
    } else {
        double kns, kss, dpn, dps;
        dpn = d.dpn[0];
        dps = d.dps[0];
        if (wall) {
            kns = d.kn[0]; kss = d.ks[0];
        } else {
            kns = 0.5 * d.kn[0]; kss = 0.5 * d.ks[0];   // two equal springs in series
        }
        const double c = 2. * sqrt64(kns * ms);
        const double Cn = dpn * c;
        const double Ct = dps * c;
        kt = kss;
        gt = Ct;
        F0 = -kns * gap - Cn * vc[0];
    }
    for (int a = 0; a < 3; ++a) shear[a] += inc[a];
    const double ts[3] = {-kt * shear[0], -kt * shear[1], -kt * shear[2]};
    const double tl = sqrt64(dot3(ts, ts));
    F[0] = F0;
    if (tl >= mu * F0 && tl > 0.0) {
        // sliding: the spring is set to the friction limit, F = -kt shear
        const double ratio = div64(mu * F0, tl);
        shear[1] *= ratio;
        shear[2] *= ratio;
        F[1] = -kt * shear[1];
        F[2] = -kt * shear[2];
    } else {
        F[1] = ts[1] - gt * vc[1];
        F[2] = ts[2] - gt * vc[2];
    }
}

__device__ __forceinline__ void periodic_delta(const lbdem_dem &d, const double *pi, const double *pj, double *dv) {
    // demsolver.py:483-512
    for (int a = 0; a < 3; ++a) {
        dv[a] = pj[a] - pi[a];
        if (d.periodic[a]) {
            const double L = d.dom_max[a] - d.dom_min[a];
            if (dv[a] > 0.5 * L) dv[a] -= L;
            else if (dv[a] < -0.5 * L) dv[a] += L;
        }
    }
}

// State of particle i held in registers by its contact lanes.
struct PState {
    double p[3], v[3], w[3], rad, mass;
};

// The evaluated part of resolve(i, j) (demsolver.py:676-740) for a touching
// pair, on values in registers: dv is the minimum-image vector i -> j, len its
// length and il the reciprocal of that, sh the pair's shear history (updated).
// Gives the contact point, the force in the contact frame, the lever arms and
// the force on j (that on i is its exact negative).
__device__ __forceinline__ void pair_force(const DemArgs &A, const double *pi, const double *vi, const double *wi,
                                           double rad_i, const double *vj, const double *wj, double Rs, double ms,
                                           const double *dv, double len, double il, double gap, double *sh, double *cp_out,
                                           double *F_out, double *ri, double *rj, double *Fj) {
    const double a[3] = {div64(dv[0], len, il), div64(dv[1], len, il), div64(dv[2], len, il)};
    const M3 R = rot_to_x(a);
    const double delta_n = -gap;
    for (int t = 0; t < 3; ++t) {
        const double cp = pi[t] + a[t] * (rad_i - delta_n);
        cp_out[t] = cp;
        ri[t] = cp - pi[t];
        rj[t] = cp - (pi[t] + dv[t]);
    }
    double vci[3], vcj[3], dvc[3], vc[3];
    cross3(wi, ri, vci);
    cross3(wj, rj, vcj);
    for (int t = 0; t < 3; ++t) {
        vci[t] += vi[t];
        vcj[t] += vj[t];
        dvc[t] = vcj[t] - vci[t];
    }
    mv(R, dvc, vc);
    double F[3];
    contact_force(A, Rs, ms, false, sh, delta_n, vc, F);
    for (int t = 0; t < 3; ++t) F_out[t] = F[t];
    mtv(R, F, Fj);
}

// resolve(i, j) (demsolver.py:638-740); forces on i accumulated in Fi/Mi,
// forces on j added atomically.  hk: i's first contact slots (the partner of
// an active slot, -1 for an inactive one) as they were when the sub-step
// started (only i's lanes touch i's slots, each for its own partner).
__device__ __forceinline__ void resolve_pair(const DemArgs &A, int i, const PState &P, int n_i, const int *hk,
                                             int j, double *Fi_acc, double *Mi_acc) {
    const lbdem_dem &d = A.d;
    const size_t base = (size_t)i * d.maxc;
    // partner state: all loads issued together
    double pj[3], vj[3], wj[3];
    for (int t = 0; t < 3; ++t) {
        pj[t] = d.pos[3 * j + t];
        vj[t] = d.vel[3 * j + t];
        wj[t] = d.omega[3 * j + t];
    }
    const double rad_j = d.radius[j], mass_j = d.mass[j];
    int off = -1;
    const int nreg = min(n_i, min(d.maxc, SLOTS_IN_REGS));
#pragma unroll
    for (int o = SLOTS_IN_REGS - 1; o >= 0; --o)   // lowest matching slot wins, as a forward search
        if (o < nreg && hk[o] == j) off = o;
    if (off < 0)
        for (int o = SLOTS_IN_REGS; o < n_i && o < d.maxc; ++o)
            if (d.cf_j[base + o] == j && d.cf_active[base + o]) {
                off = o;
                break;
            }
    double dv[3];
    periodic_delta(d, P.p, pj, dv);
    const double d2 = dot3(dv, dv), il = rsqrt64(d2), len = sqrt64(d2, il);
    const double gap = len - P.rad - rad_j;
    bool eval = false;
    if (off >= 0) {
        if (gap < 0) eval = true;
        else d.cf_active[base + off] = 0;
    } else if (gap < 0) {
        // append_contact_offset (demsolver.py:352-359); several lanes of the
        // same particle may append in one sub-step
        off = n_i + atomicAdd(d.cf_add + i, 1);
        if (off >= d.maxc) {
            atomicOr(d.status, (int)LBDEM_ST_CONTACT_OVERFLOW);
            return;
        }
        d.cf_j[base + off] = j;
        d.cf_active[base + off] = 1;
        for (int a = 0; a < 3; ++a)
            d.cf_shear[3 * (base + off) + a] = d.cf_pos[3 * (base + off) + a] = d.cf_force[3 * (base + off) + a] = 0.0;
        eval = true;
    }
    if (!eval) return;
    const size_t s = base + off;
    double sh[3] = {d.cf_shear[3 * s], d.cf_shear[3 * s + 1], d.cf_shear[3 * s + 2]};
    double ri[3], rj[3], Fj[3], Mi[3], Mj[3], Rs, ms;
    pair_effective(P.rad, rad_j, P.mass, mass_j, Rs, ms);
    pair_force(A, P.p, P.v, P.w, P.rad, vj, wj, Rs, ms, dv, len, il, gap, sh, d.cf_pos + 3 * s, d.cf_force + 3 * s, ri,
               rj, Fj);
    const double Fi[3] = {-Fj[0], -Fj[1], -Fj[2]};
    cross3(ri, Fi, Mi);
    cross3(rj, Fj, Mj);
    for (int t = 0; t < 3; ++t) {
        d.cf_shear[3 * s + t] = sh[t];
        Fi_acc[t] += Fi[t];
        Mi_acc[t] += Mi[t];
        atomicAdd(d.acc_force + 3 * j + t, Fj[t]);
        atomicAdd(d.acc_moment + 3 * j + t, Mj[t]);
    }
}

// evaluate_wall (demsolver.py:742-807) on values in registers: sh is the wall
// contact's shear history (updated), cp and F receive the contact point and
// the force in the contact frame.
__device__ __forceinline__ void wall_force(const DemArgs &A, const PState &P, int w, double *sh, double *cp, double *F,
                                           double *Fi_acc, double *Mi_acc) {
    const lbdem_dem &d = A.d;
    const double *nrm = d.wall_n + 3 * w;
    const M3 R = rot_to_x(nrm);
    const double *p = P.p;
    const double delta_n = (dot3(p, nrm) - d.wall_d[w]) + P.rad;
    const double distance = P.rad - delta_n;
    double ri[3];
    for (int t = 0; t < 3; ++t) {
        ri[t] = distance * nrm[t];
        cp[t] = p[t] + ri[t];
    }
    double vci[3], m[3], vc[3];
    cross3(P.w, ri, vci);
    for (int t = 0; t < 3; ++t) m[t] = -(vci[t] + P.v[t]);
    mv(R, m, vc);
    contact_force(A, P.rad, P.mass, true, sh, delta_n, vc, F);
    const double mF[3] = {-F[0], -F[1], -F[2]};
    double Fi[3], Mi[3];
    mtv(R, mF, Fi);
    cross3(ri, Fi, Mi);
    for (int t = 0; t < 3; ++t) {
        Fi_acc[t] += Fi[t];
        Mi_acc[t] += Mi[t];
    }
}

__device__ void wall_contact(const DemArgs &A, int i, const PState &P, int w, double *Fi_acc, double *Mi_acc) {
    const lbdem_dem &d = A.d;
    const size_t s = (size_t)i * 6 + w;
    double sh[3] = {d.wcf_shear[3 * s], d.wcf_shear[3 * s + 1], d.wcf_shear[3 * s + 2]}, cp[3], F[3];
    wall_force(A, P, w, sh, cp, F, Fi_acc, Mi_acc);
    for (int t = 0; t < 3; ++t) {
        d.wcf_pos[3 * s + t] = cp[t];
        d.wcf_shear[3 * s + t] = sh[t];
        d.wcf_force[3 * s + t] = F[t];
    }
}

// Eight lanes per particle: lane k probes the k-th cell of the reference's
// probe list (own cell + octant, bpcd.py:133-142) and, for k < 6, wall k
// (demsolver.py:809-838); the lanes' forces on the particle are summed with
// shuffles before one atomic per component.
// One lane of the contact phase: lane k of particle i = tid / 8.  All 32 lanes
// of the warp must call it together (shuffle reduction over groups of 8).
// WRAP: also probe around the particle's periodic images (lbdem_dem.wrap_pairs).
template <bool WRAP>
__device__ __forceinline__ void contact_lane(const DemArgs &A, const int32_t *count, int tid) {
    const lbdem_dem &d = A.d;
    const int i = tid >> 3, k = tid & 7;
    const bool act = i < d.n;
    double Fi[3] = {0.0, 0.0, 0.0}, Mi[3] = {0.0, 0.0, 0.0};
    if (act) {
        // particle state, contact-slot snapshot and wall flag fetched together
        PState P;
        for (int t = 0; t < 3; ++t) {
            P.p[t] = d.pos[3 * i + t];
            P.v[t] = d.vel[3 * i + t];
            P.w[t] = d.omega[3 * i + t];
        }
        P.rad = d.radius[i];
        P.mass = d.mass[i];
        const int n_i = d.cfn[i];   // slots in use when the sub-step started
        const size_t base = (size_t)i * d.maxc;
        int hk[SLOTS_IN_REGS];
#pragma unroll
        for (int o = 0; o < SLOTS_IN_REGS; ++o) {
            const bool in = o < d.maxc;
            const int pj = in ? d.cf_j[base + o] : -1, act_o = in ? d.cf_active[base + o] : 0;
            hk[o] = act_o ? pj : -1;
        }
        const bool wall_lane = k < 6 && !d.wall_periodic[k];
        const int wact = wall_lane ? d.wcf_active[(size_t)i * 6 + k] : 0;
        // the reference's probe of lane k around a position (own cell + octant)
        auto probe = [&](const double q[3]) {
            int ijk[3], dd[3];
            ref_cell(d, q, ijk);
            for (int a = 0; a < 3; ++a) {
                const double center = (ijk[a] + 0.5) * d.cell_size + d.bp_min[a];
                dd[a] = (q[a] > center) ? 1 : -1;
            }
            const int ox = (k == 1 || k == 5 || k == 6 || k == 7) ? dd[0] : 0;
            const int oy = (k == 2 || k == 4 || k == 6 || k == 7) ? dd[1] : 0;
            const int oz = (k == 3 || k == 4 || k == 5 || k == 7) ? dd[2] : 0;
            const int c = cell_index(d, ijk[0] + ox, ijk[1] + oy, ijk[2] + oz);
            if (c >= 0) {
                const int n = min(count[c], d.cell_cap);
                const int32_t *lst = d.cell_list + (size_t)c * d.cell_cap;
                for (int t = 0; t < n; ++t) {
                    const int j = lst[t];
                    if (j > i) resolve_pair(A, i, P, n_i, hk, j, Fi, Mi);
                }
            }
        };
        if constexpr (!WRAP) {
            // the union of the eight probed cells' lists (own cell + octant, in
            // the reference's order), shared round-robin by the particle's eight
            // lanes so that a crowded cell does not make one lane the phase's
            // last: lane k takes candidates k, k + 8, ... of the concatenation
            int ijk[3], dd[3];
            ref_cell(d, P.p, ijk);
            for (int a = 0; a < 3; ++a) {
                const double center = (ijk[a] + 0.5) * d.cell_size + d.bp_min[a];
                dd[a] = (P.p[a] > center) ? 1 : -1;
            }
            int cidx[8], pre[8], total = 0;   // cell and exclusive prefix of the counts (static indices only)
#pragma unroll
            for (int kk = 0; kk < 8; ++kk) {
                const int ox = (kk == 1 || kk == 5 || kk == 6 || kk == 7) ? dd[0] : 0;
                const int oy = (kk == 2 || kk == 4 || kk == 6 || kk == 7) ? dd[1] : 0;
                const int oz = (kk == 3 || kk == 4 || kk == 5 || kk == 7) ? dd[2] : 0;
                cidx[kk] = cell_index(d, ijk[0] + ox, ijk[1] + oy, ijk[2] + oz);
                pre[kk] = total;
                total += cidx[kk] >= 0 ? min(count[cidx[kk]], d.cell_cap) : 0;
            }
            for (int t = k; t < total; t += 8) {
                // the last probed cell whose first index is <= t holds candidate t
                int cc = cidx[0], bb = 0;
#pragma unroll
                for (int kk = 1; kk < 8; ++kk)
                    if (t >= pre[kk]) { cc = cidx[kk]; bb = pre[kk]; }
                const int j = d.cell_list[(size_t)cc * d.cell_cap + (t - bb)];
                if (j > i) resolve_pair(A, i, P, n_i, hk, j, Fi, Mi);
            }
        } else {
            // the particle and its periodic images when it lies within one
            // broad-phase cell of a periodic face; the pair geometry is the
            // minimum image either way (periodic_delta)
            double sh[3] = {0.0, 0.0, 0.0};
            int nimg[3] = {1, 1, 1};
            for (int a = 0; a < 3; ++a) {
                if (!d.periodic[a]) continue;
                const double L = d.dom_max[a] - d.dom_min[a];
                if (P.p[a] < d.dom_min[a] + d.cell_size) { sh[a] = L; nimg[a] = 2; }
                else if (P.p[a] > d.dom_max[a] - d.cell_size) { sh[a] = -L; nimg[a] = 2; }
            }
            for (int ia = 0; ia < nimg[0]; ++ia)
                for (int ja = 0; ja < nimg[1]; ++ja)
                    for (int ka = 0; ka < nimg[2]; ++ka) {
                        const double q[3] = {P.p[0] + ia * sh[0], P.p[1] + ja * sh[1], P.p[2] + ka * sh[2]};
                        probe(q);
                    }
        }
        if (wall_lane) {
            const int w = k;
            const size_t s = (size_t)i * 6 + w;
            const double sep = -(dot3(P.p, d.wall_n + 3 * w) - d.wall_d[w]);
            if (wact) {
                if (sep > P.rad) d.wcf_active[s] = 0;
                else wall_contact(A, i, P, w, Fi, Mi);
            } else if (sep <= P.rad) {
                d.wcf_active[s] = 1;
                for (int t = 0; t < 3; ++t) d.wcf_shear[3 * s + t] = d.wcf_pos[3 * s + t] = d.wcf_force[3 * s + t] = 0.0;
                wall_contact(A, i, P, w, Fi, Mi);
            }
        }
    }
#pragma unroll
    for (int off = 1; off < 8; off <<= 1)
        for (int t = 0; t < 3; ++t) {
            Fi[t] += __shfl_xor_sync(0xffffffffu, Fi[t], off);
            Mi[t] += __shfl_xor_sync(0xffffffffu, Mi[t], off);
        }
    if (act && k == 0)
        for (int t = 0; t < 3; ++t) {
            atomicAdd(d.acc_force + 3 * i + t, Fi[t]);
            atomicAdd(d.acc_moment + 3 * i + t, Mi[t]);
        }
}

template <bool WRAP>
__global__ void __launch_bounds__(128) k_contacts(const __grid_constant__ DemArgs A) {
    grid_dependency();
    contact_lane<WRAP>(A, A.d.cell_count + (size_t)A.parity * A.ncell, blockIdx.x * blockDim.x + threadIdx.x);
}

// quaternion to rotation matrix (demsolver/utils.py:34-61)
__device__ M3 quat2rot(const double *q) {
    const double w2 = q[0] * q[0], i2 = q[1] * q[1], j2 = q[2] * q[2], k2 = q[3] * q[3];
    const double twoij = 2.0 * q[1] * q[2], twoik = 2.0 * q[1] * q[3], twojk = 2.0 * q[2] * q[3];
    const double twoiw = 2.0 * q[1] * q[0], twojw = 2.0 * q[2] * q[0], twokw = 2.0 * q[3] * q[0];
    M3 r;
    r.m[0][0] = w2 + i2 - j2 - k2; r.m[0][1] = twoij - twokw; r.m[0][2] = twojw + twoik;
    r.m[1][0] = twoij + twokw; r.m[1][1] = w2 - i2 + j2 - k2; r.m[1][2] = twojk - twoiw;
    r.m[2][0] = twoik - twojw; r.m[2][1] = twojk + twoiw; r.m[2][2] = w2 - i2 - j2 + k2;
    return r;
}

// Angular acceleration (demsolver.py:590-613) R^-1 I^-1 (R M - (R w) x I (R w)).
// For a multiple of the unit tensor -- every sphere -- it is M / I whatever the
// orientation, which takes the quaternion and eight dependent products out of
// a sub-step's chain; other tensors (the field is the user's) take the general
// form.
__device__ __forceinline__ bool inertia_iso(const double I[9]) {
    return I[0] == I[4] && I[0] == I[8] && I[1] == 0.0 && I[2] == 0.0 && I[3] == 0.0 && I[5] == 0.0 && I[6] == 0.0 &&
           I[7] == 0.0;
}
__device__ __noinline__ void angular_general(const double *q, const double *w, const double *mom, const double *inertia,
                                             double *alpha) {
    const M3 Rm = quat2rot(q);
    M3 I;
    for (int r = 0; r < 3; ++r)
        for (int c = 0; c < 3; ++c) I.m[r][c] = inertia[3 * r + c];
    double ml[3], wl[3], Iw[3], cw[3], rhs[3], wdl[3];
    mv(Rm, mom, ml);
    mv(Rm, w, wl);
    mv(I, wl, Iw);
    cross3(wl, Iw, cw);
    for (int t = 0; t < 3; ++t) rhs[t] = ml[t] - cw[t];
    mv(inv3(I), rhs, wdl);
    mv(inv3(Rm), wdl, alpha);
}

// Euler rotation update (demsolver.py:614-636) on values already in registers:
// w (3), wd (3, the previous angular acceleration) and the new one; q (4).
__device__ __forceinline__ void spin_update(double dt, double w[3], double wd[3], const double alpha[3]) {
    for (int t = 0; t < 3; ++t) w[t] += 0.5 * (wd[t] + alpha[t]) * dt;
    for (int t = 0; t < 3; ++t) wd[t] = alpha[t];
}
__device__ __forceinline__ void quat_update(double dt, double q[4], const double w[3]) {
    const double dq0 = -0.5 * (q[1] * w[0] + q[2] * w[1] + q[3] * w[2]);
    const double dq1 = +0.5 * (q[0] * w[0] - q[3] * w[1] + q[2] * w[2]);
    const double dq2 = +0.5 * (q[3] * w[0] + q[0] * w[1] + q[1] * w[2]);
    const double dq3 = +0.5 * (-q[2] * w[0] + q[1] * w[1] + q[0] * w[2]);
    q[0] += dq0 * dt; q[1] += dq1 * dt; q[2] += dq2 * dt; q[3] += dq3 * dt;
    // within 3.5 half-ulps of q / |q|, as a root and a division would be, which
    // are the longest chain of a lone particle's sub-step: they took 10 of them
    // from 13.0 to 14.1 us, this from 12.7 to 13.3
    const double il = rsqrt64_round((q[0] * q[0] + q[1] * q[1]) + (q[2] * q[2] + q[3] * q[3]));
    for (int t = 0; t < 4; ++t) q[t] *= il;
}

__device__ __forceinline__ void wrap_position(const lbdem_dem &d, double *p) {
    // demsolver.py:451-480
    for (int a = 0; a < 3; ++a) {
        if (!d.periodic[a]) continue;
        const double L = d.dom_max[a] - d.dom_min[a];
        if (p[a] > d.dom_max[a]) p[a] = p[a] - L;
        else if (p[a] < d.dom_min[a]) p[a] = p[a] + L;
    }
}

// update (demsolver.py:514-589), translation on values in registers; the
// position is not wrapped yet.  imass: rcp64(mass).
__device__ __forceinline__ void translate_update(double dt, int fixed, double mass, double imass, const double force[3],
                                                 double p[3], double v[3], double acc[3]) {
    if (fixed) {
        for (int t = 0; t < 3; ++t) p[t] += v[t] * dt;
        return;
    }
    double a[3];
    for (int t = 0; t < 3; ++t) a[t] = div64(force[t], mass, imass);
    for (int t = 0; t < 3; ++t) v[t] += 0.5 * (acc[t] + a[t]) * dt;
    for (int t = 0; t < 3; ++t) p[t] += v[t] * dt + 0.5 * a[t] * (dt * dt);
    for (int t = 0; t < 3; ++t) acc[t] = a[t];
}

__device__ void integrate_particle(const lbdem_dem &d, int ncell, int parity, int i, int role);
__device__ __forceinline__ void integrate_unit(const lbdem_dem &d, int ncell, int parity, int u);

__global__ void __launch_bounds__(128) k_integrate(const __grid_constant__ DemArgs A) {
    grid_dependency();
    const lbdem_dem &d = A.d;
    const int tid = blockIdx.x * blockDim.x + threadIdx.x;
    // clear the counts consumed by this sub-step (the other half receives the new binning)
    int32_t *used = d.cell_count + (size_t)A.parity * A.ncell;
    for (int c = tid; c < A.ncell; c += gridDim.x * blockDim.x) used[c] = 0;
    if (tid < 3 * d.n) integrate_unit(d, A.ncell, A.parity, tid);
}

// late_clear_state / remove_inactive_contact (demsolver.py:371-386, 431-436):
// slots are only moved when an inactive one precedes an active one.  Returns
// the number of active slots among the first `used`.
__device__ __forceinline__ int compact_slots(const lbdem_dem &d, int i, int used) {
    const size_t base = (size_t)i * d.maxc;
    int act[SLOTS_IN_REGS];
#pragma unroll
    for (int o = 0; o < SLOTS_IN_REGS; ++o) act[o] = o < d.maxc ? d.cf_active[base + o] : 0;
    const int cnt = min(used, d.maxc);
    int w_ = 0;
    auto keep = [&](int o) {
        if (w_ != o) {
            const size_t dd = base + w_, ss = base + o;
            d.cf_j[dd] = d.cf_j[ss];
            d.cf_active[dd] = 1;
            for (int t = 0; t < 3; ++t) {
                d.cf_shear[3 * dd + t] = d.cf_shear[3 * ss + t];
                d.cf_pos[3 * dd + t] = d.cf_pos[3 * ss + t];
                d.cf_force[3 * dd + t] = d.cf_force[3 * ss + t];
            }
        }
        ++w_;
    };
#pragma unroll
    for (int o = 0; o < SLOTS_IN_REGS; ++o)
        if (o < cnt && act[o]) keep(o);
    for (int o = SLOTS_IN_REGS; o < cnt; ++o)
        if (d.cf_active[base + o]) keep(o);
    for (int o = w_; o < cnt; ++o) d.cf_active[base + o] = 0;
    return w_;
}

__device__ void integrate_particle(const lbdem_dem &d, int ncell, int parity, int i, int role) {
    const double dt = d.dt;
    const int frozen = d.freeze[i], fixed = d.fixvel[i];
    if (role == 0) {
        // clear_state (demsolver.py:422-429) + contacts, then apply_body_force (:437-448): the force;
        // update (demsolver.py:514-589): translation; then the binning for the next sub-step.  Every
        // input is fetched before any store, so the loads overlap.
        double af[3], ffl[3], p[3], v[3], acc[3];
        for (int t = 0; t < 3; ++t) {
            af[t] = d.acc_force[3 * i + t];
            ffl[t] = d.force_fluid[3 * i + t];
            p[t] = d.pos[3 * i + t];
            v[t] = d.vel[3 * i + t];
            acc[t] = d.acc[3 * i + t];
        }
        const double mass = d.mass[i];
        double force[3];
        for (int t = 0; t < 3; ++t) {
            double f = af[t];
            f += mass * d.g[t];
            f += ffl[t];
            force[t] = f;
        }
        if (!frozen) {
            translate_update(dt, fixed, mass, rcp64(mass), force, p, v, acc);
            wrap_position(d, p);
        }
        for (int t = 0; t < 3; ++t) {
            d.acc_force[3 * i + t] = 0.0;
            d.force[3 * i + t] = force[t];
            d.pos[3 * i + t] = p[t];
            d.vel[3 * i + t] = v[t];
            d.acc[3 * i + t] = acc[t];
        }
        // bin the new position for the next sub-step
        int ijk[3];
        ref_cell(d, p, ijk);
        const int c = cell_index(d, ijk[0], ijk[1], ijk[2]);
        if (c < 0) {
            atomicOr(d.status, (int)LBDEM_ST_GRID_OVERFLOW);
            return;
        }
        int32_t *count = d.cell_count + (size_t)(parity ^ 1) * ncell;
        const int rank = atomicAdd(count + c, 1);
        if (rank < d.cell_cap) d.cell_list[(size_t)c * d.cell_cap + rank] = i;
        else atomicOr(d.status, (int)LBDEM_ST_CELL_OVERFLOW);
    } else if (role == 1) {
        // the moment and the Euler rotation update (demsolver.py:590-636)
        double am[3], mfl[3], w[3], wd[3], q[4], I[9];
        for (int t = 0; t < 3; ++t) {
            am[t] = d.acc_moment[3 * i + t];
            mfl[t] = d.moment_fluid[3 * i + t];
            w[t] = d.omega[3 * i + t];
            wd[t] = d.omega_dot[3 * i + t];
        }
        for (int t = 0; t < 4; ++t) q[t] = d.quat[4 * i + t];
        for (int t = 0; t < 9; ++t) I[t] = d.inertia[9 * i + t];
        double moment[3];
        for (int t = 0; t < 3; ++t) {
            double m = am[t];
            m += 0.0;
            m += mfl[t];
            moment[t] = m;
        }
        if (!frozen) {
            double alpha[3];
            if (inertia_iso(I)) {
                const double iI = rcp64(I[0]);
                for (int t = 0; t < 3; ++t) alpha[t] = moment[t] * iI;
            } else {
                angular_general(q, w, moment, I, alpha);
            }
            spin_update(dt, w, wd, alpha);
            quat_update(dt, q, w);
        }
        for (int t = 0; t < 3; ++t) {
            d.acc_moment[3 * i + t] = 0.0;
            d.moment[3 * i + t] = moment[t];
            d.omega[3 * i + t] = w[t];
            d.omega_dot[3 * i + t] = wd[t];
        }
        for (int t = 0; t < 4; ++t) d.quat[4 * i + t] = q[t];
    } else {
        const int w_ = compact_slots(d, i, d.cfn[i] + d.cf_add[i]);
        d.cfn[i] = w_;
        d.cf_add[i] = 0;
    }
}

// Integration of unit u of 3 n: role u / n (0 translation and binning, 1
// rotation, 2 contact-slot compaction) of particle u % n.  The three parts
// read and write disjoint state, so they run as three independent chains in
// different warps.
__device__ __forceinline__ void integrate_unit(const lbdem_dem &d, int ncell, int parity, int u) {
    const int role = u / d.n;
    integrate_particle(d, ncell, parity, u - role * d.n, role);
}

// All sub-steps of one call in ONE launch: a single thread-block cluster (up
// to 16 CTAs) grid-strides over the contact lanes, then over the particles;
// the two phases of every sub-step are separated by hardware cluster
// barriers (barrier.cluster arrive.release / wait.acquire), which order the
// global-memory writes of one phase before the reads of the next for every
// thread of the cluster.  Same per-lane/per-particle code as the two kernels.
template <bool WRAP>
__global__ void __launch_bounds__(512) k_dem_cluster(const __grid_constant__ DemArgs A, int nsub) {
    cg::cluster_group cl = cg::this_cluster();
    const lbdem_dem &d = A.d;
    const int nthr = (int)cl.num_threads();
    const int me = (int)cl.thread_rank();
    const int nlanes = 8 * d.n;
    for (int s = 0; s < nsub; ++s) {
        const int parity = (A.parity + s) & 1;
        const int32_t *count = d.cell_count + (size_t)parity * A.ncell;
        for (int base = 0; base < nlanes; base += nthr) contact_lane<WRAP>(A, count, base + me);
        cl.sync();
        int32_t *used = d.cell_count + (size_t)parity * A.ncell;
        for (int c = me; c < A.ncell; c += nthr) used[c] = 0;
        for (int u = me; u < 3 * d.n; u += nthr) integrate_unit(d, A.ncell, parity, u);
        cl.sync();
    }
}

// All sub-steps in one 128-thread block (at most 16 particles): the phases are
// separated by __syncthreads, which orders the block's global-memory writes of
// one phase before the reads of the next; the same per-lane/per-particle code
// without the cluster form's register cap (512 threads), so nothing spills.
template <bool WRAP>
__global__ void __launch_bounds__(128) k_dem_block(const __grid_constant__ DemArgs A, int nsub) {
    grid_dependency();
    const lbdem_dem &d = A.d;
    const int nthr = (int)blockDim.x, me = (int)threadIdx.x;
    const int nlanes = 8 * d.n;
    for (int s = 0; s < nsub; ++s) {
        const int parity = (A.parity + s) & 1;
        const int32_t *count = d.cell_count + (size_t)parity * A.ncell;
        for (int base = 0; base < nlanes; base += nthr) contact_lane<WRAP>(A, count, base + me);
        __syncthreads();
        int32_t *used = d.cell_count + (size_t)parity * A.ncell;
        for (int c = me; c < A.ncell; c += nthr) used[c] = 0;
        for (int u = me; u < 3 * d.n; u += nthr) integrate_unit(d, A.ncell, parity, u);
        __syncthreads();
    }
}

// ---------------------------------------------------------------------------
// All sub-steps of one call in ONE cooperative launch (without a workspace; also
// what k_dem_flow falls back to): every block of the grid is resident
// (cudaLaunchCooperativeKernel), the contact lanes and the particles are
// grid-strided, and the two phases of each sub-step are separated by a grid
// barrier.  The barrier is an arrival counter in caller-owned memory, zero at
// launch; its wait is bounded: after 2^22 looks (some seconds) it sets
// LBDEM_ST_WAIT_TIMEOUT and continues, so a fault can never hang the GPU.
// ---------------------------------------------------------------------------
__device__ __forceinline__ unsigned ld_acquire_gpu(const unsigned *p) {
    unsigned v;
    asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ void st_release_gpu(unsigned *p, unsigned v) {
    asm volatile("st.release.gpu.global.u32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}

__device__ __forceinline__ void red_release_gpu(unsigned *p, unsigned v) {
    asm volatile("red.release.gpu.global.add.u32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}

// Arrivals count up monotonically in sync[0] (zero at launch: k_dem_coop's caller
// zeroes it, k_dem_flow finds it as barrier_release left it): the k-th barrier is
// passed when the count reaches k * gridDim.x.  One release reduction per block
// and barrier (after the block barrier, which orders the block's writes of the
// phase before thread 0, so the release publishes them all), then polling with
// acquire loads; no reset.
__device__ __forceinline__ void grid_wait(uint32_t *sync, unsigned gen, int32_t *status) {
    if (gridDim.x > 1 && threadIdx.x == 0) {
        const unsigned target = gen * gridDim.x;
        unsigned it = 0;
        while (ld_acquire_gpu(sync) < target) {
            if (++it > (1u << 22)) {
                atomicOr(status, (int)LBDEM_ST_WAIT_TIMEOUT);
                break;
            }
            __nanosleep(32);
        }
    }
    __syncthreads();
}
__device__ __forceinline__ void grid_barrier(uint32_t *sync, unsigned &gen, int32_t *status) {
    __syncthreads();
    if (gridDim.x > 1 && threadIdx.x == 0) red_release_gpu(sync, 1u);
    gen += 1;
    grid_wait(sync, gen, status);
}

// The last block to leave a launch that used grid_barrier resets its counter
// (sync[1] counts the blocks past their last barrier); true in that thread.
__device__ __forceinline__ bool barrier_release(uint32_t *sync) {
    __syncthreads();
    if (threadIdx.x != 0 || atomicAdd(sync + 1, 1u) != gridDim.x - 1) return false;
    sync[0] = 0u;
    sync[1] = 0u;
    return true;
}

template <bool WRAP>
__global__ void __launch_bounds__(128, 1) k_dem_coop(const __grid_constant__ DemArgs A, int nsub) {
    const lbdem_dem &d = A.d;
    const int nthr = gridDim.x * blockDim.x;
    const int me = blockIdx.x * blockDim.x + threadIdx.x;
    const int nlanes = 8 * d.n;
    unsigned gen = 0;
    for (int s = 0; s < nsub; ++s) {
        const int parity = (A.parity + s) & 1;
        const int32_t *count = d.cell_count + (size_t)parity * A.ncell;
        for (int base = 0; base < nlanes; base += nthr) contact_lane<WRAP>(A, count, base + me);
        grid_barrier(d.sync, gen, d.status);
        int32_t *used = d.cell_count + (size_t)parity * A.ncell;
        for (int c = me; c < A.ncell; c += nthr) used[c] = 0;
        for (int u = me; u < 3 * d.n; u += nthr) integrate_unit(d, A.ncell, parity, u);
        grid_barrier(d.sync, gen, d.status);
    }
    barrier_release(d.sync);
}

// ---------------------------------------------------------------------------
// All sub-steps of one call in ONE launch without a grid barrier per sub-step:
// LPP lanes own a particle for the whole call, its state stays in registers (its
// pairs' data, indexed at run time, in local memory), and a particle waits only
// for the particles it can touch.
//
// What bounds the sub-steps is latency: two grid barriers and a chain of
// dependent loads (cell, list, partner, contact slot) per sub-step, for a few
// thousand threads.  But a particle moves a fraction of its radius per call,
// so the pairs that can touch during a chunk of sub-steps are known at its
// start, and most particles of a suspension have none.  Per chunk:
//   build   every particle's partners: gap <= m_i + m_j, m the displacement
//           that its velocity and known acceleration allow (times two) plus
//           FLOW_SLACK radii.  The test is symmetric bit for bit, so both sides
//           list the pair.  Shear histories of known contacts are copied to
//           registers on BOTH sides.
//   flow    a lane evaluates its pairs from the lower index's perspective (the
//           same arithmetic on the same values on both sides, so both copies of
//           the history agree) and keeps its own side's force: no atomics.
//           A particle with partners publishes its state after a sub-step as
//           nine 16-byte packets (value, sub-step) in one of two slots; a
//           partner polls those packets, which is wait and transfer in one
//           round trip.  Partners are at most one sub-step apart (each needs
//           the other's state), so two slots suffice.  A warp publishes before
//           it polls, and every warp is resident, so every wait ends; they are
//           bounded all the same.
//   commit  after a grid barrier: state, contact slots and broad-phase lists.
// Nothing is written before the commit, so a chunk whose assumptions fail -- a
// particle moved farther than m, more than FLOW_NBR partners, a full contact
// list, a particle leaving the grid or outside a periodic face, a slot in use
// that the two-phase form may drop -- is done by that form instead, in the same
// launch.
// 10 sub-steps, against the two-phase form (B200): 2000 spheres of a 256^3
// suspension, a fifth of them in contact, 44 us (106); one sphere 14 us alone and
// 18 between the kernels of a coupled step (60); others at flow_forms.  What
// bounds it now: FP64 latency of an isolated particle's sub-step 0.7 us, of one
// with a contact 1.9 us (half of it the exchange through L2), and 7 us (one
// block) to 12 of search, barrier and commit per call.
// ---------------------------------------------------------------------------
constexpr int FLOW_THREADS = 128;
constexpr int FLOW_NBR = 16;          // partners of a particle
constexpr int FLOW_CHUNK = 16;        // sub-steps between two partner searches
constexpr double FLOW_SLACK = 0.02;   // radii
constexpr int COOP_MIN_SUBSTEPS = 3;
// In more than one block, fewer sub-steps than this run the two-phase form: a
// partner search and commit cost 12-20 us (2000 / 10,000 particles: 29 / 46 us
// for one sub-step against 18 / 21, 29 / 48 for two against 26 / 40, 31 / 50
// for three against 35 / 59).
constexpr int FLOW_MIN_SUBSTEPS = 3;
// In one block (16 particles) the two-phase form needs no grid barrier, and a few
// sub-steps are the shorter by it where particles touch: particles apart /
// touching, two-phase against this form, us: one sub-step of 1, 8 and 16 particles
// 6.3 / 6.3, 6.7 / 6.9, 6.4 / 7.1 against 8.1 / 10.9, 9.7 / 20.7, 10.2 / 23.3; two
// of 1, 2, 8 and 16 11.0 / 10.7, 10.9 / 11.6, 11.4 / 11.3, 11.1 / 10.6 against 9.1
// / 12.0, 9.2 / 14.2, 10.6 / 22.9, 10.7 / 25.2; three of 8 and 16 15.9 / 16.6, 16.6
// / 18.0 against 11.0 / 24.0, 11.4 / 26.8; ten 49 / 42, 48 / 55 against 16 / 36, 17
// / 39.  With periodic images, whose cells the two-phase form looks up in every
// sub-step: one of 16 9.5 / 11.1 against 10.4 / 23.2, two 17.0 / 20.3 against 10.2
// / 24.7.
static int flow_min_one_block(const lbdem_dem *D) {
    return D->wrap_pairs || D->n <= 2 ? 2 : D->n <= 8 ? 3 : 4;
}
constexpr size_t FLOW_HEADER = 256;   // workspace: two failure words (by chunk parity), the epoch, the hold, then the packets
// After a chunk that failed, this many chunks at most go to the two-phase form
// without a search (1, 3, 7, ... while they keep failing; FlowHold): what breaks
// an assumption lasts -- a frozen particle outside a face, a large sphere amid
// small ones.  10 sub-steps of beds with such a particle, us, this / every chunk
// tried first / the cooperative or split form: 2000 spheres 186 / 273 / 181,
// 6000 310 / 482 / 182, 20,000 599 / 916 / 330 (the forms of 4 and 2 lanes per
// particle keep their grid for it).
constexpr unsigned FLOW_HOLD_MAX = 31;
constexpr int FLOW_STRIDE = 16;       // packets between two slots: no 128-byte line is polled and written for two
constexpr int FLOW_STATE = 9;         // doubles of a published state: position, velocity, angular velocity
constexpr int FLOW_TAGS = 2 * FLOW_CHUNK;   // tags of a chunk: no packet of an earlier chunk or call has one of them

struct FlowHold {
    unsigned left, length;   // chunks left to the two-phase form, and their number in all
};

struct FlowArgs {
    DemArgs A;
    unsigned char *work;
    int nsub;
};

__device__ __forceinline__ ulonglong2 *flow_packets(const FlowArgs &f, int i, int slot) {
    return reinterpret_cast<ulonglong2 *>(f.work + FLOW_HEADER) + ((size_t)i * 2 + slot) * FLOW_STRIDE;
}
// a packet is one 128-bit relaxed access: value and tag arrive together
__device__ __forceinline__ void packet_store(bool on, ulonglong2 *p, double v, unsigned long long tag) {
    const unsigned __int128 w = ((unsigned __int128)tag << 64) | (unsigned long long)__double_as_longlong(v);
    asm volatile("{\n .reg .pred q;\n setp.ne.u32 q, %2, 0;\n @q st.relaxed.gpu.global.b128 [%0], %1;\n}\n" ::"l"(p),
                 "q"(w), "r"((unsigned)on)
                 : "memory");
}
__device__ __forceinline__ void packet_load(const ulonglong2 *p, unsigned long long &v, unsigned long long &tag) {
    unsigned __int128 w;
    asm volatile("ld.relaxed.gpu.global.b128 %0, [%1];" : "=q"(w) : "l"(p) : "memory");
    v = (unsigned long long)w;
    tag = (unsigned long long)(w >> 64);
}
// one look at a partner's packets: true when all are of sub-step `tag`
__device__ __forceinline__ bool flow_look(const ulonglong2 *p, unsigned long long tag, double o[FLOW_STATE]) {
    bool ok = true;
#pragma unroll
    for (int c = 0; c < FLOW_STATE; ++c) {
        unsigned long long v, t;
        packet_load(p + c, v, t);
        ok = ok && t == tag;
        o[c] = __longlong_as_double((long long)v);
    }
    return ok;
}

// Displacement allowed to particle i during T: twice that of its velocity and
// of the body and fluid force, plus the slack that contacts may use.
__device__ __forceinline__ double flow_budget(const lbdem_dem &d, int i, double T, double rad, double mass) {
    // sums of magnitudes, in FP32: a bound needs no more, and FP32 divides in a few cycles
    float v = 0.f, a = 0.f, g = 0.f;
    for (int t = 0; t < 3; ++t) {
        v += fabsf((float)d.vel[3 * i + t]);
        a += fabsf((float)d.force_fluid[3 * i + t]);
        g += fabsf((float)d.g[t]);
    }
    const float Tf = (float)T;
    return (double)(2.f * Tf * (v + Tf * (a / (float)mass + g))) + FLOW_SLACK * rad;
}

// minimum-image vector pi -> pj (periodic_delta) and which periods it took:
// bits 2a (minus) and 2a + 1 (plus) of axis a
__device__ __forceinline__ int image_delta(const lbdem_dem &d, const double *pi, const double *pj, double *dv) {
    int m = 0;
    for (int a = 0; a < 3; ++a) {
        dv[a] = pj[a] - pi[a];
        if (d.periodic[a]) {
            const double L = d.dom_max[a] - d.dom_min[a];
            if (dv[a] > 0.5 * L) { dv[a] -= L; m |= 1 << (2 * a); }
            else if (dv[a] < -0.5 * L) { dv[a] += L; m |= 2 << (2 * a); }
        }
    }
    return m;
}

// Whether the broad phase proposes the pair (i, j), i the lower index: j's
// cell among i's own and its octant's (bpcd.py:133-142), or, with periodic
// images, those of i's images (contact_lane).
template <bool WRAP>
__device__ __noinline__ bool flow_proposed(const lbdem_dem &d, double px, double py, double pz, double ox, double oy,
                                           double oz) {
    const double pi[3] = {px, py, pz}, pj[3] = {ox, oy, oz};
    int cj[3];
    ref_cell(d, pj, cj);
    double sh[3] = {0.0, 0.0, 0.0};
    if (WRAP)
        for (int a = 0; a < 3; ++a) {
            if (!d.periodic[a]) continue;
            const double L = d.dom_max[a] - d.dom_min[a];
            if (pi[a] < d.dom_min[a] + d.cell_size) sh[a] = L;
            else if (pi[a] > d.dom_max[a] - d.cell_size) sh[a] = -L;
        }
    for (int im = 0; im < (WRAP ? 8 : 1); ++im) {
        bool in = true;
        for (int a = 0; a < 3; ++a) {
            const bool img = (im >> a) & 1;
            if (img && sh[a] == 0.0) in = false;
            const double q = pi[a] + (img ? sh[a] : 0.0);
            const int c = (int)floor((q - d.bp_min[a]) / d.cell_size);
            const double center = (c + 0.5) * d.cell_size + d.bp_min[a];
            const int o = cj[a] - c;
            in = in && (o == 0 || o == (q > center ? 1 : -1));
        }
        if (in) return true;
    }
    return false;
}

// Whether the broad phase may propose the pair (i, j), i the lower index, at
// some time while the two move by no more than mi and mj: flow_proposed over
// those ranges.  On an axis the probed cells of i are the two from
// floor((h - 1) / 2), h the half cell it lies in.  Near a periodic face, where
// a particle can wrap or gain an image, the axis counts as proposed.
template <bool WRAP>
__device__ __forceinline__ bool flow_may_propose(const lbdem_dem &d, int i, int j, double mi, double mj) {
    for (int a = 0; a < 3; ++a) {
        const double pi = d.pos[3 * i + a], pj = d.pos[3 * j + a];
        if (d.periodic[a]) {
            const double img = WRAP ? d.cell_size : 0.0;
            if (!(pi - mi >= d.dom_min[a] + img && pi + mi <= d.dom_max[a] - img && pj - mj >= d.dom_min[a] &&
                  pj + mj <= d.dom_max[a]))
                continue;
        }
        const double h = 0.5 * d.cell_size, x = pi - d.bp_min[a], y = pj - d.bp_min[a];
        const int lo = ((int)floor((x - mi) / h) - 1) >> 1, hi = ((int)floor((x + mi) / h) - 1) >> 1;
        if ((int)floor((y + mj) / d.cell_size) < lo || (int)floor((y - mj) / d.cell_size) > hi + 1) return false;
    }
    return true;
}

// Whether a lane's share of i's slots in use holds one whose partner is not among
// the nn listed and may be proposed within the chunk.
template <bool WRAP>
__device__ __forceinline__ bool flow_stale_slots(const lbdem_dem &d, int i, int k, int lanes, int used, int nn,
                                                 const int *list, double m, double T) {
    for (int o = k; o < min(used, d.maxc); o += lanes) {
        const size_t s = (size_t)i * d.maxc + o;
        if (!d.cf_active[s]) continue;
        const int j = d.cf_j[s];
        bool listed = false;
        for (int e = 0; e < nn; ++e) listed = listed || list[e] == j;
        if (!listed && flow_may_propose<WRAP>(d, i, j, m, flow_budget(d, j, T, d.radius[j], d.mass[j]))) return true;
    }
    return false;
}
// Called, as pair_effective in a chunk, so that the sub-steps' code stays together:
// between other kernels its instructions come from L2 each time, and a step of one
// settling sphere takes 39.6 us instead of 41.0.  With 2 lanes per particle this
// call costs spills (20,000 spheres 239 us, inline 233).
template <bool WRAP>
__device__ __noinline__ bool flow_stale_slots_called(const lbdem_dem &d, int i, int k, int lanes, int used, int nn,
                                                     const int *list, double m, double T) {
    return flow_stale_slots<WRAP>(d, i, k, lanes, used, nn, list, m, T);
}
__device__ __noinline__ void pair_effective_called(double rad_i, double rad_j, double mass_i, double mass_j, double &Rs,
                                                   double &ms) {
    pair_effective(rad_i, rad_j, mass_i, mass_j, Rs, ms);
}

// the two-phase form over the sub-steps of a chunk whose lists are binned in
// half `parity` (the body of k_dem_coop).  Inlined: called, it read every member
// of A through a generic pointer (2000 spheres 244 us instead of 183).
template <bool WRAP>
__device__ __forceinline__ void flow_two_phase(const DemArgs &A, int parity, int nsub, unsigned &gen) {
    const lbdem_dem &d = A.d;
    const int nthr = gridDim.x * blockDim.x, me = blockIdx.x * blockDim.x + threadIdx.x;
    for (int s = 0; s < nsub; ++s) {
        const int par = (parity + s) & 1;
        int32_t *count = d.cell_count + (size_t)par * A.ncell;
        for (int base = 0; base < 8 * d.n; base += nthr) contact_lane<WRAP>(A, count, base + me);
        grid_barrier(d.sync, gen, d.status);
        for (int c = me; c < A.ncell; c += nthr) count[c] = 0;
        for (int u = me; u < 3 * d.n; u += nthr) integrate_unit(d, A.ncell, par, u);
        grid_barrier(d.sync, gen, d.status);
    }
}

// One chunk: S sub-steps from the lists binned in half `parity`.  True when it
// failed: nothing was written then, and the lists are binned as before.
template <bool WRAP, int LPP>
__device__ __forceinline__ bool flow_chunk(const FlowArgs &f, int parity, int S, int chunk, unsigned long long epoch0,
                                           unsigned &gen) {
    constexpr int GPB = FLOW_THREADS / LPP;          // particles per block
    constexpr int K = FLOW_NBR / LPP;                // pairs per lane
    constexpr int NW = (6 + LPP - 1) / LPP;          // walls per lane
    __shared__ int s_cnt[GPB], s_list[GPB][FLOW_NBR];
    __shared__ double s_I[GPB][9];                   // inertia tensors
    const DemArgs &A = f.A;
    const lbdem_dem &d = A.d;
    const int nthr = gridDim.x * blockDim.x, me = blockIdx.x * blockDim.x + threadIdx.x;
    const int g = threadIdx.x / LPP, k = threadIdx.x % LPP;
    const int i = blockIdx.x * GPB + g;
    const bool act = i < d.n;
    const double rmax = 0.25 * d.cell_size;
    int *fail_words = reinterpret_cast<int *>(f.work);
    const unsigned long long tag0 = epoch0 + (unsigned long long)chunk * FLOW_TAGS;
    volatile int *fail = fail_words + (chunk & 1);
    int32_t *count = d.cell_count + (size_t)parity * A.ncell;
    // ------------------------------------------------------------ build
    PState P = {};
    double acc[3] = {}, wd[3] = {}, q[4] = {}, ffl[3] = {}, mfl[3] = {}, af[3] = {}, am[3] = {};
    double m = 0.0, imass = 0.0, iI = 0.0;
    int frozen = 1, fixed = 0, n_used = 0;
    bool bad = false, iso = true;
    if (k == 0) s_cnt[g] = 0;
    __syncwarp();
    if (act) {
        for (int t = 0; t < 3; ++t) {
            P.p[t] = d.pos[3 * i + t];
            P.v[t] = d.vel[3 * i + t];
            P.w[t] = d.omega[3 * i + t];
            acc[t] = d.acc[3 * i + t];
            wd[t] = d.omega_dot[3 * i + t];
            ffl[t] = d.force_fluid[3 * i + t];
            mfl[t] = d.moment_fluid[3 * i + t];
            af[t] = d.acc_force[3 * i + t];
            am[t] = d.acc_moment[3 * i + t];
        }
        for (int t = 0; t < 4; ++t) q[t] = d.quat[4 * i + t];
        P.rad = d.radius[i];
        P.mass = d.mass[i];
        frozen = d.freeze[i];
        fixed = d.fixvel[i];
        n_used = d.cfn[i];
        double I[9];
        for (int t = 0; t < 9; ++t) I[t] = d.inertia[9 * i + t];
        iso = inertia_iso(I);
        iI = rcp64(I[0]);
        imass = rcp64(P.mass);
        if (!iso && k == 0)
            for (int t = 0; t < 9; ++t) s_I[g][t] = I[t];
        const double T = S * d.dt, mcap = 0.25 * rmax;
        m = flow_budget(d, i, T, P.rad, P.mass);
        // cells that hold every possible partner: centres within reach, of
        // the particle and of its periodic images.  (rmax bounds a partner's
        // radius; one written above it later would be listed by its owner only.)
        bad = !(m <= mcap) || P.rad > rmax;
        const double reach = P.rad + rmax + m + mcap;
        // (a superset: a reciprocal and a slack do).  Per axis: n0 cells of
        // the particle from lo0, then n1 of its image from lo1
        const double icell = rcp64(d.cell_size);
        int lo0[3], lo1[3], n0[3], n1[3], code[3];
        for (int a = 0; a < 3; ++a) {
            const double x = P.p[a] - d.bp_min[a];
            bad = bad || !(x - m > -d.cell_size && x + m < (d.gdim[a] - 1) * d.cell_size);
            lo0[a] = max(-1, (int)floor((x - reach) * icell - 1e-9));
            n0[a] = max(0, min(d.gdim[a] - 2, (int)floor((x + reach) * icell + 1e-9)) - lo0[a] + 1);
            lo1[a] = n1[a] = code[a] = 0;
            if (!d.periodic[a]) continue;
            // The image within reach of the opposite face finds every partner only where both centres lie in
            // the box: of two across a face, the one outside would list the other and not be listed by it.
            // (An unwrapped packing's first call, or a frozen particle, which is never wrapped.)
            bad = bad || !(P.p[a] >= d.dom_min[a] && P.p[a] <= d.dom_max[a]);
            const double L = d.dom_max[a] - d.dom_min[a];
            double sh = 0.0;
            if (P.p[a] < d.dom_min[a] + reach) { sh = L; code[a] = 1 << (2 * a); }
            else if (P.p[a] > d.dom_max[a] - reach) { sh = -L; code[a] = 2 << (2 * a); }
            if (sh != 0.0) {
                lo1[a] = max(-1, (int)floor((x + sh - reach) * icell - 1e-9));
                n1[a] = max(0, min(d.gdim[a] - 2, (int)floor((x + sh + reach) * icell + 1e-9)) - lo1[a] + 1);
            }
        }
        const int nx = n0[0] + n1[0], nxy = nx * (n0[1] + n1[1]), tot = bad ? 0 : nxy * (n0[2] + n1[2]);
        const float inx = 1.f / (float)nx, inxy = 1.f / (float)nxy;
        auto consider = [&](int j, const double *pj, double rj, int image) {
            double dv[3];
            if (image_delta(d, P.p, pj, dv) != image) return;        // found through another image
            const double d2 = dot3(dv, dv), far = P.rad + rj + (m + mcap);
            if (!(d2 <= far * far)) return;
            const double near = P.rad + rj + (m + flow_budget(d, j, T, rj, d.mass[j]));
            if (!(d2 <= near * near)) return;
            const int at = atomicAdd(&s_cnt[g], 1);
            if (at < FLOW_NBR) s_list[g][at] = j;
            else bad = true;
        };
        for (int c0 = k; c0 < tot; c0 += 2 * LPP) {
            // two cells at a time: counts and first two entries in one round
            // trip, those particles' positions in a second
            int ci[2], nj[2], image[2], e[2][2];
            double pj[2][2][3], rj[2][2];
#pragma unroll
            for (int u = 0; u < 2; ++u) {
                const int c = c0 + u * LPP;
                ci[u] = image[u] = nj[u] = e[u][0] = e[u][1] = 0;
                if (c >= tot) continue;
                const int iz = (int)(((float)c + 0.5f) * inxy), r = c - iz * nxy;
                const int iy = (int)(((float)r + 0.5f) * inx), ix = r - iy * nx;
                const bool bx = ix >= n0[0], by = iy >= n0[1], bz = iz >= n0[2];
                image[u] = (bx ? code[0] : 0) | (by ? code[1] : 0) | (bz ? code[2] : 0);
                ci[u] = cell_index(d, bx ? lo1[0] + ix - n0[0] : lo0[0] + ix, by ? lo1[1] + iy - n0[1] : lo0[1] + iy,
                                   bz ? lo1[2] + iz - n0[2] : lo0[2] + iz);
                const int32_t *lst = d.cell_list + (size_t)ci[u] * d.cell_cap;
                nj[u] = count[ci[u]];
                e[u][0] = lst[0];
                e[u][1] = d.cell_cap > 1 ? lst[1] : 0;
            }
#pragma unroll
            for (int u = 0; u < 2; ++u) {
                bad = bad || nj[u] > d.cell_cap;
                nj[u] = min(nj[u], d.cell_cap);
#pragma unroll
                for (int t = 0; t < 2; ++t) {
                    if (t >= nj[u]) e[u][t] = i;
                    const int j = e[u][t];
                    for (int a = 0; a < 3; ++a) pj[u][t][a] = d.pos[3 * j + a];
                    rj[u][t] = d.radius[j];
                }
            }
#pragma unroll
            for (int u = 0; u < 2; ++u) {
#pragma unroll
                for (int t = 0; t < 2; ++t)
                    if (e[u][t] != i) consider(e[u][t], pj[u][t], rj[u][t], image[u]);
                for (int t = 2; t < nj[u]; ++t) {
                    const int j = d.cell_list[(size_t)ci[u] * d.cell_cap + t];
                    const double p[3] = {d.pos[3 * j], d.pos[3 * j + 1], d.pos[3 * j + 2]};
                    if (j != i) consider(j, p, d.radius[j], image[u]);
                }
            }
        }
    }
    __syncwarp();
    // this lane's pairs: partner, its constants, and the shear history of a
    // contact that the lower index already lists
    const int nn = act ? min(s_cnt[g], FLOW_NBR) : 0;
    int pj[K], pslot[K];                       // partner; slot of the lower index, -1: none yet
    unsigned pact = 0, pdirty = 0;             // bit e: pair e is in contact / was evaluated
    double prad[K], pRs[K], pms[K], psh[K][3], pcp[K][3], pF[K][3];
    int np = 0, matched = 0;
    for (int e = k; e < nn; e += LPP, ++np) {
        const int j = s_list[g][e], own = min(i, j), other = max(i, j);
        pj[np] = j;
        prad[np] = d.radius[j];
        pair_effective_called(P.rad, prad[np], P.mass, d.mass[j], pRs[np], pms[np]);
        const int no = min(d.cfn[own], d.maxc);
        int off = -1;
        for (int o = 0; o < no && off < 0; ++o)
            if (d.cf_j[(size_t)own * d.maxc + o] == other && d.cf_active[(size_t)own * d.maxc + o]) off = o;
        pslot[np] = off;
        for (int t = 0; t < 3; ++t) psh[np][t] = off >= 0 ? d.cf_shear[3 * ((size_t)own * d.maxc + off) + t] : 0.0;
        if (off >= 0) {
            pact |= 1u << np;
            matched += own == i;
        }
    }
    __syncwarp();
    for (int o = 1; o < LPP; o <<= 1) matched += __shfl_xor_sync(0xffffffffu, matched, o);
    const int np_most = __reduce_max_sync(0xffffffffu, np);
    const int room = d.maxc - (n_used - matched);     // slots for listed pairs
    // A slot in use whose partner is not listed: a contact that opened where the broad phase did not propose
    // the pair, or positions written since.  The two-phase form drops it when the pair is proposed again, so
    // where that can happen in this chunk it takes over; elsewhere the slot stays, as there.
    if (act && n_used > matched) {
        const double T = S * d.dt;
        if (LPP > 2 ? flow_stale_slots_called<WRAP>(d, i, k, LPP, n_used, nn, s_list[g], m, T)
                    : flow_stale_slots<WRAP>(d, i, k, LPP, n_used, nn, s_list[g], m, T))
            bad = true;
    }
    int wact = 0, wdirty = 0, wnear = 0;
    double wsh[NW][3], wcp[NW][3], wF[NW][3];
    for (int e = 0; e < NW; ++e) {
        const int w = k + e * LPP;
        if (!act || w >= 6 || d.wall_periodic[w]) continue;
        if (d.wcf_active[(size_t)i * 6 + w]) wact |= 1 << e;
        // walls within the particle's displacement (normals are unit vectors; any other length only widens it)
        const double *nrm = d.wall_n + 3 * w;
        const double sep = -(dot3(P.p, nrm) - d.wall_d[w]);
        if (((wact >> e) & 1) || !(sep > P.rad + m * (fabs(nrm[0]) + fabs(nrm[1]) + fabs(nrm[2])))) wnear |= 1 << e;
        for (int t = 0; t < 3; ++t) wsh[e][t] = d.wcf_shear[3 * ((size_t)i * 6 + w) + t];
    }
    if (bad) *fail = 1;
    // half a grid barrier: the lists may be cleared once every block has built
    __syncthreads();
    if (threadIdx.x == 0 && gridDim.x > 1) red_release_gpu(d.sync, 1u);
    ++gen;
    bool failed;
    {
        // -------------------------------------------------------- flow
        double D[3] = {0.0, 0.0, 0.0}, force[3], moment[3];
        bool lost = false, late = false;
        const bool walls = __any_sync(0xffffffffu, wnear != 0);
        for (int s = 0; s < S; ++s) {
            double F[3] = {0.0, 0.0, 0.0}, M[3] = {0.0, 0.0, 0.0};
            int held = 0, fresh = 0;
            bool hit = false;                         // this lane evaluated a contact
            for (int e = 0; e < np_most; ++e) {
                const bool have = e < np;
                const int j = have ? pj[e] : i;
                const bool own = i < j;
                double o[FLOW_STATE];
                if (s == 0) {
                    if (have)
                        for (int t = 0; t < 3; ++t) {
                            o[t] = d.pos[3 * j + t];
                            o[3 + t] = d.vel[3 * j + t];
                            o[6 + t] = d.omega[3 * j + t];
                        }
                } else {
                    // The warp polls as one: a lane spinning by itself leaves the warp split, and every
                    // later exchange between its lanes then costs hundreds of cycles (a contact between
                    // two SMs: 14,300 cycles per sub-step with a loop per lane).  Bounded: about 2^20 looks.
                    bool wait = have && !lost;
                    for (unsigned it = 0; __any_sync(0xffffffffu, wait); ++it) {
                        if (wait) {
                            const int failed = *fail;
                            wait = !flow_look(flow_packets(f, j, s & 1), tag0 + s, o);
                            if (wait && (failed || it >= (1u << 20))) {
                                late = late || !failed;
                                lost = true;          // the chunk has failed: no more waits
                                wait = false;
                            }
                        }
                    }
                }
                if (have && !lost) {
                    double lp[3], hp[3], dv[3];
                    for (int t = 0; t < 3; ++t) {
                        lp[t] = own ? P.p[t] : o[t];
                        hp[t] = own ? o[t] : P.p[t];
                    }
                    const int img = image_delta(d, lp, hp, dv);
                    const bool on = (pact >> e) & 1u;
                    held += own && on;
                    const double lr = own ? P.rad : prad[e], hr = own ? prad[e] : P.rad;
                    const double d2 = dot3(dv, dv), il = rsqrt64(d2), len = sqrt64(d2, il), gap = len - lr - hr;
                    // (the reference proposes no pair across a periodic face)
                    const bool proposed = WRAP || img == 0;
                    if (proposed && !(gap < 0) && on &&
                        flow_proposed<WRAP>(d, lp[0], lp[1], lp[2], hp[0], hp[1], hp[2]))
                        pact &= ~(1u << e);
                    if (proposed && gap < 0) {
                        double lv[3], lw[3], hv[3], hw[3], shr[3], cp[3], Fc[3], ri[3], rj[3], Fj[3], Ms[3];
                        for (int t = 0; t < 3; ++t) {
                            lv[t] = own ? P.v[t] : o[3 + t];
                            lw[t] = own ? P.w[t] : o[6 + t];
                            hv[t] = own ? o[3 + t] : P.v[t];
                            hw[t] = own ? o[6 + t] : P.w[t];
                            shr[t] = on ? psh[e][t] : 0.0;
                        }
                        fresh += own && !on;
                        pact |= 1u << e;
                        pdirty |= 1u << e;
                        pair_force(A, lp, lv, lw, lr, hv, hw, pRs[e], pms[e], dv, len, il, gap, shr, cp, Fc, ri, rj, Fj);
                        hit = true;
                        for (int t = 0; t < 3; ++t) {
                            psh[e][t] = shr[t];
                            pcp[e][t] = cp[t];
                            pF[e][t] = Fc[t];
                            ri[t] = own ? ri[t] : rj[t];
                            Fj[t] = own ? -Fj[t] : Fj[t];
                        }
                        cross3(ri, Fj, Ms);
                        for (int t = 0; t < 3; ++t) {
                            F[t] += Fj[t];
                            M[t] += Ms[t];
                        }
                    }
                }
                __syncwarp();
            }
            if (__any_sync(0xffffffffu, fresh != 0)) {
                // as the two-phase form counts: slots in use when the sub-step began, plus the new ones
                int used = held + fresh, any = fresh;
                for (int o = 1; o < LPP; o <<= 1) {
                    used += __shfl_xor_sync(0xffffffffu, used, o);
                    any += __shfl_xor_sync(0xffffffffu, any, o);
                }
                if (any && used > room) *fail = 1;
            }
            if (walls) {
                for (int e = 0; e < NW; ++e) {
                    const int w = k + e * LPP;
                    if (!((wnear >> e) & 1)) continue;
                    const double sep = -(dot3(P.p, d.wall_n + 3 * w) - d.wall_d[w]);
                    const bool on = (wact >> e) & 1;
                    if (on && sep > P.rad) {
                        wact &= ~(1 << e);
                        wdirty |= 1 << e;
                    } else if (on || sep <= P.rad) {
                        double shr[3], cp[3], Fc[3];
                        for (int t = 0; t < 3; ++t) shr[t] = on ? wsh[e][t] : 0.0;
                        wall_force(A, P, w, shr, cp, Fc, F, M);
                        hit = true;
                        for (int t = 0; t < 3; ++t) {
                            wsh[e][t] = shr[t];
                            wcp[e][t] = cp[t];
                            wF[e][t] = Fc[t];
                        }
                        wact |= 1 << e;
                        wdirty |= 1 << e;
                    }
                }
            }
            __syncwarp();
            const bool hits = __any_sync(0xffffffffu, hit);
            if (hits) {
#pragma unroll
                for (int o = 1; o < LPP; o <<= 1)
                    for (int t = 0; t < 3; ++t) {
                        F[t] += __shfl_xor_sync(0xffffffffu, F[t], o);
                        M[t] += __shfl_xor_sync(0xffffffffu, M[t], o);
                    }
            }
            // integration, by every lane of the particle alike (integrate_particle, roles 0 and 1); lanes
            // without a particle stay with their warp (theirs counts as frozen)
            for (int t = 0; t < 3; ++t) {
                double x = F[t] + (s == 0 ? af[t] : 0.0);
                x += P.mass * d.g[t];
                x += ffl[t];
                force[t] = x;
                moment[t] = M[t] + (s == 0 ? am[t] : 0.0) + mfl[t];
            }
            double x[3] = {P.p[0], P.p[1], P.p[2]}, y[3];
            if (!frozen) {
                translate_update(d.dt, fixed, P.mass, imass, force, P.p, P.v, acc);
                for (int t = 0; t < 3; ++t) y[t] = P.p[t];
                wrap_position(d, P.p);
                double alpha[3];
                if (iso)
                    for (int t = 0; t < 3; ++t) alpha[t] = moment[t] * iI;
                else
                    angular_general(q, P.w, moment, s_I[g], alpha);
                spin_update(d.dt, P.w, wd, alpha);
            }
            // publish at once; what no partner waits for comes after
            if (np_most > 0 && s + 1 < S) {
                ulonglong2 *out = flow_packets(f, i, (s + 1) & 1);
                const unsigned long long tag = tag0 + s + 1;
#pragma unroll
                for (int t = 0; t < 3; ++t) {
                    packet_store(nn > 0 && t % LPP == k, out + t, P.p[t], tag);
                    packet_store(nn > 0 && (3 + t) % LPP == k, out + 3 + t, P.v[t], tag);
                    packet_store(nn > 0 && (6 + t) % LPP == k, out + 6 + t, P.w[t], tag);
                }
            }
            if (!frozen) {
                quat_update(d.dt, q, P.w);
                for (int t = 0; t < 3; ++t) D[t] += y[t] - x[t];
                if (y[0] != P.p[0] || y[1] != P.p[1] || y[2] != P.p[2]) {
                    int c[3];
                    ref_cell(d, P.p, c);
                    if (cell_index(d, c[0], c[1], c[2]) < 0) *fail = 1;
                }
                if (!(dot3(D, D) <= 0.999 * (m * m))) *fail = 1;
            }
        }
        if (late) {
            atomicOr(d.status, (int)LBDEM_ST_WAIT_TIMEOUT);
            *fail = 1;
        }
        // every block has built by now: clear the lists it read
        grid_wait(d.sync, gen, d.status);
        for (int c = me; c < A.ncell; c += nthr) count[c] = 0;
        if (me == 0) fail_words[(chunk + 1) & 1] = 0;
        grid_barrier(d.sync, gen, d.status);
        failed = *fail != 0;
        if (!failed) {
            // -------------------------------------------------- commit
            const size_t base = (size_t)i * d.maxc;
            int drop = 0, born = 0;
            if (act) {
                if (k == 0) {
                    for (int t = 0; t < 3; ++t) {
                        d.pos[3 * i + t] = P.p[t];
                        d.vel[3 * i + t] = P.v[t];
                        d.acc[3 * i + t] = acc[t];
                        d.force[3 * i + t] = force[t];
                        d.acc_force[3 * i + t] = 0.0;
                    }
                    bin_particle(d, i, d.cell_count + (size_t)(parity ^ (S & 1)) * A.ncell);
                }
                if (k == LPP - 1) {
                    for (int t = 0; t < 3; ++t) {
                        d.omega[3 * i + t] = P.w[t];
                        d.omega_dot[3 * i + t] = wd[t];
                        d.moment[3 * i + t] = moment[t];
                        d.acc_moment[3 * i + t] = 0.0;
                    }
                    for (int t = 0; t < 4; ++t) d.quat[4 * i + t] = q[t];
                }
                for (int e = 0; e < NW; ++e) {
                    if (!((wdirty >> e) & 1)) continue;
                    const size_t s = (size_t)i * 6 + k + e * LPP;
                    d.wcf_active[s] = (wact >> e) & 1;
                    if ((wact >> e) & 1)
                        for (int t = 0; t < 3; ++t) {
                            d.wcf_shear[3 * s + t] = wsh[e][t];
                            d.wcf_pos[3 * s + t] = wcp[e][t];
                            d.wcf_force[3 * s + t] = wF[e][t];
                        }
                }
                // listed contacts in their slots; dropped ones leave gaps
                for (int e = 0; e < np; ++e) {
                    if (pj[e] < i) continue;
                    const bool on = (pact >> e) & 1u;
                    if (pslot[e] < 0) {
                        born += on;
                    } else if (!on) {
                        d.cf_active[base + pslot[e]] = 0;
                        drop = 1;
                    } else if ((pdirty >> e) & 1u) {
                        const size_t s = base + pslot[e];
                        for (int t = 0; t < 3; ++t) {
                            d.cf_shear[3 * s + t] = psh[e][t];
                            d.cf_pos[3 * s + t] = pcp[e][t];
                            d.cf_force[3 * s + t] = pF[e][t];
                        }
                    }
                }
            }
            // close the gaps, then append the new contacts in lane order
            int before = 0, all = born, drops = drop;
#pragma unroll
            for (int o = 1; o < LPP; o <<= 1) {
                const int x = __shfl_xor_sync(0xffffffffu, all, o);
                before += (k & o) ? x : 0;
                all += x;
                drops += __shfl_xor_sync(0xffffffffu, drops, o);
            }
            __syncwarp();
            int kept = n_used;
            if (act && k == 0 && drops) kept = compact_slots(d, i, n_used);
            __syncwarp();
            kept = __shfl_sync(0xffffffffu, kept, 0, LPP);
            if (act) {
                int at = kept + before;
                for (int e = 0; e < np; ++e) {
                    if (pj[e] < i || pslot[e] >= 0 || !((pact >> e) & 1u)) continue;
                    const size_t s = base + at++;
                    d.cf_j[s] = pj[e];
                    d.cf_active[s] = 1;
                    for (int t = 0; t < 3; ++t) {
                        d.cf_shear[3 * s + t] = psh[e][t];
                        d.cf_pos[3 * s + t] = pcp[e][t];
                        d.cf_force[3 * s + t] = pF[e][t];
                    }
                }
                if (k == 0 && (drops || all)) d.cfn[i] = kept + all;
            }
        } else {
            // the lists were cleared: bin the untouched positions again
            if (act && k == 0) bin_particle(d, i, count);
            grid_barrier(d.sync, gen, d.status);
        }
    }
    return failed;
}

// MB: resident blocks per SM that the registers are cut for (255 at 2, 168 at 3)
template <bool WRAP, int LPP, int MB>
__global__ void __launch_bounds__(FLOW_THREADS, MB) k_dem_flow(const __grid_constant__ FlowArgs f) {
    grid_dependency();
    const lbdem_dem &d = f.A.d;
    int *fail_words = reinterpret_cast<int *>(f.work);
    unsigned long long *epoch = reinterpret_cast<unsigned long long *>(f.work + 16);
    FlowHold *hold_word = reinterpret_cast<FlowHold *>(f.work + 24);
    const unsigned long long epoch0 = *epoch;
    FlowHold hold = *hold_word;               // (the same in every thread throughout)
    unsigned gen = 0;
    int parity = f.A.parity, done = 0, chunk = 0;
    while (done < f.nsub) {
        const int S = min(f.nsub - done, FLOW_CHUNK);
        // (expected, so that the two-phase form stays out of the sub-steps' code: a lone sphere 14.4 us otherwise, 14.1)
        bool failed = hold.left > 0;
        if (__builtin_expect(failed, 0)) {
            --hold.left;
            // (the next chunk's failure word, as flow_chunk clears it; all have read it: the last use was before a barrier)
            if (blockIdx.x == 0 && threadIdx.x == 0) fail_words[(chunk + 1) & 1] = 0;
        } else {
            failed = flow_chunk<WRAP, LPP>(f, parity, S, chunk, epoch0, gen);
            hold.length = failed ? min(2 * hold.length + 1, FLOW_HOLD_MAX) : 0;
            hold.left = hold.length;
        }
        if (__builtin_expect(failed, 0)) flow_two_phase<WRAP>(f.A, parity, S, gen);
        parity ^= S & 1;
        done += S;
        ++chunk;
        if (done < f.nsub && !failed) grid_barrier(d.sync, gen, d.status);
    }
    // leave the barrier and the failure words clear for the next launch
    if (gridDim.x == 1) {
        __syncthreads();
        if (threadIdx.x < 2) fail_words[threadIdx.x] = 0;
        if (threadIdx.x == 0) {
            *epoch = epoch0 + (unsigned long long)chunk * FLOW_TAGS;
            *hold_word = hold;
        }
    } else if (barrier_release(d.sync)) {
        fail_words[0] = fail_words[1] = 0;
        *epoch = epoch0 + (unsigned long long)chunk * FLOW_TAGS;
        *hold_word = hold;
    }
}

// The per-material Hertz constants of DemArgs, from
// hertz.py:45-97 (particle-particle: the restitution 0.5 (e + e)) and
// hertz.py:99-153 (particle-wall).
static void contact_constants(DemArgs &A) {
    const lbdem_dem &d = A.d;
    for (int tj = 0; tj < 2; ++tj) {
        const double Ys = 1.0 / ((1.0 - d.nu[0] * d.nu[0]) / d.E[0] + (1.0 - d.nu[tj] * d.nu[tj]) / d.E[tj]);
        const double Gs = 1.0 / (2.0 * (2.0 - d.nu[0]) * (1.0 + d.nu[0]) / d.E[0] +
                                 2.0 * (2.0 - d.nu[tj]) * (1.0 + d.nu[tj]) / d.E[tj]);
        const double e = tj == 0 ? 0.5 * (d.e[0] + d.e[0]) : d.e[1];
        const double lne = log(e);
        const double beta = lne / sqrt(lne * lne + M_PI * M_PI);
        A.hz_kn[tj] = 4.0 / 3.0 * Ys;
        A.hz_kt[tj] = 8.0 * Gs;
        A.hz_gn[tj] = -2.0 * beta * sqrt(5.0 / 6.0 * 2.0 * Ys);    // Sn = 2 Ys x
        A.hz_gt[tj] = -2.0 * beta * sqrt(5.0 / 6.0 * 8.0 * Gs);    // St = 8 Gs x
    }
}

static int check_dem(const lbdem_dem *D) {
    if (!D || D->n < 0 || D->maxc < 0 || !D->status) {
        set_error("dem: bad descriptor");
        return LBDEM_ERR_ARG;
    }
    if (D->n > 0 && (!D->pos || !D->vel || !D->cell_count ||
                     !D->cfn || !D->cf_add || !D->wcf_active || !D->acc_force || !D->acc_moment || !D->cell_list ||
                     D->cell_cap <= 0)) {
        set_error("dem: missing buffers");
        return LBDEM_ERR_ARG;
    }
    if (D->gdim[0] <= 0 || D->gdim[1] <= 0 || D->gdim[2] <= 0 || !(D->cell_size > 0.0)) {
        set_error("dem: bad broad-phase grid");
        return LBDEM_ERR_ARG;
    }
    if (D->wrap_pairs)
        for (int a = 0; a < 3; ++a)
            if (D->periodic[a] && D->dom_max[a] - D->dom_min[a] < 4.0 * D->cell_size) {
                // a pair must not be reachable both directly and through an image
                set_error("dem: periodic images need every periodic length >= 4 broad-phase cells (axis %d)", a);
                return LBDEM_ERR_ARG;
            }
    return LBDEM_OK;
}

}  // namespace lbdem

using namespace lbdem;

extern "C" {

// (Re)bin the current positions into the active half of cell_count.
int lbdem_dem_bin(lbdem_dem *D, void *stream) {
    int rc = check_dem(D);
    if (rc) return rc;
    if (D->n == 0) return LBDEM_OK;
    cudaStream_t st = (cudaStream_t)stream;
    DemArgs A;
    A.d = *D;
    A.ncell = D->gdim[0] * D->gdim[1] * D->gdim[2];
    A.parity = D->parity;
    if (cudaMemsetAsync(D->cell_count + (size_t)A.parity * A.ncell, 0, sizeof(int32_t) * A.ncell, st) != cudaSuccess)
        return check_launch("dem_bin memset");
    k_bin<<<(D->n + 127) / 128, 128, 0, st>>>(A);
    return check_launch("dem_bin");
}

static thread_local int g_dem_launches = 0;

// Cooperative-launch support, SM count and resident blocks per SM of the
// cooperative kernel (128 threads, no dynamic shared memory) on device `dev`:
// constant for a device, so looked up once per device and form (the host
// launch of every call would otherwise repeat three driver queries).
static bool coop_residency(int dev, int form, const void *kcoop, int &coop, int &nsm, int &per_sm) {
    constexpr int MAXDEV = 64;
    static std::mutex mu;
    static int cached[10][MAXDEV][3];   // form: k_dem_coop without / with images, then the forms of k_dem_flow likewise
    static bool have[10][MAXDEV] = {};
    if (dev < 0 || dev >= MAXDEV) return false;
    std::lock_guard<std::mutex> lock(mu);
    if (!have[form][dev]) {
        int c = 0, n = 0, p = 0;
        cudaDeviceGetAttribute(&c, cudaDevAttrCooperativeLaunch, dev);
        cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev);
        if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&p, kcoop, 128, 0) != cudaSuccess) {
            cudaGetLastError();
            return false;
        }
        cached[form][dev][0] = c;
        cached[form][dev][1] = n;
        cached[form][dev][2] = p;
        have[form][dev] = true;
    }
    coop = cached[form][dev][0];
    nsm = cached[form][dev][1];
    per_sm = cached[form][dev][2];
    return true;
}

int lbdem_dem_launches_last(void) { return g_dem_launches; }

// Forms of the one launch without per-sub-step barriers, in the order of
// preference: all particles must be resident at once, and the first form that
// allows it is taken (148 SMs: up to 4736, 9472, 14208 and 28416 particles).
// 11 sub-steps with the forms that still fit: 8000 spheres of a dense bed, all
// in contact, 101, 130 and 127 us (two-phase 250); 10,000 of a channel 76 and
// 87 us (two-phase 210).
struct FlowForm {
    int lanes;
    void (*kern[2])(const FlowArgs);   // without / with periodic images
};
constexpr int FLOW_FORMS = 4;
static const FlowForm flow_forms[FLOW_FORMS] = {
    {8, {k_dem_flow<false, 8, 2>, k_dem_flow<true, 8, 2>}},
    {4, {k_dem_flow<false, 4, 2>, k_dem_flow<true, 4, 2>}},
    {4, {k_dem_flow<false, 4, 3>, k_dem_flow<true, 4, 3>}},
    {2, {k_dem_flow<false, 2, 3>, k_dem_flow<true, 2, 3>}},
};

// The form for D's particles (index), or -1 where none applies.  Periodic axes
// must be longer than 2.5 broad-phase cells, so that no pair is near both
// directly and through an image.
static int flow_form(const lbdem_dem *D, int dev, int *blocks) {
    if (D->n > 1)
        for (int a = 0; a < 3; ++a)
            if (D->periodic[a] && !(D->dom_max[a] - D->dom_min[a] > 2.5 * D->cell_size)) return -1;
    const bool wrap = D->wrap_pairs != 0;
    for (int l = 0; l < FLOW_FORMS; ++l) {
        const int gpb = FLOW_THREADS / flow_forms[l].lanes, nb = (D->n + gpb - 1) / gpb;
        *blocks = nb;
        if (nb == 1) return l;
        int coop = 0, nsm = 0, per_sm = 0;
        if (!D->sync || !coop_residency(dev, 2 + 2 * l + wrap, (const void *)flow_forms[l].kern[wrap], coop, nsm, per_sm) || !coop)
            return -1;
        if (nb <= per_sm * nsm) return l;
    }
    return -1;
}

size_t lbdem_dem_flow_bytes(const lbdem_dem *D) {
    int dev = 0, nb = 0;
    if (check_dem(D) || D->n == 0 || cudaGetDevice(&dev) != cudaSuccess || flow_form(D, dev, &nb) < 0) return 0;
    return LBDEM_DEM_FLOW_BYTES(D->n);
}

int lbdem_dem_substeps_flow(lbdem_dem *D, int32_t nsub, void *work, void *stream) {
    int rc = check_dem(D);
    if (rc) return rc;
    const char *mode = getenv("LBDEM_DEM_KERNELS");
    int dev = 0, nb = 0, form = -1;
    cudaGetDevice(&dev);
    if (work && D->n > 0 && nsub > 0 && (!mode || strcmp(mode, "flow") == 0)) form = flow_form(D, dev, &nb);
    const int least = nb > 1 ? FLOW_MIN_SUBSTEPS : flow_min_one_block(D);
    // (the barrier's arrival counter must stay far from wrapping)
    if (form < 0 || (!mode && nsub < least) || 8ll * nsub * nb >= (1ll << 30))
        return lbdem_dem_substeps(D, nsub, stream);
    g_dem_launches = 0;
    FlowArgs f;
    f.A.d = *D;
    f.A.ncell = D->gdim[0] * D->gdim[1] * D->gdim[2];
    f.A.parity = D->parity;
    contact_constants(f.A);
    f.work = static_cast<unsigned char *>(work);
    f.nsub = nsub;
    cudaStream_t st = (cudaStream_t)stream;
    auto *kern = flow_forms[form].kern[D->wrap_pairs != 0];
    void *args[] = {&f};
    const int threads = nb > 1 ? FLOW_THREADS : (flow_forms[form].lanes * D->n + 31) / 32 * 32;
    const cudaError_t e = nb > 1 ? cudaLaunchCooperativeKernel((const void *)kern, dim3(nb), dim3(threads), args, 0, st)
                                 : launch_chained(kern, dim3(1), dim3(threads), 0, st, f);
    if (e != cudaSuccess) {
        cudaGetLastError();
        return lbdem_dem_substeps(D, nsub, stream);
    }
    D->parity ^= (nsub & 1);
    g_dem_launches = 1;
    return check_launch("dem_substeps (flow)");
}

int lbdem_dem_substeps(lbdem_dem *D, int32_t nsub, void *stream) {
    g_dem_launches = 0;
    int rc = check_dem(D);
    if (rc) return rc;
    if (D->n == 0 || nsub <= 0) return LBDEM_OK;
    cudaStream_t st = (cudaStream_t)stream;
    DemArgs A;
    A.d = *D;
    A.ncell = D->gdim[0] * D->gdim[1] * D->gdim[2];
    contact_constants(A);
    const int nb_int = max((3 * D->n + 127) / 128, min(148, (A.ncell + 127) / 128));   // 3 units per particle
    const int nb_con = (int)((8ll * D->n + 127) / 128);
    // "cluster": all sub-steps in one launch of a single thread-block cluster
    // (opt-in: it confines the contact phase to <= 16 SMs and measured slower
    // than two launches per sub-step spread over the whole GPU).  It is the
    // default when one 512-thread block holds every contact lane (n <= 64):
    // block barriers instead of grid barriers (one sphere: 90 us for 10
    // sub-steps against 107 us cooperative).
    const char *mode = getenv("LBDEM_DEM_KERNELS");
    const bool wrap = D->wrap_pairs != 0;
    auto *kcl = wrap ? k_dem_cluster<true> : k_dem_cluster<false>;
    auto *kcoop = wrap ? k_dem_coop<true> : k_dem_coop<false>;
    // (one block on one SM also runs beside a step on another stream)
    const bool one_block = !mode && 8ll * D->n <= 512;
    if (one_block && 8ll * D->n <= 128) {
        A.parity = D->parity;
        launch_chained(wrap ? k_dem_block<true> : k_dem_block<false>, dim3(1), dim3(128), 0, st, A, (int)nsub);
        D->parity ^= (nsub & 1);
        g_dem_launches = 1;
        return check_launch("dem_substeps (one block)");
    }
    if ((mode && strcmp(mode, "cluster") == 0) || one_block) {
        // one cluster of up to 16 CTAs x 512 threads, sized to the contact lanes
        int ncta = (int)((8ll * D->n + 511) / 512);
        ncta = ncta < 1 ? 1 : (ncta > 16 ? 16 : ncta);
        cudaFuncSetAttribute(kcl, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
        for (; ncta >= 1; ncta >>= 1) {
            cudaLaunchConfig_t cfg = {};
            cfg.gridDim = dim3(ncta, 1, 1);
            cfg.blockDim = dim3(512, 1, 1);
            cfg.dynamicSmemBytes = 0;
            cfg.stream = st;
            cudaLaunchAttribute attr[1];
            attr[0].id = cudaLaunchAttributeClusterDimension;
            attr[0].val.clusterDim.x = ncta;
            attr[0].val.clusterDim.y = 1;
            attr[0].val.clusterDim.z = 1;
            cfg.attrs = attr;
            cfg.numAttrs = 1;
            int nclusters = 0;
            if (cudaOccupancyMaxActiveClusters(&nclusters, kcl, &cfg) != cudaSuccess || nclusters < 1) {
                cudaGetLastError();
                continue;
            }
            A.parity = D->parity;
            if (cudaLaunchKernelEx(&cfg, kcl, A, (int)nsub) == cudaSuccess) {
                D->parity ^= (nsub & 1);
                g_dem_launches = 1;
                return check_launch("dem_substeps (cluster)");
            }
            cudaGetLastError();
        }
    }
    // default: one cooperative launch for all sub-steps when one resident wave
    // covers the contact lanes ("split" forces two launches per sub-step), from
    // three sub-steps on.  On the GPU alone two chained launches per sub-step are
    // the shorter (2000 particles, 1-4 sub-steps: 15, 25, 33, 43 us against 18,
    // 27, 37, 47; 150 particles 13, 22, 32, 39 against 18, 27, 35, 43), but each
    // takes the host 2-3 us to issue, which a longer call does not hide
    if (D->sync && !(mode && strcmp(mode, "split") == 0) && (mode || nsub >= COOP_MIN_SUBSTEPS)) {
        int dev = 0, coop = 0, nsm = 0, per_sm = 0;
        cudaGetDevice(&dev);
        if (coop_residency(dev, wrap, (const void *)kcoop, coop, nsm, per_sm) && coop && per_sm > 0) {
            // one resident wave must cover every contact lane: beyond that the
            // grid-stride loop serialises the phases' memory-latency chains and
            // two launches per sub-step (all lanes in flight) are faster
            const int nb = max(nb_con, nb_int);
            // the arrival counter reaches 2 nsub nb within the launch: keep it far from wrapping
            if (nb <= per_sm * nsm && 2ll * nsub * nb < (1ll << 30)) {
                if (cudaMemsetAsync(D->sync, 0, 2 * sizeof(uint32_t), st) != cudaSuccess)
                    return check_launch("dem_substeps (barrier reset)");
                A.parity = D->parity;
                int nsub_arg = nsub;
                void *args[] = {&A, &nsub_arg};
                if (cudaLaunchCooperativeKernel((void *)kcoop, dim3(nb), dim3(128), args, 0, st) ==
                    cudaSuccess) {
                    D->parity ^= (nsub & 1);
                    g_dem_launches = 1;
                    return check_launch("dem_substeps (cooperative)");
                }
            }
        }
        cudaGetLastError();
    }
    // two launches per sub-step, in 64-thread blocks: each block's registers
    // (~10 K) fit in the room one retiring block of the fused step frees, so
    // the sub-steps can interleave with a step running on another stream
    const int nb_con64 = (int)((8ll * D->n + 63) / 64), nb_int64 = 2 * nb_int;
    for (int s = 0; s < nsub; ++s) {
        A.parity = D->parity;
        launch_chained(wrap ? k_contacts<true> : k_contacts<false>, dim3(nb_con64), dim3(64), 0, st, A);
        launch_chained(k_integrate, dim3(nb_int64), dim3(64), 0, st, A);
        D->parity ^= 1;
    }
    g_dem_launches = 2 * nsub;
    return check_launch("dem_substeps");
}

}  // extern "C"
