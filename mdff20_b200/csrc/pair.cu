// Real-space pair kernels: n-m Lennard-Jones, BHMFT(D) with Tang-Toennies damping and
// the real-space multipole Ewald sum (charges + dipoles).  One warp per ion over that
// ion's FULL neighbour list; each lane takes every 32nd neighbour, per-ion sums are
// combined with warp shuffles and written by lane 0 (no atomics); energies and
// virials go to per-block partial sums reduced in a fixed order.
#include "pairq.cuh"
#include "sr_pair.cuh"
#include "step.cuh"

namespace mdffgpu {

constexpr int PAIR_WARPS = 8;  // warps (= ions) per block

// block-level sum of NV per-warp values into part[(slot+v)*stride + blockIdx.x]
template <int NV>
__device__ __forceinline__ void block_partials(const double (&v)[NV], double *part, int slot, int stride) {
    __shared__ double sh[PAIR_WARPS][NV];
    int w = threadIdx.x >> 5, l = threadIdx.x & 31;
    if (l == 0)
        for (int k = 0; k < NV; k++) sh[w][k] = v[k];
    __syncthreads();
    if (threadIdx.x < NV) {
        double a = 0.0;
        for (int k = 0; k < PAIR_WARPS; k++) a += sh[k][threadIdx.x];
        part[(size_t)(slot + threadIdx.x) * stride + blockIdx.x] = a;
    }
}

// ---------------------------------------------------------------- short range
// engforce_nmlj_pbc (src/nmlj.c:254-385) when LJ, engforce_bhmftd_pbc
// (src/bhmftd.c:117-271) otherwise.  Adds forces into f; slot gets u (x2) and the
// virial sum over the full list of (r_a f_b + r_b f_a).  (The queue of pairq.cuh does not pay
// here: 24000 ions 45 us without, 56 with.)  FP64 in mixed precision too: in FP32 the
// repulsion A exp(-B r) carries the rounding of r times B r (about 8 at Si-O contact), which
// measured an 8e-6 relative force error on the bench system.
// The sums of the slots follow in the last block (fin.ticket set) or in a launch of their own.
struct SrFin {
    unsigned *ticket;
    double *scal;
    double inveOmegaPU, *u, *pvir, *tau;
};
template <bool LJ>
__global__ void __launch_bounds__(PAIR_WARPS * 32, LJ ? 1 : 3) k_sr(int n, Cell c, const double4 *__restrict__ s,
                                                        const int *__restrict__ typ, const PairSR *__restrict__ pr,
                                                        int nt, const int *__restrict__ nbl,
                                                        const int *__restrict__ nbn, int cap, double srcutsq,
                                                        int trunctype, int damped, double3 *__restrict__ f,
                                                        double *__restrict__ part, int slot, int stride, SrFin fin) {
    grid_dep();
    int i = blockIdx.x * PAIR_WARPS + (threadIdx.x >> 5);
    int lane = threadIdx.x & 31;
    double acc[7] = {0, 0, 0, 0, 0, 0, 0};  // u, Vxx Vxy Vxz Vyy Vyz Vzz
    double fx = 0, fy = 0, fz = 0;
    if (i < n) {
        double4 si = s[i];
        int ti = typ[i];
        const int m = min(nbn[i], cap);
        const int *L = nbl + (size_t)i * cap;
        // neighbour types and positions one round ahead, indices two rounds ahead
        int jc = lane < m ? L[lane] : 0;
        int jn = lane + 32 < m ? L[lane + 32] : 0;
        int tc = lane < m ? typ[jc] : 0;
        double4 sc = lane < m ? s[jc] : si;
        for (int k = lane; k < m; k += 32) {
            int tj = tc;
            double4 sj = sc;
            if (k + 32 < m) {
                tc = typ[jn];
                sc = s[jn];
            }
            if (k + 64 < m) jn = L[k + 64];
            const PairSR &P = pr[ti * nt + tj];
            if (!LJ && P.A == 0.0) continue;
            double3 r = pbc_frac(c, dsub(si.x, sj.x), dsub(si.y, sj.y), dsub(si.z, sj.z));
            double r2 = norm2_exact(r);
            if (!(r2 < srcutsq)) continue;
            double u, w;
            if (LJ) lj_pair(P, r2, trunctype, u, w);
            else bhm_pair(P, r2, damped, u, w);
            sr_accumulate(r, u, w, fx, fy, fz, acc);
        }
    }
    fx = warp_sum(fx);
    fy = warp_sum(fy);
    fz = warp_sum(fz);
#pragma unroll
    for (int k = 0; k < 7; k++) acc[k] = warp_sum(acc[k]);
    if (i < n && lane == 0) {
        double3 o = f[i];
        f[i] = make_double3(o.x + fx, o.y + fy, o.z + fz);
    }
    if (i >= n) {
#pragma unroll
        for (int k = 0; k < 7; k++) acc[k] = 0.0;
    }
    block_partials<7>(acc, part, slot, stride);
    if (!fin.ticket) return;
    const int slots[7] = {slot, slot + 1, slot + 2, slot + 3, slot + 4, slot + 5, slot + 6};
    if (last_block_warps(part, stride, slots, 7, fin.scal, fin.ticket) && threadIdx.x == 0)
        finalize_sr(fin.scal, slot, fin.inveOmegaPU, fin.u, fin.pvir, fin.tau);
}

// the slot sums and their composition in one block, four warps per slot (with one warp per slot
// 1700 partials took 7.1 us)
__global__ void __launch_bounds__(896) k_sum_sr(const double *part, int stride, int nparts, int slot, SrFin fin) {
    grid_dep();
    __shared__ double sh[28];
    const int w = threadIdx.x >> 5, l = threadIdx.x & 31;
    const double *p = part + (size_t)(slot + (w >> 2)) * stride;
    double a = 0.0;
#pragma unroll 8
    for (int k = 32 * (w & 3) + l; k < nparts; k += 128) a += p[k];
    a = warp_sum(a);
    if (l == 0) sh[w] = a;
    __syncthreads();
    if (threadIdx.x < 7) {
        const double *q = sh + 4 * threadIdx.x;
        fin.scal[slot + threadIdx.x] = (q[0] + q[1]) + (q[2] + q[3]);
    }
    __syncthreads();
    if (threadIdx.x == 0) finalize_sr(fin.scal, slot, fin.inveOmegaPU, fin.u, fin.pvir, fin.tau);
}

// whether a pair kernel's last block sums its slots: up to one wave of blocks (n <= 4736), where
// it saves two launches of 2 us each; with several waves the arrivals of the blocks cost more
bool sum_in_last(const Engine &e, int blocks) { return blocks <= 4 * e.nsm; }

void launch_sr(Engine &e, bool lj) {
    int nb = ceil_div(e.n, PAIR_WARPS);
    DevScalars *o = e.d_out;
    const int slot = lj ? S_LJ_U : S_BH_U;
    SrFin fin{sum_in_last(e, nb) ? e.d_ticket + 7 : nullptr, e.d_scal, e.cell.inveOmegaPU, lj ? &o->u_lj : &o->u_bh,
              lj ? &o->pvir_lj : &o->pvir_bh, lj ? o->tau_lj : o->tau_bh};
    if (lj)
        MDFF_LAUNCH(e, k_sr<true>, nb, PAIR_WARPS * 32, 0, e.n, e.cell, e.d_s, e.d_typ, e.d_pair, e.nt, e.d_nb,
                    e.d_nbn, e.cap_nb, e.srcutsq, e.p.trunctype, 0, e.d_f, e.d_part, (int)S_LJ_U,
                    e.part_stride, fin);
    else
        MDFF_LAUNCH(e, k_sr<false>, nb, PAIR_WARPS * 32, 0, e.n, e.cell, e.d_s, e.d_typ, e.d_pair, e.nt, e.d_nb,
                    e.d_nbn, e.cap_nb, e.srcutsq, e.p.trunctype, e.p.lbhmftd, e.d_f, e.d_part, (int)S_BH_U,
                    e.part_stride, fin);
    if (!fin.ticket) MDFF_LAUNCH(e, k_sum_sr, 1, 896, 0, e.d_part, e.part_stride, nb, slot, fin);
}

// ---------------------------------------------------------------- real-space Ewald
// multipole_ES_dir (src/ewald.c:353-871) for charges and dipoles, from ion i's side.
// For each neighbour j within cutlongrange (d2 <= lrcutsq, src/ewald.c:486) the
// tensors T0..T3 (src/ewald.c:562-620) are contracted directly with q and mu:
//   field at i      : -qj T1 (+ qj T1D1 damped)  and  T2 mu_j (only if mu_i, mu_j != 0)
//   force on i      : -f_ij with f_ij as src/ewald.c:719-812
//   EFG at i        : -qj T2 + T3 . mu_j
//   energy, virial  : half of the pair value (each pair is seen from both ions)
// Template flags select what is computed; FORCES also computes energy and virial.
struct DirArgs {
    int n, nt, cap;
    Cell c;
    const double4 *s;
    const double *q;
    const double3 *mu;
    const int *typ;
    const PairDamp *damp;
    const int *col, *con;
    double lrcutsq, alpha;
    TT tt;
    int lq, ld, ldamp, efg_q;
    double3 *ef;
    double *efg;
    double3 *f;
    double *part;
    int slot, stride;
    double *scal;
    unsigned *ticket;            // the last block sums the slots (null: a launch of its own does)
};

//
// Bound by the FP64 pipe and the latency of its long dependent chains (128 registers: 16 warps
// per SM): per pair one reciprocal square root, one exponential, one erfc and up to two
// Tang-Toennies functions.  Pairs are taken in full groups of 32 from the queue of pairq.cuh,
// divisions by d^2 are products, a damping function is evaluated only where it enters (a zero
// dipole or c = 0 leaves it out exactly), energy and virial only when asked for.  6000 ions, cut
// off 10 + 1 A: forces 118 -> 84 us, field 89 -> 64; 3000 ions 73 -> 55 and 56 -> 43.  A third
// block per SM (80 registers, 240 bytes spilled) took the forces to 112 us; erfcx times the
// exponential at hand in place of erfc changed nothing (82.6 / 61.4 us).
template <bool FORCES, bool EF, bool EFG>
__global__ void __launch_bounds__(PAIR_WARPS * 32) k_dir(DirArgs a) {
    grid_dep();
    int i = blockIdx.x * PAIR_WARPS + (threadIdx.x >> 5);
    int lane = threadIdx.x & 31;
    double acc[7] = {0, 0, 0, 0, 0, 0, 0};   // u, V6
    double fi[3] = {0, 0, 0}, ei[3] = {0, 0, 0};
    double gi[9] = {0, 0, 0, 0, 0, 0, 0, 0, 0};
    const bool en = a.part != nullptr;   // energy and virial wanted
    __shared__ PairQ queue[PAIR_WARPS];
    if (i < a.n) {
        double4 si = a.s[i];
        double qi = a.lq ? a.q[i] : 0.0;
        double3 mi = a.ld ? a.mu[i] : make_double3(0, 0, 0);
        bool dip_i = (mi.x != 0.0) || (mi.y != 0.0) || (mi.z != 0.0);
        int ti = a.typ[i];
        auto pair = [&](int j, const double3 &r, double d2) {
            double qj = a.lq ? a.q[j] : 0.0;
            double3 mj = a.ld ? a.mu[j] : make_double3(0, 0, 0);
            bool dip_j = (mj.x != 0.0) || (mj.y != 0.0) || (mj.z != 0.0);
            const Screened v = screened(d2, a.alpha);
            const double d = v.d, dm1 = v.dm1, dm3 = v.dm3, dm5 = v.dm5, F0 = v.F0, F1 = v.F1, F2 = v.F2;
            // Tang-Toennies damping of the charge->dipole field, src/ewald.c:505-539: of the charge j
            // at i's dipole (1; the field at any i) and of the charge i at j's dipole (2)
            double F1d1 = 0.0, F1d2 = 0.0, F2d1 = 0.0, F2d2 = 0.0;
            bool damp = false;
            if (a.ldamp && a.lq) {
                const PairDamp &D = a.damp[ti * a.nt + a.typ[j]];
                if (D.ldamp) {
                    damp = true;
                    double f, fd;
                    if ((EF || dip_i) && D.c1 != 0.0) {   // (c = 0: f = 1)
                        tt_damp(a.tt, D.b1, D.c1, d, D.k1, f, fd);
                        F1d1 = 1.0 - f;
                        F2d1 = F1d1 + d * (1.0 / 3.0) * fd;
                    }
                    if (dip_j && D.c2 != 0.0) {
                        tt_damp(a.tt, D.b2, D.c2, d, D.k2, f, fd);
                        F1d2 = 1.0 - f;
                        F2d2 = F1d2 + d * (1.0 / 3.0) * fd;
                    }
                }
            }
            double F1_dm3 = F1 * dm3, F2_dm5 = 3.0 * F2 * dm5;
            double u = 0.0;
            double fij[3] = {0, 0, 0};
            // charge-charge, src/ewald.c:703-731
            if (a.lq) {
                u += qi * qj * (dm1 * F0);
                if (EF) {
                    double cfe = qj * dm3 * (F1 - F1d1);   // -qj T1 + qj T1D1
                    ei[0] += cfe * r.x;
                    ei[1] += cfe * r.y;
                    ei[2] += cfe * r.z;
                }
                if (FORCES) {
                    double cf = -qi * qj * F1_dm3;        // qij T1
                    fij[0] = cf * r.x;
                    fij[1] = cf * r.y;
                    fij[2] = cf * r.z;
                }
                if (EFG && a.efg_q) {
                    double rr[3] = {r.x, r.y, r.z};
                    for (int p = 0; p < 3; p++)
                        for (int q = 0; q < 3; q++)
                            gi[3 * p + q] += -qj * (rr[p] * rr[q] * F2_dm5 - (p == q ? F1_dm3 : 0.0));
                }
            }
            double rmi = r.x * mi.x + r.y * mi.y + r.z * mi.z;
            double rmj = r.x * mj.x + r.y * mj.y + r.z * mj.z;
            // dipole-dipole, src/ewald.c:737-761 (both dipoles non-zero)
            if (a.ld && dip_i && dip_j) {
                double mm = mi.x * mj.x + mi.y * mj.y + mi.z * mj.z;
                u += F1_dm3 * mm - F2_dm5 * rmi * rmj;
                if (EF) {
                    ei[0] += F2_dm5 * rmj * r.x - F1_dm3 * mj.x;
                    ei[1] += F2_dm5 * rmj * r.y - F1_dm3 * mj.y;
                    ei[2] += F2_dm5 * rmj * r.z - F1_dm3 * mj.z;
                }
                // F3 = F2 + 8 (alpha d)^5 exp / 15
                const double ad2 = a.alpha * a.alpha * d2;
                const double F3_dm7 =
                    (15.0 * F2 + 8.0 * (ad2 * ad2 * a.alpha * d) * v.ex) * (dm5 * dm1 * dm1);
                if (FORCES) {
                    double c1 = -F3_dm7 * rmi * rmj, c2 = F2_dm5;
                    fij[0] -= c1 * r.x + c2 * (mm * r.x + mi.x * rmj + mj.x * rmi);
                    fij[1] -= c1 * r.y + c2 * (mm * r.y + mi.y * rmj + mj.y * rmi);
                    fij[2] -= c1 * r.z + c2 * (mm * r.z + mi.z * rmj + mj.z * rmi);
                }
                if (EFG) {
                    double rr[3] = {r.x, r.y, r.z}, mv[3] = {mj.x, mj.y, mj.z};
                    for (int p = 0; p < 3; p++)
                        for (int q = 0; q < 3; q++)
                            gi[3 * p + q] += -F3_dm7 * rmj * rr[p] * rr[q] +
                                             F2_dm5 * ((p == q ? rmj : 0.0) + mv[p] * rr[q] + rr[p] * mv[q]);
                }
            }
            // charge-dipole, src/ewald.c:767-812
            if (a.lq && a.ld && (dip_i || dip_j)) {
                u += F1_dm3 * (qi * rmj - qj * rmi);
                if (FORCES) {
                    double wx = qj * mi.x - qi * mj.x, wy = qj * mi.y - qi * mj.y, wz = qj * mi.z - qi * mj.z;
                    double rw = r.x * wx + r.y * wy + r.z * wz;
                    fij[0] += F2_dm5 * rw * r.x - F1_dm3 * wx;
                    fij[1] += F2_dm5 * rw * r.y - F1_dm3 * wy;
                    fij[2] += F2_dm5 * rw * r.z - F1_dm3 * wz;
                }
                if (damp) {
                    u += dm3 * (-qi * F1d2 * rmj + qj * F1d1 * rmi);
                    if (FORCES) {
                        double a1 = 3.0 * F2d1 * dm5, b1 = F1d1 * dm3;
                        double a2 = 3.0 * F2d2 * dm5, b2 = F1d2 * dm3;
                        fij[0] += -qj * (a1 * rmi * r.x - b1 * mi.x) + qi * (a2 * rmj * r.x - b2 * mj.x);
                        fij[1] += -qj * (a1 * rmi * r.y - b1 * mi.y) + qi * (a2 * rmj * r.y - b2 * mj.y);
                        fij[2] += -qj * (a1 * rmi * r.z - b1 * mi.z) + qi * (a2 * rmj * r.z - b2 * mj.z);
                    }
                }
            }
            if (FORCES) {
                fi[0] -= fij[0];
                fi[1] -= fij[1];
                fi[2] -= fij[2];
            }
            if (en) {
                acc[0] += u;
                if (FORCES) {
                    acc[1] += -(r.x * fij[0] + r.x * fij[0]);
                    acc[2] += -(r.x * fij[1] + r.y * fij[0]);
                    acc[3] += -(r.x * fij[2] + r.z * fij[0]);
                    acc[4] += -(r.y * fij[1] + r.y * fij[1]);
                    acc[5] += -(r.y * fij[2] + r.z * fij[1]);
                    acc[6] += -(r.z * fij[2] + r.z * fij[2]);
                }
            }
        };
        pairs_in_cut<false>(a.c, a.s, si, a.col + (size_t)i * a.cap, min(a.con[i], a.cap), a.lrcutsq,
                            queue[threadIdx.x >> 5], pair);
    }
    if (en) {
#pragma unroll
        for (int k = 0; k < 7; k++) acc[k] = warp_sum(acc[k]);
    }
    if (FORCES) {
        for (int k = 0; k < 3; k++) fi[k] = warp_sum(fi[k]);
    }
    if (EF) {
        for (int k = 0; k < 3; k++) ei[k] = warp_sum(ei[k]);
    }
    if (EFG) {
        for (int k = 0; k < 9; k++) gi[k] = warp_sum(gi[k]);
    }
    if (i < a.n && lane == 0) {
        if (FORCES && a.f) a.f[i] = make_double3(fi[0], fi[1], fi[2]);
        if (EF && a.ef) a.ef[i] = make_double3(ei[0], ei[1], ei[2]);
        if (EFG && a.efg)
            for (int k = 0; k < 9; k++) a.efg[(size_t)i * 9 + k] = gi[k];
    }
    if (i >= a.n) {
#pragma unroll
        for (int k = 0; k < 7; k++) acc[k] = 0.0;
    }
    if (!a.part) return;
    block_partials<7>(acc, a.part, a.slot, a.stride);
    if (!a.ticket) return;
    const int slots[7] = {a.slot, a.slot + 1, a.slot + 2, a.slot + 3, a.slot + 4, a.slot + 5, a.slot + 6};
    last_block_warps(a.part, a.stride, slots, 7, a.scal, a.ticket);
}

void launch_dir(Engine &e, const double *q, const double3 *mu, double alpha, bool lq, bool ld, bool damp,
                bool forces, bool ef, bool efg, bool efg_q, double3 *out_ef, double *out_efg, double3 *out_f,
                bool energy) {
    const double4 *s = e.d_s;
    DirArgs a;
    a.n = e.n;
    a.nt = e.nt;
    a.cap = e.cap_co;
    a.c = e.cell;
    a.s = s;
    a.q = q;
    a.mu = mu;
    a.typ = e.d_typ;
    a.damp = e.d_damp;
    a.col = e.d_co;
    a.con = e.d_con;
    a.lrcutsq = e.lrcutsq;
    a.alpha = alpha;
    a.tt.E[0] = 1.0;
    for (int k = 1; k < 9; k++) a.tt.E[k] = a.tt.E[k - 1] / (double)k;
    a.lq = lq;
    a.ld = ld;
    a.ldamp = damp;
    a.efg_q = efg_q;
    a.ef = out_ef;
    a.efg = out_efg;
    a.f = out_f;
    int nb = ceil_div(e.n, PAIR_WARPS);
    a.part = energy ? e.d_part : nullptr;
    a.slot = S_DIR_U;
    a.stride = e.part_stride;
    a.scal = e.d_scal;
    a.ticket = energy && sum_in_last(e, nb) ? e.d_ticket + 8 : nullptr;
    if (efg || (ef && forces))
        MDFF_LAUNCH(e, (k_dir<true, true, true>), nb, PAIR_WARPS * 32, 0, a);
    else if (forces)
        MDFF_LAUNCH(e, (k_dir<true, false, false>), nb, PAIR_WARPS * 32, 0, a);
    else
        MDFF_LAUNCH(e, (k_dir<false, true, false>), nb, PAIR_WARPS * 32, 0, a);
    if (energy && !a.ticket) e.reduce(S_DIR_U, 7, nb);
}

// ---------------------------------------------------------------- cached dipole field
// Within one force evaluation the positions are fixed while the induced dipoles are
// iterated (src/pim.c:236-278), so the screened pair factors F1/d^3 and 3 F2/d^5 of
// the dipole field (the T2 tensor, src/ewald.c:581-603) are computed once per pair
// and reused by every iteration: the iteration kernel then does no erfc/exp.  Induced dipoles
// sit on polarisable ions and act on those only, so the records are the pairs of polarisable
// ions inside the cut-off, in list order: pcol, pcon and coef.  Bound by the FP64 pipe (prep) and
// by the gathers of 88 bytes per pair from L2 (field).  6000 ions, silica, cut-off 10 + 1 A, against
// factors for every list entry (three per record): prep 47 -> 22 us, field 18 -> 11 us; 3000 ions
// prep 25 -> 12, field 13 -> 6.
__global__ void __launch_bounds__(PAIR_WARPS * 32) k_dir_prep(int n, Cell c, const double4 *__restrict__ s,
                                                             const int *__restrict__ polar,
                                                             const int *__restrict__ col,
                                                             const int *__restrict__ con, int cap, double lrcutsq,
                                                             double alpha, int *__restrict__ pcol,
                                                             int *__restrict__ pcon, double2 *__restrict__ coef) {
    grid_dep();
    int i = blockIdx.x * PAIR_WARPS + (threadIdx.x >> 5);
    int lane = threadIdx.x & 31;
    if (i >= n) return;
    int cnt = 0;
    if (polar[i]) {
        __shared__ PairQ queue[PAIR_WARPS];
        int *P = pcol + (size_t)i * cap;
        double2 *C = coef + (size_t)i * cap;
        pairs_in_cut<false>(c, s, s[i], col + (size_t)i * cap, min(con[i], cap), lrcutsq, queue[threadIdx.x >> 5],
                            [&](int j) { return polar[j] != 0; }, cnt,
                            [&](int at, int j, const double3 &, double d2) {
                                const Screened v = screened(d2, alpha);
                                P[at] = j;
                                C[at] = make_double2(v.F1 * v.dm3, 3.0 * v.F2 * v.dm5);
                            });
    }
    if (lane == 0) pcon[i] = cnt;
}

// field of the dipoles mu from the cached factors: E_i = sum_j (3F2/d^5 (r.mu_j) r - F1/d^3 mu_j),
// only when mu_i and mu_j are non-zero (src/ewald.c:737-749)
__global__ void __launch_bounds__(PAIR_WARPS * 32) k_dir_field_cached(int n, Cell c, const double4 *__restrict__ s,
                                                                     const int *__restrict__ pcol,
                                                                     const int *__restrict__ pcon, int cap,
                                                                     const double2 *__restrict__ coef,
                                                                     const double3 *__restrict__ mu,
                                                                     double3 *__restrict__ ef) {
    grid_dep();
    int i = blockIdx.x * PAIR_WARPS + (threadIdx.x >> 5);
    int lane = threadIdx.x & 31;
    if (i >= n) return;
    double ex = 0.0, ey = 0.0, ez = 0.0;
    const int m = pcon[i];
    if (m > 0) {
        double3 mi = mu[i];
        if ((mi.x != 0.0) || (mi.y != 0.0) || (mi.z != 0.0)) {
            double4 si = s[i];
            const int *L = pcol + (size_t)i * cap;
            const double2 *C = coef + (size_t)i * cap;
            int jn = lane < m ? L[lane] : 0;
#pragma unroll 2
            for (int k = lane; k < m; k += 32) {
                const int j = jn;
                if (k + 32 < m) jn = L[k + 32];
                const double2 cf = C[k];
                const double3 mj = mu[j];
                const double4 sj = s[j];
                const double3 r = pbc_frac(c, dsub(si.x, sj.x), dsub(si.y, sj.y), dsub(si.z, sj.z));
                const double rmj = r.x * mj.x + r.y * mj.y + r.z * mj.z;
                ex += cf.y * rmj * r.x - cf.x * mj.x;
                ey += cf.y * rmj * r.y - cf.x * mj.y;
                ez += cf.y * rmj * r.z - cf.x * mj.z;
            }
        }
    }
    ex = warp_sum(ex);
    ey = warp_sum(ey);
    ez = warp_sum(ez);
    if (lane == 0) ef[i] = make_double3(ex, ey, ez);
}

void launch_dir_prep(Engine &e, double alpha) {
    int nb = ceil_div(e.n, PAIR_WARPS);
    MDFF_LAUNCH(e, k_dir_prep, nb, PAIR_WARPS * 32, 0, e.n, e.cell, e.d_s, e.d_polar, e.d_co, e.d_con, e.cap_co,
                e.lrcutsq, alpha, e.d_pcol, e.d_pcon, e.d_coef);
}

void launch_dir_field_cached(Engine &e, const double3 *mu, double3 *out_ef) {
    int nb = ceil_div(e.n, PAIR_WARPS);
    int pd = -1;
    e.prof_begin("k_dir", &pd);
    MDFF_LAUNCH(e, k_dir_field_cached, nb, PAIR_WARPS * 32, 0, e.n, e.cell, e.d_s, e.d_pcol, e.d_pcon, e.cap_co,
                e.d_coef, mu, out_ef);
    e.prof_end("k_dir", pd, 0.0);
}

}  // namespace mdffgpu
