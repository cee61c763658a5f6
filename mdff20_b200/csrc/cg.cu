// The vector part of the induced-dipole solves on thread-block clusters: an iteration's
// p.Ap, updates, norms, loop test and new direction in one launch, the start and the end of a
// solve in one launch each.
//
// What bounds it: latency.  At a few hundred to some thousand ions the vectors take well under
// a microsecond of memory time; the separate launches each paid a grid's start, a fence, an
// arrival counter and a last block's reduction (7 + 2 us per iteration at 128 dipoles).  One
// cluster of at most eight blocks holds its ions in registers across the phases, and the sums cross the cluster through distributed shared memory in rank order (the
// same bits on every run).
#include <cooperative_groups.h>

#include <algorithm>

#include "engine.cuh"

namespace cg = cooperative_groups;

namespace mdffgpu {

constexpr int CGT = 512;                  // threads per block
constexpr int CG_CLUSTER_MAX = 8 * CGT;   // one ion per thread of eight blocks; with four ions per
                                          // thread 16000 dipoles took 17.9 us, the grid kernels 12
// carried rho(k) per thread from which a larger cluster shares them out: in one block they are a
// serial chain of reads from L2.  FP64 force evaluations with the fused CG, one block / at most 4
// per thread: 96 ions nk 12194 300 / 264 us, nk 137312 702 / 440 us, 300 ions 331 / 297 and 862 /
// 609 us; below 4096 (kmax 10) no difference
constexpr int CG_RHO = 4;

// sums of NV values over the cluster, in warp order then rank order; sh: [NV][16 + 1] of this
// phase alone (read by the other blocks until the next cluster barrier)
template <int NV>
__device__ __forceinline__ void cluster_sum(cg::cluster_group cl, double (&v)[NV], double (*sh)[CGT / 32 + 1]) {
    const int w = threadIdx.x >> 5, l = threadIdx.x & 31;
#pragma unroll
    for (int k = 0; k < NV; k++) {
        v[k] = warp_sum(v[k]);
        if (l == 0) sh[k][w] = v[k];
    }
    __syncthreads();
    if (threadIdx.x < NV) {
        double a = 0.0;
#pragma unroll
        for (int q = 0; q < CGT / 32; q++) a += sh[threadIdx.x][q];
        sh[threadIdx.x][CGT / 32] = a;
    }
    cl.sync();
    const int nr = (int)cl.num_blocks();
#pragma unroll
    for (int k = 0; k < NV; k++) {
        double a = 0.0;
        for (int r = 0; r < nr; r++) a += *cl.map_shared_rank(&sh[k][CGT / 32], r);
        v[k] = a;
    }
}

__device__ __forceinline__ double3 alpha_times(const double *__restrict__ P, double3 e) {
    return make_double3(P[0] * e.x + P[3] * e.y + P[6] * e.z, P[1] * e.x + P[4] * e.y + P[7] * e.z,
                        P[2] * e.x + P[5] * e.y + P[8] * e.z);
}

struct CgArgs {
    int cnt, nk;
    const int *idx;              // the polarisable ions
    const double *pol, *invpol;
    double *scal;
    double3 *p;
    const double3 *ap;
    double3 *x, *r;
    const double2 *__restrict__ rho_p;   // rho(k) of p, and of the iterate (null: not carried)
    double2 *__restrict__ acc;
    const double3 *efs, *tx, *rhs;
    CgTest test;
    CgComb comb;                 // A p to be formed (part set) in place of ap
};

// A p of the t-th ion i from the slice partials of the FP32 ion pass: alpha^-1 p - T p, k_combine32's
// terms in its order.  A launch less per iteration than with k_combine32 between: the fit of
// 48 configurations 10.18 -> 9.72 ms.
__device__ __forceinline__ double3 comb_ap(const CgComb &b, int cnt, int t, int i, const double3 &p,
                                           const double *__restrict__ I) {
    double S[3] = {0, 0, 0};
#pragma unroll 8
    for (int s = 0; s < b.nslice; s++) {
        const double *o = b.part + ((size_t)s * cnt + t) * 3;
        for (int k = 0; k < 3; k++) S[k] += o[k];
    }
    const double3 d = b.ef_dir[i];
    const double sp[3] = {b.self2 * p.x + d.x, b.self2 * p.y + d.y, b.self2 * p.z + d.z};
    double T[3];
    for (int k = 0; k < 3; k++) {
        const double g = TPI_D * (b.c.B[k][0] * S[0] + b.c.B[k][1] * S[1] + b.c.B[k][2] * S[2]);
        T[k] = sp[k] + (-b.tfpiV * g);
    }
    return make_double3(I[0] * p.x + I[1] * p.y + I[2] * p.z - T[0], I[3] * p.x + I[4] * p.y + I[5] * p.z - T[1],
                        I[6] * p.x + I[7] * p.y + I[8] * p.z - T[2]);
}

// r, z = alpha r, p = z, r.z, r.r and the test before the first iteration; one ion per thread
__global__ void __launch_bounds__(CGT) k_cg_begin(CgArgs a) {
    grid_dep();
    cg::cluster_group cl = cg::this_cluster();
    __shared__ double sh[2][CGT / 32 + 1];
    const int t = (int)cl.block_rank() * CGT + threadIdx.x;
    double v[2] = {0.0, 0.0};
    if (t < a.cnt) {
        const int i = a.idx[t];
        double3 r;
        if (a.rhs) {
            r = a.rhs[i];
            a.x[i] = make_double3(0, 0, 0);
        } else {
            const double3 e = a.efs ? a.efs[i] : make_double3(0, 0, 0), f = a.tx[i], m = a.x[i];
            const double *I = a.invpol + (size_t)i * 9;
            r = make_double3(e.x + f.x - (I[0] * m.x + I[1] * m.y + I[2] * m.z),
                             e.y + f.y - (I[3] * m.x + I[4] * m.y + I[5] * m.z),
                             e.z + f.z - (I[6] * m.x + I[7] * m.y + I[8] * m.z));
        }
        const double3 z = alpha_times(a.pol + (size_t)i * 9, r);
        a.r[i] = r;
        a.p[i] = z;
        v[0] = r.x * z.x + r.y * z.y + r.z * z.z;
        v[1] = r.x * r.x + r.y * r.y + r.z * r.z;
    }
    cluster_sum<2>(cl, v, sh);
    if (t == 0) {
        a.scal[S_RZ] = v[0];
        a.scal[S_RR] = v[1];
        if (a.test.mode) {
            *a.test.guard = 0u;
            cg_test(a.test, v[1], 1);
        }
    }
    cl.sync();
}

// one iteration after A p: a = r.z / p.Ap, x += a p, r -= a Ap, rho(k) of the iterate, z =
// alpha r, r.z and r.r, the loop test (with its backstop: past maxit iterations the loop ends
// whatever the test says) and p = z + beta p.  All of an ion's operands are read before the
// first cluster barrier.
__global__ void __launch_bounds__(CGT) k_cg_update(CgArgs a) {
    grid_dep();
    cg::cluster_group cl = cg::this_cluster();
    __shared__ double sh1[1][CGT / 32 + 1], sh2[2][CGT / 32 + 1];
    const int T = CGT * (int)cl.num_blocks(), t = (int)cl.block_rank() * CGT + threadIdx.x;
    const double rz = a.scal[S_RZ];
    const bool on = t < a.cnt;
    const int i = on ? a.idx[t] : 0;
    double3 p = make_double3(0, 0, 0), q = p, x = p, r = p, z = p;
    double P[9] = {0, 0, 0, 0, 0, 0, 0, 0, 0};
    if (on) {
        p = a.p[i];
        q = a.comb.part ? comb_ap(a.comb, a.cnt, t, i, p, a.invpol + (size_t)i * 9) : a.ap[i];
        x = a.x[i];
        r = a.r[i];
#pragma unroll
        for (int k = 0; k < 9; k++) P[k] = a.pol[(size_t)i * 9 + k];
    }
    double u[1] = {p.x * q.x + p.y * q.y + p.z * q.z};
    cluster_sum<1>(cl, u, sh1);
    const double al = rz / u[0];
    r = make_double3(r.x - al * q.x, r.y - al * q.y, r.z - al * q.z);
    z = alpha_times(P, r);
    double v[2] = {r.x * z.x + r.y * z.y + r.z * z.z, r.x * r.x + r.y * r.y + r.z * r.z};
    if (on) {
        a.x[i] = make_double3(x.x + al * p.x, x.y + al * p.y, x.z + al * p.z);
        a.r[i] = r;
    }
    if (a.acc) {
#pragma unroll 4
        for (int k = t; k < a.nk; k += T) {
            const double2 w = a.rho_p[k], s = a.acc[k];
            a.acc[k] = make_double2(s.x + al * w.x, s.y + al * w.y);
        }
    }
    cluster_sum<2>(cl, v, sh2);
    const double beta = v[0] / rz;
    if (on) a.p[i] = make_double3(z.x + beta * p.x, z.y + beta * p.y, z.z + beta * p.z);
    if (t == 0) {
        a.scal[S_RZ] = v[0];
        a.scal[S_RZOLD] = rz;
        a.scal[S_RR] = v[1];
        if (a.test.mode) {
            cg_test(a.test, v[1], 0);
            if (++*a.test.guard > (unsigned)a.test.maxit) {
                atomicOr(a.test.status, (unsigned)ST_SCF);
                cudaGraphSetConditional(a.test.h, 0);
            }
        }
    }
    cl.sync();
}

// the predictor (k_aspc_predict) and the total dipoles of the first field pass
__global__ void k_pim_begin(int n, AspcCoef cf, int es, double *__restrict__ hist, const double3 *__restrict__ mus,
                            double3 *__restrict__ mu, double3 *__restrict__ tot) {
    grid_dep();
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    double *h = hist + (size_t)i * ASPC_DEPTH * 3;
    double m[3] = {0.0, 0.0, 0.0}, o[18];
#pragma unroll
    for (int k = 0; k < 18; k++) o[k] = h[k];
#pragma unroll
    for (int k = 0; k < 6; k++)
        if (k < cf.ne)
            for (int c = 0; c < 3; c++) m[c] += cf.c[k] * o[3 * k + c];
#pragma unroll
    for (int k = 5; k > 0; k--)
        if (k <= es)
            for (int c = 0; c < 3; c++) h[3 * k + c] = o[3 * (k - 1) + c];
    mu[i] = make_double3(m[0], m[1], m[2]);
    const double3 s = mus[i];
    tot[i] = make_double3(s.x + m[0], s.y + m[1], s.z + m[2]);
}

// total dipoles, history, and the sums mu.alpha^-1.mu (u_pol), q^2, |mu|^2 (self terms)
__global__ void __launch_bounds__(256) k_pim_finish(int n, int pim, const double *__restrict__ invpol,
                                                    const double3 *__restrict__ mus, const double3 *__restrict__ ind,
                                                    double3 *__restrict__ tot, double *__restrict__ hist,
                                                    const double *__restrict__ q, double coul, double *part, int stride,
                                                    double *scal, unsigned *ticket, DevScalars *out) {
    grid_dep();
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    double v[2] = {0.0, 0.0}, u[1] = {0.0};
    if (i < n) {
        double3 t = mus[i];
        if (pim) {
            const double3 m = ind[i];
            const double *I = invpol + (size_t)i * 9;
            const double mm[3] = {m.x, m.y, m.z};
#pragma unroll
            for (int a = 0; a < 3; a++)
#pragma unroll
                for (int b = 0; b < 3; b++) u[0] += mm[a] * I[3 * a + b] * mm[b];
            double *h = hist + (size_t)i * ASPC_DEPTH * 3;
            h[0] = m.x, h[1] = m.y, h[2] = m.z;
            t = make_double3(t.x + m.x, t.y + m.y, t.z + m.z);
        }
        tot[i] = t;
        const double qi = q[i];
        v[0] = qi * qi;
        v[1] = t.x * t.x + t.y * t.y + t.z * t.z;
    }
    block_sum_to_part<2>(v, part, S_Q2, stride);
    if (pim) block_sum_to_part<1>(u, part, S_UPOL, stride);
    const int slots[3] = {S_Q2, S_MU2, S_UPOL};
    if (last_block_warps(part, stride, slots, pim ? 3 : 2, scal, ticket) && pim && threadIdx.x == 0)
        out->u_pol = 0.5 * scal[S_UPOL] * coul;
}

bool cg_clustered(const Engine &e) { return e.npol <= CG_CLUSTER_MAX; }

static CgArgs cg_args(Engine &e, double3 *x, const CgTest &t) {
    CgArgs a{};
    a.cnt = e.npol;
    a.nk = e.nk;
    a.idx = e.d_pidx;
    a.pol = e.d_pol;
    a.invpol = e.d_invpol;
    a.scal = e.d_scal;
    a.p = e.d_cg_p;
    a.ap = e.d_cg_ap;
    a.x = x;
    a.r = e.d_cg_r;
    a.test = t;
    return a;
}

// the smallest cluster with one ion per thread and at most CG_RHO of the nk carried rho(k), up to
// eight blocks (the portable limit).  (Blocks past the ions add zeros: the same bits.)
static int cluster_of(int cnt, int nk = 0) {
    int cs = 1;
    while (cs < 8 && (cnt > CGT * cs || nk > CG_RHO * CGT * cs)) cs *= 2;
    return cs;
}

void launch_cg_begin(Engine &e, const double3 *efs, const double3 *tx, const double3 *rhs, double3 *x,
                     const CgTest &t) {
    CgArgs a = cg_args(e, x, t);
    a.efs = efs;
    a.tx = tx;
    a.rhs = rhs;
    const int cs = cluster_of(a.cnt);
    MDFF_LAUNCH_C(e, cs, k_cg_begin, cs, CGT, 0, a);
}

void launch_cg_update(Engine &e, double3 *x, const double2 *rho_p, double2 *acc, const CgTest &t) {
    CgArgs a = cg_args(e, x, t);
    a.rho_p = rho_p;
    a.acc = acc;
    a.comb = e.cg_comb;
    e.cg_comb.part = nullptr;
    const int cs = cluster_of(a.cnt, acc ? e.nk : 0);
    MDFF_LAUNCH_C(e, cs, k_cg_update, cs, CGT, 0, a);
}

void launch_pim_begin(Engine &e, const AspcCoef &cf, int es) {
    MDFF_LAUNCH(e, k_pim_begin, ceil_div(e.n, 256), 256, 0, e.n, cf, es, e.d_hist, e.d_mu_static, e.d_mu_ind,
                e.d_mu_tot);
}

void launch_pim_finish(Engine &e, bool pim) {
    MDFF_LAUNCH(e, k_pim_finish, ceil_div(e.n, 256), 256, 0, e.n, (int)pim, e.d_invpol, e.d_mu_static, e.d_mu_ind,
                e.d_mu_tot, e.d_hist, e.d_q, e.coul_unit, e.d_part, e.part_stride, e.d_scal, e.d_ticket + 3, e.d_out);
}

}  // namespace mdffgpu
