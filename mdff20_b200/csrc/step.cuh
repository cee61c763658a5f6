// Device pieces shared by the kernels that close an MD step: the displacement test of
// check_verletlist and the composition of the reference's energy globals.
#pragma once

#include "engine.cuh"

namespace mdffgpu {

// ---------------------------------------------------------------- check_verletlist
// displacement since the last build, largest and second largest (src/verlet.c:134-147)
__device__ __forceinline__ void top2_insert(double &m1, double &m2, double d) {
    if (d > m1) {
        m2 = m1;
        m1 = d;
    } else if (d > m2) {
        m2 = d;
    }
}

// warp merge of per-lane top-2 pairs (the two largest values, whatever the order they
// are met in)
__device__ __forceinline__ void top2_warp(double &m1, double &m2) {
    for (int o = 16; o > 0; o >>= 1) {
        double o1 = __shfl_xor_sync(0xffffffffu, m1, o);
        double o2 = __shfl_xor_sync(0xffffffffu, m2, o);
        double n1 = fmax(m1, o1);
        double n2 = fmax(fmin(m1, o1), fmax(m2, o2));
        m1 = n1;
        m2 = n2;
    }
}

struct CheckArgs {
    int on;                      // 0: no list check in this launch
    int n, ncell;
    Cell c;
    double4 *s;                  // fractional coordinates of the current positions
    const double4 *svl;          // ... at the last build
    double *part1, *part2;
    double skindiff;
    int *rebuild, *cell_cnt;
    DevScalars *out;
    cudaGraphConditionalHandle h;   // condition of the IF node that holds the rebuild (use_h)
    int use_h;
};
CheckArgs check_args(Engine &e, const cudaGraphConditionalHandle *h);

__device__ __forceinline__ double check_moved(const CheckArgs &a, double4 si, int i) {
    const double4 b = a.svl[i];
    return __dsqrt_rn(norm2_exact(pbc_frac(a.c, dsub(si.x, b.x), dsub(si.y, b.y), dsub(si.z, b.z))));
}

// the block's two largest displacements (256 threads); the caller's block fences and arrives
__device__ __forceinline__ void check_block(const CheckArgs &a, double m1) {
    __shared__ double sm1[8], sm2[8];
    double m2 = 0.0;
    top2_warp(m1, m2);
    if ((threadIdx.x & 31) == 0) {
        sm1[threadIdx.x >> 5] = m1;
        sm2[threadIdx.x >> 5] = m2;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        double a1 = 0.0, a2 = 0.0;
        for (int k = 0; k < (int)(blockDim.x >> 5); k++) {
            top2_insert(a1, a2, sm1[k]);
            top2_insert(a1, a2, sm2[k]);
        }
        a.part1[blockIdx.x] = a1;
        a.part2[blockIdx.x] = a2;
    }
}

// the last block: merges the block pairs, tests them against the skin (src/verlet.c:148) and on
// a rebuild zeroes the cell counts the binning adds to
__device__ __forceinline__ void check_last(const CheckArgs &a) {
    __shared__ int rb_s;
    if (threadIdx.x < 32) {
        double b1 = 0.0, b2 = 0.0;
#pragma unroll 4
        for (int k = threadIdx.x; k < (int)gridDim.x; k += 32) {
            top2_insert(b1, b2, __ldcg(a.part1 + k));
            top2_insert(b1, b2, __ldcg(a.part2 + k));
        }
        top2_warp(b1, b2);
        if (threadIdx.x == 0) {
            const int rb = (b1 + b2 > a.skindiff) ? 1 : 0;
            *a.rebuild = rb;
            a.out->rebuild = rb;
            if (rb) a.out->nbuilds += 1;
            if (a.use_h) cudaGraphSetConditional(a.h, rb ? 1u : 0u);
            rb_s = rb;
        }
    }
    __syncthreads();
    if (rb_s)
        for (int k = threadIdx.x; k < a.ncell; k += blockDim.x) a.cell_cnt[k] = 0;
}

// ---------------------------------------------------------------- composition
// u, pvir, tau of a short-range evaluator from its slots (src/nmlj.c:351-363):
// slot 0 holds the full-list energy sum (each pair twice), slots 1..6 the full-list
// sum of r_a f_b + r_b f_a.
__device__ __forceinline__ void finalize_sr(const double *scal, int slot, double inveOmegaPU, double *u, double *pvir,
                                            double *tau) {
    *u = 0.5 * scal[slot];
    double t[6];
    for (int k = 0; k < 6; k++) t[k] = 0.25 * scal[slot + 1 + k] * inveOmegaPU;
    double full[9] = {t[0], t[1], t[2], t[1], t[3], t[4], t[2], t[4], t[5]};
    double pv = 0.0;
    for (int k = 0; k < 9; k++) tau[k] = full[k];
    for (int k = 0; k < 3; k++) pv += full[4 * k] * (1.0 / 3.0);
    *pvir = pv;
}

// u_coul, tau_coul (src/ewald.c:209-307): dir (full-list sums), rec, self
__device__ __forceinline__ void finalize_coul(const CoulFin &c) {
    const double *scal = c.scal;
    const double rpi = 1.7724538509055160273;
    double alpha2 = c.alpha * c.alpha, selfa = c.alpha / rpi, selfa2 = 2.0 * selfa * alpha2 / 3.0;
    double u_self = -selfa * scal[S_Q2] + -selfa2 * scal[S_MU2];
    double u_dir = c.do_dir ? 0.5 * scal[S_DIR_U] : 0.0;
    double u_rec = c.do_rec ? scal[S_REC_U] * c.ttpiV : 0.0;
    *c.u = (u_dir + u_rec + u_self) * c.coul;
    if (c.do_stress) {
        double td[6], tr[6];
        for (int k = 0; k < 6; k++) {
            td[k] = 0.25 * scal[S_DIR_TAU + k] * c.inveOmegaPU;
            tr[k] = scal[S_REC_TAU + k] * c.ttpiV * c.inveOmegaPU;
        }
        int map[9] = {0, 1, 2, 1, 3, 4, 2, 4, 5};
        for (int k = 0; k < 9; k++) {
            double t = 0.0;
            if (c.do_dir) t += td[map[k]] * c.coul;
            if (c.do_rec) t += tr[map[k]] * c.coul;
            c.tau[k] = t;
        }
    }
    double pv = 0.0;
    for (int k = 0; k < 3; k++) pv += c.tau[4 * k] * (1.0 / 3.0);
    *c.pvir = pv;
}

}  // namespace mdffgpu
