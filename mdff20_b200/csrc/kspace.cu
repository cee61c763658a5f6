// Reciprocal-space multipole Ewald sum: multipole_ES_rec (src/ewald.c:876-1051) with
// the structure factors of struct_fact / charge_density_* (src/kspace.c:154-302).
//
// The reference tabulates cos/sin(k.r) for every (k, ion) pair (N*nk doubles twice,
// src/kspace.c:35-38).  Here no table exists: with k = 2*pi*B*n (n integer, the
// reference's own k-vectors, src/kspace.c:87-89) the phase factorises,
//     exp(i k.r) = E0[nx] * E1[ny] * E2[nz],   E_d[m] = exp(2*pi*i*m*t_d),  t = B^T r,
// and only the factors are tabulated, one short row per ion.  Two passes:
//   rho pass : rho(k) = sum_i (q_i + i k.mu_i) exp(i k.r_i), per-ion-chunk partial sums,
//              reduced in a fixed order;
//   ion pass : per ion the k sums for field, force and EFG, over slices of the rows,
//              combined and mapped to Cartesian k once per ion.
// FP64: kspace64.cu.  Mixed precision: kspace32.cu, kspace_tc.cu, kspace_ion_tc.cu, with the
// chunk sums, Ak rho(k) and the energy below.
#include "engine.cuh"

namespace mdffgpu {

// one warp, one k per lane: store Ak*rho(k); warp partials of u_rec = sum Ak|rho|^2 and
// of the k-space virial (src/ewald.c:945-1006) into ppart[slot..slot+6][blockIdx.x]
__device__ __forceinline__ void rho_finish(int k, int nk, double2 rho, const double *__restrict__ Ak,
                                           const double *__restrict__ kcoe, const double3 *__restrict__ kv,
                                           double2 *__restrict__ rho_s, double *__restrict__ ppart, int slot,
                                           int stride, bool energy) {
    int l = threadIdx.x & 31;
    double v[7] = {0, 0, 0, 0, 0, 0, 0};
    if (k < nk) {
        double ak = Ak[k], co = kcoe[k];
        double3 kk = kv[k];
        double str = (rho.x * rho.x + rho.y * rho.y) * ak;
        rho_s[k] = make_double2(ak * rho.x, ak * rho.y);
        v[0] = str;
        v[1] = (1.0 - co * kk.x * kk.x) * str;
        v[2] = -co * kk.x * kk.y * str;
        v[3] = -co * kk.x * kk.z * str;
        v[4] = (1.0 - co * kk.y * kk.y) * str;
        v[5] = -co * kk.y * kk.z * str;
        v[6] = (1.0 - co * kk.z * kk.z) * str;
    }
    if (!energy) return;
#pragma unroll
    for (int q = 0; q < 7; q++) v[q] = warp_sum(v[q]);
    if (l < 7) {
        double a = v[0];
#pragma unroll
        for (int q = 1; q < 7; q++)
            if (l == q) a = v[q];
        ppart[(size_t)(slot + l) * stride + blockIdx.x] = a;
    }
}

// sum the ion-chunk partials of rho(k) in a fixed order, then rho_finish. A block owns
// RHOR_K consecutive k (one per lane); its 8 warps take every 8th chunk and warp 0 adds
// the 8 warp sums in warp order. rho_raw (optional) receives rho(k) itself.  Partials
// are FP32 sums over one chunk of ions, added in FP64.  scal set: energies too, the k sums by the
// last block.
__global__ void __launch_bounds__(256) k_rho_reduce(int nk, int nchunks, const float2 *__restrict__ part,
                                                    const double *__restrict__ Ak, const double *__restrict__ kcoe,
                                                    const double3 *__restrict__ kv, double2 *__restrict__ rho_s,
                                                    double2 *__restrict__ rho_raw, double *__restrict__ ppart,
                                                    int slot, int stride, double *scal, unsigned *ticket) {
    grid_dep();
    __shared__ double2 ws[8][RHOR_K];
    int w = threadIdx.x >> 5, l = threadIdx.x & 31;
    int k = blockIdx.x * RHOR_K + l;
    // chunks w, w + 8, ...: four loads in flight into four accumulators (fixed order)
    double2 a0 = make_double2(0.0, 0.0), a1 = a0, a2 = a0, a3 = a0;
    if (k < nk) {
        int c = w;
        for (; c + 24 < nchunks; c += 32) {
            float2 p0 = part[(size_t)c * nk + k], p1 = part[(size_t)(c + 8) * nk + k];
            float2 p2 = part[(size_t)(c + 16) * nk + k], p3 = part[(size_t)(c + 24) * nk + k];
            a0.x += (double)p0.x, a0.y += (double)p0.y;
            a1.x += (double)p1.x, a1.y += (double)p1.y;
            a2.x += (double)p2.x, a2.y += (double)p2.y;
            a3.x += (double)p3.x, a3.y += (double)p3.y;
        }
        for (; c < nchunks; c += 8) {
            float2 p = part[(size_t)c * nk + k];
            a0.x += (double)p.x, a0.y += (double)p.y;
        }
    }
    double2 acc = make_double2((a0.x + a1.x) + (a2.x + a3.x), (a0.y + a1.y) + (a2.y + a3.y));
    ws[w][l] = acc;
    __syncthreads();
    if (w == 0) {
        double2 rho = ws[0][l];
#pragma unroll
        for (int q = 1; q < 8; q++) {
            rho.x += ws[q][l].x;
            rho.y += ws[q][l].y;
        }
        if (rho_raw && k < nk) rho_raw[k] = rho;
        rho_finish(k, nk, rho, Ak, kcoe, kv, rho_s, ppart, slot, stride, scal != nullptr);
    }
    if (!scal) return;
    const int slots[7] = {slot, slot + 1, slot + 2, slot + 3, slot + 4, slot + 5, slot + 6};
    last_block_warps(ppart, stride, slots, 7, scal, ticket);
}

// rho_finish on a rho(k) assembled elsewhere (one warp per RHOR_K k)
__global__ void __launch_bounds__(32) k_rho_from_acc(int nk, const double2 *__restrict__ acc,
                                                     const double *__restrict__ Ak, const double *__restrict__ kcoe,
                                                     const double3 *__restrict__ kv, double2 *__restrict__ rho_s,
                                                     double *__restrict__ ppart, int slot, int stride, double *scal,
                                                     unsigned *ticket) {
    grid_dep();
    int k = blockIdx.x * RHOR_K + threadIdx.x;
    double2 rho = k < nk ? acc[k] : make_double2(0.0, 0.0);
    rho_finish(k, nk, rho, Ak, kcoe, kv, rho_s, ppart, slot, stride, scal != nullptr);
    if (!scal) return;
    const int slots[7] = {slot, slot + 1, slot + 2, slot + 3, slot + 4, slot + 5, slot + 6};
    last_block_warps(ppart, stride, slots, 7, scal, ticket);
}

// ---------------------------------------------------------------- launcher
// rho pass + reduction + ion pass.  `o` says where the per-ion results go:
//   o.ef  = self2*mu + o.ef_dir + E_rec          (when o.ef)
//   o.f   = o.f + o.f_dir*coul + F_rec*coul      (when o.f)
//   o.efg = self + o.efg_dir + EFG_rec (upper)   (when o.efg)
// mixed precision: kspace32.cu passes, FP64 reduction of the FP32 chunk partials
static void launch_rec32(Engine &e, const double *q, const double3 *mu, bool lq, bool ld, const RecOut &o) {
    int nbr = ceil_div(e.nk, RHOR_K);
    int cnt = o.idx ? o.cnt : e.n;
    double *scal = o.energy ? e.d_scal : nullptr;   // energy and virial sums wanted
    if (o.rho_acc) {
        MDFF_LAUNCH(e, k_rho_from_acc, nbr, 32, 0, e.nk, o.rho_acc, e.d_Ak, e.d_kcoe, e.d_kvec, e.d_rho, e.d_part,
                    (int)S_REC_U, e.part_stride, scal, e.d_ticket + 2);
    } else {
        launch_rho32(e, q, mu, lq, ld, o.idx, cnt);
        MDFF_LAUNCH(e, k_rho_reduce, nbr, 256, 0, e.nk, e.rho_chunks_used, e.d_rho_part32, e.d_Ak, e.d_kcoe,
                    e.d_kvec, e.d_rho, o.rho_raw, e.d_part, (int)S_REC_U, e.part_stride, scal, e.d_ticket + 2);
    }
    if (!o.ef && !o.f) return;
    if (o.out_idx) launch_ion32(e, lq ? q : nullptr, mu, ld, o, o.out_idx, o.out_cnt);
    else launch_ion32(e, lq ? q : nullptr, mu, ld, o, o.idx, cnt);
}

void launch_rec(Engine &e, const double *q, const double3 *mu, bool lq, bool ld, const RecOut &o) {
    // FP32 passes in mixed precision (no FP32 EFG: EFG requests run in FP64, as do few ions)
    if (e.use32 && e.rec32 && !e.rec64 && o.efg == nullptr) {
        launch_rec32(e, q, mu, lq, ld, o);
        return;
    }
    launch_rec64(e, q, mu, lq, ld, o);
}

}  // namespace mdffgpu
