// FP64 reciprocal-space passes on the FP64 matrix instructions (mma.sync m8n8k4.f64).
//
// With exp(i k.r) = E0[nx] E1[ny] E2[nz] (kspace.cu) and E2[+-z] = c_z +- i d_z, both ion x k
// passes are contractions over the pairs +-z of each row (nx, ny):
//
//   rho pass   the summand of k = (nx, ny, nz) is (B1 + nz B2) E2[nz], B1 = (q + i c0) b,
//              B2 = i c1 b, b = E0 E1, c0 + nz c1 = k.mu.  The sums over the ions
//                  C[coef, row][col] = sum_i A[coef, row][i] E[i][col],
//              coef = (B1x, B1y, B2x, B2y), col = (c_0, d_0, c_1, d_1, ...), give rho at +z
//              and -z: 4 FMA per k-vector (2 for charges only) instead of 6 + the table.
//   ion pass   G = sum_z Y(z), H = sum_z z Y(z), K = sum_z z^2 Y(z), Y = Ak rho conj(E2), per
//              (ion, row) are D[i][comp, row] = sum_col E[i][col] W[comp, row][col] with the
//              weights W of the folded +-z sums: 4 FMA per k-vector for the field, 6 with
//              forces or EFG.  The row phase conj(E0 E1) and the factors nx, ny follow per
//              (ion, row); the sums S = sum k Im, Hm = sum k k^T Re give field, force and EFG.
//
// What bounds it: the FP64 pipe.  mma.f64 reaches 36.9 TFLOP/s on B200 with one warp per
// scheduler (DFMA: 32 with one, 35.3 with four) and takes one issue slot and no shared-memory
// operand traffic per 256 FMA, so the passes run near the pipe instead of on LDS and issue.
// The operand layouts fall out of the fragments: a lane of the rho pass holds (row, ion) of
// all four coefficients, so A is formed in registers; its accumulators hold (c_z, d_z) of one
// (row, z), so rho(+-z) is formed in the lane.  A lane of the ion pass holds G, H, K of one
// (ion, row).
//
// Measured (B200, 4000 dipoles of 6000 ions, nk 12194, kmax 14): rho pass 89 -> 24.7 us (16
// TFLOP/s of the 8-flop count), ion pass and combine 68 -> 25.9 us, with forces 104 -> 48.6 us;
// at 128 of 192 ions (kmax 10) the rho pass 32 -> 3.6 us, the ion pass and combine 25 -> 7.6 us.  The thread-per-segment passes these replaced were slower at
// every size, so no other FP64 path is kept.
//
// |nz| beyond 15 is split in groups of 16 (rho: a grid dimension, ion: more units of work).
#include <algorithm>
#include <type_traits>

#include "step.cuh"

namespace mdffgpu {

constexpr int R64_WARPS = 8;     // rho pass: warps per block, 8 rows each
constexpr int R64_ROWS = 8 * R64_WARPS;
constexpr int R64_TI = 16;       // ions per stage
constexpr int I64_WARPS = 4;     // ion pass: warps per block, MT tiles of 8 ions each
constexpr int ZG = 16;           // |nz| values per group (32 table columns)

__device__ __forceinline__ void dmma(double (&c)[2], double a, double b) {
    asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1},{%2},{%3},{%0,%1};"
        : "+d"(c[0]), "+d"(c[1])
        : "d"(a), "d"(b));
}

__device__ __forceinline__ void cp_async16(void *dst, const void *src) {
    const unsigned d = (unsigned)__cvta_generic_to_shared(dst);
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(d), "l"(src) : "memory");
}

__device__ __forceinline__ double3 to_phase(const Cell &c, double x, double y, double z) {
    return make_double3(c.B[0][0] * x + c.B[1][0] * y + c.B[2][0] * z,
                        c.B[0][1] * x + c.B[1][1] * y + c.B[2][1] * z,
                        c.B[0][2] * x + c.B[1][2] * y + c.B[2][2] * z);
}

// ---------------------------------------------------------------- phase tables
// one row of the table per ion: E0[0..K0] | E1[-K1..K1] | (c_z, d_z) for z = 0..16 nzg - 1
// (zero past K2), each from its own reduced argument (no recurrence: the chain of K complex
// products per ion was most of a small system's rho pass, 32 of its 35 us at 192 ions)
struct Tab64 {
    int K0, K1, K2, nzg;
    int e1, z, w;      // offsets of E1 and Z, row width (double2)
};
__global__ void __launch_bounds__(256) k_phase64(int n, Cell c, Tab64 t, const double4 *__restrict__ r,
                                                 double2 *__restrict__ tab) {
    grid_dep();
    // entries computed: E0[0..K0], E1[0..K1] (and the conjugates), Z[0..16 nzg - 1]
    const int ne = t.K0 + 1 + t.K1 + 1 + ZG * t.nzg;
    const long long id = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    const int i = (int)(id / ne);
    if (i >= n) return;
    int m = (int)(id - (long long)i * ne);
    const double4 ri = r[i];
    const double3 p = to_phase(c, ri.x, ri.y, ri.z);
    int dim = 0;
    double x = p.x;
    if (m > t.K0) {
        m -= t.K0 + 1;
        dim = 1;
        x = p.y;
        if (m > t.K1) {
            m -= t.K1 + 1;
            dim = 2;
            x = p.z;
        }
    }
    x -= rint(x);
    double a = (double)m * x;
    a -= rint(a);
    double sn, cs;
    sincospi(2.0 * a, &sn, &cs);
    double2 *T = tab + (size_t)i * t.w;
    if (dim == 0) {
        T[m] = make_double2(cs, sn);
    } else if (dim == 1) {
        T[t.e1 + t.K1 + m] = make_double2(cs, sn);
        if (m) T[t.e1 + t.K1 - m] = make_double2(cs, -sn);
    } else {
        T[t.z + m] = m <= t.K2 ? make_double2(cs, sn) : make_double2(0.0, 0.0);
    }
}

// ---------------------------------------------------------------- rho pass
struct Rho64Args {
    int n, chunk, nrow, nk;      // n: ions in the pass (idx[n] when set); chunk: a multiple of R64_TI
    Tab64 t;
    Cell c;
    int stw;                     // stage row width (double2), 2 mod 8: conflict-free fragment loads
    int nbuf;                    // stage buffers: 2, or 1 where two do not fit (kmax in the hundreds)
    const double2 *tab;
    const double *q;
    const double3 *mu;
    const int *idx;
    const KRow *row;
    double2 *part;               // [chunks][nk]
};

// grid (row blocks, ion chunks, z groups).  KS: k steps of 4 columns that hold |nz| values,
// NTL = ceil(KS / 2) column tiles of 8.
template <int KS, bool LQ, bool LD>
__global__ void __launch_bounds__(32 * R64_WARPS, 2) k_rho64(Rho64Args a) {
    grid_dep();
    constexpr int NTL = (KS + 1) / 2, NCO = LD ? 4 : 2;
    extern __shared__ double2 sm[];
    double2 *qm = sm + a.nbuf * R64_TI * a.stw;  // [nbuf][R64_TI][2]: (q, m0), (m1, m2)
    const int l = threadIdx.x & 31, w = threadIdx.x >> 5, lk = l & 3, lr = l >> 2;
    const int zg = blockIdx.z;
    const int rr = blockIdx.x * R64_ROWS + 8 * w + lr;
    const KRow R = a.row[min(rr, a.nrow - 1)];
    const int i0 = blockIdx.y * a.chunk, i1 = min(a.n, i0 + a.chunk);
    const int ns = (i1 - i0 + R64_TI - 1) / R64_TI;
    const int zs = a.t.e1 + 2 * a.t.K1 + 1;      // stage offset of the Z columns
    // 16 threads per ion copy its row; positions past the chunk repeat a valid row and carry
    // q = mu = 0.  The ion's index, charge and dipole are read one stage before they are used.
    const int ki = threadIdx.x >> 4, xi = threadIdx.x & 15;
    int ia = 0;
    double qn = 0.0;
    double3 mn = make_double3(0.0, 0.0, 0.0);
    auto fetch = [&](int s) {
        const int pos = i0 + s * R64_TI + ki, pc = min(pos, i1 - 1);
        ia = a.idx ? a.idx[pc] : pc;
        if (xi == 0) {
            qn = 0.0;
            mn = make_double3(0.0, 0.0, 0.0);
            if (pos < i1) {
                if (LQ) qn = a.q[ia];
                if (LD) mn = a.mu[ia];
            }
        }
    };
    auto issue = [&](int b) {
        const double2 *src = a.tab + (size_t)ia * a.t.w;
        double2 *dst = sm + (b * R64_TI + ki) * a.stw;
        for (int x = xi; x < zs; x += 16) cp_async16(dst + x, src + x);
        for (int x = xi; x < 4 * NTL; x += 16) cp_async16(dst + zs + x, src + a.t.z + ZG * zg + x);
        if (xi == 0) {
            const double3 m = LD ? to_phase(a.c, TPI_D * mn.x, TPI_D * mn.y, TPI_D * mn.z) : make_double3(0, 0, 0);
            qm[(b * R64_TI + ki) * 2] = make_double2(qn, m.x);
            qm[(b * R64_TI + ki) * 2 + 1] = make_double2(m.y, m.z);
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    double acc[NCO][NTL][2];
#pragma unroll
    for (int f = 0; f < NCO; f++)
#pragma unroll
        for (int j = 0; j < NTL; j++) acc[f][j][0] = acc[f][j][1] = 0.0;
    const double nx = (double)R.nx, ny = (double)R.ny;
    const int x0 = R.nx, x1 = a.t.e1 + a.t.K1 + R.ny;
    const bool two = a.nbuf == 2;
    fetch(0);
    if (two) {
        issue(0);
        fetch(1);
    }
    for (int s = 0; s < ns; s++) {
        const int b = two ? s & 1 : 0;
        if (!two) {
            issue(0);
            fetch(s + 1);
        }
        if (two && s + 1 < ns) {
            issue(b ^ 1);
            fetch(s + 2);
            asm volatile("cp.async.wait_group 1;" ::: "memory");
        } else {
            asm volatile("cp.async.wait_group 0;" ::: "memory");
        }
        __syncthreads();
#pragma unroll
        for (int k4 = 0; k4 < R64_TI / 4; k4++) {
            const int k = b * R64_TI + 4 * k4 + lk;
            const double2 *T = sm + k * a.stw;
            const double2 e0 = T[x0], e1 = T[x1];
            const double2 qa = qm[2 * k];
            const double bx = e0.x * e1.x - e0.y * e1.y, by = e0.x * e1.y + e0.y * e1.x;
            double A[NCO];
            if (LD) {
                const double2 m12 = qm[2 * k + 1];
                const double c0 = nx * qa.y + ny * m12.x, c1 = m12.y;
                A[0] = LQ ? qa.x * bx - c0 * by : -c0 * by;
                A[1] = LQ ? qa.x * by + c0 * bx : c0 * bx;
                A[NCO - 2] = -c1 * by;
                A[NCO - 1] = c1 * bx;
            } else {
                A[0] = qa.x * bx;
                A[1] = qa.x * by;
            }
            const double *Z = (const double *)(T + zs) + lr;
#pragma unroll
            for (int j = 0; j < NTL; j++) {
                const double e = Z[8 * j];
#pragma unroll
                for (int f = 0; f < NCO; f++) dmma(acc[f][j], A[f], e);
            }
        }
        __syncthreads();
    }
    if (rr >= a.nrow) return;
    double2 *P = a.part + (size_t)blockIdx.y * a.nk + R.koff;
#pragma unroll
    for (int j = 0; j < NTL; j++) {
        const int z = ZG * zg + 4 * j + lk;
        if (z > a.t.K2) continue;
        const double zf = (double)z;
        double p1 = acc[0][j][0], p2 = acc[0][j][1], p3 = acc[1][j][0], p4 = acc[1][j][1];
        double q1 = 0.0, q2 = 0.0, q3 = 0.0, q4 = 0.0;
        if (LD) {
            q1 = zf * acc[NCO - 2][j][0], q2 = zf * acc[NCO - 2][j][1];
            q3 = zf * acc[NCO - 1][j][0], q4 = zf * acc[NCO - 1][j][1];
        }
        if (z >= R.z0) P[z - R.z0] = make_double2((p1 - p4) + (q1 - q4), (p2 + p3) + (q2 + q3));
        if (z > 0 && -z >= R.z0) P[-z - R.z0] = make_double2((p1 + p4) - (q1 + q4), (p3 - p2) - (q3 - q2));
    }
}

// ---------------------------------------------------------------- chunk sums, weights, energy
// One lane per (row, z >= 0): the chunk partials of rho(+z) and rho(-z) in a fixed order (8
// warps take every 8th chunk, warp 0 adds the warp sums), the ion pass's weights, and, when
// asked, the energy and virial sums over k (src/ewald.c:945-1006), reduced by the last block.
struct Red64Args {
    int npair, nchunk, nk, nrg, ks;
    Tab64 t;
    const double2 *part;
    const KRow *row;
    const double *Ak, *kcoe;
    const double3 *kv;
    double2 *rho_raw;            // null: not wanted
    double *w;                   // weights (null: not wanted)
    int wk;                      // the K weights too
    int energy;
    double *ppart, *scal;
    int slot, stride;
    unsigned *ticket;
};
__device__ __forceinline__ void k_energy(double (&v)[7], double2 rho, double ak, double co, double3 k) {
    const double str = (rho.x * rho.x + rho.y * rho.y) * ak;
    v[0] += str;
    v[1] += (1.0 - co * k.x * k.x) * str;
    v[2] += -co * k.x * k.y * str;
    v[3] += -co * k.x * k.z * str;
    v[4] += (1.0 - co * k.y * k.y) * str;
    v[5] += -co * k.y * k.z * str;
    v[6] += (1.0 - co * k.z * k.z) * str;
}
__global__ void __launch_bounds__(256) k_rho64_sum(Red64Args a) {
    grid_dep();
    __shared__ double2 wp[8][32], wm[8][32];
    const int w = threadIdx.x >> 5, l = threadIdx.x & 31, Z1 = a.t.K2 + 1;
    const int p = blockIdx.x * 32 + l;
    const bool act = p < a.npair;
    const int rr = act ? p / Z1 : 0, z = act ? p - rr * Z1 : 0;
    const KRow R = a.row[rr];
    const bool okp = act && z >= R.z0, okm = act && z > 0 && -z >= R.z0;
    const int kp = R.koff + z - R.z0, km = R.koff - z - R.z0;
    double2 sp = make_double2(0.0, 0.0), sn = sp;
    if (a.nchunk > 1) {
#pragma unroll 4
        for (int c = w; c < a.nchunk; c += 8) {
            const double2 *P = a.part + (size_t)c * a.nk;
            if (okp) {
                const double2 u = P[kp];
                sp.x += u.x, sp.y += u.y;
            }
            if (okm) {
                const double2 u = P[km];
                sn.x += u.x, sn.y += u.y;
            }
        }
        wp[w][l] = sp;
        wm[w][l] = sn;
        __syncthreads();
        if (w == 0) {
#pragma unroll
            for (int q = 1; q < 8; q++) {
                sp.x += wp[q][l].x, sp.y += wp[q][l].y;
                sn.x += wm[q][l].x, sn.y += wm[q][l].y;
            }
        }
    } else if (w == 0) {
        if (okp) sp = a.part[kp];
        if (okm) sn = a.part[km];
    }
    if (w == 0) {
        if (a.rho_raw) {
            if (okp) a.rho_raw[kp] = sp;
            if (okm) a.rho_raw[km] = sn;
        }
        const double akp = okp ? a.Ak[kp] : 0.0, akm = okm ? a.Ak[km] : 0.0;
        if (a.energy) {
            double v[7] = {0, 0, 0, 0, 0, 0, 0};
            if (okp) k_energy(v, sp, akp, a.kcoe[kp], a.kv[kp]);
            if (okm) k_energy(v, sn, akm, a.kcoe[km], a.kv[km]);
#pragma unroll
            for (int q = 0; q < 7; q++) {
                v[q] = warp_sum(v[q]);
                if (l == q) a.ppart[(size_t)(a.slot + q) * a.stride + blockIdx.x] = v[q];
            }
        }
        if (a.w && act) {
            // s = Ak (rho+ + rho-), d = Ak (rho+ - rho-): columns c_z and d_z of G, H, K
            const double sx = akp * sp.x + akm * sn.x, sy = akp * sp.y + akm * sn.y;
            const double dx = akp * sp.x - akm * sn.x, dy = akp * sp.y - akm * sn.y;
            const double zf = (double)z, zz = zf * zf;
            const int unit = (z / ZG) * a.nrg + (rr >> 2), zl = z % ZG;
            // fragment order: [unit][G|H|K][k step][lane], lane = 4 (2 (row % 4) + comp) + col % 4
            double *o = a.w + ((size_t)unit * 3 * a.ks + (zl >> 1)) * 32 + 4 * (2 * (rr & 3)) + 2 * (zl & 1);
            const size_t tile = (size_t)a.ks * 32;
            o[0] = sx, o[4] = sy, o[1] = dy, o[5] = -dx;
            o += tile;
            o[0] = zf * dx, o[4] = zf * dy, o[1] = zf * sy, o[5] = -zf * sx;
            if (a.wk) {
                o += tile;
                o[0] = zz * sx, o[4] = zz * sy, o[1] = zz * dy, o[5] = -zz * dx;
            }
        }
    }
    if (a.energy) {
        const int slots[7] = {a.slot, a.slot + 1, a.slot + 2, a.slot + 3, a.slot + 4, a.slot + 5, a.slot + 6};
        last_block_warps(a.ppart, a.stride, slots, 7, a.scal, a.ticket);
    }
}

// ---------------------------------------------------------------- ion pass
struct Ion64Args {
    int cnt;                 // output ions (idx[cnt], or all)
    const int *idx;
    int nrg, units, slices;  // row groups of 4, units = z groups x row groups, slices of the units
    Tab64 t;
    Cell c;
    const double2 *tab;
    const double *w;
    const double2 *rowxy;    // (nx, ny), padded to whole groups
    double *part;            // [slice][cnt][3 or 9]
    unsigned *btick;         // one per block of ions
    double tfpiV, self2, coul;
    int ld;
    const double *q;         // charges of the force (null: none)
    const double3 *mu;       // dipoles of the force
    const double3 *ef_dir;
    double3 *ef;
    const double3 *f_dir;
    double3 *f;
    double *efg;
    const double *efg_dir;
    const double *qself;     // self terms use q and mu whatever lq/ld (src/ewald.c:201-224)
    const double3 *muself;
    CgAp cg;
    CoulFin fin;
};

// the results of one ion from its sums S = sum n Im, Hm = sum n n^T Re (n-space)
template <bool WF>
__device__ __forceinline__ double ion64_write(const Ion64Args &a, int i, const double (&S)[9]) {
    const Cell &c = a.c;
    const double tpi = TPI_D;
    double gS[3], pap = 0.0;
#pragma unroll
    for (int k = 0; k < 3; k++) gS[k] = tpi * (c.B[k][0] * S[0] + c.B[k][1] * S[1] + c.B[k][2] * S[2]);
    if (a.ef) {
        const double3 mu = a.muself ? a.muself[i] : make_double3(0, 0, 0);
        double3 b = make_double3(a.self2 * mu.x, a.self2 * mu.y, a.self2 * mu.z);
        if (a.ef_dir) {
            const double3 d = a.ef_dir[i];
            b.x += d.x, b.y += d.y, b.z += d.z;
        }
        const double3 t = make_double3(b.x - a.tfpiV * gS[0], b.y - a.tfpiV * gS[1], b.z - a.tfpiV * gS[2]);
        a.ef[i] = t;
        if (!WF && a.cg.ap) {   // ap = invpol p - T p, and p.ap (k_cg_ap)
            const double3 m = a.cg.p[i];
            const double *I = a.cg.invpol + (size_t)i * 9;
            const double3 ap = make_double3(I[0] * m.x + I[1] * m.y + I[2] * m.z - t.x,
                                            I[3] * m.x + I[4] * m.y + I[5] * m.z - t.y,
                                            I[6] * m.x + I[7] * m.y + I[8] * m.z - t.z);
            a.cg.ap[i] = ap;
            pap = m.x * ap.x + m.y * ap.y + m.z * ap.z;
        }
    }
    if (WF) {
        const double H[3][3] = {{S[3], S[4], S[5]}, {S[4], S[6], S[7]}, {S[5], S[7], S[8]}};
        if (a.f) {
            double gP[3] = {0.0, 0.0, 0.0};
            if (a.ld) {   // sum_k k (k.mu) Re = (2 pi)^2 B H (B^T mu)
                const double3 mu = a.mu[i];
                const double3 m = to_phase(c, mu.x, mu.y, mu.z);
                double P[3];
#pragma unroll
                for (int k = 0; k < 3; k++) P[k] = H[k][0] * m.x + H[k][1] * m.y + H[k][2] * m.z;
#pragma unroll
                for (int k = 0; k < 3; k++)
                    gP[k] = tpi * tpi * (c.B[k][0] * P[0] + c.B[k][1] * P[1] + c.B[k][2] * P[2]);
            }
            const double qi = a.q ? a.q[i] : 0.0;
            double3 fo = a.f[i];
            if (a.f_dir) {
                const double3 d = a.f_dir[i];
                fo.x += d.x * a.coul, fo.y += d.y * a.coul, fo.z += d.z * a.coul;
            }
            double fr[3];
#pragma unroll
            for (int k = 0; k < 3; k++) fr[k] = a.tfpiV * (-qi * gS[k] + gP[k]);
            a.f[i] = make_double3(fo.x + fr[0] * a.coul, fo.y + fr[1] * a.coul, fo.z + fr[2] * a.coul);
        }
        if (a.efg) {   // (2 pi)^2 B H B^T, upper triangle only as in src/ewald.c:977-984
            for (int p = 0; p < 3; p++) {
                double BH[3];
                for (int k = 0; k < 3; k++)
                    BH[k] = c.B[p][0] * H[0][k] + c.B[p][1] * H[1][k] + c.B[p][2] * H[2][k];
                for (int k = 0; k < 3; k++) {
                    double v = 0.0;
                    if (k >= p)
                        v = a.tfpiV * tpi * tpi * (BH[0] * c.B[k][0] + BH[1] * c.B[k][1] + BH[2] * c.B[k][2]);
                    double b0 = (p == k && a.qself) ? -a.self2 * a.qself[i] : 0.0;
                    if (a.efg_dir) b0 += a.efg_dir[(size_t)i * 9 + 3 * p + k];
                    a.efg[(size_t)i * 9 + 3 * p + k] = b0 + v;
                }
            }
        }
    }
    return pap;
}

// WS = 1: grid (blocks of 32 MT ions, slices), the block's four warps hold four tiles of 8 MT
// ions.  WS = 8: grid (blocks of 8 MT ions, slices / 8), the block's eight warps take eight row
// slices of the same ions and add them in shared memory (few ions: the chip fills without
// partial sums in memory and their arrival counters, 11.8 -> 7.6 us at 128 ions, kmax 10).  A warp keeps
// its ions' table columns (the A fragments of all k steps) in registers and streams the
// weights (coalesced); with more than one slice in the grid the last block of an ion block to
// finish sums them in slice order and writes the results.
template <int KS, bool WF, int MT, int WS>
__global__ void __launch_bounds__(WS == 1 ? 32 * I64_WARPS : 32 * WS) k_ion64(Ion64Args a) {
    grid_dep();
    if (WF && a.fin.on && blockIdx.x == 0 && blockIdx.y == 0 && threadIdx.x == 0) finalize_coul(a.fin);
    constexpr int NTT = WF ? 3 : 2, NV = WF ? 9 : 3, IW = WS == 1 ? I64_WARPS : 1;   // warps over the ions
    const int l = threadIdx.x & 31, w = threadIdx.x >> 5, lk = l & 3, lr = l >> 2;
    const int base = (blockIdx.x * IW + (WS == 1 ? w : 0)) * 8 * MT;
    const double2 *T[MT];
#pragma unroll
    for (int m = 0; m < MT; m++) {
        const int pos = min(base + 8 * m + lr, a.cnt - 1);
        T[m] = a.tab + (size_t)(a.idx ? a.idx[pos] : pos) * a.t.w;
    }
    const int ns = a.slices * WS, sl = WS == 1 ? blockIdx.y : blockIdx.y * WS + w;
    const int u0 = (int)((long long)sl * a.units / ns);
    const int u1 = (int)((long long)(sl + 1) * a.units / ns);
    double A[MT][KS], S[MT][NV];
#pragma unroll
    for (int m = 0; m < MT; m++)
#pragma unroll
        for (int v = 0; v < NV; v++) S[m][v] = 0.0;
    // the next unit's weights are read into the registers each k step frees, its rows' phase
    // factors before the products, the (nx, ny) of its rows one unit earlier still
    double B[NTT * KS];
    double2 xy, e0[MT], e1[MT];
    auto rows_of = [&](int u) { return a.rowxy[4 * (min(u, u1 - 1) % a.nrg) + lk]; };
    auto factors = [&](double2 r) {
        const int x0 = (int)r.x, x1 = a.t.e1 + a.t.K1 + (int)r.y;
#pragma unroll
        for (int m = 0; m < MT; m++) e0[m] = T[m][x0], e1[m] = T[m][x1];
    };
    int zg = -1;
    if (u0 < u1) {
        const double *W = a.w + (size_t)u0 * 3 * KS * 32 + l;
#pragma unroll
        for (int s = 0; s < NTT * KS; s++) B[s] = W[s * 32];
        xy = rows_of(u0);
        factors(xy);
    }
    double2 xn = u0 < u1 ? rows_of(u0 + 1) : make_double2(0.0, 0.0);
    for (int u = u0; u < u1; u++) {
        const int g = u / a.nrg;
        if (g != zg) {
            zg = g;
#pragma unroll
            for (int m = 0; m < MT; m++)
#pragma unroll
                for (int s = 0; s < KS; s++) A[m][s] = ((const double *)(T[m] + a.t.z + ZG * g))[4 * s + lk];
        }
        const double fx = xy.x, fy = xy.y;
        double2 ph[MT];
#pragma unroll
        for (int m = 0; m < MT; m++)
            ph[m] = make_double2(e0[m].x * e1[m].x - e0[m].y * e1[m].y, e0[m].x * e1[m].y + e0[m].y * e1[m].x);
        xy = xn;
        factors(xy);
        xn = rows_of(u + 2);
        double acc[MT][NTT][2];
#pragma unroll
        for (int m = 0; m < MT; m++)
#pragma unroll
            for (int t = 0; t < NTT; t++) acc[m][t][0] = acc[m][t][1] = 0.0;
        const double *W = a.w + (size_t)min(u + 1, u1 - 1) * 3 * KS * 32 + l;
#pragma unroll
        for (int s = 0; s < KS; s++)
#pragma unroll
            for (int t = 0; t < NTT; t++) {
#pragma unroll
                for (int m = 0; m < MT; m++) dmma(acc[m][t], A[m][s], B[t * KS + s]);
                B[t * KS + s] = W[(t * KS + s) * 32];
            }
#pragma unroll
        for (int m = 0; m < MT; m++) {
            const double wx = ph[m].x, wy = ph[m].y;
            const double Rg = wx * acc[m][0][1] - wy * acc[m][0][0], Rh = wx * acc[m][1][1] - wy * acc[m][1][0];
            S[m][0] += fx * Rg;
            S[m][1] += fy * Rg;
            S[m][2] += Rh;
            if (WF) {
                const double Q0 = wx * acc[m][0][0] + wy * acc[m][0][1];
                const double Q1 = wx * acc[m][1][0] + wy * acc[m][1][1];
                const double Q2 = wx * acc[m][NTT - 1][0] + wy * acc[m][NTT - 1][1];
                const double a0 = fx * Q0, a1 = fy * Q0;
                S[m][NV - 6] += fx * a0;
                S[m][NV - 5] += fx * a1;
                S[m][NV - 4] += fx * Q1;
                S[m][NV - 3] += fy * a1;
                S[m][NV - 2] += fy * Q1;
                S[m][NV - 1] += Q2;
            }
        }
    }
    // the block's sums: per ion of the block, WS row slices each, in shared memory
    constexpr int NI = 8 * MT * IW;   // ions of the block
    __shared__ double red[WS][NI][NV];
#pragma unroll
    for (int m = 0; m < MT; m++)
#pragma unroll
        for (int v = 0; v < NV; v++) {
            double s = S[m][v];
            s += __shfl_xor_sync(0xffffffffu, s, 1);
            s += __shfl_xor_sync(0xffffffffu, s, 2);
            if (lk == 0) red[WS == 1 ? 0 : w][(WS == 1 ? 8 * MT * w : 0) + 8 * m + lr][v] = s;
        }
    __syncthreads();
    const int i0 = blockIdx.x * NI, ni = min(NI, a.cnt - i0);
    for (int k = threadIdx.x; k < NI * NV; k += blockDim.x) {
        const int q = k / NV, v = k - q * NV;
        double s = red[0][q][v];
#pragma unroll
        for (int x = 1; x < WS; x++) s += red[x][q][v];
        if (a.slices == 1) red[0][q][v] = s;
        else if (q < ni) a.part[((size_t)blockIdx.y * a.cnt + i0 + q) * NV + v] = s;
    }
    if (a.slices > 1) {   // the last slice of this ion block goes on, with all slices added
        __shared__ bool last;
        __threadfence();
        __syncthreads();
        if (threadIdx.x == 0) {
            last = atomicAdd(a.btick + blockIdx.x, 1u) == (unsigned)a.slices - 1u;
            if (last) a.btick[blockIdx.x] = 0u;
        }
        __syncthreads();
        if (!last) return;
        __threadfence();
        for (int k = threadIdx.x; k < ni * NV; k += blockDim.x) {
            const double *o = a.part + (size_t)i0 * NV + k;
            double s = 0.0;
#pragma unroll 4
            for (int x = 0; x < a.slices; x++) s += __ldcg(o + (size_t)x * a.cnt * NV);
            red[0][k / NV][k % NV] = s;
        }
    }
    __syncthreads();
    double pap[1] = {0.0};
    if ((int)threadIdx.x < ni) {
        double t[9] = {0, 0, 0, 0, 0, 0, 0, 0, 0};
#pragma unroll
        for (int v = 0; v < NV; v++) t[v] = red[0][threadIdx.x][v];
        pap[0] = ion64_write<WF>(a, a.idx ? a.idx[i0 + threadIdx.x] : i0 + threadIdx.x, t);
    }
    if (!WF && a.cg.ap && a.cg.part) {
        block_sum_to_part<1>(pap, a.cg.part, S_PAP, a.cg.stride);
        last_block_slots(a.cg.part, a.cg.stride, S_PAP, 1, a.cg.scal, a.cg.ticket);
    }
}

// ---------------------------------------------------------------- set-up and launchers
// algorithmic flops per (ion, k), FMA = 2
static double rho_flops_per_pair(bool lq, bool ld) { return ld ? 8.0 : (lq ? 4.0 : 0.0); }
static double ion_flops_per_pair(bool wf) { return wf ? 12.0 : 8.0; }

static Tab64 layout64(const Engine &e) {
    Tab64 t;
    t.K0 = e.kmax[0];
    t.K1 = e.kmax[1];
    t.K2 = e.kmax[2];
    t.nzg = ceil_div(t.K2 + 1, ZG);
    t.e1 = t.K0 + 1;
    t.z = t.e1 + 2 * t.K1 + 1;
    t.w = t.z + ZG * t.nzg;
    return t;
}

// k steps of 4 columns, (c_z, d_z) per |nz|, of one z group
static int ksteps64(const Engine &e) {
    const int cols = 2 * std::min(e.kmax[2] + 1, ZG);
    return cols <= 8 ? 2 : std::max(4, ceil_div(cols, 4));
}

// Mixed precision of few ions: the matrix instructions run at half the FP32 rate, but with two
// launches fewer per pass and no table of their own.  Up to REC64_IONS ions, unless padding or the
// size of the passes takes that back: both precisions pad |nz| (here to whole groups of ZG, there
// to kz_of), counted below in (ion, row, padded |nz|).  Measured, FP32 on CUDA cores against FP64.
// Polarisable MD, 10 steps, kmax 14: 192 ions 2885 / 2126 us, 648 ions 2187 / 1725, 1536 ions 2740 /
// 2580, 3000 ions 3396 / 3429.  Force evaluations, rigid and with dipoles: 1920 ions kmax 12 97 / 84
// and 417 / 409 us, kmax 15 109 / 97 and 484 / 457.  One |nz| past a group: kmax 16 999 ions (0.87e7
// more here) 99 / 101 and 462 / 447, 1296 ions (1.1e7) 101 / 122 and 478 / 530, 1920 ions 110 / 146 and
// 489 / 629; kmax 32 300 ions (1.0e7) 203 / 138 and 770 / 623, 648 ions (2.2e7) 212 / 198 and 849 /
// 932.  Large passes: 1296 ions kmax 24 (5.0e7 here) 197 / 171 and 812 / 704, 1920 ions kmax 20 (5.2e7)
// 195 / 232 and 762 / 820, 1536 ions kmax 31 (9.8e7) 309 / 270 and 1099 / 1282.
bool few_for_rec32(const Engine &e) {
    constexpr int REC64_IONS = 2048;
    constexpr double MORE = 1.05e7, MOST = 5e7;
    const double rows = (double)e.n * e.nrow;
    const double w64 = rows * ZG * ceil_div(e.kmax[2] + 1, ZG), w32 = rows * kz_of(e.kmax[2]);
    return e.n < REC64_IONS && w64 - w32 <= MORE && w64 <= MOST;
}

void setup_kspace64(Engine &e, const std::vector<KRow> &rows) {
    const Tab64 t = layout64(e);
    const int nrg = ceil_div(rows.size(), 4);
    e.tab64_w = t.w;
    e.rho64_chunks_max = std::max(1, std::min(64, ceil_div(e.n, R64_TI)));
    e.ion64_slices_max = std::max(1, std::min({t.nzg * nrg, 32, std::max(4, 65536 / e.n)}));
    // one allocation (each of more than half a megabyte costs 0.35 ms here and 0.27 ms when it is
    // freed), zeroed: padding rows and columns of the weights stay so
    size_t bytes = 0;
    auto take = [&](size_t b) {
        const size_t at = bytes;
        bytes += (b + 255) / 256 * 256;
        return at;
    };
    const size_t tab = take(sizeof(double2) * e.n * t.w), w = take(sizeof(double) * t.nzg * nrg * 3 * ksteps64(e) * 32),
                 rowxy = take(sizeof(double2) * nrg * 4), part = take(sizeof(double2) * e.rho64_chunks_max * e.nk),
                 btick = take(sizeof(unsigned) * (ceil_div(e.n, 8) + 1)),
                 ion_part = take(sizeof(double) * e.ion64_slices_max * e.n * 9);
    e.d_k64 = dalloc<char>(bytes);
    e.d_tab64 = (double2 *)(e.d_k64 + tab);
    e.d_w64 = (double *)(e.d_k64 + w);
    e.d_rowxy = (double2 *)(e.d_k64 + rowxy);
    e.d_rho_part = (double2 *)(e.d_k64 + part);
    e.d_btick = (unsigned *)(e.d_k64 + btick);
    e.d_ion_part = (double *)(e.d_k64 + ion_part);
    std::vector<double2> xy((size_t)nrg * 4, make_double2(0.0, 0.0));
    for (size_t r = 0; r < rows.size(); r++) xy[r] = make_double2(rows[r].nx, rows[r].ny);
    MDFF_CK(cudaMemcpy(e.d_rowxy, xy.data(), sizeof(double2) * xy.size(), cudaMemcpyHostToDevice));
}

static void launch_phase64(Engine &e) {
    const Tab64 t = layout64(e);
    const long long items = (long long)e.n * (t.K0 + 1 + t.K1 + 1 + ZG * t.nzg);
    MDFF_LAUNCH(e, k_phase64, ceil_div(items, 256), 256, 0, e.n, e.cell, t, e.d_r, e.d_tab64);
    e.phase64_ready = true;
}

template <int KS>
static void rho64_ks(Engine &e, const Rho64Args &a, dim3 grid, size_t smem, bool lq, bool ld) {
    auto go = [&](auto kernel) {
        if (smem > 48 * 1024)
            MDFF_CK(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
        MDFF_LAUNCH(e, kernel, grid, 32 * R64_WARPS, smem, a);
    };
    if (lq && ld) go(k_rho64<KS, true, true>);
    else if (lq) go(k_rho64<KS, true, false>);
    else go(k_rho64<KS, false, true>);
}

template <int KS, bool WF>
static void ion64_mt(Engine &e, const Ion64Args &a, dim3 grid, int mt, int ws) {
    constexpr int M4 = WF ? 2 : 4;
    if (ws == 8 && mt == 2) MDFF_LAUNCH(e, (k_ion64<KS, WF, 2, 8>), grid, 256, 0, a);
    else if (ws == 8) MDFF_LAUNCH(e, (k_ion64<KS, WF, 1, 8>), grid, 256, 0, a);
    else if (mt == 4) MDFF_LAUNCH(e, (k_ion64<KS, WF, M4, 1>), grid, 32 * I64_WARPS, 0, a);
    else MDFF_LAUNCH(e, (k_ion64<KS, WF, 2, 1>), grid, 32 * I64_WARPS, 0, a);
}

template <int KS>
static void ion64_ks(Engine &e, const Ion64Args &a, dim3 grid, int mt, int ws, bool wf) {
    if (wf) ion64_mt<KS, true>(e, a, grid, mt, ws);
    else ion64_mt<KS, false>(e, a, grid, mt, ws);
}

template <class F>
static void by_ksteps(int ks, F &&f) {
    switch (ks) {
    case 2: f(std::integral_constant<int, 2>()); break;
    case 4: f(std::integral_constant<int, 4>()); break;
    case 5: f(std::integral_constant<int, 5>()); break;
    case 6: f(std::integral_constant<int, 6>()); break;
    case 7: f(std::integral_constant<int, 7>()); break;
    default: f(std::integral_constant<int, 8>()); break;
    }
}

// rho(k) of (q, mu) over ions idx[cnt] (all when null), or the given rho_acc; weights,
// energies and rho_raw as `o` asks
static void rho64(Engine &e, const double *q, const double3 *mu, bool lq, bool ld, const int *idx, int cnt,
                  const RecOut &o, bool weights, bool wk) {
    const Tab64 t = layout64(e);
    const int ks = ksteps64(e);
    int chunks = 1;
    const double2 *part = o.rho_acc;
    if (!part) {
        // ion chunks: enough blocks for whole waves of the SMs without splitting the chunk
        // sums further than that (a stage of 16 ions is the unit of work; starting a block
        // costs about as much as one, each further chunk partial a little)
        const int rb = ceil_div(e.nrow, R64_ROWS) * t.nzg, stages = ceil_div(std::max(cnt, 1), R64_TI);
        double best = 1e300;
        int per = stages;
        for (int c = 1; c <= std::min(e.rho64_chunks_max, stages); c++) {
            const int p = ceil_div(stages, c), used = ceil_div(stages, p);
            const double cost = ceil_div(rb * used, e.split_sm) * (p + 1.0) + 0.02 * used;
            if (cost < best) {
                best = cost;
                per = p;
            }
        }
        chunks = ceil_div(stages, per);
        part = e.d_rho_part;
        if (!lq && !ld) {
            MDFF_CK(cudaMemsetAsync(e.d_rho_part, 0, sizeof(double2) * (size_t)e.nk * chunks, e.stream));
        } else {
            Rho64Args a;
            a.n = cnt;
            a.chunk = per * R64_TI;
            a.nrow = e.nrow;
            a.nk = e.nk;
            a.t = t;
            a.c = e.cell;
            const int ntl = (ks + 1) / 2;
            a.stw = t.z + 4 * ntl;
            a.stw += ((2 - a.stw) % 8 + 8) % 8;
            a.tab = e.d_tab64;
            a.q = q;
            a.mu = mu;
            a.idx = idx;
            a.row = e.d_row;
            a.part = e.d_rho_part;
            const size_t buf = sizeof(double2) * R64_TI * (a.stw + 2);
            a.nbuf = 2 * buf <= 227 * 1024 ? 2 : 1;
            const size_t smem = a.nbuf * buf;
            if (smem > 227 * 1024) throw Error(MDFFGPU_ERR_ARG, "kmax too large for the FP64 k-space pass");
            const dim3 grid(ceil_div(e.nrow, R64_ROWS), chunks, t.nzg);
            int ps = -1;
            e.prof_begin("k_rho", &ps);
            by_ksteps(ks, [&](auto k) { rho64_ks<decltype(k)::value>(e, a, grid, smem, lq, ld); });
            e.prof_end("k_rho", ps, rho_flops_per_pair(lq, ld) * (double)cnt * e.nk);
        }
    }
    Red64Args r;
    r.npair = e.nrow * (t.K2 + 1);
    r.nchunk = chunks;
    r.nk = e.nk;
    r.nrg = ceil_div(e.nrow, 4);
    r.ks = ks;
    r.t = t;
    r.part = part;
    r.row = e.d_row;
    r.Ak = e.d_Ak;
    r.kcoe = e.d_kcoe;
    r.kv = e.d_kvec;
    r.rho_raw = o.rho_raw;
    r.w = weights ? e.d_w64 : nullptr;
    r.wk = wk;
    r.energy = o.energy;
    r.ppart = e.d_part;
    r.scal = e.d_scal;
    r.slot = (int)S_REC_U;
    r.stride = e.part_stride;
    r.ticket = e.d_ticket + 2;
    MDFF_LAUNCH(e, k_rho64_sum, ceil_div(r.npair, 32), 256, 0, r);
}

void launch_rec64(Engine &e, const double *q, const double3 *mu, bool lq, bool ld, const RecOut &o) {
    if (!e.phase64_ready) launch_phase64(e);
    // ion subsets: the rho pass sums over o.idx (all ions when null; q and mu vanish
    // elsewhere), the ion pass writes at o.out_idx, else at o.idx, else at every ion
    const int *out_idx = o.out_idx ? o.out_idx : o.idx;
    const int out_n = o.out_idx ? o.out_cnt : (o.idx ? o.cnt : e.n);
    const bool wf = o.f || o.efg, any = wf || o.ef;
    rho64(e, q, mu, lq, ld, o.idx, o.idx ? o.cnt : e.n, o, any, wf);
    if (!any) return;
    if (o.cg.ap && (wf || !o.ef)) throw Error(MDFFGPU_ERR_STATE, "the CG product needs a field-only pass");
    // what the results add to may have run beside the passes above
    e.join_side(Engine::SIDE_DIR);
    e.join_side(Engine::SIDE_SR);
    e.join_side(Engine::SIDE_PREP);
    e.join_side(Engine::SIDE_BODY);
    e.join_side(Engine::SIDE_FIELD);
    const Tab64 t = layout64(e);
    Ion64Args a;
    a.cnt = out_n;
    a.idx = out_idx;
    a.nrg = ceil_div(e.nrow, 4);
    a.units = a.nrg * t.nzg;
    a.t = t;
    a.c = e.cell;
    a.tab = e.d_tab64;
    a.w = e.d_w64;
    a.rowxy = e.d_rowxy;
    a.part = e.d_ion_part;
    a.btick = e.d_btick;
    a.tfpiV = 2.0 * 2.0 * TPI_D * e.cell.inveOmega;
    a.self2 = o.self2;
    a.coul = o.coul;
    a.ld = ld;
    a.q = lq ? q : nullptr;
    a.mu = mu;
    a.ef_dir = o.ef_dir;
    a.ef = o.ef;
    a.f_dir = o.f_dir;
    a.f = o.f;
    a.efg = o.efg;
    a.efg_dir = o.efg_dir;
    a.qself = o.self_q;
    a.muself = o.self_mu;
    a.cg = o.cg;
    a.fin = o.fin;
    // tiles of 8 ions per warp, row slices within the block (ws) and of the grid: time in units
    // of one (row group, tile) per scheduler, plus the start of the block (8 units) and, with
    // slices in memory, the arrival and second read (16); several tiles per warp share each
    // weight load
    int mt = 1, ws = 8;
    a.slices = 1;
    double best = 1e300;
    for (int w = 1; w <= 8; w += 7)
        for (int m = w == 8 ? 1 : 2; m <= ((w == 8 || wf) ? 2 : 4); m *= 2) {
            const int blocks = ceil_div(std::max(out_n, 1), w == 8 ? 8 * m : 8 * m * I64_WARPS);
            const double unit = m * (m == 1 ? 1.3 : (m == 2 ? 1.1 : 1.0)) * (w == 8 ? 2.0 : 1.0);
            for (int s = 1; s <= e.ion64_slices_max && s * w <= std::max(a.units, 8); s++) {
                const double cost =
                    ceil_div(blocks * s, e.split_sm) * ceil_div(a.units, s * w) * unit + 8.0 + (s > 1 ? 16.0 : 0.0);
                if (cost < best) {
                    best = cost;
                    mt = m;
                    ws = w;
                    a.slices = s;
                }
            }
        }
    const int per_block = ws == 8 ? 8 * mt : 8 * mt * I64_WARPS;
    const dim3 grid(ceil_div(std::max(out_n, 1), per_block), a.slices);
    int pi = -1;
    e.prof_begin("k_rec_ion", &pi);
    by_ksteps(ksteps64(e), [&](auto k) { ion64_ks<decltype(k)::value>(e, a, grid, mt, ws, wf); });
    e.prof_end("k_rec_ion", pi, ion_flops_per_pair(wf) * (double)out_n * e.nk);
}

}  // namespace mdffgpu
