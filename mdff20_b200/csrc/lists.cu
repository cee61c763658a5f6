// Verlet neighbour lists on the GPU: gen_pbc_verletlist / check_verletlist
// (src/verlet.c:54-170) rebuilt as cell-binned, warp-per-ion FULL lists.
//
// The reference keeps a half list (each pair once, parity rule src/verlet.c:82-83)
// and scatters forces to both ions.  Here every ion keeps all its neighbours, so each
// force kernel writes only its own ion (no atomics, deterministic sums); the pair
// SET equals the reference's because every distance is computed with the reference's
// operation order (kardir, nearbyint minimum image, A-multiply, x^2+y^2+z^2, no FMA)
// and tested with the same inclusive `<= (rc+skin)^2` (src/verlet.c:90,99).
#include <algorithm>
#include <cmath>

#include "step.cuh"

namespace mdffgpu {

// s = kardir(r), w = charge; f (may be null) = 0
__global__ void k_kardir(int n, Cell c, const double4 *__restrict__ r, double4 *__restrict__ s,
                         double3 *__restrict__ f) {
    grid_dep();
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    double4 ri = r[i];
    double3 q = kardir(c, ri.x, ri.y, ri.z);
    s[i] = make_double4(q.x, q.y, q.z, ri.w);
    if (f) f[i] = make_double3(0.0, 0.0, 0.0);
}

void launch_kardir(Engine &e, const double4 *r, double4 *s, double3 *f) {
    MDFF_LAUNCH(e, k_kardir, ceil_div(e.n, 256), 256, 0, e.n, e.cell, r, s, f);
    e.phase64_ready = false;   // the positions may have moved
}

// ---------------------------------------------------------------- check_verletlist
// check_verletlist in one launch: the fractional coordinates of the current positions
// (kardir, written to s for a rebuild), each ion's displacement since the last build and
// the skin test in the last block (step.cuh).  The kernels that close a step do the same
// without a launch of their own.
__global__ void __launch_bounds__(256) k_check_list(CheckArgs a, const double4 *__restrict__ r, unsigned *ticket) {
    grid_dep();
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    double m = 0.0;
    if (i < a.n) {
        const double4 ri = r[i];
        const double3 f = kardir(a.c, ri.x, ri.y, ri.z);
        const double4 si = make_double4(f.x, f.y, f.z, ri.w);
        a.s[i] = si;
        m = check_moved(a, si, i);
    }
    check_block(a, m);
    if (last_block(ticket)) check_last(a);
}

__global__ void k_force_rebuild(int *rebuild, DevScalars *out) {
    grid_dep();
    *rebuild = 1;
    out->rebuild = 1;
    out->nbuilds += 1;
}

CheckArgs check_args(Engine &e, const cudaGraphConditionalHandle *h) {
    CheckArgs a;
    a.on = 1;
    a.n = e.n;
    a.ncell = e.ncell;
    a.c = e.cell;
    a.s = e.d_s;
    a.svl = e.d_svl;
    a.part1 = e.d_part + (size_t)S_DISP1 * e.part_stride;
    a.part2 = e.d_part + (size_t)S_DISP2 * e.part_stride;
    a.skindiff = e.p.skindiff;
    a.rebuild = e.d_rebuild;
    a.cell_cnt = e.d_cell_cnt;
    a.out = e.d_out;
    a.h = h ? *h : cudaGraphConditionalHandle{};
    a.use_h = h != nullptr;
    return a;
}

void launch_check_list(Engine &e, const cudaGraphConditionalHandle *h) {
    MDFF_LAUNCH(e, k_check_list, ceil_div(e.n, 256), 256, 0, check_args(e, h), e.d_r, e.d_ticket + 5);
}

// ---------------------------------------------------------------- cell binning
__device__ __forceinline__ int cell_coord(double s, int ncd) {
    double u = s - floor(s);
    int c = (int)(u * (double)ncd);
    return c < 0 ? 0 : (c >= ncd ? ncd - 1 : c);
}

// svl (may be null): the positions of this build
__global__ void k_bin(int n, int3 nc, const double4 *__restrict__ s, int *__restrict__ cell_of,
                      int *__restrict__ cnt, double4 *__restrict__ svl, const int *__restrict__ rebuild) {
    grid_dep();
    if (!*rebuild) return;
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    double4 si = s[i];
    int cx = cell_coord(si.x, nc.x), cy = cell_coord(si.y, nc.y), cz = cell_coord(si.z, nc.z);
    int c = (cx * nc.y + cy) * nc.z + cz;
    cell_of[i] = c;
    if (svl) svl[i] = si;
    atomicAdd(&cnt[c], 1);
}

// exclusive scan of the cell counts (one block), resets the fill cursors
__global__ void k_scan_cells(int ncell, const int *__restrict__ cnt, int *__restrict__ start, int *__restrict__ cur,
                             int cell_cap, unsigned *status, const int *__restrict__ rebuild) {
    grid_dep();
    if (!*rebuild) return;
    __shared__ int carry;
    __shared__ int wsum[32];
    if (threadIdx.x == 0) carry = 0;
    __syncthreads();
    for (int base = 0; base < ncell; base += blockDim.x) {
        int i = base + threadIdx.x;
        int v = (i < ncell) ? cnt[i] : 0;
        if (i < ncell && v > cell_cap) atomicOr(status, ST_CELL_OVERFLOW);
        int x = v;
        int l = threadIdx.x & 31, w = threadIdx.x >> 5;
        for (int o = 1; o < 32; o <<= 1) {
            int y = __shfl_up_sync(0xffffffffu, x, o);
            if (l >= o) x += y;
        }
        if (l == 31) wsum[w] = x;
        __syncthreads();
        if (w == 0) {
            int t = (l < (int)(blockDim.x >> 5)) ? wsum[l] : 0;
            for (int o = 1; o < 32; o <<= 1) {
                int y = __shfl_up_sync(0xffffffffu, t, o);
                if (l >= o) t += y;
            }
            wsum[l] = t;
        }
        __syncthreads();
        int excl = x - v + (w > 0 ? wsum[w - 1] : 0) + carry;
        if (i < ncell) {
            start[i] = excl;
            cur[i] = 0;
        }
        __syncthreads();
        if (threadIdx.x == blockDim.x - 1) carry = excl + v;
        __syncthreads();
    }
}

__global__ void k_fill_cells(int n, const int *__restrict__ cell_of, const int *__restrict__ start,
                             int *__restrict__ cur, int *__restrict__ ions, const int *__restrict__ rebuild) {
    grid_dep();
    if (!*rebuild) return;
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    int c = cell_of[i];
    int k = atomicAdd(&cur[c], 1);
    ions[start[c] + k] = i;
}

// sort each cell's ion indices ascending (bitonic in shared memory) so that the list
// order, hence every pair sum, is the same from run to run; pk receives, in that order, the
// fractional coordinates wrapped to [-1/2, 1/2] in FP32 with the index in w (the candidates
// of k_build's first test, read there without a gather).  An ion 2^20 boxes away or more gets NaN:
// its differences to other ions round by more than k_build's shells allow for, so FP64 decides
// all its pairs.
__global__ void k_sort_cells(int ncell, int cell_cap, const int *__restrict__ start, const int *__restrict__ cnt,
                             int *__restrict__ ions, const double4 *__restrict__ s, float4 *__restrict__ pk,
                             const int *__restrict__ rebuild) {
    grid_dep();
    if (!*rebuild) return;
    extern __shared__ int sh[];
    int c = blockIdx.x;
    if (c >= ncell) return;
    int m = cnt[c];
    int b = start[c];
    auto pack = [&](int k, int j) {
        const double4 p = s[j];
        const bool far = !(fmax(fabs(p.x), fmax(fabs(p.y), fabs(p.z))) < 1048576.0);
        pk[b + k] = make_float4(far ? __int_as_float(0x7fffffff) : (float)(p.x - rint(p.x)),
                                (float)(p.y - rint(p.y)), (float)(p.z - rint(p.z)), __int_as_float(j));
    };
    if (m <= 1 || m > cell_cap) {
        for (int k = threadIdx.x; k < m; k += blockDim.x) pack(k, ions[b + k]);
        return;
    }
    int p2 = 1;
    while (p2 < m) p2 <<= 1;
    for (int k = threadIdx.x; k < p2; k += blockDim.x) sh[k] = (k < m) ? ions[b + k] : 0x7fffffff;
    __syncthreads();
    for (int size = 2; size <= p2; size <<= 1) {
        for (int stride = size >> 1; stride > 0; stride >>= 1) {
            for (int k = threadIdx.x; k < p2; k += blockDim.x) {
                int j = k ^ stride;
                if (j > k) {
                    bool up = ((k & size) == 0);
                    int a = sh[k], bb = sh[j];
                    if ((a > bb) == up) {
                        sh[k] = bb;
                        sh[j] = a;
                    }
                }
            }
            __syncthreads();
        }
    }
    for (int k = threadIdx.x; k < m; k += blockDim.x) {
        ions[b + k] = sh[k];
        pack(k, sh[k]);
    }
}

// ---------------------------------------------------------------- list build
// Each warp takes G consecutive ions of the cell order (mostly one cell's) and scans their 27
// (or fewer, for thin cells) neighbour cells in a fixed order, appending, in order, every j with
// |r_ij|^2 <= cut^2 to both lists of each ion.  Bound by instructions (8 candidates per
// neighbour): the pair is decided in FP32 where that is certain, and by the reference's FP64
// operations only in a shell around each radius (BuildCut, about 1e-4 A wide: a few candidates
// per ion), so the pair sets stay exact; a candidate is loaded and placed once for the G ions.
// Measured against testing every candidate in FP64 (B200, cuts 8 and 11 A): 24000 ions 367 ->
// 275 us (G = 4), 6000 ions 120 -> 79 us (G = 2), 3000 ions 62 -> 60 us (G = 1: few warps, so
// ions per warp would cost more occupancy than they save).  All ions in one cell (whole call): 4000
// ions 234 -> 223 us (G = 2; 237 with G = 1), 6000 ions 505 -> 399, 2048 ions 137 -> 125 (G = 1; 128
// with G = 2), 8000 ions 604 -> 571.
// NEAR (at least three cells in each dimension, orthorhombic): candidates are placed relative
// to the cell's centre, which fixes the periodic image of every pair within the cut.
struct BuildCut {
    float lo_nb, hi_nb, lo_co, hi_co;   // r^2 below lo: inside; above hi: outside; between: FP64 decides
    double rsq_nb, rsq_co;
};
struct BuildArgs {
    int n;
    Cell c;
    int3 nc;
    const double4 *s;
    const int *cell_of, *start, *cnt;
    const float4 *pk;
    BuildCut cut;
    int cap_nb, *nbl, *nbn, cap_co, *col, *con;
    unsigned *status;
    const int *rebuild;
};
constexpr int BUILD_WARPS = 8;
template <int G, bool NEAR>
__global__ void __launch_bounds__(BUILD_WARPS * 32) k_build(BuildArgs a) {
    grid_dep();
    if (!*a.rebuild) return;
    const int p0 = ((blockIdx.x * blockDim.x + threadIdx.x) >> 5) * G;
    const int lane = threadIdx.x & 31;
    if (p0 >= a.n) return;
    const int ng = min(G, a.n - p0);
    // lane g holds ion g
    const float4 me = a.pk[min(p0 + lane, a.n - 1)];
    const int my_i = __float_as_int(me.w), my_cell = a.cell_of[my_i];
    const int3 nc = a.nc;
    const int rx = nc.x >= 3 ? 1 : 0, ry = nc.y >= 3 ? 1 : 0, rz = nc.z >= 3 ? 1 : 0;
    float A[9];
#pragma unroll
    for (int k = 0; k < 9; k++) A[k] = (float)a.c.A[k / 3][k % 3];
    const BuildCut q = a.cut;
    const float hi = fmaxf(q.hi_nb, q.hi_co);
    // the shells as |r^2 - mid| <= half (4e-7 for the roundings of that form): three instructions
    // fewer per candidate.  One ion per warp over its cells keeps the comparisons of r^2 itself
    // (2048 ions 67 us, 75 with this form)
    constexpr bool MID = !NEAR || G > 1;
    const float mid_nb = 0.5f * (q.lo_nb + q.hi_nb), half_nb = 0.5f * (q.hi_nb - q.lo_nb) + 4e-7f * q.hi_nb;
    const float mid_co = 0.5f * (q.lo_co + q.hi_co), half_co = 0.5f * (q.hi_co - q.lo_co) + 4e-7f * q.hi_co;
    const unsigned lt = (1u << lane) - 1u;
    int knb[G], kco[G];
#pragma unroll
    for (int g = 0; g < G; g++) knb[g] = kco[g] = 0;
    unsigned left = (1u << ng) - 1u;
    while (left) {
        // the next run of ions that share a cell
        const int ci = __shfl_sync(0xffffffffu, my_cell, __ffs(left) - 1);
        const unsigned run = __ballot_sync(0xffffffffu, my_cell == ci) & left;
        left &= ~run;
        const int cx = ci / (nc.y * nc.z), cy = (ci / nc.z) % nc.y, cz = ci % nc.z;
        const float ox = ((float)cx + 0.5f) / (float)nc.x, oy = ((float)cy + 0.5f) / (float)nc.y,
                    oz = ((float)cz + 0.5f) / (float)nc.z;
        float mx = me.x, my = me.y, mz = me.z;
        if (NEAR) {
            mx -= ox, my -= oy, mz -= oz;
            mx = (mx - rintf(mx)) * A[0], my = (my - rintf(my)) * A[4], mz = (mz - rintf(mz)) * A[8];
        }
        int ig[G];
        float gx[G], gy[G], gz[G];
#pragma unroll
        for (int g = 0; g < G; g++) {
            ig[g] = __shfl_sync(0xffffffffu, my_i, g);
            gx[g] = __shfl_sync(0xffffffffu, mx, g);
            gy[g] = __shfl_sync(0xffffffffu, my, g);
            gz[g] = __shfl_sync(0xffffffffu, mz, g);
        }
        auto scan = [&](int b, int e) {
            float4 p = a.pk[min(b + lane, a.n - 1)];
            for (int base = b; base < e; base += 32) {
                const bool in = base + lane < e;
                const int j = __float_as_int(p.w);
                float px = p.x, py = p.y, pz = p.z;
                bool edge = false;
                p = a.pk[min(base + 32 + lane, a.n - 1)];
                if (NEAR) {
                    px -= ox, py -= oy, pz -= oz;
                    px -= rintf(px), py -= rintf(py), pz -= rintf(pz);
                    // next to the half box edge FP32 may pick the other image: FP64 decides
                    edge = fmaxf(fabsf(px), fmaxf(fabsf(py), fabsf(pz))) > 0.4999f;
                    px *= A[0], py *= A[4], pz *= A[8];
                }
#pragma unroll
                for (int g = 0; g < G; g++) {
                    if (!(run >> g & 1u)) continue;
                    float x = px - gx[g], y = py - gy[g], z = pz - gz[g];
                    if (!NEAR) {
                        x -= rintf(x), y -= rintf(y), z -= rintf(z);
                        edge = fmaxf(fabsf(x), fmaxf(fabsf(y), fabsf(z))) > 0.4999f;
                        const float u = x, v = y, w = z;
                        x = u * A[0] + v * A[3] + w * A[6];
                        y = u * A[1] + v * A[4] + w * A[7];
                        z = u * A[2] + v * A[5] + w * A[8];
                    }
                    const float r2 = x * x + y * y + z * z;
                    bool in_nb, in_co, open;
                    if (MID) {
                        const bool cand = in && j != ig[g];
                        const float d = fminf(fabsf(r2 - mid_nb) - half_nb, fabsf(r2 - mid_co) - half_co);
                        open = cand && (edge || !(d > 0.0f));
                        in_nb = cand && r2 < mid_nb, in_co = cand && r2 < mid_co;
                    } else {
                        const bool cand = in && j != ig[g] && (edge || !(r2 > hi));
                        in_nb = cand && !edge && r2 < q.lo_nb, in_co = cand && !edge && r2 < q.lo_co;
                        open = cand && (edge || (!in_nb && !(r2 > q.hi_nb)) || (!in_co && !(r2 > q.hi_co)));
                    }
                    if (__any_sync(0xffffffffu, open)) {
                        if (open) {
                            const double4 si = a.s[ig[g]], sj = a.s[j];
                            const double3 d = pbc_frac(a.c, dsub(si.x, sj.x), dsub(si.y, sj.y), dsub(si.z, sj.z));
                            const double e2 = norm2_exact(d);
                            in_nb = (e2 <= q.rsq_nb);
                            in_co = (e2 <= q.rsq_co);
                        }
                    }
                    const unsigned bnb = __ballot_sync(0xffffffffu, in_nb);
                    const unsigned bco = __ballot_sync(0xffffffffu, in_co);
                    if (in_nb) {
                        const int pos = knb[g] + __popc(bnb & lt);
                        if (pos < a.cap_nb) a.nbl[(size_t)ig[g] * a.cap_nb + pos] = j;
                    }
                    if (in_co) {
                        const int pos = kco[g] + __popc(bco & lt);
                        if (pos < a.cap_co) a.col[(size_t)ig[g] * a.cap_co + pos] = j;
                    }
                    knb[g] += __popc(bnb);
                    kco[g] += __popc(bco);
                }
            }
        };
        for (int dx = -rx; dx <= rx; dx++) {
            int x = cx + dx;
            x += x < 0 ? nc.x : (x >= nc.x ? -nc.x : 0);
            for (int dy = -ry; dy <= ry; dy++) {
                int y = cy + dy;
                y += y < 0 ? nc.y : (y >= nc.y ? -nc.y : 0);
                const int row = (x * nc.y + y) * nc.z;
                if (rz == 1 && cz > 0 && cz < nc.z - 1) {   // the three cells are one run
                    scan(a.start[row + cz - 1], a.start[row + cz + 1] + a.cnt[row + cz + 1]);
                } else {
                    for (int dz = -rz; dz <= rz; dz++) {
                        int z = cz + dz;
                        z += z < 0 ? nc.z : (z >= nc.z ? -nc.z : 0);
                        scan(a.start[row + z], a.start[row + z] + a.cnt[row + z]);
                    }
                }
            }
        }
    }
    bool over = false;
#pragma unroll
    for (int g = 0; g < G; g++)
        if (lane == g && g < ng) {
            a.nbn[my_i] = knb[g];
            a.con[my_i] = kco[g];
            over = knb[g] > a.cap_nb || kco[g] > a.cap_co;
        }
    if (over) atomicOr(a.status, ST_LIST_OVERFLOW);
}

// The FP32 shell of one list radius: FP32 decides outside it.  Wrapped fractional coordinates
// in FP32 are off by at most 2^-26 each; a component difference, taken through the cell centre
// and with its image, by less than 2.5e-7; a Cartesian component by less than 3.5e-7 times the
// sum of |A|, and the distance by sqrt(3) of that.  The shell is three times as wide.
static void build_shell(const Cell &c, double r, float *lo, float *hi) {
    double sum = 0.0;
    for (int k = 0; k < 9; k++) sum += std::fabs(c.A[k / 3][k % 3]);
    const double w = 2e-6 * (sum + r), l = std::max(0.0, r - w), h = r + w;
    *lo = (float)(l * l * (1.0 - 1e-6));
    *hi = (float)(h * h * (1.0 + 1e-6));
}

void run_build(cudaStream_t st, bool pdl, int n, const Cell &c, const int nc[3], const double4 *s, const int *cell_of,
               const int *start, const int *cnt, const float4 *pk, double cut_nb, double cut_co, int cap_nb, int *nbl,
               int *nbn, int cap_co, int *col, int *con, unsigned *status, const int *rebuild) {
    BuildArgs a;
    a.n = n;
    a.c = c;
    a.nc = make_int3(nc[0], nc[1], nc[2]);
    a.s = s;
    a.cell_of = cell_of;
    a.start = start;
    a.cnt = cnt;
    a.pk = pk;
    build_shell(c, cut_nb, &a.cut.lo_nb, &a.cut.hi_nb);
    build_shell(c, cut_co, &a.cut.lo_co, &a.cut.hi_co);
    a.cut.rsq_nb = cut_nb * cut_nb;
    a.cut.rsq_co = cut_co * cut_co;
    a.cap_nb = cap_nb;
    a.nbl = nbl;
    a.nbn = nbn;
    a.cap_co = cap_co;
    a.col = col;
    a.con = con;
    a.status = status;
    a.rebuild = rebuild;
    cudaLaunchAttribute at;
    at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at.val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t cfg = {};
    cfg.blockDim = dim3(BUILD_WARPS * 32);
    cfg.stream = st;
    cfg.attrs = &at;
    cfg.numAttrs = pdl ? 1 : 0;
    const bool near = nc[0] >= 3 && nc[1] >= 3 && nc[2] >= 3;
    auto go = [&](auto kernel, int g) {
        cfg.gridDim = dim3(ceil_div(n, g * BUILD_WARPS));
        MDFF_CK(cudaLaunchKernelEx(&cfg, kernel, a));
    };
    if (!near && n >= 3000) go(k_build<2, false>, 2);
    else if (!near) go(k_build<1, false>, 1);
    else if (n >= 16384) go(k_build<4, true>, 4);
    else if (n >= 4096) go(k_build<2, true>, 2);
    else go(k_build<1, true>, 1);
}

void launch_build_lists(Engine &e, bool force) {
    if (force) MDFF_LAUNCH(e, k_force_rebuild, 1, 1, 0, e.d_rebuild, e.d_out);
    int3 nc = make_int3(e.nc[0], e.nc[1], e.nc[2]);
    // after k_check_list the counts are zero already when a rebuild is due
    if (force) MDFF_CK(cudaMemsetAsync(e.d_cell_cnt, 0, sizeof(int) * e.ncell, e.stream));
    MDFF_LAUNCH(e, k_bin, ceil_div(e.n, 256), 256, 0, e.n, nc, e.d_s, e.d_cell_of, e.d_cell_cnt, e.d_svl,
                e.d_rebuild);
    MDFF_LAUNCH(e, k_scan_cells, 1, 1024, 0, e.ncell, e.d_cell_cnt, e.d_cell_start, e.d_cell_cur, e.cell_cap,
                e.d_status, e.d_rebuild);
    MDFF_LAUNCH(e, k_fill_cells, ceil_div(e.n, 256), 256, 0, e.n, e.d_cell_of, e.d_cell_start, e.d_cell_cur,
                e.d_cell_ions, e.d_rebuild);
    MDFF_LAUNCH(e, k_sort_cells, e.ncell, 256, sizeof(int) * e.cell_cap, e.ncell, e.cell_cap, e.d_cell_start,
                e.d_cell_cnt, e.d_cell_ions, e.d_s, e.d_cell_pk, e.d_rebuild);
    double cnb = e.p.cutshortrange + e.p.skindiff, cco = e.p.cutlongrange + e.p.skindiff;
    if (!e.p.lverletL) {  // no lists in the reference: every pair inside the cutoff itself
        cnb = e.p.cutshortrange;
        cco = e.p.cutlongrange;
    }
    run_build(e.stream, e.pdl, e.n, e.cell, e.nc, e.d_s, e.d_cell_of, e.d_cell_start, e.d_cell_cnt, e.d_cell_pk, cnb, cco,
              e.cap_nb, e.d_nb, e.d_nbn, e.cap_co, e.d_co, e.d_con, e.d_status, e.d_rebuild);
    e.launches++;
}

// ---------------------------------------------------------------- CSR half list
// verlet_nb / verlet_coul (src/verlet.h:8-16) from the full rows: (i, j) is kept when the
// parity rule of src/verlet.c:82-83 holds, j ascending.  Bound by the copy of the result to
// the host: the host loop with a sort per row over the copied padded rows took 93 ms for the
// two lists of 6000 ions (1.5 M pairs), these kernels 0.03 ms.
__device__ __forceinline__ bool half_keep(int i, int j) { return i > j ? ((i + j) & 1) == 0 : (i < j && ((i + j) & 1)); }

// one warp per row: pairs of the row in the half list
__global__ void __launch_bounds__(256) k_half_count(int n, int cap, const int *__restrict__ list,
                                                    const int *__restrict__ cnt, int *__restrict__ out) {
    grid_dep();
    const int i = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, l = threadIdx.x & 31;
    if (i >= n) return;
    const int m = min(cnt[i], cap);
    const int *L = list + (size_t)i * cap;
    int c = 0;
    for (int k = l; k < m; k += 32) c += half_keep(i, L[k]);
    for (int o = 16; o > 0; o >>= 1) c += __shfl_xor_sync(0xffffffffu, c, o);
    if (l == 0) out[i] = c;
}

// inclusive sums of one value per thread over a block (w: 32 ints of shared memory)
__device__ __forceinline__ int block_scan(int v, int *w) {
    const int l = threadIdx.x & 31, q = threadIdx.x >> 5;
    for (int o = 1; o < 32; o <<= 1) {
        const int y = __shfl_up_sync(0xffffffffu, v, o);
        if (l >= o) v += y;
    }
    if (l == 31) w[q] = v;
    __syncthreads();
    int b = 0;
    for (int k = 0; k < q; k++) b += w[k];
    return v + b;
}

// row starts point[0..n] from the row counts in point[1..n] (one block, each thread a run of rows)
__global__ void __launch_bounds__(1024) k_half_scan(int n, int *__restrict__ point) {
    grid_dep();
    __shared__ int w[32];
    const int per = (n + (int)blockDim.x - 1) / (int)blockDim.x;
    const int b = min(n, (int)threadIdx.x * per), e = min(n, b + per);
    int s = 0;
    for (int k = b; k < e; k++) s += point[k + 1];
    int run = block_scan(s, w) - s;
    for (int k = b; k < e; k++) {
        run += point[k + 1];
        point[k + 1] = run;
    }
    if (threadIdx.x == 0) point[0] = 0;
}

// one block per row: the kept j as bits of a window of HALF_WIN ions in shared memory, read
// back in ascending order (no sort); the first `room` entries of the list
constexpr int HALF_WIN = 65536;
__global__ void __launch_bounds__(128) k_half_fill(int n, int cap, const int *__restrict__ list,
                                                   const int *__restrict__ cnt, const int *__restrict__ point,
                                                   int *__restrict__ out, size_t room) {
    grid_dep();
    extern __shared__ unsigned bits[];
    __shared__ int w[32];
    const int i = blockIdx.x, m = min(cnt[i], cap);
    const int *L = list + (size_t)i * cap;
    int at = point[i];
    for (int w0 = 0; w0 < n; w0 += HALF_WIN) {
        const int nw = (min(n - w0, HALF_WIN) + 31) >> 5;
        for (int k = threadIdx.x; k < nw; k += blockDim.x) bits[k] = 0u;
        __syncthreads();
        for (int k = threadIdx.x; k < m; k += blockDim.x) {
            const int j = L[k];
            if (half_keep(i, j) && j >= w0 && j - w0 < HALF_WIN)
                atomicOr(&bits[(j - w0) >> 5], 1u << ((j - w0) & 31));
        }
        __syncthreads();
        const int per = (nw + (int)blockDim.x - 1) / (int)blockDim.x;
        const int b = min(nw, (int)threadIdx.x * per), e = min(nw, b + per);
        int c = 0;
        for (int k = b; k < e; k++) c += __popc(bits[k]);
        const int incl = block_scan(c, w);
        int pos = at + incl - c;
        for (int k = b; k < e; k++)
            for (unsigned u = bits[k]; u; u &= u - 1, pos++)
                if ((size_t)pos < room) out[pos] = w0 + 32 * k + __ffs(u) - 1;
        __syncthreads();
        if (threadIdx.x == blockDim.x - 1) w[0] = incl;
        __syncthreads();
        at += w[0];
        __syncthreads();
    }
}

// the list in CSR form into host arrays point[n + 1], list[cap] (list may be null); *count: pairs
void Engine::half_list(int which, int *point, int *list, int cap, int *count) {
    if (!list_ready) throw Error(MDFFGPU_ERR_STATE, "no Verlet list built");
    const int c = which ? cap_co : cap_nb;
    const int *L = which ? d_co : d_nb, *m = which ? d_con : d_nbn;
    if (!d_csr_point) d_csr_point = dalloc<int>((size_t)n + 1);
    MDFF_LAUNCH(*this, k_half_count, ceil_div((long long)n * 32, 256), 256, 0, n, c, L, m, d_csr_point + 1);
    MDFF_LAUNCH(*this, k_half_scan, 1, 1024, 0, n, d_csr_point);
    const size_t smem = sizeof(unsigned) * ((std::min(n, HALF_WIN) + 31) / 32);
    auto fill = [&](size_t room) {
        if (room > csr_room) {
            // kept between calls, for either list at the present capacities (a pair is in two rows of
            // the full list): one allocation for the first calls of a context
            if (d_csr_list) MDFF_CK(cudaFree(d_csr_list));
            d_csr_list = nullptr;
            csr_room = 0;
            d_csr_list = dalloc<int>(room);
            csr_room = room;
        }
        MDFF_LAUNCH(*this, k_half_fill, n, 128, smem, n, c, L, m, d_csr_point, d_csr_list, csr_room);
    };
    // filled while the row starts are on their way (launched after their wait: 32 ions 65 us for both
    // calls of a list, so 62; 256 ions 78 and 76)
    if (list) fill((size_t)n * std::max(cap_nb, cap_co) / 2);
    MDFF_CK(cudaMemcpyAsync(point, d_csr_point, sizeof(int) * (n + 1), cudaMemcpyDeviceToHost, stream));
    MDFF_CK(cudaStreamSynchronize(stream));
    const int tot = point[n];
    if (count) *count = tot;
    if (list && tot > 0) {
        if ((size_t)tot > csr_room) fill(tot);
        MDFF_CK(cudaMemcpyAsync(list, d_csr_list, sizeof(int) * std::min(tot, std::max(cap, 0)), cudaMemcpyDeviceToHost,
                                stream));
        MDFF_CK(cudaStreamSynchronize(stream));
    }
    if (list && tot > cap) throw Error(MDFFGPU_ERR_ARG, "list buffer too small");
}

}  // namespace mdffgpu
