// Radial distribution function on the GPU: the pair histogram of get_gr
// (src/radial_distribution.c:180-230) for one configuration after another.
//
// get_gr counts every ordered pair (ia, ja != ia) whose minimum-image distance is below
// cutgr into bin (int)(r / resg) of gr[bin][type(ia)][type(ja)], with the distance
// computed as everywhere in the reference: positions to fractional coordinates
// (kardir), difference, nearbyint shift, back to Cartesian with A (pbc,
// src/pbc.c:7-14), r^2 = x^2 + y^2 + z^2, sqrt.  The kernel does the same FP64
// operations, each rounded once (no contraction), so every pair lands in the
// reference's bin and the integer counts are identical.  A pair's distance is the same
// both ways round (negation is exact through every step), so each unordered pair is
// evaluated and counted once; mdffgpu_rdf_counts adds the two orders up.
//
// What bounds it: instructions per pair (n^2 / 2 of them; half the pairs lie inside half the
// box width).  The exact distance, square root and division in FP64 are about 100 issue slots;
// only whether a pair is in range and its bin matter, so both are decided in FP32 where that is
// certain, and by the FP64 operations where the distance is within its error of a bin edge or of
// the cut-off (0.02% of the pairs at bins of 0.1 A and 35 A).  Coordinates are 32-bit fixed-point
// fractions, whose differences wrap to the minimum image by themselves and keep the relative
// error of the components; the error bound is GrErr's.  24000 ions, 351 bins: 965 -> 494 us a
// configuration (46 issue slots per 32 pairs, 0.82 issued per cycle).
//
// Layout: persistent blocks over (i tile, j tile) pairs of the upper triangle, the j tile in
// shared memory, one or two i per thread; each pair is counted once, under (type i, type j), in
// a block-private shared histogram, and added to both orders of the global 64-bit histogram when
// the block ends (global atomics directly when the histogram does not fit in shared memory).
#include <algorithm>
#include <cmath>
#include <cstring>
#include <string>
#include <type_traits>
#include <vector>

#include "engine.cuh"
#include "wrap32.h"

namespace mdffgpu {

constexpr int GR_THREADS = 256;
constexpr int GR_JT = 256;                // most ions of a j tile
constexpr int GR_SMEM_COUNTERS = 10240;   // 40 KB of 32-bit block counters (+ 4 KB of tile)

// positions (one array per component, or null: r) -> exact fractions s, fixed-point fractions
// with the type; *bad is set when a coordinate is not finite or so far out that its fraction
// loses digits (every pair is then decided in FP64)
__global__ void __launch_bounds__(256) k_gr_pack(int n, Cell c, const double *__restrict__ soa,
                                                 const double4 *__restrict__ r, const int *__restrict__ typ,
                                                 double4 *__restrict__ s, int4 *__restrict__ fx, int *bad) {
    grid_dep();
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    double x, y, z;
    if (soa) {
        x = soa[i], y = soa[n + i], z = soa[2 * (size_t)n + i];
    } else {
        const double4 q = r[i];
        x = q.x, y = q.y, z = q.z;
    }
    const double3 f = kardir(c, x, y, z);
    s[i] = make_double4(f.x, f.y, f.z, 0.0);
    if (!(fabs(f.x) < 1e6 && fabs(f.y) < 1e6 && fabs(f.z) < 1e6)) *bad = 1;
    auto fix = [](double u) { return (int)(unsigned)__double2ll_rn((u - rint(u)) * 4294967296.0); };
    fx[i] = make_int4(fix(f.x), fix(f.y), fix(f.z), typ[i]);
}

// FP32 decision: a[k] lattice entries x 2^-32 (row-major), bin coordinate r / resg known to
// within e1 (r / resg) + e0, in range below lo2 and out of range above hi2
struct GrErr {
    float a[9], inv, e1, e0, lo2, hi2;
};
struct GrArgs {
    int n, nt, nbins, jt, priv;
    Cell c;
    GrErr w;
    const double4 *s;
    const int4 *fx;
    double cut2, resg;
    unsigned long long *hist;
    const int *bad;
};

// the reference's bin of a pair, or -1 (outside)
__device__ __forceinline__ int gr_bin(const GrArgs &a, const double4 &si, const double4 &sj) {
    const double3 d = pbc_frac(a.c, dsub(si.x, sj.x), dsub(si.y, sj.y), dsub(si.z, sj.z));
    const double r2 = norm2_exact(d);
    if (!(r2 < a.cut2)) return -1;
    const int b = (int)__ddiv_rn(sqrt(r2), a.resg);
    return b < 0 || b >= a.nbins ? -1 : b;   // never past the end for nbins > cutgr / resg
}
__device__ __noinline__ int gr_exact(const GrArgs &a, int i, int j) { return gr_bin(a, a.s[i], a.s[j]); }

__device__ __forceinline__ float rsqrt_approx(float x) {
    float y;
    asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}

// the block's counters added to the histogram and cleared
__device__ __forceinline__ void gr_flush(const GrArgs &a, unsigned *h, int nh) {
    __syncthreads();
    for (int k = threadIdx.x; k < nh; k += GR_THREADS) {
        const unsigned c = h[k];
        if (!c) continue;
        atomicAdd(&a.hist[k], (unsigned long long)c);
        h[k] = 0u;
    }
    __syncthreads();
}

template <int IPT, bool ORTHO, bool PRIV>
__global__ void __launch_bounds__(GR_THREADS) k_gr_pairs(const __grid_constant__ GrArgs a) {
    grid_dep();
    extern __shared__ unsigned h_sh[];
    __shared__ int4 tile[GR_JT];
    const int np = a.nt * a.nt, nh = a.nbins * np;
    if (PRIV)
        for (int k = threadIdx.x; k < nh; k += GR_THREADS) h_sh[k] = 0u;
    const int nbi = (a.n + GR_THREADS * IPT - 1) / (GR_THREADS * IPT), nbj = (a.n + a.jt - 1) / a.jt;
    GrErr w = a.w;
    if (*a.bad != 0) w.hi2 = __int_as_float(0x7f800000), w.e0 = 1.0f;   // every pair in FP64
    const float thr0 = 0.5f - w.e0 - 0.5f * w.e1;
    // the certain counts of one block stay below 2^31 up to about 10^6 ions; past that they are
    // added to the global histogram on the way
    long long seen = 0;
    for (long long t = blockIdx.x; t < (long long)nbi * nbj; t += gridDim.x) {
        const int bi = (int)(t / nbj), bj = (int)(t - (long long)bi * nbj);
        const int i0 = bi * GR_THREADS * IPT, j0 = bj * a.jt, jn = min(a.jt, a.n - j0);
        if (j0 + jn - 1 <= i0) continue;   // no j > i here
        __syncthreads();
        for (int k = threadIdx.x; k < jn; k += GR_THREADS) tile[k] = a.fx[j0 + k];
        __syncthreads();
        int4 me[IPT];
        int lo[IPT];   // first j of the tile past i
#pragma unroll
        for (int m = 0; m < IPT; m++) {
            const int i = i0 + m * GR_THREADS + threadIdx.x;
            me[m] = a.fx[min(i, a.n - 1)];
            me[m].w *= a.nt;
            lo[m] = i < a.n ? max(0, i + 1 - j0) : jn;
        }
        // straight-line per pair; the one branch is the FP64 decision of the warp's open pairs
        auto scan = [&](auto diag) {
            constexpr bool DIAG = decltype(diag)::value;   // tiles that hold pairs with j <= i, or i >= n
#pragma unroll 2
            for (int jj = 0; jj < jn; jj++) {
                const int4 o = tile[jj];
#pragma unroll
                for (int m = 0; m < IPT; m++) {
                    const int dx = wrap_diff(me[m].x, o.x), dy = wrap_diff(me[m].y, o.y), dz = wrap_diff(me[m].z, o.z);
                    const float u = (float)dx, v = (float)dy, q = (float)dz;
                    float x, y, z;
                    bool edge = false;
                    if (ORTHO) {
                        x = u * w.a[0], y = v * w.a[4], z = q * w.a[8];
                    } else {
                        x = u * w.a[0] + v * w.a[3] + q * w.a[6];
                        y = u * w.a[1] + v * w.a[4] + q * w.a[7];
                        z = u * w.a[2] + v * w.a[5] + q * w.a[8];
                        // next to a half box edge the two images differ in a triclinic cell
                        edge = fmaxf(fabsf(u), fmaxf(fabsf(v), fabsf(q))) > 2147483000.0f;
                    }
                    const float r2 = x * x + y * y + z * z;
                    bool in = r2 < w.hi2 || edge;
                    if (DIAG) in = in && jj >= lo[m];
                    // floor by rounding x - 1/2; its distance to the halfway points is the
                    // distance to the bin edges (a NaN or a bin past 2^22 fails the test)
                    const float h = r2 * rsqrt_approx(r2) * w.inv - 0.5f;
                    const float y0 = h + 12582912.0f, fr = h - (y0 - 12582912.0f);
                    int b = __float_as_int(y0) - 0x4b400000;
                    const bool sure = fabsf(fr) < thr0 - w.e1 * h && r2 < w.lo2 && !edge;
                    if (__any_sync(0xffffffffu, in && !sure)) {
                        if (in && !sure) {
                            b = gr_exact(a, i0 + m * GR_THREADS + threadIdx.x, j0 + jj);
                            in = b >= 0;
                        }
                    }
                    const int k = b * np + me[m].w + o.w;
                    if (in) {
                        if (PRIV) atomicAdd(&h_sh[k], 1u);
                        else atomicAdd(&a.hist[k], 1ull);
                    }
                }
            }
        };
        if (j0 < i0 + GR_THREADS * IPT) scan(std::true_type());
        else scan(std::false_type());
        seen += (long long)GR_THREADS * IPT * jn;
        if (PRIV && seen > (1ll << 30)) {
            gr_flush(a, h_sh, nh);
            seen = 0;
        }
    }
    if (PRIV) gr_flush(a, h_sh, nh);
}

// Every pair by the FP64 operations, for bins so fine that FP32 would leave most warps an open pair
// (gr_fine): the same loop over tiles with one i per thread, the exact fractions in shared memory.
template <bool PRIV>
__global__ void __launch_bounds__(GR_THREADS) k_gr_fine(const __grid_constant__ GrArgs a) {
    grid_dep();
    extern __shared__ unsigned h_sh[];
    __shared__ double4 tile[GR_JT];
    __shared__ int ttile[GR_JT];
    const int np = a.nt * a.nt, nh = a.nbins * np;
    if (PRIV)
        for (int k = threadIdx.x; k < nh; k += GR_THREADS) h_sh[k] = 0u;
    const int nbi = (a.n + GR_THREADS - 1) / GR_THREADS, nbj = (a.n + a.jt - 1) / a.jt;
    long long seen = 0;
    for (long long t = blockIdx.x; t < (long long)nbi * nbj; t += gridDim.x) {
        const int bi = (int)(t / nbj), bj = (int)(t - (long long)bi * nbj);
        const int i0 = bi * GR_THREADS, j0 = bj * a.jt, jn = min(a.jt, a.n - j0);
        if (j0 + jn - 1 <= i0) continue;   // no j > i here
        __syncthreads();
        for (int k = threadIdx.x; k < jn; k += GR_THREADS) {
            tile[k] = a.s[j0 + k];
            ttile[k] = a.fx[j0 + k].w;
        }
        __syncthreads();
        const int i = i0 + threadIdx.x;
        if (i < a.n) {
            const double4 si = a.s[i];
            const int ti = a.fx[i].w * a.nt;
#pragma unroll 2
            for (int jj = max(0, i + 1 - j0); jj < jn; jj++) {
                const int b = gr_bin(a, si, tile[jj]);
                if (b < 0) continue;
                const int k = b * np + ti + ttile[jj];
                if (PRIV) atomicAdd(&h_sh[k], 1u);
                else atomicAdd(&a.hist[k], 1ull);
            }
        }
        seen += (long long)GR_THREADS * jn;
        if (PRIV && seen > (1ll << 30)) {
            gr_flush(a, h_sh, nh);
            seen = 0;
        }
    }
    if (PRIV) gr_flush(a, h_sh, nh);
}

// Whether to take k_gr_fine: a pair is open in FP32 with a chance of about 2 (e0 + 3/4 e1 nbins) (most
// pairs lie in the outer bins), and a warp is done by FP32 only where none of its 32 is.  Measured, in
// us, FP32 decision / all in FP64, bins to 0.45 of the box: triclinic cell, 1 type, 9000 ions, chance
// 0.020 211 / 216, 0.030 234 / 216; 20000 ions 0.030 859 / 880, 0.040 955 / 879; 40000 ions 0.030 3026 /
// 3184, 0.040 3358 / 3187; orthorhombic, 2 types, 20000 ions, 0.030 826 / 818, 0.040 909 / 822.
static bool gr_fine(const GrErr &w, int nbins) {
    return 2.0 * ((double)w.e0 + 0.75 * (double)w.e1 * nbins) > 0.033;
}

// lattice (src/cell.c:13-91) as far as kardir and pbc need it: A, B = (A_j x A_k) / omega
static Cell cell_of(const double *A9) {
    Cell c;
    memset(&c, 0, sizeof c);
    memcpy(c.A, A9, sizeof(c.A));
    const int nx[3] = {1, 2, 0}, ny[3] = {2, 0, 1};
    for (int i = 0; i < 3; i++) {
        const double *u = c.A[nx[i]], *v = c.A[ny[i]];
        c.B[i][0] = u[1] * v[2] - u[2] * v[1];
        c.B[i][1] = u[2] * v[0] - u[0] * v[2];
        c.B[i][2] = u[0] * v[1] - u[1] * v[0];
    }
    double omega = c.B[0][0] * c.A[0][0] + c.B[1][0] * c.A[1][0] + c.B[2][0] * c.A[2][0];
    if (!(omega > 0.0)) throw Error(MDFFGPU_ERR_ARG, "cell volume must be positive");
    c.omega = omega;
    c.inveOmega = 1.0 / omega;
    for (int i = 0; i < 3; i++)
        c.w[i] = omega / std::sqrt(c.B[0][i] * c.B[0][i] + c.B[1][i] * c.B[1][i] + c.B[2][i] * c.B[2][i]);
    for (int i = 0; i < 3; i++)
        for (int j = 0; j < 3; j++) c.B[i][j] = c.B[i][j] * c.inveOmega;
    return c;
}

}  // namespace mdffgpu

using mdffgpu::Engine;
using mdffgpu::Error;

struct mdffgpu_rdf {
    int n = 0, nt = 0, nbins = 0, device = 0, nconf = 0;
    double cut2 = 0.0, resg = 0.0;
    cudaStream_t stream = nullptr;
    double *d_soa = nullptr;      // positions of the configuration, one array per component
    double4 *d_s = nullptr;
    int4 *d_fx = nullptr;
    int *d_typ = nullptr, *d_bad = nullptr;
    unsigned long long *d_hist = nullptr;
    double *h_soa = nullptr;      // pinned staging
    long long launches = 0;
    std::string err;
};

namespace {

template <typename F>
int rdf_guarded(mdffgpu_rdf *r, F &&f) {
    if (!r) return MDFFGPU_ERR_ARG;
    try {
        MDFF_CK(cudaSetDevice(r->device));
        f(*r);
        return MDFFGPU_OK;
    } catch (const Error &x) {
        r->err = x.what();
        return x.code;
    } catch (const std::exception &x) {
        r->err = x.what();
        return MDFFGPU_ERR_CUDA;
    }
}

// one configuration: soa, or the positions of a context
void launch_gr(mdffgpu_rdf &r, const mdffgpu::Cell &c, const double *soa, const double4 *d_r, const int *d_typ,
               cudaStream_t st) {
    using namespace mdffgpu;
    MDFF_CK(cudaMemsetAsync(r.d_bad, 0, sizeof(int), st));
    k_gr_pack<<<ceil_div(r.n, 256), 256, 0, st>>>(r.n, c, soa, d_r, d_typ, r.d_s, r.d_fx, r.d_bad);
    MDFF_CK(cudaGetLastError());
    GrArgs a;
    a.n = r.n;
    a.nt = r.nt;
    a.nbins = r.nbins;
    a.c = c;
    a.s = r.d_s;
    a.fx = r.d_fx;
    a.cut2 = r.cut2;
    a.resg = r.resg;
    a.hist = r.d_hist;
    a.bad = r.d_bad;
    const int nh = r.nbins * r.nt * r.nt;
    a.priv = nh <= GR_SMEM_COUNTERS ? 1 : 0;
    const size_t smem = a.priv ? sizeof(unsigned) * nh : 0;
    // Error of the FP32 distance.  Each component: conversion of the fixed-point difference,
    // lattice entry and product, 3 x 2^-24 relative of its terms; squares, sum and root of r^2
    // half of 3 x 2^-24 more, the reciprocal root 2^-22, two products and 1 / resg 3 x 2^-24:
    // below 7e-7 of r in an orthorhombic cell (e1 takes 1.2e-6).  In a triclinic one the terms
    // cancel, which leaves 2e-7 of the lattice entries (e0 takes 1e-6 of their sum).  The
    // fixed-point rounding is 2^-32 of a lattice entry per component (2e-9 taken).
    double sum = 0.0;
    bool ortho = true;
    for (int k = 0; k < 9; k++) {
        const double v = c.A[k / 3][k % 3];
        sum += std::fabs(v);
        if (k / 3 != k % 3 && v != 0.0) ortho = false;
        a.w.a[k] = (float)(v / 4294967296.0);
    }
    const double abs_err = (ortho ? 2e-9 : 1e-6) * sum;
    const double cut = std::min(std::sqrt(r.cut2), r.nbins * r.resg);   // certain pairs have a bin
    a.w.inv = (float)(1.0 / r.resg);
    a.w.e1 = 1.2e-6f;
    a.w.e0 = (float)(abs_err / r.resg + 1e-7);
    const double m = 1.2e-6 * cut + abs_err, l = std::max(0.0, cut - m), h = std::sqrt(r.cut2) * (1.0 + 1.2e-6) + abs_err;
    a.w.lo2 = (float)(l * l * (1.0 - 2e-6));
    a.w.hi2 = (float)(h * h * (1.0 + 2e-6));
    int nsm = 148;
    cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, r.device);
    // two i per thread once that leaves several tile pairs per block; j tiles short enough for
    // the same (a block's start and its flush cost about as much as 20000 pairs)
    const bool fine = gr_fine(a.w, r.nbins);
    const int ipt = r.n >= 12288 && !fine ? 2 : 1, few = 4 * nsm;
    a.jt = fine ? GR_JT / 4 : GR_JT;
    while (a.jt > 32 && (long long)ceil_div(r.n, GR_THREADS * ipt) * ceil_div(r.n, a.jt) < 8ll * few) a.jt /= 2;
    const long long tiles = (long long)ceil_div(r.n, GR_THREADS * ipt) * ceil_div(r.n, a.jt);
    // in FP64 a tile is long, so blocks are handed out as others end: 16 per SM where each has counters
    // to add up, one per tile otherwise (us, tiles of 256 j at 4 blocks per SM / so, triclinic cell: 20000
    // ions, 5000 bins 1093 / 882, 30000 bins of 2 types 1126 / 822; 9000 ions 254 / 218 and 259 / 217)
    const long long most = !fine ? few : a.priv ? 4 * few : 1ll << 30;
    const int grid = (int)std::min(most, tiles);
    auto go = [&](auto kernel) { kernel<<<grid, GR_THREADS, smem, st>>>(a); };
    auto by_cell = [&](auto two, auto priv) {
        constexpr int I = decltype(two)::value ? 2 : 1;
        if (ortho) go(k_gr_pairs<I, true, decltype(priv)::value>);
        else go(k_gr_pairs<I, false, decltype(priv)::value>);
    };
    if (fine && a.priv) {   // (with its tile of fractions past the default limit)
        MDFF_CK(cudaFuncSetAttribute(k_gr_fine<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
        go(k_gr_fine<true>);
    } else if (fine) go(k_gr_fine<false>);
    else if (ipt == 2 && a.priv) by_cell(std::true_type(), std::true_type());
    else if (ipt == 2) by_cell(std::true_type(), std::false_type());
    else if (a.priv) by_cell(std::false_type(), std::true_type());
    else by_cell(std::false_type(), std::false_type());
    MDFF_CK(cudaGetLastError());
    r.launches += 2;
}

}  // namespace

mdffgpu::Engine *mdffgpu_engine_of(mdffgpu_ctx *ctx);

extern "C" {

int mdffgpu_rdf_create(int nion, int ntype, const int *nionit, double cutgr, double resg, int nbins, int device,
                       mdffgpu_rdf **out) {
    if (!out || !nionit || nion <= 0 || ntype <= 0 || ntype > MDFFGPU_NTMAX || !(resg > 0.0) || !(cutgr > 0.0) ||
        nbins <= 0)
        return MDFFGPU_ERR_ARG;
    *out = nullptr;
    long long tot = 0;
    for (int t = 0; t < ntype; t++) tot += nionit[t] < 0 ? -1000000000LL : nionit[t];
    if (tot != nion) return MDFFGPU_ERR_ARG;
    if ((long long)nbins * ntype * ntype > (1LL << 28)) return MDFFGPU_ERR_ARG;
    mdffgpu_rdf *r = new mdffgpu_rdf();
    r->n = nion;
    r->nt = ntype;
    r->nbins = nbins;
    r->device = device;
    r->cut2 = cutgr * cutgr;
    r->resg = resg;
    int rc = rdf_guarded(r, [&](mdffgpu_rdf &x) {
        MDFF_CK(cudaStreamCreateWithFlags(&x.stream, cudaStreamNonBlocking));
        x.d_soa = mdffgpu::dalloc<double>(3 * (size_t)nion);
        x.d_s = mdffgpu::dalloc<double4>(nion);
        x.d_fx = mdffgpu::dalloc<int4>(nion);
        x.d_bad = mdffgpu::dalloc<int>(1);
        x.d_typ = mdffgpu::dalloc<int>(nion);
        x.d_hist = mdffgpu::dalloc<unsigned long long>((size_t)nbins * ntype * ntype);
        MDFF_CK(cudaMallocHost((void **)&x.h_soa, 3 * sizeof(double) * nion));
        std::vector<int> typ(nion);
        for (int t = 0, ia = 0; t < ntype; t++)
            for (int k = 0; k < nionit[t]; k++) typ[ia++] = t;
        MDFF_CK(cudaMemcpy(x.d_typ, typ.data(), sizeof(int) * nion, cudaMemcpyHostToDevice));
        // (from pageable memory it may return before the device has it; the kernels run on their own
        // stream.  Not the whole device: a stream another thread records on must not be waited for)
        MDFF_CK(cudaStreamSynchronize(0));
    });
    if (rc != MDFFGPU_OK) {
        mdffgpu_rdf_destroy(r);
        return rc;
    }
    *out = r;
    return MDFFGPU_OK;
}

int mdffgpu_rdf_destroy(mdffgpu_rdf *r) {
    if (!r) return MDFFGPU_ERR_ARG;
    cudaSetDevice(r->device);
    cudaFree(r->d_soa);
    cudaFree(r->d_s);
    cudaFree(r->d_fx);
    cudaFree(r->d_bad);
    cudaFree(r->d_typ);
    cudaFree(r->d_hist);
    if (r->h_soa) cudaFreeHost(r->h_soa);
    if (r->stream) cudaStreamDestroy(r->stream);
    delete r;
    return MDFFGPU_OK;
}

const char *mdffgpu_rdf_last_error(const mdffgpu_rdf *r) { return r ? r->err.c_str() : "null rdf"; }

int mdffgpu_rdf_reset(mdffgpu_rdf *r) {
    return rdf_guarded(r, [&](mdffgpu_rdf &x) {
        MDFF_CK(cudaMemsetAsync(x.d_hist, 0, sizeof(unsigned long long) * x.nbins * x.nt * x.nt, x.stream));
        MDFF_CK(cudaStreamSynchronize(x.stream));
        x.nconf = 0;
    });
}

int mdffgpu_rdf_add(mdffgpu_rdf *r, const double *cell, const double *rx, const double *ry, const double *rz) {
    if (!cell || !rx || !ry || !rz) return MDFFGPU_ERR_ARG;
    return rdf_guarded(r, [&](mdffgpu_rdf &x) {
        mdffgpu::Cell c = mdffgpu::cell_of(cell);
        const size_t b = sizeof(double) * x.n;
        memcpy(x.h_soa, rx, b);
        memcpy(x.h_soa + x.n, ry, b);
        memcpy(x.h_soa + 2 * (size_t)x.n, rz, b);
        MDFF_CK(cudaMemcpyAsync(x.d_soa, x.h_soa, 3 * b, cudaMemcpyHostToDevice, x.stream));
        launch_gr(x, c, x.d_soa, nullptr, x.d_typ, x.stream);
        MDFF_CK(cudaStreamSynchronize(x.stream));
        x.nconf++;
    });
}

int mdffgpu_rdf_add_ctx(mdffgpu_rdf *r, mdffgpu_ctx *ctx) {
    Engine *e = mdffgpu_engine_of(ctx);
    if (!e) return MDFFGPU_ERR_ARG;
    return rdf_guarded(r, [&](mdffgpu_rdf &x) {
        if (e->n != x.n || e->nt != x.nt || e->device != x.device)
            throw Error(MDFFGPU_ERR_ARG, "rdf_add_ctx: the context holds another system or device");
        // the context's positions and types, on its stream (one less host round trip)
        launch_gr(x, e->cell, nullptr, e->d_r, e->d_typ, e->stream);
        MDFF_CK(cudaStreamSynchronize(e->stream));
        x.nconf++;
    });
}

int mdffgpu_rdf_counts(mdffgpu_rdf *r, long long *pairs, int *nconf) {
    if (!pairs) return MDFFGPU_ERR_ARG;
    return rdf_guarded(r, [&](mdffgpu_rdf &x) {
        size_t nh = (size_t)x.nbins * x.nt * x.nt;
        MDFF_CK(cudaMemcpyAsync(pairs, x.d_hist, sizeof(unsigned long long) * nh, cudaMemcpyDeviceToHost, x.stream));
        MDFF_CK(cudaStreamSynchronize(x.stream));
        // both orders of every pair: (ti, tj) and (tj, ti) hold their sum, like pairs count twice
        for (size_t b = 0; b < (size_t)x.nbins; b++) {
            long long *h = pairs + b * x.nt * x.nt;
            for (int ti = 0; ti < x.nt; ti++)
                for (int tj = ti; tj < x.nt; tj++)
                    h[ti * x.nt + tj] = h[tj * x.nt + ti] = h[ti * x.nt + tj] + h[tj * x.nt + ti];
        }
        if (nconf) *nconf = x.nconf;
    });
}

}  // extern "C"
