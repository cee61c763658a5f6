// One warp over the neighbour list of one ion: the pairs inside the cut-off are queued in shared
// memory and handed out 32 at a time, so that the pair terms run with every lane at work.  A
// list that holds the skin is 1.4 to 2 times longer than the cut-off sphere (its ions sit at
// random places of the list), and without the queue the lanes outside wait for the FP64
// exponentials, error function and division of the others.
// STRICT: pairs with d2 < cutsq, else those with !(d2 > cutsq); of them those with want(j);
// f(k, j, r, d2) for the k-th, count of them in `total`.
#pragma once

#include "common.cuh"

namespace mdffgpu {

struct PairQ {
    double x[64], y[64], z[64];
    int j[64];
};

template <bool STRICT, class W, class F>
__device__ __forceinline__ void pairs_in_cut(const Cell &c, const double4 *__restrict__ s, const double4 &si,
                                             const int *__restrict__ L, int m, double cutsq, PairQ &q, W &&want,
                                             int &total, F &&f) {
    const int lane = threadIdx.x & 31;
    int cnt = 0;
    total = 0;
    // positions one chunk ahead, indices two chunks ahead
    int jc = lane < m ? L[lane] : 0;
    int jn = lane + 32 < m ? L[lane + 32] : 0;
    double4 sc = lane < m ? s[jc] : si;
    for (int k0 = 0;; k0 += 32) {   // one round more than the list has: the rest of the queue
        if (k0 < m) {
            const int k = k0 + lane, j = jc;
            const double4 sj = sc;
            if (k + 32 < m) sc = s[jn];
            jc = jn;
            if (k + 64 < m) jn = L[k + 64];
            const double3 r = pbc_frac(c, dsub(si.x, sj.x), dsub(si.y, sj.y), dsub(si.z, sj.z));
            const double d2 = norm2_exact(r);
            const bool keep = k < m && (STRICT ? d2 < cutsq : !(d2 > cutsq)) && want(j);
            const unsigned b = __ballot_sync(0xffffffffu, keep);
            if (keep) {
                const int p = cnt + __popc(b & ((1u << lane) - 1u));
                q.j[p] = j;
                q.x[p] = r.x;
                q.y[p] = r.y;
                q.z[p] = r.z;
            }
            cnt += __popc(b);
            __syncwarp();
            if (cnt < 32) continue;
        }
        if (lane < cnt) {
            const double3 r = make_double3(q.x[lane], q.y[lane], q.z[lane]);
            f(total + lane, q.j[lane], r, norm2_exact(r));
        }
        __syncwarp();
        total += cnt < 32 ? cnt : 32;
        if (k0 >= m) break;
        cnt -= 32;
        if (lane < cnt) {   // the rest moves to the front (distinct halves)
            q.j[lane] = q.j[32 + lane];
            q.x[lane] = q.x[32 + lane];
            q.y[lane] = q.y[32 + lane];
            q.z[lane] = q.z[32 + lane];
        }
        __syncwarp();
    }
}

template <bool STRICT, class F>
__device__ __forceinline__ void pairs_in_cut(const Cell &c, const double4 *__restrict__ s, const double4 &si,
                                             const int *__restrict__ L, int m, double cutsq, PairQ &q, F &&f) {
    int total;
    pairs_in_cut<STRICT>(
        c, s, si, L, m, cutsq, q, [](int) { return true; }, total,
        [&](int, int j, const double3 &r, double d2) { f(j, r, d2); });
}

// the screened factors of src/ewald.c:562-603 at squared distance d2: erfc(alpha d) and the F_k
// from one exponential and one reciprocal square root
struct Screened {
    double d, dm1, dm3, dm5, F0, F1, F2, ex;   // ex = exp(-alpha^2 d^2) / sqrt(pi)
};
__device__ __forceinline__ Screened screened(double d2, double alpha) {
    Screened v;
    v.dm1 = rsqrt(d2);
    v.d = d2 * v.dm1;
    const double dm2 = v.dm1 * v.dm1, ad = alpha * v.d;
    v.dm3 = v.dm1 * dm2;
    v.dm5 = v.dm3 * dm2;
    v.ex = exp(-alpha * alpha * d2) * 0.56418958354775628695;
    v.F0 = erfc(ad);
    v.F1 = v.F0 + 2.0 * ad * v.ex;
    v.F2 = v.F1 + (4.0 / 3.0) * (ad * ad * ad) * v.ex;
    return v;
}

}  // namespace mdffgpu
