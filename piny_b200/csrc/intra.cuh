// Pieces of the intramolecular terms shared by their kernels: block sums of
// energies and virial, one bend, one excluded pair.
#pragma once

#include "common.cuh"

namespace pinyb200 {

// Per-thread sums v of a block, thread t holding bead t % P (P a power of two
// up to 64, blockDim a multiple of 32 and P up to 256), added to
// acc[bead][slot]: lanes of one bead by shuffles, then the block's warps
// through shared memory, then one global atomic per (bead, slot).  Every
// thread of the block must call it.  (Shared FP64 atomics instead of the
// shuffles serialise: with one bead all 256 threads of a block met at 7
// addresses, and each of the three intramolecular kernels took 35-41 us of
// the 256- and 4096-molecule boxes.)
template <int NV>
__device__ __forceinline__ void block_acc(double *acc, int P, const int *slot, const double *v)
{
    __shared__ double sh[NV][8][32];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, nw = blockDim.x >> 5;
    const int G = P < 32 ? P : 32;
#pragma unroll
    for (int c = 0; c < NV; c++) {
        const double t = warp_sum_strided(v[c], G);
        if (lane < G) sh[c][w][lane] = t;
    }
    __syncthreads();
    const int wstep = P > 32 ? P / 32 : 1;  // warps w, w + wstep, ... hold the same beads
    for (int i = threadIdx.x; i < P * NV; i += blockDim.x) {
        const int c = i / P, b = i - c * P;
        double t = 0.0;
        for (int k = b >> 5; k < nw; k += wstep) t += sh[c][k][b & 31];
        if (t != 0.0) atomicAdd(&acc[(size_t)b * S_NSLOT + slot[c]], t);
    }
}

// One bend of three sites (bend.c:186-330): forces on the outer sites f1, f3
// (the middle one takes -(f1 + f3)), the bond vectors for the virial, and
// the energy.
struct BendTerm {
    double dx12, dy12, dz12, dx23, dy23, dz23;
    double fx1, fy1, fz1, fx3, fy3, fz3;
    double v;
};

__device__ __forceinline__ void bend_eval(double x1, double y1, double z1, double x2, double y2, double z2, double x3,
                                          double y3, double z3, const double *c, const double *s, const double *dc,
                                          const double *ds, BendTerm &t)
{
    const double dx12 = x1 - x2, dy12 = y1 - y2, dz12 = z1 - z2;
    const double dx23 = x3 - x2, dy23 = y3 - y2, dz23 = z3 - z2;
    const double r122i = 1.0 / (dx12 * dx12 + dy12 * dy12 + dz12 * dz12);
    const double r12i = sqrt(r122i);
    const double r322i = 1.0 / (dx23 * dx23 + dy23 * dy23 + dz23 * dz23);
    const double r32i = sqrt(r322i);
    const double rpmag = r12i * r32i;
    double cost = (dx12 * dx23 + dy12 * dy23 + dz12 * dz23) * rpmag;
    cost = cost < 1.0 ? cost : 1.0;
    cost = cost > -1.0 ? cost : -1.0;
    double sint = sqrt(1.0 - cost * cost);
    sint = sint > 1.0e-8 ? sint : 1.0e-8;
    const double cos122 = cost * r122i, cos322 = cost * r322i;
    const double vc = ((((((c[6] * cost + c[5]) * cost + c[4]) * cost + c[3]) * cost + c[2]) * cost + c[1]) * cost +
                       c[0]);
    const double sisum = (((((s[6] * sint + s[5]) * sint + s[4]) * sint + s[3]) * sint + s[2]) * sint);
    t.v = vc + (sisum * cost + s[1] * sint);
    const double dvc = (((((dc[6] * cost + dc[5]) * cost + dc[4]) * cost + dc[3]) * cost + dc[2]) * cost + dc[1]);
    double dvs = ((((ds[6] * sint + ds[5]) * sint + ds[4]) * sint + ds[3]) * sint + ds[2]);
    dvs = dvs * cost + ds[1];
    const double pre = -(dvc + sisum - dvs * cost / sint);
    t.fx1 = (dx23 * rpmag - dx12 * cos122) * pre;
    t.fy1 = (dy23 * rpmag - dy12 * cos122) * pre;
    t.fz1 = (dz23 * rpmag - dz12 * cos122) * pre;
    t.fx3 = (dx12 * rpmag - dx23 * cos322) * pre;
    t.fy3 = (dy12 * rpmag - dy23 * cos322) * pre;
    t.fz3 = (dz12 * rpmag - dz23 * cos322) * pre;
    t.dx12 = dx12; t.dy12 = dy12; t.dz12 = dz12;
    t.dx23 = dx23; t.dy23 = dy23; t.dz23 = dz23;
}

// Excluded-pair correction of one pair at distance r (ecorr.c): energy and
// force factor from the interval coefficients, before the charge product.
__device__ __forceinline__ void ecor_eval(double r, int nsplin, double rmin, double dr, double dri,
                                          const double4 *__restrict__ tab, double &v, double &dv)
{
    int k = __double2int_rz(__dadd_rn(__dmul_rn(__dsub_rn(r, rmin), dri), 0.5)) + 3;
    k = k < nsplin - 2 ? k : nsplin - 2;
    k = k > 3 ? k : 3;
    const double rsp = __dadd_rn(__dmul_rn((double)(k - 3), dr), rmin);
    const double del = __dmul_rn(__dsub_rn(r, rsp), dri);
    v = spline_eval<double4, double>(tab[k - 1], del);
    dv = spline_eval<double4, double>(tab[nsplin + k - 1], del);
}

}  // namespace pinyb200
