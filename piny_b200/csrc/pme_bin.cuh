// PME records: stencil origins, the per-bead tile bins, and filing one charge.
#pragma once

#include "common.cuh"

namespace pinyb200 {

struct PmeArgs {
    int natm, P, nchrg;
    const int *ichrg;
    const double *charge;
    const double *posT;
    int Na, Nb, Nc, n;
    void *grid;  // real [P][Nc][Nb][Na]
    double *forceP;  // PME forces [nchrg][3][P]
    int4 *rhead;  // per (charge, bead) records, see RecGeom
    void *rw;
    unsigned long long *stamp;
};

// Scaled coordinate of one charge along one axis, wrapped to (0,1] and
// multiplied by the grid size; returns floor and fraction (FP64, PINY order).
__device__ __forceinline__ void scaled(double s, int N, int &i0, double &frac)
{
    s = __dsub_rn(s, nint_rn(__dsub_rn(s, 0.5)));
    double xs = __dmul_rn(s, (double)N);
    i0 = (int)xs;
    frac = __dsub_rn(xs, (double)i0);
    // s == 1 exactly (a coordinate on a cell face) and non-finite positions
    // would index outside the grid; keep every access in bounds.
    if (i0 == N) i0 = 0;
    if (!(i0 >= 0 && i0 < N)) { i0 = 0; frac = 0.0; }
}

// First grid index per axis of one charge's stencil and the fractional
// offsets.  PINY's points ia-(j-2), j = 1..n, are the n consecutive indices
// ia-n+1 .. ia (wrapped), and point j carries weight m[j]; so grid index
// lo + t (t = 0..n-1) carries m[n - t].  Evaluated once per charge and bead, when
// its record is written; the tile kernels read the record.
__device__ __forceinline__ void stencil_of(const PmeArgs &a, const Cell &cell, double x, double y, double z, int ni,
                                           int &la, int &lb, int &lc, double &fa, double &fb, double &fc)
{
    const double sa = __dadd_rn(__dadd_rn(__dmul_rn(x, cell.hi[0]), __dmul_rn(y, cell.hi[3])), __dmul_rn(z, cell.hi[6]));
    const double sb = __dadd_rn(__dadd_rn(__dmul_rn(x, cell.hi[1]), __dmul_rn(y, cell.hi[4])), __dmul_rn(z, cell.hi[7]));
    const double sc = __dadd_rn(__dadd_rn(__dmul_rn(x, cell.hi[2]), __dmul_rn(y, cell.hi[5])), __dmul_rn(z, cell.hi[8]));
    int ia, ib, ic;
    scaled(sa, a.Na, ia, fa);
    scaled(sb, a.Nb, ib, fb);
    scaled(sc, a.Nc, ic, fc);
    la = ia - ni + 1;
    if (la < 0) la += a.Na;
    lb = ib - ni + 1;
    if (lb < 0) lb += a.Nb;
    lc = ic - ni + 1;
    if (lc < 0) lc += a.Nc;
}

struct TileArgs {
    int T;  // tile edge (grid points)
    int nshare;  // blocks that share a bin's records (spread and gather)
    float qfix, qfix_inv;  // FP32 spread: fixed-point scale 2^S of the shared tile, and 2^-S
    int nta, ntb, ntc, ntile, cap;
    int *cnt;  // [P][ntile], then the overflow count
    int *bin;  // [P][ntile][cap] record numbers k*P + b
    int *ovf;  // [nchrg * P] record numbers that did not fit their bin
};

// One (charge k, bead b) record, number k P + b, at position (x, y, z):
// stencil origin in FP64 with PINY's operation order and the fractional
// offsets with the charge in R; returns the bin (bead and tile of its origin).
template <typename R>
__device__ __forceinline__ int pme_write_record(const PmeArgs &a, const TileArgs &t, const Cell &cell, int at, int k,
                                                int b, double x, double y, double z)
{
    const int idx = k * a.P + b;
    int la, lb, lc;
    double fa, fb, fc;
    stencil_of(a, cell, x, y, z, a.n, la, lb, lc, fa, fb, fc);
    typename Vec4<R>::T fr;
    fr.x = (R)fa;
    fr.y = (R)fb;
    fr.z = (R)fc;
    fr.w = (R)a.charge[at];
    ((typename Vec4<R>::T *)a.rw)[idx] = fr;
    a.rhead[idx] = make_int4(at, la, lb, lc);
    const int sh = t.T == 8 ? 3 : 4;  // tile edges are 8 or 16
    return b * t.ntile + ((lc >> sh) * t.ntb + (lb >> sh)) * t.nta + (la >> sh);
}

// Record idx into place `slot` of its bin, or the overflow list.
__device__ __forceinline__ void pme_put_record(const PmeArgs &a, const TileArgs &t, int bin, int slot, int idx)
{
    if (slot < t.cap) t.bin[(size_t)bin * t.cap + slot] = idx;
    else t.ovf[atomicAdd(&t.cnt[a.P * t.ntile], 1)] = idx;
}

template <typename R>
__device__ __forceinline__ void pme_file_record(const PmeArgs &a, const TileArgs &t, const Cell &cell, int at, int k,
                                                int b, double x, double y, double z)
{
    const int bin = pme_write_record<R>(a, t, cell, at, k, b, x, y, z);
    pme_put_record(a, t, bin, atomicAdd(&t.cnt[bin], 1), k * a.P + b);
}

// Kernel arguments of a context's mesh, and of its tile bins for spline order
// NI and tile edge TT.
PmeArgs pme_args_of(pinyb200_ctx *c);
TileArgs tile_args_of(pinyb200_ctx *c, int NI, int TT);

}  // namespace pinyb200
