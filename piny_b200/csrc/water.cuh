// Staging and finishing of one evaluation for boxes of identical water
// molecules: what comes before the pair and mesh kernels, and what comes
// after them, as one kernel each, a thread per (molecule, bead).
//
//   stage   positions into [site][xyz][bead], M sites placed, site forces
//           cleared, mode-1 positions kept (or the bead centroid), the
//           molecular extent bound, and every charge's PME record and bin
//   finish  bonds, bend and excluded-pair correction of the molecule, the
//           pair and mesh forces added, M-site forces distributed, forces
//           out in PINY's [bead][site][xyz] order, energies and virial
//
// Each replaces five or six small launches that passed the same arrays
// through memory between them.  Bound: launch latency for small boxes; for
// large ones the reads and writes of positions and forces.  Blocks cover
// blockDim / P molecules with all their beads, so both layouts are read and
// written in whole rows through a shared tile.
#pragma once

#include "boxtab.cuh"
#include "common.cuh"
#include "intra.cuh"
#include "pme_bin.cuh"

namespace pinyb200 {

struct StageArgs {
    int natm, nmol, P;
    const double *pos;     // [P][natm][3]
    double *posT, *forceT; // [natm][3][P]
    float *offT;           // [natm][3][P] FP32 offsets from the first site, or nullptr
    const double *xm_src;  // mode-1 positions [natm][3], or nullptr: the bead centroid (P > 1)
    double *xm_dst;        // kept copy (may be xm_src itself)
    unsigned long long *ext;
    const double *gcoef;   // [nmol][3] M-site coefficients (four sites)
    int bin;               // PME records wanted
};

// Site charges of the molecule: four sites, the first uncharged (q-TIP4P/F),
// or every site charged.
template <typename R, int NS, bool Q0>
__device__ __forceinline__ void water_stage_body(const StageArgs &a, const PmeArgs &pm, const TileArgs &tl,
                                                 const Cell &cell, const VBlk vb)
{
    extern __shared__ double wtile[];  // [P][W + 1]
    constexpr int NC = 3 * NS;
    const int P = a.P, MB = (int)blockDim.x / P, W = MB * NC;
    const int m0 = vb.x * MB, nm = min(MB, a.nmol - m0), cols = nm * NC;
    const size_t row = (size_t)a.natm * 3;
    for (int i = threadIdx.x; i < P * W; i += blockDim.x) {
        const int b = i / W, j = i - b * W;
        if (j < cols) wtile[b * (W + 1) + j] = a.pos[b * row + (size_t)m0 * NC + j];
    }
    __syncthreads();
    if (P > 1) {
        // mode-1 positions: the caller's, or the centroid of the beads as given
        for (int j = threadIdx.x; j < cols; j += blockDim.x) {
            double v;
            if (a.xm_src) {
                v = a.xm_src[(size_t)m0 * NC + j];
            } else {
                double s = 0.0;
                for (int b = 0; b < P; b++) s += wtile[b * (W + 1) + j];
                v = s / (double)P;
            }
            if (a.xm_dst != a.xm_src) a.xm_dst[(size_t)m0 * NC + j] = v;
        }
    }
    const int ml = threadIdx.x / P, b = threadIdx.x - ml * P, m = m0 + ml;
    double ext = 0.0;
    if (ml < nm) {
        double x[NC];
        const double *src = wtile + b * (W + 1) + ml * NC;
#pragma unroll
        for (int k = 0; k < NC; k++) x[k] = src[k];
        if (NS == 4) {
            const double c0 = a.gcoef[3 * m], c1 = a.gcoef[3 * m + 1], c2 = a.gcoef[3 * m + 2];
#pragma unroll
            for (int d = 0; d < 3; d++)
                x[(NS - 1) * 3 + d] = __dadd_rn(
                    __dadd_rn(__dadd_rn(0.0, __dmul_rn(c0, x[d])), __dmul_rn(c1, x[3 + d])), __dmul_rn(c2, x[6 + d]));
        }
        const size_t o = (size_t)m * NC * P + b;
#pragma unroll
        for (int k = 0; k < NC; k++) {
            a.posT[o + (size_t)k * P] = x[k];
            a.forceT[o + (size_t)k * P] = 0.0;
        }
        if (a.offT) {
#pragma unroll
            for (int k = 3; k < NC; k++) a.offT[o + (size_t)k * P] = (float)(x[k] - x[k % 3]);
        }
        if (P == 1) {
#pragma unroll
            for (int k = 3; k < NC; k++) ext = fmax(ext, fabs(x[k] - x[k % 3]));
        }
        if (a.bin) {
            // the counters' replies are waited for together
            constexpr int NQ = Q0 ? NS : NS - 1, S0 = Q0 ? 0 : 1;
            int bin[NQ], slot[NQ];
#pragma unroll
            for (int q = 0; q < NQ; q++) {
                const int s = S0 + q;
                bin[q] = pme_write_record<R>(pm, tl, cell, m * NS + s, m * NQ + q, b, x[3 * s], x[3 * s + 1],
                                             x[3 * s + 2]);
            }
#pragma unroll
            for (int q = 0; q < NQ; q++) slot[q] = atomicAdd(&tl.cnt[bin[q]], 1);
#pragma unroll
            for (int q = 0; q < NQ; q++) pme_put_record(pm, tl, bin[q], slot[q], (m * NQ + q) * P + b);
        }
    }
    if (P > 1) {
        __syncthreads();
        // the extent bound from the mode-1 positions (written above by this block, or the caller's)
        const double *xm = a.xm_src ? a.xm_src : a.xm_dst;
        for (int j = threadIdx.x; j < cols; j += blockDim.x) {
            const int mm = j / NC, k = j - mm * NC;
            const double *r = xm + (size_t)(m0 + mm) * NC;
            ext = fmax(ext, fabs(r[k] - r[k % 3]));
        }
    }
    // one atomic per block, and only where it raises the bound: thousands of
    // warps meeting at this address took most of the kernel's time
    __shared__ double bext[8];
#pragma unroll
    for (int o = 16; o >= 1; o >>= 1) ext = fmax(ext, __shfl_xor_sync(0xffffffffu, ext, o));
    if ((threadIdx.x & 31) == 0) bext[threadIdx.x >> 5] = ext;
    __syncthreads();
    if (threadIdx.x == 0) {
        for (int w = 1; w < (int)(blockDim.x >> 5); w++) ext = fmax(ext, bext[w]);
        const unsigned long long bits = (unsigned long long)__double_as_longlong(ext);
        if (ext > 0.0 && bits > __ldcg(a.ext)) atomicMax(a.ext, bits);
    }
}

struct FinishArgs {
    int natm, nmol, P;
    const double *posT, *forceT;
    const double *forceP;    // PME forces [nchrg][3][P], or nullptr
    double *forceT_out;      // complete site forces kept in [site][xyz][bead], or nullptr
    double *out;             // [P][natm][3]
    double *acc;
    int energy, distrib;
    const double *bond_eq, *bond_c, *bond_dc;                 // the molecule's bond type
    const double *bend_c, *bend_s, *bend_dc, *bend_ds;        // and bend type
    int ecor_nsplin;
    double ecor_rmin, ecor_dr, ecor_dri;
    const double4 *ecor_tab;
    double q[4];
    const double *gcoef;
};

template <int NS, bool Q0>
__device__ __forceinline__ void water_finish_body(const FinishArgs &a, const VBlk vb)
{
    extern __shared__ double wtile[];  // [P][W + 1]
    constexpr int NC = 3 * NS, NQ = Q0 ? NS : NS - 1, S0 = Q0 ? 0 : 1;
    const int P = a.P, MB = (int)blockDim.x / P, W = MB * NC;
    const int m0 = vb.x * MB, nm = min(MB, a.nmol - m0);
    const int ml = threadIdx.x / P, b = threadIdx.x - ml * P, m = m0 + ml;
    double v[9] = {0, 0, 0, 0, 0, 0, 0, 0, 0};  // vbond, vbend, vecor, pxx, pyy, pzz, pxy, pxz, pyz
    if (ml < nm) {
        const size_t o = (size_t)m * NC * P + b;
        double x[NC], f[NC];
#pragma unroll
        for (int k = 0; k < NC; k++) x[k] = a.posT[o + (size_t)k * P];
#pragma unroll
        for (int k = 0; k < NC; k++) f[k] = a.forceT[o + (size_t)k * P];
        auto pair = [&](int i, int j, double dx, double dy, double dz, double pre) {
            const double fx = dx * pre, fy = dy * pre, fz = dz * pre;
            f[3 * i] += fx;
            f[3 * i + 1] += fy;
            f[3 * i + 2] += fz;
            f[3 * j] -= fx;
            f[3 * j + 1] -= fy;
            f[3 * j + 2] -= fz;
            v[3] += dx * fx;
            v[4] += dy * fy;
            v[5] += dz * fz;
            v[6] += dx * fy;
            v[7] += dx * fz;
            v[8] += dy * fz;
        };
        // bonds O-H1, O-H2 (bond_both.c:29-420)
#pragma unroll
        for (int h = 1; h <= 2; h++) {
            const double dx = x[0] - x[3 * h], dy = x[1] - x[3 * h + 1], dz = x[2] - x[3 * h + 2];
            const double r = sqrt(dx * dx + dy * dy + dz * dz);
            const double rr0 = r - a.bond_eq[0];
            const double *c = a.bond_c, *d = a.bond_dc;
            v[0] += (((((c[6] * rr0 + c[5]) * rr0 + c[4]) * rr0 + c[3]) * rr0 + c[2]) * rr0 + c[1]) * rr0 + c[0];
            const double dv = ((((d[6] * rr0 + d[5]) * rr0 + d[4]) * rr0 + d[3]) * rr0 + d[2]) * rr0 + d[1];
            pair(0, h, dx, dy, dz, -dv / r);
        }
        // bend H1-O-H2
        {
            BendTerm g;
            bend_eval(x[3], x[4], x[5], x[0], x[1], x[2], x[6], x[7], x[8], a.bend_c, a.bend_s, a.bend_dc, a.bend_ds,
                      g);
            v[1] = g.v;
            f[3] += g.fx1;
            f[4] += g.fy1;
            f[5] += g.fz1;
            f[0] -= g.fx1 + g.fx3;
            f[1] -= g.fy1 + g.fy3;
            f[2] -= g.fz1 + g.fz3;
            f[6] += g.fx3;
            f[7] += g.fy3;
            f[8] += g.fz3;
            v[3] += g.dx12 * g.fx1 + g.dx23 * g.fx3;
            v[4] += g.dy12 * g.fy1 + g.dy23 * g.fy3;
            v[5] += g.dz12 * g.fz1 + g.dz23 * g.fz3;
            v[6] += g.dx12 * g.fy1 + g.dx23 * g.fy3;
            v[7] += g.dx12 * g.fz1 + g.dx23 * g.fz3;
            v[8] += g.dy12 * g.fz1 + g.dy23 * g.fz3;
        }
        // excluded charged pairs
        if (a.ecor_tab) {
#pragma unroll
            for (int i = S0 + 1; i < NS; i++)
#pragma unroll
                for (int j = S0; j < i; j++) {
                    const double dx = x[3 * i] - x[3 * j], dy = x[3 * i + 1] - x[3 * j + 1],
                                 dz = x[3 * i + 2] - x[3 * j + 2];
                    const double r =
                        __dsqrt_rn(__dadd_rn(__dadd_rn(__dmul_rn(dx, dx), __dmul_rn(dy, dy)), __dmul_rn(dz, dz)));
                    double ev, dv;
                    ecor_eval(r, a.ecor_nsplin, a.ecor_rmin, a.ecor_dr, a.ecor_dri, a.ecor_tab, ev, dv);
                    const double q12 = a.q[i] * a.q[j];
                    v[2] += ev * q12;
                    pair(i, j, dx, dy, dz, dv * q12);
                }
        }
        if (a.forceP) {
#pragma unroll
            for (int k = 0; k < 3 * NQ; k++) f[3 * S0 + k] += a.forceP[((size_t)m * 3 * NQ + k) * P + b];
        }
        if (NS == 4 && a.distrib) {
            const double c[3] = {a.gcoef[3 * m], a.gcoef[3 * m + 1], a.gcoef[3 * m + 2]};
#pragma unroll
            for (int d = 0; d < 3; d++) {
                const double fg = f[(NS - 1) * 3 + d];
#pragma unroll
                for (int s = 0; s < 3; s++) f[3 * s + d] += c[s] * fg;
                f[(NS - 1) * 3 + d] = 0.0;
            }
        }
        double *dst = wtile + b * (W + 1) + ml * NC;
#pragma unroll
        for (int k = 0; k < NC; k++) dst[k] = f[k];
        if (a.forceT_out) {
#pragma unroll
            for (int k = 0; k < NC; k++) a.forceT_out[o + (size_t)k * P] = f[k];
        }
    }
    __syncthreads();
    const size_t row = (size_t)a.natm * 3;
    const int cols = nm * NC;
    for (int i = threadIdx.x; i < P * W; i += blockDim.x) {
        const int bb = i / W, j = i - bb * W;
        if (j < cols) a.out[bb * row + (size_t)m0 * NC + j] = wtile[bb * (W + 1) + j];
    }
    if (a.energy) {
        const int slot[9] = {S_VBOND, S_VBEND, S_VECOR, S_PXX, S_PYY, S_PZZ, S_PXY, S_PXZ, S_PYZ};
        block_acc<9>(a.acc, P, slot, v);
    }
}

}  // namespace pinyb200
