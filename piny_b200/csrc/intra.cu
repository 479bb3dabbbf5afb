// Intramolecular terms, Ewald exclusion correction, ghost sites and the
// layout transposes, all in FP64 for every bead.
//
//   bonds   bond_both (src/energy/intra/bond_both.c:29-420): power series
//           V = sum c_n (r - r0)^n by Horner, F = -dV/dr d/r
//   bends   bend (src/energy/intra/bend.c:28-440): cos/sin series with the
//           sin clamp at 1e-8 and PINY's chain-rule forces
//   ecor    ecor (src/energy/intra/ecorr.c:28-274): q_i q_j S(cv0),
//           spline of -erf(alpha r)/r plus the finite-k correction
//   ghosts  get_ghost_pos / distrib_ghost_force
//           (src/energy/intra_con/ghost_control.c:28-129)
#include <algorithm>

#include <vector>

#include "boxtab.cuh"
#include "common.cuh"
#include "intra.cuh"

namespace pinyb200 {

// out[c][r] = in[r][c] for an rows x cols matrix of doubles, through a
// 32 x 32 shared tile (padded against bank conflicts): both the global reads
// and the global writes are 256-byte rows.  Positions in: in = [P][natm*3]
// (PINY's bead-major order), out = [natm*3][P]; forces out the reverse.
__device__ __forceinline__ void transpose_tiled_body(const double *__restrict__ in, double *__restrict__ out, int rows,
                                                     long long cols, const VBlk vb)
{
    __shared__ double tile[32][33];
    const long long c0 = (long long)vb.x * 32;
    const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;
    for (int r0 = vb.y * 32; r0 < rows; r0 += vb.gy * 32) {
#pragma unroll
        for (int k = 0; k < 32; k += 8) {
            const int r = r0 + ty + k;
            const long long c = c0 + tx;
            if (r < rows && c < cols) tile[ty + k][tx] = in[(size_t)r * cols + c];
        }
        __syncthreads();
#pragma unroll
        for (int k = 0; k < 32; k += 8) {
            const long long c = c0 + ty + k;
            const int r = r0 + tx;
            if (r < rows && c < cols) out[(size_t)c * rows + r] = tile[tx][ty + k];
        }
        __syncthreads();
    }
}

__global__ void __launch_bounds__(256) transpose_tiled_kernel(const double *__restrict__ in, double *__restrict__ out,
                                                              int rows, long long cols)
{
    transpose_tiled_body(in, out, rows, cols, hw_blk());
}

__device__ __forceinline__ void ghost_pos_body(double *__restrict__ posT, int P, int nghost, int ncomp,
                                 const int *__restrict__ gatom, const int *__restrict__ gcomp,
                                 const double *__restrict__ gcoef, const VBlk vb)
{
    const long long t = (long long)vb.x * blockDim.x + threadIdx.x;
    if (t >= (long long)nghost * P) return;
    const int b = (int)(t % P);
    const int g = (int)(t / P);
    const int gl = gatom[g];
#pragma unroll
    for (int d = 0; d < 3; d++) {
        double v = 0.0;
        for (int c = 0; c < ncomp; c++) {
            const int at = gcomp[g * ncomp + c];
            if (at < 0) continue;
            v = __dadd_rn(v, __dmul_rn(gcoef[g * ncomp + c], posT[(3 * (size_t)at + d) * P + b]));
        }
        posT[(3 * (size_t)gl + d) * P + b] = v;
    }
}

__global__ void ghost_pos_kernel(double *__restrict__ posT, int P, int nghost, int ncomp,
                                 const int *__restrict__ gatom, const int *__restrict__ gcomp,
                                 const double *__restrict__ gcoef)
{
    ghost_pos_body(posT, P, nghost, ncomp, gatom, gcomp, gcoef, hw_blk());
}

__device__ __forceinline__ void ghost_distrib_body(double *__restrict__ fT, int P, int nghost, int ncomp,
                                     const int *__restrict__ gatom, const int *__restrict__ gcomp,
                                     const double *__restrict__ gcoef, const VBlk vb)
{
    const long long t = (long long)vb.x * blockDim.x + threadIdx.x;
    if (t >= (long long)nghost * P) return;
    const int b = (int)(t % P);
    const int g = (int)(t / P);
    const int gl = gatom[g];
#pragma unroll
    for (int d = 0; d < 3; d++) {
        const double fg = fT[(3 * (size_t)gl + d) * P + b];
        for (int c = 0; c < ncomp; c++) {
            const int at = gcomp[g * ncomp + c];
            if (at < 0) continue;
            fT[(3 * (size_t)at + d) * P + b] += gcoef[g * ncomp + c] * fg;
        }
        fT[(3 * (size_t)gl + d) * P + b] = 0.0;
    }
}

__global__ void ghost_distrib_kernel(double *__restrict__ fT, int P, int nghost, int ncomp,
                                     const int *__restrict__ gatom, const int *__restrict__ gcomp,
                                     const double *__restrict__ gcoef)
{
    ghost_distrib_body(fT, P, nghost, ncomp, gatom, gcomp, gcoef, hw_blk());
}

struct IntraArgs {
    int natm, P;
    const double *posT;
    double *forceT;
    double *acc;
    const double *charge;
    int energy;
};

__device__ __forceinline__ void add_f(double *fT, int P, int at, int b, double fx, double fy, double fz)
{
    atomicAdd(&fT[(3 * (size_t)at + 0) * P + b], fx);
    atomicAdd(&fT[(3 * (size_t)at + 1) * P + b], fy);
    atomicAdd(&fT[(3 * (size_t)at + 2) * P + b], fz);
}

__device__ __forceinline__ void load_x(const double *posT, int P, int at, int b, double &x, double &y, double &z)
{
    x = posT[(3 * (size_t)at + 0) * P + b];
    y = posT[(3 * (size_t)at + 1) * P + b];
    z = posT[(3 * (size_t)at + 2) * P + b];
}

__device__ __forceinline__ void bond_body(const IntraArgs &a, int nbond, const int *__restrict__ bj,
                                                   const double *__restrict__ eq, const double *__restrict__ cc,
                                                   const double *__restrict__ dc, const VBlk vb)
{
    const long long t0 = (long long)vb.x * blockDim.x + threadIdx.x;
    const long long stride = (long long)vb.gx * blockDim.x;  // a multiple of P
    const int b = (int)(t0 % a.P);
    double v = 0, p[6] = {0, 0, 0, 0, 0, 0};
    for (long long t = t0; t < (long long)nbond * a.P; t += stride) {
        const int ib = (int)(t / a.P);
        const int j1 = bj[3 * ib], j2 = bj[3 * ib + 1], ty = bj[3 * ib + 2];
        double x1, y1, z1, x2, y2, z2;
        load_x(a.posT, a.P, j1, b, x1, y1, z1);
        load_x(a.posT, a.P, j2, b, x2, y2, z2);
        const double dx = x1 - x2, dy = y1 - y2, dz = z1 - z2;
        const double r = sqrt(dx * dx + dy * dy + dz * dz);
        const double rr0 = r - eq[ty];
        const double *c = cc + 7 * ty, *d = dc + 7 * ty;
        v += (((((c[6] * rr0 + c[5]) * rr0 + c[4]) * rr0 + c[3]) * rr0 + c[2]) * rr0 + c[1]) * rr0 + c[0];
        const double dv = ((((d[6] * rr0 + d[5]) * rr0 + d[4]) * rr0 + d[3]) * rr0 + d[2]) * rr0 + d[1];
        const double pre = -dv / r;
        const double fx = dx * pre, fy = dy * pre, fz = dz * pre;
        add_f(a.forceT, a.P, j1, b, fx, fy, fz);
        add_f(a.forceT, a.P, j2, b, -fx, -fy, -fz);
        p[0] += dx * fx; p[1] += dy * fy; p[2] += dz * fz; p[3] += dx * fy; p[4] += dx * fz; p[5] += dy * fz;
    }
    if (a.energy) {
        const int slot[7] = {S_VBOND, S_PXX, S_PYY, S_PZZ, S_PXY, S_PXZ, S_PYZ};
        const double vals[7] = {v, p[0], p[1], p[2], p[3], p[4], p[5]};
        block_acc<7>(a.acc, a.P, slot, vals);
    }
}

__global__ void __launch_bounds__(256) bond_kernel(const __grid_constant__ IntraArgs a, int nbond, const int *__restrict__ bj,
                                                   const double *__restrict__ eq, const double *__restrict__ cc,
                                                   const double *__restrict__ dc)
{
    bond_body(a, nbond, bj, eq, cc, dc, hw_blk());
}

// One bend of one bead from the position array.
__device__ __forceinline__ void bend_term(const double *posT, int P, int a1, int a2, int a3, int b,
                                          const double *c, const double *s, const double *dc, const double *ds,
                                          BendTerm &t)
{
    double x1, y1, z1, x2, y2, z2, x3, y3, z3;
    load_x(posT, P, a1, b, x1, y1, z1);
    load_x(posT, P, a2, b, x2, y2, z2);
    load_x(posT, P, a3, b, x3, y3, z3);
    bend_eval(x1, y1, z1, x2, y2, z2, x3, y3, z3, c, s, dc, ds, t);
}

__device__ __forceinline__ void bend_body(const IntraArgs &a, int nbend, const int *__restrict__ bj,
                                                   const double *__restrict__ bc, const double *__restrict__ bs,
                                                   const double *__restrict__ bdc, const double *__restrict__ bds, const VBlk vb)
{
    const long long t0 = (long long)vb.x * blockDim.x + threadIdx.x;
    const long long stride = (long long)vb.gx * blockDim.x;  // a multiple of P
    const int b = (int)(t0 % a.P);
    double v = 0, p[6] = {0, 0, 0, 0, 0, 0};
    for (long long t = t0; t < (long long)nbend * a.P; t += stride) {
        const int ib = (int)(t / a.P);
        const int a1 = bj[4 * ib], a2 = bj[4 * ib + 1], a3 = bj[4 * ib + 2], ty = bj[4 * ib + 3];
        BendTerm g;
        bend_term(a.posT, a.P, a1, a2, a3, b, bc + 7 * ty, bs + 7 * ty, bdc + 7 * ty, bds + 7 * ty, g);
        v += g.v;
        add_f(a.forceT, a.P, a1, b, g.fx1, g.fy1, g.fz1);
        add_f(a.forceT, a.P, a2, b, -(g.fx1 + g.fx3), -(g.fy1 + g.fy3), -(g.fz1 + g.fz3));
        add_f(a.forceT, a.P, a3, b, g.fx3, g.fy3, g.fz3);
        p[0] += g.dx12 * g.fx1 + g.dx23 * g.fx3;
        p[1] += g.dy12 * g.fy1 + g.dy23 * g.fy3;
        p[2] += g.dz12 * g.fz1 + g.dz23 * g.fz3;
        p[3] += g.dx12 * g.fy1 + g.dx23 * g.fy3;
        p[4] += g.dx12 * g.fz1 + g.dx23 * g.fz3;
        p[5] += g.dy12 * g.fz1 + g.dy23 * g.fz3;
    }
    if (a.energy) {
        const int slot[7] = {S_VBEND, S_PXX, S_PYY, S_PZZ, S_PXY, S_PXZ, S_PYZ};
        const double vals[7] = {v, p[0], p[1], p[2], p[3], p[4], p[5]};
        block_acc<7>(a.acc, a.P, slot, vals);
    }
}

__global__ void __launch_bounds__(256) bend_kernel(const __grid_constant__ IntraArgs a, int nbend, const int *__restrict__ bj,
                                                   const double *__restrict__ bc, const double *__restrict__ bs,
                                                   const double *__restrict__ bdc, const double *__restrict__ bds)
{
    bend_body(a, nbend, bj, bc, bs, bdc, bds, hw_blk());
}

__device__ __forceinline__ void ecor_body(const IntraArgs &a, int necor, const int *__restrict__ j1s,
                                                   const int *__restrict__ j2s, int nsplin, double rmin, double dr,
                                                   double dri, const double4 *__restrict__ tab, const VBlk vb)
{
    const long long t0 = (long long)vb.x * blockDim.x + threadIdx.x;
    const long long stride = (long long)vb.gx * blockDim.x;  // a multiple of P
    const int b = (int)(t0 % a.P);
    double v = 0, p[6] = {0, 0, 0, 0, 0, 0};
    for (long long t = t0; t < (long long)necor * a.P; t += stride) {
        const int ie = (int)(t / a.P);
        const int j1 = j1s[ie], j2 = j2s[ie];
        double x1, y1, z1, x2, y2, z2;
        load_x(a.posT, a.P, j1, b, x1, y1, z1);
        load_x(a.posT, a.P, j2, b, x2, y2, z2);
        const double dx = x1 - x2, dy = y1 - y2, dz = z1 - z2;
        const double r = __dsqrt_rn(__dadd_rn(__dadd_rn(__dmul_rn(dx, dx), __dmul_rn(dy, dy)), __dmul_rn(dz, dz)));
        double ev, edv;
        ecor_eval(r, nsplin, rmin, dr, dri, tab, ev, edv);
        const double q12 = a.charge[j1] * a.charge[j2];
        v += ev * q12;
        const double dvt = edv * q12;
        const double fx = dx * dvt, fy = dy * dvt, fz = dz * dvt;
        add_f(a.forceT, a.P, j1, b, fx, fy, fz);
        add_f(a.forceT, a.P, j2, b, -fx, -fy, -fz);
        p[0] += dx * fx; p[1] += dy * fy; p[2] += dz * fz; p[3] += dx * fy; p[4] += dx * fz; p[5] += dy * fz;
    }
    if (a.energy) {
        const int slot[7] = {S_VECOR, S_PXX, S_PYY, S_PZZ, S_PXY, S_PXZ, S_PYZ};
        const double vals[7] = {v, p[0], p[1], p[2], p[3], p[4], p[5]};
        block_acc<7>(a.acc, a.P, slot, vals);
    }
}

__global__ void __launch_bounds__(256) ecor_kernel(const __grid_constant__ IntraArgs a, int necor, const int *__restrict__ j1s,
                                                   const int *__restrict__ j2s, int nsplin, double rmin, double dr,
                                                   double dri, const double4 *__restrict__ tab)
{
    ecor_body(a, necor, j1s, j2s, nsplin, rmin, dr, dri, tab, hw_blk());
}

// ---- RESPA: weighted intramolecular forces, no energies -------------------
// Bonds at an inter level (bond_both.c:270-420): the full series at eq and
// the RESPA series at eq_res, combined as w_res F_res + w_both (F - F_res).
// At an intra-only level (bond.c:113-118, :270-278): one series, at eq_res
// when use_res, times w_res.
__global__ void __launch_bounds__(256) bond_w_kernel(int P, const double *__restrict__ posT, double *__restrict__ fW,
                                                     int nbond, const int *__restrict__ bj,
                                                     const double *__restrict__ eq, const double *__restrict__ eq_res,
                                                     const double *__restrict__ dc, int both, int use_res,
                                                     double w_res, double w_both)
{
    const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= (long long)nbond * P) return;
    const int ib = (int)(t / P), b = (int)(t % P);
    const int j1 = bj[3 * ib], j2 = bj[3 * ib + 1], ty = bj[3 * ib + 2];
    double x1, y1, z1, x2, y2, z2;
    load_x(posT, P, j1, b, x1, y1, z1);
    load_x(posT, P, j2, b, x2, y2, z2);
    const double dx = x1 - x2, dy = y1 - y2, dz = z1 - z2;
    const double r = sqrt(dx * dx + dy * dy + dz * dz);
    const double *d = dc + 7 * ty;
    double fx, fy, fz;
    if (both) {
        const double rr0 = r - eq[ty], rr0r = r - eq_res[ty];
        const double dv = ((((d[6] * rr0 + d[5]) * rr0 + d[4]) * rr0 + d[3]) * rr0 + d[2]) * rr0 + d[1];
        const double dvr = ((((d[6] * rr0r + d[5]) * rr0r + d[4]) * rr0r + d[3]) * rr0r + d[2]) * rr0r + d[1];
        const double pre = -dv / r, prer = -dvr / r;
        const double f1x = dx * pre, f1y = dy * pre, f1z = dz * pre;
        const double f2x = dx * prer, f2y = dy * prer, f2z = dz * prer;
        fx = w_res * f2x + w_both * (f1x - f2x);
        fy = w_res * f2y + w_both * (f1y - f2y);
        fz = w_res * f2z + w_both * (f1z - f2z);
    } else {
        const double rr0 = r - (use_res ? eq_res[ty] : eq[ty]);
        const double dv = ((((d[6] * rr0 + d[5]) * rr0 + d[4]) * rr0 + d[3]) * rr0 + d[2]) * rr0 + d[1];
        const double pre = -dv / r;
        fx = dx * pre * w_res;
        fy = dy * pre * w_res;
        fz = dz * pre * w_res;
    }
    add_f(fW, P, j1, b, fx, fy, fz);
    add_f(fW, P, j2, b, -fx, -fy, -fz);
}

// Bends x w (bend.c:144, :380-393).
__global__ void __launch_bounds__(256) bend_w_kernel(int P, const double *__restrict__ posT, double *__restrict__ fW,
                                                     int nbend, const int *__restrict__ bj,
                                                     const double *__restrict__ bc, const double *__restrict__ bs,
                                                     const double *__restrict__ bdc, const double *__restrict__ bds,
                                                     double w)
{
    const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= (long long)nbend * P) return;
    const int ib = (int)(t / P), b = (int)(t % P);
    const int a1 = bj[4 * ib], a2 = bj[4 * ib + 1], a3 = bj[4 * ib + 2], ty = bj[4 * ib + 3];
    BendTerm g;
    bend_term(posT, P, a1, a2, a3, b, bc + 7 * ty, bs + 7 * ty, bdc + 7 * ty, bds + 7 * ty, g);
    const double fx2 = -(g.fx1 + g.fx3), fy2 = -(g.fy1 + g.fy3), fz2 = -(g.fz1 + g.fz3);
    add_f(fW, P, a1, b, g.fx1 * w, g.fy1 * w, g.fz1 * w);
    add_f(fW, P, a2, b, fx2 * w, fy2 * w, fz2 * w);
    add_f(fW, P, a3, b, g.fx3 * w, g.fy3 * w, g.fz3 * w);
}

// Ewald exclusion correction (ecorr.c): table 0, the force table x w
// (:100, :229-245); 1, the RESPA table x w (:103-106); 2, ecor_both's
// w F + (w_res - w) F_res with w_res = wght_ter_res (:349-351, :497-505).
__global__ void __launch_bounds__(256) ecor_w_kernel(int P, const double *__restrict__ posT, double *__restrict__ fW,
                                                     const double *__restrict__ charge, int necor,
                                                     const int *__restrict__ j1s, const int *__restrict__ j2s,
                                                     int nsplin, double rmin, double dr, double dri,
                                                     const double4 *__restrict__ tab,
                                                     const double4 *__restrict__ tab_res, int table, double w,
                                                     double w_res)
{
    const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= (long long)necor * P) return;
    const int ie = (int)(t / P), b = (int)(t % P);
    const int j1 = j1s[ie], j2 = j2s[ie];
    double x1, y1, z1, x2, y2, z2;
    load_x(posT, P, j1, b, x1, y1, z1);
    load_x(posT, P, j2, b, x2, y2, z2);
    const double dx = x1 - x2, dy = y1 - y2, dz = z1 - z2;
    const double r = __dsqrt_rn(__dadd_rn(__dadd_rn(__dmul_rn(dx, dx), __dmul_rn(dy, dy)), __dmul_rn(dz, dz)));
    int k = __double2int_rz(__dadd_rn(__dmul_rn(__dsub_rn(r, rmin), dri), 0.5)) + 3;
    k = k < nsplin - 2 ? k : nsplin - 2;
    k = k > 3 ? k : 3;
    const double rsp = __dadd_rn(__dmul_rn((double)(k - 3), dr), rmin);
    const double del = __dmul_rn(__dsub_rn(r, rsp), dri);
    const double q12 = charge[j1] * charge[j2];
    double fx, fy, fz;
    if (table == 0 || table == 1) {
        const double dvt = spline_eval<double4, double>(table == 0 ? tab[nsplin + k - 1] : tab_res[k - 1], del) * q12;
        fx = dx * dvt * w;
        fy = dy * dvt * w;
        fz = dz * dvt * w;
    } else {
        const double dvt = spline_eval<double4, double>(tab[nsplin + k - 1], del) * q12;
        const double dvr = spline_eval<double4, double>(tab_res[k - 1], del) * q12;
        const double wd = w_res - w;
        fx = w * (dx * dvt) + wd * (dx * dvr);
        fy = w * (dy * dvt) + wd * (dy * dvr);
        fz = w * (dz * dvt) + wd * (dz * dvr);
    }
    add_f(fW, P, j1, b, fx, fy, fz);
    add_f(fW, P, j2, b, -fx, -fy, -fz);
}

static inline unsigned nblk(long long n, int t) { return (unsigned)((n + t - 1) / t); }

// grid-stride launch size for the intramolecular kernels
static inline unsigned nblk_gs(pinyb200_ctx *c, long long n)
{
    long long b = (n + 255) / 256, cap = (long long)c->sm_count * 4;
    return (unsigned)(b < cap ? (b > 0 ? b : 1) : cap);
}

cudaError_t launch_transpose_in(pinyb200_ctx *c, const double *d_aos)
{
    const long long M = (long long)c->sys.natm * 3;
    const dim3 grid((unsigned)((M + 31) / 32), (unsigned)((c->P + 31) / 32));
    transpose_tiled_kernel<<<grid, 256, 0, c->stream>>>(d_aos, c->d_posT, c->P, M);
    return cudaGetLastError();
}

cudaError_t launch_transpose_out(pinyb200_ctx *c, double *d_aos, const double *fT)
{
    const long long M = (long long)c->sys.natm * 3;
    const dim3 grid((unsigned)((c->P + 31) / 32), (unsigned)std::min<long long>((M + 31) / 32, 65535));
    transpose_tiled_kernel<<<grid, 256, 0, c->stream>>>(fT ? fT : c->d_forceT, d_aos, (int)M, c->P);
    return cudaGetLastError();
}

cudaError_t launch_ghost_pos(pinyb200_ctx *c)
{
    const DeviceSystem &s = c->sys;
    if (s.nghost == 0) return cudaSuccess;
    ghost_pos_kernel<<<nblk((long long)s.nghost * c->P, 256), 256, 0, c->stream>>>(
        c->d_posT, c->P, s.nghost, s.ghost_ncomp, s.ghost_atom, s.ghost_comp, s.ghost_coef);
    return cudaGetLastError();
}

cudaError_t launch_ghost_distrib(pinyb200_ctx *c, double *fT)
{
    const DeviceSystem &s = c->sys;
    if (s.nghost == 0) return cudaSuccess;
    ghost_distrib_kernel<<<nblk((long long)s.nghost * c->P, 256), 256, 0, c->stream>>>(
        fT ? fT : c->d_forceT, c->P, s.nghost, s.ghost_ncomp, s.ghost_atom, s.ghost_comp, s.ghost_coef);
    return cudaGetLastError();
}

cudaError_t launch_intra(pinyb200_ctx *c, const Cell &cell, bool energy)
{
    (void)cell;
    const DeviceSystem &s = c->sys;
    IntraArgs a;
    a.natm = s.natm;
    a.P = c->P;
    a.posT = c->d_posT;
    a.forceT = c->d_forceT;
    a.acc = c->d_acc;
    a.charge = s.charge;
    a.energy = energy ? 1 : 0;
    if (s.nbond)
        bond_kernel<<<nblk_gs(c, (long long)s.nbond * c->P), 256, 0, c->stream>>>(a, s.nbond, s.bond_j, s.bond_eq,
                                                                                  s.bond_c, s.bond_dc);
    if (s.nbend)
        bend_kernel<<<nblk_gs(c, (long long)s.nbend * c->P), 256, 0, c->stream>>>(a, s.nbend, s.bend_j, s.bend_c,
                                                                                  s.bend_s, s.bend_dc, s.bend_ds);
    if (s.necor)
        ecor_kernel<<<nblk_gs(c, (long long)s.necor * c->P), 256, 0, c->stream>>>(
            a, s.necor, s.ecor_j1, s.ecor_j2, s.ecor_nsplin, s.ecor_rmin, s.ecor_dr, s.ecor_dri, s.ecor_tab);
    return cudaGetLastError();
}

// Weighted bonds and bends of one RESPA level into target: bond_both's
// combination when both (inter levels), else bond() with PINY's ires_bond
// choice of equilibrium; bends x wght_tra_res.
cudaError_t launch_intra_respa(pinyb200_ctx *c, bool both, double *target)
{
    const DeviceSystem &s = c->sys;
    const double w_both = c->r_int_res_inter ? c->r_wter_res : c->r_wter;  // bond_both.c:156-161
    if (s.nbond)
        bond_w_kernel<<<nblk((long long)s.nbond * c->P, 256), 256, 0, c->stream>>>(
            c->P, c->d_posT, target, s.nbond, s.bond_j, s.bond_eq, c->d_bond_eq_res, s.bond_dc, both ? 1 : 0,
            c->r_ires_bond, c->r_wtra_res, w_both);
    if (s.nbend)
        bend_w_kernel<<<nblk((long long)s.nbend * c->P, 256), 256, 0, c->stream>>>(
            c->P, c->d_posT, target, s.nbend, s.bend_j, s.bend_c, s.bend_s, s.bend_dc, s.bend_ds, c->r_wtra_res);
    return cudaGetLastError();
}

cudaError_t launch_ecor_weighted(pinyb200_ctx *c, double w, double *target, int table)
{
    const DeviceSystem &s = c->sys;
    if (!s.necor) return cudaSuccess;
    ecor_w_kernel<<<nblk((long long)s.necor * c->P, 256), 256, 0, c->stream>>>(
        c->P, c->d_posT, target, s.charge, s.necor, s.ecor_j1, s.ecor_j2, s.ecor_nsplin, s.ecor_rmin, s.ecor_dr,
        s.ecor_dri, s.ecor_tab, (const double4 *)c->d_ecor_res_tab, table, w, c->r_wter_res);
    return cudaGetLastError();
}


// ---------------------------------------------------------------------------
// Many boxes per launch (the batched evaluation): ranges cleared and sums
// copied for every box in one persistent launch each.

struct ZeroBox {
    unsigned *p;
    long long n;  // 4-byte words
};

// 1024 words per block, 16-byte stores where the range allows
__device__ __forceinline__ void zero_body(unsigned *p, long long n, const VBlk vb)
{
    const long long w = ((long long)vb.x * blockDim.x + threadIdx.x) * 4;
    if (w >= n) return;
    if (w + 4 <= n && (((uintptr_t)(p + w)) & 15) == 0) {
        *(uint4 *)(p + w) = make_uint4(0u, 0u, 0u, 0u);
    } else {
        for (long long k = w; k < n && k < w + 4; k++) p[k] = 0u;
    }
}

__global__ void __launch_bounds__(256) zero_batch_kernel(const __grid_constant__ BoxTab<ZeroBox> t)
{
    PINYB200_BOX_LOOP(t, i, vb, (zero_body(t.arg[i].p, t.arg[i].n, vb)));
}

__global__ void __launch_bounds__(256) copy_batch_kernel(const __grid_constant__ BoxTab<CopySeg> t)
{
    PINYB200_BOX_LOOP(t, i, vb, {
        const CopySeg &c = t.arg[i];
        const long long k = (long long)vb.x * blockDim.x + threadIdx.x;
        if (k < c.n) c.dst[k] = c.src[k];
    });
}

cudaError_t launch_zero_batch(const std::vector<std::pair<void *, size_t>> &seg, int sm_count, cudaStream_t st)
{
    BoxTabBuilder<ZeroBox> tb;
    for (const auto &z : seg) {
        const long long n = (long long)(z.second / 4);
        tb.add(ZeroBox{(unsigned *)z.first, n}, (int)((n + 1023) / 1024), 1, (double)n);
    }
    return launch_tables(tb, (const void *)zero_batch_kernel, 256, 0, sm_count,
                         [&](const BoxTab<ZeroBox> &t, int g) { zero_batch_kernel<<<g, 256, 0, st>>>(t); });
}

cudaError_t launch_copy_batch(const std::vector<CopySeg> &seg, int sm_count, cudaStream_t st)
{
    BoxTabBuilder<CopySeg> tb;
    for (const CopySeg &c : seg) tb.add(c, (int)((c.n + 255) / 256), 1, (double)c.n);
    return launch_tables(tb, (const void *)copy_batch_kernel, 256, 0, sm_count,
                         [&](const BoxTab<CopySeg> &t, int g) { copy_batch_kernel<<<g, 256, 0, st>>>(t); });
}

}  // namespace pinyb200
