// Smooth PME for all beads: charge spreading, batched 3D FFT, k-sphere
// convolution with energy and virial, force gather.
//
// Restates ewald3d_recip_pme_none (src/energy/inter/recip3d/ewald3d_pme.c:
// 95-600): scaled coordinates wrapped to (0,1] (:231-256), order-n cardinal
// B-splines by PINY's recursion and their derivatives from the order n-1
// splines (:301-338, :512-532), grid points ia - (j-2) wrapped (:274-300),
// the half-space spherical k list with preg = exp(-g^2/4a^2)/(g^2 V/4pi) and
// the B-spline weights (:366-425), and the gather F = -q sum grad(M) phi
// (:534-559).  PINY spreads into a complex grid with zero imaginary part and
// runs unnormalised complex FFTs (para_fft_gen3d_bck_to_g / _fwd_to_r).
// The device spreads into a real grid and keeps half of the spectrum
// (a <= Na/2): the charge grid is real, so the other half is its complex
// conjugate.  Filtering with the symmetric influence function equals PINY's
// half-list convolution plus Hermitian fill (pme_sngl_pack_coef,
// fft_package.c:458-503); half of the full-grid sum is PINY's energy.
//
// Kernels per evaluation (all beads in each launch):
//   bin         (charge, bead) -> grid tile of its stencil origin (water boxes
//               do this in their staging kernel)
//   spread      per (tile, bead): shared-memory copy of the tile, added to
//               the real grid once (FP32: 16-byte vector atomics)
//   plane_fwd   per (bead, c) plane: FFT along a then b in shared memory,
//               half spectrum out (cubic meshes of PINY's lengths: the
//               compile-time transforms of fft.cuh, others the ones here)
//   conv_c      per (bead, b): FFT along c, filter + energy + virial,
//               inverse FFT along c
//   plane_inv   per (bead, c): inverse FFT along b, Hermitian completion,
//               inverse FFT along a, real potential out
//   gather      per (tile, bead): forces from a shared copy of the tile's
//               potential
#include <algorithm>
#include <map>
#include <tuple>
#include <vector>

#include "boxtab.cuh"
#include "common.cuh"
#include "fft.cuh"
#include "pme_bin.cuh"

namespace pinyb200 {

// Largest value of the order-n cardinal B-spline (PINY's m[] over the
// fractional offset, ewald3d_pme.c:301-338), sampled finely: a bound for the
// fixed-point spread.
static double bspline_peak_of(int n)
{
    double best = 0.0;
    for (int k = 0; k <= 1024; k++) {
        const double f = k / 1024.0;
        double m[16] = {0}, u[16];
        for (int j = 1; j <= n; j++) u[j] = f + (double)(j - 1);
        m[1] = 1.0 - std::fabs(u[1] - 1.0);
        m[2] = 1.0 - std::fabs(u[2] - 1.0);
        for (int nn = 3; nn <= n; nn++) {
            const double rn1 = 1.0 / (double)(nn - 1);
            for (int j = nn; j >= 2; j--) m[j] = (u[j] * m[j] + ((double)nn - u[j]) * m[j - 1]) * rn1;
            m[1] = u[1] * m[1] * rn1;
        }
        for (int j = 1; j <= n; j++) best = std::max(best, m[j]);
    }
    return best * (1.0 + 1e-6);
}
static double bspline_peak(int n)
{
    // once per order: 1025 samples of the recursion are 50 us of host time
    static const std::vector<double> peak = [] {
        std::vector<double> p(13, 0.0);
        for (int k = 3; k <= 12; k++) p[k] = bspline_peak_of(k);
        return p;
    }();
    return peak[std::min(12, std::max(3, n))];
}

// Stencil points per axis, padded.
template <int NI>
struct RecGeom {
    static constexpr int NIP = NI <= 4 ? 4 : (NI <= 8 ? 8 : 12);
};

// Tile geometry: T^3 grid points own the charges whose stencil starts in
// them; the shared copy spans E = T + NI - 1 points per edge (the stencils
// reach NI - 1 beyond), rows padded to PA.
// With PA = 24 (E <= 24) the 4 b rows x 8 a points of a warp fall in 32
// distinct banks (row offsets 0, 24, 48, 72 = 0, 24, 16, 8 mod 32).
template <int NI, int TT>
struct TileGeom {
    static constexpr int T = TT;
    static constexpr int E = T + NI - 1;
    static constexpr int PA = E <= 24 ? 24 : ((E + 3) & ~3);
    static constexpr int NPT = E * E * PA;
};

// i mod N for 0 <= i < k N with small k.
__device__ __forceinline__ int wrapi(int i, int N)
{
    while (i >= N) i -= N;
    return i;
}

// The E^3 points of the tile with corner (ta0, tb0, tc0) of grid g into the
// block's shared copy: asynchronous 16-byte copies where the rows allow (all
// in flight at once; the padding columns take what the grid holds there),
// else plain loads.  The caller's barrier follows.
template <typename R, typename TG>
__device__ __forceinline__ void load_tile(R *tl, const R *g, int Na, int Nb, int Nc, int ta0, int tb0, int tc0)
{
    constexpr int NROW = TG::E * TG::E, V = 16 / sizeof(R), NQ = TG::PA / V;
    if ((Na & (V - 1)) == 0) {
        for (int i = threadIdx.x; i < NROW * NQ; i += blockDim.x) {
            const int row = i / NQ, q = i - row * NQ;
            const int cz = row / TG::E, by = row - cz * TG::E;
            cp_async16(tl + row * TG::PA + V * q,
                       g + ((size_t)wrapi(tc0 + cz, Nc) * Nb + wrapi(tb0 + by, Nb)) * Na + wrapi(ta0 + V * q, Na));
        }
        cp_async_wait();
    } else {
        for (int i = threadIdx.x; i < NROW * TG::PA; i += blockDim.x) {
            const int row = i / TG::PA, ax = i - row * TG::PA;
            const int cz = row / TG::E, by = row - cz * TG::E;
            tl[i] = ax < TG::E ? g[((size_t)wrapi(tc0 + cz, Nc) * Nb + wrapi(tb0 + by, Nb)) * Na + wrapi(ta0 + ax, Na)]
                               : (R)0;
        }
    }
}

// Weights of one record that a lane of an 8-lane group needs: its own a
// points (l8 and l8 + 8) and all b and c points; DERIV adds the derivatives.
template <typename R, int NI, bool DERIV>
struct LaneW {
    typedef RecGeom<NI> RG;
    R wa0, wa1, da0, da1;
    R mb[RG::NIP], mc[RG::NIP], db[DERIV ? RG::NIP : 1], dc[DERIV ? RG::NIP : 1];
};

// Shared copy of a tile.
template <typename R, int NI, int TT>
size_t spread_smem()
{
    return (size_t)TileGeom<NI, TT>::NPT * sizeof(R);
}

// Gather sums of one record for lane l8: d/ds_a, d/ds_b, d/ds_c of
// sum M_a M_b M_c phi over the lane's a points; phi(tc, tb, ta) reads the
// potential at stencil point (tc, tb, ta).  The a weights factor out of the
// b and c sums, so a stencil point costs one load and two FMAs.
template <typename R, int NI, typename PHI>
__device__ __forceinline__ void gather_lane(PHI phi, const LaneW<R, NI, true> &lw, int l8, double &ea, double &eb,
                                            double &ec)
{
    ea = eb = ec = 0.0;
    if (l8 >= NI) return;
    R xa = 0, xb = 0, xc = 0;
#pragma unroll
    for (int j = 0; j < (NI > 8 ? 2 : 1); j++) {
        if (j == 1 && l8 + 8 >= NI) break;
        const int ta = l8 + 8 * j;
        R sa = 0, sb = 0, sc = 0;
#pragma unroll
        for (int tc = 0; tc < NI; tc++) {
            R um = 0, ud = 0;
#pragma unroll
            for (int tb = 0; tb < NI; tb++) {
                const R p = phi(tc, tb, ta);
                um += lw.mb[tb] * p;
                ud += lw.db[tb] * p;
            }
            sa += lw.mc[tc] * um;
            sb += lw.mc[tc] * ud;
            sc += lw.dc[tc] * um;
        }
        const R wa = j ? lw.wa1 : lw.wa0, da = j ? lw.da1 : lw.da0;
        xa += da * sa;
        xb += wa * sb;
        xc += wa * sc;
    }
    ea = (double)xa;
    eb = (double)xb;
    ec = (double)xc;
}

// Force of one record from its three sums (summed over the 8-lane group;
// lane 0 writes): F = -q h^-T (N_a e_a, N_b e_b, N_c e_c), stored (not
// added) at the record's slot idx = k * P + b of the PME force buffer
// [nchrg][3][P]; every record is written exactly once per evaluation.
__device__ __forceinline__ void gather_store(const PmeArgs &a, const Cell &cell, int at, int idx, double ea,
                                             double eb, double ec, int l8)
{
#pragma unroll
    for (int o = 4; o >= 1; o >>= 1) {
        ea += __shfl_xor_sync(0xffffffffu, ea, o);
        eb += __shfl_xor_sync(0xffffffffu, eb, o);
        ec += __shfl_xor_sync(0xffffffffu, ec, o);
    }
    if (l8 != 0) return;
    ea *= (double)a.Na;
    eb *= (double)a.Nb;
    ec *= (double)a.Nc;
    const double q = a.charge[at];
    const double gx = ea * cell.hi[0] + eb * cell.hi[1] + ec * cell.hi[2];
    const double gy = ea * cell.hi[3] + eb * cell.hi[4] + ec * cell.hi[5];
    const double gz = ea * cell.hi[6] + eb * cell.hi[7] + ec * cell.hi[8];
    const int k = idx / a.P, b = idx - k * a.P;
    double *f = a.forceP;
    f[(3 * (size_t)k + 0) * a.P + b] = -gx * q;
    f[(3 * (size_t)k + 1) * a.P + b] = -gy * q;
    f[(3 * (size_t)k + 2) * a.P + b] = -gz * q;
}

// Adds the PME forces [nchrg][3][P] to the site forces [natm][3][P].
__device__ __forceinline__ void pme_force_add_body(int nchrg, int P, const int *__restrict__ ichrg,
                                                   const double *__restrict__ fP, double *__restrict__ fT, const VBlk vb)
{
    const long long t = (long long)vb.x * blockDim.x + threadIdx.x;
    if (t >= (long long)nchrg * 3 * P) return;
    const long long kd = t / P;
    const int b = (int)(t - kd * P);
    const int k = (int)(kd / 3), d = (int)(kd - 3LL * k);
    fT[(3 * (size_t)ichrg[k] + d) * P + b] += fP[t];
}

__global__ void __launch_bounds__(256) pme_force_add_kernel(int nchrg, int P, const int *__restrict__ ichrg,
                                                            const double *__restrict__ fP, double *__restrict__ fT)
{
    pme_force_add_body(nchrg, P, ichrg, fP, fT, hw_blk());
}

// RESPA outer level: PME forces x wght_ter into another buffer
// (ewald3d_pme.c: forces x wght_now before they are added).
__global__ void __launch_bounds__(256) pme_force_add_scaled_kernel(int nchrg, int P, const int *__restrict__ ichrg,
                                                                   const double *__restrict__ fP, double w,
                                                                   double *__restrict__ fT)
{
    const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= (long long)nchrg * 3 * P) return;
    const long long kd = t / P;
    const int b = (int)(t - kd * P);
    const int k = (int)(kd / 3), d = (int)(kd - 3LL * k);
    fT[(3 * (size_t)ichrg[k] + d) * P + b] += fP[t] * w;
}

// ---------------------------------------------------------------------------
// B-spline weights as polynomials of the fractional offset.  PINY's
// recursion (ewald3d_pme.c:301-338) makes the weight m[j] of order NI (at
// u = f + j - 1) a polynomial of degree NI - 1 in f on [0, 1), and the
// derivative weight dm[j] = m'[j] - m'[j - 1] formed from the order NI - 1
// splines (:512-532) one of degree NI - 2.  BsplinePoly runs that recursion
// on coefficient arrays at compile time; the kernels evaluate each lane's
// weights by Horner.  The bin kernel writes, per (charge, bead), the stencil
// origin and the three fractional offsets with the charge (32 bytes in
// FP32), and spread and gather read the next record while they work on the
// current one.
template <int NI>
struct BsplinePoly {
    double m[NI][NI];   // m[p][d]: coefficient of f^d of PINY's m[p + 1]
    double dm[NI][NI];  // dm[p][d]: of PINY's dm[p + 1]
    constexpr BsplinePoly() : m(), dm()
    {
        double cur[NI + 1][NI + 1] = {};
        cur[1][1] = 1.0;   // m[1] = 1 - |u_1 - 1| = f
        cur[2][0] = 1.0;   // m[2] = 1 - |u_2 - 1| = 1 - f
        cur[2][1] = -1.0;
        for (int nn = 3; nn <= NI; nn++) {
            const double rn1 = 1.0 / (double)(nn - 1);
            // m[j] = (u_j m[j] + (nn - u_j) m[j - 1]) / (nn - 1), u_j = f + j - 1
            for (int j = nn; j >= 2; j--) {
                double nw[NI + 1] = {};
                for (int d = 0; d < NI; d++) {
                    nw[d] += (double)(j - 1) * cur[j][d] + (double)(nn - j + 1) * cur[j - 1][d];
                    nw[d + 1] += cur[j][d] - cur[j - 1][d];
                }
                for (int d = 0; d <= NI; d++) cur[j][d] = nw[d] * rn1;
            }
            double nw1[NI + 1] = {};
            for (int d = 0; d < NI; d++) nw1[d + 1] = cur[1][d];
            for (int d = 0; d <= NI; d++) cur[1][d] = nw1[d] * rn1;
            if (nn == NI - 1)
                for (int j = 1; j <= NI; j++)
                    for (int d = 0; d < NI; d++) dm[j - 1][d] = cur[j][d] - (j >= 2 ? cur[j - 1][d] : 0.0);
        }
        for (int j = 1; j <= NI; j++)
            for (int d = 0; d < NI; d++) m[j - 1][d] = cur[j][d];
    }
};

template <int NI>
__constant__ BsplinePoly<NI> kBspline = BsplinePoly<NI>();

// Shared copy of the polynomials in R, rows padded to a multiple of 4.
template <typename R, int NI>
struct PolyTab {
    static constexpr int NP4 = (NI + 3) & ~3;
    R m[NI][NP4], dm[NI][NP4];
    __device__ __forceinline__ void fill(bool deriv)
    {
        for (int i = threadIdx.x; i < NI * NP4; i += blockDim.x) {
            const int p = i / NP4, d = i - p * NP4;
            m[p][d] = d < NI ? (R)kBspline<NI>.m[p][d] : (R)0;
            if (deriv) dm[p][d] = d < NI ? (R)kBspline<NI>.dm[p][d] : (R)0;
        }
    }
};

// Weight of stencil point t (grid index lo + t carries PINY's m[NI - t],
// piece NI - 1 - t) from its coefficient row, by Horner.
template <typename R, int NI>
__device__ __forceinline__ R poly_eval(const R (&row)[PolyTab<R, NI>::NP4], R f)
{
    constexpr int NP4 = PolyTab<R, NI>::NP4;
    R c[NP4];
    if constexpr (sizeof(R) == 4) {
#pragma unroll
        for (int i = 0; i < NP4; i += 4) {
            const float4 v = *(const float4 *)&row[i];
            c[i] = v.x;
            c[i + 1] = v.y;
            c[i + 2] = v.z;
            c[i + 3] = v.w;
        }
    } else {
#pragma unroll
        for (int i = 0; i < NP4; i += 2) {
            const double2 v = *(const double2 *)&row[i];
            c[i] = v.x;
            c[i + 1] = v.y;
        }
    }
    R w = c[NI - 1];
#pragma unroll
    for (int d = NI - 2; d >= 0; d--) w = w * f + c[d];
    return w;
}

// The piece of one stencil point (t of a lane of an 8-lane group, order up to
// 8) in registers: its weight at f, and the weight's derivative (which is
// dm: the difference of the order n - 1 splines is the derivative of the
// order n one) from the same Horner pass.
template <typename R, int NI>
struct Piece {
    R c[NI];
    __device__ __forceinline__ void load(int t)
    {
        const int p = NI - 1 - (t < NI ? t : NI - 1);
#pragma unroll
        for (int d = 0; d < NI; d++) c[d] = t < NI ? (R)kBspline<NI>.m[p][d] : (R)0;
    }
    __device__ __forceinline__ R value(R f) const
    {
        R w = c[NI - 1];
#pragma unroll
        for (int d = NI - 2; d >= 0; d--) w = w * f + c[d];
        return w;
    }
    // second derivative
    __device__ __forceinline__ R second(R f) const
    {
        R w = c[NI - 1], dw = (R)0, d2 = (R)0;
#pragma unroll
        for (int d = NI - 2; d >= 0; d--) {
            d2 = d2 * f + dw;
            dw = dw * f + w;
            w = w * f + c[d];
        }
        return (R)2 * d2;
    }
    __device__ __forceinline__ void both(R f, R &w, R &dw) const
    {
        w = c[NI - 1];
        dw = (R)0;
#pragma unroll
        for (int d = NI - 2; d >= 0; d--) {
            dw = dw * f + w;
            w = w * f + c[d];
        }
    }
};

template <typename R>
__device__ __forceinline__ typename Vec4<R>::T load_frac(const void *rw, int idx)
{
    if constexpr (sizeof(R) == 4) return __ldg((const float4 *)rw + idx);
    else return ldg4((const double4 *)rw + idx);
}

// Bin kernel of the compact path: one thread per (charge, bead), stencil
// origin in FP64 with PINY's operation order, record
// (atom, la, lb, lc) + (fa, fb, fc, q), record number filed under its tile.
template <typename R>
__device__ __forceinline__ void pme_bin_compact_body(const PmeArgs &a, const Cell &cell, const TileArgs &t,
                                                     const VBlk vb)
{
    const long long idx = (long long)vb.x * blockDim.x + threadIdx.x;
    if (idx >= (long long)a.nchrg * a.P) return;
    const int b = (int)(idx % a.P);
    const int k = (int)(idx / a.P);
    const int at = a.ichrg[k];
    pme_file_record<R>(a, t, cell, at, k, b, a.posT[(3 * (size_t)at + 0) * a.P + b],
                       a.posT[(3 * (size_t)at + 1) * a.P + b], a.posT[(3 * (size_t)at + 2) * a.P + b]);
}

template <typename R>
__global__ void __launch_bounds__(256) pme_bin_compact_kernel(const __grid_constant__ PmeArgs a,
                                                              const __grid_constant__ Cell cell,
                                                              const __grid_constant__ TileArgs t)
{
    pme_bin_compact_body<R>(a, cell, t, hw_blk());
}

// Weights one spread lane needs (lanes = 8 a points x 4 b rows): its a
// points la8 (+8), its b rows lb4 + 4 i, and all c points.  Up to order 8 a
// lane evaluates the three axes at point la8 from its piece in registers and
// the b and c weights are shuffled from lanes 0..7 (weights from a shared
// table took 12 of the 60 shared-memory wavefronts of a record); order 10
// evaluates from the table.  Every lane of the warp calls it.
template <typename R, int NI>
struct SpreadPoly {
    PolyTab<R, NI> *pt;
    Piece<R, NI <= 8 ? NI : 4> piece;
    __device__ __forceinline__ void init(PolyTab<R, NI> *tab, int lane)
    {
        pt = tab;
        if constexpr (NI <= 8) piece.load(lane & 7);
    }
};
template <typename R, int NI>
struct SpreadW {
    static constexpr int NTB = (NI + 3) / 4, NSA = (NI + 7) / 8;
    R wa[NSA], mb[NTB], mc[NI];
    __device__ __forceinline__ void eval(const SpreadPoly<R, NI> &sp, const typename Vec4<R>::T &fr, int lane)
    {
        const int la8 = lane & 7, lb4 = lane >> 3;
        if constexpr (NI <= 8) {
            wa[0] = sp.piece.value(fr.x);
            const R wb = sp.piece.value(fr.y), wc = sp.piece.value(fr.z);
#pragma unroll
            for (int i = 0; i < NTB; i++) mb[i] = __shfl_sync(0xffffffffu, wb, (lb4 + 4 * i) & 7);
#pragma unroll
            for (int tc = 0; tc < NI; tc++) mc[tc] = __shfl_sync(0xffffffffu, wc, tc);
        } else {
            const PolyTab<R, NI> &pt = *sp.pt;
#pragma unroll
            for (int s = 0; s < NSA; s++)
                wa[s] = la8 + 8 * s < NI ? poly_eval<R, NI>(pt.m[NI - 1 - (la8 + 8 * s)], fr.x) : (R)0;
#pragma unroll
            for (int i = 0; i < NTB; i++)
                mb[i] = lb4 + 4 * i < NI ? poly_eval<R, NI>(pt.m[NI - 1 - (lb4 + 4 * i)], fr.y) : (R)0;
            const R mcl = lane < NI ? poly_eval<R, NI>(pt.m[NI - 1 - lane], fr.z) : (R)0;
#pragma unroll
            for (int tc = 0; tc < NI; tc++) mc[tc] = __shfl_sync(0xffffffffu, mcl, tc);
        }
    }
};

// One record spread straight into the grid g of its bead (origin outside
// the block's tile, or an overflow record); a warp, lanes as SpreadW.
template <typename R, int NI>
__device__ __forceinline__ void spread_warp_global(const PmeArgs &a, R *g, int la, int lb, int lc,
                                                   const SpreadW<R, NI> &w, R q, int lane)
{
    const int la8 = lane & 7, lb4 = lane >> 3;
#pragma unroll
    for (int s = 0; s < SpreadW<R, NI>::NSA; s++) {
        if (la8 + 8 * s >= NI) break;
        const int ga = wrapi(la + la8 + 8 * s, a.Na);
        const R qa = q * w.wa[s];
#pragma unroll
        for (int tc = 0; tc < NI; tc++) {
            const int gc = wrapi(lc + tc, a.Nc);
            const R cq = qa * w.mc[tc];
#pragma unroll
            for (int i = 0; i < SpreadW<R, NI>::NTB; i++)
                if (lb4 + 4 * i < NI) atomicAdd(g + ((size_t)gc * a.Nb + wrapi(lb + lb4 + 4 * i, a.Nb)) * a.Na + ga, cq * w.mb[i]);
        }
    }
}

// Spread, FP32 and the boxes of a batch (one block per (tile,
// bead), one warp per record into a shared copy of the tile, the copy added
// to the grid once), with the weights evaluated in the block and the next
// record read ahead.
template <int NI, int TT>
__device__ __forceinline__ void spread_tile_c_body(const PmeArgs &a, const TileArgs &t, const VBlk vb)
{
    typedef float R;
    typedef TileGeom<NI, TT> TG;
    typedef typename Vec4<R>::T R4;
    constexpr int NTB = SpreadW<R, NI>::NTB;
    extern __shared__ unsigned char smem_raw[];
    R *tl = (R *)smem_raw;
    __shared__ __align__(16) PolyTab<R, NI> pt;
    for (int i = threadIdx.x; i < TG::NPT; i += blockDim.x) tl[i] = (R)0;
    if (NI > 8) pt.fill(false);
    SpreadPoly<R, NI> sp;
    sp.init(&pt, threadIdx.x & 31);
    __syncthreads();
    const int tile = vb.x, b = vb.y / t.nshare, z = vb.y - b * t.nshare;
    const int ta0 = (tile % t.nta) * TG::T, tb0 = ((tile / t.nta) % t.ntb) * TG::T, tc0 = (tile / (t.nta * t.ntb)) * TG::T;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarp = blockDim.x >> 5;
    const int la8 = lane & 7, lb4 = lane >> 3;
    const int n = min(t.cnt[b * t.ntile + tile], t.cap);
    const int *list = t.bin + ((size_t)b * t.ntile + tile) * t.cap;
    R *g = (R *)a.grid + (size_t)b * a.Na * a.Nb * a.Nc;
    int4 hn = make_int4(0, 0, 0, 0);
    R4 fn = {};
    const int e0 = z * nwarp + warp, estep = nwarp * t.nshare;
    if (e0 < n) {
        const int idx = list[e0];
        hn = a.rhead[idx];
        fn = load_frac<R>(a.rw, idx);
    }
    for (int e = e0; e < n; e += estep) {
        const int4 h = hn;
        const R4 fr = fn;
        if (e + estep < n) {
            const int idx = list[e + estep];
            hn = a.rhead[idx];
            fn = load_frac<R>(a.rw, idx);
        }
        SpreadW<R, NI> w;
        w.eval(sp, fr, lane);
        const R q = fr.w;
        const int oa = h.y - ta0, ob = h.z - tb0, oc = h.w - tc0;
        if (oa >= 0 && oa < TG::T && ob >= 0 && ob < TG::T && oc >= 0 && oc < TG::T) {
            const int off0 = (oc * TG::E + ob + lb4) * TG::PA + oa + la8;
#pragma unroll
            for (int s = 0; s < SpreadW<R, NI>::NSA; s++) {
                if (la8 + 8 * s >= NI) break;
                const R qa = q * w.wa[s];
#pragma unroll
                for (int tc = 0; tc < NI; tc++) {
                    const R cq = qa * w.mc[tc];
#pragma unroll
                    for (int i = 0; i < NTB; i++) {
                        if (lb4 + 4 * i >= NI) continue;
                        const int o = off0 + (tc * TG::E + 4 * i) * TG::PA + 8 * s;
                        // fixed point: v 2^S + 1.5 2^23 is exact to the nearest
                        // integer for |v 2^S| < 2^22, whose bits less those of
                        // 1.5 2^23 are that integer; integer shared atomics run
                        // at five times the rate of FP32 ones
                        const float y = fmaf(cq * w.mb[i], t.qfix, 12582912.0f);
                        atomicAdd((int *)tl + o, __float_as_int(y) - 0x4B400000);
                    }
                }
            }
        } else {
            spread_warp_global<R, NI>(a, g, h.y, h.z, h.w, w, q, lane);
        }
    }
    // overflow records: one warp each, straight into the grid
    const int nov = t.cnt[a.P * t.ntile];
    const int gid = vb.y * vb.gx + vb.x, nblk = vb.gx * vb.gy;
    for (int e = gid * nwarp + warp; e < nov; e += nblk * nwarp) {
        const int idx = t.ovf[e];
        const int4 h = a.rhead[idx];
        const R4 fr = load_frac<R>(a.rw, idx);
        SpreadW<R, NI> w;
        w.eval(sp, fr, lane);
        R *g2 = (R *)a.grid + (size_t)(idx % a.P) * a.Na * a.Nb * a.Nc;
        spread_warp_global<R, NI>(a, g2, h.y, h.z, h.w, w, fr.w, lane);
    }
    __syncthreads();
    constexpr int NROW = TG::E * TG::E;
    if ((a.Na & 3) == 0) {
        constexpr int NQ = TG::PA / 4;
        constexpr int RPI = 32 / NQ;
        for (int r0 = warp * RPI; r0 < NROW; r0 += nwarp * RPI) {
            const int row = r0 + lane / NQ, q4 = lane % NQ;
            if (lane >= RPI * NQ || row >= NROW) continue;
            const int4 iv = ((const int4 *)tl)[row * NQ + q4];
            if ((iv.x | iv.y | iv.z | iv.w) == 0) continue;
            const float4 v = make_float4((float)iv.x * t.qfix_inv, (float)iv.y * t.qfix_inv,
                                         (float)iv.z * t.qfix_inv, (float)iv.w * t.qfix_inv);
            const int cz = row / TG::E, by = row - cz * TG::E;
            const int gc = wrapi(tc0 + cz, a.Nc), gb = wrapi(tb0 + by, a.Nb), ga = wrapi(ta0 + 4 * q4, a.Na);
            atomicAdd((float4 *)((float *)g + ((size_t)gc * a.Nb + gb) * a.Na + ga), v);
        }
    } else {
        for (int row = warp; row < NROW; row += nwarp) {
            const int cz = row / TG::E, by = row - cz * TG::E;
            R *dst = g + ((size_t)wrapi(tc0 + cz, a.Nc) * a.Nb + wrapi(tb0 + by, a.Nb)) * a.Na;
            for (int ax = lane; ax < TG::E; ax += 32) {
                const R v = (float)((const int *)tl)[row * TG::PA + ax] * t.qfix_inv;
                if (v != (R)0) atomicAdd(dst + wrapi(ta0 + ax, a.Na), v);
            }
        }
    }
}

// FP64 spread: shared FP64 atomics are compare-and-swap loops, so here every
// c plane of the shared tile belongs to one warp (plane c to warp c mod 8)
// and is added to by plain loads and stores.  The block stages 16 records'
// weights at a time in shared memory (8 threads a record, one barrier a
// batch); each warp then walks the records, whose stencil holds one plane of
// its own for every order up to 8, and adds its 8 a x 8 b points, 32 at a
// time.  4096 TIP4P/F x 32 beads, 64^3, order 8: 525 us with atomics.
constexpr int kOwnBatch = 16;  // two blocks of 16-point tiles still fit an SM
template <int NI, int TT>
constexpr size_t spread_own_smem()
{
    return sizeof(double) * ((size_t)TileGeom<NI, TT>::NPT + 2 * kOwnBatch * 3 * RecGeom<NI>::NIP);
}

template <int NI, int TT>
__global__ void __launch_bounds__(256, 2) spread_own_kernel(const __grid_constant__ PmeArgs a,
                                                            const __grid_constant__ TileArgs t)
{
    stamp_start(a.stamp, T_PME0);
    typedef TileGeom<NI, TT> TG;
    constexpr int NIP = RecGeom<NI>::NIP, NTB = (NI + 3) / 4, NS8 = (NI + 7) / 8;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    double *tl = (double *)smem_raw;
    double *wst = tl + TG::NPT;  // [2][kOwnBatch][3][NIP]: M_a, M_b, q M_c by stencil point
    __shared__ __align__(16) PolyTab<double, NI> pt;
    __shared__ int4 org[2][kOwnBatch];  // stencil origin in the tile, record number (~record: outside the tile)
    for (int i = threadIdx.x; i < TG::NPT; i += 256) tl[i] = 0.0;
    pt.fill(false);
    SpreadPoly<double, NI> sp;
    sp.init(&pt, threadIdx.x & 31);
    __syncthreads();
    const int tile = blockIdx.x, b = blockIdx.y / t.nshare, z = blockIdx.y - b * t.nshare;
    const int ta0 = (tile % t.nta) * TG::T, tb0 = ((tile / t.nta) % t.ntb) * TG::T, tc0 = (tile / (t.nta * t.ntb)) * TG::T;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int la8 = lane & 7, lb4 = lane >> 3;
    const int n = min(t.cnt[b * t.ntile + tile], t.cap);
    const int *list = t.bin + ((size_t)b * t.ntile + tile) * t.cap;
    double *g = (double *)a.grid + (size_t)b * a.Na * a.Nb * a.Nc;
    int buf = 0;
    for (int e0 = kOwnBatch * z; e0 < n; e0 += kOwnBatch * t.nshare, buf ^= 1) {
        const int nb = min(kOwnBatch, n - e0);
        {
            const int r = threadIdx.x >> 3, j0 = threadIdx.x & 7;
            if (r < nb) {
                const int idx = list[e0 + r];
                const double4 fr = load_frac<double>(a.rw, idx);
                double *w = wst + (buf * kOwnBatch + r) * 3 * NIP;
#pragma unroll
                for (int s = 0; s < NS8; s++) {
                    const int j = j0 + 8 * s;
                    if (j >= NI) break;
                    w[j] = poly_eval<double, NI>(pt.m[NI - 1 - j], fr.x);
                    w[NIP + j] = poly_eval<double, NI>(pt.m[NI - 1 - j], fr.y);
                    w[2 * NIP + j] = fr.w * poly_eval<double, NI>(pt.m[NI - 1 - j], fr.z);
                }
                if (j0 == 0) {
                    const int4 h = a.rhead[idx];
                    const int oa = h.y - ta0, ob = h.z - tb0, oc = h.w - tc0;
                    const bool in = oa >= 0 && oa < TG::T && ob >= 0 && ob < TG::T && oc >= 0 && oc < TG::T;
                    org[buf][r] = make_int4(oa, ob, oc, in ? idx : ~idx);
                }
            }
        }
        __syncthreads();  // the other buffer's readers are done when its writers come back
        for (int r = 0; r < nb; r++) {
            const int4 o = org[buf][r];
            const double *w = wst + (buf * kOwnBatch + r) * 3 * NIP;
            if (o.w >= 0) {
#pragma unroll
                for (int s8 = 0; s8 < NS8; s8++) {
                    const int p = ((warp - o.z) & 7) + 8 * s8;
                    if (p >= NI) break;
                    const double mc = w[2 * NIP + p];
                    double *row = tl + ((o.z + p) * TG::E + o.y + lb4) * TG::PA + o.x + la8;
#pragma unroll
                    for (int s = 0; s < NS8; s++) {
                        if (la8 + 8 * s >= NI) break;
                        const double ca = mc * w[la8 + 8 * s];
#pragma unroll
                        for (int i = 0; i < NTB; i++)
                            if (lb4 + 4 * i < NI) row[4 * i * TG::PA + 8 * s] += ca * w[NIP + lb4 + 4 * i];
                    }
                }
            } else if (warp == 0) {
                // origin outside the tile (none is expected): straight into the grid
                const int idx = ~o.w;
                const int4 h = a.rhead[idx];
                const double4 fr = load_frac<double>(a.rw, idx);
                SpreadW<double, NI> sw;
                sw.eval(sp, fr, lane);
                spread_warp_global<double, NI>(a, g, h.y, h.z, h.w, sw, fr.w, lane);
            }
            __syncwarp();
        }
    }
    // overflow records: one warp each, straight into the grid
    const int nov = t.cnt[a.P * t.ntile];
    const int gid = blockIdx.y * gridDim.x + blockIdx.x, nblk = gridDim.x * gridDim.y;
    for (int e = gid * 8 + warp; e < nov; e += nblk * 8) {
        const int idx = t.ovf[e];
        const int4 h = a.rhead[idx];
        const double4 fr = load_frac<double>(a.rw, idx);
        SpreadW<double, NI> sw;
        sw.eval(sp, fr, lane);
        spread_warp_global<double, NI>(a, (double *)a.grid + (size_t)(idx % a.P) * a.Na * a.Nb * a.Nc, h.y, h.z, h.w,
                                       sw, fr.w, lane);
    }
    __syncthreads();
    constexpr int NROW = TG::E * TG::E;
    for (int i = threadIdx.x; i < NROW * TG::PA; i += 256) {
        const double v = tl[i];
        if (v == 0.0) continue;
        const int row = i / TG::PA, ax = i - row * TG::PA;
        const int cz = row / TG::E, by = row - cz * TG::E;
        atomicAdd(g + ((size_t)wrapi(tc0 + cz, a.Nc) * a.Nb + wrapi(tb0 + by, a.Nb)) * a.Na + wrapi(ta0 + ax, a.Na), v);
    }
}

template <int NI, int TT>
__global__ void __launch_bounds__(256) spread_tile_c_kernel(const __grid_constant__ PmeArgs a,
                                                            const __grid_constant__ TileArgs t)
{
    stamp_start(a.stamp, T_PME0);
    spread_tile_c_body<NI, TT>(a, t, hw_blk());
}

// Gather weights of one record for lane l8 of an 8-lane group: its a
// points (l8, l8 + 8) with derivatives, and all b and c points, evaluated by
// lane t % 8 of the group and shuffled; up to order 8 from the lane's piece
// in registers.  Every lane of the warp calls it.
template <typename R, int NI>
__device__ __forceinline__ void gather_weights(const PolyTab<R, NI> &pt, const Piece<R, NI <= 8 ? NI : 4> &piece,
                                               const typename Vec4<R>::T &fr, int l8, LaneW<R, NI, true> &lw)
{
    R ob[2], odb[2], oc[2], odc[2];
    if constexpr (NI <= 8) {
        piece.both(fr.x, lw.wa0, lw.da0);
        piece.both(fr.y, ob[0], odb[0]);
        piece.both(fr.z, oc[0], odc[0]);
        lw.wa1 = lw.da1 = ob[1] = odb[1] = oc[1] = odc[1] = (R)0;
    } else {
        const bool t0 = l8 < NI, t1 = NI > 8 && l8 + 8 < NI;
        const int p0 = NI - 1 - (t0 ? l8 : 0), p1 = NI - 1 - (t1 ? l8 + 8 : 0);
        lw.wa0 = t0 ? poly_eval<R, NI>(pt.m[p0], fr.x) : (R)0;
        lw.da0 = t0 ? poly_eval<R, NI>(pt.dm[p0], fr.x) : (R)0;
        lw.wa1 = t1 ? poly_eval<R, NI>(pt.m[p1], fr.x) : (R)0;
        lw.da1 = t1 ? poly_eval<R, NI>(pt.dm[p1], fr.x) : (R)0;
        ob[0] = t0 ? poly_eval<R, NI>(pt.m[p0], fr.y) : (R)0;
        odb[0] = t0 ? poly_eval<R, NI>(pt.dm[p0], fr.y) : (R)0;
        oc[0] = t0 ? poly_eval<R, NI>(pt.m[p0], fr.z) : (R)0;
        odc[0] = t0 ? poly_eval<R, NI>(pt.dm[p0], fr.z) : (R)0;
        ob[1] = t1 ? poly_eval<R, NI>(pt.m[p1], fr.y) : (R)0;
        odb[1] = t1 ? poly_eval<R, NI>(pt.dm[p1], fr.y) : (R)0;
        oc[1] = t1 ? poly_eval<R, NI>(pt.m[p1], fr.z) : (R)0;
        odc[1] = t1 ? poly_eval<R, NI>(pt.dm[p1], fr.z) : (R)0;
    }
#pragma unroll
    for (int s = 0; s < RecGeom<NI>::NIP; s++) {
        if (s >= NI) {
            lw.mb[s] = lw.mc[s] = lw.db[s] = lw.dc[s] = (R)0;
            continue;
        }
        const int h = s >= 8 ? 1 : 0;
        lw.mb[s] = __shfl_sync(0xffffffffu, ob[h], s & 7, 8);
        lw.db[s] = __shfl_sync(0xffffffffu, odb[h], s & 7, 8);
        lw.mc[s] = __shfl_sync(0xffffffffu, oc[h], s & 7, 8);
        lw.dc[s] = __shfl_sync(0xffffffffu, odc[h], s & 7, 8);
    }
}

// Gather: one block per (tile, bead), the tile's potential copied to shared
// memory once, 8 lanes per record, the weights evaluated in the block and the
// next record read ahead.  Bound by shared-memory wavefronts (80 % of the
// pipe), 60 % of the loads' being bank conflicts of four records at unrelated
// origins: 132 -> 125 us at 4096 TIP4P/F x 32, 64^3, order 8; FP64 401 -> 193.
template <typename R, int NI, int TT>
__device__ __forceinline__ void gather_tile_c_body(const PmeArgs &a, const Cell &cell, const TileArgs &t, const VBlk vb)
{
    typedef TileGeom<NI, TT> TG;
    typedef typename Vec4<R>::T R4;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    R *tl = (R *)smem_raw;
    __shared__ __align__(16) PolyTab<R, NI> pt;
    if (NI > 8) pt.fill(true);
    Piece<R, NI <= 8 ? NI : 4> piece;
    piece.load(threadIdx.x & 7);
    const int tile = vb.x, b = vb.y / t.nshare, z = vb.y - b * t.nshare;
    const int ta0 = (tile % t.nta) * TG::T, tb0 = ((tile / t.nta) % t.ntb) * TG::T, tc0 = (tile / (t.nta * t.ntb)) * TG::T;
    const R *g = (const R *)a.grid + (size_t)b * a.Na * a.Nb * a.Nc;
    const int n = min(t.cnt[b * t.ntile + tile], t.cap);
    const int grp = threadIdx.x >> 3, l8 = threadIdx.x & 7, ngrp = blockDim.x >> 3;
    if (n > z * ngrp) load_tile<R, TG>(tl, g, a.Na, a.Nb, a.Nc, ta0, tb0, tc0);
    __syncthreads();
    const int *list = t.bin + ((size_t)b * t.ntile + tile) * t.cap;
    const int eb = z * ngrp, estep = ngrp * t.nshare;
    const int nr = n > eb ? (n - eb + estep - 1) / estep : 0;  // same trip count in every group of a warp (shuffles)
    int4 hn = make_int4(0, 0, 0, 0);
    R4 fn = {};
    int in = 0;
    if (eb + grp < n) {
        in = list[eb + grp];
        hn = a.rhead[in];
        fn = load_frac<R>(a.rw, in);
    }
    for (int r = 0; r < nr; r++) {
        const int e = eb + r * estep + grp;
        const bool act = e < n;
        const int idx = in;
        const int4 h = hn;
        const R4 fr = fn;
        if (e + estep < n) {
            in = list[e + estep];
            hn = a.rhead[in];
            fn = load_frac<R>(a.rw, in);
        }
        LaneW<R, NI, true> lw;
        gather_weights<R, NI>(pt, piece, fr, l8, lw);
        double ea = 0, eb = 0, ec = 0;
        if (act) {
            const int oa = h.y - ta0, ob = h.z - tb0, oc = h.w - tc0;
            if (oa >= 0 && oa < TG::T && ob >= 0 && ob < TG::T && oc >= 0 && oc < TG::T) {
                const R *base = tl + (oc * TG::E + ob) * TG::PA + oa;
                gather_lane<R, NI>([&](int tc, int tb, int ta) { return base[(tc * TG::E + tb) * TG::PA + ta]; }, lw,
                                   l8, ea, eb, ec);
            } else {
                gather_lane<R, NI>(
                    [&](int tc, int tb, int ta) {
                        return g[((size_t)wrapi(h.w + tc, a.Nc) * a.Nb + wrapi(h.z + tb, a.Nb)) * a.Na +
                                 wrapi(h.y + ta, a.Na)];
                    },
                    lw, l8, ea, eb, ec);
            }
        }
        gather_store(a, cell, h.x, idx, ea, eb, ec, act ? l8 : 1);
    }
    const int nov = t.cnt[a.P * t.ntile];
    const int gid = vb.y * vb.gx + vb.x, nblk = vb.gx * vb.gy;
    const int nr2 = (nov + nblk * ngrp - 1) / (nblk * ngrp);
    for (int r = 0; r < nr2; r++) {
        const int e = (r * nblk + gid) * ngrp + grp;
        const bool act = e < nov;
        int idx = 0;
        int4 h = make_int4(0, 0, 0, 0);
        R4 fr = {};
        if (act) {
            idx = t.ovf[e];
            h = a.rhead[idx];
            fr = load_frac<R>(a.rw, idx);
        }
        LaneW<R, NI, true> lw;
        gather_weights<R, NI>(pt, piece, fr, l8, lw);
        double ea = 0, eb = 0, ec = 0;
        if (act) {
            const R *g2 = (const R *)a.grid + (size_t)(idx % a.P) * a.Na * a.Nb * a.Nc;
            gather_lane<R, NI>(
                [&](int tc, int tb, int ta) {
                    return g2[((size_t)wrapi(h.w + tc, a.Nc) * a.Nb + wrapi(h.z + tb, a.Nb)) * a.Na +
                              wrapi(h.y + ta, a.Na)];
                },
                lw, l8, ea, eb, ec);
        }
        gather_store(a, cell, h.x, idx, ea, eb, ec, act ? l8 : 1);
    }
}

// Resident blocks per SM the FP32 gather (order <= 8) is compiled for: its
// shared tile of 16-point edges allows 4; at 4 the 64-register cap spills
// 60 bytes and the C3 evaluation is still 2.8 % faster than at 3 (80
// registers).  The others hold 2 (128 registers).
#ifndef PINYB200_GATHER_BLOCKS
#define PINYB200_GATHER_BLOCKS 4
#endif
template <typename R, int NI, int TT>
__global__ void __launch_bounds__(256, sizeof(R) == 4 && NI <= 8 ? PINYB200_GATHER_BLOCKS : 2)
    gather_tile_c_kernel(const __grid_constant__ PmeArgs a,
                                                            const __grid_constant__ Cell cell,
                                                            const __grid_constant__ TileArgs t)
{
    gather_tile_c_body<R, NI, TT>(a, cell, t, hw_blk());
    stamp_end(a.stamp, T_PME1);
}

// ---------------------------------------------------------------------------
// In-place FFTs of `nl` lines of length N held in shared memory: element n of
// line l at sm[l * ls + n * es].  Unnormalised, exp(sign 2 pi i n k / N);
// tw[2m], tw[2m+1] = cos, sin(2 pi m / N).  Power-of-two lengths up to 256
// use Stockham autosort passes of radix 8 and 4 (16 = 4x4, 32 = 8x4,
// 64 = 8x8, 128 = 8x4x4, 256 = 8x8x4): one butterfly per thread and pass,
// read into registers, barrier, written back in place.  Other lengths use a
// direct DFT done a block of lines at a time.  Every thread of the block
// must call these.

// R-point DFT in registers, exp(SIGN 2 pi i r k / R), R = 2, 4, 8.
template <typename R, int RAD, int SIGN>
__device__ __forceinline__ void dft_small(typename Cplx<R>::T *v)
{
    typedef typename Cplx<R>::T C2;
    if (RAD == 2) {
        const C2 a = v[0], b = v[1];
        v[0].x = a.x + b.x;
        v[0].y = a.y + b.y;
        v[1].x = a.x - b.x;
        v[1].y = a.y - b.y;
    } else if (RAD == 4) {
        const R s = (R)SIGN;
        const C2 t0 = {v[0].x + v[2].x, v[0].y + v[2].y}, t1 = {v[0].x - v[2].x, v[0].y - v[2].y};
        const C2 t2 = {v[1].x + v[3].x, v[1].y + v[3].y};
        // (v1 - v3) * (SIGN i)
        const C2 t3 = {-s * (v[1].y - v[3].y), s * (v[1].x - v[3].x)};
        v[0].x = t0.x + t2.x;
        v[0].y = t0.y + t2.y;
        v[2].x = t0.x - t2.x;
        v[2].y = t0.y - t2.y;
        v[1].x = t1.x + t3.x;
        v[1].y = t1.y + t3.y;
        v[3].x = t1.x - t3.x;
        v[3].y = t1.y - t3.y;
    } else {
        // radix 2 over two 4-point DFTs: X_k = E_k + w^k O_k, X_k+4 = E_k - w^k O_k
        C2 e[4] = {v[0], v[2], v[4], v[6]}, o[4] = {v[1], v[3], v[5], v[7]};
        dft_small<R, 4, SIGN>(e);
        dft_small<R, 4, SIGN>(o);
        const R s = (R)SIGN, h = (R)0.70710678118654752440;  // cos(pi/4)
        C2 w[4];
        w[0] = o[0];
        w[1] = {h * (o[1].x - s * o[1].y), h * (o[1].y + s * o[1].x)};   // (1 + s i) / sqrt 2
        w[2] = {-s * o[2].y, s * o[2].x};                                  // s i
        w[3] = {h * (-o[3].x - s * o[3].y), h * (-o[3].y + s * o[3].x)};  // (-1 + s i) / sqrt 2
#pragma unroll
        for (int k = 0; k < 4; k++) {
            v[k].x = e[k].x + w[k].x;
            v[k].y = e[k].y + w[k].y;
            v[k + 4].x = e[k].x - w[k].x;
            v[k + 4].y = e[k].y - w[k].y;
        }
    }
}

__host__ __device__ constexpr int stockham_radix(int rem) { return rem == 16 ? 4 : (rem % 8 == 0 ? 8 : rem); }
__host__ __device__ constexpr int stockham_min_radix(int n, int ns)
{
    return ns >= n ? 8 : (stockham_radix(n / ns) < stockham_min_radix(n, ns * stockham_radix(n / ns))
                              ? stockham_radix(n / ns)
                              : stockham_min_radix(n, ns * stockham_radix(n / ns)));
}

// One Stockham pass (stride NS) over lines l0 .. l0+nlg-1, then the next.
// Consecutive threads take consecutive lines (G lines per round) and share
// the butterfly index j: a half-warp then touches 16 different lines at the
// same position, which fall in 16 different bank pairs both for lines along
// the fast axis (odd line stride) and across it (line stride 1), and reads
// one twiddle (a broadcast).
template <typename R, int N, int NS, int SIGN>
__device__ __forceinline__ void stockham_pass(typename Cplx<R>::T *sm, int l0, int nlg, int G, int ls, int es,
                                              const R *tw)
{
    typedef typename Cplx<R>::T C2;
    constexpr int RAD = stockham_radix(N / NS);
    constexpr int BPL = N / RAD;  // butterflies per line
    const int l = threadIdx.x % G, j = threadIdx.x / G;
    const bool act = l < nlg && j < BPL;
    C2 v[RAD];
    C2 *p = sm + (size_t)(l0 + (act ? l : 0)) * ls;
    if (act) {
#pragma unroll
        for (int r = 0; r < RAD; r++) v[r] = p[(j + r * BPL) * es];
        if (NS > 1) {
            const int k = j % NS;
#pragma unroll
            for (int r = 1; r < RAD; r++) {
                const int m = r * k * (N / (NS * RAD));
                const R wr = tw[2 * m], wi = (R)SIGN * tw[2 * m + 1];
                const R xr = v[r].x * wr - v[r].y * wi, xi = v[r].x * wi + v[r].y * wr;
                v[r].x = xr;
                v[r].y = xi;
            }
        }
        dft_small<R, RAD, SIGN>(v);
    }
    __syncthreads();
    if (act) {
        const int d = (j / NS) * NS * RAD + j % NS;
#pragma unroll
        for (int r = 0; r < RAD; r++) p[(d + r * NS) * es] = v[r];
    }
    __syncthreads();
    if constexpr (NS * RAD < N) stockham_pass<R, N, NS * RAD, SIGN>(sm, l0, nlg, G, ls, es, tw);
}

template <typename R, int N, int SIGN>
__device__ __forceinline__ void fft_pow2_inl(typename Cplx<R>::T *sm, int nl, int ls, int es, const R *tw)
{
    constexpr int BPLMAX = N / stockham_min_radix(N, 1);
    const int G = (int)blockDim.x / BPLMAX > 0 ? (int)blockDim.x / BPLMAX : 1;  // lines per round
    for (int l0 = 0; l0 < nl; l0 += G) stockham_pass<R, N, 1, SIGN>(sm, l0, min(G, nl - l0), G, ls, es, tw);
}

// Out-of-line copy for kernels whose lengths are known only at run time.
template <typename R, int N, int SIGN>
__device__ __noinline__ void fft_pow2(typename Cplx<R>::T *sm, int nl, int ls, int es, const R *tw)
{
    fft_pow2_inl<R, N, SIGN>(sm, nl, ls, es, tw);
}

template <typename R, int SIGN>
__device__ bool fft_pow2_dispatch(typename Cplx<R>::T *sm, int N, int nl, int ls, int es, const R *tw)
{
    switch (N) {
    case 2: fft_pow2<R, 2, SIGN>(sm, nl, ls, es, tw); return true;
    case 4: fft_pow2<R, 4, SIGN>(sm, nl, ls, es, tw); return true;
    case 8: fft_pow2<R, 8, SIGN>(sm, nl, ls, es, tw); return true;
    case 16: fft_pow2<R, 16, SIGN>(sm, nl, ls, es, tw); return true;
    case 32: fft_pow2<R, 32, SIGN>(sm, nl, ls, es, tw); return true;
    case 64: fft_pow2<R, 64, SIGN>(sm, nl, ls, es, tw); return true;
    case 128: fft_pow2<R, 128, SIGN>(sm, nl, ls, es, tw); return true;
    case 256: fft_pow2<R, 256, SIGN>(sm, nl, ls, es, tw); return true;
    default: return false;
    }
}

template <typename R>
__device__ void smem_fft(typename Cplx<R>::T *sm, int N, int nl, int ls, int es, const R *tw, int sign)
{
    typedef typename Cplx<R>::T C2;
    const int nt = blockDim.x;
    if (N == 1) return;
    if (sign > 0 ? fft_pow2_dispatch<R, 1>(sm, N, nl, ls, es, tw) : fft_pow2_dispatch<R, -1>(sm, N, nl, ls, es, tw))
        return;
    {
        const int per = nt / N;  // lines per pass
        for (int l0 = 0; l0 < nl; l0 += per) {
            const int l = l0 + threadIdx.x / N, k = threadIdx.x % N;
            R sr = 0, si = 0;
            const bool act = threadIdx.x < per * N && l < nl;
            if (act) {
                const C2 *p = sm + l * ls;
                for (int n = 0; n < N; n++) {
                    const int e = (int)(((long long)n * k) % N);
                    const R wr = tw[2 * e], wi = (R)sign * tw[2 * e + 1];
                    const C2 v = p[n * es];
                    sr += v.x * wr - v.y * wi;
                    si += v.x * wi + v.y * wr;
                }
            }
            __syncthreads();
            if (act) {
                sm[l * ls + k * es].x = sr;
                sm[l * ls + k * es].y = si;
            }
            __syncthreads();
        }
    }
}

// Plane and slab kernels of meshes whose lengths are known only at run time
// (not cubic, or an edge fft.cuh does not build): one complex line per real
// row, every length from order to 256.

template <typename R>
__device__ __forceinline__ void load_twiddles(R *dst, const R *src, int N)
{
    for (int i = threadIdx.x; i < 2 * N; i += blockDim.x) dst[i] = src[i];
}

// Forward transform of one (bead, c) plane along a then b; half spectrum
// (a <= Na/2) out.  Shared: plane [Nb][Na+1] complex, twiddles.
template <typename R>
__device__ __forceinline__ void plane_fwd_body(const R *__restrict__ q, typename Cplx<R>::T *__restrict__ spec, int Na,
                                               int Nb, int Nc, const R *__restrict__ twa, const R *__restrict__ twb,
                                               const VBlk vb)
{
    (void)Nc;
    typedef typename Cplx<R>::T C2;
    extern __shared__ unsigned char smem_raw[];
    C2 *pl = (C2 *)smem_raw;
    const int ls = Na + 1;
    R *ta = (R *)(pl + (size_t)Nb * ls);
    R *tb = ta + 2 * Na;
    const int Nh = Na / 2 + 1;
    const size_t plane = vb.x;  // bead * Nc + c
    load_twiddles(ta, twa, Na);
    load_twiddles(tb, twb, Nb);
    const R *src = q + plane * Na * Nb;
    for (int idx = threadIdx.x; idx < Na * Nb; idx += blockDim.x) {
        C2 v;
        v.x = src[idx];
        v.y = (R)0;
        pl[(idx / Na) * ls + idx % Na] = v;
    }
    __syncthreads();
    smem_fft<R>(pl, Na, Nb, ls, 1, ta, +1);   // along a, every row
    smem_fft<R>(pl, Nb, Nh, 1, ls, tb, +1);   // along b, columns a <= Na/2
    C2 *dst = spec + plane * (size_t)Nb * Nh;
    for (int idx = threadIdx.x; idx < Nb * Nh; idx += blockDim.x) dst[idx] = pl[(idx / Nh) * ls + idx % Nh];
}

template <typename R>
__global__ void __launch_bounds__(256) plane_fwd_kernel(const R *__restrict__ q, typename Cplx<R>::T *__restrict__ spec,
                                                        int Na, int Nb, int Nc, const R *__restrict__ twa,
                                                        const R *__restrict__ twb)
{
    plane_fwd_body<R>(q, spec, Na, Nb, Nc, twa, twb, hw_blk());
}

// Inverse of plane_fwd: half spectrum in, along b, Hermitian completion of
// each row (U(Na-a) = conj U(a) once b and c are back in real space), along
// a, real part out.
template <typename R>
__device__ __forceinline__ void plane_inv_body(const typename Cplx<R>::T *__restrict__ spec, R *__restrict__ phi, int Na,
                                               int Nb, int Nc, const R *__restrict__ twa, const R *__restrict__ twb,
                                               const VBlk vb)
{
    (void)Nc;
    typedef typename Cplx<R>::T C2;
    extern __shared__ unsigned char smem_raw[];
    C2 *pl = (C2 *)smem_raw;
    const int ls = Na + 1;
    R *ta = (R *)(pl + (size_t)Nb * ls);
    R *tb = ta + 2 * Na;
    const int Nh = Na / 2 + 1;
    const size_t plane = vb.x;
    load_twiddles(ta, twa, Na);
    load_twiddles(tb, twb, Nb);
    const C2 *src = spec + plane * (size_t)Nb * Nh;
    for (int idx = threadIdx.x; idx < Nb * Nh; idx += blockDim.x) pl[(idx / Nh) * ls + idx % Nh] = src[idx];
    __syncthreads();
    smem_fft<R>(pl, Nb, Nh, 1, ls, tb, -1);
    for (int idx = threadIdx.x; idx < Nb * Na; idx += blockDim.x) {
        const int b = idx / Na, a = idx % Na;
        if (a >= Nh) {
            C2 v = pl[b * ls + (Na - a)];
            v.y = -v.y;
            pl[b * ls + a] = v;
        }
    }
    __syncthreads();
    smem_fft<R>(pl, Na, Nb, ls, 1, ta, -1);
    R *dst = phi + plane * Na * Nb;
    for (int idx = threadIdx.x; idx < Na * Nb; idx += blockDim.x) dst[idx] = pl[(idx / Na) * ls + idx % Na].x;
}

template <typename R>
__global__ void __launch_bounds__(256) plane_inv_kernel(const typename Cplx<R>::T *__restrict__ spec, R *__restrict__ phi,
                                                        int Na, int Nb, int Nc, const R *__restrict__ twa,
                                                        const R *__restrict__ twb)
{
    plane_inv_body<R>(spec, phi, Na, Nb, Nc, twa, twb, hw_blk());
}

// One (bead, b) slab of the half spectrum: FFT along c, energy and virial
// of the k-sphere terms (ewald3d_pme.c:366-425), multiplication by the
// influence function, inverse FFT along c.  Half-spectrum points with
// 0 < a < Na/2 stand for two full-grid points; E = 1/2 sum_full w |S|^2.
template <typename R>
__device__ __forceinline__ void conv_c_body(typename Cplx<R>::T *__restrict__ spec, const R *__restrict__ filt, int Na,
                                            int Nb, int Nc, const R *__restrict__ twc, const Cell &cell, double alp,
                                            double *__restrict__ acc, int energy, const VBlk vb)
{
    typedef typename Cplx<R>::T C2;
    extern __shared__ unsigned char smem_raw[];
    C2 *sl = (C2 *)smem_raw;
    const int Nh = Na / 2 + 1;
    const int ls = Nh + 1;  // padded line stride: element c of column a at sl[c * ls + a]
    R *tc = (R *)(sl + (size_t)Nc * ls);
    __shared__ double red[7][8];
    const int bead = vb.x / Nb, b = vb.x % Nb;
    load_twiddles(tc, twc, Nc);
    C2 *base = spec + ((size_t)bead * Nc * Nb + b) * Nh;
    const size_t cstride = (size_t)Nb * Nh;
    for (int idx = threadIdx.x; idx < Nc * Nh; idx += blockDim.x) {
        const int c = idx / Nh, a = idx % Nh;
        sl[c * ls + a] = base[c * cstride + a];
    }
    __syncthreads();
    smem_fft<R>(sl, Nc, Nh, 1, ls, tc, +1);
    // per-point energy and virial terms in R (FP32 for MIXED), summed in FP64
    double e = 0, pxx = 0, pyy = 0, pzz = 0, pxy = 0, pxz = 0, pyz = 0;
    const R kb = (R)(b <= Nb / 2 ? b : b - Nb);
    const R tpi = (R)(2.0 * M_PI), falp2 = (R)(4.0 * alp * alp);
    R hi[9];
#pragma unroll
    for (int k = 0; k < 9; k++) hi[k] = (R)cell.hi[k];
    for (int idx = threadIdx.x; idx < Nc * Nh; idx += blockDim.x) {
        const int c = idx / Nh, a = idx % Nh;
        const R w = filt[((size_t)c * Nb + b) * Na + a];
        C2 s = sl[c * ls + a];
        if (w != (R)0 && energy) {
            const R ka = (R)a, kc = (R)(c <= Nc / 2 ? c : c - Nc);
            const R xk = tpi * (ka * hi[0] + kb * hi[1] + kc * hi[2]);
            const R yk = tpi * (ka * hi[3] + kb * hi[4] + kc * hi[5]);
            const R zk = tpi * (ka * hi[6] + kb * hi[7] + kc * hi[8]);
            const R g2 = xk * xk + yk * yk + zk * zk;
            const R mult = (a == 0 || 2 * a == Na) ? (R)0.5 : (R)1.0;
            const R sm = mult * (s.x * s.x + s.y * s.y) * w;
            const R prep = (R)-2.0 * ((g2 / falp2) + (R)1.0) / g2 * sm;
            e += (double)sm;
            pxx += (double)(prep * xk * xk);
            pyy += (double)(prep * yk * yk);
            pzz += (double)(prep * zk * zk);
            pxy += (double)(prep * xk * yk);
            pxz += (double)(prep * xk * zk);
            pyz += (double)(prep * yk * zk);
        }
        s.x *= w;
        s.y *= w;
        sl[c * ls + a] = s;
    }
    __syncthreads();
    smem_fft<R>(sl, Nc, Nh, 1, ls, tc, -1);
    for (int idx = threadIdx.x; idx < Nc * Nh; idx += blockDim.x) {
        const int c = idx / Nh, a = idx % Nh;
        base[c * cstride + a] = sl[c * ls + a];
    }
    if (!energy) return;
    double v[7] = {e, pxx, pyy, pzz, pxy, pxz, pyz};
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
#pragma unroll
    for (int k = 0; k < 7; k++) {
        double t = warp_sum(v[k]);
        if (lane == 0) red[k][wid] = t;
    }
    __syncthreads();
    if (threadIdx.x < 7) {
        double t = 0;
        for (int w2 = 0; w2 < (int)(blockDim.x >> 5); w2++) t += red[threadIdx.x][w2];
        const int slot[7] = {S_VRECIP, S_PXX, S_PYY, S_PZZ, S_PXY, S_PXZ, S_PYZ};
        atomicAdd(&acc[(size_t)bead * S_NSLOT + slot[threadIdx.x]], t);
        if (threadIdx.x == 0) {
            // diagonal vnow term of the pressure tensor (ewald3d_pme.c:415-417)
            atomicAdd(&acc[(size_t)bead * S_NSLOT + S_PXX], t);
            atomicAdd(&acc[(size_t)bead * S_NSLOT + S_PYY], t);
            atomicAdd(&acc[(size_t)bead * S_NSLOT + S_PZZ], t);
        }
    }
}

template <typename R>
__global__ void __launch_bounds__(256) conv_c_kernel(typename Cplx<R>::T *__restrict__ spec, const R *__restrict__ filt,
                                                     int Na, int Nb, int Nc, const R *__restrict__ twc,
                                                     const __grid_constant__ Cell cell, double alp,
                                                     double *__restrict__ acc, int energy)
{
    conv_c_body<R>(spec, filt, Na, Nb, Nc, twc, cell, alp, acc, energy, hw_blk());
}

// ---------------------------------------------------------------------------
// Influence function on the full grid: preg * bweight for grid points whose
// k (or -k) is on PINY's list, zero elsewhere.
__global__ void filter_kernel(int Na, int Nb, int Nc, const int *__restrict__ kmask, const int *__restrict__ kvec,
                              const double *__restrict__ bw, Cell cell, double alp, double *__restrict__ f64,
                              float *__restrict__ f32)
{
    const size_t G = (size_t)Na * Nb * Nc;
    const size_t g = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (g >= G) return;
    const int idx = kmask[g];
    double w = 0.0;
    if (idx >= 0) {
        const double tpi = 2.0 * M_PI;
        const double aka = tpi * (double)kvec[3 * idx], akb = tpi * (double)kvec[3 * idx + 1],
                     akc = tpi * (double)kvec[3 * idx + 2];
        const double xk = (aka * cell.hi[0] + akb * cell.hi[1] + akc * cell.hi[2]);
        const double yk = (aka * cell.hi[3] + akb * cell.hi[4] + akc * cell.hi[5]);
        const double zk = (aka * cell.hi[6] + akb * cell.hi[7] + akc * cell.hi[8]);
        const double g2 = xk * xk + yk * yk + zk * zk;
        const double falp2 = 4.0 * alp * alp;
        const double pivol = cell.vol / (4.0 * M_PI);
        w = exp((-g2 / falp2)) / (g2 * pivol) * bw[idx];
    }
    f64[g] = w;
    f32[g] = (float)w;
}

// Shared memory of the plane and slab kernels.
size_t pme_plane_smem(int Na, int Nb, bool fp64)
{
    const size_t cs = fp64 ? 16 : 8, rs = fp64 ? 8 : 4;
    return cs * (size_t)Nb * (Na + 1) + rs * 2 * (size_t)(Na + Nb);
}
size_t pme_slab_smem(int Na, int Nc, bool fp64)
{
    const size_t cs = fp64 ? 16 : 8, rs = fp64 ? 8 : 4;
    return cs * (size_t)Nc * (Na / 2 + 2) + rs * 2 * (size_t)Nc;
}

// The three FFT kernels for meshes of run-time lengths.
template <typename R>
static cudaError_t launch_fft_rt(pinyb200_ctx *c, const PmeArgs &a, const Cell &cell, typename Cplx<R>::T *spec,
                                const R *filt, const R *const *tw, size_t sp, size_t ss, bool energy)
{
    cudaError_t err = cudaSuccess;
    // opt in to more than 48 KB of dynamic shared memory where a plane needs it
    if (sp > 48 * 1024) {
        err = smem_optin((const void *)plane_fwd_kernel<R>, (int)sp);
        if (err == cudaSuccess)
            err = smem_optin((const void *)plane_inv_kernel<R>, (int)sp);
        if (err != cudaSuccess) return err;
    }
    if (ss > 48 * 1024) {
        err = smem_optin((const void *)conv_c_kernel<R>, (int)ss);
        if (err != cudaSuccess) return err;
    }
    plane_fwd_kernel<R><<<a.P * a.Nc, 256, sp, c->stream>>>((const R *)a.grid, spec, a.Na, a.Nb, a.Nc, tw[0],
                                                                tw[1]);
    if ((err = kt_mark(c, "pme_plane_fwd")) != cudaSuccess) return err;
    conv_c_kernel<R><<<a.P * a.Nb, 256, ss, c->stream>>>(spec, filt, a.Na, a.Nb, a.Nc, tw[2], cell, c->alp_ewd,
                                                             c->d_acc, energy ? 1 : 0);
    if ((err = kt_mark(c, "pme_conv_c")) != cudaSuccess) return err;
    plane_inv_kernel<R><<<a.P * a.Nc, 256, sp, c->stream>>>(spec, (R *)a.grid, a.Na, a.Nb, a.Nc, tw[0], tw[1]);
    if ((err = kt_mark(c, "pme_plane_inv")) != cudaSuccess) return err;
    return cudaGetLastError();
}

// Kernel arguments of a context's PME mesh.
PmeArgs pme_args_of(pinyb200_ctx *c)
{
    const DeviceSystem &s = c->sys;
    PmeArgs a;
    a.natm = s.natm;
    a.P = c->P;
    a.nchrg = s.nchrg;
    a.ichrg = s.ichrg;
    a.charge = s.charge;
    a.posT = c->d_posT;
    a.Na = s.ngrid[0];
    a.Nb = s.ngrid[1];
    a.Nc = s.ngrid[2];
    a.n = s.n_interp;
    a.grid = c->d_grid;
    a.forceP = c->d_forceP;
    a.rhead = (int4 *)c->d_pme_head;
    a.rw = c->d_pme_w;
    a.stamp = (unsigned long long *)(c->d_acc + (size_t)c->P * S_NSLOT);
    return a;
}

static FftArgs fft_args(void *grid, void *spec, const void *filt, const void *tw, const Cell &cell, pinyb200_ctx *c,
                        bool energy)
{
    FftArgs f;
    f.grid = grid;
    f.spec = spec;
    f.filt = filt;
    f.tw = tw;
    f.cell = cell;
    f.alp = c->alp_ewd;
    f.acc = c->d_acc;
    f.energy = energy ? 1 : 0;
    return f;
}

// Transforms, convolution and inverse transforms of one context's mesh: the
// kernels of compile-time edge where built (every cubic mesh PINY chooses up
// to 128^3), else those of run-time lengths.
template <typename R>
static cudaError_t launch_fft(pinyb200_ctx *c, const PmeArgs &a, const Cell &cell, typename Cplx<R>::T *spec,
                              const R *filt, const R *const *tw, size_t sp, size_t ss, bool energy)
{
    if (fft_fixed_edge(a.Na, a.Nb, a.Nc))
        return launch_fft_fixed<R>(c, a.Na, a.P, fft_args(a.grid, spec, filt, tw[0], cell, c, energy));
    return launch_fft_rt<R>(c, a, cell, spec, filt, tw, sp, ss, energy);
}

// Zeroes the charge grid.
cudaError_t launch_pme_clear(pinyb200_ctx *c)
{
    if (c->sys.nchrg == 0 || c->sys.nktot == 0) return cudaSuccess;
    const size_t G = (size_t)c->sys.ngrid[0] * c->sys.ngrid[1] * c->sys.ngrid[2];
    return cudaMemsetAsync(c->d_grid, 0, (c->precision == PINYB200_FP64 ? sizeof(double) : sizeof(float)) * G * c->P,
                           c->stream);
}

// Tile binning arguments of a context's PME mesh for spline order NI and
// tile edge TT.
TileArgs tile_args_of(pinyb200_ctx *c, int NI, int TT)
{
    TileArgs t;
    t.T = TT;
    // fixed-point scale of the FP32 spread tile: every contribution q M_a M_b
    // M_c (bounded by max |q| times the B-spline's peak cubed) below 2^22
    // after scaling, the range the rounding trick is exact in; at most 2^24 (a
    // resolution of 6e-8 against contributions of up to ~0.15), or 2^25 where
    // even a full bin's charges on one grid point stay below 2^31 (order 8 of
    // q-TIP4P/F: the force gradient of 1024 x 16 on 32^3 is 1.3e-7 off FP64 at
    // 2^24, 5e-8 at 2^25 and with FP32 sums).  At 2^24 that takes 128 charges
    // of one sign on a point.
    {
        const double peak = bspline_peak(NI), most = c->q_max * peak * peak * peak;
        int S = 25;
        while (S > 8 && std::ldexp(most, S) >= 0.99 * std::ldexp(1.0, 22)) S--;
        if (S == 25 && c->pme_cap * std::ldexp(most, S) >= std::ldexp(1.0, 31)) S = 24;
        t.qfix = (float)std::ldexp(1.0, S);
        t.qfix_inv = (float)std::ldexp(1.0, -S);
    }
    // few bins (small meshes of few beads): several blocks per bin, each with
    // at least 16 of its records on average
    const int bins = c->pme_ntile * c->P, mean = c->sys.nchrg / std::max(1, c->pme_ntile);
    t.nshare = std::max(1, std::min(std::min(4, 2 * c->sm_count / std::max(1, bins)), mean / 16));
    t.nta = c->pme_nt[0];
    t.ntb = c->pme_nt[1];
    t.ntc = c->pme_nt[2];
    t.ntile = c->pme_ntile;
    t.cap = c->pme_cap;
    t.cnt = c->d_pme_cnt;
    t.bin = c->d_pme_bin;
    t.ovf = c->d_pme_ovf;
    return t;
}

template <typename R, int NI, int TT>
static cudaError_t launch_pme_t(pinyb200_ctx *c, const Cell &cell, bool energy, bool staged)
{
    typedef typename Cplx<R>::T C2;
    const PmeArgs a = pme_args_of(c);
    const size_t G = (size_t)a.Na * a.Nb * a.Nc;
    constexpr bool f64 = sizeof(R) == 8;
    const TileArgs t = tile_args_of(c, NI, TT);
    cudaError_t err = cudaSuccess;
    if (!staged) {
        err = launch_pme_clear(c);
        if (err != cudaSuccess) return err;
        if ((err = kt_mark(c, "pme_grid_clear (memset)")) != cudaSuccess) return err;
        err = cudaMemsetAsync(t.cnt, 0, ((size_t)a.P * t.ntile + 1) * sizeof(int), c->stream);
        if (err != cudaSuccess) return err;
        const long long nt = (long long)a.nchrg * a.P;
        const int threads = 256;
        pme_bin_compact_kernel<R><<<(unsigned)((nt + threads - 1) / threads), threads, 0, c->stream>>>(a, cell, t);
        if ((err = kt_mark(c, "pme_bin")) != cudaSuccess) return err;
    }
    const size_t st = (size_t)TileGeom<NI, TT>::NPT * sizeof(R), ss_spread = spread_smem<R, NI, TT>();
    if (ss_spread > 48 * 1024 - sizeof(PolyTab<R, NI>)) {
        if constexpr (!f64) err = smem_optin((const void *)spread_tile_c_kernel<NI, TT>, (int)ss_spread);
        if (err != cudaSuccess) return err;
    }
    if constexpr (f64) {
        err = smem_optin((const void *)spread_own_kernel<NI, TT>, (int)spread_own_smem<NI, TT>());
        if (err != cudaSuccess) return err;
    }
    if (st > 48 * 1024 - sizeof(PolyTab<R, NI>)) {
        err = smem_optin((const void *)gather_tile_c_kernel<R, NI, TT>, (int)st);
        if (err != cudaSuccess) return err;
    }
    const dim3 tgrid((unsigned)t.ntile, (unsigned)(a.P * t.nshare));
    if constexpr (f64) spread_own_kernel<NI, TT><<<tgrid, 256, spread_own_smem<NI, TT>(), c->stream>>>(a, t);
    else spread_tile_c_kernel<NI, TT><<<tgrid, 256, ss_spread, c->stream>>>(a, t);
    if ((err = kt_mark(c, "pme_spread")) != cudaSuccess) return err;
    const R *twbase = (const R *)(f64 ? (const void *)c->d_twiddle64 : (const void *)c->d_twiddle32);
    const R *tw[3] = {twbase, twbase + 2 * 256, twbase + 4 * 256};
    const size_t sp = pme_plane_smem(a.Na, a.Nb, f64), ss = pme_slab_smem(a.Na, a.Nc, f64);
    C2 *spec = (C2 *)c->d_spec;
    const R *filt = f64 ? (const R *)c->d_filter : (const R *)((const double *)c->d_filter + G);
    err = launch_fft<R>(c, a, cell, spec, filt, tw, sp, ss, energy);
    if (err != cudaSuccess) return err;
    gather_tile_c_kernel<R, NI, TT><<<tgrid, 256, st, c->stream>>>(a, cell, t);
    if ((err = kt_mark(c, "pme_gather")) != cudaSuccess) return err;
    return cudaGetLastError();
}

template <typename R, int TT>
static cudaError_t launch_pme_rt(pinyb200_ctx *c, const Cell &cell, bool energy, bool staged)
{
    switch (c->sys.n_interp) {
    case 4: return launch_pme_t<R, 4, TT>(c, cell, energy, staged);
    case 5: return launch_pme_t<R, 5, TT>(c, cell, energy, staged);
    case 6: return launch_pme_t<R, 6, TT>(c, cell, energy, staged);
    case 7: return launch_pme_t<R, 7, TT>(c, cell, energy, staged);
    case 8: return launch_pme_t<R, 8, TT>(c, cell, energy, staged);
    case 10: return launch_pme_t<R, 10, TT>(c, cell, energy, staged);
    default: return cudaErrorInvalidValue;
    }
}

template <typename R>
static cudaError_t launch_pme_r(pinyb200_ctx *c, const Cell &cell, bool energy, bool staged)
{
    return c->pme_tile == 8 ? launch_pme_rt<R, 8>(c, cell, energy, staged)
                            : launch_pme_rt<R, 16>(c, cell, energy, staged);
}

cudaError_t launch_pme_force_add(pinyb200_ctx *c)
{
    if (c->sys.nchrg == 0 || c->sys.nktot == 0) return cudaSuccess;
    const long long n = (long long)c->sys.nchrg * 3 * c->P;
    pme_force_add_kernel<<<(unsigned)((n + 255) / 256), 256, 0, c->stream>>>(c->sys.nchrg, c->P, c->sys.ichrg,
                                                                            c->d_forceP, c->d_forceT);
    return cudaGetLastError();
}

cudaError_t launch_pme_force_add_scaled(pinyb200_ctx *c, double w, double *target)
{
    if (c->sys.nchrg == 0 || c->sys.nktot == 0) return cudaSuccess;
    const long long n = (long long)c->sys.nchrg * 3 * c->P;
    pme_force_add_scaled_kernel<<<(unsigned)((n + 255) / 256), 256, 0, c->stream>>>(c->sys.nchrg, c->P,
                                                                                   c->sys.ichrg, c->d_forceP, w,
                                                                                   target);
    return cudaGetLastError();
}

// The influence function of the context's mesh for this cell, on st, unless
// it is the one already there.
static cudaError_t launch_filter(pinyb200_ctx *c, const Cell &cell, cudaStream_t st)
{
    bool same = c->filter_ok;
    for (int i = 0; i < 9 && same; i++) same = c->filter_h[i] == cell.h[i];
    if (same) return cudaSuccess;
    const size_t G = (size_t)c->sys.ngrid[0] * c->sys.ngrid[1] * c->sys.ngrid[2];
    filter_kernel<<<(unsigned)((G + 255) / 256), 256, 0, st>>>(
        c->sys.ngrid[0], c->sys.ngrid[1], c->sys.ngrid[2], c->sys.kmask, c->sys.kvec, c->sys.bweight, cell,
        c->alp_ewd, (double *)c->d_filter, (float *)((double *)c->d_filter + G));
    for (int i = 0; i < 9; i++) c->filter_h[i] = cell.h[i];
    c->filter_ok = true;
    return cudaGetLastError();
}

cudaError_t pme_filters_ready(pinyb200_ctx *c, const Cell &cell, cudaStream_t st)
{
    if (c->sys.nchrg == 0) return cudaSuccess;
    cudaError_t e = c->sys.nktot > 0 ? launch_filter(c, cell, st) : cudaSuccess;
    if (e == cudaSuccess && c->pme_res.on) {
        pme_swap(c, c->pme_res);
        e = launch_filter(c, cell, st);
        pme_swap(c, c->pme_res);
    }
    return e;
}

cudaError_t launch_pme(pinyb200_ctx *c, const Cell &cell, bool energy, bool staged)
{
    if (c->sys.nchrg == 0 || c->sys.nktot == 0) return cudaSuccess;
    const cudaError_t err = launch_filter(c, cell, c->stream);
    if (err != cudaSuccess) return err;
    if (c->precision == PINYB200_FP64) return launch_pme_r<double>(c, cell, energy, staged);
    return launch_pme_r<float>(c, cell, energy, staged);
}

// ---------------------------------------------------------------------------
// Many boxes per launch (the batched evaluation): every forward PME kernel of
// the compact FP32 path over a table of boxes, one persistent launch per
// group of boxes that share the kernel's compile-time shape.

struct PmeBox {
    PmeArgs a;
    TileArgs t;
    Cell cell;
};

// Resident blocks per SM of the multi-box gather (its run-time argument table
// costs registers over the one-box kernel's): 4 (64 registers).
#ifndef PINYB200_GATHER_BATCH_BLOCKS
#define PINYB200_GATHER_BATCH_BLOCKS 4
#endif

struct FftBox {
    const void *q;      // real grid (forward input, inverse output)
    void *spec;         // half spectrum
    const void *filt;   // influence function (FP32)
    const void *tw[3];  // twiddles per axis
    int Na, Nb, Nc;
    Cell cell;
    double alp;
    double *acc;
    int energy;
};

template <int NI, int TT>
__global__ void __launch_bounds__(256) spread_batch_kernel(const __grid_constant__ BoxTab<PmeBox> t)
{
    PINYB200_BOX_LOOP(t, i, vb, (spread_tile_c_body<NI, TT>(t.arg[i].a, t.arg[i].t, vb)));
}

template <typename R, int NI, int TT>
__global__ void __launch_bounds__(256, NI <= 8 ? PINYB200_GATHER_BATCH_BLOCKS : 1)
    gather_batch_kernel(const __grid_constant__ BoxTab<PmeBox> t)
{
    PINYB200_BOX_LOOP(t, i, vb, (gather_tile_c_body<R, NI, TT>(t.arg[i].a, t.arg[i].cell, t.arg[i].t, vb)));
}

template <typename R>
__global__ void __launch_bounds__(256) plane_fwd_batch_kernel(const __grid_constant__ BoxTab<FftBox> t)
{
    typedef typename Cplx<R>::T C2;
    PINYB200_BOX_LOOP(t, i, vb,
                      (plane_fwd_body<R>((const R *)t.arg[i].q, (C2 *)t.arg[i].spec, t.arg[i].Na, t.arg[i].Nb,
                                             t.arg[i].Nc, (const R *)t.arg[i].tw[0], (const R *)t.arg[i].tw[1], vb)));
}

template <typename R>
__global__ void __launch_bounds__(256) conv_c_batch_kernel(const __grid_constant__ BoxTab<FftBox> t)
{
    typedef typename Cplx<R>::T C2;
    PINYB200_BOX_LOOP(t, i, vb,
                      (conv_c_body<R>((C2 *)t.arg[i].spec, (const R *)t.arg[i].filt, t.arg[i].Na, t.arg[i].Nb,
                                          t.arg[i].Nc, (const R *)t.arg[i].tw[2], t.arg[i].cell, t.arg[i].alp,
                                          t.arg[i].acc, t.arg[i].energy, vb)));
}

template <typename R>
__global__ void __launch_bounds__(256) plane_inv_batch_kernel(const __grid_constant__ BoxTab<FftBox> t)
{
    typedef typename Cplx<R>::T C2;
    PINYB200_BOX_LOOP(t, i, vb,
                      (plane_inv_body<R>((const C2 *)t.arg[i].spec, (R *)t.arg[i].q, t.arg[i].Na, t.arg[i].Nb,
                                             t.arg[i].Nc, (const R *)t.arg[i].tw[0], (const R *)t.arg[i].tw[1], vb)));
}

// stage 0 spread, 1 gather for the boxes of one (order, tile edge) group
template <int NI, int TT>
static cudaError_t pme_batch_tiles(const std::vector<PmeBox> &bx, const std::vector<int> &P, int sm_count,
                                   cudaStream_t st, int stage)
{
    typedef float R;
    BoxTabBuilder<PmeBox> tb;
    for (size_t i = 0; i < bx.size(); i++) {
        const double work = (double)bx[i].a.nchrg * P[i];
        tb.add(bx[i], bx[i].t.ntile, P[i] * bx[i].t.nshare, work);
    }
    if (stage == 0) {
        const size_t ss = spread_smem<R, NI, TT>();
        return launch_tables(tb, (const void *)spread_batch_kernel<NI, TT>, 256, ss, sm_count,
                             [&](const BoxTab<PmeBox> &t, int g) { spread_batch_kernel<NI, TT><<<g, 256, ss, st>>>(t); });
    }
    const size_t sg = (size_t)TileGeom<NI, TT>::NPT * sizeof(R);
    return launch_tables(tb, (const void *)gather_batch_kernel<R, NI, TT>, 256, sg, sm_count,
                         [&](const BoxTab<PmeBox> &t, int g) { gather_batch_kernel<R, NI, TT><<<g, 256, sg, st>>>(t); });
}

template <int TT>
static cudaError_t pme_batch_tiles_n(int NI, const std::vector<PmeBox> &bx, const std::vector<int> &P, int sm_count,
                                     cudaStream_t st, int stage)
{
    switch (NI) {
    case 4: return pme_batch_tiles<4, TT>(bx, P, sm_count, st, stage);
    case 5: return pme_batch_tiles<5, TT>(bx, P, sm_count, st, stage);
    case 6: return pme_batch_tiles<6, TT>(bx, P, sm_count, st, stage);
    case 7: return pme_batch_tiles<7, TT>(bx, P, sm_count, st, stage);
    case 8: return pme_batch_tiles<8, TT>(bx, P, sm_count, st, stage);
    case 10: return pme_batch_tiles<10, TT>(bx, P, sm_count, st, stage);
    default: return cudaErrorInvalidValue;
    }
}

// stage 0 forward plane FFT, 1 c-axis FFT with the convolution, 2 inverse
// plane FFT for the boxes of one mesh of run-time lengths
static cudaError_t pme_batch_fft(const std::vector<FftBox> &bx, const std::vector<int> &P, int sm_count,
                                 cudaStream_t st, int stage)
{
    typedef float R;
    size_t sp = 0, ss = 0;
    BoxTabBuilder<FftBox> tb;
    for (size_t i = 0; i < bx.size(); i++) {
        sp = std::max(sp, pme_plane_smem(bx[i].Na, bx[i].Nb, false));
        ss = std::max(ss, pme_slab_smem(bx[i].Na, bx[i].Nc, false));
        const double work = (double)bx[i].Na * bx[i].Nb * bx[i].Nc * P[i];
        tb.add(bx[i], P[i] * (stage == 1 ? bx[i].Nb : bx[i].Nc), 1, work);
    }
    if (stage == 0)
        return launch_tables(tb, (const void *)plane_fwd_batch_kernel<R>, 256, sp, sm_count,
                             [&](const BoxTab<FftBox> &t, int g) { plane_fwd_batch_kernel<R><<<g, 256, sp, st>>>(t); });
    if (stage == 1)
        return launch_tables(tb, (const void *)conv_c_batch_kernel<R>, 256, ss, sm_count,
                             [&](const BoxTab<FftBox> &t, int g) { conv_c_batch_kernel<R><<<g, 256, ss, st>>>(t); });
    return launch_tables(tb, (const void *)plane_inv_batch_kernel<R>, 256, sp, sm_count,
                         [&](const BoxTab<FftBox> &t, int g) { plane_inv_batch_kernel<R><<<g, 256, sp, st>>>(t); });
}

static cudaError_t pme_batch_tiles_group(const std::pair<int, int> &key, const std::vector<PmeBox> &bx,
                                         const std::vector<int> &P, int sm_count, cudaStream_t st, int stage)
{
    return key.second == 8 ? pme_batch_tiles_n<8>(key.first, bx, P, sm_count, st, stage)
                           : pme_batch_tiles_n<16>(key.first, bx, P, sm_count, st, stage);
}

// Forward PME of many MIXED contexts on stream st, as launch_pme does for
// one whose grids are clear and charges binned: spread, transformed,
// convolved (energies and virials into each context's per-bead sums when
// `energy`), transformed back and gathered into each context's PME forces.
cudaError_t launch_pme_batch(const std::vector<pinyb200_ctx *> &box, const std::vector<Cell> &cells, bool energy,
                             int sm_count, cudaStream_t st)
{
    // groups: tiles by (order, tile edge), FFTs by mesh
    std::map<std::pair<int, int>, std::pair<std::vector<PmeBox>, std::vector<int>>> tiles;
    std::map<std::tuple<int, int, int>, std::pair<std::vector<FftBox>, std::vector<int>>> ffts;
    for (size_t i = 0; i < box.size(); i++) {
        pinyb200_ctx *c = box[i];
        if (c->sys.nchrg == 0 || c->sys.nktot == 0) continue;
        if (c->precision != PINYB200_MIXED) return cudaErrorInvalidValue;
        const Cell &cell = cells[i];
        const size_t G = (size_t)c->sys.ngrid[0] * c->sys.ngrid[1] * c->sys.ngrid[2];
        const cudaError_t ef = launch_filter(c, cell, st);
        if (ef != cudaSuccess) return ef;
        PmeBox pb;
        pb.a = pme_args_of(c);
        pb.t = tile_args_of(c, c->sys.n_interp, c->pme_tile);
        pb.cell = cell;
        auto &tg = tiles[std::make_pair(c->sys.n_interp, c->pme_tile)];
        tg.first.push_back(pb);
        tg.second.push_back(c->P);
        FftBox fb;
        fb.q = c->d_grid;
        fb.spec = c->d_spec;
        fb.filt = (const void *)((const double *)c->d_filter + G);
        fb.tw[0] = c->d_twiddle32;
        fb.tw[1] = c->d_twiddle32 + 2 * 256;
        fb.tw[2] = c->d_twiddle32 + 4 * 256;
        fb.Na = c->sys.ngrid[0];
        fb.Nb = c->sys.ngrid[1];
        fb.Nc = c->sys.ngrid[2];
        fb.cell = cell;
        fb.alp = c->alp_ewd;
        fb.acc = c->d_acc;
        fb.energy = energy ? 1 : 0;
        auto &fg = ffts[std::make_tuple(fb.Na, fb.Nb, fb.Nc)];
        fg.first.push_back(fb);
        fg.second.push_back(c->P);
    }
    cudaError_t err = cudaSuccess;
    for (auto &kv : tiles) {
        err = pme_batch_tiles_group(kv.first, kv.second.first, kv.second.second, sm_count, st, 0);
        if (err != cudaSuccess) break;
    }
    for (int stage = 0; stage < 3 && err == cudaSuccess; stage++)
        for (auto &kv : ffts) {
            const int Na = std::get<0>(kv.first), Nb = std::get<1>(kv.first), Nc = std::get<2>(kv.first);
            if (fft_fixed_edge(Na, Nb, Nc)) {
                std::vector<FftArgs> fx;
                for (const FftBox &b : kv.second.first) {
                    FftArgs f;
                    f.grid = const_cast<void *>(b.q);
                    f.spec = b.spec;
                    f.filt = b.filt;
                    f.tw = b.tw[0];
                    f.cell = b.cell;
                    f.alp = b.alp;
                    f.acc = b.acc;
                    f.energy = b.energy;
                    fx.push_back(f);
                }
                err = launch_fft_fixed_batch(Na, fx, kv.second.second, sm_count, st, stage);
            } else {
                err = pme_batch_fft(kv.second.first, kv.second.second, sm_count, st, stage);
            }
            if (err != cudaSuccess) break;
        }
    for (auto &kv : tiles) {
        if (err != cudaSuccess) break;
        err = pme_batch_tiles_group(kv.first, kv.second.first, kv.second.second, sm_count, st, 1);
    }
    return err;
}

}  // namespace pinyb200

namespace pinyb200 {

// ---------------------------------------------------------------------------
// Adjoint of the reciprocal-space term (parameter gradients).
//
// With u the adjoint of the raw site forces, Q_u(g) = sum_s q_s u_s . grad
// M_s(g) is spread, convolved with the same influence function as the charge
// grid (chi = theta * Q_u), and gathered; with phi the forward potential:
//   charge tangent dq:   dE += sum_s dq_s phi_s
//                        dF += -sum_s dq_s (u_s . grad phi_s + chi_s)
//   ghost position w:    dF += -sum_s q_s (w_s . grad chi_s + u_s^T (grad grad phi)_s w_s)
// (symmetry of the influence function moves the convolution onto Q_u).

// Second-derivative weights of the order-NI B-spline at offset f, PINY's
// index j = 1..NI: d2[j] = m[j] - 2 m[j-1] + m[j-2] with m of order NI-2.
template <typename R, int NI>
__device__ __forceinline__ void bspline_d2(R f, R *d2)
{
    R u[NI + 1], m[NI + 1];
#pragma unroll
    for (int j = 1; j <= NI; j++) u[j] = f + (R)(j - 1);
    m[0] = (R)0;
    m[1] = (R)1 - fabs(u[1] - (R)1);
    m[2] = (R)1 - fabs(u[2] - (R)1);
#pragma unroll
    for (int j = 3; j <= NI; j++) m[j] = (R)0;
#pragma unroll
    for (int nn = 3; nn <= NI - 2; nn++) {
        const R rn = (R)nn, rn1 = (R)1 / (R)(nn - 1);
#pragma unroll
        for (int j = nn; j >= 2; j--) m[j] = (u[j] * m[j] + (rn - u[j]) * m[j - 1]) * rn1;
        m[1] = u[1] * m[1] * rn1;
    }
#pragma unroll
    for (int j = 1; j <= NI; j++) d2[j] = m[j] - (R)2 * (j >= 2 ? m[j - 1] : (R)0) + (j >= 3 ? m[j - 2] : (R)0);
}

// u (or w) in scaled-grid units: t_d = N_d sum_alpha hi[d + 3 alpha] v_alpha.
__device__ __forceinline__ void scaled_vec(const PmeArgs &a, const Cell &cell, double vx, double vy, double vz,
                                           double *t)
{
    const int N[3] = {a.Na, a.Nb, a.Nc};
#pragma unroll
    for (int d = 0; d < 3; d++) t[d] = N[d] * (cell.hi[d] * vx + cell.hi[d + 3] * vy + cell.hi[d + 6] * vz);
}

// Q_u: one warp per record, lanes 8 a points x 4 b rows, FP32/FP64 atomics.
template <typename R, int NI>
__global__ void __launch_bounds__(256) pme_dipole_spread_kernel(const __grid_constant__ PmeArgs a,
                                                                const __grid_constant__ Cell cell,
                                                                const double *__restrict__ uT, R *__restrict__ grid2)
{
    constexpr int NTB = (NI + 3) / 4, NSA = (NI + 7) / 8;
    __shared__ __align__(16) PolyTab<R, NI> pt;
    if (NI > 8) pt.fill(true);
    Piece<R, NI <= 8 ? NI : 4> piece;
    piece.load(threadIdx.x & 7);
    __syncthreads();
    const int lane = threadIdx.x & 31, la8 = lane & 7, lb4 = lane >> 3;
    const long long nrec = (long long)a.nchrg * a.P;
    const size_t G = (size_t)a.Na * a.Nb * a.Nc;
    for (long long idx = ((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5; idx < nrec;
         idx += ((long long)gridDim.x * blockDim.x) >> 5) {
        const int b = (int)(idx % a.P);
        const int4 h = a.rhead[idx];
        const typename Vec4<R>::T fr = load_frac<R>(a.rw, (int)idx);
        const int at = h.x;
        const double ux = uT[(3 * (size_t)at + 0) * a.P + b], uy = uT[(3 * (size_t)at + 1) * a.P + b],
                     uz = uT[(3 * (size_t)at + 2) * a.P + b];
        if (ux == 0.0 && uy == 0.0 && uz == 0.0) continue;
        double ut[3];
        scaled_vec(a, cell, ux, uy, uz, ut);
        R wa[NSA], da[NSA], mb[NTB], db[NTB], mcl = 0, dcl = 0;
        if constexpr (NI <= 8) {
            R wb, eb;
            piece.both(fr.x, wa[0], da[0]);
            piece.both(fr.y, wb, eb);
            piece.both(fr.z, mcl, dcl);
#pragma unroll
            for (int i = 0; i < NTB; i++) {
                mb[i] = __shfl_sync(0xffffffffu, wb, (lb4 + 4 * i) & 7);
                db[i] = __shfl_sync(0xffffffffu, eb, (lb4 + 4 * i) & 7);
            }
        } else {
#pragma unroll
            for (int s = 0; s < NSA; s++) {
                const int p = NI - 1 - min(la8 + 8 * s, NI - 1);
                wa[s] = poly_eval<R, NI>(pt.m[p], fr.x);
                da[s] = poly_eval<R, NI>(pt.dm[p], fr.x);
            }
#pragma unroll
            for (int i = 0; i < NTB; i++) {
                const int p = NI - 1 - min(lb4 + 4 * i, NI - 1);
                mb[i] = poly_eval<R, NI>(pt.m[p], fr.y);
                db[i] = poly_eval<R, NI>(pt.dm[p], fr.y);
            }
            const int p = NI - 1 - min(lane, NI - 1);
            mcl = poly_eval<R, NI>(pt.m[p], fr.z);
            dcl = poly_eval<R, NI>(pt.dm[p], fr.z);
        }
        const R q = fr.w;
        R *g = grid2 + (size_t)b * G;
#pragma unroll
        for (int tc = 0; tc < NI; tc++) {
            const R mc = __shfl_sync(0xffffffffu, mcl, tc), dc = __shfl_sync(0xffffffffu, dcl, tc);
            R *pc = g + (size_t)wrapi(h.w + tc, a.Nc) * a.Nb * a.Na;
#pragma unroll
            for (int s = 0; s < NSA; s++) {
                if (la8 + 8 * s >= NI) continue;
                const R ma = q * wa[s], ga = q * da[s];
                const R cm = (R)ut[0] * ga * mc + (R)ut[2] * ma * dc, cd = (R)ut[1] * ma * mc;
                const int ia = wrapi(h.y + la8 + 8 * s, a.Na);
#pragma unroll
                for (int i = 0; i < NTB; i++)
                    if (lb4 + 4 * i < NI)
                        atomicAdd(pc + (size_t)wrapi(h.z + lb4 + 4 * i, a.Nb) * a.Na + ia, cm * mb[i] + cd * db[i]);
            }
        }
    }
}

// Sums of one potential at one record over this lane's a points: value and
// derivatives along a, b, c; phi(tc, tb, ta) reads the potential.  A plane's b
// sums are in R, the sum over planes is compensated (Kahan's, four operations a
// term: as good as FP64, whose conversions take 5 us more of 530 at 1024 TIP4P/F
// x 16), everything beyond it in FP64.
template <typename R>
struct KahanSum {
    R s = 0, c = 0;
    __device__ __forceinline__ void add(R a, R b)  // a b
    {
        if constexpr (sizeof(R) == 8) {
            s += a * b;
        } else {
            const R y = a * b - c, t = s + y;
            c = (t - s) - y;
            s = t;
        }
    }
    __device__ __forceinline__ double value() const { return (double)s - (double)c; }
};
template <typename R, int NI, typename PHI>
__device__ __forceinline__ void adjoint_lane(PHI phi, const LaneW<R, NI, true> &lw, int l8, double *s)
{
    s[0] = s[1] = s[2] = s[3] = 0.0;
#pragma unroll
    for (int j = 0; j < (NI > 8 ? 2 : 1); j++) {
        const int ta = l8 + 8 * j;
        if (ta >= NI) break;
        KahanSum<R> smm, sdm, smd;
#pragma unroll
        for (int tc = 0; tc < NI; tc++) {
            R um = 0, ud = 0;
#pragma unroll
            for (int tb = 0; tb < NI; tb++) {
                const R p = phi(tc, tb, ta);
                um += lw.mb[tb] * p;
                ud += lw.db[tb] * p;
            }
            smm.add(lw.mc[tc], um);
            sdm.add(lw.mc[tc], ud);
            smd.add(lw.dc[tc], um);
        }
        const double wa = j ? lw.wa1 : lw.wa0, da = j ? lw.da1 : lw.da0;
        s[0] += wa * smm.value();
        s[1] += da * smm.value();
        s[2] += wa * sdm.value();
        s[3] += wa * smd.value();
    }
}

// Second derivatives aa, bb, cc, ab, ac, bc of one potential at one record,
// this lane's share, in FP64; the 8 lanes of the group call it together.
template <typename R, int NI, typename PHI>
__device__ __forceinline__ void adjoint_hessian(PHI phi, const Piece<R, NI <= 8 ? NI : 4> &piece,
                                                const typename Vec4<R>::T &fr, const LaneW<R, NI, true> &lw, int l8,
                                                double *hs)
{
    R d2a[2] = {0, 0}, d2b[NI], d2c[NI];
    if constexpr (NI <= 8) {
        const unsigned mask = 0xffu << (threadIdx.x & 24);
        d2a[0] = piece.second(fr.x);
        const R sb = piece.second(fr.y), sc = piece.second(fr.z);
#pragma unroll
        for (int k = 0; k < NI; k++) {
            d2b[k] = __shfl_sync(mask, sb, k, 8);
            d2c[k] = __shfl_sync(mask, sc, k, 8);
        }
    } else {
        R d2[NI + 1];  // grid order: point lo + t carries index NI - t
        bspline_d2<R, NI>(fr.y, d2);
#pragma unroll
        for (int k = 0; k < NI; k++) d2b[k] = d2[NI - k];
        bspline_d2<R, NI>(fr.z, d2);
#pragma unroll
        for (int k = 0; k < NI; k++) d2c[k] = d2[NI - k];
        bspline_d2<R, NI>(fr.x, d2);
#pragma unroll
        for (int k = 0; k < NI; k++) {
            if (k == l8) d2a[0] = d2[NI - k];
            if (k == l8 + 8) d2a[1] = d2[NI - k];
        }
    }
#pragma unroll
    for (int j = 0; j < (NI > 8 ? 2 : 1); j++) {
        const int ta = l8 + 8 * j;
        if (ta >= NI) break;
        double smm = 0, s2m = 0, sm2 = 0, sdm = 0, smd = 0, sdd = 0;  // b and c weights
#pragma unroll
        for (int tc = 0; tc < NI; tc++) {
            double um = 0, ud = 0, u2 = 0;
#pragma unroll
            for (int tb = 0; tb < NI; tb++) {
                const double p = (double)phi(tc, tb, ta);
                um += (double)lw.mb[tb] * p;
                ud += (double)lw.db[tb] * p;
                u2 += (double)d2b[tb] * p;
            }
            smm += (double)lw.mc[tc] * um;
            s2m += (double)lw.mc[tc] * u2;
            sm2 += (double)d2c[tc] * um;
            sdm += (double)lw.mc[tc] * ud;
            smd += (double)lw.dc[tc] * um;
            sdd += (double)lw.dc[tc] * ud;
        }
        const double wa = j ? lw.wa1 : lw.wa0, da = j ? lw.da1 : lw.da0;
        hs[0] += (double)d2a[j] * smm;
        hs[1] += wa * s2m;
        hs[2] += wa * sm2;
        hs[3] += da * sdm;
        hs[4] += da * smd;
        hs[5] += wa * sdd;
    }
}

// Gathers phi, grad phi, chi, grad chi (and grad grad phi at sites with a
// ghost tangent) per record and contracts them with every channel.  As the
// gather: a block per (tile, bead, share), the tile's potential in shared
// memory (phi, then chi in its place), 8 lanes a record.  The contraction is
// linear, so each potential's terms are added on their own.  Bound:
// shared-memory reads, 128 a record and lane.  1024 TIP4P/F x 16 beads, 32^3,
// FP32: 277 us as one thread per record reading global memory, 127 here.
template <typename R, int NI, int TT>
__global__ void __launch_bounds__(256, sizeof(R) == 4 && NI <= 8 ? 2 : 1) pme_adjoint_gather_kernel(const __grid_constant__ PmeArgs a,
                                                                 const __grid_constant__ Cell cell,
                                                                 const __grid_constant__ TileArgs t,
                                                                 const __grid_constant__ GradArgs g,
                                                                 const R *__restrict__ phi, const R *__restrict__ chi)
{
    typedef TileGeom<NI, TT> TG;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    R *tl = (R *)smem_raw;
    __shared__ __align__(16) PolyTab<R, NI> pt;
    __shared__ double sh[2 * PINYB200_MAX_TAN];
    if (NI > 8) pt.fill(true);
    Piece<R, NI <= 8 ? NI : 4> piece;
    piece.load(threadIdx.x & 7);
    double acc[2 * PINYB200_MAX_TAN];
    for (int k = 0; k < 2 * g.K; k++) acc[k] = 0.0;
    const size_t G = (size_t)a.Na * a.Nb * a.Nc;
    const int l8 = threadIdx.x & 7, grp = threadIdx.x >> 3, ngrp = blockDim.x >> 3;
    const int lane = threadIdx.x & 31;
    const int tile = blockIdx.x, b0 = blockIdx.y / t.nshare, z = blockIdx.y - b0 * t.nshare;
    const int ta0 = (tile % t.nta) * TG::T, tb0 = ((tile / t.nta) % t.ntb) * TG::T, tc0 = (tile / (t.nta * t.ntb)) * TG::T;
    const int n = min(t.cnt[b0 * t.ntile + tile], t.cap);
    const int *list = t.bin + ((size_t)b0 * t.ntile + tile) * t.cap;
    const int nov = t.cnt[a.P * t.ntile];
    const int gid = blockIdx.y * gridDim.x + blockIdx.x, nblk = gridDim.x * gridDim.y;
    bool any_w = false;
    for (int k = 0; k < g.K; k++) any_w |= g.ch[k].w != nullptr;

    for (int which = 0; which < 2; which++) {  // 0 phi, 1 chi
        const R *pot = which ? chi : phi;
        if (n > z * ngrp) load_tile<R, TG>(tl, pot + (size_t)b0 * G, a.Na, a.Nb, a.Nc, ta0, tb0, tc0);
        __syncthreads();
        // one record by the 8 lanes of a group; every lane of the warp calls it
        auto record = [&](bool act, int idx, bool binned) {
            const int b = idx % a.P;
            int4 h = make_int4(0, 0, 0, 0);
            typename Vec4<R>::T fr = {};
            if (act) {
                h = a.rhead[idx];
                fr = load_frac<R>(a.rw, idx);
            }
            LaneW<R, NI, true> lw;
            gather_weights<R, NI>(pt, piece, fr, l8, lw);
            double s[4] = {0, 0, 0, 0}, hs[6] = {0, 0, 0, 0, 0, 0};
            bool need_h = false;  // a ghost-position tangent at this site
            if (act && any_w)
                for (int k = 0; k < g.K; k++)
                    if (g.ch[k].w) {
                        const double *wv = g.ch[k].w + (3 * (size_t)h.x) * a.P + b;
                        need_h |= wv[0] != 0.0 || wv[a.P] != 0.0 || wv[2 * a.P] != 0.0;
                    }
            const bool hess = need_h && which == 0;
            const int oa = h.y - ta0, ob = h.z - tb0, oc = h.w - tc0;
            if (act && binned && oa >= 0 && oa < TG::T && ob >= 0 && ob < TG::T && oc >= 0 && oc < TG::T) {
                const R *base = tl + (oc * TG::E + ob) * TG::PA + oa;
                auto get = [&](int tc, int tb, int ta) { return base[(tc * TG::E + tb) * TG::PA + ta]; };
                adjoint_lane<R, NI>(get, lw, l8, s);
                if (hess) adjoint_hessian<R, NI>(get, piece, fr, lw, l8, hs);
            } else if (act) {
                const R *gb = pot + (size_t)b * G;
                auto get = [&](int tc, int tb, int ta) {
                    return gb[((size_t)wrapi(h.w + tc, a.Nc) * a.Nb + wrapi(h.z + tb, a.Nb)) * a.Na +
                              wrapi(h.y + ta, a.Na)];
                };
                adjoint_lane<R, NI>(get, lw, l8, s);
                if (hess) adjoint_hessian<R, NI>(get, piece, fr, lw, l8, hs);
            }
#pragma unroll
            for (int o = 4; o >= 1; o >>= 1) {
#pragma unroll
                for (int k = 0; k < 4; k++) s[k] += __shfl_xor_sync(0xffffffffu, s[k], o);
            }
            if (__any_sync(0xffffffffu, hess)) {
#pragma unroll
                for (int o = 4; o >= 1; o >>= 1) {
#pragma unroll
                    for (int k = 0; k < 6; k++) hs[k] += __shfl_xor_sync(0xffffffffu, hs[k], o);
                }
            }
            if (!act || l8 != 0) return;
            const int at = h.x;
            double ut[3] = {0, 0, 0};
            if (which == 0)
                scaled_vec(a, cell, g.uT[(3 * (size_t)at + 0) * a.P + b], g.uT[(3 * (size_t)at + 1) * a.P + b],
                           g.uT[(3 * (size_t)at + 2) * a.P + b], ut);
            const double q = a.charge[at];
            for (int k = 0; k < g.K; k++) {
                const GradChan &ch = g.ch[k];
                if (ch.dq) {
                    const double dq = ch.dq[at];
                    if (dq != 0.0) {
                        if (which == 0) {
                            acc[2 * k] += dq * s[0] / (double)a.P;
                            acc[2 * k + 1] -= dq * (ut[0] * s[1] + ut[1] * s[2] + ut[2] * s[3]);
                        } else {
                            acc[2 * k + 1] -= dq * s[0];
                        }
                    }
                }
                if (ch.w && need_h) {
                    double wt[3];
                    scaled_vec(a, cell, ch.w[(3 * (size_t)at) * a.P + b], ch.w[(3 * (size_t)at + 1) * a.P + b],
                               ch.w[(3 * (size_t)at + 2) * a.P + b], wt);
                    const double v = which ? wt[0] * s[1] + wt[1] * s[2] + wt[2] * s[3]
                                           : ut[0] * (hs[0] * wt[0] + hs[3] * wt[1] + hs[4] * wt[2]) +
                                                 ut[1] * (hs[3] * wt[0] + hs[1] * wt[1] + hs[5] * wt[2]) +
                                                 ut[2] * (hs[4] * wt[0] + hs[5] * wt[1] + hs[2] * wt[2]);
                    acc[2 * k + 1] -= q * v;
                }
            }
        };
        for (int e0 = ngrp * z; e0 < n; e0 += ngrp * t.nshare) {
            const int e = e0 + grp;
            record(e < n, e < n ? list[e] : 0, true);
        }
        for (int e0 = gid * ngrp; e0 < nov; e0 += nblk * ngrp) {
            const int e = e0 + grp;
            record(e < nov, e < nov ? t.ovf[e] : 0, false);
        }
        __syncthreads();
    }
    // block flush: warp sums (lanes other than a group's first hold zeros)
    for (int i = threadIdx.x; i < 2 * g.K; i += blockDim.x) sh[i] = 0.0;
    __syncthreads();
    for (int i = 0; i < 2 * g.K; i++) {
        const double v = acc[i];
        if (!__any_sync(0xffffffffu, v != 0.0)) continue;
        const double w = warp_sum(v);
        if (lane == 0) atomicAdd(&sh[i], w);
    }
    __syncthreads();
    for (int i = threadIdx.x; i < 2 * g.K; i += blockDim.x)
        if (sh[i] != 0.0) atomicAdd(&g.gacc[i], sh[i]);
}

template <typename R, int NI, int TT>
static cudaError_t launch_adjoint_gather(pinyb200_ctx *c, const PmeArgs &a, const Cell &cell, const GradArgs &g)
{
    TileArgs t = tile_args_of(c, NI, TT);
    // two passes of loads and a wide inner loop: more blocks per bin than the gather
    const int bins = t.ntile * a.P;
    t.nshare = std::max(1, std::min(8, (4 * c->sm_count + bins - 1) / bins));
    const size_t st = (size_t)TileGeom<NI, TT>::NPT * sizeof(R);
    cudaError_t err = smem_optin((const void *)pme_adjoint_gather_kernel<R, NI, TT>, (int)st);
    if (err != cudaSuccess) return err;
    pme_adjoint_gather_kernel<R, NI, TT><<<dim3((unsigned)t.ntile, (unsigned)(a.P * t.nshare)), 256, st, c->stream>>>(
        a, cell, t, g, (const R *)c->d_grid, (const R *)c->grad.d_grid2);
    return cudaGetLastError();
}

template <typename R, int NI>
static cudaError_t launch_pme_adjoint_t(pinyb200_ctx *c, const Cell &cell, const GradArgs &g)
{
    typedef typename Cplx<R>::T C2;
    PmeArgs a = pme_args_of(c);
    a.grid = c->grad.d_grid2;
    const size_t G = (size_t)a.Na * a.Nb * a.Nc;
    const bool f64 = sizeof(R) == 8;
    cudaError_t err = cudaMemsetAsync(c->grad.d_grid2, 0, sizeof(R) * G * c->P, c->stream);
    if (err != cudaSuccess) return err;
    const long long nrec = (long long)a.nchrg * a.P;
    long long blocks = (nrec * 32 + 255) / 256;
    if (blocks > (long long)c->sm_count * 16) blocks = (long long)c->sm_count * 16;
    pme_dipole_spread_kernel<R, NI><<<(unsigned)blocks, 256, 0, c->stream>>>(a, cell, g.uT, (R *)c->grad.d_grid2);
    const R *twbase = (const R *)(f64 ? (const void *)c->d_twiddle64 : (const void *)c->d_twiddle32);
    const R *tw[3] = {twbase, twbase + 2 * 256, twbase + 4 * 256};
    const size_t sp = pme_plane_smem(a.Na, a.Nb, f64), ss = pme_slab_smem(a.Na, a.Nc, f64);
    C2 *spec = (C2 *)c->d_spec;
    const R *filt = f64 ? (const R *)c->d_filter : (const R *)((const double *)c->d_filter + G);
    err = launch_fft<R>(c, a, cell, spec, filt, tw, sp, ss, false);
    if (err != cudaSuccess) return err;
    return c->pme_tile == 8 ? launch_adjoint_gather<R, NI, 8>(c, a, cell, g) : launch_adjoint_gather<R, NI, 16>(c, a, cell, g);
}

template <typename R>
static cudaError_t launch_pme_adjoint_r(pinyb200_ctx *c, const Cell &cell, const GradArgs &g)
{
    switch (c->sys.n_interp) {
    case 4: return launch_pme_adjoint_t<R, 4>(c, cell, g);
    case 5: return launch_pme_adjoint_t<R, 5>(c, cell, g);
    case 6: return launch_pme_adjoint_t<R, 6>(c, cell, g);
    case 7: return launch_pme_adjoint_t<R, 7>(c, cell, g);
    case 8: return launch_pme_adjoint_t<R, 8>(c, cell, g);
    case 10: return launch_pme_adjoint_t<R, 10>(c, cell, g);
    default: return cudaErrorInvalidValue;
    }
}

cudaError_t launch_pme_adjoint(pinyb200_ctx *c, const Cell &cell, const GradArgs &g)
{
    if (c->sys.nchrg == 0 || c->sys.nktot == 0 || !c->grad.d_grid2) return cudaSuccess;
    if (c->precision == PINYB200_FP64) return launch_pme_adjoint_r<double>(c, cell, g);
    return launch_pme_adjoint_r<float>(c, cell, g);
}

}  // namespace pinyb200
