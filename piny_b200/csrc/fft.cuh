// Batched 3D FFTs of the PME mesh for cubic meshes of compile-time edge.
//
// The charge grid is real, so a plane's two-dimensional transform is done on
// rows packed in pairs: row 2r as the real and row 2r+1 as the imaginary part
// of one complex row, an N/2 x N complex plane in shared memory.  Its
// transform W(m, k) (m over the N/2 packed rows, k along a) holds the
// transforms E and O of the even and odd rows,
//   E = (W(m, k) + conj W(-m, -k)) / 2,  O = (W(m, k) - conj W(-m, -k)) / 2i,
// and F(m, k) = E + w^m O, F(m + N/2, k) = E - w^m O with w = exp(2 pi i / N)
// are the plane's half spectrum.  The inverse packs W = E + i O from
// E = F(m) + F(m + N/2), O = w^-m (F(m) - F(m + N/2)) and reads rows 2r and
// 2r+1 off as real and imaginary part.  Against one complex line per real
// row this is half the shared memory and half the butterflies.
//
// Lines of length N = R0 R1 (both at most 16) take two passes: decimation in
// frequency forwards, the transposed passes backwards.  Every butterfly reads
// and writes the same places, so a pass needs one barrier and no second
// buffer; the forward result stands in digit-reversed order (frequency
// k = u0 + R0 u1 at place u0 R1 + u1), which the untangling step and the
// convolution index for and the inverse passes undo.  First passes read
// global memory and last passes write it directly; the convolution's second
// forward pass, filter and first inverse pass stay in registers.
//
// Bound: the L2 traffic of grid and spectrum (each read and written once per
// kernel); figures at launch_fft_n.
#pragma once

#include "boxtab.cuh"
#include "common.cuh"

namespace pinyb200 {

// cos and sin of 2 pi m / n at compile time (Taylor series on [0, pi/4]).
__host__ __device__ constexpr double ct_series(double x, bool sine)
{
    double t = sine ? x : 1.0, s = t;
    for (int k = sine ? 2 : 1; k < 28; k += 2) {
        t = -t * x * x / (double)(k * (k + 1));
        s += t;
    }
    return s;
}
__host__ __device__ constexpr double ct_cos(int m, int n)
{
    m = ((m % n) + n) % n;
    if (2 * m > n) m = n - m;
    bool neg = false;
    double num = 2.0 * m;  // the angle in units of pi / n
    if (4 * m > n) {
        num = (double)n - num;
        neg = true;
    }
    constexpr double pi = 3.14159265358979323846;
    const double x = num * pi / n;
    const double v = 4.0 * num <= (double)n ? ct_series(x, false) : ct_series(((double)n / 2.0 - num) * pi / n, true);
    return neg ? -v : v;
}
// sin(2 pi m / n) = cos(2 pi (m / n - 1 / 4))
__host__ __device__ constexpr double ct_sin(int m, int n) { return ct_cos(4 * m - n, 4 * n); }

template <typename C2, typename R>
__device__ __forceinline__ C2 cmul(const C2 &a, R wr, R wi)
{
    C2 c;
    c.x = a.x * wr - a.y * wi;
    c.y = a.x * wi + a.y * wr;
    return c;
}

// v *= exp(SIGN 2 pi i M / N) for compile-time M, N.
template <typename R, int M, int N, int SIGN, typename C2>
__device__ __forceinline__ void rot(C2 &v)
{
    constexpr int m = M % N;
    if constexpr (m == 0) {
    } else if constexpr (2 * m == N) {
        v.x = -v.x;
        v.y = -v.y;
    } else if constexpr (4 * m == N || 4 * m == 3 * N) {
        constexpr R s = (R)(4 * m == N ? SIGN : -SIGN);
        const R x = v.x;
        v.x = -s * v.y;
        v.y = s * x;
    } else {
        constexpr R wr = (R)ct_cos(m, N), wi = (R)(SIGN * ct_sin(m, N));
        v = cmul(v, wr, wi);
    }
}

// RAD-point DFT in registers, exp(SIGN 2 pi i n k / RAD): 2, 3, 4, 5 points
// directly, 6, 8, 9, 10, 12, 16 as two smaller ones.
__host__ __device__ constexpr int dft_split(int rad)
{
    return rad == 6 ? 2 : rad == 8 ? 2 : rad == 9 ? 3 : rad == 10 ? 2 : rad == 12 ? 3 : rad == 16 ? 4 : 1;
}
template <typename R, int RAD, int SIGN>
__device__ __forceinline__ void dft(typename Cplx<R>::T *v);

// The first stage of a composite radix, from column N2 on: A-point DFTs over
// n = Q n1 + N2, rotated, into w[k1 Q + N2].
template <typename R, int RAD, int SIGN, int N2, int K1, typename C2>
__device__ __forceinline__ void dft_rot_col(C2 *t, C2 *w)
{
    constexpr int A = dft_split(RAD), Q = RAD / A;
    rot<R, K1 * N2, RAD, SIGN>(t[K1]);
    w[K1 * Q + N2] = t[K1];
    if constexpr (K1 + 1 < A) dft_rot_col<R, RAD, SIGN, N2, K1 + 1>(t, w);
}
template <typename R, int RAD, int SIGN, int N2>
__device__ __forceinline__ void dft_cols(const typename Cplx<R>::T *v, typename Cplx<R>::T *w)
{
    constexpr int A = dft_split(RAD), Q = RAD / A;
    typename Cplx<R>::T t[A];
#pragma unroll
    for (int n1 = 0; n1 < A; n1++) t[n1] = v[Q * n1 + N2];
    dft<R, A, SIGN>(t);
    dft_rot_col<R, RAD, SIGN, N2, 0>(t, w);
    if constexpr (N2 + 1 < Q) dft_cols<R, RAD, SIGN, N2 + 1>(v, w);
}

template <typename R, int RAD, int SIGN>
__device__ __forceinline__ void dft(typename Cplx<R>::T *v)
{
    typedef typename Cplx<R>::T C2;
    constexpr R s = (R)SIGN;
    if constexpr (RAD == 1) {
    } else if constexpr (RAD == 2) {
        const C2 a = v[0], b = v[1];
        v[0].x = a.x + b.x;
        v[0].y = a.y + b.y;
        v[1].x = a.x - b.x;
        v[1].y = a.y - b.y;
    } else if constexpr (RAD == 3) {
        constexpr R h = (R)0.5, q = s * (R)ct_sin(1, 3);
        const C2 t = {v[1].x + v[2].x, v[1].y + v[2].y}, d = {q * (v[1].x - v[2].x), q * (v[1].y - v[2].y)};
        const C2 a = {v[0].x - h * t.x, v[0].y - h * t.y};
        v[0].x += t.x;
        v[0].y += t.y;
        v[1].x = a.x - d.y;
        v[1].y = a.y + d.x;
        v[2].x = a.x + d.y;
        v[2].y = a.y - d.x;
    } else if constexpr (RAD == 4) {
        const C2 t0 = {v[0].x + v[2].x, v[0].y + v[2].y}, t1 = {v[0].x - v[2].x, v[0].y - v[2].y};
        const C2 t2 = {v[1].x + v[3].x, v[1].y + v[3].y};
        const C2 t3 = {-s * (v[1].y - v[3].y), s * (v[1].x - v[3].x)};
        v[0].x = t0.x + t2.x;
        v[0].y = t0.y + t2.y;
        v[2].x = t0.x - t2.x;
        v[2].y = t0.y - t2.y;
        v[1].x = t1.x + t3.x;
        v[1].y = t1.y + t3.y;
        v[3].x = t1.x - t3.x;
        v[3].y = t1.y - t3.y;
    } else if constexpr (RAD == 5) {
        constexpr R c1 = (R)ct_cos(1, 5), c2 = (R)ct_cos(2, 5), s1 = s * (R)ct_sin(1, 5), s2 = s * (R)ct_sin(2, 5);
        const C2 t1 = {v[1].x + v[4].x, v[1].y + v[4].y}, t2 = {v[2].x + v[3].x, v[2].y + v[3].y};
        const C2 t3 = {v[1].x - v[4].x, v[1].y - v[4].y}, t4 = {v[2].x - v[3].x, v[2].y - v[3].y};
        const C2 a1 = {v[0].x + c1 * t1.x + c2 * t2.x, v[0].y + c1 * t1.y + c2 * t2.y};
        const C2 a2 = {v[0].x + c2 * t1.x + c1 * t2.x, v[0].y + c2 * t1.y + c1 * t2.y};
        const C2 b1 = {s1 * t3.x + s2 * t4.x, s1 * t3.y + s2 * t4.y};
        const C2 b2 = {s2 * t3.x - s1 * t4.x, s2 * t3.y - s1 * t4.y};
        v[0].x += t1.x + t2.x;
        v[0].y += t1.y + t2.y;
        v[1] = C2{a1.x - b1.y, a1.y + b1.x};
        v[4] = C2{a1.x + b1.y, a1.y - b1.x};
        v[2] = C2{a2.x - b2.y, a2.y + b2.x};
        v[3] = C2{a2.x + b2.y, a2.y - b2.x};
    } else {
        // n = Q n1 + n2, k = k1 + A k2
        constexpr int A = dft_split(RAD), Q = RAD / A;
        static_assert(A > 1, "radix not built");
        C2 w[RAD];  // w[k1 * Q + n2]
        dft_cols<R, RAD, SIGN, 0>(v, w);
#pragma unroll
        for (int k1 = 0; k1 < A; k1++) {
            dft<R, Q, SIGN>(w + k1 * Q);
#pragma unroll
            for (int k2 = 0; k2 < Q; k2++) v[k1 + A * k2] = w[k1 * Q + k2];
        }
    }
}

// The two passes of a line of length N: N = R0 R1, R0 <= R1 <= 16.
__host__ __device__ constexpr bool radix_built(int r)
{
    return (r >= 2 && r <= 6) || r == 8 || r == 9 || r == 10 || r == 12 || r == 16;
}
__host__ __device__ constexpr int fft_r0(int n)
{
    int best = 0;
    for (int r = 2; r * r <= n; r++)
        if (n % r == 0 && radix_built(r) && radix_built(n / r)) best = r;
    return best;
}
template <int N>
struct FftPlan {
    static constexpr int R0 = fft_r0(N), R1 = N / R0;
    static_assert(R0 > 0, "length not built");
    static constexpr int S = R1 | 1;  // places u0 S + u1: an odd stride keeps k-ordered reads off one bank
    static constexpr int W = R0 * S;  // places of a line
    // place of frequency k, and of the natural index a of the other pass's columns
    static __device__ __forceinline__ int place(int k) { return (k % R0) * S + k / R0; }
    static __device__ __forceinline__ int column(int a) { return (a / R1) * S + a % R1; }
};

template <int N>
struct FftGeom {
    typedef FftPlan<N> PA;      // along a (and c)
    typedef FftPlan<N / 2> PB;  // along the packed b rows
    static constexpr int H = N / 2, NH = N / 2 + 1;
    static constexpr int LS = PA::W | 1;          // row stride of the packed plane
    static constexpr int ROWS = PB::R0 * PB::R1;  // = H; the b passes keep rows unpadded
    static constexpr int LC = NH | 1;             // row stride of a slab
    static constexpr int PLANE_T = N >= 48 ? 256 : (N >= 24 ? 128 : 96);
    // slab threads: the larger pass in whole rounds of at most 320 threads
    static constexpr int CI = NH * (PA::R1 > PA::R0 ? PA::R1 : PA::R0);
    static constexpr int CROUNDS = (CI + 319) / 320;
    static constexpr int CONV_T = ((CI + CROUNDS - 1) / CROUNDS + 31) / 32 * 32;
    static constexpr int MAXRAD = PA::R1 > PB::R1 ? PA::R1 : PB::R1;
};
// register budget per thread the kernels are compiled for, as resident
// blocks: radix-10 FP32 butterflies fit 64 registers, radix 12 and 16 want
// 96; FP64 doubles both
template <typename R, int N>
__host__ __device__ constexpr int fft_blocks(int threads, bool multi_box)
{
    const int regs = (sizeof(R) == 8 ? 128 : (FftGeom<N>::MAXRAD > 10 ? 96 : 64)) + (multi_box ? 16 : 0);
    const int b = 65536 / (regs * threads);
    return b < 1 ? 1 : b;
}

template <typename R, int N>
constexpr size_t fft_plane_smem()
{
    return sizeof(typename Cplx<R>::T) * ((size_t)FftGeom<N>::H * FftGeom<N>::LS + N);
}
template <typename R, int N>
constexpr size_t fft_slab_smem()
{
    return sizeof(typename Cplx<R>::T) * ((size_t)N * FftGeom<N>::LC + N);
}

// Arguments of one box's transforms.
struct FftArgs {
    void *grid;        // real [P][N][N][N]: charges in, potential out
    void *spec;        // half spectrum [P][N][N][N/2+1]
    const void *filt;  // influence function [N][N][N]
    const void *tw;    // cos, sin of 2 pi m / N
    Cell cell;
    double alp;
    double *acc;
    int energy;
};

// One pass over the packed rows' columns (a places), and over the rows.
template <typename R, int N, int SIGN>
__device__ __forceinline__ void fft_pass_b(typename Cplx<R>::T *pl, const typename Cplx<R>::T *tw)
{
    typedef typename Cplx<R>::T C2;
    typedef FftGeom<N> G;
    typedef typename G::PA PA;
    typedef typename G::PB PB;
    auto outer = [&]() {
        for (int i = threadIdx.x; i < N * PB::R1; i += blockDim.x) {
            const int j = i / N;
            C2 *p = pl + j * G::LS + PA::column(i - j * N);
            C2 v[PB::R0];
#pragma unroll
            for (int t = 0; t < PB::R0; t++) {
                v[t] = p[t * PB::R1 * G::LS];
                if (SIGN < 0 && t > 0) {
                    const C2 w = tw[2 * j * t];
                    v[t] = cmul(v[t], w.x, -w.y);
                }
            }
            dft<R, PB::R0, SIGN>(v);
#pragma unroll
            for (int u = 0; u < PB::R0; u++) {
                if (SIGN > 0 && u > 0) {
                    const C2 w = tw[2 * j * u];
                    v[u] = cmul(v[u], w.x, w.y);
                }
                p[u * PB::R1 * G::LS] = v[u];
            }
        }
    };
    auto inner = [&]() {
        for (int i = threadIdx.x; i < N * PB::R0; i += blockDim.x) {
            const int s = i / N;
            C2 *p = pl + s * PB::R1 * G::LS + PA::column(i - s * N);
            C2 v[PB::R1];
#pragma unroll
            for (int t = 0; t < PB::R1; t++) v[t] = p[t * G::LS];
            dft<R, PB::R1, SIGN>(v);
#pragma unroll
            for (int t = 0; t < PB::R1; t++) p[t * G::LS] = v[t];
        }
    };
    if (SIGN > 0) outer();
    else inner();
    __syncthreads();
    if (SIGN > 0) inner();
    else outer();
    __syncthreads();
}

// The contiguous pass along a: R1 neighbouring places of one row.
template <typename R, int N, int SIGN>
__device__ __forceinline__ void fft_pass_a_inner(typename Cplx<R>::T *pl)
{
    typedef typename Cplx<R>::T C2;
    typedef FftGeom<N> G;
    typedef typename G::PA PA;
    for (int i = threadIdx.x; i < G::H * PA::R0; i += blockDim.x) {
        const int s = i / G::H, l = i - s * G::H;
        C2 *p = pl + l * G::LS + s * PA::S;
        C2 v[PA::R1];
#pragma unroll
        for (int t = 0; t < PA::R1; t++) v[t] = p[t];
        dft<R, PA::R1, SIGN>(v);
#pragma unroll
        for (int t = 0; t < PA::R1; t++) p[t] = v[t];
    }
    __syncthreads();
}

template <typename R, int N>
__device__ __forceinline__ typename Cplx<R>::T *fft_load_tw(typename Cplx<R>::T *dst, const void *src)
{
    for (int i = threadIdx.x; i < N; i += blockDim.x) dst[i] = __ldg((const typename Cplx<R>::T *)src + i);
    return dst;
}

// Row b = place_b(m) of the packed transform: place of packed frequency m.
template <int N>
__device__ __forceinline__ int fft_row(int m)
{
    typedef typename FftGeom<N>::PB PB;
    return (m % PB::R0) * PB::R1 + m / PB::R0;
}

// Forward transform of one (bead, c) plane, half spectrum out.
template <typename R, int N>
__device__ __forceinline__ void fft_plane_fwd_body(const FftArgs &f, const VBlk vb)
{
    typedef typename Cplx<R>::T C2;
    typedef FftGeom<N> G;
    typedef typename G::PA PA;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    C2 *pl = (C2 *)smem_raw;
    C2 *tw = fft_load_tw<R, N>(pl + G::H * G::LS, f.tw);
    const R *src = (const R *)f.grid + (size_t)vb.x * N * N;
    __syncthreads();
    for (int i = threadIdx.x; i < G::H * PA::R1; i += blockDim.x) {
        const int l = i / PA::R1, j = i - l * PA::R1;
        const R *q = src + 2 * l * N + j;
        C2 v[PA::R0];
#pragma unroll
        for (int t = 0; t < PA::R0; t++) v[t] = C2{q[t * PA::R1], q[t * PA::R1 + N]};
        dft<R, PA::R0, 1>(v);
        C2 *p = pl + l * G::LS + j;
        p[0] = v[0];
#pragma unroll
        for (int u = 1; u < PA::R0; u++) {
            const C2 w = tw[j * u];
            p[u * PA::S] = cmul(v[u], w.x, w.y);
        }
    }
    __syncthreads();
    fft_pass_a_inner<R, N, 1>(pl);
    fft_pass_b<R, N, 1>(pl, tw);
    C2 *dst = (C2 *)f.spec + (size_t)vb.x * N * G::NH;
    for (int i = threadIdx.x; i < G::H * G::NH; i += blockDim.x) {
        const int m = i / G::NH, k = i - m * G::NH;
        const C2 a = pl[fft_row<N>(m) * G::LS + PA::place(k)];
        const C2 b = pl[fft_row<N>(m ? G::H - m : 0) * G::LS + PA::place(k ? N - k : 0)];
        const R h = (R)0.5;
        const C2 e = {h * (a.x + b.x), h * (a.y - b.y)}, o = {h * (a.y + b.y), h * (b.x - a.x)};
        const C2 w = tw[m];
        const C2 t = cmul(o, w.x, w.y);
        dst[i] = C2{e.x + t.x, e.y + t.y};
        dst[i + G::H * G::NH] = C2{e.x - t.x, e.y - t.y};
    }
}

// Inverse of fft_plane_fwd_body, real potential out.
template <typename R, int N>
__device__ __forceinline__ void fft_plane_inv_body(const FftArgs &f, const VBlk vb)
{
    typedef typename Cplx<R>::T C2;
    typedef FftGeom<N> G;
    typedef typename G::PA PA;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    C2 *pl = (C2 *)smem_raw;
    C2 *tw = fft_load_tw<R, N>(pl + G::H * G::LS, f.tw);
    const C2 *src = (const C2 *)f.spec + (size_t)vb.x * N * G::NH;
    __syncthreads();
    for (int i = threadIdx.x; i < G::H * G::NH; i += blockDim.x) {
        const int m = i / G::NH, k = i - m * G::NH;
        const C2 f1 = src[i], f2 = src[i + G::H * G::NH];
        const C2 e = {f1.x + f2.x, f1.y + f2.y}, d = {f1.x - f2.x, f1.y - f2.y};
        const C2 w = tw[m];
        const C2 o = cmul(d, w.x, -w.y);
        pl[fft_row<N>(m) * G::LS + PA::place(k)] = C2{e.x - o.y, e.y + o.x};
        if (k > 0 && 2 * k < N)
            pl[fft_row<N>(m ? G::H - m : 0) * G::LS + PA::place(N - k)] = C2{e.x + o.y, o.x - e.y};
    }
    __syncthreads();
    fft_pass_b<R, N, -1>(pl, tw);
    fft_pass_a_inner<R, N, -1>(pl);
    R *dst = (R *)f.grid + (size_t)vb.x * N * N;
    for (int i = threadIdx.x; i < G::H * PA::R1; i += blockDim.x) {
        const int l = i / PA::R1, j = i - l * PA::R1;
        const C2 *p = pl + l * G::LS + j;
        C2 v[PA::R0];
        v[0] = p[0];
#pragma unroll
        for (int u = 1; u < PA::R0; u++) {
            const C2 w = tw[j * u];
            v[u] = cmul(p[u * PA::S], w.x, -w.y);
        }
        dft<R, PA::R0, -1>(v);
        R *q = dst + 2 * l * N + j;
#pragma unroll
        for (int t = 0; t < PA::R0; t++) {
            q[t * PA::R1] = v[t].x;
            q[t * PA::R1 + N] = v[t].y;
        }
    }
}

// One (bead, b) slab of the half spectrum: transform along c, energy and
// virial of the k-sphere terms (ewald3d_pme.c:366-425), multiplication by the
// influence function, inverse transform along c.  Half-spectrum points with
// 0 < a < N/2 stand for two full-grid points; E = 1/2 sum_full w |S|^2.
template <typename R, int N>
__device__ __forceinline__ void fft_conv_body(const FftArgs &f, const VBlk vb)
{
    typedef typename Cplx<R>::T C2;
    typedef FftGeom<N> G;
    typedef typename G::PA PA;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    C2 *sl = (C2 *)smem_raw;
    C2 *tw = fft_load_tw<R, N>(sl + N * G::LC, f.tw);
    __shared__ double red[7][16];
    const int bead = vb.x / N, b = vb.x - bead * N;
    C2 *base = (C2 *)f.spec + ((size_t)bead * N * N + b) * G::NH;
    constexpr int CS = N * G::NH;  // c stride
    const R *filt = (const R *)f.filt + (size_t)b * N;
    __syncthreads();
    for (int i = threadIdx.x; i < G::NH * PA::R1; i += blockDim.x) {
        const int j = i / G::NH, a = i - j * G::NH;
        const C2 *p = base + (size_t)j * CS + a;
        C2 v[PA::R0];
#pragma unroll
        for (int t = 0; t < PA::R0; t++) v[t] = p[(size_t)t * PA::R1 * CS];
        dft<R, PA::R0, 1>(v);
        C2 *q = sl + j * G::LC + a;
        q[0] = v[0];
#pragma unroll
        for (int u = 1; u < PA::R0; u++) {
            const C2 w = tw[j * u];
            q[u * PA::R1 * G::LC] = cmul(v[u], w.x, w.y);
        }
    }
    __syncthreads();
    // per-point energy and virial terms in R (FP32 for MIXED), summed in FP64
    double e = 0, pxx = 0, pyy = 0, pzz = 0, pxy = 0, pxz = 0, pyz = 0;
    const R kb = (R)(2 * b <= N ? b : b - N);
    const R tpi = (R)(2.0 * M_PI), falp2 = (R)(4.0 * f.alp * f.alp);
    for (int i = threadIdx.x; i < G::NH * PA::R0; i += blockDim.x) {
        const int s = i / G::NH, a = i - s * G::NH;
        C2 *p = sl + s * PA::R1 * G::LC + a;
        R w[PA::R1];
#pragma unroll
        for (int u = 0; u < PA::R1; u++) w[u] = __ldg(filt + (size_t)(s + PA::R0 * u) * N * N + a);
        C2 v[PA::R1];
#pragma unroll
        for (int t = 0; t < PA::R1; t++) v[t] = p[t * G::LC];
        dft<R, PA::R1, 1>(v);
        if (f.energy) {
            const R ka = (R)a;
            const R x0 = ka * (R)f.cell.hi[0] + kb * (R)f.cell.hi[1], y0 = ka * (R)f.cell.hi[3] + kb * (R)f.cell.hi[4],
                    z0 = ka * (R)f.cell.hi[6] + kb * (R)f.cell.hi[7];
            const R mult = (a == 0 || 2 * a == N) ? (R)0.5 : (R)1.0;
#pragma unroll
            for (int u = 0; u < PA::R1; u++) {
                if (w[u] == (R)0) continue;
                const int c = s + PA::R0 * u;
                const R kc = (R)(2 * c <= N ? c : c - N);
                const R xk = tpi * (x0 + kc * (R)f.cell.hi[2]);
                const R yk = tpi * (y0 + kc * (R)f.cell.hi[5]);
                const R zk = tpi * (z0 + kc * (R)f.cell.hi[8]);
                const R g2 = xk * xk + yk * yk + zk * zk;
                const R sm = mult * (v[u].x * v[u].x + v[u].y * v[u].y) * w[u];
                const R prep = (R)-2.0 * ((g2 / falp2) + (R)1.0) / g2 * sm;
                e += (double)sm;
                pxx += (double)(prep * xk * xk);
                pyy += (double)(prep * yk * yk);
                pzz += (double)(prep * zk * zk);
                pxy += (double)(prep * xk * yk);
                pxz += (double)(prep * xk * zk);
                pyz += (double)(prep * yk * zk);
            }
        }
#pragma unroll
        for (int u = 0; u < PA::R1; u++) {
            v[u].x *= w[u];
            v[u].y *= w[u];
        }
        dft<R, PA::R1, -1>(v);
#pragma unroll
        for (int t = 0; t < PA::R1; t++) p[t * G::LC] = v[t];
    }
    __syncthreads();
    for (int i = threadIdx.x; i < G::NH * PA::R1; i += blockDim.x) {
        const int j = i / G::NH, a = i - j * G::NH;
        const C2 *q = sl + j * G::LC + a;
        C2 v[PA::R0];
        v[0] = q[0];
#pragma unroll
        for (int u = 1; u < PA::R0; u++) {
            const C2 w = tw[j * u];
            v[u] = cmul(q[u * PA::R1 * G::LC], w.x, -w.y);
        }
        dft<R, PA::R0, -1>(v);
        C2 *p = base + (size_t)j * CS + a;
#pragma unroll
        for (int t = 0; t < PA::R0; t++) p[(size_t)t * PA::R1 * CS] = v[t];
    }
    if (!f.energy) return;
    const double val[7] = {e, pxx, pyy, pzz, pxy, pxz, pyz};
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
#pragma unroll
    for (int k = 0; k < 7; k++) {
        const double t = warp_sum(val[k]);
        if (lane == 0) red[k][wid] = t;
    }
    __syncthreads();
    if (threadIdx.x < 7) {
        double t = 0;
        for (int w2 = 0; w2 < (int)(blockDim.x >> 5); w2++) t += red[threadIdx.x][w2];
        double *acc = f.acc + (size_t)bead * S_NSLOT;
        // sum 0 is the energy, also the diagonal vnow term of the pressure
        // tensor (ewald3d_pme.c:415-417); 1..6 S_PXX..S_PYZ
        if (threadIdx.x == 0) {
            atomicAdd(&acc[S_VRECIP], t);
            atomicAdd(&acc[S_PXX], t);
            atomicAdd(&acc[S_PYY], t);
            atomicAdd(&acc[S_PZZ], t);
        } else {
            atomicAdd(&acc[S_PXX + threadIdx.x - 1], t);
        }
    }
}

template <typename R, int N>
__global__ void __launch_bounds__(FftGeom<N>::PLANE_T, fft_blocks<R, N>(FftGeom<N>::PLANE_T, false))
    fft_plane_fwd_kernel(const __grid_constant__ FftArgs f)
{
    fft_plane_fwd_body<R, N>(f, hw_blk());
}
template <typename R, int N>
__global__ void __launch_bounds__(FftGeom<N>::PLANE_T, fft_blocks<R, N>(FftGeom<N>::PLANE_T, false))
    fft_plane_inv_kernel(const __grid_constant__ FftArgs f)
{
    fft_plane_inv_body<R, N>(f, hw_blk());
}
template <typename R, int N>
__global__ void __launch_bounds__(FftGeom<N>::CONV_T, fft_blocks<R, N>(FftGeom<N>::CONV_T, false))
    fft_conv_kernel(const __grid_constant__ FftArgs f)
{
    fft_conv_body<R, N>(f, hw_blk());
}

// The mesh edges built: PINY's 2^a 3^b 5^c sizes that are multiples of 4, from
// 16 to 128 (set_pme_grid chooses among these).  X(N) for each.
// FP64 up to 108: a context refuses FP64 meshes above 117 points (pme_plane_smem).
#define PINYB200_FFT_MAX_FP64 108
#define PINYB200_FFT_EDGES(X)                                                                                    \
    X(16) X(20) X(24) X(32) X(36) X(40) X(48) X(60) X(64) X(72) X(80) X(96) X(100) X(108) X(120) X(128)

inline bool fft_fixed_edge(int Na, int Nb, int Nc)
{
    if (Na != Nb || Na != Nc) return false;
#define PINYB200_FFT_IS(n) \
    if (Na == n) return true;
    PINYB200_FFT_EDGES(PINYB200_FFT_IS)
#undef PINYB200_FFT_IS
    return false;
}

// The three kernels of one box on a mesh of built edge N (fft_fixed_edge),
// enqueued on c->stream with their timing marks.
template <typename R>
cudaError_t launch_fft_fixed(pinyb200_ctx *c, int N, int P, const FftArgs &f);

// One of the three kernels (stage 0 forward planes, 1 convolution, 2 inverse
// planes) of many MIXED boxes of mesh edge N as persistent launches.
cudaError_t launch_fft_fixed_batch(int N, const std::vector<FftArgs> &bx, const std::vector<int> &P, int sm_count,
                                   cudaStream_t st, int stage);

}  // namespace pinyb200
