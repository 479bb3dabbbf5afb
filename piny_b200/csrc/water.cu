// Launchers of the staging and finishing kernels (water.cuh).
#include "water.cuh"

namespace pinyb200 {

// The per-bead sums and the bin counters to zero.
// acc: the bead sums and the time stamps behind them, nacc in all.
__global__ void __launch_bounds__(256) water_clear_kernel(double *__restrict__ acc, int nacc, int *__restrict__ cnt,
                                                          int ncnt)
{
    const int t = blockIdx.x * blockDim.x + threadIdx.x, n = gridDim.x * blockDim.x;
    for (int i = t; i < nacc; i += n)
        acc[i] = i == nacc - T_NSTAMP + T_BEG ? __longlong_as_double((long long)clock_ns()) : 0.0;
    for (int i = t; i < ncnt; i += n) cnt[i] = 0;
}

template <typename R, int NS, bool Q0>
__global__ void __launch_bounds__(256) water_stage_kernel(const __grid_constant__ StageArgs a,
                                                          const __grid_constant__ PmeArgs pm,
                                                          const __grid_constant__ TileArgs t,
                                                          const __grid_constant__ Cell cell)
{
    water_stage_body<R, NS, Q0>(a, pm, t, cell, hw_blk());
}

template <int NS, bool Q0>
__global__ void __launch_bounds__(256, 2) water_finish_kernel(const __grid_constant__ FinishArgs a)
{
    unsigned long long *stamp = (unsigned long long *)(a.acc + (size_t)a.P * S_NSLOT);
    stamp_start(stamp, T_FIN0);
    water_finish_body<NS, Q0>(a, hw_blk());
    stamp_end(stamp, T_END);
}

// Threads per block: 256, fewer (down to 64, and a bead each) while that
// leaves SMs without a block.
static int water_threads(const pinyb200_ctx *c)
{
    int t = 256;
    while (t > 64 && t > c->P && (long long)c->nmol * c->P < (long long)t * c->sm_count) t /= 2;
    return t;
}
static size_t water_smem(const pinyb200_ctx *c, int threads)
{
    return sizeof(double) * (size_t)c->P * (threads / c->P * 3 * c->mol_stride + 1);
}

template <typename R>
static cudaError_t launch_stage_r(pinyb200_ctx *c, const StageArgs &a, const PmeArgs &pm, const TileArgs &t,
                                  const Cell &cell)
{
    const int th = water_threads(c), mb = th / c->P;
    const unsigned g = (unsigned)((c->nmol + mb - 1) / mb);
    const size_t sm = water_smem(c, th);
    if (c->mol_stride == 4) water_stage_kernel<R, 4, false><<<g, th, sm, c->stream>>>(a, pm, t, cell);
    else if (c->water_q0) water_stage_kernel<R, 3, true><<<g, th, sm, c->stream>>>(a, pm, t, cell);
    else water_stage_kernel<R, 3, false><<<g, th, sm, c->stream>>>(a, pm, t, cell);
    return cudaGetLastError();
}

// Kernel arguments of one context.
static StageArgs stage_args(pinyb200_ctx *c, const double *d_pos, const double *d_xmod)
{
    StageArgs a;
    a.natm = c->sys.natm;
    a.nmol = c->nmol;
    a.P = c->P;
    a.pos = d_pos;
    a.posT = c->d_posT;
    a.forceT = c->d_forceT;
    a.offT = c->mix_ok ? c->d_offT : nullptr;
    a.xm_src = c->P > 1 ? d_xmod : nullptr;
    a.xm_dst = c->d_xmod;
    a.ext = (unsigned long long *)(c->d_acc + S_EXT);
    a.gcoef = c->sys.ghost_coef;
    a.bin = c->sys.nchrg > 0 && c->sys.nktot > 0 ? 1 : 0;
    return a;
}

static FinishArgs finish_args(pinyb200_ctx *c, double *d_out, bool energy, bool distrib, bool keep_site_forces)
{
    const DeviceSystem &s = c->sys;
    FinishArgs a;
    a.natm = s.natm;
    a.nmol = c->nmol;
    a.P = c->P;
    a.posT = c->d_posT;
    a.forceT = c->d_forceT;
    a.forceP = s.nchrg > 0 && s.nktot > 0 ? c->d_forceP : nullptr;
    a.forceT_out = keep_site_forces ? c->d_forceT : nullptr;
    a.out = d_out;
    a.acc = c->d_acc;
    a.energy = energy ? 1 : 0;
    a.distrib = distrib ? 1 : 0;
    a.bond_eq = s.bond_eq + c->water_bond;
    a.bond_c = s.bond_c + 7 * c->water_bond;
    a.bond_dc = s.bond_dc + 7 * c->water_bond;
    a.bend_c = s.bend_c + 7 * c->water_bend;
    a.bend_s = s.bend_s + 7 * c->water_bend;
    a.bend_dc = s.bend_dc + 7 * c->water_bend;
    a.bend_ds = s.bend_ds + 7 * c->water_bend;
    a.ecor_nsplin = s.ecor_nsplin;
    a.ecor_rmin = s.ecor_rmin;
    a.ecor_dr = s.ecor_dr;
    a.ecor_dri = s.ecor_dri;
    a.ecor_tab = s.necor > 0 ? s.ecor_tab : nullptr;
    for (int k = 0; k < 4; k++) a.q[k] = k < c->mol_stride ? c->h_charge[k] : 0.0;
    a.gcoef = s.ghost_coef;
    return a;
}

// Positions (and mode-1 positions d_xmod, nullptr: the bead centroid) staged,
// sums and bins cleared, charges binned; enqueued on c->stream.
cudaError_t launch_water_stage(pinyb200_ctx *c, const Cell &cell, const double *d_pos, const double *d_xmod)
{
    const StageArgs a = stage_args(c, d_pos, d_xmod);
    PmeArgs pm = {};
    TileArgs t = {};
    int ncnt = 0;
    if (a.bin) {
        pm = pme_args_of(c);
        t = tile_args_of(c, c->sys.n_interp, c->pme_tile);
        ncnt = c->P * c->pme_ntile + 1;
    }
    const int nacc = c->P * S_NSLOT + T_NSTAMP;
    const int blocks = std::max(1, std::min((std::max(ncnt, nacc) + 255) / 256, c->sm_count));
    water_clear_kernel<<<blocks, 256, 0, c->stream>>>(c->d_acc, nacc, t.cnt, ncnt);
    if (c->precision == PINYB200_FP64) return launch_stage_r<double>(c, a, pm, t, cell);
    return launch_stage_r<float>(c, a, pm, t, cell);
}

// Intramolecular terms, the sum of all forces and their way out to d_out;
// keep_site_forces: the complete site forces are kept in c->d_forceT too.
cudaError_t launch_water_finish(pinyb200_ctx *c, double *d_out, bool energy, bool distrib, bool keep_site_forces)
{
    const FinishArgs a = finish_args(c, d_out, energy, distrib, keep_site_forces);
    const int th = water_threads(c), mb = th / c->P;
    const unsigned g = (unsigned)((c->nmol + mb - 1) / mb);
    const size_t sm = water_smem(c, th);
    auto go = [&](auto *kernel) {
        // static and dynamic shared memory together may pass 48 KB
        cudaError_t e = smem_optin((const void *)kernel, (int)sm);
        if (e != cudaSuccess) return e;
        kernel<<<g, th, sm, c->stream>>>(a);
        return cudaGetLastError();
    };
    if (c->mol_stride == 4) return go(water_finish_kernel<4, false>);
    if (c->water_q0) return go(water_finish_kernel<3, true>);
    return go(water_finish_kernel<3, false>);
}

// ---------------------------------------------------------------------------
// Many boxes per launch: one persistent launch per kind of molecule.

struct StageBox {
    StageArgs a;
    PmeArgs pm;
    TileArgs t;
    Cell cell;
};

template <int NS, bool Q0>
__global__ void __launch_bounds__(256) water_stage_batch_kernel(const __grid_constant__ BoxTab<StageBox> t)
{
    PINYB200_BOX_LOOP(t, i, vb,
                      (water_stage_body<float, NS, Q0>(t.arg[i].a, t.arg[i].pm, t.arg[i].t, t.arg[i].cell, vb)));
}

template <int NS, bool Q0>
__global__ void __launch_bounds__(256, 2) water_finish_batch_kernel(const __grid_constant__ BoxTab<FinishArgs> t)
{
    PINYB200_BOX_LOOP(t, i, vb, (water_finish_body<NS, Q0>(t.arg[i], vb)));
}

// Kinds of molecule: 0 four sites, 1 three charged sites, 2 three sites, two charged.
static int water_kind(const pinyb200_ctx *c) { return c->mol_stride == 4 ? 0 : (c->water_q0 ? 1 : 2); }

// Staging of MIXED contexts (as launch_water_stage; the sums, bin counters
// and charge grids are already zero).
cudaError_t launch_water_stage_batch(const std::vector<pinyb200_ctx *> &box, const std::vector<Cell> &cells,
                                     const std::vector<const double *> &pos, const std::vector<const double *> &xmod,
                                     int sm_count, cudaStream_t st)
{
    for (int kind = 0; kind < 3; kind++) {
        BoxTabBuilder<StageBox> tb;
        size_t sm = 0;
        for (size_t i = 0; i < box.size(); i++) {
            pinyb200_ctx *c = box[i];
            if (water_kind(c) != kind) continue;
            StageBox x;
            memset(&x, 0, sizeof(x));
            x.a = stage_args(c, pos[i], xmod[i]);
            if (x.a.bin) {
                x.pm = pme_args_of(c);
                x.t = tile_args_of(c, c->sys.n_interp, c->pme_tile);
            }
            x.cell = cells[i];
            const int mb = 256 / c->P;
            tb.add(x, (c->nmol + mb - 1) / mb, 1, (double)c->nmol * c->P);
            sm = std::max(sm, water_smem(c, 256));
        }
        auto go = [&](auto *kernel) {
            return launch_tables(tb, (const void *)kernel, 256, sm, sm_count,
                                 [&](const BoxTab<StageBox> &t, int g) { kernel<<<g, 256, sm, st>>>(t); });
        };
        const cudaError_t e = kind == 0   ? go(water_stage_batch_kernel<4, false>)
                              : kind == 1 ? go(water_stage_batch_kernel<3, true>)
                                          : go(water_stage_batch_kernel<3, false>);
        if (e != cudaSuccess) return e;
    }
    return cudaSuccess;
}

cudaError_t launch_water_finish_batch(const std::vector<pinyb200_ctx *> &box, const std::vector<double *> &out,
                                      bool energy, bool distrib, int sm_count, cudaStream_t st)
{
    for (int kind = 0; kind < 3; kind++) {
        BoxTabBuilder<FinishArgs> tb;
        size_t sm = 0;
        for (size_t i = 0; i < box.size(); i++) {
            pinyb200_ctx *c = box[i];
            if (water_kind(c) != kind) continue;
            const int mb = 256 / c->P;
            tb.add(finish_args(c, out[i], energy, distrib, false), (c->nmol + mb - 1) / mb, 1, (double)c->nmol * c->P);
            sm = std::max(sm, water_smem(c, 256));
        }
        auto go = [&](auto *kernel) {
            return launch_tables(tb, (const void *)kernel, 256, sm, sm_count,
                                 [&](const BoxTab<FinishArgs> &t, int g) { kernel<<<g, 256, sm, st>>>(t); });
        };
        const cudaError_t e = kind == 0   ? go(water_finish_batch_kernel<4, false>)
                              : kind == 1 ? go(water_finish_batch_kernel<3, true>)
                                          : go(water_finish_batch_kernel<3, false>);
        if (e != cudaSuccess) return e;
    }
    return cudaSuccess;
}

}  // namespace pinyb200
