"""The work that users of this framework have it do, as cases that can be timed and compared.

A case is one call (or one pair of calls) of the public Python entry points of
``piny_b200.lib`` on a seeded water box: the force and energy evaluation of all
beads of a box (``DeviceBox.energy_force_device``, ``energy_force``), with and
without PINY's list test and rebuild, many uneven boxes at once
(``DeviceBatch``), the parameter gradient (``DeviceBox.grad``) and the NVT
ring-polymer step (``DevicePimd.step``).  Launch shapes are the defaults: what
a program gets that does not call the autotuner.

``exact`` gives the same numbers in 64 bits from plain torch: direct sums over
molecule pairs, PME by scatter, torch's FFT and gather, and the integrator as
array operations.  The set-up arrays (spline tables, k list, B-spline weights,
bond and bend series) are the call's inputs and are taken as they are.
"""
from __future__ import annotations

import dataclasses
import math

import numpy as np
import torch

from piny_b200 import params, pimd, system, water
from piny_b200.lib import NORMAL_MODES, STAGING, DeviceBatch, DeviceBox, DevicePimd

ENERGIES = ("vreal", "vvdw", "vcoul", "vrecip", "vself", "vbgr", "vecor", "vlong", "vbond", "vbend", "vintert",
            "vintrat")
AU_PER_AMU = 1822.888486
MODELS = {"spcfw": water.SPC_FW, "tip4pf": water.TIP4P_F}


# ---------------------------------------------------------------------------
# the cases

def listed():
    return [
        # classical MD of a small box: one bead, every kernel a few microseconds, so launches and latency count
        _box("classical_256_fp64", "spcfw", 256, 1, 32, 6, "fp64"),
        # classical MD of a large box: one bead, lanes have to come from sites instead of beads
        _box("classical_4096_mixed", "tip4pf", 4096, 1, 64, 8, "mixed"),
        # path-integral water, small box
        _box("pimd_256x32_mixed", "spcfw", 256, 32, 32, 6, "mixed"),
        # path-integral water, the benchmark's box, in both precisions (the largest call)
        _box("pimd_4096x32_mixed", "tip4pf", 4096, 32, 64, 8, "mixed"),
        _box("pimd_4096x32_fp64", "tip4pf", 4096, 32, 64, 8, "fp64"),
        # a box whose mesh is one of PINY's 2^a 3^b 5^c sizes that is no power of two, molecule count odd
        _box("pimd_1501x8_mesh36_mixed", "tip4pf", 1501, 8, 36, 8, "mixed"),
        # the call a host program makes: positions in and forces out in host memory
        _box("host_1024x16_mixed", "tip4pf", 1024, 16, 32, 8, "mixed", kind="host"),
        # force calls of an MD step in which PINY's list test fires, so that the list is rebuilt on the device
        _box("rebuild_8000x4_mixed", "tip4pf", 8000, 4, 80, 6, "mixed", kind="rebuild"),
        # replicas of many sizes in one call (parameter fitting, many thermodynamic states)
        {"name": "batch_24_mixed", "kind": "batch", "boxes": 24, "nmin": 64, "nmax": 1024, "mix": 2024,
         "precision": "mixed"},
        # force matching: forward evaluation and adjoint for the 9 model parameters
        _box("grad_1024x16_mixed", "tip4pf", 1024, 16, 32, 8, "mixed", kind="grad"),
        # PINY's NVT ring-polymer step: chains, transforms, springs, list test and forces
        _box("step_1024x32_mixed", "tip4pf", 1024, 32, 32, 8, "mixed", kind="step", modes="normal"),
    ]


def _box(name, model, nmol, beads, grid, order, precision, kind="eval", modes=""):
    c = {"name": name, "kind": kind, "model": model, "nmol": nmol, "beads": beads, "grid": grid, "order": order,
         "precision": precision}
    if kind == "step":
        c["modes"] = modes
    return c


def draw(rng):
    kind = rng.choice(["eval", "eval", "eval", "eval", "host", "rebuild", "batch", "grad", "step"])
    if kind == "batch":
        return {"kind": "batch", "boxes": rng.randint(3, 24), "nmin": 64, "nmax": rng.randint(200, 1024),
                "mix": rng.randint(1, 10 ** 6), "precision": "mixed"}
    precision = rng.choice(["mixed", "mixed", "mixed", "fp64"])
    model = "tip4pf" if kind == "grad" else rng.choice(["tip4pf", "tip4pf", "spcfw"])
    beads = rng.choice([4, 8, 16, 32]) if kind == "step" else rng.choice([1, 1, 2, 4, 8, 16, 32, 64])
    # molecules x beads, so that a drawn pass stays below the longest listed ones
    most = {"eval": 65536, "rebuild": 20000}.get(kind, 32768)
    most = int((most if precision == "mixed" else most / 2) / beads)
    nmol = int(round(math.exp(rng.uniform(math.log(216), math.log(max(217, min(16384, most)))))))
    # meshes a user picks: PINY's sizes from about one point per Angstrom up to 1.4 (grid point spacing 0.7 A)
    edge = water.density_box_edge(nmol)
    sizes = [n for n in range(16, 129, 4) if _smooth(n)]
    fit = [n for n in sizes if edge <= n <= 1.4 * edge + 4]
    c = {"kind": kind, "model": model, "nmol": nmol, "beads": beads, "grid": rng.choice(fit),
         "order": rng.choice([6, 8]), "precision": precision}
    if kind == "step":
        c["modes"] = rng.choice(["normal", "staging"])
    return c


def _smooth(n):
    for p in (2, 3, 5):
        while n % p == 0:
            n //= p
    return n == 1


# ---------------------------------------------------------------------------
# inputs

def _spec(case, seed):
    edge = water.density_box_edge(case["nmol"])
    return water.BoxSpec(MODELS[case["model"]], case["nmol"], edge, case["beads"], 298.0, seed,
                         cutoff=min(9.0, 0.47 * edge), grid=case["grid"], order=case["order"])


def _batch_specs(case, seed):
    """Boxes as in water.c4_specs: sizes and bead counts from the case's mix, positions from the seed."""
    rng = np.random.default_rng(case["mix"])
    out = []
    for i in range(case["boxes"]):
        n = int(round(float(np.exp(rng.uniform(np.log(case["nmin"]), np.log(case["nmax"]))))))
        beads = int(rng.choice([1, 4, 8, 16, 32, 64]))
        edge = water.density_box_edge(n)
        out.append(water.BoxSpec(water.TIP4P_F, n, edge, beads, 298.0, seed * 1000 + i,
                                 grid=1 << int(np.ceil(np.log2(edge))), order=8))
    return out


def _positions(spec):
    """Bead positions and mode-1 positions (None for one bead), Bohr."""
    pos = water.build_positions(spec) / water.BOHR
    return pos, (pos.mean(axis=0) if spec.nbeads > 1 else None)


def _moved(spec, pos, seed):
    """Every molecule moved as a whole by 0.6 skin in a random direction: past PINY's rebuild threshold (skin / 2)."""
    rng = np.random.default_rng(seed + 77)
    d = rng.normal(size=(spec.nmol, 3))
    d *= 0.6 * spec.skin / water.BOHR / np.linalg.norm(d, axis=1, keepdims=True)
    return pos + np.repeat(d, spec.model.nsite, axis=0)[None]


def _fbar(pos, seed):
    """Upstream gradient of the forces, of the size of a force-matching residual (Hartree/Bohr)."""
    return 1e-3 * np.random.default_rng(seed + 5).normal(size=pos.shape)


def _step_setup(case, spec, S):
    ghost = np.zeros(S["natm"], bool)
    if S["nghost"]:
        ghost[np.asarray(S["ghost_atom"])] = True
    mass = np.tile(np.asarray(spec.model.masses, np.float64), spec.nmol) * AU_PER_AMU
    modes = NORMAL_MODES if case["modes"] == "normal" else STAGING
    setup = pimd.nvt_setup(mass, ghost, spec.nbeads, modes, spec.temperature, 10.0, 800.0, len_nhc=4, nyosh=3)
    rng = np.random.default_rng(spec.seed + 9)
    v = rng.normal(size=(spec.nbeads, S["natm"], 3))
    v *= np.sqrt(spec.temperature / water.BOLTZ / setup["bead_mass"])[:, :, None]
    v[:, ghost, :] = 0.0
    return setup, v


def _device(a):
    return None if a is None else torch.from_numpy(np.ascontiguousarray(a)).cuda()


def _ptr(t):
    return None if t is None else t.data_ptr()


class _One:
    """One box with its list, and its positions on the GPU."""

    def __init__(self, spec, precision):
        self.spec = spec
        self.pos, self.xmod = _positions(spec)
        self.S = system.build_system(spec, self.pos)
        self.hmat = self.S["hmat"]
        self.box = DeviceBox(self.S, spec.nbeads, precision)
        self.box.build_list(self.pos[0], self.xmod, self.hmat, self.S["cutskin2"])
        self.d_pos, self.d_xmod = _device(self.pos), _device(self.xmod)
        self.d_force = torch.empty_like(self.d_pos)


class _State:
    pass


def prepare(case, seed):
    s = _State()
    s.kind = case["kind"]
    s.stream = torch.cuda.current_stream().cuda_stream
    if s.kind == "batch":
        s.boxes = [_One(spec, case["precision"]) for spec in _batch_specs(case, seed)]
        s.batch = DeviceBatch([b.box for b in s.boxes])
        s.args = ([_ptr(b.d_pos) for b in s.boxes], [_ptr(b.d_xmod) for b in s.boxes], [b.hmat for b in s.boxes],
                  [_ptr(b.d_force) for b in s.boxes])
        return s
    s.one = one = _One(_spec(case, seed), case["precision"])
    if s.kind == "rebuild":
        moved = _moved(one.spec, one.pos, seed)
        s.places = [(_device(p), _device(p.mean(axis=0) if one.spec.nbeads > 1 else None),
                     torch.empty_like(one.d_pos)) for p in (moved, one.pos)]
        one.box.list_set_spread(one.S["spread"])
    elif s.kind == "grad":
        one.box.grad_prepare(params.tangents(one.spec, params.theta_of(one.spec.model), one.S))
        s.d_fbar = _device(_fbar(one.pos, seed))
    elif s.kind == "step":
        setup, v = _step_setup(case, one.spec, one.S)
        s.pimd = DevicePimd(setup)
        s.d_v = _device(v)
        s.pimd.forces(one.box, _ptr(one.d_pos), _ptr(one.d_force), one.hmat, stream=s.stream)
        one.box.list_set_spread(one.S["spread"])
    return s


# ---------------------------------------------------------------------------
# one pass

def _energies(e):
    return np.array([e[k] for k in ENERGIES])


def run(s):
    if s.kind == "batch":
        e = s.batch.energy_force_device(*s.args, stream=s.stream, distribute_ghosts=True)
        # one array each: 24 boxes' energies and tensors
        return {"forces": [b.d_force for b in s.boxes], "energies": np.array([_energies(x) for x in e]),
                "pvten": np.array([x["pvten"] for x in e])}
    one = s.one
    if s.kind == "eval":
        e = one.box.energy_force_device(_ptr(one.d_pos), _ptr(one.d_xmod), one.hmat, _ptr(one.d_force),
                                        stream=s.stream, distribute_ghosts=True)
        return {"force": one.d_force, "energies": _energies(e), "pvten": e["pvten"]}
    if s.kind == "host":
        f, e = one.box.energy_force(one.pos, one.xmod, one.hmat, distribute_ghosts=True)
        return {"force": f, "energies": _energies(e), "pvten": e["pvten"]}
    if s.kind == "rebuild":
        out = []
        for d_pos, d_xmod, d_force in s.places:
            e = one.box.energy_force_device(_ptr(d_pos), _ptr(d_xmod), one.hmat, _ptr(d_force), stream=s.stream,
                                            distribute_ghosts=True, update_list=True)
            out.append({"force": d_force, "energies": _energies(e), "pvten": e["pvten"]})
        return out
    if s.kind == "grad":
        dE, dF = one.box.grad(_ptr(one.d_pos), _ptr(one.d_xmod), one.hmat, _ptr(s.d_fbar), stream=s.stream)
        return {"dE": dE, "dF": dF}
    e = s.pimd.step(one.box, _ptr(one.d_pos), _ptr(s.d_v), _ptr(one.d_force), one.hmat, stream=s.stream)
    return {"x": one.d_pos, "v": s.d_v, "f": one.d_force, "energies": _energies(e),
            "estimators": np.array([e["kin_harm"], e["akvirx"]]), "pvten": e["pvten"], "pvten_tot": e["pvten_tot"],
            "pvten_mode_tot": e["pvten_mode_tot"]}


# ---------------------------------------------------------------------------
# what a pass cannot do without

def work(case):
    if case["kind"] == "batch":
        parts = [_work_box(s.model, s.nmol, s.nbeads, s.grid, s.order, s.L, s.cutoff) for s in _batch_specs(case, 0)]
        return {"bytes": sum(b for b, _ in parts), "flops": sum(f for _, f in parts)}
    s = _spec(case, 0)
    b, f = _work_box(s.model, s.nmol, s.nbeads, s.grid, s.order, s.L, s.cutoff)
    if case["kind"] == "rebuild":
        # two evaluations, each with a test of every molecule pair of the 27 cells around a molecule
        return {"bytes": 2 * b, "flops": 2 * (f + 10.0 * s.nmol * s.nmol / 2)}
    if case["kind"] == "grad":
        return {"bytes": 2 * b, "flops": 2.5 * f}
    if case["kind"] == "step":
        n = s.natm * 3 * s.nbeads
        return {"bytes": b + 8.0 * n * 4, "flops": f + n * (6.0 * s.nbeads + 200.0)}
    return {"bytes": b, "flops": f}


def _work_box(model, nmol, beads, grid, order, edge, cutoff):
    """Positions in, forces out; 45 operations per site pair within the cutoff that carries a charge product or a
    Lennard-Jones term, PME as spread, two real FFTs and gather, and 150 per molecule for its bonds and bend."""
    ns = model.nsite
    nq = sum(1 for q in model.charges if q != 0.0)
    active = nq * nq + (0 if model.charges[0] != 0.0 else 1)
    pairs = 0.5 * nmol * (4.0 / 3.0 * math.pi * cutoff ** 3) * nmol / edge ** 3 * active
    g = float(grid) ** 3
    pme = nmol * nq * order ** 3 * 10.0 + 2 * 2.5 * g * math.log2(g) + 8.0 * g
    return 48.0 * nmol * ns * beads, beads * (45.0 * pairs + pme + 150.0 * nmol)


def tolerance(case):
    # Against 64 bits FP32 pair and mesh arithmetic with FP64 sums is 1e-7 to 5e-7 off in forces and virial, 2e-8 in
    # energies and up to 7e-7 in the parameter gradient; FP64 runs are 1e-15 to 2e-13 off, and a separation that
    # rounds to the spline's neighbouring interval moves one pair's force by up to 1e-9 of itself.
    if case["precision"] == "fp64":
        return {"rel": 1e-11, "max": 1e-9}
    if case["kind"] == "grad":
        return {"rel": 2e-6, "max": 1e-5}
    return {"rel": 1e-6, "max": 4e-5}


# ---------------------------------------------------------------------------
# the same numbers in 64 bits

_DEV = "cuda" if torch.cuda.is_available() else "cpu"


def _t(a, dtype=torch.float64):
    return torch.as_tensor(np.ascontiguousarray(a), dtype=dtype, device=_DEV)


def _nint(x):
    return torch.where(x >= 0, torch.floor(x + 0.5), torch.ceil(x - 0.5))


def _spline(table, r, rmin, dr, dri, nsplin):
    """PINY's 4-point cubic on r_i = dr (i - 3) + rmin, i from 1."""
    k = torch.clamp(((r.detach() - rmin) * dri + 0.5).to(torch.int64) + 3, 3, nsplin - 2)
    t = (r - ((k - 3).to(r.dtype) * dr + rmin)) * dri
    c0, fp1, fm1, fm2 = table[k - 1], table[k], table[k - 2], table[k - 3]
    c1 = fp1 / 3.0 + 0.5 * c0 - fm1 + fm2 / 6.0
    c2 = 0.5 * fp1 - c0 + 0.5 * fm1
    c3 = fp1 / 6.0 - 0.5 * c0 + 0.5 * fm1 - fm2 / 6.0
    return c0 + t * (c1 + t * (c2 + t * c3))


def _bspline(u, n):
    """Weights M_n(u + j), j = 0..n-1, and their derivatives, for fractions u in [0, 1): the last axis is j."""
    j = torch.arange(n, dtype=u.dtype, device=u.device)
    x = u[..., None] + j
    m = torch.where(j < 2, 1.0 - torch.abs(x - 1.0), torch.zeros_like(x))
    d = None

    def shifted(w):
        return torch.cat([torch.zeros_like(w[..., :1]), w[..., :-1]], dim=-1)

    for k in range(3, n + 1):
        if k == n:
            d = m - shifted(m)
        m = (x * m + (k - x) * shifted(m)) / (k - 1)
    return m, d


class _Exact:
    """Plain evaluation of one box from its set-up arrays; `tangents` and `eps` move the parameters."""

    def __init__(self, spec, S, pos, xmod, tangents=None):
        self.spec, self.S, self.ns = spec, S, spec.model.nsite
        self.P, self.natm = spec.nbeads, int(S["natm"])
        self.h = float(S["hmat"][0])
        self.eps = torch.zeros(len(tangents or ()), dtype=torch.float64, device=_DEV,
                               requires_grad=bool(tangents))
        tan = tangents or []

        def moved(key, dkey):
            a = _t(S[key])
            for k, tk in enumerate(tan):
                if tk.get(dkey) is not None:
                    a = a + self.eps[k] * _t(tk[dkey])
            return a

        self.q = moved("charge", "dcharge")
        self.cv0, self.cdv0 = moved("cv0", "dcv0"), moved("cdv0", "dcdv0")
        self.coef = moved("ghost_coef", "dghost_coef") if S["nghost"] else None
        self.bond_eq, self.bond_c = moved("bond_eq", "dbond_eq"), moved("bond_c", "dbond_c")
        self.bond_dc = torch.cat([self.bond_c[1:2], self.bond_c[1:2], self.bond_c[2:] * _t(np.arange(2.0, 7.0))])
        self.bend = {k: moved("bend_" + k, "dbend_" + k) for k in ("c", "s", "dc", "ds")}
        self.clong = torch.tensor(float(S["clong"]), dtype=torch.float64, device=_DEV)
        for k, tk in enumerate(tan):
            if tk.get("dclong"):
                self.clong = self.clong + self.eps[k] * float(tk["dclong"])
        self.charged = torch.nonzero(_t(S["charge"]) != 0.0).flatten()
        self._mol_pairs(pos, xmod)
        self._filter()

    def _mol_pairs(self, pos, xmod):
        """Molecule pairs that can have a site pair within the cutoff, from mode-1 positions and a margin."""
        S, ns = self.S, self.ns
        ref = _t(pos[0] if xmod is None else xmod)
        self.xref = ref
        o = ref[::ns]
        out = float((_t(pos).reshape(self.P, -1, ns, 3) - o[None, :, None, :]).norm(dim=-1).max())
        reach2 = (float(np.max(S["cutoff"])) + 2.0 * out) ** 2
        n = o.shape[0]
        i_l, j_l = [], []
        rows = max(1, 8_000_000 // n)
        for a in range(0, n, rows):
            d = o[a:a + rows, None, :] - o[None, :, :]
            d = d - self.h * torch.round(d / self.h)
            ij = torch.nonzero((d * d).sum(-1) <= reach2)
            ij[:, 0] += a
            ij = ij[ij[:, 0] > ij[:, 1]]
            i_l.append(ij[:, 0])
            j_l.append(ij[:, 1])
        self.mi, self.mj = torch.cat(i_l), torch.cat(j_l)

    def _filter(self):
        """Influence function on the half spectrum and the k sphere's sums (ewald3d_recip_pme)."""
        S = self.S
        na, nb, nc = int(S["ngrid_a"]), int(S["ngrid_b"]), int(S["ngrid_c"])
        self.grid = (nc, nb, na)
        k = torch.stack([_t(S["kastr"], torch.int64), _t(S["kbstr"], torch.int64), _t(S["kcstr"], torch.int64)], -1)
        g = k.to(torch.float64) * (2.0 * math.pi / self.h)
        g2 = (g * g).sum(-1)
        falp2 = 4.0 * S["alp_ewd"] ** 2
        preg = torch.exp(-g2 / falp2) / (g2 * (self.h ** 3 / (4.0 * math.pi)))
        bw = _t(S["bweight"])
        self.kidx = ((k[:, 2] % nc) * nb + (k[:, 1] % nb)) * na + (k[:, 0] % na)
        kneg = (((-k[:, 2]) % nc) * nb + ((-k[:, 1]) % nb)) * na + ((-k[:, 0]) % na)
        self.preg, self.kbw, self.kg = preg, bw, g
        self.kprep = -2.0 * preg * (g2 / falp2 + 1.0) / g2
        full = torch.zeros(na * nb * nc, dtype=torch.float64, device=_DEV)
        full[self.kidx] = preg * bw
        full[kneg] = preg * bw
        self.infl = full.reshape(self.grid)

    def ghosts(self, x):
        """x [natm, 3] with the M sites put back from their components; also the coefficients' list."""
        S = self.S
        if not S["nghost"]:
            return x
        nc = int(S["ghost_ncomp"])
        comp = _t(S["ghost_comp"], torch.int64).reshape(-1, nc)
        g = (self.coef.reshape(-1, nc)[:, :, None] * x[comp]).sum(1)
        return x.index_copy(0, _t(S["ghost_atom"], torch.int64), g)

    def distribute(self, f):
        S = self.S
        if not S["nghost"]:
            return f
        nc = int(S["ghost_ncomp"])
        comp = _t(S["ghost_comp"], torch.int64)
        atom = _t(S["ghost_atom"], torch.int64)
        add = (self.coef.reshape(-1, nc)[:, :, None] * f[atom][:, None, :]).reshape(-1, 3)
        f = f.index_add(0, comp, add)
        return f.index_copy(0, atom, torch.zeros_like(f[atom]))

    def pairs(self, x):
        """(force, vvdw, vcoul, virial) of the real-space pairs within the cutoff."""
        S, ns = self.S, self.ns
        f = torch.zeros_like(x)
        vv = vc = torch.zeros((), dtype=x.dtype, device=x.device)
        pv = torch.zeros(3, 3, dtype=x.dtype, device=x.device)
        nsplin = int(S["nsplin"])
        typ, charge = np.asarray(S["atm_typ"])[:ns], np.asarray(S["charge"])[:ns]
        for a in range(ns):
            for b in range(ns):
                p = system._pair_index(int(typ[a]), int(typ[b]), int(S["ntyp"]))
                u = int(S["inter_map"][p])
                lj = bool(np.any(np.asarray(S["cv0"])[u * nsplin:(u + 1) * nsplin]))
                if charge[a] * charge[b] == 0.0 and not lj:
                    continue
                i, j = self.mi * ns + a, self.mj * ns + b
                d = x[i] - x[j]
                ref = self.xref[i] - self.xref[j] if self.P > 1 else d.detach()
                d = d - self.h * _nint(ref / self.h)
                near = (d.detach() ** 2).sum(-1).sqrt() < float(S["cutoff"][p])
                i, j, d = i[near], j[near], d[near]
                r = (d * d).sum(-1).sqrt()
                grid = (float(S["rmin_spl"][u]), float(S["dr_spl"][u]), float(S["dri_spl"][u]), nsplin)
                off = u * nsplin
                dv = torch.zeros_like(r)
                if charge[a] * charge[b] != 0.0:
                    q2 = self.q[i] * self.q[j]
                    dv = dv + q2 * _spline(_t(S["cdv0_c"])[off:off + nsplin], r, *grid)
                    vc = vc + (q2 * _spline(_t(S["cv0_c"])[off:off + nsplin], r, *grid)).sum()
                if lj:
                    dv = dv + _spline(self.cdv0[off:off + nsplin], r, *grid)
                    vv = vv + _spline(self.cv0[off:off + nsplin], r, *grid).sum()
                g = d * dv[:, None]
                f = f.index_add(0, i, g).index_add(0, j, -g)
                pv = pv + d.T @ g
        return f, vv, vc, pv

    def pme(self, x):
        """(force, vrecip, virial) of the reciprocal sum."""
        S, n = self.S, int(self.S["n_interp"])
        nc, nb, na = self.grid
        size = _t([na, nb, nc])
        xc, q = x[self.charged], self.q[self.charged]
        s = xc / self.h
        s = s - _nint((s - 0.5).detach())
        s = s * size
        i0 = s.detach().to(torch.int64)
        m, d = _bspline(s - i0.to(s.dtype), n)
        off = torch.arange(n, device=_DEV)
        idx = (i0[:, :, None] - off) % size.to(torch.int64)[:, None]
        flat = ((idx[:, 2, :, None, None] * nb + idx[:, 1, None, :, None]) * na + idx[:, 0, None, None, :])
        w = m[:, 2, :, None, None] * m[:, 1, None, :, None] * m[:, 0, None, None, :]
        grid = torch.zeros(na * nb * nc, dtype=x.dtype, device=x.device)
        grid = grid.index_add(0, flat.reshape(-1), (w * q[:, None, None, None]).reshape(-1)).reshape(self.grid)
        spec = torch.fft.fftn(grid)
        smag = spec.reshape(-1)[self.kidx].abs().square() * self.kbw
        v = (smag * self.preg).sum()
        pv = torch.einsum("k,ki,kj->ij", smag * self.kprep, self.kg, self.kg) + v * torch.eye(
            3, dtype=x.dtype, device=x.device)
        phi = (torch.fft.ifftn(spec * self.infl).real * float(na * nb * nc)).reshape(-1)[flat]
        fa = torch.einsum("pcba,pc,pb,pa->p", phi, m[:, 2], m[:, 1], d[:, 0]) * na
        fb = torch.einsum("pcba,pc,pb,pa->p", phi, m[:, 2], d[:, 1], m[:, 0]) * nb
        fc = torch.einsum("pcba,pc,pb,pa->p", phi, d[:, 2], m[:, 1], m[:, 0]) * nc
        force = -torch.stack([fa, fb, fc], -1) * (q / self.h)[:, None]
        return torch.zeros_like(x).index_add(0, self.charged, force), v, pv

    def intra(self, x):
        """(force, vecor, vbond, vbend, virial) of the excluded-pair correction, bonds and bends."""
        S = self.S
        f = torch.zeros_like(x)
        i, j = _t(S["ecor_j1"], torch.int64), _t(S["ecor_j2"], torch.int64)
        d = x[i] - x[j]
        r = (d * d).sum(-1).sqrt()
        grid = (float(S["ecor_rmin"]), float(S["ecor_dr"]), float(S["ecor_dri"]), int(S["ecor_nsplin"]))
        q2 = self.q[i] * self.q[j]
        vecor = (q2 * _spline(_t(S["ecor_cv0"]), r, *grid)).sum()
        g = d * (q2 * _spline(_t(S["ecor_cdv0"]), r, *grid))[:, None]
        f = f.index_add(0, i, g).index_add(0, j, -g)
        pv = d.T @ g

        def series(c, t, low):
            v = torch.zeros_like(t)
            for k in range(6, low - 1, -1):
                v = v * t + c[k]
            return v

        i, j = _t(S["bond_j1"], torch.int64), _t(S["bond_j2"], torch.int64)
        d = x[i] - x[j]
        r = (d * d).sum(-1).sqrt()
        t = r - self.bond_eq[0]
        vbond = series(self.bond_c, t, 0).sum()
        g = d * (-series(self.bond_dc, t, 1) / r)[:, None]
        f = f.index_add(0, i, g).index_add(0, j, -g)
        pv = pv + d.T @ g

        a1, a2, a3 = (_t(S["bend_j%d" % k], torch.int64) for k in (1, 2, 3))
        d1, d3 = x[a1] - x[a2], x[a3] - x[a2]
        r1, r3 = (d1 * d1).sum(-1).sqrt(), (d3 * d3).sum(-1).sqrt()
        cost = torch.clamp((d1 * d3).sum(-1) / (r1 * r3), -1.0, 1.0)
        sint = torch.clamp((1.0 - cost * cost).sqrt(), min=1e-8)
        bc, bs, bdc, bds = (self.bend[k] for k in ("c", "s", "dc", "ds"))
        sisum = series(bs, sint, 2) * sint
        vbend = (series(bc, cost, 0) + sisum * cost + bs[1] * sint).sum()
        dvs = series(bds, sint, 2) * cost + bds[1]
        pre = -(series(bdc, cost, 1) + sisum - dvs * cost / sint)
        f1 = (d3 / (r1 * r3)[:, None] - d1 * (cost / r1 ** 2)[:, None]) * pre[:, None]
        f3 = (d1 / (r1 * r3)[:, None] - d3 * (cost / r3 ** 2)[:, None]) * pre[:, None]
        f = f.index_add(0, a1, f1).index_add(0, a3, f3).index_add(0, a2, -(f1 + f3))
        pv = pv + d1.T @ f1 + d3.T @ f3
        return f, vecor, vbond, vbend, pv

    def constants(self):
        """(vself, vbgr, vlong)."""
        S, vol = self.S, self.h ** 3
        vself = -(self.q * self.q).sum() * S["alp_ewd"] * S["self_erf"] / math.sqrt(math.pi)
        vbgr = -0.5 * self.q.sum() ** 2 * math.pi / (S["alp_ewd"] ** 2 * vol)
        return vself, vbgr, self.clong / vol

    def bead(self, x):
        """(raw site forces, [vvdw, vcoul, vrecip, vecor, vbond, vbend], virial) of one bead."""
        f1, vv, vc, p1 = self.pairs(x)
        f2, vrec, p2 = self.pme(x)
        f3, vecor, vbond, vbend, p3 = self.intra(x)
        return f1 + f2 + f3, torch.stack([vv, vc, vrec, vecor, vbond, vbend]), p1 + p2 + p3

    def energy_force(self, pos):
        """Distributed forces [P, natm, 3], the energy vector and the bead-summed pressure tensor."""
        force, e, pv = [], 0.0, 0.0
        for b in range(self.P):
            f, eb, pb = self.bead(self.ghosts(_t(pos[b])))
            force.append(self.distribute(f))
            e, pv = e + eb, pv + pb
        P = float(self.P)
        vv, vc, vrec, vecor, vbond, vbend = (float(v) / P for v in e)
        vself, vbgr, vlong = (float(v) for v in self.constants())
        # the pressure tensor's lower half repeats the upper one
        pv = pv.cpu().numpy() + np.eye(3) * (vlong + vbgr) * P
        pv = np.triu(pv) + np.triu(pv, 1).T
        inter = vv + vc + vlong + vrec + vself + vbgr + vecor
        energies = np.array([vv + vc, vv + vlong, vc + vrec + vself + vbgr + vecor, vrec, vself, vbgr, vecor, vlong,
                             vbond, vbend, inter, vbond + vbend])
        return torch.stack(force).cpu().numpy(), energies, pv.reshape(9)


def _exact_eval(spec, pos, xmod):
    S = system.build_system(spec, pos)
    f, e, pv = _Exact(spec, S, pos, xmod).energy_force(pos)
    return {"force": f, "energies": e, "pvten": pv}


def _exact_grad(spec, seed):
    """dE = d(vintert + vintrat) / d theta and dF = fbar . dF / d theta by torch's reverse mode."""
    pos, xmod = _positions(spec)
    S = system.build_system(spec, pos)
    X = _Exact(spec, S, pos, xmod, params.tangents(spec, params.theta_of(spec.model), S))
    fbar = _fbar(pos, seed)
    dE, dF = torch.zeros_like(X.eps), torch.zeros_like(X.eps)

    def slope(v):
        (g,) = torch.autograd.grad(v, X.eps, allow_unused=True, retain_graph=True)
        return torch.zeros_like(X.eps) if g is None else g

    for b in range(X.P):
        x = X.ghosts(_t(pos[b]))
        f, _, _ = X.bead(x)
        dF += slope((X.distribute(f) * _t(fbar[b])).sum())
        # the energy's slope at fixed sites, and what the moving M sites do to it by their forces
        _, e, _ = X.bead(x.detach())
        dE += (slope(e.sum()) - slope((f.detach() * x).sum())) / X.P
    dE += slope(sum(X.constants()))
    return {"dE": dE.cpu().numpy(), "dF": dF.cpu().numpy()}


def _mode_matrices(P, modes):
    """(beads -> modes, modes -> beads, bead forces -> mode forces) of PINY's transforms as P x P matrices."""
    back = np.zeros((P, P))
    if modes == STAGING:
        for m in range(P):
            v = np.zeros(P + 1)
            v[m + 1] = 1.0
            v[P] += v[1]
            for ip in range(P - 1, 1, -1):
                v[ip] += (ip - 1.0) / ip * v[ip + 1] + v[1] / ip
            back[:, m] = v[1:]
    else:
        j = np.arange(P)
        back[:, 0] = 1.0
        back[:, P - 1] = (-1.0) ** j
        for k in range(1, P // 2):
            back[:, 2 * k - 1] = 2.0 * np.cos(2.0 * np.pi * j * k / P)
            back[:, 2 * k] = 2.0 * np.sin(2.0 * np.pi * j * k / P)
    return np.linalg.inv(back), back, back.T


def _chains(v, mass, c, state):
    """PINY's chain operator for one chain per coordinate: v [natm, 3], state (x, v) [len, num]."""
    on = np.asarray(c["inhc"]).T < c["num_nhc"]
    which = np.asarray(c["inhc"]).T[on]
    order = np.argsort(which)
    mn, gk, xn, vn = np.asarray(c["mass_nhc"]), np.asarray(c["gkt"]), state[0], state[1]
    kin = (mass[:, None] * v * v)[on][order]
    scale, last = np.ones_like(kin), len(mn) - 1
    fn = np.empty_like(mn)
    fn[0] = (kin - gk[0]) / mn[0]
    fn[1:] = (mn[:-1] * vn[:-1] ** 2 - gk[1:]) / mn[1:]
    for _ in range(int(c["nres_nhc"])):
        for w in c["wdti"]:
            vn[last] += fn[last] * w / 4
            for k in range(last - 1, -1, -1):
                a = np.exp(-w / 8 * vn[k + 1])
                vn[k] = vn[k] * a * a + w / 4 * fn[k] * a
            a = np.exp(-w / 2 * vn[0])
            scale, kin = scale * a, kin * a * a
            xn += vn * w / 2
            fn[0] = (kin - gk[0]) / mn[0]
            for k in range(last):
                a = np.exp(-w / 8 * vn[k + 1])
                vn[k] = vn[k] * a * a + w / 4 * fn[k] * a
                fn[k + 1] = (mn[k] * vn[k] ** 2 - gk[k + 1]) / mn[k + 1]
            vn[last] += fn[last] * w / 4
    out = v.copy()
    back = np.empty_like(scale)
    back[order] = scale
    out[on] *= back
    return out


def _exact_step(case, spec):
    pos, xmod = _positions(spec)
    S = system.build_system(spec, pos)
    st, v = _step_setup(case, spec, S)
    P, dt = spec.nbeads, st["dt"]
    to_modes, to_beads, force_modes = _mode_matrices(P, st["kind"])
    bm = st["bead_mass"][:, :, None]
    state = [(np.zeros_like(st["class_nhc"]["mass_nhc"]), np.zeros_like(st["class_nhc"]["mass_nhc"]))] + \
        [(np.zeros_like(st["bead_nhc"]["mass_nhc"]), np.zeros_like(st["bead_nhc"]["mass_nhc"])) for _ in range(P - 1)]

    def chains(v):
        return np.stack([_chains(v[b], st["mass"] if b == 0 else st["bead_mass"][b],
                                 st["class_nhc"] if b == 0 else st["bead_nhc"], state[b]) for b in range(P)])

    def forces(x, u):
        X = _Exact(spec, S, x, u[0])
        x = np.stack([X.ghosts(_t(x[b])).cpu().numpy() for b in range(P)])
        f, e, pv = X.energy_force(x)
        fk = st["prekf"][None, :, None] * st["path_eig"][:, None, None]
        fm = -2.0 * fk * u
        kin_harm, mode = float((fk * u * u).sum()), np.einsum("bni,bnj->ij", u, fm)
        f = f / P
        corr = np.einsum("bni,bnj->ij", x - u[0][None], f)
        akv = 0.5 * (3.0 * st["nfree_atoms"] / st["beta"] - np.trace(corr))
        tot = pv / P - corr.reshape(9)
        return x, np.einsum("mb,bni->mni", force_modes, f) + fm * st["wght_pimd"], e, kin_harm, akv, tot, mode.reshape(9)

    _, f, *_ = forces(pos, np.einsum("mb,bni->mni", to_modes, pos))
    v = chains(v)
    v = v + f * (dt / 2.0) / bm
    u = np.einsum("mb,bni->mni", to_modes, pos) + v * dt
    x, f, e, kin_harm, akv, tot, mode = forces(np.einsum("bm,mni->bni", to_beads, u), u)
    v = chains(v + f * (dt / 2.0) / bm)
    return {"x": x, "v": v, "f": f, "energies": e, "estimators": np.array([kin_harm, akv]), "pvten": tot,
            "pvten_tot": tot, "pvten_mode_tot": mode}


def exact(case, seed):
    if case["kind"] == "batch":
        parts = [_exact_eval(s, *_positions(s)) for s in _batch_specs(case, seed)]
        return {"forces": [p["force"] for p in parts], "energies": np.array([p["energies"] for p in parts]),
                "pvten": np.array([p["pvten"] for p in parts])}
    spec = _spec(case, seed)
    if case["kind"] == "grad":
        return _exact_grad(spec, seed)
    if case["kind"] == "step":
        return _exact_step(case, spec)
    pos, xmod = _positions(spec)
    if case["kind"] == "rebuild":
        moved = _moved(spec, pos, seed)
        return [_exact_eval(dataclasses.replace(spec), p, p.mean(axis=0) if spec.nbeads > 1 else None)
                for p in (moved, pos)]
    return _exact_eval(spec, pos, xmod)
