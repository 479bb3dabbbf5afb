"""Kernels at the sizes where they can go wrong, against the oracle: every mesh
edge the mesh transforms are compiled for, tiles of both edges, bead counts and
molecule counts around the pair kernels' chunks, boxes in which most molecule
pairs are near half a box, and the water staging and finishing kernels against
the general ones."""
import numpy as np
import pytest

from piny_b200 import params, system, water

pytestmark = pytest.mark.gpu

# FP64 follows the oracle's operation order up to summation order; MIXED
# evaluates pairs and mesh in FP32 (2^-24 per operation, a few hundred terms
# per force): the bounds of the parity tests
TOL = {"fp64": (1e-12, 1e-11), "mixed": (1e-5, 1e-6)}


def _box(model, nmol, beads, grid, order, seed=11, cutoff=None, edge=None):
    L = water.density_box_edge(nmol) if edge is None else edge
    spec = water.BoxSpec(model, nmol, L, beads, 298.0, seed, cutoff=cutoff or min(9.0, 0.47 * L), grid=grid,
                         order=order)
    pos = water.build_positions(spec) / water.BOHR
    return spec, system.build_system(spec, pos), pos, (pos.mean(axis=0) if beads > 1 else None)


def _oracle(oracle, S, pos, xmod, distribute=False):
    pi, pj = oracle.verlist(S, pos[0], xmod, S["hmat"], S["cutskin2"])
    f, e = oracle.energy_force(S, pos, xmod, S["hmat"], pi, pj, distribute_ghosts=distribute)
    return f, e


def _device(S, pos, xmod, precision, tuning=None, distribute=False):
    from piny_b200.lib import DeviceBox
    box = DeviceBox(S, pos.shape[0], precision)
    box.build_list(pos[0], xmod, S["hmat"], S["cutskin2"])
    if tuning:
        ch = box.tuning()
        for k, v in tuning.items():
            ch[k] = v
        box.set_tuning(ch)
    f, e = box.energy_force(pos, xmod, S["hmat"], distribute_ghosts=distribute)
    box.close()
    return f, e


def _check(precision, f, e, fref, eref):
    ftol, etol = TOL[precision]
    assert np.linalg.norm(f - fref) <= ftol * np.linalg.norm(fref)
    scale = abs(eref["vvdw"]) + abs(eref["vcoul"]) + abs(eref["vself"])
    for k in ("vintert", "vrecip", "vecor", "vbond", "vbend"):
        assert abs(e[k] - eref[k]) <= etol * scale, k
    assert np.abs(e["pvten"] - eref["pvten"]).max() <= 10 * etol * scale * f.shape[0]


@pytest.mark.parametrize("grid", [16, 20, 24, 32, 36, 40, 48, 60, 64, 72, 80, 96, 100, 108, 120, 128])
def test_mesh_edges(oracle, grid):
    spec, S, pos, xmod = _box(water.SPC_FW, 27, 1, grid, 6, edge=12.4, cutoff=5.5)
    assert S["ngrid_a"] == grid
    fref, eref = _oracle(oracle, S, pos, xmod)
    # a context refuses FP64 meshes above 117 points a side, as before these
    # transforms: a plane of the run-time-length ones does not fit a block
    for precision in ("fp64", "mixed") if grid <= 108 else ("mixed",):
        f, e = _device(S, pos, xmod, precision)
        _check(precision, f, e, fref, eref)


@pytest.mark.parametrize("order", [4, 5, 6, 7, 8, 10])
@pytest.mark.parametrize("tile", [8, 16])
def test_orders_and_tiles(oracle, order, tile):
    spec, S, pos, xmod = _box(water.TIP4P_F, 65, 2, 32, order)
    fref, eref = _oracle(oracle, S, pos, xmod)
    for precision in ("fp64", "mixed"):
        f, e = _device(S, pos, xmod, precision, tuning={0: tile})
        _check(precision, f, e, fref, eref)


@pytest.mark.parametrize("beads", [1, 2, 8, 32, 64])
@pytest.mark.parametrize("model, nmol, cutoff", [(water.TIP4P_F, 33, 4.5), (water.TIP4P_F, 64, 9.0),
                                                 (water.SPC_FW, 65, 9.0)])
def test_pairs_near_half_a_box(oracle, model, nmol, cutoff, beads):
    """Boxes of 10 to 12.5 Angstrom: with a cutoff beyond half the box every
    image decision matters, and each site pair has to get its own."""
    spec, S, pos, xmod = _box(model, nmol, beads, 16, 6, cutoff=cutoff)
    fref, eref = _oracle(oracle, S, pos, xmod, distribute=True)
    for precision in ("fp64", "mixed"):
        for variant in (0, 2):
            f, e = _device(S, pos, xmod, precision, tuning={1: variant}, distribute=True)
            _check(precision, f, e, fref, eref)


def _two_types(S):
    """The same box with its second half's bonds and bends under a second type
    of equal constants: not the one-type water of the fused kernels."""
    T = dict(S)
    T["nbond_typ"] = T["nbend_typ"] = 2
    T["bond_typ"] = np.array(S["bond_typ"]).copy()
    T["bond_typ"][len(T["bond_typ"]) // 2:] = 1
    T["bend_typ"] = np.array(S["bend_typ"]).copy()
    T["bend_typ"][len(T["bend_typ"]) // 2:] = 1
    for k in ("bond_eq", "bond_c", "bond_dc", "bend_eq", "bend_c", "bend_s", "bend_dc", "bend_ds"):
        T[k] = np.concatenate([S[k], S[k]])
    return T


def _turned(S):
    """The same box with bonds, bends and exclusion pairs listed backwards and turned round."""
    T = dict(S)
    for a, b in (("bond_j1", "bond_j2"), ("bend_j1", "bend_j3"), ("ecor_j1", "ecor_j2")):
        T[a], T[b] = np.ascontiguousarray(S[b][::-1]), np.ascontiguousarray(S[a][::-1])
    T["bend_j2"] = np.ascontiguousarray(S["bend_j2"][::-1])
    return T


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("model, nmol, beads", [(water.TIP4P_F, 65, 1), (water.TIP4P_F, 33, 4), (water.SPC_FW, 65, 2),
                                                (water.SPC_FW, 27, 64), (water.TIP4P_F, 27, 32)])
def test_water_kernels_equal_the_general_ones(model, nmol, beads, precision):
    import torch

    from piny_b200.lib import DeviceBox
    spec, S, pos, xmod = _box(model, nmol, beads, 20, 6)
    got = []
    for T in (S, _two_types(S), _turned(S)):
        for distribute in (False, True):
            got.append(_device(T, pos, xmod, precision, distribute=distribute))
        # without mode-1 positions: the bead centroid
        box = DeviceBox(T, beads, precision)
        box.build_list(pos[0], xmod, S["hmat"], S["cutskin2"])
        d = torch.from_numpy(pos).cuda()
        f = torch.full_like(d, float("nan"))
        e = box.energy_force_device(d.data_ptr(), None, S["hmat"], f.data_ptr(), distribute_ghosts=True, energy=False)
        got.append((f.cpu().numpy(), e))
        box.close()
    # FP64 sums in another order; in MIXED the same FP32 terms summed in FP64
    tol = 1e-13 if precision == "fp64" else 1e-9
    for k in range(3, 9):
        f0, e0 = got[k % 3]
        f, e = got[k]
        assert np.linalg.norm(f - f0) <= tol * np.linalg.norm(f0)
        scale = abs(e0["vreal"]) + abs(e0["vself"]) + 1.0
        assert abs(e["vintert"] - e0["vintert"]) <= 10 * tol * scale
        assert np.abs(e["pvten"] - e0["pvten"]).max() <= 100 * tol * scale * beads


@pytest.mark.parametrize("nmol, beads, cutoff", [(65, 1, None), (64, 4, 9.0), (130, 16, None), (27, 64, None)])
def test_gradient_pair_kernels(nmol, beads, cutoff):
    """The molecule-pair adjoint (MIXED), the site-list one (MIXED, two bond
    types) and FP64 give the same derivatives."""
    import torch

    from piny_b200.lib import DeviceBox
    spec, S, pos, xmod = _box(water.TIP4P_F, nmol, beads, 20, 6, cutoff=cutoff)
    tan = params.tangents(spec, params.theta_of(spec.model), S)
    tan2 = [{k: (np.concatenate([v, v]) if k.startswith(("dbond", "dbend")) else v) for k, v in t.items()}
            for t in tan]
    rng = np.random.default_rng(3)
    d, x = torch.from_numpy(pos).cuda(), None if xmod is None else torch.from_numpy(xmod).cuda()
    fbar = torch.from_numpy(rng.normal(size=pos.shape)).cuda()
    out = []
    for T, t, precision in ((S, tan, "fp64"), (S, tan, "mixed"), (_two_types(S), tan2, "mixed")):
        box = DeviceBox(T, beads, precision)
        box.build_list(pos[0], xmod, S["hmat"], S["cutskin2"])
        box.grad_prepare(t)
        out.append(box.grad(d.data_ptr(), None if x is None else x.data_ptr(), S["hmat"], fbar.data_ptr()))
        box.close()
    for dE, dF in out[1:]:
        # FP32 pair and mesh terms: 1e-6 of the largest component, single ones within 1e-3 of it as elsewhere
        assert np.abs(dE - out[0][0]).max() <= 1e-5 * np.abs(out[0][0]).max()
        assert np.abs(dF - out[0][1]).max() <= 1e-5 * np.abs(out[0][1]).max()


@pytest.mark.parametrize("nsplin", [2000, 4096, 4097, 9000])
@pytest.mark.parametrize("model,nmol,beads", [(water.TIP4P_F, 700, 4), (water.SPC_FW, 300, 8), (water.TIP4P_F, 300, 16),
                                              (water.TIP4P_F, 300, 32), (water.SPC_FW, 216, 64)])
def test_pair_tables_in_shared_memory(oracle, model, nmol, beads, nsplin):
    # boxes large enough for the one-block-per-SM kernel; tables that fit its shared memory up to the
    # last point, and ones that do not
    L = water.density_box_edge(nmol)
    spec = water.BoxSpec(model, nmol, L, beads, 298.0, 5, cutoff=min(9.0, 0.45 * L), grid=24, order=6, nsplin=nsplin)
    pos = water.build_positions(spec) / water.BOHR
    S = system.build_system(spec, pos)
    xmod = pos.mean(axis=0)
    fref, eref = _oracle(oracle, S, pos, xmod)
    f, e = _device(S, pos, xmod, "mixed")
    _check("mixed", f, e, fref, eref)


@pytest.mark.parametrize("nmol,beads", [(65, 32), (700, 32), (700, 64)])
def test_fp64_pairs_by_chunk_queue(oracle, nmol, beads):
    # fewer and more than two chunks to a warp
    spec, S, pos, xmod = _box(water.TIP4P_F, nmol, beads, 24, 6)
    fref, eref = _oracle(oracle, S, pos, xmod)
    f, e = _device(S, pos, xmod, "fp64", tuning={2: 1})
    _check("fp64", f, e, fref, eref)


@pytest.mark.parametrize("model, nmol, beads", [(water.SPC_FW, 65, 1), (water.SPC_FW, 64, 16), (water.TIP4P_F, 65, 1),
                                                (water.TIP4P_F, 64, 16)])
def test_gradient_of_tables_without_a_term(oracle, model, nmol, beads):
    """A table tangent on the table that is zero in the model (the slope along a
    term not there yet), alone and together with one on the O-O table: the same
    derivatives in MIXED and FP64, and where every site pair is charged, so that
    every one of them is listed, the oracle's difference quotient (energy and
    forces are linear in the tables)."""
    import torch

    from piny_b200.lib import DeviceBox
    spec, S, pos, xmod = _box(model, nmol, beads, 20, 6)
    ns, nu = int(S["nsplin"]), int(S["ninter_unique"])
    null = [u for u in range(nu) if not np.any(np.asarray(S["cv0"])[u * ns:(u + 1) * ns])]
    assert len(null) == 1 and nu == 2
    r = float(S["rmin_spl"][0]) + float(S["dr_spl"][0]) * np.arange(-2, ns - 2)
    v, dv = np.exp(-0.3 * r), 0.3 * np.exp(-0.3 * r) / r

    def on(tables):
        return {"dcv0": np.concatenate([v if u in tables else 0 * v for u in range(nu)]),
                "dcdv0": np.concatenate([dv if u in tables else 0 * v for u in range(nu)])}

    tan = [on(null), on([0, 1]), on([1 - null[0]])]
    d, x = torch.from_numpy(pos).cuda(), None if xmod is None else torch.from_numpy(xmod).cuda()
    fbar = np.random.default_rng(3).normal(size=pos.shape)
    dfbar = torch.from_numpy(fbar).cuda()
    out = {}
    for precision in ("fp64", "mixed"):
        box = DeviceBox(S, beads, precision)
        box.build_list(pos[0], xmod, S["hmat"], S["cutskin2"])
        box.grad_prepare(tan)
        out[precision] = box.grad(d.data_ptr(), None if x is None else x.data_ptr(), S["hmat"], dfbar.data_ptr())
        box.close()
    for got, ref in zip(out["mixed"], out["fp64"]):
        assert np.all(ref != 0.0)
        assert np.all(np.abs(got - ref) <= 1e-5 * np.abs(ref))
    if model is not water.SPC_FW:
        return
    pi, pj = oracle.verlist(S, pos[0], xmod, S["hmat"], S["cutskin2"])
    f0, e0 = oracle.energy_force(S, pos, xmod, S["hmat"], pi, pj, distribute_ghosts=True)
    for k, t in enumerate(tan):
        T = dict(S, cv0=np.asarray(S["cv0"]) + t["dcv0"], cdv0=np.asarray(S["cdv0"]) + t["dcdv0"])
        f1, e1 = oracle.energy_force(T, pos, xmod, S["hmat"], pi, pj, distribute_ghosts=True)
        dE, dF = e1["vintert"] - e0["vintert"], float(((f1 - f0) * fbar).sum())
        # both are differences of sums of this size, to 1e-13 of it
        escale = abs(e0["vreal"]) + abs(e0["vself"]) + abs(dE)
        assert abs(out["fp64"][0][k] - dE) <= 1e-12 * escale
        assert abs(out["fp64"][1][k] - dF) <= 1e-12 * np.abs(f1 * fbar).sum()


def _pairs_only(S):
    """Without bonds, bends and exclusion correction, which see no images."""
    return dict(S, nbond=0, nbend=0, necor=0, nghost=0)


@pytest.mark.parametrize("model, nmol, cutoff", [(water.SPC_FW, 64, 5.5), (water.TIP4P_F, 65, 5.5),
                                                 (water.SPC_FW, 130, 9.0)])
@pytest.mark.parametrize("beads", [1, 2, 8, 32, 64])
def test_sites_in_different_cells(oracle, model, nmol, cutoff, beads):
    """Every site moved by lattice vectors of its own, as a program does that
    wraps atoms one by one: a site pair's shift then differs from its molecules'
    first sites' by up to four cells, and its image is what it was."""
    spec, S, pos, xmod = _box(model, nmol, beads, 20, 6, cutoff=cutoff)
    S = _pairs_only(S)
    h = float(S["hmat"][0])
    n = np.random.default_rng(5).integers(-1, 2, size=(pos.shape[1], 3))
    moved = pos + h * n[None]
    xm = None if xmod is None else xmod + h * n
    f0, e0 = _oracle(oracle, S, pos, xmod)
    fref, eref = _oracle(oracle, S, moved, xm)
    assert np.linalg.norm(fref - f0) <= 1e-9 * np.linalg.norm(f0)
    for precision in ("fp64", "mixed"):
        for variant in (0, 2, 1):
            f, e = _device(S, moved, xm, precision, tuning={1: variant})
            _check(precision, f, e, fref, eref)
            if precision == "fp64":
                break


def test_gradient_with_sites_in_different_cells():
    """As above for the pair adjoint: each molecule's sites stay together for
    bonds and exclusions, so one molecule of every three is moved as a whole and
    the rest by sites would break them; whole cells' moves of whole molecules
    leave every derivative as it was."""
    import torch

    from piny_b200.lib import DeviceBox
    spec, S, pos, xmod = _box(water.TIP4P_F, 65, 8, 20, 6)
    h = float(S["hmat"][0])
    n = np.repeat(np.random.default_rng(5).integers(-2, 3, size=(65, 3)), 4, axis=0)
    tan = params.tangents(spec, params.theta_of(spec.model), S)
    fbar = torch.from_numpy(np.random.default_rng(3).normal(size=pos.shape)).cuda()
    out = []
    for p, x in ((pos, xmod), (pos + h * n[None], xmod + h * n)):
        box = DeviceBox(S, 8, "mixed")
        box.build_list(p[0], x, S["hmat"], S["cutskin2"])
        box.grad_prepare(tan)
        d, dx = torch.from_numpy(p).cuda(), torch.from_numpy(x).cuda()
        out.append(box.grad(d.data_ptr(), dx.data_ptr(), S["hmat"], fbar.data_ptr()))
        box.close()
    for a, b in zip(*out):
        assert np.abs(a - b).max() <= 1e-6 * np.abs(a).max()


@pytest.mark.parametrize("model, nmol, beads, cutoff", [(water.SPC_FW, 65, 1, None), (water.SPC_FW, 216, 8, 5.0),
                                                        (water.TIP4P_F, 216, 1, 5.0), (water.TIP4P_F, 300, 32, None),
                                                        (water.TIP4P_F, 64, 4, 9.0)])
@pytest.mark.parametrize("apart", [0.6, 0.0])
def test_pairs_closer_than_the_tables(oracle, model, nmol, beads, cutoff, apart):
    """Two hydrogens nearer than the tables' first point, down to the same place:
    PINY continues the first interval's cubic there."""
    import torch

    from piny_b200.lib import DeviceBox
    spec, S, pos, xmod = _box(model, nmol, beads, 24, 6, cutoff=cutoff)
    ns, last = spec.model.nsite, spec.nmol - 1
    r = float(S["rmin_spl"][0])
    # the last molecule: the first one's mirror image in a point half of `apart` rmin beyond its first hydrogen
    out = pos[:, 1] - pos[:, 0]
    c = pos[:, 1] + 0.5 * apart * r * out / np.linalg.norm(out, axis=1, keepdims=True)
    pos[:, last * ns:] = 2.0 * c[:, None, :] - pos[:, :ns]
    xmod = None if xmod is None else pos.mean(axis=0)
    fref, eref = _oracle(oracle, S, pos, xmod, distribute=True)
    force, grads = {}, {}
    tan = None if ns == 3 else params.tangents(spec, params.theta_of(spec.model), S)
    for precision in ("fp64", "mixed"):
        force[precision], e = _device(S, pos, xmod, precision, distribute=True)
        escale = abs(eref["vreal"]) + abs(eref["vself"])
        assert abs(e["vintert"] - eref["vintert"]) <= (1e-11 if precision == "fp64" else 1e-4) * escale
        if ns == 3 or apart == 0.0:  # at r = 0 the derivative along a moving M site has no value
            continue
        box = DeviceBox(S, beads, precision)
        box.build_list(pos[0], xmod, S["hmat"], S["cutskin2"])
        box.grad_prepare(tan)
        d, x = torch.from_numpy(pos).cuda(), None if xmod is None else torch.from_numpy(xmod).cuda()
        fbar = torch.from_numpy(np.random.default_rng(3).normal(size=pos.shape)).cuda()
        grads[precision] = box.grad(d.data_ptr(), None if x is None else x.data_ptr(), S["hmat"], fbar.data_ptr())
        box.close()
    norm = np.linalg.norm(fref)
    assert np.linalg.norm(force["fp64"] - fref) <= 1e-12 * norm
    # FP32 separations are sums of three values up to the box edge L, each
    # rounded to 2^-24: 3 L 2^-24 of the pair's r = 0.11 Bohr, up to 1e-4
    assert np.linalg.norm(force["mixed"] - fref) <= 1e-4 * norm
    for a, b in zip(grads.get("mixed", ()), grads.get("fp64", ())):
        assert np.abs(a - b).max() <= 1e-4 * np.abs(b).max()


@pytest.mark.parametrize("nmol, beads, grid, bound", [(216, 8, 32, 3e-6), (4096, 2, 64, 4e-6)])
def test_mesh_forces_resolve_small_weights(nmol, beads, grid, bound):
    """Mesh forces alone (no pair tables): MIXED within the rounding of a spread at
    2^-25 (2.1e-6 and 2.8e-6 of the mesh force; 4.0e-6 and 5.4e-6 at 2^-24)."""
    spec, S, pos, xmod = _box(water.TIP4P_F, nmol, beads, grid, 8, seed=3)
    S = dict(S, nbond=0, nbend=0, necor=0, **{k: 0.0 * np.asarray(S[k]) for k in ("cv0", "cdv0", "cv0_c", "cdv0_c")})
    f64, _ = _device(S, pos, xmod, "fp64")
    f32, _ = _device(S, pos, xmod, "mixed")
    assert np.linalg.norm(f32 - f64) <= bound * np.linalg.norm(f64)


@pytest.mark.parametrize("nmol, beads", [(216, 1), (216, 8), (130, 32)])
def test_gradient_under_a_common_force(nmol, beads):
    """An upstream gradient with a large common part, which no force sum sees:
    it cancels in the FP64 differences of the pair adjoint (without the mesh,
    whose FP32 spread holds the common part)."""
    import torch

    from piny_b200.lib import DeviceBox
    spec, S, pos, xmod = _box(water.TIP4P_F, nmol, beads, 20, 6, seed=5)
    S = dict(S, nktot=0)
    tan = params.tangents(spec, params.theta_of(spec.model), S)
    d, x = torch.from_numpy(pos).cuda(), None if xmod is None else torch.from_numpy(xmod).cuda()
    fbar = torch.from_numpy(1e4 + np.random.default_rng(3).normal(size=pos.shape)).cuda()
    out = []
    for precision in ("fp64", "mixed"):
        box = DeviceBox(S, beads, precision)
        box.build_list(pos[0], xmod, S["hmat"], S["cutskin2"])
        box.grad_prepare(tan)
        out.append(box.grad(d.data_ptr(), None if x is None else x.data_ptr(), S["hmat"], fbar.data_ptr())[1])
        box.close()
    # FP32 pair terms: 1e-6 of a component, up to 1e-5 of one that is small by
    # cancellation; differences of u rounded to FP32 were 5e-5 to 9e-3 off
    assert np.all(np.abs(out[1] - out[0]) <= 3e-5 * np.abs(out[0]))


def _atoms(n, edge, cutoff, beads, seed):
    """A fluid of one-site molecules with the O-O term of q-SPC/Fw and no charges (Bohr)."""
    spec = water.BoxSpec(water.SPC_FW, n, edge, beads, 298.0, seed, cutoff=cutoff, grid=16, order=6)
    W = system.build_system(spec, water.build_positions(spec) / water.BOHR)
    S = dict(W, natm=n, atm_typ=np.zeros(n, np.int32), charge=np.zeros(n), excl_off=np.zeros(n + 1, np.int32),
             excl_j=np.zeros(1, np.int32), nktot=0, necor=0, nbond=0, nbend=0, nghost=0)
    rng = np.random.default_rng(seed)
    g = int(np.ceil(n ** (1 / 3)))
    cell = np.stack(np.meshgrid(*[np.arange(g)] * 3, indexing="ij"), -1).reshape(-1, 3)[:n] * (edge / g)
    pos = cell[None] + rng.normal(scale=0.05, size=(beads, n, 3))
    return S, pos / water.BOHR


@pytest.mark.parametrize("beads", [1, 8, 32])
def test_device_rebuild_keeps_its_room(beads):
    """A denser configuration whose pairs still fit the reserved lists (a quarter
    and 1024 more than at the host build): the chunks cut from it fit theirs."""
    import torch

    from piny_b200.lib import DeviceBox
    S, pos = _atoms(216, 30.0, 5.0, beads, 3)
    closer = pos * 0.8 + 1.0
    xmod, xm2 = (pos.mean(axis=0), closer.mean(axis=0)) if beads > 1 else (None, None)
    box = DeviceBox(S, beads, "fp64")
    n0 = box.build_list(pos[0], xmod, S["hmat"], S["cutskin2"])
    box.list_set_spread(0.0)
    d = torch.from_numpy(closer).cuda()
    dx = None if xm2 is None else torch.from_numpy(xm2).cuda()
    f = torch.zeros_like(d)
    e = box.energy_force_device(d.data_ptr(), None if dx is None else dx.data_ptr(), S["hmat"], f.data_ptr(),
                                update_list=True)
    st = box.list_status()
    assert st["rebuilt_last"] == 1 and n0 * 1.25 + 300 < st["npairs"] < n0 * 1.25 + 1024
    fresh = DeviceBox(S, beads, "fp64")
    fresh.build_list(closer[0], xm2, S["hmat"], S["cutskin2"])
    fref, eref = fresh.energy_force(closer, xm2, S["hmat"])
    assert np.linalg.norm(f.cpu().numpy() - fref) <= 1e-12 * np.linalg.norm(fref)
    assert abs(e["vintert"] - eref["vintert"]) <= 1e-11 * abs(eref["vintert"])
    box.close()
    fresh.close()
