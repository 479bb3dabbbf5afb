"""Graph replay of the single-box entry points.

A call with the same pointers, cell, flags and stream as the one before is
a replay of one captured CUDA graph; the inputs behind the pointers may
change between calls.  Every call (plain, captured, replayed) must give the
oracle's forces and energies for the positions it was given: FP64 relative
RMS 1e-12.
"""
import numpy as np
import pytest

from helpers import load_fixture, rel_rms, respa_from_fixture

pytestmark = pytest.mark.gpu


def test_replayed_evaluations_follow_the_inputs(oracle):
    import torch

    from piny_b200.lib import DeviceBox

    F = load_fixture("tip4pf_64_p4")
    P = int(F["nbeads"])
    xmod = F["xmod"]
    box = DeviceBox(F, P, "fp64")
    box.build_list(F["pos"][0], xmod, F["hmat"], F["cutskin2"])
    pi, pj = box.get_list()
    rng = np.random.default_rng(3)
    inputs = [F["pos"] + rng.normal(scale=0.01, size=F["pos"].shape) for _ in range(4)]
    dev = torch.device("cuda:0")
    d = torch.from_numpy(np.ascontiguousarray(inputs[0])).to(dev)
    dx = torch.from_numpy(np.ascontiguousarray(xmod)).to(dev)
    f = torch.zeros_like(d)
    for k in [0, 0, 1, 2, 3, 1]:  # plain, captured, then replays with new contents
        d.copy_(torch.from_numpy(inputs[k]))
        e = box.energy_force_device(d.data_ptr(), dx.data_ptr(), F["hmat"], f.data_ptr())
        fref, eref = oracle.energy_force(F, inputs[k], xmod, F["hmat"], pi, pj)
        assert rel_rms(f.cpu().numpy(), fref) < 1e-12, k
        assert abs(e["vintert"] - eref["vintert"]) <= 1e-11 * max(1.0, abs(eref["vintert"])), k
        assert abs(e["vintrat"] - eref["vintrat"]) <= 1e-11 * max(1.0, abs(eref["vintrat"])), k
        assert box.last_timing()[0] > 0.0
    # the host-buffer entry replays its own graph the same way
    for k in [2, 2, 0, 3]:
        fh, eh = box.energy_force(inputs[k], xmod, F["hmat"])
        fref, eref = oracle.energy_force(F, inputs[k], xmod, F["hmat"], pi, pj)
        assert rel_rms(fh, fref) < 1e-12, k
        assert abs(eh["vintert"] - eref["vintert"]) <= 1e-11 * max(1.0, abs(eref["vintert"])), k
    # a new cell is a new graph
    h2 = np.asarray(F["hmat"]) * 1.002
    for k in [1, 1, 1]:
        fh, eh = box.energy_force(inputs[k], xmod, h2)
        fref, eref = oracle.energy_force(F, inputs[k], xmod, h2, pi, pj)
        assert rel_rms(fh, fref) < 1e-12
    box.close()


def _two_cells(F):
    return np.asarray(F["hmat"]), np.asarray(F["hmat"]) * 1.004


@pytest.mark.parametrize("entry", ["device", "host"])
def test_replay_after_another_cell(oracle, entry):
    """Cells A, A, A, B, A, as in a rejected volume move: the influence function
    belongs to the last cell evaluated, the graph to the one before."""
    import torch

    from piny_b200.lib import DeviceBox

    F = load_fixture("tip4pf_64_p4")
    A, B = _two_cells(F)
    xmod = F["xmod"]
    box = DeviceBox(F, int(F["nbeads"]), "fp64")
    box.build_list(F["pos"][0], xmod, A, F["cutskin2"])
    pi, pj = box.get_list()
    ref = {id(h): oracle.energy_force(F, F["pos"], xmod, h, pi, pj) for h in (A, B)}
    d = torch.from_numpy(np.ascontiguousarray(F["pos"])).cuda()
    dx = torch.from_numpy(np.ascontiguousarray(xmod)).cuda()
    f = torch.zeros_like(d)
    for k, h in enumerate([A, A, A, B, A, A, B, B, B, A]):
        if entry == "device":
            e = box.energy_force_device(d.data_ptr(), dx.data_ptr(), h, f.data_ptr())
            got = f.cpu().numpy()
        else:
            got, e = box.energy_force(F["pos"], xmod, h)
        fref, eref = ref[id(h)]
        assert rel_rms(got, fref) < 1e-12, k
        assert abs(e["vrecip"] - eref["vrecip"]) <= 1e-11 * abs(eref["vrecip"]), k
    box.close()


@pytest.mark.parametrize("branches", [True, False])
def test_batch_replay_after_another_cell(oracle, branches):
    """A batch's graph replayed after one of its boxes was evaluated at another cell."""
    import torch

    from piny_b200.lib import DeviceBatch, DeviceBox

    F = load_fixture("tip4pf_64_p4")
    A, B = _two_cells(F)
    P, xmod = int(F["nbeads"]), F["xmod"]
    prec, tol = ("fp64", 1e-12) if branches else ("mixed", 1e-5)
    boxes = [DeviceBox(F, P, prec) for _ in range(2)]
    for b in boxes:
        b.build_list(F["pos"][0], xmod, A, F["cutskin2"])
    pi, pj = boxes[0].get_list()
    fref, eref = oracle.energy_force(F, F["pos"], xmod, A, pi, pj)
    d = torch.from_numpy(np.ascontiguousarray(F["pos"])).cuda()
    dx = torch.from_numpy(np.ascontiguousarray(xmod)).cuda()
    f = [torch.zeros_like(d) for _ in boxes]
    batch = DeviceBatch(boxes)
    args = ([d.data_ptr()] * 2, [dx.data_ptr()] * 2, [A, A], [t.data_ptr() for t in f])
    for k in range(4):
        if k >= 2:
            boxes[1].energy_force(F["pos"], xmod, B)
        es = batch.energy_force_device(*args, branches=branches, kernels=not branches)
        for i in range(2):
            assert rel_rms(f[i].cpu().numpy(), fref) < tol, (k, i)
            assert abs(es[i]["vrecip"] - eref["vrecip"]) <= 10 * tol * abs(eref["vrecip"]), (k, i)
    batch.close()
    for b in boxes:
        b.close()


@pytest.mark.parametrize("name", ["tip4pf_64_p4", "respa_pmegrid_tip4pf_64_p4"])
def test_step_replay_after_another_cell(name):
    """A ring-polymer trajectory with the force context used at another cell
    between its steps equals the one without (graph replays from step 3 on;
    with RESPA, the influence functions of both meshes)."""
    import torch

    from piny_b200 import pimd, water
    from piny_b200 import respa as R
    from piny_b200.lib import NORMAL_MODES, DeviceBox, DevicePimd

    F = load_fixture(name)
    A, B = _two_cells(F)
    P, natm, pos, xmod = int(F["nbeads"]), int(F["natm"]), F["pos"], F["xmod"]
    respa = name.startswith("respa")
    ghost = np.zeros(natm, bool)
    ghost[np.asarray(F["ghost_atom"])] = True
    mass = np.tile(np.asarray(water.TIP4P_F.masses, np.float64), natm // 4) * 1822.888486
    setup = pimd.nvt_setup(mass, ghost, P, NORMAL_MODES, 298.0, 20.0, 800.0, len_nhc=3, nyosh=3)
    if respa:
        setup["nres"] = (2, 1, 2, 1)
    v0 = np.random.default_rng(5).normal(size=pos.shape) * np.sqrt(298.0 / water.BOLTZ / setup["bead_mass"])[:, :, None]
    v0[:, ghost, :] = 0.0
    runs = []
    for disturb in (False, True):
        box = DeviceBox(F, P, "fp64")
        box.build_list(pos[0], xmod, A, F["cutskin2"])
        if respa:
            box.set_respa(respa_from_fixture(F))
        pm = DevicePimd(setup)
        dx, dv = torch.from_numpy(pos.copy()).cuda(), torch.from_numpy(v0.copy()).cuda()
        df, d0 = torch.zeros_like(dx), torch.from_numpy(pos.copy()).cuda()
        pm.forces(box, dx.data_ptr(), df.data_ptr(), A)
        for step in range(5):
            if disturb and step >= 3:
                box.energy_force(pos, xmod, B)
                if respa:
                    f0 = torch.zeros_like(d0)
                    box.respa_force_device(d0.data_ptr(), None, B, R.FULL_INTER | R.RES_INTER | R.FULL_INTRA,
                                           f0.data_ptr())
            e = pm.step(box, dx.data_ptr(), dv.data_ptr(), df.data_ptr(), A)
        runs.append((df.cpu().numpy(), dv.cpu().numpy(), e["vrecip"]))
        pm.close()
        box.close()
    # sums of atomics in another order, five steps long
    assert rel_rms(runs[1][0], runs[0][0]) < 1e-11
    assert rel_rms(runs[1][1], runs[0][1]) < 1e-11
    assert abs(runs[1][2] - runs[0][2]) <= 1e-11 * abs(runs[0][2])
