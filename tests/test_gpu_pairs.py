"""The pair kernels where their paths change: a water group's union cut into
parts and chunks of every size, forces too large for the water-water kernel's
32-bit j sums, odd water counts, batch members that differ in cutoff.  Forces
against the float64 oracle (per-atom relative RMS <= 1e-5, the engine's
specification), virials to 1e-5 of the sum's largest part."""
import numpy as np
import pytest

from dynamics_b200 import md, synth

from .systems import mixed, rel_rms, water_only
from .test_gpu_native import FORCE_RTOL, PE_RTOL, _cfg, _compare, _oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("split,chunk", [(1, 0), (1, 32), (1, 160), (2, 0), (3, 64), (5, 32), (8, 0), (8, 32)])
@pytest.mark.parametrize("mode", ["reference", "corrected"])
def test_water_water_parts(gpu_lib, split, chunk, mode):
    sysd = water_only()
    sysd["water_pos"] = sysd["water_pos"][:-5]  # 338 waters: a partly empty group
    sysd["water_vel"] = sysd["water_vel"][:-5]
    cfg = _cfg(sysd, mode, ww_split=split, ww_union_chunk=chunk)
    st = md.MdState(sysd, cfg)
    got = st.forces()
    ref = _oracle(sysd, cfg, st)
    assert _compare(got, ref) < FORCE_RTOL
    assert abs(got["potential"] - ref["pe"]) <= PE_RTOL * abs(ref["pe"])
    # after steps with prunes the parts' list offsets are the prune kernel's
    st.step(0.002, 30)
    s = st.state()
    assert st.energies()["list_prunes"] > st.energies()["list_rebuilds"]
    got = st.forces()
    ref = _oracle({**sysd, "water_pos": s["water_pos"]}, cfg, st)
    assert _compare(got, ref) < FORCE_RTOL
    st.close()


@pytest.mark.parametrize("distance", [1.3, 1.7])
def test_large_forces(gpu_lib, distance):
    """Two waters too close: some of their site forces exceed what the 32-bit
    sums hold (1000 kcal/mol/A); the others must not suffer."""
    sysd = water_only()
    wp = sysd["water_pos"].copy()
    for i, j in ((3, 4), (200, 120)):
        wp[j] += wp[i, 0] + np.float32(distance / np.sqrt(3.0)) - wp[j, 0]
    sysd["water_pos"] = wp
    st = md.MdState(sysd, _cfg(sysd))
    got = st.forces()
    ref = _oracle(sysd, st.cfg, st)
    assert np.abs(ref["f_water"]).max() > 1000.0
    close = np.array([3, 4, 200, 120])
    far = np.setdiff1d(np.arange(st.n_water), close)
    assert rel_rms(got["f_water"][close], ref["f_water"][close]) < FORCE_RTOL
    # float32 sums on the far waters hold no term above the largest pair force
    # they take part in
    assert rel_rms(got["f_water"][far], ref["f_water"][far]) < FORCE_RTOL
    st.close()


def test_batch_members_of_other_cutoffs(gpu_lib):
    systems = [water_only(), mixed(), mixed(seed=4)]
    cfgs = [_cfg(s, spme_interval=1, ww_split=1, seed=7) for s in systems]
    cfgs[1].coulomb_cutoff = cfgs[1].lj_cutoff = 7.5
    cfgs[2].spme_alpha = 0.37
    b = md.MdBatch(systems, cfgs)
    b.step(0.001, 6)
    for m, s, c in zip(b.members, systems, cfgs):
        alone = md.MdState(s, c)
        alone.step(0.001, 6)
        want, got = alone.state(), m.state()
        for k in want:
            np.testing.assert_array_equal(got[k], want[k])
        alone.close()
    b.close()


@pytest.mark.parametrize("n_side,mol_len", [(7, 5), (19, 5), (19, 0)])
def test_forces_output(gpu_lib, n_side, mol_len):
    """The forces handed to the host, at a size that passes through the
    device's scratch at once and at one that takes two turns (6,314 waters a
    turn): against the oracle; the same bits from a second call, whose energies
    come from the partial sums the scratch shares, and for each output alone."""
    from dynamics_b200 import _lib

    sysd = mixed(n_side=n_side, mol_len=mol_len) if mol_len else water_only(n_side)
    cfg = _cfg(sysd, "corrected")
    st = md.MdState(sysd, cfg)
    st.step(0.001, 3)
    got = st.forces()
    s = st.state()
    ref = _oracle({**sysd, "water_pos": s["water_pos"], "atom_pos": s["atom_pos"]}, cfg, st)
    assert _compare(got, ref) < FORCE_RTOL
    again = st.forces()
    for k in got:
        np.testing.assert_array_equal(got[k], again[k])
    for k in ("f_atoms", "f_water"):
        part = np.full_like(got[k], np.nan)
        a, w = (_lib.ptr(part), None) if k == "f_atoms" else (None, _lib.ptr(part))
        _lib.check(_lib.lib().dyn_sys_forces(st.handle, a, w, None))
        np.testing.assert_array_equal(part, got[k])
    st.close()
