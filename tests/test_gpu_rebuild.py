"""The list rebuild where its kernels change path: water columns longer than
a CTA and than one chunk of sort keys, water groups whose union exceeds one
chunk of the prune, water counts that leave a group or cluster partly empty,
exclusions across clusters, static atoms.  Every interacting pair inside the
cutoff must be in the lists (periodic k-d trees), and no excluded pair or
pair of two static atoms."""
import numpy as np
import pytest

from dynamics_b200 import md, synth

from .coverage import covered_pairs
from .systems import mixed, water_only
from .test_gpu_lists import check_lists, run_until_rebuild

pytestmark = pytest.mark.gpu


def _cfg(rc, grid, **kw):
    return md.MdConfig(coulomb_cutoff=rc, lj_cutoff=rc, spme_alpha=synth.ewald_alpha(rc), spme_grid=grid,
                       integrator=md.LangevinMiddle(gamma=1.0), seed=3, **kw)


def _tiled(cell, nz, drop=0):
    """nz copies of a water box along z, the last ``drop`` waters left out."""
    box = float(cell["box_hi"][0])
    s = dict(cell)
    off = np.arange(nz)[:, None, None, None] * np.array([0.0, 0.0, box], np.float32)
    for k, o in (("water_pos", off), ("water_vel", 0.0 * off)):
        a = (cell[k][None] + o).reshape(-1, 3, 3).astype(np.float32)
        s[k] = a[:len(a) - drop]
    s["box_hi"] = np.array([box, box, nz * box], np.float32)
    return s


# 4 columns of about 43 (one warp), 600 (more than the CTA's 512 threads) and
# 1115 waters (more than one chunk of 1024 keys); the water counts are not
# multiples of a cluster (8) or a group (32)
@pytest.mark.parametrize("nz,drop", [(1, 171), (7, 1), (13, 0)])
def test_columns(gpu_lib, nz, drop):
    sysd = _tiled(synth.water_box(343, 21.7, seed=5), nz, drop)
    st = md.MdState(sysd, _cfg(8.0, (24, 24, 24 * nz)))
    check_lists(st, sysd, 8.0)
    run_until_rebuild(st, sysd, 8.0)
    st.close()


def test_union_of_several_prune_chunks(gpu_lib):
    sysd = water_only(n_side=12)
    st = md.MdState(sysd, _cfg(14.0, (36, 36, 36)))
    assert st.energies()["list_union_max"] > 1024
    run_until_rebuild(st, sysd, 14.0)
    assert st.energies()["list_prunes"] > st.energies()["list_rebuilds"]
    st.close()


@pytest.mark.parametrize("static", [False, True])
def test_masks(gpu_lib, static):
    sysd = mixed(n_mol=9, mol_len=7)
    na = len(sysd["atom_pos"])
    if static:
        sysd["atom_static"] = np.arange(na) % 3 != 0
    st = md.MdState(sysd, _cfg(8.0, (24, 24, 24)))
    check_lists(st, sysd, 8.0)
    got = covered_pairs(st, st.n_water, na)[2]
    skip = np.concatenate([np.asarray(sysd[k], np.int64).reshape(-1, 2) for k in ("excl", "pair14")])
    skip = np.minimum(skip[:, 0], skip[:, 1]) * na + np.maximum(skip[:, 0], skip[:, 1])
    assert not np.isin(got, skip).any()
    assert len(np.unique(got)) == len(st.list_pairs(2))
    if static:
        m = sysd["atom_static"]
        assert not (m[got // na] & m[got % na]).any()
    st.close()
