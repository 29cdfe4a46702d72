"""The list build by molecule gives the rows of the build by cell: the same
partners in the same order, so forces agree to the last bit.  Its three lane
counts (8, 16 and 32 a molecule, by density), boxes of three cells per axis
(every cell at a face), molecules exactly on the lower faces (binned in halo
cells), cells of more than 32 and more than 128 molecules, bonds, both sides of
the size where the build by warp takes over, and rows that overflow."""
import numpy as np
import pytest

from flowmol_b200 import api, lattice, polymer
from helpers import WCA_RC

pytestmark = pytest.mark.gpu


def _setup(r, v, dom, rc, mode, mono=None, **kw):
    p = api.make_params(len(r), dom, rc, list_build=mode, threads_per_molecule=1, **kw)
    s = api.MDSystem(p)
    s.upload(r, v)
    if mono is not None:
        s.upload_monomers(*mono)
    s.setup()
    out = list(s.pair_list()) + [s.download()[2]] + (list(s.bonds()) if mono is not None else [])
    s.close()
    return out


CASES = {
    "three_cells": ([5, 6, 5], 0.7, 2.5),
    "lanes_8": ([8, 8, 8], 0.8, WCA_RC),
    "lanes_16": ([9, 10, 8], 0.8, 1.45),
    "lanes_32": ([16, 17, 15], 0.8442, 2.5),
    "below_the_line": ([25, 25, 26], 0.8, WCA_RC),
    "above_the_line": ([26, 25, 27], 0.8442, 2.5),
    "cells_of_60": ([14, 13, 15], 0.8442, 3.9),
    "cells_of_300": ([13, 13, 13], 1.78, 5.3),
    "faces": ([7, 7, 7], 0.8, WCA_RC),
    "faces_dense": ([9, 9, 9], 0.8442, 2.5),
}


@pytest.mark.parametrize("name", sorted(CASES))
def test_rows_equal_the_build_by_cell(gpu_lib, name):
    nu, rho, rc = CASES[name]
    r, v, dom = lattice.lj_fluid(nu, rho, 1.0, 81)
    if name.startswith("faces"):
        r = r - r.min(axis=0) - 0.5 * np.asarray(dom)
    else:
        r = lattice.jitter(r, 0.04, 82, dom)
    for x, y in zip(_setup(r, v, dom, rc, api.LIST_BUILD_AUTO, density=rho),
                    _setup(r, v, dom, rc, api.LIST_BUILD_CELLS, density=rho)):
        assert np.array_equal(x, y)


@pytest.mark.parametrize("chains,beads", [(300, 8), (2100, 8), (9000, 8)])
def test_polymer_rows_and_bonds_equal_the_build_by_cell(gpu_lib, chains, beads):
    r, v, ch, sub, _, bf, dom = polymer.fene_melt(chains, beads)
    got = [_setup(r, v, dom, WCA_RC, m, (ch, sub, bf), density=0.85, potential_flag=1, k_c=30.0, R_0=1.5)
           for m in (api.LIST_BUILD_AUTO, api.LIST_BUILD_CELLS)]
    for x, y in zip(*got):
        assert np.array_equal(x, y)


@pytest.mark.parametrize("nu", [[8, 8, 8], [26, 25, 27]])
def test_overflow_grows_the_rows(gpu_lib, nu):
    """A list capacity too small for the liquid ends with the rows of a large one."""
    r, v, dom = lattice.lj_fluid(nu, 0.8442, 1.0, 83)
    r = lattice.jitter(r, 0.04, 84, dom)
    for x, y in zip(_setup(r, v, dom, 2.5, api.LIST_BUILD_AUTO, density=0.8442, nlist_capacity=40),
                    _setup(r, v, dom, 2.5, api.LIST_BUILD_CELLS, density=0.8442)):
        assert np.array_equal(x, y)


@pytest.mark.parametrize("tpm", [1, 2, 4, 8, 16])
@pytest.mark.parametrize("precision", [api.PRECISION_FP64, api.PRECISION_FP32])
def test_lanes_of_the_force_kernel_read_every_entry_once(gpu_lib, tpm, precision):
    """Rows of 0 to 100 entries (a gas with a dense drop) walked by every number
    of lanes: the lanes differ in the order of a sum of at most 120 FP64 terms of
    up to 1e3, 120 x 2^-53 x 1e3 = 1.4e-11 absolute."""
    rng = np.random.default_rng(3)
    r, v, dom = lattice.lj_fluid([12, 12, 12], 0.9, 1.0, 85)
    keep = (np.linalg.norm(r, axis=1) < 6.0) | (rng.random(len(r)) < 0.15)
    r, v = lattice.jitter(r[keep], 0.04, 86, dom), v[keep]
    out = []
    for t in (tpm, 1):
        s = api.MDSystem(api.make_params(len(r), dom, 2.5, threads_per_molecule=t, precision=precision))
        s.upload(r, v)
        s.setup()
        n = np.bincount(np.searchsorted(np.arange(1, len(r) + 1), s.pair_list()[0]), minlength=len(r))
        out.append((s.download()[2], *s.per_molecule()))
        s.close()
    assert n.min() <= 6 and n.max() > 64
    for x, y in zip(*out):
        assert np.abs(x - y).max() <= 1.4e-11


def test_numbers_and_records_after_a_device_upload(gpu_lib):
    """Global numbers of a state uploaded without any are 1 .. n, before and
    after a sort renumbers them; records come in order across the ring's end."""
    import ctypes as C
    import torch
    r, v, dom = lattice.lj_fluid([6, 6, 6], 0.8, 1.0, 87)
    r = lattice.jitter(r, 0.04, 88, dom)
    s = api.MDSystem(api.make_params(len(r), dom, WCA_RC, density=0.8, tplot=1))
    d = [torch.tensor(x, device="cuda") for x in (r, v)]
    api.check(gpu_lib.fm_upload_state_device(s.h, len(r), *[C.c_void_p(x.data_ptr()) for x in d]))
    assert np.array_equal(s.download()[3], np.arange(1, len(r) + 1))
    s.set_sort(1, 1, 1)
    s.setup()
    s.simulation_md(5)
    assert np.array_equal(np.sort(s.download()[3]), np.arange(1, len(r) + 1))
    assert [x["iter"] for x in s.records()] == list(range(6))
    s.simulation_md(4094)
    first = s.records(7)
    assert [x["iter"] for x in first] == list(range(6, 13))
    s.simulation_md(4)
    assert [x["iter"] for x in s.records()] == list(range(4100, 4104))
    s.close()
