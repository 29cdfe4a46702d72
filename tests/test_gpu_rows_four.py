"""The list build by fours, which dense systems of 16,384 to 65,536 molecules
take: its rows are those of the builds by cell and by 2x2x2 cells, partner for
partner, just above the line and at its upper end, in ragged boxes, with cells
of more than 20 molecules (a warp takes several fours), of more than 128, and
of 1 to 3 left over, in boxes of three cells per axis, with molecules in halo
cells (coordinates on the lower faces), with rows that overflow, and in a
subdomain."""
import numpy as np
import pytest

from flowmol_b200 import api, lattice
from flowmol_b200 import domain as D

pytestmark = pytest.mark.gpu


def _rows(r, v, dom, rc, rho, mode, **kw):
    s = api.MDSystem(api.make_params(len(r), dom, rc, list_build=mode, threads_per_molecule=1, density=rho, **kw))
    s.upload(r, v)
    s.setup()
    out = [*s.pair_list(), s.download()[2]]
    s.close()
    return out


CASES = {
    "just_above": ([17, 16, 17], 0.8442, 2.5, api.LIST_BUILD_CELLS),
    "ragged": ([20, 19, 20], 0.75, 2.5, api.LIST_BUILD_CELLS),
    "thin": ([23, 20, 21], 0.45, 2.5, api.LIST_BUILD_CELLS),
    "cells_of_60": ([18, 17, 19], 0.8442, 3.9, api.LIST_BUILD_CELLS),
    "cells_of_300": ([17, 17, 17], 1.78, 5.3, api.LIST_BUILD_CELLS),
    "three_cells": ([17, 16, 16], 0.8442, 8.0, api.LIST_BUILD_CELLS),
    "faces": ([17, 17, 17], 0.8442, 2.5, api.LIST_BUILD_CELLS),
    "largest": ([32, 32, 16], 0.8442, 2.5, api.LIST_BUILD_CELLS),
    "by_blocks": ([25, 24, 25], 0.8442, 2.5, api.LIST_BUILD_BLOCKS),
    "by_warp_above": ([26, 25, 27], 0.8442, 2.5, api.LIST_BUILD_BLOCKS),  # past the line: by cell against by 2x2x2
}


@pytest.mark.parametrize("name", sorted(CASES))
def test_rows_equal_the_builds_by_warp(gpu_lib, name):
    nu, rho, rc, other = CASES[name]
    r, v, dom = lattice.lj_fluid(nu, rho, 1.0, 71)
    if name == "faces":
        r = r - r.min(axis=0) - 0.5 * np.asarray(dom)
    else:
        r = lattice.jitter(r, 0.04, 72, dom)
    assert (len(r) <= 65536) == (name != "by_warp_above") and len(r) >= 16384
    for x, y in zip(_rows(r, v, dom, rc, rho, api.LIST_BUILD_AUTO), _rows(r, v, dom, rc, rho, other)):
        assert np.array_equal(x, y)


def test_remainders_and_empty_cells(gpu_lib):
    """A drop in a thin gas: cells of every size from none to some thirty."""
    rho = 0.8442
    r, v, dom = lattice.lj_fluid([24, 24, 24], rho, 1.0, 73)
    rng = np.random.default_rng(74)
    keep = (np.linalg.norm(r, axis=1) < 0.38 * dom[0]) | (rng.random(len(r)) < 0.12)
    r, v = lattice.jitter(r[keep], 0.04, 75, dom), v[keep]
    assert 16384 <= len(r) <= 65536
    auto = _rows(r, v, dom, 2.5, rho, api.LIST_BUILD_AUTO)
    _, g = api.derive_geometry(api.make_params(len(r), dom, 2.5, density=rho))
    cell = np.ceil((r + 0.5 * np.asarray(dom)) / np.array(g["cellside"])).astype(int) - 1
    n = np.bincount(np.ravel_multi_index(cell.T, g["ncells"]), minlength=np.prod(g["ncells"]))
    assert {0, 1, 2, 3, 4, 5} <= set(n.tolist()) and n.max() > 20
    for x, y in zip(auto, _rows(r, v, dom, 2.5, rho, api.LIST_BUILD_CELLS)):
        assert np.array_equal(x, y)


@pytest.mark.parametrize("name", ["liquid", "faces"])
def test_overflow(gpu_lib, name):
    r, v, dom = lattice.lj_fluid([17, 17, 18], 0.8442, 1.0, 76)
    r = r - r.min(axis=0) - 0.5 * np.asarray(dom) if name == "faces" else lattice.jitter(r, 0.04, 77, dom)
    for x, y in zip(_rows(r, v, dom, 2.5, 0.8442, api.LIST_BUILD_AUTO, nlist_capacity=40),
                    _rows(r, v, dom, 2.5, 0.8442, api.LIST_BUILD_CELLS)):
        assert np.array_equal(x, y)


@pytest.mark.parametrize("dims", [(1, 1, 1), (2, 1, 1), (2, 2, 1)])
def test_subdomains_equal_the_undivided_system(gpu_lib, dims):
    """Subdomains of 39,000, 23,000 and 13,000 entries, halo copies among them: after
    rebuilds and migration every position and velocity is the undivided
    system's, bit for bit (the undivided one by cell)."""
    rho = 0.8442
    r, v, dom = lattice.lj_fluid([17, 18, 19], rho, 1.0, 78)
    r = lattice.jitter(r, 0.05, 79, dom)
    kw = dict(tplot=10, density=rho, threads_per_molecule=4)
    s = api.MDSystem(api.make_params(len(r), dom, 2.5, list_build=api.LIST_BUILD_CELLS, **kw))
    s.upload(r, v)
    s.setup()
    s.simulation_md(30)
    rs, vs, _, _ = s.download()
    s.close()
    sysd = D.local_system(api.make_params(len(r), dom, 2.5, **kw), r, v, dims=dims, capacity_factor=1.5)
    try:
        sysd.setup()
        sysd.run(30)
        rd, vd, gid = sysd.state()
        assert np.array_equal(np.sort(gid), np.arange(len(r)))
        assert np.array_equal(rd, rs[gid]) and np.array_equal(vd, vs[gid])
    finally:
        sysd.close()
