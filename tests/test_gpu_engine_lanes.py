"""Every number of lanes of the engine's force kernel meets each entry of a row
once (rows of 0 to 100 entries, so every remainder of a chunk of eight), and
its two list builds give the same jobs on both sides of the line between them."""
import numpy as np
import pytest

from flowmol_b200 import api, lattice

pytestmark = pytest.mark.gpu


def _drop_in_gas():
    rng = np.random.default_rng(3)
    r, v, dom = lattice.lj_fluid([12, 12, 12], 0.9, 1.0, 85)
    keep = (np.linalg.norm(r, axis=1) < 6.0) | (rng.random(len(r)) < 0.15)
    return lattice.jitter(r[keep], 0.04, 86, dom), v[keep], dom


def _row_lengths(r, v, dom):
    s = api.MDSystem(api.make_params(len(r), dom, 2.5))
    s.upload(r, v)
    s.setup()
    n = np.bincount(s.pair_list()[0] - 1, minlength=len(r))
    s.close()
    return n


@pytest.mark.parametrize("tpm", [1, 2, 4, 8])
@pytest.mark.parametrize("precision", [api.PRECISION_FP64, api.PRECISION_FP32])
def test_lanes_agree(gpu_lib, tpm, precision):
    """One velocity-Verlet step against the 16-lane kernel. The lanes differ in
    the order of a sum of at most 120 FP64 terms of up to 1e3, so a differs by
    at most 1.4e-11 and v by dt 1.4e-11 = 7e-14; an ulp of r (1.8e-15) times a
    stiffness of 1e4 adds dt/2 1.8e-11 = 4.5e-14: below 2e-13 in all."""
    r, v, dom = _drop_in_gas()
    n = _row_lengths(r, v, dom)
    assert n.min() <= 6 and n.max() > 64 and len(np.unique(n % 8)) == 8
    out = []
    for t in (tpm, 16):
        e = api.Engine(8192, 40000, 8192 * 160, 2, threads_per_molecule=t, precision=precision, ticks_per_chunk=4)
        job = e.submit(api.make_job(len(r), dom, 2.5, 1, tplot=1), r, v)
        e.run()
        assert e.results()[0]["status"] == 0
        out.append(e.job_state(job, len(r)))
        e.close()
    for x, y in zip(*out):
        assert np.abs(x - y).max() <= 2e-13


# a dense liquid's molecule is a warp of the build by molecule, four molecules
# share one at WCA range: 16,384 warps, one job more, and a mixture of both
JOBS = {
    "at_the_line": [([16, 16, 16], 0.8442, 2.5)],
    "above_the_line": [([16, 17, 16], 0.8442, 2.5)],
    "together_above": [([15, 16, 16], 0.8442, 2.5), ([8, 8, 8], 0.8, 2.5)],
    "mixed_ranges": [([14, 15, 14], 0.8442, 2.5), ([12, 12, 13], 0.8, 2.0 ** (1.0 / 6.0)), ([10, 10, 9], 0.8, 1.45)],
}


@pytest.mark.parametrize("name", sorted(JOBS))
def test_rows_by_molecule_and_by_cell_give_the_same_jobs(gpu_lib, name):
    """Both sides of the line below which a tick builds by molecule: the same
    rows in the same order, so the same trajectories to the last bit."""
    out = []
    for mode in (api.LIST_BUILD_AUTO, api.LIST_BUILD_CELLS):
        e = api.Engine(40000, 160000, 40000 * 160, 4, threads_per_molecule=1, list_build=mode, ticks_per_chunk=8)
        ids = []
        for k, (nu, rho, rc) in enumerate(JOBS[name]):
            r, v, dom = lattice.lj_fluid(nu, rho, 1.0, 91 + k)
            ids.append((e.submit(api.make_job(len(r), dom, rc, 30, tplot=10), lattice.jitter(r, 0.04, 92, dom), v), len(r)))
        e.run()
        assert all(x["status"] == 0 for x in e.results())
        out.append([e.job_state(*j) for j in ids])
        e.close()
    for x, y in zip(*out):
        assert np.array_equal(x[0], y[0]) and np.array_equal(x[1], y[1])


def test_sparse_job_with_dense_cells(gpu_lib):
    """A liquid drop in a thin gas: on average two molecules a cell, so the cells
    are sorted four a warp, but up to twenty in the drop's, which one lane
    sorts.  As in the other engine tests, positions follow the single system to
    1e-9, here over 40 steps."""
    rng = np.random.default_rng(41)
    r, v, dom = lattice.lj_fluid([20, 20, 20], 0.85, 1.0, 42)
    keep = (np.linalg.norm(r - [3.0, -2.0, 1.0], axis=1) < 6.0) | (rng.random(len(r)) < 0.05)
    r, v = lattice.jitter(r[keep], 0.03, 43, dom), v[keep]
    nc = np.floor(np.asarray(dom) / 2.8).astype(int)
    cell = np.ceil((r / dom + 0.5) * nc).astype(int) - 1
    n = np.bincount(np.ravel_multi_index(cell.T, nc), minlength=nc.prod())
    assert n.mean() < 3.3 and n.max() > 16 and np.any((n > 3) & (n <= 8)) and np.any(n == 0)
    e = api.Engine(8192, 40000, 8192 * 160, 2, threads_per_molecule=4, ticks_per_chunk=8)
    job = e.submit(api.make_job(len(r), dom, 2.5, 40, tplot=20), r, v)
    e.run()
    assert e.results()[0]["status"] == 0
    got = e.job_state(job, len(r))
    e.close()
    s = api.MDSystem(api.make_params(len(r), dom, 2.5, tplot=20, threads_per_molecule=4))
    s.upload(r, v)
    s.setup()
    s.simulation_md(40)
    want = s.download()
    s.close()
    for x, y in zip(got, want):
        assert np.abs(x - y).max() <= 1e-9
