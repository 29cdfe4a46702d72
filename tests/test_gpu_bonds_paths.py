"""Bonds on the paths where they are found in another way than by one look-up
after the gather path's list build: by scanning (a named bead has several
copies), after the tiled path's build, in runs through the rebuild graph on
both paths, and more of them than a bead can hold."""
import numpy as np
import pytest

from flowmol_b200 import api, polymer
from helpers import WCA_RC
from test_gpu_bonds import _expected

pytestmark = pytest.mark.gpu


def _system(r, v, ch, sub, bf, dom, R_0, **kw):
    p = api.make_params(len(r), dom, WCA_RC, density=0.85, potential_flag=1, k_c=30.0, R_0=R_0, **kw)
    _, g = api.derive_geometry(p)
    s = api.MDSystem(p)
    s.upload(r, v)
    s.upload_monomers(ch, sub, bf)
    return s, np.array(g["ncells"]), np.array(g["cellside"])


@pytest.mark.parametrize("copies", [2, 8])
@pytest.mark.parametrize("path", [api.FORCE_PATH_GATHER, api.FORCE_PATH_TILES])
def test_copies_of_a_named_bead(gpu_lib, path, copies):
    """Chains numbered alike in groups: up to four beads in the cells around an
    owner's answer to a name, every one a bond.  With eight copies in a small
    box there are more than four and the setup says so."""
    r, v, ch, sub, _, bf, dom = polymer.fene_melt(300 if copies == 2 else 24, 8)
    groups = ch.max() // copies
    s, nc, cs = _system(r, v, (ch - 1) % groups + 1, sub, bf, dom, 6.0, force_path=path)
    want = _expected(r, (ch - 1) % groups + 1, sub, bf, dom, nc, cs)
    most = np.bincount([o for o, _ in want]).max()
    if copies == 8:
        assert most > 4
        with pytest.raises(api.FlowmolError):
            s.setup()
    else:
        assert 2 < most <= 4
        s.setup()
        o, q, _ = s.bonds()
        assert sorted(zip(o.tolist(), q.tolist())) == want
    s.close()


@pytest.mark.parametrize("graphs", ["1", "0"])
@pytest.mark.parametrize("solvent", [0, 1])
def test_tiled_path_finds_the_same_bonds(gpu_lib, monkeypatch, solvent, graphs):
    """After a run with rebuilds: the same bonds, and the trajectories of the two
    force paths differ by the order of their FP64 sums (a few ulp of forces of
    up to 1e3, 2e-13 each, grown 100-fold at most over 60 steps of 0.005: 1e-9)."""
    monkeypatch.setenv("FM_STEP_GRAPHS", graphs)
    r, v, ch, sub, _, bf, dom = (polymer.fene_solution if solvent else polymer.fene_melt)(500, 8)
    out = []
    for path in (api.FORCE_PATH_GATHER, api.FORCE_PATH_TILES):
        s, _, _ = _system(r, v, ch, sub, bf, dom, 1.5, force_path=path, solvent_flag=solvent, threads_per_molecule=4)
        s.setup()
        s.simulation_md(60)
        assert s.force_path()[0] == path and s.counters()["rebuilds"] > 1
        o, q, _ = s.bonds()
        assert len(o) == 2 * 7 * len(np.unique(ch[np.any(bf != 0, axis=1)]))
        out.append((sorted(zip(o.tolist(), q.tolist())), s.download()[0]))
        s.close()
    assert out[0][0] == out[1][0]
    assert np.abs(out[0][1] - out[1][1]).max() <= 1e-9
