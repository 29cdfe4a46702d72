"""Bonds by table look-up and by scan: every bead of the 27 cells around an
owner's that has its chain and whose subchain bit its flags name, for unique
beads, for chains numbered alike (a named bead then has several copies), with
molecules in halo cells (coordinates on the lower faces), in boxes of three
cells per axis, and in a mixture with solvent."""
import numpy as np
import pytest

from flowmol_b200 import api, polymer
from helpers import WCA_RC

pytestmark = pytest.mark.gpu


def _expected(r, ch, sub, bf, dom, nc, cs):
    """(owner, partner) pairs, 1-based; halo cells 0 and nc + 1 are the cells on
    the far side."""
    cell = np.ceil((r + 0.5 * np.asarray(dom)) / cs).astype(int)
    out = []
    for c in np.unique(ch):
        idx = np.flatnonzero(ch == c)
        if not np.any(bf[idx]):
            continue
        for i in idx:
            d = cell[idx] - cell[i]
            near = np.all((np.abs(d) <= 1) | (np.abs(np.abs(d) - nc) <= 1), axis=1)
            pos = sub[idx] - 1
            named = (bf[i][np.clip(pos // 31, 0, 3)] >> (pos % 31)) & 1
            out += [(i + 1, j + 1) for j in idx[near & (named == 1) & (idx != i)]]
    return sorted(out)


@pytest.mark.parametrize("case", ["unique", "alike", "three_cells", "solution", "long_chains", "faces"])
@pytest.mark.parametrize("force_path", [api.FORCE_PATH_AUTO, api.FORCE_PATH_GATHER])
def test_bonds(gpu_lib, case, force_path):
    chains, beads, kw = {"three_cells": (13, 8, {}), "long_chains": (60, 36, {"fill": 0.5}),
                         "solution": (300, 8, {})}.get(case, (300, 8, {}))
    make = polymer.fene_solution if case == "solution" else polymer.fene_melt
    r, v, ch, sub, _, bf, dom = make(chains, beads, **kw)
    if case == "alike":
        ch = (ch - 1) % 60 + 1
    if case == "faces":
        r = r - r.min(axis=0) - 0.5 * np.asarray(dom)
    # R_0 6: a copy of a named bead anywhere in the 27 cells is a bond the force accepts
    p = api.make_params(len(r), dom, WCA_RC, density=0.85, potential_flag=1, k_c=30.0, R_0=6.0, force_path=force_path)
    _, g = api.derive_geometry(p)
    s = api.MDSystem(p)
    s.upload(r, v)
    s.upload_monomers(ch, sub, bf)
    want = _expected(r, ch, sub, bf, dom, np.array(g["ncells"]), np.array(g["cellside"]))
    most = np.bincount([o for o, _ in want]).max()
    if most > 4:
        with pytest.raises(api.FlowmolError):
            s.setup()
    else:
        s.setup()
        o, q, _ = s.bonds()
        if case == "faces":  # a bead on a face pairs with one side only
            assert set(zip(o.tolist(), q.tolist())) <= set(want) and len(o) > 0.8 * len(want)
        else:
            assert sorted(zip(o.tolist(), q.tolist())) == want
    s.close()
