"""A list that overflows grows once, to the longest row of the whole system,
also where the build by molecule has more blocks than fit on the GPU at once
and the short rows come first."""
import numpy as np
import pytest

from flowmol_b200 import api, lattice

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nu", [[16, 16, 32], [22, 22, 32]])  # by molecule, by fours
def test_growth_covers_every_row(gpu_lib, nu):
    r, v, dom = lattice.lj_fluid(nu, 0.9, 1.0, 61)
    rng = np.random.default_rng(62)
    # from a gas in the lower cells, which the first blocks take, to a liquid in the top ones
    keep = rng.random(len(r)) < 0.1 + 0.9 * (r[:, 2] / dom[2] + 0.5) ** 2
    r, v = lattice.jitter(r[keep], 0.04, 63, dom), v[keep]
    assert 10000 < len(r) < 65536 and (len(r) >= 16384) == (nu[0] == 22)
    out = []
    for mode, cap in ((api.LIST_BUILD_AUTO, 8), (api.LIST_BUILD_CELLS, 160)):
        s = api.MDSystem(api.make_params(len(r), dom, 2.5, density=0.9, list_build=mode, threads_per_molecule=1,
                                         nlist_capacity=cap))
        s.upload(r, v)
        s.setup()
        rows = s.pair_list()
        out.append([*rows, s.download()[2]])
        if cap == 8:
            most = np.bincount(rows[0] - 1).max()
            want = -(-(int(np.ceil(1.2 * most)) + 8) // 8) * 8
            assert s.counters()["nlist_capacity"] == want
        s.close()
    for x, y in zip(*out):
        assert np.array_equal(x, y)
