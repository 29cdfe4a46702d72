"""All pairs by lanes on both sides of the size where their number changes, and
where one lane per molecule was once taken: the forces of the neighbour list."""
import numpy as np
import pytest

from flowmol_b200 import api, lattice

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nu", [[12, 13, 13], [16, 16, 8], [13, 13, 13], [21, 20, 20]])
@pytest.mark.parametrize("record", [True, False])
def test_all_pairs_equal_the_list(gpu_lib, nu, record):
    """A pair's distance differs by two ulp of half a box, 7e-15, times a
    stiffness of at most 1.1e3 and some 12 near neighbours: below 2e-10."""
    r, v, dom = lattice.lj_fluid(nu, 0.8, 1.0, 51)
    r = lattice.jitter(r, 0.02, 52, dom)
    out = []
    for pairs in (0, 3):
        s = api.MDSystem(api.make_params(len(r), dom, 2.5, density=0.8, force_list=pairs, threads_per_molecule=1,
                                         tplot=1 if record else 100))
        s.upload(r, v)
        s.setup()
        if not record:
            s.iter = 1
            s.simulation_compute_forces()
        out.append((s.download()[2], s.records()[0]["potenergy"]))
        s.close()
    assert np.abs(out[0][0] - out[1][0]).max() <= 2e-10
    assert out[0][1] == pytest.approx(out[1][1], rel=1e-12)
