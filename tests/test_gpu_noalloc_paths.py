"""Forces without allocation: the one-block binning up to 4,096 molecules and
the kernels above it, 8, 16 and 32 lanes per molecule, cells of more than 32
molecules, and molecules exactly on the lower faces, against fm_setup.  Both
sum the same FP64 terms in another order: the parity tolerance 1e-12 (floor 1)."""
import ctypes as C

import numpy as np
import pytest

from flowmol_b200 import api, lattice
from helpers import WCA_RC, rel_err

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nu,rho,rc,faces", [
    ([8, 16, 8], 0.8442, 2.5, False), ([16, 8, 8], 0.8, WCA_RC, False), ([9, 15, 8], 0.8442, 2.5, False),
    ([13, 17, 16], 0.8, 1.45, False), ([8, 9, 9], 1.2, 3.5, False), ([7, 7, 8], 0.8, WCA_RC, True),
    ([12, 11, 12], 0.8442, 2.5, True), ([5, 5, 5], 0.7, 2.2, False)])
def test_noalloc_equals_setup(gpu_lib, nu, rho, rc, faces):
    import torch
    r, v, dom = lattice.lj_fluid(nu, rho, 1.0, 61)
    r = r - r.min(axis=0) - 0.5 * np.asarray(dom) if faces else lattice.jitter(r, 0.05, 62, dom)
    p = api.make_params(len(r), dom, rc, density=rho)
    f = gpu_lib.fm_compute_forces_noalloc
    f.argtypes = [C.POINTER(api.FmParams), C.c_int32] + [C.c_void_p] * 5
    d = torch.tensor(r, device="cuda")
    a, pe, vir = torch.empty_like(d), torch.empty(len(r), dtype=torch.float64, device="cuda"), \
        torch.empty(len(r), dtype=torch.float64, device="cuda")
    assert f(C.byref(p), len(r), d.data_ptr(), a.data_ptr(), pe.data_ptr(), vir.data_ptr(), None) == 0
    s = api.MDSystem(p)
    s.upload(r, v)
    s.setup()
    assert rel_err(a.cpu().numpy(), s.download()[2], 1.0).max() <= 1e-12
    for x, y in zip((pe, vir), s.per_molecule()):
        y = np.asarray(y)
        assert (np.abs(x.cpu().numpy() - y) / np.maximum(np.abs(y), 1.0)).max() <= 1e-12
    s.close()
