"""update_halo over arrays of random contents, halos included.

Whatever the halos held before the call, every element must equal the oracle's:
the one-launch update (three or more cells per axis), whose x- and y-face
fluxes keep mirrors of a z halo plane's old values, and the per-axis passes
(thinner grids, an array given for two fields)."""
import ctypes

import numpy as np
import pytest

import cloverleaf3d_ref_b200 as C
import hydro_harness as H
import oracle_lib as O

pytestmark = pytest.mark.gpu

FIELDS = ["density0", "density1", "energy0", "energy1", "pressure", "viscosity", "soundspeed", "xvel0", "xvel1",
          "yvel0", "yvel1", "zvel0", "zvel1", "vol_flux_x", "vol_flux_y", "vol_flux_z", "mass_flux_x",
          "mass_flux_y", "mass_flux_z"]
# the argument order of update_halo_kernel (density0, energy0, pressure, ...)
ORDER = ["density0", "energy0", "pressure", "viscosity", "soundspeed", "density1", "energy1", "xvel0", "yvel0",
         "zvel0", "xvel1", "yvel1", "zvel1", "vol_flux_x", "vol_flux_y", "vol_flux_z", "mass_flux_x",
         "mass_flux_y", "mass_flux_z"]


def call(lib, name, a, n, fields, depth):
    nb = (ctypes.c_int * 6)(*[-1] * 6)
    bounds = [H.I(v) for v in (1, n[0], 1, n[1], 1, n[2])]
    getattr(lib, name)(*bounds, nb, nb, *[H.p(a[f]) for f in ORDER], (ctypes.c_int * 19)(*fields), H.I(depth))


@pytest.mark.parametrize("alias", [False, True])
@pytest.mark.parametrize("depth", [1, 2])
@pytest.mark.parametrize("n", [(3, 3, 3), (4, 3, 5), (33, 9, 34), (29, 40, 7), (30, 31, 9), (2, 5, 4), (5, 1, 3)])
def test_random_contents(n, depth, alias):
    rng = np.random.default_rng(sum(n) + depth)
    a = {f: np.asfortranarray(rng.standard_normal(O.shape(H.ARRAYS_3D[f], *n))) for f in FIELDS}
    fields = [1] * 19
    if alias:  # one array for two fields of one kind; every third field left out
        a["energy1"] = a["density1"]
        fields = [0 if i % 3 == 2 else 1 for i in range(19)]
    want = {f: v.copy(order="F") for f, v in a.items()}
    if alias:
        want["energy1"] = want["density1"]
    L = C.lib()
    L.clover_gpu_release()
    L.clover_gpu_clear_status()
    for _ in range(2):  # the second call meets the halos the first one left
        call(O.load(), "oracle_update_halo_kernel", want, n, fields, depth)
        call(L, "clover_update_halo_kernel", a, n, fields, depth)
    L.clover_gpu_sync_to_host()
    assert L.clover_gpu_status() == 0
    for f in FIELDS:
        assert np.array_equal(a[f], want[f]), f
    L.clover_gpu_release()
