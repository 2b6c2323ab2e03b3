"""Staged tiles of 16-bit cavities whose rows are not whole 16-byte units, in
launches large enough to be staged by default, against the one-cell kernels."""
from __future__ import annotations

import numpy as np
import pytest

from helpers import n_diff

pytestmark = pytest.mark.gpu


def _lattice(api, dims, storage, shape, cs):
    L = api.Lattice(*dims, storage, True, True)
    tau = np.float32(0.53)
    L.set_params(api.Params.make(float(np.float32(1) / tau), float(tau), api.les_coefficient(cs), (0, 0, 0), 0.08))
    L.init([api.FLAG_OBSTACLE, api.FLAG_GHOST_LAYER, 1, 1, 1, 1])
    nx, ny, nz = dims
    L.write(api.FIELD_FLAGS, np.full((nz - 2) * (nx - 2), api.FLAG_VELOCITY_INJECTION, np.int32),
            origin=(1, ny - 2, 1), size=(nx - 2, 1, nz - 2))
    L.perturb((0, 0, 0), dims, 7, 1e-2)
    L.set_kernel_shape(shape)
    return L


@pytest.mark.parametrize("cs", [0.0, 0.17])
@pytest.mark.parametrize("storage", ["f16", "bf16", "c16"])
@pytest.mark.parametrize("dims", [(3, 60, 40), (9, 17, 19), (33, 40, 21), (130, 33, 9), (523, 11, 5), (101, 99, 81), (104, 109, 121), (145, 141, 131)])
def test_staged_rows_equal_one_cell_kernels(capi, dims, storage, cs):
    """Odd, even and wide rows, fewer cells than a tile, more tiles than blocks; shape 0 at the three largest."""
    api = capi
    st = api.STORAGE_NAMES[storage]
    a = _lattice(api, dims, st, 1, cs)
    b = _lattice(api, dims, st, 0 if dims[0] in (101, 104, 145) else 3, cs)
    for k in range(4):
        a.step(k & 1)
        b.step(k & 1)
    for field in (api.FIELD_DD, api.FIELD_VELOCITY, api.FIELD_DENSITY):
        assert n_diff(a.read(field), b.read(field)) == 0
    api.synchronize()


def test_staged_ensemble_of_uneven_rows(capi):
    """One launch over cavities of all row lengths, large enough to be staged."""
    api = capi
    C = api.Cavity.make
    cav = [C((97, 80, 61), api.F16, 0.53, 0.17, 0.05, 7, 1, 1e-2), C((64, 90, 70), api.F16, 0.55, 0.17, 0.08, 9, 2, 1e-2),
           C((33, 130, 75), api.F16, 0.52, 0.17, 0.1, 5, 3, 1e-2), C((10, 11, 12), api.F16, 0.6, 0.17, 0.05, 9, 4, 1e-2),
           C((102, 70, 50), api.F16, 0.54, 0.0, 0.06, 8, 5, 1e-2), C((90, 81, 47), api.C16, 0.54, 0.17, 0.06, 8, 6, 1e-2),
           C((77, 120, 115), api.C16, 0.56, 0.17, 0.04, 9, 7, 1e-2),
           C((101, 103, 99), api.F16, 0.56, 0.17, 0.04, 6, 8, 1e-2), C((110, 101, 90), api.C16, 0.56, 0.17, 0.04, 9, 9, 1e-2)]
    out = {}
    for shape in (1, 3):
        B = api.Batch(cav, store_velocity=True)
        B.set_kernel_shape(shape)
        B.reset()
        B.run()
        out[shape] = [(L.read(api.FIELD_DD), L.read(api.FIELD_VELOCITY)) for L in B.lattices]
    for (a, u), (b, v) in zip(out[1], out[3]):
        assert n_diff(a, b) == 0 and n_diff(u, v) == 0
