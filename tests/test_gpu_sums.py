"""Conservation sums and velocity errors of arbitrary populations.

The kernels sum cells whose populations are ordinary (the moving ones within
[2^-8, 2^-3), the one at rest below 2^-1) in integers and every other cell in
compensated double arithmetic; both must give the sums of the stored values.
Tolerance: every sum is exact or compensated and rounds a few times at the
end, so 2^-48 of the sum of the magnitudes bounds it; squares of the double
cells' momenta add a few roundings of their own (2^-46).
"""
from __future__ import annotations

import math

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

E = np.array([[1, -1, 0, 0, 1, -1, 1, -1, 1, -1, 1, -1, 0, 0, 0, 0, 0, 0, 0],
              [0, 0, 1, -1, 1, -1, -1, 1, 0, 0, 0, 0, 1, -1, 1, -1, 0, 0, 0],
              [0, 0, 0, 0, 0, 0, 0, 0, 1, -1, -1, 1, 1, -1, -1, 1, 1, -1, 0]], dtype=np.float64)
W = np.array([1 / 18] * 4 + [1 / 36] * 12 + [1 / 18] * 2 + [1 / 3])


def _filled(api, dims, storage, odd, seed):
    """A lattice of populations near rest; with `odd`, a share of the cells holds values outside the ordinary range."""
    rng = np.random.default_rng(seed)
    shape = (19, dims[2], dims[1], dims[0])
    f = W[:, None, None, None] * (1 + 0.2 * rng.uniform(-1, 1, shape))
    if odd:
        n = rng.random(shape[1:]) < 0.05
        f[:, n] = rng.choice([-0.02, 0.0, 1e-9, 0.13, 0.6, 2.0 ** -8, 2.0 ** -3, 2.0 ** -1], (19, int(n.sum())))
    L = api.Lattice(*dims, storage, False, False)
    L.init([api.FLAG_OBSTACLE, api.FLAG_GHOST_LAYER] * 3)
    L.write(api.FIELD_DD, f)
    return L, L.read(api.FIELD_DD).astype(np.float64), L.read(api.FIELD_FLAGS)[0] == api.FLAG_FLUID


def _close(got, terms, bits):
    assert abs(got - math.fsum(terms.ravel())) <= 2.0 ** -bits * math.fsum(np.abs(terms).ravel()) + 1e-300


@pytest.mark.parametrize("odd", [False, True])
@pytest.mark.parametrize("dims", [(3, 3, 3), (5, 4, 3), (17, 9, 8), (67, 33, 21)])
@pytest.mark.parametrize("storage", ["f32", "f64", "f16", "bf16", "c16"])
def test_sums_of_arbitrary_populations(capi, storage, dims, odd):
    api = capi
    L, f, fluid = _filled(api, dims, api.STORAGE_NAMES[storage], odd, 11)
    f = f[:, fluid]
    for layout in (0, 1):
        e = -E if layout else E
        for got in (L.reduce_conserved(layout), L.reduce_conserved_noalloc(layout)):
            _close(got[0], f, 48)
            for a in range(3):
                _close(got[1 + a], e[a][:, None] * f, 48)
            _close(got[4], 0.5 * (e @ f) ** 2, 40)


@pytest.mark.parametrize("odd", [False, True])
@pytest.mark.parametrize("a,b", [("f16", "f64"), ("f32", "f32"), ("f64", "f32"), ("c16", "bf16"), ("f64", "f64")])
def test_velocity_error_of_arbitrary_populations(capi, a, b, odd):
    api = capi
    dims = (35, 18, 13)
    A, fa, fluid = _filled(api, dims, api.STORAGE_NAMES[a], odd, 21)
    B, fb, _ = _filled(api, dims, api.STORAGE_NAMES[b], odd, 22)
    for la, lb in ((0, 0), (1, 0), (1, 1)):
        ua, ub = (-E if la else E) @ fa[:, fluid], (-E if lb else E) @ fb[:, fluid]
        d2, r2 = ((ua - ub) ** 2).sum(0), (ub ** 2).sum(0)
        r = api.compare_velocity(A, la, B, lb)
        n = int(fluid.sum())
        assert r["cells"] == n
        for key, want in (("max_abs", math.sqrt(d2.max())), ("rms", math.sqrt(d2.sum() / n)),
                          ("ref_rms", math.sqrt(r2.sum() / n)), ("ref_max", math.sqrt(r2.max()))):
            assert r[key] == pytest.approx(want, rel=2.0 ** -40)


def test_not_a_number_reaches_the_sums(capi):
    api = capi
    L, f, _ = _filled(api, (9, 8, 7), api.F32, False, 3)
    f[4, 3, 3, 3] = np.nan
    L.write(api.FIELD_DD, f)
    got = L.reduce_conserved(0)
    assert np.isnan(got[0]) and np.isnan(got[1]) and np.isnan(got[4])
