"""Sums of squares that are small beside the populations: velocity errors of
double lattices a few last places apart, kinetic energy of nearly still ones.

The expected values are exact (Python integers in units of 2^-61).  The sums
are exact too and round once; the mean, the square root and the expectation
round once each, so 2^-50 bounds the relative difference.
"""
from __future__ import annotations

import math
from fractions import Fraction

import numpy as np
import pytest

from test_gpu_sums import E, W

pytestmark = pytest.mark.gpu
DIMS = (21, 12, 9)


def _lattice(api, storage, f):
    L = api.Lattice(*DIMS, api.STORAGE_NAMES[storage], False, False)
    L.init([api.FLAG_OBSTACLE, api.FLAG_GHOST_LAYER] * 3)
    L.write(api.FIELD_DD, f)
    return L, L.read(api.FIELD_FLAGS)[0] == api.FLAG_FLUID


def _momenta(L, api, fluid, sign=1):
    """Exact momenta of the fluid cells, integers in units of 2^-61."""
    f = np.ldexp(L.read(api.FIELD_DD).astype(np.float64)[:, fluid], 61)
    p = np.array([[int(v) for v in plane] for plane in f], dtype=object)
    return sign * (E.astype(int).astype(object) @ p)


def _root_mean(total, n):
    return math.sqrt(float(Fraction(int(total), (1 << 122) * n)))


def _base(seed):
    rng = np.random.default_rng(seed)
    return rng, W[:, None, None, None] * (1 + 0.1 * rng.uniform(-1, 1, (19, DIMS[2], DIMS[1], DIMS[0])))


@pytest.mark.parametrize("a,b", [("f64", "f64"), ("f64", "f32"), ("f32", "f64")])
@pytest.mark.parametrize("places", [1, 64, 1 << 20])
def test_velocity_error_of_a_few_last_places(capi, places, a, b):
    api = capi
    rng, f = _base(places)
    g = f.astype(np.float32).astype(np.float64) if "f32" in (a, b) else f
    h = (g.view(np.int64) + rng.integers(-places, places + 1, g.shape)).view(np.float64)
    A, fluid = _lattice(api, a, h if a == "f64" else g)
    B, _ = _lattice(api, b, h if a == "f32" else g)
    n = int(fluid.sum())
    for la, lb in ((0, 0), (1, 1), (1, 0)):
        ua, ub = _momenta(A, api, fluid, -1 if la else 1), _momenta(B, api, fluid, -1 if lb else 1)
        d2, r2 = ((ua - ub) ** 2).sum(0), (ub ** 2).sum(0)
        r = api.compare_velocity(A, la, B, lb)
        for key, want in (("rms", _root_mean(d2.sum(), n)), ("ref_rms", _root_mean(r2.sum(), n)),
                          ("max_abs", _root_mean(max(d2), 1)), ("ref_max", _root_mean(max(r2), 1))):
            assert r[key] == pytest.approx(want, rel=2.0 ** -50, abs=0), (key, la, lb)
        assert r["rms"] > 0


@pytest.mark.parametrize("storage,u", [("f64", 1e-15), ("f64", 1e-12), ("f64", 1e-9), ("f64", 1e-4), ("f32", 1e-4), ("f16", 1e-4)])
def test_energy_of_nearly_still_flow(capi, storage, u):
    api = capi
    rng = np.random.default_rng(7)
    f = W[:, None, None, None] + u * rng.uniform(-1, 1, (19, DIMS[2], DIMS[1], DIMS[0]))
    L, fluid = _lattice(api, storage, f)
    j2 = int((_momenta(L, api, fluid) ** 2).sum())
    want = float(Fraction(j2, 1 << 123))
    assert want > 0
    for got in (L.reduce_conserved(0), L.reduce_conserved(1), L.reduce_conserved_noalloc(0)):
        assert got[4] == pytest.approx(want, rel=2.0 ** -50, abs=0)
