"""Double lattices under parameters that the binding accepts but no ordinary
flow has: the step is the double arithmetic's, not-a-number results included."""
from __future__ import annotations

import math
import subprocess
from pathlib import Path

import numpy as np
import pytest

ROOT = Path(__file__).resolve().parent.parent


def test_integer_collision_refuses_or_equals_double_arithmetic(tmp_path):
    exe = tmp_path / "fix64_params_probe"
    subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-x", "c++",
                    "-I", str(ROOT / "turbulent_lbm_multigpu_gb300" / "csrc"),
                    str(ROOT / "tests/cpp/fix64_params_probe.cpp"), "-o", str(exe)], check=True)
    r = subprocess.run([str(exe), "20000"], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout


@pytest.mark.gpu
@pytest.mark.parametrize("inv_tau,tau0,les", [
    (1.9, 0.53, -1.0), (1.9, 0.53, -50.0), (1.9, 0.53, math.inf), (1.9, 0.53, math.nan), (1.9, math.inf, 0.7),
    (1.9, 1e30, 0.7), (1.9, 1e14, 1e29), (math.inf, 0.0, 0.0), (math.nan, 0.0, 0.0), (0.0, 0.0, 0.0), (-0.5, 0.0, 0.0)])
def test_steps_with_any_parameters_match_oracle(capi, oracle_mod, inv_tau, tau0, les):
    api, O = capi, oracle_mod
    dims = (19, 11, 9)
    rng = np.random.default_rng(9)
    w = np.array([1 / 18] * 4 + [1 / 36] * 12 + [1 / 18] * 2 + [1 / 3])
    state = w[:, None, None, None] * (1 + 0.1 * rng.uniform(-1, 1, (19,) + dims[::-1]))
    for parity in (0, 1):
        L = api.Lattice(*dims, api.F64, True, True)
        L.set_params(api.Params.make(inv_tau, tau0, les, (0, 0, 0), 0.05))
        L.init([1] * 6)
        L.write(api.FIELD_DD, state)
        s = O.single(O.OracleKernels("f64"), dims, O.Params(inv_tau, tau0, les, (0, 0, 0), 0.05), "f64")
        s.lat.flags[...] = L.read(api.FIELD_FLAGS).reshape(s.lat.flags.shape)
        s.lat.dd[...] = state.reshape(s.lat.dd.shape)
        s.lat.counter = parity
        L.step(parity)
        s.step()
        for what, want in ((api.FIELD_DD, s.lat.dd), (api.FIELD_VELOCITY, s.lat.vel), (api.FIELD_DENSITY, s.lat.rho)):
            got = L.read(what)
            np.testing.assert_array_equal(got, want.reshape(got.shape))
