"""Fast flows of double lattices: the integer collision takes them up to
|u_a| + |u_b| = 0.25 and gives the bits of the double arithmetic."""
from __future__ import annotations

import subprocess
from pathlib import Path

import numpy as np
import pytest

from helpers import n_diff

ROOT = Path(__file__).resolve().parent.parent


@pytest.mark.parametrize("seed", [1, 2])
def test_fast_flows_are_accepted_and_equal_double_arithmetic(tmp_path, seed):
    exe = tmp_path / "fix64_fast_probe"
    subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-x", "c++",
                    "-I", str(ROOT / "turbulent_lbm_multigpu_gb300" / "csrc"), str(ROOT / "tests/cpp/fix64_fast_probe.cpp"),
                    "-o", str(exe)], check=True)
    r = subprocess.run([str(exe), str(seed), "1000000"], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout


@pytest.mark.gpu
@pytest.mark.parametrize("cs", [0.0, 0.17])
@pytest.mark.parametrize("u", [(0.2, 0.03, 0.0), (-0.05, 0.0, 0.19), (0.13, 0.12, -0.1), (0.24, 0.02, 0.01)])
def test_steps_of_fast_flows_match_oracle(capi, oracle_mod, u, cs):
    api, O = capi, oracle_mod
    dims = (37, 14, 11)
    rng = np.random.default_rng(3)
    p = O.Params.lattice(0.6, 0.3, cs, dtype=np.float64)
    L = api.Lattice(*dims, api.F64, True, True)
    L.set_params(api.Params.make(p.inv_tau, p.tau0, p.les_c, p.gravity, p.lid))
    L.init([1] * 6)
    L.write(api.FIELD_FLAGS, np.full((dims[2] - 2) * (dims[0] - 2), api.FLAG_VELOCITY_INJECTION, np.int32),
            origin=(1, dims[1] - 2, 1), size=(dims[0] - 2, 1, dims[2] - 2))
    from test_gpu_sums import E, W
    s = (np.array(u)[:, None] * E).sum(0)
    eq = W * (1 + 3 * s + 4.5 * s * s - 1.5 * np.dot(u, u))
    state = eq[:, None, None, None] * (1 + 0.02 * rng.uniform(-1, 1, (19,) + dims[::-1]))
    L.write(api.FIELD_DD, state)
    o = O.single(O.OracleKernels("f64"), dims, p, "f64")
    o.lat.dd[...] = state.reshape(o.lat.dd.shape)
    for k in range(6):
        L.step(k & 1)
        o.step()
        for what, want in ((api.FIELD_DD, o.lat.dd), (api.FIELD_VELOCITY, o.lat.vel), (api.FIELD_DENSITY, o.lat.rho)):
            got = L.read(what)
            assert n_diff(got, want.reshape(got.shape)) == 0, (k, what)
