"""The integer collision of double populations: bit for bit the double one.

On the CPU the header that the kernels compile is compared with plain double
arithmetic over random cells, noise from 1e-12 to 0.5, flows up to and beyond
the accepted speeds, and values that refuse it.  On the GPU the step kernels
are compared with the oracle from states whose cells take every way: the
integer one, the refusal to double arithmetic for populations, densities or
speeds out of range, lid speeds on and off the grid, walls, ghosts and flags
that only stream.
"""
from __future__ import annotations

import subprocess
from pathlib import Path

import numpy as np
import pytest

from helpers import n_diff

ROOT = Path(__file__).resolve().parent.parent


@pytest.mark.parametrize("seed", [1, 2])
def test_integer_collision_equals_double_arithmetic(tmp_path, seed):
    exe = tmp_path / "fix64_probe"
    subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-x", "c++",
                    "-I", str(ROOT / "turbulent_lbm_multigpu_gb300" / "csrc"), str(ROOT / "tests/cpp/fix64_probe.cpp"),
                    "-o", str(exe)], check=True)
    r = subprocess.run([str(exe), str(seed), "1000000"], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout


def _wild(rng, dims, lo, hi):
    """Populations around rest, with cells of low and high density, high speed, negative, zero and boundary values."""
    w = np.array([1 / 18] * 4 + [1 / 36] * 12 + [1 / 18] * 2 + [1 / 3])
    n = dims[0] * dims[1] * dims[2]
    f = w[:, None] * (1 + 0.01 * rng.standard_normal((19, n)))
    kind = rng.integers(0, 10, n)
    f[:, kind == 0] *= lo  # densities on either side of the accepted ones
    f[:, kind == 1] *= hi
    f[0, kind == 2] *= 3.5  # a speed of 0.13
    k = kind == 3
    f[:, k] = rng.choice([-0.02, 0.0, 2.0 ** -9, 2.0 ** -3, np.nextafter(2.0 ** -3, 0), 0.05], (19, int(k.sum())))
    f[18, kind == 4] = rng.choice([0.5, np.nextafter(0.5, 0), 0.1])
    k = kind == 5  # large differences from equilibrium, ordinary populations
    f[:18, k] = np.exp2(rng.uniform(-6.5, -4, (18, int(k.sum()))))
    return f.reshape(19, dims[2], dims[1], dims[0])


@pytest.mark.gpu
@pytest.mark.parametrize("cs", [0.0, 0.17])
@pytest.mark.parametrize("lid", [0.1, -0.06, 0.0, 1e-4, 0.3])
@pytest.mark.parametrize("dims", [(13, 9, 8), (40, 17, 11)])
def test_steps_from_wild_states_match_oracle(capi, oracle_mod, dims, lid, cs):
    api, O = capi, oracle_mod
    rng = np.random.default_rng(5)
    p = O.Params.lattice(0.56, lid, cs, dtype=np.float64)
    flags = np.full(dims[::-1], api.FLAG_FLUID, np.int32)
    flags[0], flags[:, 0], flags[:, :, -1] = 1, 8, 1
    flags[1:-1, -2, 1:-1] = api.FLAG_VELOCITY_INJECTION
    flags[2, 3, 3:7] = 16  # streams unchanged
    state = _wild(rng, dims, 0.8, 1.9)
    for parity in (0, 1):
        L = api.Lattice(*dims, api.F64, True, True)
        L.set_params(api.Params.make(p.inv_tau, p.tau0, p.les_c, p.gravity, p.lid))
        L.init([1] * 6)
        s = O.single(O.OracleKernels("f64"), dims, p, "f64")
        for what, a in ((api.FIELD_FLAGS, flags), (api.FIELD_DD, state)):
            L.write(what, a)
        s.lat.flags[...] = flags.reshape(s.lat.flags.shape)
        s.lat.dd[...] = state.reshape(s.lat.dd.shape)
        if parity:
            s.lat.counter = 1
        for k in range(2):
            L.step((parity + k) & 1)
            s.step()
            for what, want in ((api.FIELD_DD, s.lat.dd), (api.FIELD_VELOCITY, s.lat.vel), (api.FIELD_DENSITY, s.lat.rho)):
                got = L.read(what)
                assert n_diff(got, want.reshape(got.shape)) == 0, (parity, k, what)
