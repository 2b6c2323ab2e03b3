"""The solve server keeps released solves' device memory for later ones: that
must not keep a solve out that fits the budget, change a result, or hold
memory while the server has nothing to run."""
from __future__ import annotations

import pytest
import torch

from helpers import n_diff
from test_gpu_batch import lone

pytestmark = pytest.mark.gpu


def _bytes(dims):
    """Budget share of a cavity's fields: 19 float planes, flags, velocity."""
    n = dims[0] * dims[1] * dims[2]
    up = lambda v, m: (v + m - 1) // m * m
    return up(n, 64) * 19 * 4 + up(n, 256) + n * 12 + 4096


def _finish(S, ids):
    left = set(ids)
    for _ in range(1000):
        if not left:
            return
        S.tick()
        left -= set(S.poll())
    raise AssertionError("solves did not finish")


def test_kept_memory_keeps_no_solve_out(capi):
    """A small solve after a released larger one, and solves that fill the rest of the budget: all run at once."""
    api = capi
    big, small = (40, 40, 40), (40, 40, 33)
    make = lambda d, k: api.Cavity.make(d, api.F32, 0.56, 0.17, 0.05, 6, k, 1e-2)
    S = api.Server(hbm_budget_bytes=_bytes(small) + 8 * _bytes(big))
    first = S.submit(make(big, 1))
    _finish(S, [first])
    S.release(first)
    cav = [make(small, 2)] + [make(big, 3 + k) for k in range(8)]
    ids = [S.submit(c) for c in cav]
    assert S.tick(max_steps=1) == 9
    assert S.status()["hbm_used"] == _bytes(small) + 8 * _bytes(big)
    _finish(S, ids)
    for sid, c in ((ids[0], cav[0]), (ids[1], cav[1]), (ids[8], cav[8])):
        assert n_diff(S.lattice(sid).read(api.FIELD_DD), lone(api, c).read(api.FIELD_DD)) == 0
    for sid in ids:
        S.release(sid)


def test_an_idle_server_holds_no_memory(capi):
    api = capi
    dims = (160, 160, 128)
    S = api.Server(hbm_budget_bytes=64 * _bytes(dims))
    warm = api.Lattice(32, 32, 32, api.F32, True, False)  # context and modules are loaded before the first look
    warm.run(0, 2)
    api.synchronize()
    free = torch.cuda.mem_get_info()[0]
    ids = [S.submit(api.Cavity.make(dims, api.F32, 0.56, 0.17, 0.05, 4, k, 1e-2)) for k in range(3)]
    _finish(S, ids)
    for sid in ids:
        S.release(sid)
    assert S.tick() == 0
    assert torch.cuda.mem_get_info()[0] >= free - (64 << 20)
    again = S.submit(api.Cavity.make(dims, api.F32, 0.56, 0.17, 0.05, 4, 9, 1e-2))
    _finish(S, [again])
    assert n_diff(S.lattice(again).read(api.FIELD_DD),
                  lone(api, api.Cavity.make(dims, api.F32, 0.56, 0.17, 0.05, 4, 9, 1e-2)).read(api.FIELD_DD)) == 0
