"""GPU: waits of the ring kernel (square d = 6, n = 6..8 with a workspace) that
run out.  With a bound of one poll the computing warps give up on their first
item, some of a group's warps perhaps finding its copies landed: the group
leaves as a whole, its taker and publisher with it.  With a few polls more, the
takers give up on parts of other blocks.  Either way the kernel returns, the
status word reads 1, each element of y is untouched or complete (one add an
element, at the end of its part), and the next call is clean and correct."""
import numpy as np
import pytest

import kronmult_b200 as kb
import oracle
from tests.golden_cases import rel_err
from tests.gpu_util import dev, host

pytestmark = pytest.mark.gpu

D = 6
TOL = {"f64": 1e-13, "f32": 1e-5}


@pytest.fixture(autouse=True)
def _forced():
    kb.tune_clear()
    for n in (6, 7, 8):
        for prec in ("f64", "f32"):
            kb.tune_set(D, n, prec, "big", kb.BIG_RING)
    yield
    kb.lib().kron_set_wait_limit(0)
    kb.tune_clear()


@pytest.mark.parametrize("prec,n,batch", [("f64", 6, 200), ("f64", 7, 90), ("f64", 8, 40),
                                          ("f32", 7, 90), ("f32", 8, 40)])
def test_ring_wait_runs_out(gpu_lib, prec, n, batch):
    import torch

    lib, L = kb.lib(), n ** D
    dt = torch.float64 if prec == "f64" else torch.float32
    f = kb.kronmult_batched if prec == "f64" else kb.kronmult_batched_f32
    rng = np.random.default_rng(860 + n)
    A = rng.standard_normal(n * n * D * batch) / np.sqrt(n)
    X, Y0 = rng.uniform(-1, 1, L * batch), rng.uniform(-1, 1, L * batch)
    Yref = Y0.copy()
    oracle.kronmult_batched(D, n, A, X, Yref)
    dA, dX = dev(A, dt), dev(X, dt)
    W = torch.empty(L * batch, dtype=dt, device="cuda")
    old = host(dev(Y0, dt)).astype(np.float64)
    near = 100 * TOL[prec] * np.abs(Yref).max()  # an element against the norm's bar
    assert lib.kron_device_status(1) in (0, 1)
    for limit in (1, 6, 40):
        dY = dev(Y0, dt)
        assert lib.kron_set_wait_limit(limit) == 0
        f(D, n, dA, dX, dY, W)
        torch.cuda.synchronize()
        assert lib.kron_set_wait_limit(0) == 0
        status, got = lib.kron_device_status(1), host(dY).astype(np.float64)
        done = np.abs(got - Yref) <= near
        assert np.all(done | (got == old))
        assert status == 1 or (limit > 1 and np.all(done))
        dY = dev(Y0, dt)
        f(D, n, dA, dX, dY, W)
        assert rel_err(host(dY).astype(np.float64), Yref) <= TOL[prec]
        assert lib.kron_device_status(1) == 0
