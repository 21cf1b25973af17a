"""GPU: the resident kernel (square d = 6, n = 6 in FP32; the vector in one
block's shared memory, no workspace) against the oracle, through the C ABI.

Sizes where it can go wrong: one entry, fewer entries than blocks, several
entries a block (the rows' buffer and mbarriers are used again), x and y off
16-byte alignment, and a wait that runs out.  Bar: normwise relative error
<= 1e-5."""
import numpy as np
import pytest

import kronmult_b200 as kb
import oracle
from tests.golden_cases import rel_err
from tests.gpu_util import dev, host

pytestmark = pytest.mark.gpu

D, N = 6, 6
L = N ** D
TOL = 1e-5


@pytest.fixture(autouse=True)
def _forced():
    kb.tune_set(D, N, "f32", "slab", kb.SLAB_RESIDENT)
    kb.lib().kron_set_wait_limit(1 << 20)
    yield
    kb.lib().kron_set_wait_limit(0)
    kb.tune_clear()


def _inputs(batch, seed):
    rng = np.random.default_rng(seed)
    A = rng.standard_normal(N * N * D * batch) / np.sqrt(N)
    return A, rng.uniform(-1, 1, L * batch), rng.uniform(-1, 1, L * batch)


@pytest.mark.parametrize("batch", [1, 50, 149, 320])
def test_resident_batched(gpu_lib, batch):
    import torch

    dt = torch.float32
    A, X, Y0 = _inputs(batch, 800 + batch)
    Yref = Y0.copy()
    oracle.kronmult_batched(D, N, A, X, Yref)
    dA, dX, dY = dev(A, dt), dev(X, dt), dev(Y0, dt)
    X0 = dX.clone()
    f = kb.kronmult_batched_f32
    f(D, N, dA, dX, dY, None)
    assert rel_err(host(dY).astype(np.float64), Yref) <= TOL
    assert torch.equal(dX, X0), "x must be preserved"
    assert kb.lib().kron_device_status(1) == 0


@pytest.mark.parametrize("off", [1, 2])
def test_resident_unaligned(gpu_lib, off):
    """x and y `off` elements off 16-byte alignment."""
    import torch

    batch = 160
    dt = torch.float32
    A, X, Y0 = _inputs(batch, 830 + off)
    Yref = Y0.copy()
    oracle.kronmult_batched(D, N, A, X, Yref)
    dX = torch.empty(L * batch + off, dtype=dt, device="cuda")[off:]
    dY = torch.empty(L * batch + off, dtype=dt, device="cuda")[off:]
    dX.copy_(dev(X, dt))
    dY.copy_(dev(Y0, dt))
    f = kb.kronmult_batched_f32
    f(D, N, dev(A, dt), dX, dY, None)
    assert rel_err(host(dY).astype(np.float64), Yref) <= TOL
    assert kb.lib().kron_device_status(1) == 0


def test_resident_wait_runs_out(gpu_lib):
    """A bound of one poll: the first entry's copies are not there yet.  The
    status word reads 1, y of that block's entries is untouched or complete,
    and the next call is clean."""
    import torch

    lib, batch = kb.lib(), 300
    dt = torch.float32
    A, X, Y0 = _inputs(batch, 850)
    f = kb.kronmult_batched_f32
    dA, dX, dY = dev(A, dt), dev(X, dt), dev(Y0, dt)
    assert lib.kron_device_status(1) in (0, 1)
    assert lib.kron_set_wait_limit(1) == 0
    f(D, N, dA, dX, dY, None)
    torch.cuda.synchronize()
    assert lib.kron_set_wait_limit(1 << 20) == 0
    assert lib.kron_device_status(1) == 1
    Yref = Y0.copy()
    oracle.kronmult_batched(D, N, A, X, Yref)
    got, old = host(dY).astype(np.float64).reshape(batch, L), Y0.reshape(batch, L)
    for k in range(batch):
        same = np.array_equal(got[k], old[k].astype(np.float32))
        assert same or rel_err(got[k], Yref.reshape(batch, L)[k]) <= TOL
    dY = dev(Y0, dt)
    f(D, N, dA, dX, dY, None)
    assert rel_err(host(dY).astype(np.float64), Yref) <= TOL
    assert lib.kron_device_status(1) == 0
