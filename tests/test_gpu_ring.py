"""GPU: the ring kernel (square d = 6, n = 6..8, FP64 and FP32, with a
workspace) against the oracle, through the C ABI.

Sizes where it can go wrong: three entries (the fewest it takes), batches
below and beyond the ring, so that its slots are written again, a workspace
of three vectors (a ring of two), x and y off 16-byte alignment, factors with
lda > n, outputs that alias, and factors with an infinite element (n = 7 runs
zero padded to 8 on the tensor cores).
FP64 bar: normwise relative error <= 1e-13; FP32 <= 1e-5."""
import numpy as np
import pytest

import kronmult_b200 as kb
import oracle
from tests.golden_cases import rel_err
from tests.gpu_util import dev, host, ptrs

pytestmark = pytest.mark.gpu

D = 6
TOL = {"f64": 1e-13, "f32": 1e-5}


@pytest.fixture(autouse=True)
def _forced():
    kb.tune_clear()
    for n in (6, 7, 8):
        for prec in ("f64", "f32"):
            kb.tune_set(D, n, prec, "big", kb.BIG_RING)
    kb.lib().kron_set_wait_limit(1 << 20)
    yield
    kb.lib().kron_set_wait_limit(0)
    kb.tune_clear()


def _inputs(n, batch, seed):
    rng = np.random.default_rng(seed)
    L = n ** D
    A = rng.standard_normal(n * n * D * batch) / np.sqrt(n)
    return A, rng.uniform(-1, 1, L * batch), rng.uniform(-1, 1, L * batch)


@pytest.mark.parametrize("prec", ["f64", "f32"])
@pytest.mark.parametrize("n,batch", [(6, 3), (6, 10), (6, 330), (7, 3), (7, 90), (8, 3), (8, 45)])
def test_ring_batched(gpu_lib, prec, n, batch):
    import torch

    dt = torch.float64 if prec == "f64" else torch.float32
    A, X, Y0 = _inputs(n, batch, 900 + n + batch)
    Yref = Y0.copy()
    oracle.kronmult_batched(D, n, A, X, Yref)
    dA, dX, dY = dev(A, dt), dev(X, dt), dev(Y0, dt)
    X0 = dX.clone()
    W = torch.full((n ** D * batch,), float("nan"), dtype=dt, device="cuda")
    f = kb.kronmult_batched if prec == "f64" else kb.kronmult_batched_f32
    f(D, n, dA, dX, dY, W)
    assert rel_err(host(dY).astype(np.float64), Yref) <= TOL[prec]
    assert torch.equal(dX, X0), "x must be preserved"
    assert kb.lib().kron_device_status(1) == 0


@pytest.mark.parametrize("n", [6, 7, 8])
@pytest.mark.parametrize("xoff,yoff,slots", [(0, 0, 4), (1, 0, 24), (0, 1, 40), (1, 1, 4)])
def test_ring_xbatched(gpu_lib, n, xoff, yoff, slots):
    """lda > n, x and y shifted by one element, aliasing outputs, rings of
    three vectors and more."""
    import torch

    batch, lda, npool, L = 21, n + 2, 5, n ** D
    rng = np.random.default_rng(940 + n + xoff + 2 * yoff)
    Apool = rng.standard_normal(lda * n * npool * D) / np.sqrt(n)
    X = rng.uniform(-1, 1, L * batch + xoff)
    Y0 = rng.uniform(-1, 1, L * batch + yoff)
    aidx = rng.integers(0, npool, size=(batch, D))
    yl = rng.integers(0, 9, size=batch)
    aoff = [lda * n * (l * npool + int(aidx[k, l])) for k in range(batch) for l in range(D)]
    Yref = Y0.copy()
    oracle.kronmult_general(D, [n] * D, [n] * D, [Apool.ctypes.data + 8 * o for o in aoff],
                            [lda] * D, [X.ctypes.data + 8 * (xoff + L * k) for k in range(batch)],
                            [Yref.ctypes.data + 8 * (yoff + L * int(k)) for k in yl])
    dAp, dX, dY = dev(Apool), dev(X), dev(Y0)
    W = torch.empty(L * slots, dtype=torch.float64, device="cuda")
    pA = ptrs(dAp, aoff)
    pX = ptrs(dX, [xoff + L * k for k in range(batch)])
    pY = ptrs(dY, [yoff + L * int(k) for k in yl])
    pW = ptrs(W, [L * s for s in range(slots)])
    kb.kronmult_xbatched(D, n, pA, lda, pX, pY, pW, subbatch=slots // 2)
    assert rel_err(host(dY), Yref) <= TOL["f64"]
    assert kb.lib().kron_device_status(1) == 0


@pytest.mark.parametrize("n", [6, 7, 8])
@pytest.mark.parametrize("mode", range(D))
def test_ring_infinite_factor(gpu_lib, n, mode):
    """An infinite element in row i of A_l spoils the outputs with i_l = i and
    no others."""
    import torch

    batch, L = 3, n ** D
    A, X, Y0 = _inputs(n, batch, 970 + n)
    A.reshape(batch, D, n, n)[1, mode, 2, 4] = np.inf  # column 2, row 4
    dY = dev(Y0)
    W = torch.empty(L * batch, dtype=torch.float64, device="cuda")
    kb.kronmult_batched(D, n, dev(A), dev(X), dY, W)
    Yref = Y0.copy()
    oracle.kronmult_batched(D, n, A, X, Yref)
    got, ref = host(dY), Yref
    fine = np.isfinite(ref)
    assert np.array_equal(np.isfinite(got), fine)
    assert rel_err(got[fine], ref[fine]) <= TOL["f64"]
