"""GPU: the pipelined and the cluster two-phase kernel at shapes where the
built-in order now prefers others (the pair and the ring kernel), asked for
through the tuning table: enough entries that every pipeline stage is used
again, odd vector lengths, pointer layouts with vectors off 16-byte alignment
and lda > n, outputs that alias.  Against the oracle, normwise relative error <=
1e-13 (FP64), 1e-5 (FP32)."""
import numpy as np
import pytest

import kronmult_b200 as kb
import oracle
from tests.golden_cases import rel_err
from tests.gpu_util import dev, host, ptrs

pytestmark = pytest.mark.gpu

TOL = {"f64": 1e-13, "f32": 1e-5}


@pytest.fixture(autouse=True)
def _clean():
    kb.tune_clear()
    yield
    kb.tune_clear()


def _case(d, n, batch, seed):
    rng = np.random.default_rng(seed)
    L = n ** d
    return (rng.standard_normal(n * n * d * batch) / np.sqrt(n), rng.uniform(-1, 1, L * batch),
            rng.uniform(-1, 1, L * batch))


@pytest.mark.parametrize("variant,d,n,prec,batch", [
    ("pipe", 6, 3, "f64", 1200), ("pipe", 5, 5, "f64", 1200), ("pipe", 4, 5, "f64", 1200),
    ("pipe", 6, 4, "f64", 1200), ("pipe", 5, 4, "f64", 1200), ("pipe", 6, 4, "f32", 1800),
    ("pipe", 5, 4, "f32", 1800), ("pipe", 5, 5, "f32", 1800), ("pipe", 6, 5, "f32", 900),
    ("pipe", 4, 5, "f32", 3), ("big", 6, 7, "f64", 3), ("big", 6, 7, "f64", 40),
    ("big", 6, 8, "f64", 5), ("big", 6, 7, "f32", 5), ("big", 6, 8, "f32", 5),
])
def test_forced_batched(gpu_lib, variant, d, n, prec, batch):
    import torch

    kb.tune_set(d, n, prec, variant, 0)
    dt = torch.float64 if prec == "f64" else torch.float32
    A, X, Y0 = _case(d, n, batch, 600 + 10 * d + n + batch)
    Yref = Y0.copy()
    oracle.kronmult_batched(d, n, A, X, Yref)
    dY = dev(Y0, dt)
    W = torch.empty(n ** d * batch, dtype=dt, device="cuda") if variant == "big" else None
    f = kb.kronmult_batched if prec == "f64" else kb.kronmult_batched_f32
    f(d, n, dev(A, dt), dev(X, dt), dY, W)
    assert rel_err(host(dY).astype(np.float64), Yref) <= TOL[prec]
    assert kb.lib().kron_device_status(1) == 0


@pytest.mark.parametrize("variant,d,n,batch", [("pipe", 6, 3, 700), ("pipe", 4, 5, 900),
                                               ("pipe", 5, 5, 700), ("pipe", 6, 4, 700),
                                               ("pipe", 5, 4, 700), ("big", 6, 7, 9),
                                               ("big", 6, 8, 7)])
@pytest.mark.parametrize("off", [0, 1])
def test_forced_xbatched(gpu_lib, variant, d, n, batch, off):
    import torch

    kb.tune_set(d, n, "f64", variant, 0)
    L, lda, npool, slots = n ** d, n + 1, 6, 6
    rng = np.random.default_rng(650 + 10 * d + n + off)
    A = rng.standard_normal(lda * n * npool * d) / np.sqrt(n)
    X, Y0 = rng.uniform(-1, 1, L * batch + off), rng.uniform(-1, 1, L * batch + off)
    yl = np.sort(rng.integers(0, (batch + 1) // 2, size=batch))
    aoff = [lda * n * int(q) for q in rng.integers(0, npool * d, size=batch * d)]
    Yref = Y0.copy()
    oracle.kronmult_general(d, [n] * d, [n] * d, [A.ctypes.data + 8 * o for o in aoff], [lda] * d,
                            [X.ctypes.data + 8 * (off + L * k) for k in range(batch)],
                            [Yref.ctypes.data + 8 * (off + L * int(k)) for k in yl])
    dA, dX, dY = dev(A), dev(X), dev(Y0)
    W = torch.empty(L * slots, dtype=torch.float64, device="cuda")
    kb.kronmult_xbatched(d, n, ptrs(dA, aoff), lda, ptrs(dX, [off + L * k for k in range(batch)]),
                         ptrs(dY, [off + L * int(k) for k in yl]),
                         ptrs(W, [L * s for s in range(slots)]), subbatch=slots // 2)
    assert rel_err(host(dY), Yref) <= TOL["f64"]
    assert kb.lib().kron_device_status(1) == 0
