"""GPU: the pair kernel (a block an entry, two modes a pass) against the
oracle, through the C ABI: every (d, n) it takes, one entry and several a
block (both stages, the single one, the pointer prefetch), x off 16-byte
alignment, factors with lda > n, runs of equal outputs, and the segmented
mode's bitwise reproducibility.  FP64 bar: normwise relative error <= 1e-13;
FP32 <= 1e-5."""
import numpy as np
import pytest

import kronmult_b200 as kb
import oracle
from tests.golden_cases import rel_err
from tests.gpu_util import dev, host

pytestmark = pytest.mark.gpu

SHAPES = [(6, 3), (5, 4), (4, 5), (5, 5), (6, 5), (4, 6), (5, 6), (4, 7), (5, 7), (4, 8)]
TOL = {"f64": 1e-13, "f32": 1e-5}


@pytest.fixture(autouse=True)
def _forced():
    for d, n in SHAPES:
        for prec in ("f64", "f32"):
            kb.tune_set(d, n, prec, "sq", kb.SQ_PAIR)
    yield
    kb.tune_clear()


@pytest.mark.parametrize("prec", ["f64", "f32"])
@pytest.mark.parametrize("d,n", SHAPES)
def test_pair_batched(gpu_lib, prec, d, n):
    import torch

    dt = torch.float64 if prec == "f64" else torch.float32
    L = n ** d
    for batch, off in ((1, 0), (11, 1), (min(5003, 24_000_000 // L), 0)):
        rng = np.random.default_rng(100 * d + n + batch)
        A = rng.uniform(-1, 1, n * n * d * batch)
        X, Y0 = (rng.uniform(-1, 1, L * batch) for _ in "xy")
        Yref = Y0.copy()
        oracle.kronmult_batched(d, n, A, X, Yref)
        dX = torch.empty(L * batch + off, dtype=dt, device="cuda")[off:]
        dX.copy_(dev(X, dt))
        dY = dev(Y0, dt)
        f = kb.kronmult_batched if prec == "f64" else kb.kronmult_batched_f32
        f(d, n, dev(A, dt), dX, dY, None)
        assert rel_err(host(dY).astype(np.float64), Yref) <= TOL[prec], (batch, off)
        assert np.array_equal(host(dX), X.astype(host(dX).dtype)), "x must be preserved"


@pytest.mark.parametrize("d,n", SHAPES)
def test_pair_xbatched_and_segmented(gpu_lib, d, n):
    import torch

    L, lda, npool = n ** d, n + 3, 7
    batch = min(5003, 24_000_000 // L)
    rng = np.random.default_rng(17 * d + n)
    A = rng.uniform(-1, 1, lda * n * npool)
    X, Y0 = rng.uniform(-1, 1, L * 50), rng.uniform(-1, 1, L * 300)
    xl = rng.integers(0, 50, size=batch)
    yl = np.repeat(rng.integers(0, 300, size=batch), rng.integers(1, 6, size=batch))[:batch]
    al = rng.integers(0, npool, size=batch * d)
    Yref = Y0.copy()
    oracle.kronmult_general(d, [n] * d, [n] * d, A.ctypes.data + 8 * lda * n * al, [lda] * d,
                            X.ctypes.data + 8 * L * xl, Yref.ctypes.data + 8 * L * yl)
    dA, dX = dev(A), dev(X)
    at = lambda t, o: t.data_ptr() + 8 * torch.from_numpy(np.asarray(o)).cuda()  # noqa: E731
    pA, pX = at(dA, lda * n * al), at(dX, L * xl)
    dY = dev(Y0)
    kb.kronmult_xbatched(d, n, pA, lda, pX, at(dY, L * yl))
    assert rel_err(host(dY), Yref) <= TOL["f64"]
    out = []
    for _ in range(2):
        dY = dev(Y0)
        pY = at(dY, L * yl)
        seg = kb.Segments(pY)
        kb.kronmult_xbatched_segmented(d, n, pA, lda, pX, pY, seg)
        out.append(host(dY))
    assert rel_err(out[0], Yref) <= TOL["f64"]
    assert np.array_equal(out[0], out[1])


@pytest.mark.parametrize("d,n", [(4, 8), (5, 4), (4, 6)])
def test_segments_equal_square_kernel(gpu_lib, d, n):
    """Segmented sums do not depend on which kernel a batch's size selects."""
    import torch

    L, npool, groups = n ** d, 5, 60
    rng = np.random.default_rng(n)
    yl = np.repeat(np.arange(groups), rng.integers(1, 9, groups))
    batch = len(yl)
    dA, dX, Y0 = (rng.uniform(-1, 1, s) for s in (n * n * npool, L * 20, L * groups))
    dA, dX = dev(dA), dev(dX)
    at = lambda t, o: t.data_ptr() + 8 * torch.from_numpy(np.asarray(o)).cuda()  # noqa: E731
    pA = at(dA, n * n * rng.integers(0, npool, batch * d))
    pX = at(dX, L * rng.integers(0, 20, batch))
    out = []
    for param in (kb.SQ_PAIR, 0):
        kb.tune_set(d, n, "f64", "sq", param)
        dY = dev(Y0)
        pY = at(dY, L * yl)
        kb.kronmult_xbatched_segmented(d, n, pA, n, pX, pY, kb.Segments(pY))
        out.append(host(dY))
    assert np.array_equal(out[0], out[1])
