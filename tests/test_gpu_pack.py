"""GPU: the packed kernel (several short vectors a warp) against the oracle,
through the C ABI: every (d, n) it takes, one entry, a partly filled warp and
several steps a warp (both stages and the pointer prefetch), x off 16-byte
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

SHAPES = [(3, 2), (4, 2), (5, 2), (6, 2), (3, 3), (4, 3), (5, 3), (3, 4), (4, 4), (3, 5)]
TOL = {"f64": 1e-13, "f32": 1e-5}


@pytest.fixture(autouse=True)
def _forced():
    for d, n in SHAPES:
        for prec in ("f64", "f32"):
            kb.tune_set(d, n, prec, "sq", kb.SQ_PACK)
    yield
    kb.tune_clear()


@pytest.mark.parametrize("prec", ["f64", "f32"])
@pytest.mark.parametrize("d,n", SHAPES)
def test_pack_batched(gpu_lib, prec, d, n):
    import torch

    dt = torch.float64 if prec == "f64" else torch.float32
    L = n ** d
    for batch, off in ((1, 0), (11, 1), (50003, 0)):
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
def test_pack_xbatched_and_segmented(gpu_lib, d, n):
    import torch

    L, lda, npool, batch = n ** d, n + 3, 7, 50003
    rng = np.random.default_rng(17 * d + n)
    A = rng.uniform(-1, 1, lda * n * npool)
    X, Y0 = rng.uniform(-1, 1, L * 50), rng.uniform(-1, 1, L * 900)
    xl = rng.integers(0, 50, size=batch)
    yl = np.repeat(rng.integers(0, 900, size=batch), rng.integers(1, 6, size=batch))[:batch]
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


@pytest.mark.parametrize("n", [3, 4, 5])
def test_builtin_choice_at_d3(gpu_lib, n):
    """Either side of the built-in rule's lines at d = 3: batched entries, and
    shared factors with and without segments."""
    import torch

    kb.tune_clear()
    L, npool = n ** 3, 7
    rng = np.random.default_rng(n)
    for batch in (39999, 40000):
        A, X, Y0 = (rng.uniform(-1, 1, s * batch) for s in (3 * n * n, L, L))
        for prec, dt, f in (("f64", torch.float64, kb.kronmult_batched),
                            ("f32", torch.float32, kb.kronmult_batched_f32)):
            Yref = Y0.copy()
            oracle.kronmult_batched(3, n, A, X, Yref)
            dY = dev(Y0, dt)
            f(3, n, dev(A, dt), dev(X, dt), dY, None)
            assert rel_err(host(dY).astype(np.float64), Yref) <= TOL[prec], batch
    A, X = rng.uniform(-1, 1, n * n * npool), rng.uniform(-1, 1, L * 50)
    dA, dX = dev(A), dev(X)
    at = lambda t, o: t.data_ptr() + 8 * torch.from_numpy(np.asarray(o)).cuda()  # noqa: E731
    for groups in (2367, 2369, 4000):
        Y0 = rng.uniform(-1, 1, L * groups)
        yl = np.repeat(np.arange(groups), 2)
        xl, al = rng.integers(0, 50, 2 * groups), rng.integers(0, npool, 6 * groups)
        Yref = Y0.copy()
        oracle.kronmult_general(3, [n] * 3, [n] * 3, A.ctypes.data + 8 * n * n * al, [n] * 3,
                                X.ctypes.data + 8 * L * xl, Yref.ctypes.data + 8 * L * yl)
        pA, pX = at(dA, n * n * al), at(dX, L * xl)
        dY = dev(Y0)
        kb.kronmult_xbatched(3, n, pA, n, pX, at(dY, L * yl))
        assert rel_err(host(dY), Yref) <= TOL["f64"], groups
        dY = dev(Y0)
        pY = at(dY, L * yl)
        kb.kronmult_xbatched_segmented(3, n, pA, n, pX, pY, kb.Segments(pY))
        assert rel_err(host(dY), Yref) <= TOL["f64"], groups


@pytest.mark.parametrize("groups,hi", [(1, 300), (4000, 2), (4737, 3), (9000, 60), (20001, 2)])
def test_segment_ranges(gpu_lib, groups, hi):
    """Groups of very unequal length, so that warps' ranges start far from
    where equal ones would: fewer groups than warps, and more."""
    import torch

    d, n, L, npool = 3, 2, 8, 5
    rng = np.random.default_rng(groups)
    runs = np.sort(rng.integers(1, hi + 1, groups))
    runs[groups // 3] = 3000
    yl = np.repeat(np.arange(groups), runs)
    batch = len(yl)
    A, X, Y0 = (rng.uniform(-1, 1, s) for s in (4 * npool, L * 50, L * groups))
    xl, al = rng.integers(0, 50, batch), rng.integers(0, npool, d * batch)
    Yref = Y0.copy()
    oracle.kronmult_general(d, [n] * d, [n] * d, A.ctypes.data + 32 * al, [n] * d,
                            X.ctypes.data + 8 * L * xl, Yref.ctypes.data + 8 * L * yl)
    dA, dX, dY = dev(A), dev(X), dev(Y0)
    at = lambda t, o: t.data_ptr() + 8 * torch.from_numpy(np.asarray(o)).cuda()  # noqa: E731
    pY = at(dY, L * yl)
    kb.tune_clear()
    kb.kronmult_xbatched_segmented(d, n, at(dA, 4 * al), n, at(dX, L * xl), pY, kb.Segments(pY))
    assert rel_err(host(dY), Yref) <= TOL["f64"]
