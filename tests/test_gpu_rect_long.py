"""GPU: the runtime-shape kernel at sizes beyond 8, which it runs a thread an
output element: against the oracle at the edges of its group and block sizes
(one group, several, one block of 512 threads, the largest that fits), and no
slower than the general kernel on short vectors with long modes, where a thread
a fibre left most of a group idle (d = 2, n = 32: four times slower).  Normwise
relative error <= 1e-13."""
import os

import numpy as np
import pytest

import kronmult_b200 as kb
import oracle
from tests.golden_cases import rel_err
from tests.gpu_util import dev, host

pytestmark = pytest.mark.gpu

SHAPES = [
    ([9], [1]), ([1], [9]), ([255], [17]), ([17], [255]), ([64], [64]), ([118], [118]),
    ([119], [118]), ([255, 1], [2, 9]), ([32, 33], [31, 32]), ([48, 48], [48, 48]),
    ([9, 9, 9], [9, 9, 9]), ([16, 4, 4], [4, 4, 16]), ([13, 13, 13], [13, 13, 13]),
    ([18, 18, 18], [18, 18, 18]), ([21, 21, 21], [20, 21, 21]), ([21, 21, 21], [22, 21, 22]),
    ([2, 9, 2, 9], [9, 2, 9, 2]), ([7, 8, 7, 8], [8, 7, 8, 7]), ([8, 8, 8, 8, 2], [7, 8, 7, 8, 2]),
    ([9, 9, 9, 9], [9, 9, 9, 9]),
]


@pytest.mark.parametrize("m,n", SHAPES)
@pytest.mark.parametrize("batch", [1, 700])
def test_rect_long_modes(gpu_lib, m, n, batch):
    import torch

    d, N, M = len(m), int(np.prod(n)), int(np.prod(m))
    rng = np.random.default_rng(N * 5 + M + batch)
    off = np.cumsum([0] + [a * b for a, b in zip(m, n)])
    batch = min(batch, 4_000_000 // max(N, M, int(off[-1])) + 1)
    A, X = rng.uniform(-1, 1, off[-1] * batch), rng.uniform(-1, 1, (N + 1) * batch)
    Y0 = rng.uniform(-1, 1, M * batch)
    ao = (off[:-1][None, :] + off[-1] * np.arange(batch)[:, None]).reshape(-1)
    xo, yo = (N + 1) * np.arange(batch), M * np.arange(batch)
    Yref = Y0.copy()
    oracle.kronmult_general(d, m, n, A.ctypes.data + 8 * ao, m, X.ctypes.data + 8 * xo,
                            Yref.ctypes.data + 8 * yo)
    at = lambda t, o: t.data_ptr() + 8 * torch.from_numpy(np.asarray(o)).cuda()  # noqa: E731
    dA, dX, dY = dev(A), dev(X), dev(Y0)
    W = torch.empty(4 * (N + M) * batch, dtype=torch.float64, device="cuda")
    kb.kronmult_vbatched(m, n, at(dA, ao), at(dX, xo), at(dY, yo), W)
    assert rel_err(host(dY), Yref) <= 1e-13


def _time(f):
    import torch

    start, end = (torch.cuda.Event(enable_timing=True) for _ in range(2))
    best = 1e9
    for _ in range(7):
        start.record()
        for _ in range(20):
            f()
        end.record()
        end.synchronize()
        best = min(best, start.elapsed_time(end))
    return best


@pytest.mark.parametrize("d,n,batch", [(1, 64, 500), (2, 16, 5000), (2, 32, 100), (3, 16, 500)])
def test_no_slower_than_the_general_kernel(gpu_lib, d, n, batch):
    import torch

    A = torch.rand(batch * d * n * n, dtype=torch.float64, device="cuda")
    X = torch.rand(batch * n ** d, dtype=torch.float64, device="cuda")
    Y = torch.zeros_like(X)
    call = lambda: kb.kronmult_batched(d, n, A, X, Y)  # noqa: E731
    built_in = _time(call)
    os.environ["KRON_DISABLE_RECT"] = "1"
    try:
        general = _time(call)
    finally:
        del os.environ["KRON_DISABLE_RECT"]
    assert built_in <= 1.25 * general, (built_in, general)
