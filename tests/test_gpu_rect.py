"""GPU: the runtime-shape kernel (kronmult{d}_vbatched, vectors in shared
memory) against the oracle: sizes with and without a compiled fibre pass (1,
8, 9, 17), every group size, one entry and several entries a group, x on and
off 16-byte alignment, distinct and aliasing outputs.  Normwise relative
error <= 1e-13."""
import numpy as np
import pytest

import kronmult_b200 as kb
import oracle
from tests.golden_cases import rel_err
from tests.gpu_util import dev, host

pytestmark = pytest.mark.gpu

SHAPES = [
    ([1], [1]), ([8], [5]), ([17], [9]), ([2, 3], [4, 1]), ([1, 1, 1], [3, 2, 5]),
    ([4, 6, 3, 8], [6, 3, 8, 4]), ([9, 2, 5], [3, 11, 4]), ([2, 2, 2, 2, 2, 2], [3, 2, 3, 2, 3, 2]),
    ([8, 8, 7], [7, 8, 8]), ([5, 8, 6, 5], [8, 6, 7, 6]), ([6, 6, 5, 6, 3], [5, 4, 6, 6, 7]),
    ([13, 40], [21, 12]),
]


@pytest.mark.parametrize("m,n", SHAPES)
@pytest.mark.parametrize("batch,alias", [(1, False), (37, True), (6007, False)])
def test_rect_vbatched(gpu_lib, m, n, batch, alias):
    import torch

    d, N, M = len(m), int(np.prod(n)), int(np.prod(m))
    batch = min(batch, 4_000_000 // max(N, M) + 1)
    rng = np.random.default_rng(N * 7 + M + batch)
    asz = [a * b for a, b in zip(m, n)]
    off = np.cumsum([0] + asz)
    A = rng.uniform(-1, 1, off[-1] * batch)
    xo = np.arange(batch) * (N + 1)  # every other x off 16-byte alignment when N is even
    X = rng.uniform(-1, 1, (N + 1) * batch)
    ny = (batch + 2) // 3 if alias else batch
    yl = rng.integers(0, ny, size=batch) if alias else np.arange(batch)
    Y0 = rng.uniform(-1, 1, M * ny)
    ao = (off[:-1][None, :] + off[-1] * np.arange(batch)[:, None]).reshape(-1)
    Yref = Y0.copy()
    oracle.kronmult_general(d, m, n, A.ctypes.data + 8 * ao, m, X.ctypes.data + 8 * xo,
                            Yref.ctypes.data + 8 * M * yl)
    at = lambda t, o: t.data_ptr() + 8 * torch.from_numpy(np.asarray(o)).cuda()  # noqa: E731
    dA, dX, dY = dev(A), dev(X), dev(Y0)
    kb.kronmult_vbatched(m, n, at(dA, ao), at(dX, xo), at(dY, M * yl))
    assert rel_err(host(dY), Yref) <= 1e-13
    assert np.array_equal(host(dX), X), "x must be preserved"
