"""GPU: the tensor-core kgemm kernel with several entries a block or warp, so
that its loop runs: the next entry's operands and pointers in flight, one stage
or two used again, padding zeroed once for every later entry.  Every form of
it (a warp an entry, whole and ragged; two by two warps, whole and ragged; four
along the rows; four along the columns), leading dimensions that vary from
entry to entry between odd and even, each entry against its product in numpy:
||C - ref|| <= 1e-13 (|alpha| ||A|| ||B|| + |beta| ||C0||)."""
import numpy as np
import pytest

import kronmult_b200 as kb
from tests.gpu_util import dev, host

pytestmark = pytest.mark.gpu

# (mm, nn, kk, entries): more than the blocks an SM times the groups a block
SIZES = [
    (32, 32, 32, 6001), (32, 32, 5, 6001), (32, 32, 64, 6001),  # a warp, whole tiles
    (1, 1, 1, 20003), (8, 8, 8, 20003), (17, 9, 33, 6001), (31, 32, 64, 6001),  # a warp, ragged
    (64, 64, 64, 2503), (64, 64, 16, 2503), (64, 64, 1, 2503),  # 2 x 2 warps, whole
    (64, 40, 64, 2503), (33, 64, 29, 2503), (49, 41, 7, 2503),  # 2 x 2 warps, ragged
    (64, 8, 64, 2503), (50, 24, 9, 2503),                       # along the rows
    (16, 64, 64, 2503), (48, 32, 40, 2503), (9, 57, 31, 2503),  # along the columns
]


class _Stack:
    """`batch` column-major matrices of rows x cols, entry e with leading
    dimension rows + e % 3, in slots of (rows + 2) cols elements (and one, so
    that every other one starts off 16-byte alignment)."""

    def __init__(self, rows, cols, batch, rng):
        self.rows, self.cols, self.batch = rows, cols, batch
        self.slot = (rows + 2) * cols + 1
        self.flat = rng.uniform(-1, 1, (batch, self.slot))
        self.ld = rows + np.arange(batch) % 3

    def dense(self, flat=None):
        flat = self.flat if flat is None else flat.reshape(self.batch, self.slot)
        out = np.empty((self.batch, self.rows, self.cols))
        for c in range(3):
            ld = self.rows + c
            part = flat[c::3, :ld * self.cols].reshape(-1, self.cols, ld)
            out[c::3] = part[:, :, :self.rows].transpose(0, 2, 1)
        return out

    def device(self):
        import torch

        t = dev(self.flat.reshape(-1))
        at = t.data_ptr() + 8 * self.slot * torch.arange(self.batch, device="cuda")
        return t, at, torch.from_numpy(self.ld.astype(np.int32)).cuda()


@pytest.mark.parametrize("op", ["nn", "nt", "tt"])
@pytest.mark.parametrize("mm,nn,kk,batch", SIZES)
def test_kgemm_many_entries(gpu_lib, op, mm, nn, kk, batch):
    rng = np.random.default_rng(mm * 64 * 64 + nn * 64 + kk)
    A = _Stack(*((kk, mm) if op == "tt" else (mm, kk)), batch, rng)
    B = _Stack(*((kk, nn) if op == "nn" else (nn, kk)), batch, rng)
    C = _Stack(mm, nn, batch, rng)
    a, b, c = A.dense(), B.dense(), C.dense()
    if op == "tt":
        a = a.transpose(0, 2, 1)
    if op != "nn":
        b = b.transpose(0, 2, 1)
    ab = np.matmul(a, b)
    norm = lambda t: np.sqrt((t * t).sum(axis=(1, 2)))  # noqa: E731
    tA, pA, ldA = A.device()
    tB, pB, ldB = B.device()
    for alpha, beta in ((1.3, 1.0), (0.7, 0.0), (-1.1, 0.5)):
        tC, pC, ldC = C.device()
        kb.kgemm_batched(op, mm, nn, kk, alpha, pA, ldA, pB, ldB, beta, pC, ldC)
        got = host(tC)
        err = norm(C.dense(got) - (alpha * ab + beta * c))
        assert np.all(err <= 1e-13 * (abs(alpha) * norm(a) * norm(b) + abs(beta) * norm(c)))
        # what lies between the columns and the entries is untouched
        left = got.reshape(batch, C.slot).copy()
        for k in range(3):
            ld = mm + k
            v = left[k::3, :ld * nn].reshape(-1, nn, ld)
            v[:, :, :mm] = C.flat[k::3, :ld * nn].reshape(-1, nn, ld)[:, :, :mm]
            left[k::3, :ld * nn] = v.reshape(v.shape[0], -1)
        assert np.array_equal(left, C.flat)
