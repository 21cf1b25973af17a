"""Which shapes an uneven-batch plan takes: those whose two buffers and factors
fit 14208 doubles of shared memory, or have a two-phase split of which each
phase does; at the edge of that (one factor of 118 x 118) plan creation neither
refuses what fits nor takes what does not.  On the CPU creation stops at the
first device allocation, which is behind the shapes' check; the GPU test runs
plans of edge shapes against the oracle (normwise relative error <= 1e-13)."""
import ctypes as C

import numpy as np
import pytest

import kronmult_b200 as kb
import oracle
from tests.golden_cases import rel_err
from tests.gpu_util import dev, host, ptrs

BUDGET = 14208
OK, NOT_SUPPORTED, ALLOC = 0, 4, 5


def _even(v):
    return (v + 1) // 2 * 2


def _largest(m, n):
    """Elements of the largest intermediate in the cheaper order (last mode
    first unless the other way is strictly cheaper)."""
    best = None
    for order in (range(len(m) - 1, -1, -1), range(len(m))):
        dims, flops, top = list(n), 0, int(np.prod(n))
        for l in order:
            flops += m[l] * int(np.prod(dims))
            dims[l] = m[l]
            top = max(top, int(np.prod(dims)))
        if best is None or flops < best[0]:
            best = (flops, top)
    return best[1]


def _fits(m, n):
    asz = [a * b for a, b in zip(m, n)]
    if 2 * _even(_largest(m, n)) + _even(sum(asz)) <= BUDGET:
        return True
    return any(2 * _largest(m[q:], n[q:]) + _even(sum(asz[q:])) + 2 <= BUDGET and
               2 * _largest(m[:q], n[:q]) + _even(sum(asz[:q])) + 2 <= BUDGET
               for q in range(1, len(m)))


def _row(m, n):
    s = np.zeros(13, dtype=np.int32)
    s[0] = len(m)
    s[1:1 + 2 * len(m):2], s[2:2 + 2 * len(m):2] = m, n
    return s


def _create(shapes):
    lib, plan = kb.lib(), C.c_void_p()
    shapes = np.ascontiguousarray(shapes, dtype=np.int32)
    rc = lib.kron_vplan_create(C.byref(plan), len(shapes), shapes.ctypes.data)
    lib.kron_vplan_destroy(plan)
    return rc


EDGE = [([k], [k]) for k in range(112, 124)] + \
       [([k, 3], [n, 2]) for k in range(110, 124) for n in (113, 116, 117, 118, 119)] + \
       [([4, k], [5, n]) for k in range(110, 124) for n in (113, 116, 117, 118, 119)] + \
       [([255, 2], [k, 2]) for k in range(48, 58)] + \
       [([3, k, 2], [2, k - 1, 9]) for k in range(112, 124)]


@pytest.mark.parametrize("m,n", EDGE)
def test_edge_shapes(m, n):
    rc = _create([_row(m, n)])
    assert rc in ((OK, ALLOC) if _fits(m, n) else (NOT_SUPPORTED,))
    # the same among shapes of every class
    rc = _create([_row([2], [3]), _row([8] * 4, [7] * 4), _row(m, n), _row([8] * 6, [8] * 6)])
    assert rc in ((OK, ALLOC) if _fits(m, n) else (NOT_SUPPORTED,))


@pytest.mark.gpu
@pytest.mark.parametrize("m,n", [([118], [118]), ([116], [120]), ([4, 118], [5, 117]),
                                 ([117, 3], [118, 2]), ([255, 2], [53, 2])])
def test_edge_plans_run(gpu_lib, m, n):
    import torch

    assert _fits(m, n)
    entries = [([2], [3]), (m, n), ([8] * 4, [7] * 4), (m, n), ([8] * 6, [8] * 6), (m, n)]
    rng = np.random.default_rng(sum(m) + sum(n))
    ao, xo, yo, na, nx, ny = [], [], [], 0, 1, 0  # x off 16-byte alignment now and then
    for mm, nn in entries:
        for l in range(6):
            ao.append(na)
            na += mm[l] * nn[l] if l < len(mm) else 0
        xo.append(nx)
        yo.append(ny)
        nx, ny = nx + int(np.prod(nn)), ny + int(np.prod(mm))
    A, X, Y0 = rng.uniform(-1, 1, na), rng.uniform(-1, 1, nx), rng.uniform(-1, 1, ny)
    Yref = Y0.copy()
    for k, (mm, nn) in enumerate(entries):
        oracle.kronmult_general(len(mm), mm, nn,
                                [A.ctypes.data + 8 * o for o in ao[6 * k:6 * k + len(mm)]], mm,
                                [X.ctypes.data + 8 * xo[k]], [Yref.ctypes.data + 8 * yo[k]])
    plan = kb.VPlan(np.stack([_row(*e) for e in entries]))
    dA, dX, dY = dev(A), dev(X), dev(Y0)
    W = torch.empty(plan.workspace_bytes // 8, dtype=torch.float64, device="cuda")
    plan.execute(ptrs(dA, ao), ptrs(dX, xo), ptrs(dY, yo), W)
    assert rel_err(host(dY), Yref) <= 1e-13
    assert kb.lib().kron_device_status(1) == 0
    plan.close()
