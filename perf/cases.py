"""The work that programs have the library do, as cases that can be timed.

A case names a layout, its sizes and its options.  The sizes are those of the
benchmark workloads (bench.py) and of the reference tests' sweeps and timing
loops, with generic odd and ragged ones between them.  Factors and vectors are
what a PDE code passes: x ~ U(-1, 1), A ~ N(0, 1)/sqrt(n) (kgemm: U(-1, 1)).

Precisions: FP64, the drop-in's, and FP32.  The hi+lo split form is slower
than FP64 on this GPU and less exact, so programs call the FP64 form instead
and no case times it.
"""
import math

import numpy as np
import torch

import kronmult_b200 as kb

UNEVEN_SIZES = "2,3,4,6,8"


def listed():
    return [
        # the smallest call: a handful of 64-element vectors, where the time
        # is that of one launch (the reference tests' sweep)
        dict(name="batched_d3_n4_b16", kind="batched", d=3, n=4, batch=16, dtype="f64"),
        # a mid-size call that fits the L2 cache
        dict(name="batched_d6_n4_b512", kind="batched", d=6, n=4, batch=512, dtype="f64"),
        # the reference tests' timing loop at an odd size, vectors beyond one
        # block's shared memory
        dict(name="batched_d6_n7_b256", kind="batched", d=6, n=7, batch=256, dtype="f64"),
        # the headline: one operator application over a large batch
        dict(name="batched_d6_n6_b4096", kind="batched", d=6, n=6, batch=4096, dtype="f64"),
        # the same in single precision
        dict(name="batched_d6_n6_b4096_f32", kind="batched", d=6, n=6, batch=4096, dtype="f32"),
        # an element grid with overlapping outputs, factors from a pool
        dict(name="xbatched_d3_n8_grid", kind="xbatched", d=3, n=8, lda=8, elements=8192,
             couplings=16, pool=64, segmented=False),
        # the same with bitwise reproducible sums
        dict(name="xbatched_d3_n8_segmented", kind="xbatched", d=3, n=8, lda=8, elements=8192,
             couplings=16, pool=64, segmented=True),
        # a grid of low-order elements: short odd vectors, factors inside
        # larger matrices (lda = n + 3, as the reference tests pass them)
        dict(name="xbatched_d4_n3_grid", kind="xbatched", d=4, n=3, lda=6, elements=4096,
             couplings=9, pool=64, segmented=False),
        # large vectors with outputs drawn at random, so that some alias
        dict(name="xbatched_d6_n8_b1024", kind="xdrawn", d=6, n=8, lda=8, batch=1024, outputs=716,
             pool=32),
        # rectangular factors, one shape for the batch (restriction or
        # prolongation between orders)
        dict(name="vbatched_d4_b4096", kind="vbatched", m="4,6,3,8", n="6,3,8,4", batch=4096),
        # every entry with its own number of modes and shapes, one plan
        dict(name="uneven_20000", kind="uneven", entries=20000, sizes=UNEVEN_SIZES, dmax=6,
             shape_seed=5),
        # batched small GEMMs at the largest size of the reference tests
        dict(name="kgemm_nn_64_b32768", kind="kgemm", op="nn", mm=64, nn=64, kk=64, pad=0,
             beta=1.0, batch=32768),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(max(lo, hi))))))


def draw(rng):
    kind = rng.choice(["batched", "batched", "batched", "xbatched", "xbatched", "xdrawn",
                       "vbatched", "uneven", "kgemm", "kgemm"])
    if kind == "batched":
        d, n = rng.choice([1, 2, 3, 4, 5, 6, 6]), rng.randint(2, 8)
        # at most 1.5 GB of x and 13 GFLOP
        hi = min(100000, int(2e8 / n ** d), int(13e9 / (2 * d * n ** (d + 1))))
        return dict(kind=kind, d=d, n=n, batch=_log_int(rng, 1, hi),
                    dtype=rng.choice(["f64", "f64", "f32"]))
    if kind == "xbatched":
        d, n = rng.randint(2, 6), rng.randint(2, 8)
        while n ** d > 4096:
            d, n = rng.randint(2, 6), rng.randint(2, 8)
        couplings = rng.randint(2, 16)
        hi = min(8192, int(3.2e7 / (couplings * n ** d)))
        return dict(kind=kind, d=d, n=n, lda=n + rng.choice([0, 0, 1, 3]),
                    elements=_log_int(rng, 16, hi), couplings=couplings,
                    pool=rng.choice([16, 32, 64]), segmented=rng.random() < 0.3)
    if kind == "xdrawn":
        d, n = rng.choice([5, 6]), rng.randint(4, 8)
        hi = min(4096, int(9e7 / n ** d))
        batch = _log_int(rng, 32, hi)
        return dict(kind=kind, d=d, n=n, lda=n, batch=batch,
                    outputs=max(1, int(batch * rng.uniform(0.5, 1.0))), pool=32)
    if kind == "vbatched":
        d = rng.randint(2, 6)
        m, n = ([rng.choice([2, 3, 4, 5, 6, 7, 8]) for _ in range(d)] for _ in "mn")
        hi = min(50000, int(4e7 / max(math.prod(m), math.prod(n))))
        return dict(kind=kind, m=",".join(map(str, m)), n=",".join(map(str, n)),
                    batch=_log_int(rng, 16, hi))
    if kind == "uneven":
        return dict(kind=kind, entries=_log_int(rng, 200, 18000),
                    sizes=rng.choice([UNEVEN_SIZES, "2,3,4", "2,3,4,5,6,7,8"]),
                    dmax=rng.randint(3, 6), shape_seed=rng.randrange(1 << 20))
    mm, nn, kk = (rng.randint(1, 64) for _ in range(3))
    hi = min(60000, int(2e8 / (mm * kk + kk * nn + mm * nn)))
    return dict(kind="kgemm", op=rng.choice(["nn", "nt", "tt"]), mm=mm, nn=nn, kk=kk,
                pad=rng.choice([0, 0, 1, 3]), beta=rng.choice([1.0, 0.0, 0.5]),
                batch=_log_int(rng, 15, hi))


# ---------------------------------------------------------------- inputs
def _dtype(case):
    return torch.float32 if case.get("dtype") == "f32" else torch.float64


def _ints(text):
    return [int(v) for v in text.split(",")]


def _pointers(t, offsets):
    return t.data_ptr() + t.element_size() * offsets.to(t.device)


def _shapes(case):
    """Uneven batch: per entry (d, m1, n1, ..., m6, n6), and the offsets of
    its factors, x and y in flat arrays."""
    rng = np.random.default_rng(case["shape_seed"])
    e, sizes = case["entries"], np.array(_ints(case["sizes"]))
    d = rng.integers(1, case["dmax"] + 1, size=e)
    m, n = (rng.choice(sizes, size=(e, 6)) for _ in "mn")
    used = np.arange(6)[None, :] < d[:, None]
    m1, n1 = np.where(used, m, 1), np.where(used, n, 1)
    asz = np.where(used, m * n, 0).reshape(-1)
    shapes = np.zeros((e, 13), dtype=np.int32)
    shapes[:, 0] = d
    shapes[:, 1::2] = np.where(used, m, 0)
    shapes[:, 2::2] = np.where(used, n, 0)
    total = lambda v: int(v.sum())  # noqa: E731
    start = lambda v: np.cumsum(v) - v  # noqa: E731
    nx, ny = n1.prod(1), m1.prod(1)
    return dict(shapes=shapes, a_off=start(asz), x_off=start(nx), y_off=start(ny), na=total(asz),
                nx=total(nx), ny=total(ny))


def _lists(case, g):
    """xbatched index lists: which x, y and pool matrices entry k takes."""
    d, dev = case["d"], g.device
    if case["kind"] == "xdrawn":
        b, cols = case["batch"], case["outputs"]
        xl = torch.arange(b, device=dev)
        yl = torch.randint(cols, (b,), generator=g, device=dev)
        nx = b
    else:
        cols, c = case["elements"], case["couplings"]
        b = cols * c
        el = torch.arange(cols, device=dev)
        nb = torch.randint(1, max(2, cols), (cols, c), generator=g, device=dev)
        nb[:, 0] = 0  # every element couples to itself first
        xl = ((el[:, None] + nb) % cols).reshape(-1)
        yl = el.repeat_interleave(c)
        nx = cols
    al = torch.randint(case["pool"], (b, d), generator=g, device=dev)
    al = al + case["pool"] * torch.arange(d, device=dev)
    return b, nx, cols, xl, yl, al


def _kgemm_dims(case):
    op, mm, nn, kk, pad = (case[k] for k in ("op", "mm", "nn", "kk", "pad"))
    ra, ca = (kk, mm) if op == "tt" else (mm, kk)
    rb, cb = (kk, nn) if op == "nn" else (nn, kk)
    return (ra + pad, ca), (rb + pad, cb), (mm + pad, nn)


def _inputs(case, seed):
    """Every random input of the case, on the GPU."""
    dev = torch.device("cuda")
    g = torch.Generator(device=dev)
    g.manual_seed(seed)
    dt = _dtype(case)
    uniform = lambda k: torch.rand(k, dtype=dt, device=dev, generator=g) * 2 - 1  # noqa: E731
    normal = lambda k: torch.randn(k, dtype=dt, device=dev, generator=g)  # noqa: E731
    kind = case["kind"]
    if kind == "batched":
        d, n, b = case["d"], case["n"], case["batch"]
        return dict(A=normal(b * d * n * n) / math.sqrt(n), X=uniform(b * n ** d),
                    Y=uniform(b * n ** d))
    if kind in ("xbatched", "xdrawn"):
        d, n, lda = case["d"], case["n"], case["lda"]
        b, nx, ny, xl, yl, al = _lists(case, g)
        return dict(A=normal(d * case["pool"] * n * lda) / math.sqrt(n), X=uniform(nx * n ** d),
                    Y=uniform(ny * n ** d), xl=xl, yl=yl, al=al)
    if kind == "vbatched":
        m, n, b = _ints(case["m"]), _ints(case["n"]), case["batch"]
        asz = sum(p * q for p, q in zip(m, n))
        return dict(A=normal(b * asz) / 2, X=uniform(b * math.prod(n)),
                    Y=uniform(b * math.prod(m)))
    if kind == "uneven":
        s = _shapes(case)
        return dict(A=uniform(s["na"]), X=uniform(s["nx"]), Y=uniform(s["ny"]), s=s)
    (la, ca), (lb, cb), (lc, cc) = _kgemm_dims(case)
    b = case["batch"]
    return dict(A=uniform(b * la * ca), B=uniform(b * lb * cb), C=uniform(b * lc * cc))


def prepare(case, seed):
    v = _inputs(case, seed)
    v["case"] = case
    dev, kind = torch.device("cuda"), case["kind"]
    v["W"] = None
    if kind == "batched":
        need = kb.lib().kron_batched_workspace_bytes(case["d"], case["n"], case["batch"])
        if need:
            v["W"] = torch.empty(need // 8, dtype=_dtype(case), device=dev)
    elif kind in ("xbatched", "xdrawn"):
        d, n, lda = case["d"], case["n"], case["lda"]
        L = n ** d
        v["pA"] = _pointers(v["A"], (v["al"] * (n * lda)).reshape(-1))
        v["pX"], v["pY"] = _pointers(v["X"], L * v["xl"]), _pointers(v["Y"], L * v["yl"])
        v["pW"], v["sub"] = None, 0
        if kb.lib().kron_batched_workspace_bytes(d, n, 1):
            # 2 subbatchCount workspace vectors, as the layout wants them
            slots = min(128, 2 * (v["pX"].numel() // 2))
            v["W"] = torch.empty(L * slots, dtype=torch.float64, device=dev)
            v["pW"] = _pointers(v["W"], L * torch.arange(slots))
            v["sub"] = slots // 2
        v["seg"] = kb.Segments(v["pY"]) if case.get("segmented") else None
    elif kind == "vbatched":
        m, n, b = _ints(case["m"]), _ints(case["n"]), case["batch"]
        sizes = np.array([p * q for p, q in zip(m, n)])
        off = (np.cumsum(sizes) - sizes)[None, :] + sizes.sum() * np.arange(b)[:, None]
        v["m"], v["n"] = m, n
        v["pA"] = _pointers(v["A"], torch.from_numpy(off.reshape(-1)))
        v["pX"] = _pointers(v["X"], math.prod(n) * torch.arange(b))
        v["pY"] = _pointers(v["Y"], math.prod(m) * torch.arange(b))
        cm, cn = (np.array(t, dtype=np.int32) for t in (m, n))
        need = kb.lib().kron_vbatched_workspace_bytes(len(m), cm.ctypes.data, cn.ctypes.data, b)
        if need:
            v["W"] = torch.empty(need // 8, dtype=torch.float64, device=dev)
    elif kind == "uneven":
        s = v["s"]
        v["plan"] = kb.VPlan(s["shapes"])
        for p, t, off in (("pA", "A", "a_off"), ("pX", "X", "x_off"), ("pY", "Y", "y_off")):
            v[p] = _pointers(v[t], torch.from_numpy(s[off]))
        need = v["plan"].workspace_bytes
        if need:
            v["W"] = torch.empty(need // 8, dtype=torch.float64, device=dev)
    else:
        b = case["batch"]
        for t, (ld, cols) in zip("ABC", _kgemm_dims(case)):
            v["p" + t] = _pointers(v[t], ld * cols * torch.arange(b))
            v["ld" + t] = torch.full((b,), ld, dtype=torch.int32, device=dev)
    return v


def run(v):
    case = v["case"]
    kind = case["kind"]
    if kind == "batched":
        f = kb.kronmult_batched_f32 if case["dtype"] == "f32" else kb.kronmult_batched
        f(case["d"], case["n"], v["A"], v["X"], v["Y"], v["W"])
    elif kind in ("xbatched", "xdrawn"):
        if v["seg"] is not None:
            kb.kronmult_xbatched_segmented(case["d"], case["n"], v["pA"], case["lda"], v["pX"],
                                           v["pY"], v["seg"], v["pW"])
        else:
            kb.kronmult_xbatched(case["d"], case["n"], v["pA"], case["lda"], v["pX"], v["pY"],
                                 v["pW"], subbatch=v["sub"])
    elif kind == "vbatched":
        kb.kronmult_vbatched(v["m"], v["n"], v["pA"], v["pX"], v["pY"], v["W"])
    elif kind == "uneven":
        v["plan"].execute(v["pA"], v["pX"], v["pY"], v["W"])
    else:
        kb.kgemm_batched(case["op"], case["mm"], case["nn"], case["kk"], 1.0, v["pA"], v["ldA"],
                         v["pB"], v["ldB"], case["beta"], v["pC"], v["ldC"])
        return v["C"]
    return v["Y"]


# ---------------------------------------------------------------- bounds
def _kron_flops(m, n):
    """Fewest flops of the mode products, first mode first or last first."""
    best = math.inf
    for order in (range(len(m)), range(len(m) - 1, -1, -1)):
        dims, total = list(n), 0
        for l in order:
            total += 2 * m[l] * math.prod(dims)
            dims[l] = m[l]
        best = min(best, total)
    return best


def work(case):
    kind = case["kind"]
    if kind == "batched":
        d, n, b = case["d"], case["n"], case["batch"]
        es = 4 if case["dtype"] == "f32" else 8
        return dict(bytes=es * b * (3 * n ** d + d * n * n), flops=b * 2 * d * n ** (d + 1))
    if kind in ("xbatched", "xdrawn"):
        d, n = case["d"], case["n"]
        L = n ** d
        if kind == "xdrawn":
            b, nx = case["batch"], case["batch"]
            ny = case["outputs"] * (1 - (1 - 1 / case["outputs"]) ** b)  # distinct, expected
        else:
            b, nx = case["elements"] * case["couplings"], case["elements"]
            ny = nx
        pool = d * case["pool"] * n * n
        return dict(bytes=8 * (L * nx + 2 * L * ny + pool + b * (d + 2)),
                    flops=b * 2 * d * n ** (d + 1))
    if kind == "vbatched":
        m, n, b = _ints(case["m"]), _ints(case["n"]), case["batch"]
        per = math.prod(n) + 2 * math.prod(m) + sum(p * q for p, q in zip(m, n)) + len(m) + 2
        return dict(bytes=8 * b * per, flops=b * _kron_flops(m, n))
    if kind == "uneven":
        s = _shapes(case)
        flops = 0
        for r in s["shapes"].tolist():
            flops += _kron_flops(r[1:1 + 2 * r[0]:2], r[2:2 + 2 * r[0]:2])
        return dict(bytes=8 * (s["nx"] + 2 * s["ny"] + s["na"] + 8 * case["entries"]),
                    flops=flops)
    mm, nn, kk, b = case["mm"], case["nn"], case["kk"], case["batch"]
    cs = 1 if case["beta"] == 0.0 else 2
    return dict(bytes=8 * b * (mm * kk + kk * nn + cs * mm * nn + 3), flops=2 * b * mm * nn * kk)


def _kron64(A, x, m, n):
    """A: per mode (batch, n_l, m_l) (column-major factors as rows); x:
    (batch, prod n), the last mode's index fastest."""
    b, d = x.shape[0], len(m)
    z = x.double()
    for l in range(d):
        outer = math.prod(m[:l])
        z = z.reshape(b, outer, n[l], -1)
        z = torch.einsum("bji,bojr->boir", A[l].double(), z)
    return z.reshape(b, -1)


def exact(case, seed):
    v = _inputs(case, seed)
    kind = case["kind"]
    if kind == "batched":
        d, n, b = case["d"], case["n"], case["batch"]
        L, step = n ** d, max(1, int(5e7) // n ** d)
        A, X, y = v["A"].view(b, d, n, n), v["X"].view(b, L), v["Y"].double().view(b, L)
        for k in range(0, b, step):
            a = A[k:k + step]
            y[k:k + step] += _kron64([a[:, l] for l in range(d)], X[k:k + step], [n] * d, [n] * d)
        return y.view(-1)
    if kind in ("xbatched", "xdrawn"):
        d, n, lda = case["d"], case["n"], case["lda"]
        L = n ** d
        P, X, y = v["A"].view(-1, n, lda)[:, :, :n], v["X"].view(-1, L), v["Y"].view(-1, L).clone()
        b, step = v["xl"].numel(), max(1, int(5e7) // L)
        for k in range(0, b, step):
            s = slice(k, min(b, k + step))
            y.index_add_(0, v["yl"][s], _kron64([P[v["al"][s, l]] for l in range(d)],
                                                X[v["xl"][s]], [n] * d, [n] * d))
        return y.view(-1)
    if kind == "vbatched":
        m, n, b = _ints(case["m"]), _ints(case["n"]), case["batch"]
        A = v["A"].view(b, -1)
        split = torch.split(A, [p * q for p, q in zip(m, n)], dim=1)
        F = [a.reshape(b, q, p) for a, p, q in zip(split, m, n)]
        return v["Y"] + _kron64(F, v["X"].view(b, -1), m, n).reshape(-1)
    if kind == "uneven":
        s = v["s"]
        A, X, y = (v[t].cpu().numpy() for t in "AXY")
        for k, r in enumerate(s["shapes"].tolist()):
            d = r[0]
            m, n = r[1:1 + 2 * d:2], r[2:2 + 2 * d:2]
            z = X[s["x_off"][k]:s["x_off"][k] + math.prod(n)].reshape(1, -1)
            for l in range(d):
                o = s["a_off"][6 * k + l]
                a = A[o:o + m[l] * n[l]].reshape(n[l], m[l])
                # the mode that goes first is contracted and comes out last
                z = z.reshape(n[l], -1).T @ a
            y[s["y_off"][k]:s["y_off"][k] + math.prod(m)] += z.reshape(-1)
        return y
    b, op = case["batch"], case["op"]
    (la, ca), (lb, cb), (lc, cc) = _kgemm_dims(case)
    mm, nn, kk = case["mm"], case["nn"], case["kk"]
    A, B = v["A"].view(b, ca, la), v["B"].view(b, cb, lb)  # column major: [column, row]
    A = A[:, :, :kk] if op == "tt" else A[:, :, :mm].transpose(1, 2)
    B = B[:, :, :kk].transpose(1, 2) if op == "nn" else B[:, :, :nn]
    C = v["C"].view(b, cc, lc)
    C[:, :, :mm] = case["beta"] * C[:, :, :mm] + torch.bmm(A, B).transpose(1, 2)
    return v["C"]
