"""The kernel that a committed DRAM-traffic line names is the one that the
built-in order runs for that workload: on the GPU each workload's call, smaller
but on the same side of every dispatch rule, is traced and its longest kernel
compared with the line."""
import argparse
import glob
import math
import os
import re

import numpy as np
import pytest

import bench
import kronmult_b200 as kb

KEYS = ["cfg1", "cfg2", "cfg3", "cfg3-f32", "cfg3-split", "cfg3-n6", "cfg3-f32-n6", "cfg4", "cfg5",
        "cfg6"]


@pytest.mark.parametrize("key", KEYS)
def test_line_names_a_kernel_of_the_library(key):
    traffic, kernel, src = bench.read_profile_line(key)
    assert traffic > 0 and os.path.exists(os.path.join(bench.ROOT, src))
    text = "".join(open(f).read() for f in glob.glob(os.path.join(bench.ROOT, "kronmult_b200",
                                                                  "csrc", "*.cu*")))
    assert re.search(rf"\b{kernel}\s*\(\s*(const __grid_constant__|int )", text), kernel


def test_one_line_a_workload():
    text = "".join(open(f).read() for f in glob.glob(os.path.join(bench.ROOT, "profiles", "*.md")))
    keys = re.findall(r"^traffic_bytes_per_launch\[([^\]]+)\]", text, flags=re.M)
    assert sorted(keys) == sorted(KEYS)


def test_unknown_key_reads_as_none():
    assert bench.read_profile_line("cfg9") == (None, None, None)
    assert bench.profile_key(argparse.Namespace(config=3, precision="f32", mode="atomic",
                                                entries=0, n=6)) == "cfg3-f32-n6"


def _call(key):
    import torch

    u = lambda k, dt=torch.float64: torch.rand(k, dtype=dt, device="cuda")  # noqa: E731
    at = lambda t, o: t.data_ptr() + t.element_size() * o.to(t.device)  # noqa: E731
    if key in ("cfg2", "cfg5"):
        d, n, b, cols = (3, 8, 20000, 1250) if key == "cfg2" else (6, 8, 24, 17)
        L, nw = n ** d, 8
        A, X, Y, W = u(d * 16 * n * n), u(b * L), u(cols * L), u(nw * L)
        pA = at(A, n * n * torch.randint(16 * d, (b * d,)))
        pX, pY = at(X, L * torch.arange(b)), at(Y, L * (torch.arange(b) * cols // b))
        pW = at(W, L * torch.arange(nw))
        return lambda: kb.kronmult_xbatched(d, n, pA, n, pX, pY, pW, subbatch=nw // 2), (A, X, Y, W)
    if key == "cfg4":
        rng = np.random.default_rng(5)
        sh = np.zeros((400, 13), dtype=np.int32)
        sh[:, 0] = rng.integers(1, 7, 400)
        sh[:, 1:] = rng.choice([2, 3, 4, 6, 8], (400, 12))
        a, x, y, na, nx, ny = [], [], [], 0, 0, 0
        for s in sh:
            s[1 + 2 * s[0]:] = 0
            m, n = [int(v) for v in s[1:1 + 2 * s[0]:2]], [int(v) for v in s[2:2 + 2 * s[0]:2]]
            for l in range(6):
                a.append(na)
                na += m[l] * n[l] if l < len(m) else 0
            x.append(nx)
            y.append(ny)
            nx, ny = nx + math.prod(n), ny + math.prod(m)
        plan = kb.VPlan(sh)
        A, X, Y, W = u(na), u(nx), u(ny), u(plan.workspace_bytes // 8)
        pA, pX, pY = (at(t, torch.tensor(o)) for t, o in ((A, a), (X, x), (Y, y)))
        return lambda: plan.execute(pA, pX, pY, W), (A, X, Y, W, plan)
    if key == "cfg6":
        b = 2000
        A, B, Cc = u(b * 4096), u(b * 4096), u(b * 4096)
        p = [at(t, 4096 * torch.arange(b)) for t in (A, B, Cc)]
        ld = torch.full((b,), 64, dtype=torch.int32, device="cuda")
        return lambda: kb.kgemm_batched("nn", 64, 64, 64, 1.0, p[0], ld, p[1], ld, 1.0, p[2],
                                        ld), (A, B, Cc)
    n, b = (6, 220) if key.endswith("n6") else (4, 512)
    dt = torch.float32 if "f32" in key else torch.float64
    f = {"f32": kb.kronmult_batched_f32, "split": kb.kronmult_batched_split}
    f = next((v for k, v in f.items() if k in key), kb.kronmult_batched)
    A, X, Y, W = (u(b * s, dt) for s in (6 * n * n, n ** 6, n ** 6, n ** 6))
    return lambda: f(6, n, A, X, Y, W), ()


@pytest.mark.gpu
@pytest.mark.parametrize("key", KEYS)
def test_line_names_the_kernel_that_runs(gpu_lib, key):
    import torch
    from torch.profiler import ProfilerActivity, profile

    kb.tune_clear()
    call, keep = _call(key)
    call()
    torch.cuda.synchronize()
    with profile(activities=[ProfilerActivity.CUDA, ProfilerActivity.CPU]) as prof:
        call()
        torch.cuda.synchronize()
    times = {}
    for e in prof.events():
        if str(e.device_type).endswith("CUDA"):
            times[e.name] = times.get(e.name, 0) + e.device_time_total
    if not times:
        pytest.skip("no kernel records from the profiler on this machine")
    longest = max(times, key=times.get)
    kernel = bench.read_profile_line(key)[1]
    assert re.search(rf"\b{kernel}\b", longest), (kernel, times)
    del keep
