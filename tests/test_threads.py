"""Contexts in several threads at once, each with its own mesh: passes, updates,
stream switches and calls that move buffers; every pass gives a fresh context's
sizes and flags."""
import threading
import time

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SECONDS = 3.0


def test_contexts_in_threads(gpu_lib):
    import torch
    import core_gb300 as cg
    from core_gb300 import workload
    meshes = [workload.box(n, jitter=0.2, seed=n) for n in (9, 14, 23)]
    us = [workload.bump_field(m.coords, seed=1) for m in meshes]
    want = {}
    for p in ("fp32", "fp64", "learned"):
        for i, m in enumerate(meshes):
            with cg.Context(m, precision=p) as c:
                want[p, i] = c.estimate_and_mark(us[i], 0.1)[:2]
    wrong, passes, failed = [], [], []

    def work(p, seed):
        rng = np.random.default_rng(seed)
        streams = [torch.cuda.Stream() for _ in range(2)]
        i, end = int(rng.integers(3)), time.time() + SECONDS
        try:
            with cg.Context(meshes[i], precision=p) as c:
                while time.time() < end:
                    what = int(rng.integers(6))
                    if what == 0:
                        c.set_stream(streams[int(rng.integers(2))].cuda_stream)
                    elif what == 1:
                        i = int(rng.integers(3))
                        c.update_mesh(meshes[i])
                    elif what == 2:
                        c.recoverField(c.getGradIPField(np.stack([us[i]] * 3, 1)))
                    elif what == 3:
                        c.set_stream(0)
                    got = c.estimate_and_mark(us[i], 0.1)[:2]
                    passes.append(p)
                    if not (np.array_equal(got[0], want[p, i][0]) and np.array_equal(got[1], want[p, i][1])):
                        wrong.append((p, i, what))
                c.set_stream(0)
        except Exception as e:  # a thread's own failure fails the test
            failed.append(repr(e))
    threads = [threading.Thread(target=work, args=(p, k)) for k, p in enumerate(("fp32", "fp64", "learned") * 2)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not failed and not wrong and set(passes) == {"fp32", "fp64", "learned"}


def test_update_while_another_thread_captures(gpu_lib):
    """After a stream switch an update waits for the whole device; a capture under
    way in another thread neither refuses that nor is broken by it."""
    import torch
    import core_gb300 as cg
    from core_gb300 import workload
    a, b = (workload.box(n, jitter=0.2, seed=n) for n in (6, 8))
    u = [workload.bump_field(m.coords, seed=1) for m in (a, b)]
    with cg.Context(b) as c:
        want = c.estimate_and_mark(u[1], 0.1)[:2]
    x = torch.zeros(1024, device="cuda")
    captured, updated = threading.Event(), threading.Event()
    result = {}

    def capture():
        s, g = torch.cuda.Stream(), torch.cuda.CUDAGraph()
        with torch.cuda.stream(s):
            g.capture_begin(capture_error_mode="thread_local")
            x.add_(1)
            captured.set()
            updated.wait(60)
            g.capture_end()
            g.replay()
        s.synchronize()
        result["x"] = float(x[0])
    with cg.Context(a) as c:
        stream = torch.cuda.Stream()
        c.estimate_and_mark(u[0], 0.1)
        c.set_stream(stream.cuda_stream)
        c.estimate_and_mark(u[0], 0.1)
        t = threading.Thread(target=capture)
        t.start()
        assert captured.wait(60)
        try:
            c.update_mesh(b)
            got = c.estimate_and_mark(u[1], 0.1)[:2]
        finally:
            updated.set()
            t.join()
        c.set_stream(0)
    assert np.array_equal(got[0], want[0]) and np.array_equal(got[1], want[1])
    assert result["x"] == 1.0
