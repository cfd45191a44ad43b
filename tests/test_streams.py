"""A context that moves between streams: the work left on one of them is
ordered before what follows on the next."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", ["fp32", "fp64", "learned"])
def test_update_then_another_stream(gpu_lib, precision):
    """Pass, update and pass with a stream switch between any two of them and no
    wait: the pass before an update sees the old mesh, the one after it the new
    one with its whole adjacency."""
    import torch
    import core_gb300 as cg
    from core_gb300 import workload
    meshes = [workload.box(n, jitter=0.2, seed=s) for n, s in ((30, 1), (34, 2), (28, 3), (34, 4))]
    us = [workload.sine_field(m.coords) for m in meshes]
    want = []
    for m, u in zip(meshes, us):
        with cg.Context(m, precision=precision) as c:
            want.append(c.estimate_and_mark(u, 0.05)[1])
    streams = [torch.cuda.Stream() for _ in range(3)]
    d_us = [torch.from_numpy(u).cuda() for u in us]
    bits = [torch.zeros((2, (m.n_edges + 31) // 32), dtype=torch.int32, device="cuda") for m in meshes]
    torch.cuda.synchronize()
    with cg.Context(meshes[0], precision=precision) as c:
        for i, m in enumerate(meshes):
            if i:
                c.set_stream(streams[(2 * i) % 3].cuda_stream)
                c.update_mesh(m)
            c.set_stream(streams[(2 * i + 1) % 3].cuda_stream)
            c.estimate_and_mark_resident(d_us[i].data_ptr(), 0.05, bits[i][0].data_ptr(), bits[i][1].data_ptr())
        torch.cuda.synchronize()
        c.set_stream(0)
    for m, b, flags in zip(meshes, bits, want):
        e = np.arange(m.n_edges)
        b = b.cpu().numpy().view(np.uint32)
        assert np.array_equal((b[0][e >> 5] >> (e & 31)) & 1, flags & 1)
        assert np.array_equal((b[1][e >> 5] >> (e & 31)) & 1, (flags >> 2) & 1)
