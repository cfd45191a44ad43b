"""Where a resident pass's field may lie."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", ["fp32", "fp64", "learned"])
@pytest.mark.parametrize("offset", [0, 4, 8, 9])
@pytest.mark.parametrize("graph", [False, True])
def test_field_at_any_address(gpu_lib, precision, offset, graph):
    """A field inside a larger buffer, at an address that is no multiple of a
    double's size too: copied before the pass reads it."""
    import torch
    import core_gb300 as cg
    from core_gb300 import workload
    m = workload.box(7, jitter=0.2, seed=2)
    us = [workload.bump_field(m.coords, seed=s) for s in (1, 2)]
    stream = torch.cuda.Stream()
    with cg.Context(m, precision=precision) as c, torch.cuda.stream(stream):
        want = [c.estimate_and_mark(u, 0.1)[1] for u in us]
        c.set_stream(stream.cuda_stream)
        raw = torch.zeros(8 * m.n_verts + 16, dtype=torch.uint8, device="cuda")
        field = raw[offset:offset + 8 * m.n_verts]
        bits = torch.zeros((2, (m.n_edges + 31) // 32), dtype=torch.int32, device="cuda")
        args = (field.data_ptr(), 0.1, bits[0].data_ptr(), bits[1].data_ptr())
        e = np.arange(m.n_edges)
        for k, (u, flags) in enumerate(zip(us, want)):
            field.copy_(torch.from_numpy(u.view(np.uint8)))
            if graph and k == 0:
                c.graph_capture(*args)
            if graph:
                bits.zero_()
                c.graph_replay()
            else:
                c.estimate_and_mark_resident(*args)
            stream.synchronize()
            b = bits.cpu().numpy().view(np.uint32)
            assert np.array_equal((b[0][e >> 5] >> (e & 31)) & 1, flags & 1)
            assert np.array_equal((b[1][e >> 5] >> (e & 31)) & 1, (flags >> 2) & 1)
        c.set_stream(0)


@pytest.mark.parametrize("precision", ["fp32", "fp64"])
@pytest.mark.parametrize("offset", [0, 4, 8])
def test_anisotropic_field_at_any_address(gpu_lib, precision, offset):
    import torch
    import core_gb300 as cg
    from core_gb300 import workload
    m, u, (eps, hmin, hmax) = workload.aniso2d(24)
    out = []
    for at in (0, offset):
        raw = torch.zeros(8 * m.n_verts + 16, dtype=torch.uint8, device="cuda")
        field = raw[at:at + 8 * m.n_verts]
        field.copy_(torch.from_numpy(u.view(np.uint8)))
        bits = torch.zeros((2, (m.n_edges + 31) // 32), dtype=torch.int32, device="cuda")
        q = torch.zeros(m.n_elems, dtype=torch.float64, device="cuda")
        torch.cuda.synchronize()
        with cg.Context(m, precision=precision) as c:
            c.aniso_estimate_and_mark_resident(field.data_ptr(), eps, hmin, hmax, bits[0].data_ptr(), bits[1].data_ptr(),
                                               q.data_ptr())
            torch.cuda.synchronize()
        out.append((bits.cpu().numpy(), q.cpu().numpy()))
    assert out[0][0].any() and np.array_equal(out[0][0], out[1][0]) and np.array_equal(out[0][1], out[1][1])
