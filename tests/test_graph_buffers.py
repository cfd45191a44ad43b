"""Captured passes and the buffers they hold: a call that makes one of the
context's buffers move lies between two replays, and the next replay still gives
a fresh context's marks."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

RATIO = 0.1


def box(n=9, seed=1):
    from core_gb300 import workload
    m = workload.box(n, jitter=0.2, seed=seed)
    return m, [workload.bump_field(m.coords, seed=s) for s in (1, 2, 3)]


def fresh(m, u, precision="fp64"):
    import core_gb300 as cg
    with cg.Context(m, precision=precision) as c:
        return c.estimate_and_mark(u, RATIO)[:4]


def same(a, b):
    return np.array_equal(a[0], b[0]) and np.array_equal(a[1], b[1]) and a[2:] == b[2:]


def vector_calls(c, m):
    """ip, rec and the slab grow from 3 to 9 components, f threefold."""
    v = np.stack([np.sin(3 * m.coords[:, k]) for k in range(3)], 1)
    return c.recoverField(c.getGradIPField(v))


@pytest.mark.parametrize("precision", ["fp64", "fp32", "learned"])
def test_host_passes_around_a_vector_recovery(gpu_lib, precision):
    import core_gb300 as cg
    m, us = box()
    with cg.Context(m, precision=precision) as c:
        for u in (us[0], us[1], us[0], us[2]):  # captured on the third
            got = c.estimate_and_mark(u, RATIO)[:4]
        assert same(got, fresh(m, us[2], precision))
        vec = vector_calls(c, m)
        for u in us + us:
            assert same(c.estimate_and_mark(u, RATIO)[:4], fresh(m, u, precision))
        assert np.array_equal(vector_calls(c, m), vec)


@pytest.mark.parametrize("precision", ["fp64", "fp32", "learned"])
@pytest.mark.parametrize("moved_by", ["vector", "pairs", "aniso"])
def test_user_graph_around_a_call_that_moves_buffers(gpu_lib, precision, moved_by):
    """Also with the context's settings changed between: the replay is the pass
    that was captured."""
    import torch
    import core_gb300 as cg
    m, us = box()
    nw = (m.n_edges + 31) // 32
    e = np.arange(m.n_edges)
    stream = torch.cuda.Stream()
    with cg.Context(m, precision=precision) as c, torch.cuda.stream(stream):
        c.set_stream(stream.cuda_stream)
        d_u = torch.from_numpy(us[0]).cuda()
        bits = torch.zeros((2, nw), dtype=torch.int32, device="cuda")
        c.graph_capture(d_u.data_ptr(), RATIO, bits[0].data_ptr(), bits[1].data_ptr())
        if moved_by == "vector":
            vector_calls(c, m)
        elif moved_by == "pairs":
            for k in (1, 40):
                c.measure_vertex_pairs(np.tile(m.edge_verts, (k, 1)), size=np.full(m.n_verts, 0.1))
        else:
            c.set_precision("fp64")
            other = torch.zeros((2, nw), dtype=torch.int32, device="cuda")
            c.aniso_estimate_and_mark_resident(d_u.data_ptr(), 0.1, 0.01, 1.0, other[0].data_ptr(),
                                               other[1].data_ptr())
        for u in us + us:
            d_u.copy_(torch.from_numpy(u))
            bits.zero_()
            c.graph_replay()
            stream.synchronize()
            b = bits.cpu().numpy().view(np.uint32)
            flags = fresh(m, u, precision)[1]
            assert np.array_equal((b[0][e >> 5] >> (e & 31)) & 1, flags & 1)
            assert np.array_equal((b[1][e >> 5] >> (e & 31)) & 1, (flags >> 2) & 1)
        # on the context's own stream, which is not captured
        vector_calls(c, m)
        c.set_stream(0)
        c.graph_replay()
        c.getGradIPField(us[0])  # waits
        assert np.array_equal(bits.cpu().numpy().view(np.uint32), b)


@pytest.mark.parametrize("user_graph", [False, True])
def test_resident_gradients_after_a_replay(gpu_lib, user_graph):
    """The resident integration-point field after a replayed pass is the pass's
    (3 components), as after a direct one."""
    import torch
    import core_gb300 as cg
    from core_gb300 import _lib
    m, us = box(5)
    v = np.stack([np.sin(3 * m.coords[:, k]) for k in range(3)], 1)
    stream = torch.cuda.Stream()
    with cg.Context(m) as c:
        c.recoverField(c.getGradIPField(v))
        want = c.recoverField(c.getGradIPField(us[0]))
        if user_graph:
            c.set_stream(stream.cuda_stream)
            d_u = torch.from_numpy(us[0]).cuda()
            bits = torch.zeros((2, (m.n_edges + 31) // 32), dtype=torch.int32, device="cuda")
            torch.cuda.synchronize()
            c.graph_capture(d_u.data_ptr(), RATIO, bits[0].data_ptr(), bits[1].data_ptr())
        else:
            for _ in range(4):
                c.estimate_and_mark(us[0], RATIO)
        c.getGradIPField(v)
        if user_graph:
            c.graph_replay()
        else:
            c.estimate_and_mark(us[0], RATIO)
        out = np.empty((m.n_verts, 9))
        assert gpu_lib.sprg_recover_field(c.h, None, 9, out.ctypes.data) == _lib.SPRG_EINVAL
        out = np.empty((m.n_verts, 3))
        assert gpu_lib.sprg_recover_field(c.h, None, 3, out.ctypes.data) == _lib.SPRG_OK
        assert np.array_equal(out, want)


def marks(bits, E):
    b, e = bits.cpu().numpy().view(np.uint32), np.arange(E)
    return np.stack([(b[k][e >> 5] >> (e & 31)) & 1 for k in range(2)])


@pytest.mark.parametrize("first,then", [(([0, 0, 0, 0], 64, 8), ([4, 1, 2, 1], 48, 4)),
                                        (([4, 4, 4, 4], 1024, 8), ([4, 4, 4, 4], 64, 8)),
                                        (([1, 1, 1, 1], 64, 4), ([0, 0, 0, 0], 1024, 8))])
def test_user_graph_after_a_tiling_change(gpu_lib, first, then):
    """The captured recovery holds the tile list's length and lane mode."""
    import torch
    import core_gb300 as cg
    m, us = box(14)
    stream = torch.cuda.Stream()
    with cg.Context(m, precision="fp32") as c, torch.cuda.stream(stream):
        c.set_stream(stream.cuda_stream)
        c.set_tiling(*first)
        d_u = torch.from_numpy(us[0]).cuda()
        bits = torch.zeros((2, (m.n_edges + 31) // 32), dtype=torch.int32, device="cuda")
        c.graph_capture(d_u.data_ptr(), RATIO, bits[0].data_ptr(), bits[1].data_ptr())
        c.graph_replay()
        c.set_tiling(*then)  # a replay may still be in flight
        for u in us:
            d_u.copy_(torch.from_numpy(u))
            c.graph_replay()
            stream.synchronize()
            flags = fresh(m, u, "fp32")[1]
            assert np.array_equal(marks(bits, m.n_edges), [flags & 1, (flags >> 2) & 1])
        c.set_stream(0)


def test_user_graph_follows_the_batch(gpu_lib):
    """Other ratios for the captured batch, then another partition of the same
    meshes into batches (two boxes each, then three), then the batch cleared:
    the replay is the pass of the batch that was set last."""
    import torch
    import core_gb300 as cg
    from core_gb300 import workload
    m, u, voff, eoff, doff, ns = workload.batch_boxes(12, seed=7, lo=4, hi=12)
    K = len(ns)
    sets = [(voff, eoff, np.full(K, 0.1)), (voff, eoff, np.linspace(0.05, 0.2, K)),
            (voff[::2], eoff[::2], np.full(K // 2, 0.1)), (voff[::3], eoff[::3], np.full(K // 3, 0.07)),
            (voff, eoff, np.full(K, 0.2))]
    want = []
    for s in sets:
        with cg.Context(m, precision="fp32") as c:
            c.set_batch(*s)
            flags = c.estimate_and_mark(u, 1.0)[1]
        want.append([flags & 1, (flags >> 2) & 1])
    assert not np.array_equal(want[0], want[2])
    stream = torch.cuda.Stream()
    with cg.Context(m, precision="fp32") as c, torch.cuda.stream(stream):
        c.set_stream(stream.cuda_stream)
        d_u = torch.from_numpy(u).cuda()
        bits = torch.zeros((2, (m.n_edges + 31) // 32), dtype=torch.int32, device="cuda")
        c.set_batch(*sets[0])
        c.graph_capture(d_u.data_ptr(), 1.0, bits[0].data_ptr(), bits[1].data_ptr())
        for s, w in zip(sets[1:], want[1:]):
            c.set_batch(*s)
            for _ in range(2):
                bits.zero_()
                c.graph_replay()
                stream.synchronize()
                assert np.array_equal(marks(bits, m.n_edges), w)
        c.set_batch([], [], [])
        bits.zero_()
        c.graph_replay()
        stream.synchronize()
        assert np.array_equal(marks(bits, m.n_edges), want[-1])
        c.set_stream(0)
