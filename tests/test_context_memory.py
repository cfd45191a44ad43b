"""Contexts short of device memory.  The failures are made on the host
(sprg_test_hooks): an attempt at device memory fails as cudaMalloc does, the
context gives back what it can spare and tries again."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def fail(c, after, count=1):
    """`count` attempts at device memory fail, after the next `after`."""
    c.test_hooks(alloc_fail_after=after | count << 24)


def box(n, seed=1):
    from core_gb300 import workload
    m = workload.box(n, jitter=0.2, seed=seed)
    return m, workload.sine_field(m.coords)


def fresh(m, u, precision):
    import core_gb300 as cg
    with cg.Context(m, precision=precision) as c:
        return c.estimate_and_mark(u, 0.1)[:4]


def same(a, b):
    return np.array_equal(a[0], b[0]) and np.array_equal(a[1], b[1]) and a[2:] == b[2:]


@pytest.mark.parametrize("precision", ["fp32", "fp64", "learned"])
def test_spare_arrays_given_back(gpu_lib, precision):
    """After an update to a larger mesh every buffer of the pass grows; whichever
    allocation fails, the spare mesh arrays go and the retry holds."""
    import core_gb300 as cg
    (m0, u0), (m1, u1) = box(5), box(12, 2)
    want = fresh(m1, u1, precision)
    for k in range(64):
        with cg.Context(m0, precision=precision) as c:
            c.estimate_and_mark(u0, 0.1)
            c.update_mesh(m1)
            fail(c, k)
            assert same(c.estimate_and_mark(u1, 0.1)[:4], want), k
            assert same(c.estimate_and_mark(u1, 0.1)[:4], want), k


def test_results_go_with_their_buffers(gpu_lib):
    """A scalar field's gradients are resident; the vector field's do not fit, and
    the smaller buffer is gone: no resident field any more, then a new one."""
    import core_gb300 as cg
    from core_gb300 import _lib
    m, u = box(4)
    v = np.stack([u, u * u, 1 - u], 1)
    out = np.empty((m.n_verts, 3))
    with cg.Context(m) as c:
        ip = c.getGradIPField(u)
        want = c.recoverField(ip)
        fail(c, 1, 9)  # f grows, then ip, whatever is given back for it
        with pytest.raises(cg.SprgError) as e:
            c.getGradIPField(v)
        assert e.value.code == _lib.SPRG_ENOMEM
        c.test_hooks()
        assert gpu_lib.sprg_recover_field(c.h, None, 3, out.ctypes.data) == _lib.SPRG_ESTATE
        assert np.array_equal(c.getGradIPField(u), ip)
        assert gpu_lib.sprg_recover_field(c.h, None, 3, out.ctypes.data) == _lib.SPRG_OK
        assert np.array_equal(out, want)


@pytest.mark.parametrize("precision", ["fp32", "learned"])
@pytest.mark.parametrize("csr", [False, True])
def test_update_fails_before_the_old_mesh_goes(gpu_lib, oracle_lib, precision, csr):
    """Whichever of an update's allocations fails, the scan of its offsets
    included, the context still holds the old mesh; the next update holds."""
    import core_gb300 as cg
    (m0, u0), (m1, u1) = box(5), box(7, 2)
    if csr:
        o = oracle_lib.OracleMesh.box(7, 7, 7)
        m1.v2e_off, m1.v2e = o.v2e_off, o.v2e
    want = [fresh(m, u, precision) for m, u in ((m0, u0), (m1, u1))]
    failed = 0
    for k in range(32):
        with cg.Context(m0, precision=precision) as c:
            c.estimate_and_mark(u0, 0.1)
            fail(c, k, 100)
            try:
                c.update_mesh(m1)
            except cg.SprgError as e:
                assert e.code == 4
                failed += 1
                c.test_hooks()
                assert same(c.estimate_and_mark(u0, 0.1)[:4], want[0]), k
                c.update_mesh(m1)
            c.test_hooks()
            assert same(c.estimate_and_mark(u1, 0.1)[:4], want[1]), k
    # three arrays, staging, the out-of-range count, the box keys, and what
    # derives from the arrays: fixed-point coordinates, offsets, elements,
    # counters, the scan (as large as the old mesh's here) and the caller's order
    assert failed >= (12 if csr else 10)


def square(n, seed=1):
    from core_gb300.mesh import makeMdsBox
    m = makeMdsBox(n, n, 0)
    rng = np.random.default_rng(seed)
    inner = np.all((m.coords[:, :2] > 0) & (m.coords[:, :2] < 1), axis=1)
    m.coords[inner, :2] += rng.uniform(-0.2, 0.2, (int(inner.sum()), 2)) / n
    return m


def test_records_given_back_on_tets(gpu_lib):
    """The element records are there; each later allocation that the pass must
    have fails once, the records go, and the pass has the same bits without."""
    import core_gb300 as cg
    m, u = box(6)
    want = fresh(m, u, "fp64")
    for k in range(32):
        with cg.Context(m) as c:
            ip = c.getGradIPField(u)
            fail(c, k)
            for _ in range(5):  # a captured pass among them
                assert same(c.estimate_and_mark(u, 0.1)[:4], want), k
            assert np.array_equal(c.getGradIPField(u), ip)
    for k in range(32):  # no memory at all: an error, and the context goes on
        with cg.Context(m) as c:
            c.getGradIPField(u)
            fail(c, k, 100)
            try:
                c.estimate_and_mark(u, 0.1)
            except cg.SprgError as e:
                assert e.code == 4
            c.test_hooks()
            assert same(c.estimate_and_mark(u, 0.1)[:4], want), k


def test_user_graph_without_the_records(gpu_lib):
    """A captured FP64 pass, then another call needs the records' memory."""
    import torch
    import core_gb300 as cg
    m, u = box(6)
    flags = fresh(m, u, "fp64")[1]
    stream = torch.cuda.Stream()
    with cg.Context(m) as c, torch.cuda.stream(stream):
        c.set_stream(stream.cuda_stream)
        d_u = torch.from_numpy(u).cuda()
        bits = torch.zeros((2, (m.n_edges + 31) // 32), dtype=torch.int32, device="cuda")
        c.graph_capture(d_u.data_ptr(), 0.1, bits[0].data_ptr(), bits[1].data_ptr())
        fail(c, 0)
        c.measureQuality(np.full(m.n_verts, 0.1))
        e = np.arange(m.n_edges)
        for _ in range(3):
            bits.zero_()
            c.graph_replay()
            stream.synchronize()
            b = bits.cpu().numpy().view(np.uint32)
            assert np.array_equal((b[0][e >> 5] >> (e & 31)) & 1, flags & 1)
            assert np.array_equal((b[1][e >> 5] >> (e & 31)) & 1, (flags >> 2) & 1)
        c.set_stream(0)


@pytest.mark.parametrize("n", [3, 16])
def test_factors_given_back_on_triangles(gpu_lib, n):
    """Any allocation of the recovery fails once: the factors' own, or one for
    which they go.  Ordinary patches keep their bits; the listed ones are weighted
    sums with the factors kept and QR fits without (1e-10, as the parity tests)."""
    import core_gb300 as cg
    m = square(n)
    rng = np.random.default_rng(3)
    ip = [rng.normal(size=(m.n_elems, nc)) for nc in (3, 9, 3)]
    cnt = np.bincount(m.elem_verts.reshape(-1), minlength=m.n_verts)
    with cg.Context(m) as c:
        want = [c.recoverField(a) for a in ip]
    for k in range(24):
        with cg.Context(m) as c:
            c.getGradIPField(np.sin(m.coords[:, 0]))  # the element records
            fail(c, k)
            for a, w in zip(ip, want):
                got = c.recoverField(a)
                assert np.array_equal(got[cnt >= 4], w[cnt >= 4]), k
                assert np.abs(got - w).max() <= 1e-10 * np.abs(w).max(), k


@pytest.mark.parametrize("n", [3, 16])
def test_refined_weights_without_memory(gpu_lib, n):
    """The FP64 anisotropic pass: whichever allocation fails once, its Hessian is
    the one of the refined weights or, without them, the calls' (the factors'
    bits); both occur."""
    import torch
    import core_gb300 as cg
    from core_gb300 import workload
    m = square(n)
    u = workload.boundary_layer_field(m.coords)
    with cg.Context(m) as c:
        calls = c.recoverField(c.getGradIPField(c.recoverField(c.getGradIPField(u))))
    d_u = torch.from_numpy(u).cuda()
    bits = torch.zeros((2, (m.n_edges + 31) // 32), dtype=torch.int32, device="cuda")
    torch.cuda.synchronize()

    def hessian(c):
        c.aniso_estimate_and_mark_resident(d_u.data_ptr(), 0.1, 0.1 / n, 1.0, bits[0].data_ptr(), bits[1].data_ptr())
        torch.cuda.synchronize()
        return c.debug_read("rec", np.float64, 9 * m.n_verts).reshape(-1, 9)
    with cg.Context(m) as c:
        refined = hessian(c)
    assert not np.array_equal(refined, calls)
    with_factors = 0
    for k in range(32):
        with cg.Context(m) as c:
            c.getGradIPField(u)  # the element records, the first to go
            fail(c, k)
            first = hessian(c)
            again = hessian(c)
        for got in (first, again):
            assert np.array_equal(got, refined) or np.array_equal(got, calls), k
        with_factors += np.array_equal(first, calls)
    assert with_factors >= 2  # the weights and their flags


@pytest.mark.parametrize("precision", ["fp32", "fp64", "learned"])
def test_update_with_little_memory(gpu_lib, precision):
    """An update needs room beside the old mesh: what the old mesh's passes
    derived from it is given back for that, whichever allocation fails."""
    import core_gb300 as cg
    (m0, u0), (m1, u1) = box(6), box(9, 2)
    want = fresh(m1, u1, precision)
    # the records go first, then the rest: two attempts fail where there are both
    for count in (1, 2) if precision == "fp64" else (1,):
        for k in range(16):
            with cg.Context(m0, precision=precision) as c:
                c.estimate_and_mark(u0, 0.1)
                fail(c, k, count)
                c.update_mesh(m1)
                c.test_hooks()
                assert same(c.estimate_and_mark(u1, 0.1)[:4], want), (count, k)


@pytest.mark.parametrize("precision", ["fp32", "fp64", "learned"])
def test_failed_update_after_everything_went(gpu_lib, precision):
    """No memory at all: the old mesh's passes make their setup anew, a captured
    one too."""
    import torch
    import core_gb300 as cg
    (m0, u0), (m1, u1) = box(6), box(9, 2)
    want = fresh(m0, u0, precision)
    stream = torch.cuda.Stream()
    with cg.Context(m0, precision=precision) as c, torch.cuda.stream(stream):
        c.set_stream(stream.cuda_stream)
        d_u = torch.from_numpy(u0).cuda()
        bits = torch.zeros((2, (m0.n_edges + 31) // 32), dtype=torch.int32, device="cuda")
        c.graph_capture(d_u.data_ptr(), 0.1, bits[0].data_ptr(), bits[1].data_ptr())
        fail(c, 3, 100)
        with pytest.raises(cg.SprgError) as e:
            c.update_mesh(m1)
        assert e.value.code == 4
        c.test_hooks()
        bits.zero_()
        c.graph_replay()
        stream.synchronize()
        b, e = bits.cpu().numpy().view(np.uint32), np.arange(m0.n_edges)
        assert np.array_equal((b[0][e >> 5] >> (e & 31)) & 1, want[1] & 1)
        assert same(c.estimate_and_mark(u0, 0.1)[:4], want)
        c.update_mesh(m1)
        assert same(c.estimate_and_mark(u1, 0.1)[:4], fresh(m1, u1, precision))
        c.set_stream(0)


@pytest.mark.parametrize("precision", ["fp32", "fp64", "learned"])
def test_a_failed_call_leaves_no_error_behind(gpu_lib, precision):
    """The error of a failed allocation is that call's alone: the next calls, on
    this context and on another, do not report it."""
    import core_gb300 as cg
    m, u = box(5)
    want = fresh(m, u, precision)
    for k in (0, 2, 5):
        with cg.Context(m, precision=precision) as c:
            fail(c, k, 100)
            with pytest.raises(cg.SprgError) as e:
                c.estimate_and_mark(u, 0.1)
            assert e.value.code == 4
            with cg.Context(m, precision=precision) as other:
                assert same(other.estimate_and_mark(u, 0.1)[:4], want)
            with pytest.raises(cg.SprgError) as e:
                c.estimate_and_mark(u, 0.1)
            assert e.value.code == 4
            c.test_hooks()
            assert same(c.estimate_and_mark(u, 0.1)[:4], want)
