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
        fail(c, 1)  # f grows, then ip
        with pytest.raises(cg.SprgError) as e:
            c.getGradIPField(v)
        assert e.value.code == _lib.SPRG_ENOMEM
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
