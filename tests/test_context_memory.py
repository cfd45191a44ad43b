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
