"""Vertices whose patches grow (fewer than four tets, as at a box's corners): in
every form the recovered gradient there is the FP64 form's, bit for bit."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", ["fp32", "learned"])
@pytest.mark.parametrize("kind", ["bumps", "constant", "offset", "infinite", "thin", "large", "flat"])
def test_listed_gradients_are_the_fp64_forms(gpu_lib, precision, kind):
    import core_gb300 as cg
    from core_gb300 import workload
    for n in (2, 5):
        m = workload.box(n, jitter=0.2, seed=n)
        u = workload.bump_field(m.coords, seed=n)
        if kind == "constant":
            u[:] = 3.25
        elif kind == "offset":
            u += 1e9
        elif kind == "infinite":
            u[0] = np.inf
        elif kind == "thin":
            m.coords[:, 0] *= 1e-5
        elif kind == "large":
            m.coords *= 2.0 ** 30
        elif kind == "flat":  # a tet without volume beside a corner
            m.coords[1] = m.coords[0]
        with cg.Context(m) as c:
            want = c.recoverField(c.getGradIPField(u))
        with cg.Context(m, precision=precision) as c:
            if precision == "fp32":  # a batch: no second pass in FP64 where rounding dominates
                c.set_batch([0, m.n_verts], [0, m.n_elems], [0.1])
            c.estimate_and_mark(u, 0.1)
            got = c.debug_read("rec", np.float64, 3 * m.n_verts).reshape(-1, 3)
        grown = np.bincount(m.elem_verts.reshape(-1)) < 4
        assert grown.any()
        assert np.array_equal(got[grown], want[grown], equal_nan=True)


@pytest.mark.parametrize("precision", ["fp32", "learned"])
def test_without_memory_for_the_gradients(gpu_lib, precision):
    """Each allocation of the first pass fails once (given back for it: the listed
    patches' gradients, which the sums then compute in place)."""
    import core_gb300 as cg
    from core_gb300 import workload
    m = workload.box(4, jitter=0.2, seed=4)
    m.coords[:, 0] *= 1e-3
    u = workload.bump_field(m.coords, seed=4)
    with cg.Context(m, precision=precision) as c:
        want = c.estimate_and_mark(u, 0.1)[:4]
    passed = 0
    for k in range(56):
        with cg.Context(m, precision=precision) as c:
            c.test_hooks(alloc_fail_after=k | 1 << 24)
            try:
                got = c.estimate_and_mark(u, 0.1)[:4]
            except cg.SprgError as e:
                assert e.code == 4  # nothing there yet to give back
                continue
            passed += 1
            again = c.estimate_and_mark(u, 0.1)[:4]
        for g in (got, again):
            assert np.array_equal(g[0], want[0]) and np.array_equal(g[1], want[1]) and g[2:] == want[2:], k
    assert passed > 0
