"""The FP64 element records and what is computed from them against the
oracle, bitwise: ordinary meshes, coordinates whose determinants leave the
range of the fast quotients, degenerate and inverted elements, values that
are not finite, and the kernels' in-place form."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def mesh(oracle_lib, n, nz, kind):
    from core_gb300 import workload
    m = workload.box(n, nz=nz, jitter=0.2, seed=11)
    x = m.coords.copy()
    if kind == "tiny":        # tet determinants below 2^-500
        x *= 2.0 ** -172
    elif kind == "huge":      # above 2^500
        x *= 2.0 ** 170
    elif kind == "stretched":
        x[:, 0] *= 1e-40
        x[:, 1] *= 1e30
    elif kind == "degenerate":  # vertices of some elements coincide, others turn inside out
        x[7] = x[8]
        x[20] += 3.0 / n
    elif kind == "inf":
        x[5, 0] = np.inf
    m.coords = x
    o = oracle_lib.OracleMesh.box(n, n, nz)
    o.set_coords(x)
    m.v2e_off, m.v2e = o.v2e_off, o.v2e
    return m, o


MESHES = [(1, 1, "plain"), (5, 4, "plain"), (9, 11, "plain"), (4, 4, "tiny"), (4, 4, "huge"), (4, 3, "stretched"),
          (4, 4, "degenerate"), (3, 3, "inf"), (1, 0, "plain"), (13, 0, "plain"), (6, 0, "tiny"), (6, 0, "degenerate")]


@pytest.mark.parametrize("n,nz,kind", MESHES)
def test_gradients_bitwise(gpu_lib, oracle_lib, n, nz, kind):
    import core_gb300 as cg
    m, o = mesh(oracle_lib, n, nz, kind)
    rng = np.random.default_rng(3)
    u = rng.normal(size=m.n_verts)
    v = rng.normal(size=(m.n_verts, 3))
    v[2] = 0.0
    for hook in (-1, 2):  # 2: no memory for the records, computed in place
        with cg.Context(m) as c:
            c.test_hooks(alloc_fail_after=hook)
            got = c.getGradIPField(u)
            assert np.array_equal(got, o.grad_ip(u), equal_nan=True)
        with cg.Context(m) as c:
            c.test_hooks(alloc_fail_after=hook)
            assert np.array_equal(c.getGradIPField(v), o.grad_ip(v), equal_nan=True)
    u[1] = np.inf
    u[3] = np.nan
    with cg.Context(m) as c:
        assert np.array_equal(c.getGradIPField(u), o.grad_ip(u), equal_nan=True)


def test_records_follow_a_mesh_update(gpu_lib, oracle_lib):
    import core_gb300 as cg
    m, _ = mesh(oracle_lib, 5, 4, "plain")
    m2, o2 = mesh(oracle_lib, 5, 4, "stretched")
    u = np.random.default_rng(4).normal(size=m.n_verts)
    with cg.Context(m) as c:
        c.getGradIPField(u)
        c.update_mesh(m2)
        assert np.array_equal(c.getGradIPField(u), o2.grad_ip(u))
