"""Log-interpolated lengths of edges whose ends are infinite, NaN, far out, next
to each other or the same: the reference's values."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nz", [3, 0])
@pytest.mark.parametrize("kind", ["inf", "-inf", "nan", "two", "huge", "tiny", "equal", "far"])
def test_edges_out_of_range(gpu_lib, oracle_lib, nz, kind):
    import core_gb300 as cg
    from core_gb300 import workload
    m = workload.box(4, nz=nz, jitter=0.2, seed=3)
    x = m.coords
    v = m.n_verts // 2
    if kind in ("inf", "-inf", "nan"):
        x[v, 0] = float(kind)
    elif kind == "two":
        x[v, 0], x[v, 1] = np.inf, -np.inf
    elif kind == "huge":
        x *= 1e170
    elif kind == "tiny":
        x *= 1e-170
    elif kind == "equal":
        x[v] = x[v + 1]
    elif kind == "far":
        x[v, 1] = 1e160
    o = oracle_lib.OracleMesh.box(4, 4, nz)
    o.set_coords(x)
    rng = np.random.default_rng(5)
    V = m.n_verts
    sizes = np.exp(rng.uniform(np.log(0.02), np.log(0.4), (V, 3)))
    F = np.linalg.qr(rng.normal(size=(V, 3, 3)))[0]
    if nz == 0:
        t = rng.uniform(0, np.pi, V)
        F[:] = 0
        F[:, 0, 0], F[:, 0, 1], F[:, 1, 0], F[:, 1, 1], F[:, 2, 2] = np.cos(t), -np.sin(t), np.sin(t), np.cos(t), 1.0
    F = np.ascontiguousarray(F.reshape(V, 9))
    rc, want = o.measure_log(sizes, F)
    assert rc == 0
    with cg.Context(m) as c:
        got = c.measure_edges_log_aniso(sizes, F)
        pairs = c.measure_vertex_pairs(m.edge_verts, sizes=sizes, frames=F, log=True)
    for g in (got, pairs):
        assert np.array_equal(np.isnan(g), np.isnan(want)) and np.array_equal(np.isinf(g), np.isinf(want))
        fin = np.isfinite(want) & (want != 0)
        assert np.all(g[want == 0] == 0)
        if not fin.any():  # squares that over- or underflow throughout
            continue
        # the deflation threshold of the reference's iteration, against the
        # longest direction's weight at that edge
        d = np.linalg.norm((x[m.edge_verts[:, 1]] - x[m.edge_verts[:, 0]])[fin] / np.abs(want[fin]).max(), axis=1)
        assert np.all(np.abs(g[fin] - want[fin]) / np.abs(want[fin]).max() <= 1e-10 * d / sizes.min())
