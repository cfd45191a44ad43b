"""Per-mesh geometry of the FP32 form against extended precision."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [2, 3])
def test_largest_cofactor_norm(gpu_lib, n):
    """|cof J|_F^2 / |det J| of the worst element (the rounding-dominance test's
    measure) to FP64 rounding: on these boxes |p||q| is below 8 times a cofactor
    and the products' sum below 8 times the determinant, so the cofactors'
    squares carry 2 x 2 x 8 units of rounding, the determinant 8 + 16 and the sums
    and the quotient a few: 64."""
    import core_gb300 as cg
    from core_gb300 import workload
    for seed in range(24):
        m = workload.box(n, jitter=0.2, seed=seed)
        x = m.coords.astype(np.longdouble)
        e = [x[m.elem_verts[:, k]] - x[m.elem_verts[:, 0]] for k in (1, 2, 3)]
        cof = [np.cross(e[(i + 1) % 3], e[(i + 2) % 3]) for i in range(3)]
        q = sum((c * c).sum(1) for c in cof) / np.abs((e[0] * cof[0]).sum(1))
        with cg.Context(m, precision="fp32") as c:
            c.estimate_and_mark(workload.bump_field(m.coords, seed=1), 0.1)
            got = c.debug_read("qmax", np.float64, 1)[0]
        assert abs(got - q.max()) <= 64 * 2.0 ** -53 * q.max(), seed


def test_error_sum_on_triangles(gpu_lib):
    """The power of an error in the sum of a triangle mesh is its square root,
    correctly rounded, as the reference's pow(sqrt(err), 1); eight elements are
    summed as a tree over the lanes."""
    import core_gb300 as cg
    from core_gb300 import workload
    for seed in range(24):
        m = workload.box(2, nz=0, jitter=0.2, seed=seed)
        with cg.Context(m) as c:
            _, info = c.getSPRSizeField(c.getGradIPField(workload.bump_field(m.coords, seed=seed)), 0.1)
            err = c.debug_read("err", np.float64, m.n_elems)
        assert m.n_elems == 8 and np.all(err > 0)
        x = np.sqrt(err)
        x = x[:4] + x[4:]
        x = x[:2] + x[2:]
        assert info["error_sum"] == x[0] + x[1], seed


@pytest.mark.parametrize("n", [12, 20])
def test_pass_lengths_as_near_as_the_sequence(gpu_lib, n):
    """The FP64 pass's lengths against extended precision are no farther off than
    the reference's sequence (the measure call) on the same sizes: their rms
    errors agree to the statistics of the edges, 3 / sqrt(2 E) of 0.84 units."""
    import core_gb300 as cg
    from core_gb300 import workload
    m = workload.box(n, jitter=0.2, seed=4)
    with cg.Context(m) as c:
        size = c.estimate_and_mark(workload.bump_field(m.coords, seed=4), 1.28 / n)[0]
        L = c.debug_read("L", np.float64, m.n_edges)
        seq = c.measure_edges(size)
    Q = np.longdouble
    a, b = m.edge_verts.T
    d = m.coords.astype(Q)[b] - m.coords.astype(Q)[a]
    half = np.sqrt((d * d).sum(1)) / 2
    g = Q(0.577350269189626)
    s = size.astype(Q)
    exact = sum(half / (s[a] * ((1 - x) / 2) + s[b] * ((1 + x) / 2)) for x in (g, -g))

    def rms(x):
        return float(np.sqrt(np.mean(((x - exact) / exact * 2 ** 53) ** 2)))
    assert rms(L) <= rms(seq) * (1 + 3 / np.sqrt(2 * m.n_edges))
