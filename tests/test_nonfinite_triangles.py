"""Fields on triangles with infinite, NaN and nearly overflowing values: the
recovered values are the reference's (the oracle's fits), at vertices whose
patches grow as elsewhere."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def square(n, seed=1):
    from core_gb300 import workload
    m = workload.box(n, nz=0, jitter=0.2, seed=seed)
    return m, workload.boundary_layer_field(m.coords)


@pytest.mark.parametrize("n", [2, 5, 13])
@pytest.mark.parametrize("bad", [np.inf, -np.inf, np.nan])
def test_recovered_values(gpu_lib, oracle_lib, n, bad):
    """One bad vertex after the other: finite, infinite and NaN values in the same
    places as the oracle's, the finite ones near."""
    import core_gb300 as cg
    m, u = square(n)
    o = oracle_lib.OracleMesh.box(n, n, 0)
    o.set_coords(m.coords)
    with cg.Context(m) as c:
        for v in range(0, m.n_verts, max(1, m.n_verts // 12)):
            w = u.copy()
            w[v] = bad
            ip = c.getGradIPField(w)
            rc, want, _, _ = o.recover(ip)
            got = c.recoverField(ip)
            assert rc == 0
            assert np.array_equal(np.isnan(got), np.isnan(want)) and np.array_equal(np.isinf(got), np.isinf(want)), v
            fin = np.isfinite(want)
            assert np.abs(got[fin] - want[fin]).max(initial=0) <= 1e-10 * np.abs(want[fin]).max(initial=1)


@pytest.mark.parametrize("n", [3, 9])
@pytest.mark.parametrize("bad", [np.inf, np.nan, 1e306])
def test_anisotropic_pass(gpu_lib, n, bad):
    """The FP64 anisotropic pass's Hessian has NaN, infinite and finite values where
    the calls' (the sequence of the factors) has them, and its marks are those of
    the calls' lengths."""
    import torch
    import core_gb300 as cg
    m, u = square(n)
    e = np.arange(m.n_edges)
    with cg.Context(m) as c:
        for v in range(0, m.n_verts, max(1, m.n_verts // 12)):
            w = u.copy()
            w[v] = bad
            want = c.recoverField(c.getGradIPField(c.recoverField(c.getGradIPField(w))))
            bits = torch.zeros((2, (m.n_edges + 31) // 32), dtype=torch.int32, device="cuda")
            d_u = torch.from_numpy(w).cuda()
            torch.cuda.synchronize()
            c.aniso_estimate_and_mark_resident(d_u.data_ptr(), 0.1, 0.1 / n, 1.0, bits[0].data_ptr(),
                                               bits[1].data_ptr())
            torch.cuda.synchronize()
            got = c.debug_read("rec", np.float64, 9 * m.n_verts).reshape(-1, 9)
            assert np.array_equal(np.isnan(got), np.isnan(want)) and np.array_equal(np.isinf(got), np.isinf(want)), v
            sizes, frames = c.hessian_metric(want, 0.1, 0.1 / n, 1.0)
            L = c.measure_edges_aniso(sizes, frames)
            b = bits.cpu().numpy().view(np.uint32)
            sure = ~(np.abs(L - 1.5) < 1e-9) & ~(np.abs(L - 0.5) < 1e-9)
            assert np.array_equal(((b[0][e >> 5] >> (e & 31)) & 1)[sure], (L > 1.5)[sure]), v
            assert np.array_equal(((b[1][e >> 5] >> (e & 31)) & 1)[sure], (L < 0.5)[sure]), v


@pytest.mark.parametrize("n", [520])
def test_anisotropic_pass_on_a_large_square(gpu_lib, n):
    """From 2^18 vertices on such vertices are listed for a kernel of their own."""
    import torch
    import core_gb300 as cg
    m, u = square(n)
    assert m.n_verts > 1 << 18
    rng = np.random.default_rng(1)
    u[rng.choice(m.n_verts, 300, replace=False)] = np.inf
    u[rng.choice(m.n_verts, 300, replace=False)] = -1e306
    bits = torch.zeros((2, (m.n_edges + 31) // 32), dtype=torch.int32, device="cuda")
    d_u = torch.from_numpy(u).cuda()
    torch.cuda.synchronize()
    with cg.Context(m) as c:
        want = c.recoverField(c.getGradIPField(c.recoverField(c.getGradIPField(u))))
        c.aniso_estimate_and_mark_resident(d_u.data_ptr(), 0.1, 0.1 / n, 1.0, bits[0].data_ptr(), bits[1].data_ptr())
        torch.cuda.synchronize()
        got = c.debug_read("rec", np.float64, 9 * m.n_verts).reshape(-1, 9)
    assert np.isnan(want).any()
    assert np.array_equal(np.isnan(got), np.isnan(want)) and np.array_equal(np.isinf(got), np.isinf(want))


@pytest.mark.parametrize("n,recovery", [(9, 1), (520, 2)])
def test_launches_counted(gpu_lib, n, recovery):
    """Two gradients, two recoveries, the metric and the lengths."""
    import torch
    import core_gb300 as cg
    m, u = square(n)
    bits = torch.zeros((2, (m.n_edges + 31) // 32), dtype=torch.int32, device="cuda")
    d_u = torch.from_numpy(u).cuda()
    torch.cuda.synchronize()
    with cg.Context(m) as c:
        for _ in range(2):
            c.aniso_estimate_and_mark_resident(d_u.data_ptr(), 0.1, 0.1 / n, 1.0, bits[0].data_ptr(), bits[1].data_ptr())
        torch.cuda.synchronize()
        assert c.last_launch_count == 2 + 2 * recovery + 2
