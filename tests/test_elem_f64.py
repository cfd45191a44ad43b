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
    elif kind == "edge":      # determinants around 2^-400, cofactors around 2^-267
        x *= 2.0 ** -132
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


MESHES = [(1, 1, "plain"), (5, 4, "plain"), (9, 11, "plain"), (4, 4, "tiny"), (4, 4, "edge"), (4, 4, "huge"), (4, 3, "stretched"),
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


@pytest.mark.parametrize("n,nz", [(2, 3), (7, 6), (3, 0), (9, 0), (16, 0)])
@pytest.mark.parametrize("scale", [1e-160, 1e-70, 1.0, 1e70, 1e140])
@pytest.mark.parametrize("target", [0, 1000])
def test_element_sizes_from_errors(gpu_lib, oracle_lib, n, nz, scale, target):
    """h err^(-1/(D+2)) times the size factor, and the error integral, against
    extended precision on the errors the pass wrote.  2 ulps for the power and
    half an ulp for each of the two products after it: 7e-16 relative."""
    import core_gb300 as cg
    m, _ = mesh(oracle_lib, n, nz, "plain")
    ip = np.random.default_rng(5).normal(size=(m.n_elems, 3)) * scale
    if m.dim == 2:
        ip[:, 2] = 0.0
    with cg.Context(m) as c:
        if target:
            c.getTargetSPRSizeField(ip, target, 1e-300, 1e300)
        else:
            c.getSPRSizeField(ip, 0.1)
        err = c.debug_read("err", np.float64, m.n_elems).astype(np.longdouble)
        esize = c.debug_read("esize", np.float64, m.n_elems)
        out3 = c.debug_read("out3", np.float64, 3)
    x = m.coords[m.elem_verts]
    h = np.max([np.linalg.norm(x[:, a] - x[:, b], axis=1) for a in range(m.dim + 1) for b in range(a)], axis=0)
    ok = err > 1e-290
    power = err[ok] ** (-1 / np.longdouble(m.dim + 2))
    want = h[ok].astype(np.longdouble) * power * np.longdouble(out3[2])
    # h itself is compared as numpy sums it: two more ulps
    assert np.max(np.abs(esize[ok] - want) / want, initial=0.0) <= 7e-16 + 4.5e-16
    assert np.all(np.isinf(esize[err == 0])) or target
    if ok.all():
        G = np.sum(err ** (np.longdouble(2 * m.dim) / (m.dim + 2) / 2))
        assert abs(out3[1] - G) <= 1e-13 * G


@pytest.mark.parametrize("n,nz", [(1, 1), (5, 4), (11, 0)])
@pytest.mark.parametrize("sizes", ["random", "equal", "tiny", "huge", "odd"])
def test_iso_lengths_bitwise(gpu_lib, oracle_lib, n, nz, sizes):
    import core_gb300 as cg
    m, o = mesh(oracle_lib, n, nz, "plain")
    s = np.random.default_rng(6).uniform(0.2 / n, 3.0 / n, m.n_verts)
    if sizes == "equal":
        s[:] = 1.0 / (1.5 * n)
    elif sizes == "tiny":
        s *= 1e-200
    elif sizes == "huge":
        s *= 1e200
    elif sizes == "odd":
        s[::5] = [0.0, np.inf, np.nan, -s[0], 5e-324][:len(s[::5])] + [s[1]] * max(0, len(s[::5]) - 5)
    with cg.Context(m) as c:
        assert np.array_equal(c.measure_edges(s), o.measure(s), equal_nan=True)
        pairs = m.edge_verts[::-1]
        assert np.array_equal(c.measure_vertex_pairs(pairs, size=s), o.measure(s)[::-1], equal_nan=True)


@pytest.mark.parametrize("n,in_place", [(2, False), (7, False), (7, True)])
def test_pass_marks_are_those_of_the_bitwise_lengths(gpu_lib, oracle_lib, n, in_place):
    """The pass's marks against the reference lengths of its own sizes, with
    the adapt ratio placed so that an edge sits at each threshold; in_place:
    the last allocation of the first pass, the edge lengths', fails."""
    import core_gb300 as cg
    from core_gb300 import workload
    m, o = mesh(oracle_lib, n, n, "plain")
    u = workload.bump_field(m.coords, seed=3)
    with cg.Context(m) as c:
        L = np.sort(o.measure(c.estimate_and_mark(u, 0.1)[0]))
    for threshold in (0.5, 1.5):
        # sizes are proportional to the ratio: put the median edge on the threshold
        ratio = 0.1 * L[len(L) // 2] / threshold
        for k in range(0 if in_place else -1, 100):
            with cg.Context(m) as c:
                c.test_hooks(alloc_fail_after=k)
                try:
                    size, flags, ns, nc, _ = c.estimate_and_mark(u, ratio)
                    break
                except cg.SprgError as e:
                    assert e.code == 4
        L1 = o.measure(size)
        assert np.abs(L1 - threshold).min() < 1e-9
        assert np.array_equal((flags & 1) != 0, L1 > 1.5) and np.array_equal((flags & 4) != 0, L1 < 0.5)
        assert (ns, nc) == (int((L1 > 1.5).sum()), int((L1 < 0.5).sum()))


@pytest.mark.parametrize("n,kind", [(2, "plain"), (15, "plain"), (15, "warped"), (6, "tiny"), (6, "huge"), (9, "fan")])
@pytest.mark.parametrize("nc", [3, 9])
def test_triangle_recovery_bitwise(gpu_lib, oracle_lib, n, kind, nc):
    """Patches of 3 to 8 triangles, from the kept factors (twice, the second
    call on other samples) and factored in place; components that are 0
    everywhere, zero and infinite samples."""
    import core_gb300 as cg
    m, o = mesh(oracle_lib, n, 0, "plain")
    if kind == "warped":
        m.coords[:, 2] = np.sin(3 * m.coords[:, 0])
    elif kind in ("tiny", "huge"):
        # R's diagonal out of the fast quotients' range for huge; a tiny mesh is rank deficient below 1e-10
        m.coords *= 2.0 ** (401 if kind == "huge" else -20)
    elif kind == "fan":  # patches above 8 elements: every triangle of a block shares one vertex
        ev = m.elem_verts
        for t in range(20):
            if 40 not in ev[t]:
                ev[t][2] = 40
        m.v2e_off = m.v2e = None
    if kind == "fan":
        down = np.unique(np.sort(np.concatenate([m.elem_verts[:, [0, 1]], m.elem_verts[:, [1, 2]], m.elem_verts[:, [0, 2]]]), 1), axis=0)
        m.edge_verts = np.ascontiguousarray(down, np.int32)
    else:
        o.set_coords(m.coords)
    cnt = np.bincount(m.elem_verts.reshape(-1), minlength=m.n_verts)
    thread = (cnt >= 3) & (cnt <= 8)
    rng = np.random.default_rng(8)
    ips = [rng.normal(size=(m.n_elems, nc)) for _ in range(3)]
    ips[0][:, 2::3] = 0.0
    ips[2][:, [c for c in range(nc) if c == 2 or c > 4]] = 0.0  # a planar mesh's gradients
    ips[1][::7, 0] = 0.0
    ips[1][3, 1] = np.inf

    def answers(in_place):
        with cg.Context(m) as c:
            if in_place:  # the ninth allocation of the first call is the factors'
                c.test_hooks(alloc_fail_after=8)
                with pytest.raises(cg.SprgError):
                    c.recoverField(ips[0])
                c.test_hooks()
            return [c.recoverField(ip) for ip in ips]
    kept, placed = answers(False), answers(True)
    for a, b in zip(kept, placed):
        assert np.array_equal(a[thread], b[thread], equal_nan=True)
        # the grown patches: weighted sums with the factors kept, QR fits without
        fin = np.isfinite(a).all(axis=1) & np.isfinite(b).all(axis=1)
        assert np.abs(a[fin] - b[fin]).max() <= 1e-10 * np.abs(b[fin]).max()
    if kind == "fan":
        assert cnt.max() > 8
        return
    for ip, got in zip(ips, kept):
        rc, want, _, _ = o.recover(ip)
        assert rc == 0
        assert np.array_equal(got[thread], want[thread], equal_nan=True)


def metric_of(m, kind, seed=9):
    """sizes and frames: rotations in the plane (2D) or in space, slightly
    off orthonormal; odd: sizes and frames the fast forms hand over."""
    rng = np.random.default_rng(seed)
    V = m.n_verts
    sizes = np.exp(rng.uniform(np.log(0.02), np.log(0.4), (V, 3)))
    if m.dim == 2 and kind != "space":
        t = rng.uniform(0, np.pi, V)
        F = np.zeros((V, 3, 3))
        F[:, 0, 0], F[:, 0, 1], F[:, 1, 0], F[:, 1, 1], F[:, 2, 2] = np.cos(t), -np.sin(t), np.sin(t), np.cos(t), 1.0
        if kind == "skew":
            F[:, :2, :2] *= rng.uniform(0.5, 2.0, (V, 2, 2))
    else:
        F = np.linalg.qr(rng.normal(size=(V, 3, 3)))[0] * rng.uniform(0.5, 2.0, (V, 1, 1))
    if kind == "odd":
        sizes[::6] = 0.0
        sizes[1::11] = np.inf
        sizes[2::13] = -sizes[2::13]
        sizes[3::17] = 5e-324
        sizes[4::19] = 1e200
        F[::7] = 0.0
        F[5::23, 0, 0] = np.nan
    return sizes, np.ascontiguousarray(F.reshape(V, 9))


@pytest.mark.parametrize("n,nz", [(1, 1), (5, 4), (1, 0), (12, 0)])
@pytest.mark.parametrize("kind", ["plain", "skew", "space", "odd"])
def test_metric_lengths_and_qualities_bitwise(gpu_lib, oracle_lib, n, nz, kind):
    import core_gb300 as cg
    m, o = mesh(oracle_lib, n, nz, "plain")
    if kind == "skew" and m.dim == 2:
        m.coords[:, 2] = 0.75  # in a plane, but not z = 0
        o.set_coords(m.coords)
    sizes, F = metric_of(m, kind)
    with cg.Context(m) as c:
        L = o.measure(sizes=sizes, frames=F)
        assert np.array_equal(c.measure_edges_aniso(sizes, F), L, equal_nan=True)
        assert np.array_equal(c.measure_vertex_pairs(m.edge_verts, sizes=sizes, frames=F), L, equal_nan=True)
        assert np.array_equal(c.measureQuality(sizes=sizes, frames=F), o.quality(sizes=sizes, frames=F), equal_nan=True)
        iso = np.ascontiguousarray(sizes[:, 0])
        assert np.array_equal(c.measureQuality(iso), o.quality(iso), equal_nan=True)
        iso[:] = 0.3  # every vertex alike
        assert np.array_equal(c.measureQuality(iso), o.quality(iso), equal_nan=True)


@pytest.mark.parametrize("n,nz", [(4, 3), (9, 0)])
def test_qualities_without_the_transform_records(gpu_lib, oracle_lib, n, nz):
    """The allocation of the vertices' transforms fails: computed per element."""
    import core_gb300 as cg
    m, o = mesh(oracle_lib, n, nz, "plain")
    sizes, F = metric_of(m, "plain")
    with cg.Context(m) as c:
        c.test_hooks(alloc_fail_after=3)
        assert np.array_equal(c.measureQuality(sizes=sizes, frames=F), o.quality(sizes=sizes, frames=F))
    got = []
    for after in (4, -1):
        with cg.Context(m) as c:
            c.test_hooks(alloc_fail_after=after)
            got.append(c.measureQualityLog(sizes, F))
    assert np.array_equal(*got)


@pytest.mark.parametrize("n,nz", [(1, 1), (4, 5), (7, 0)])
@pytest.mark.parametrize("kind", ["plain", "diagonal", "isotropic", "close", "wide", "outside", "zero", "nan"])
def test_log_lengths(gpu_lib, oracle_lib, n, nz, kind):
    """Lengths under the log-interpolated field to 1e-10 (the deflation
    threshold of the reference's iteration), its failures included: frames
    along the axes, equal and nearly equal eigenvalues, sizes far apart,
    entries beyond the fast form's range."""
    import core_gb300 as cg
    m, o = mesh(oracle_lib, n, nz, "plain")
    sizes, F = metric_of(m, "plain")
    F /= np.linalg.norm(F.reshape(-1, 3, 3)[:, :, :1], axis=1, keepdims=True).reshape(-1, 1)
    if kind == "diagonal":
        F = np.tile(np.eye(3).reshape(1, 9), (m.n_verts, 1))
    elif kind == "isotropic":
        sizes[:] = sizes[:, :1]
    elif kind == "close":
        sizes[:] = 0.1 * (1 + 1e-11 * np.random.default_rng(2).normal(size=sizes.shape))
    elif kind == "wide":
        sizes[:, 0] *= 1e-9
        sizes[:, 1] *= 1e3
    elif kind == "outside":
        sizes[::3] *= 1e-60
    elif kind == "zero":
        sizes[1] = 0.0
    elif kind == "nan":
        F[2, 4] = np.nan
    rc, want = o.measure_log(sizes, F)
    with cg.Context(m) as c:
        if rc:
            with pytest.raises(cg.SprgError) as e:
                c.measure_edges_log_aniso(sizes, F)
            assert e.value.code == 7
            return
        got = c.measure_edges_log_aniso(sizes, F)
        assert np.all(np.isfinite(want)) and kind not in ("zero", "nan")
        # the deflated entries (up to 1e-10) couple the directions: against
        # the longest direction's weight at that edge
        scale = np.linalg.norm(m.coords[m.edge_verts[:, 1]] - m.coords[m.edge_verts[:, 0]], axis=1) / sizes.min()
        assert np.all(np.abs(got - want) <= 1e-10 * scale)
        assert np.abs(got - want).max() <= 1e-10 * want.max()
        L = c.getMaximumEdgeLength(sizes=sizes, frames=F, log=True)
        assert L == got.max()


@pytest.mark.parametrize("k", [5, 31, 32, 33, 64, 65, 127, 128, 129, 200])
def test_adjacency_ascends_at_every_patch_size(gpu_lib, k):
    """A fan of k triangles in shuffled order around one vertex: its size is
    the sum over its elements in ascending order, to the bit."""
    import core_gb300 as cg
    from core_gb300.mesh import Mesh
    rng = np.random.default_rng(k)
    t = np.arange(k) * 2 * np.pi / k
    x = np.zeros((k + 1, 3))
    x[1:, 0], x[1:, 1] = np.cos(t), np.sin(t)
    x[1:, :2] *= rng.uniform(0.8, 1.2, (k, 1))
    ring = 1 + np.arange(k)
    ev = np.stack([np.zeros(k, int), ring, np.roll(ring, -1)], 1)[rng.permutation(k)].astype(np.int32)
    ed = np.concatenate([np.stack([np.zeros(k, int), ring], 1), np.stack([ring, np.roll(ring, -1)], 1)]).astype(np.int32)
    ip = rng.normal(size=(k, 3))
    ip[:, 2] = 0.0
    with cg.Context(Mesh(2, x, ev, ed)) as c:
        size, _ = c.getSPRSizeField(ip, 0.1)
        esize = c.debug_read("esize", np.float64, k)
    total = 0.0
    for e in esize:
        total += e
    assert size[0] == total / k


def test_frame_of_an_updated_mesh(gpu_lib):
    """The bounding box of an update (block reductions): a mesh moved and
    stretched by sprg_update_mesh gives a fresh context's FP32 answers."""
    import core_gb300 as cg
    from core_gb300 import workload
    a, b = workload.box(11, jitter=0.2, seed=1), workload.box(11, jitter=0.2, seed=2)
    b.coords = b.coords * np.array([3.0, 0.2, 1.7]) - np.array([5.0, -0.3, 900.0])
    u = workload.sine_field(a.coords)
    with cg.Context(a, precision="fp32") as c:
        c.estimate_and_mark(u, 0.1)
        c.update_mesh(b)
        got = c.estimate_and_mark(u, 0.1)
    with cg.Context(b, precision="fp32") as c:
        want = c.estimate_and_mark(u, 0.1)
    assert np.array_equal(got[0], want[0]) and np.array_equal(got[1], want[1])


@pytest.mark.parametrize("precision", ["fp64", "fp32", "learned"])
def test_updates_in_a_row(gpu_lib, precision):
    """Growing, shrinking and moving back and forth through the spare arrays,
    with a pass after each, a failed allocation in between; every pass equals
    a fresh context's."""
    import core_gb300 as cg
    from core_gb300 import workload
    meshes = [workload.box(n, jitter=0.2, seed=s) for n, s in ((5, 1), (7, 2), (5, 3), (4, 4), (7, 5), (9, 6), (5, 1))]
    want = []
    for m in meshes:
        with cg.Context(m, precision=precision) as c:
            want.append(c.estimate_and_mark(workload.sine_field(m.coords), 0.1)[:2])
    with cg.Context(meshes[0], precision=precision) as c:
        for i, m in enumerate(meshes):
            if i:
                if m.n_verts > max(x.n_verts for x in meshes[:i]):
                    c.test_hooks(alloc_fail_after=4)
                    with pytest.raises(cg.SprgError) as e:
                        c.update_mesh(m)
                    assert e.value.code == 4
                    c.test_hooks()
                    old = meshes[i - 1]
                    got = c.estimate_and_mark(workload.sine_field(old.coords), 0.1)
                    assert np.array_equal(got[0], want[i - 1][0]) and np.array_equal(got[1], want[i - 1][1])
                c.update_mesh(m)
            got = c.estimate_and_mark(workload.sine_field(m.coords), 0.1)
            assert np.array_equal(got[0], want[i][0]) and np.array_equal(got[1], want[i][1])


@pytest.mark.parametrize("precision", ["fp32", "fp64", "learned"])
@pytest.mark.parametrize("n", [2, 8, 23])
@pytest.mark.parametrize("graph", [False, True])
def test_resident_passes_back_to_back(gpu_lib, precision, n, graph):
    """Sixty passes enqueued without a wait, the field changing between them on
    the same stream: each pass's marks are those of a fresh context (the
    kernels of a pass are launched while the ones before them drain)."""
    import torch
    import core_gb300 as cg
    from core_gb300 import workload
    m = workload.box(n, jitter=0.2, seed=2)
    E, ratio = m.n_edges, 1.28 / n
    nw = (E + 31) // 32
    us = [workload.bump_field(m.coords, seed=s) for s in (1, 2, 3)]
    want = []
    for u in us:
        with cg.Context(m, precision=precision) as c:
            want.append(c.estimate_and_mark(u, ratio)[1])
    stream = torch.cuda.Stream()
    with cg.Context(m, precision=precision) as c, torch.cuda.stream(stream):
        c.set_stream(stream.cuda_stream)
        fields = torch.from_numpy(np.stack(us)).cuda()
        d_u = fields[0].clone()
        bits = torch.zeros((2, nw), dtype=torch.int32, device="cuda")
        ptrs = (d_u.data_ptr(), ratio, bits[0].data_ptr(), bits[1].data_ptr())
        if graph:
            c.graph_capture(*ptrs)
        kept = []
        for i in range(60):
            d_u.copy_(fields[i % 3])
            if graph:
                c.graph_replay()
            else:
                c.estimate_and_mark_resident(*ptrs)
            kept.append(bits.clone())
        stream.synchronize()
        c.set_stream(0)
    e = np.arange(E)
    for i, b in enumerate(kept):
        b = b.cpu().numpy().view(np.uint32)
        flags = want[i % 3]
        assert np.array_equal((b[0][e >> 5] >> (e & 31)) & 1, flags & 1), i
        assert np.array_equal((b[1][e >> 5] >> (e & 31)) & 1, (flags >> 2) & 1), i


@pytest.mark.parametrize("n,far", [(2, 3e-7), (7, 3e-7), (7, 1e-3), (24, 3e-7)])
@pytest.mark.parametrize("threshold", [0.5, 1.5])
def test_blocks_with_many_guarded_edges(gpu_lib, n, far, threshold):
    """A quadratic on a regular box gives the interior equal sizes; the ratio puts
    the commonest length at a relative distance `far` of a threshold, so whole
    blocks of the FP32 measure kernel list their edges (or none).  The marks are
    the FP64 form's: the distance is far above FP64 rounding."""
    import core_gb300 as cg
    from core_gb300 import workload
    m = workload.box(n)
    u = (m.coords ** 2).sum(axis=1)
    with cg.Context(m) as c:
        size = c.estimate_and_mark(u, 0.1)[0]
        L = c.makeSizeField(size).measure()
        ratio = 0.1 * np.median(L) / (threshold * (1.0 + far))
        want = c.estimate_and_mark(u, ratio)[1]
    with cg.Context(m, precision="fp32") as c:
        _, flags, _, _, info = c.estimate_and_mark(u, ratio)
    assert info["n_guard_unresolved"] == 0
    if n == 24 and far < 1e-6:
        assert info["n_guard_edges"] > m.n_edges // 20
    assert np.array_equal(flags, want)


@pytest.mark.parametrize("n,extra", [(2, 0), (33, 0), (34, 0), (43, 0), (55, 0), (67, 0), (7, 2), (27, 2), (41, 2)])
def test_network_tiles_of_both_consumer_groups(gpu_lib, n, extra):
    """The inference kernel's answers from one tile in all (n = 2) to about eight
    per block, so each consumer group takes none, one or several; with more than
    sixteen neighbours for half of the vertices (extra edges) its wide form.
    Against the training kernel's forward pass: both accumulate BF16 products in
    FP32 and round each hidden activation to BF16 once, so an activation may
    differ by one BF16 unit (2^-8) where the sums' last bits straddle a boundary."""
    import torch
    import core_gb300 as cg
    from core_gb300 import learned, workload
    m = workload.box(n, jitter=0.2, seed=13)
    v = np.arange(m.n_verts // 2)
    for d in range(2, 2 + extra):
        m.edge_verts = np.concatenate([m.edge_verts, np.stack([v, v + d], 1).astype(np.int32)])
    u = workload.bump_field(m.coords, seed=13)
    with cg.Context(m, precision="fp32") as c:
        x_bits, aux = learned.features(c, u)
        p = learned.init_params(21)
        c.set_mlp_params(p)
        c.set_precision("learned")
        c.set_learned_options(True, 1e30)
        c.estimate_and_mark(u, 0.05 / n)
        rec = c.debug_read("rec16", np.float32, 8 * m.n_verts).reshape(-1, 8)[:, 4:7].astype(np.float64)
    tr = learned.Trainer(p, 64)
    z = tr.forward(torch.from_numpy(x_bits.view(np.int16)).cuda()).cpu().numpy().astype(np.float64)
    ok = aux[:, 4] == 0
    assert ok.any() or n == 2
    want = aux[ok, :3] + z[ok] * aux[ok, 3:4]
    scale = np.abs(z[ok] * aux[ok, 3:4]).max(initial=0.0) * 2e-2 + 1e-6 * np.abs(want).max(initial=0.0)
    assert np.abs(rec[ok] - want).max(initial=0.0) <= scale


@pytest.mark.parametrize("n", [1, 2, 15, 16, 33, 130])
@pytest.mark.parametrize("kind", ["layer", "odd", "nan"])
def test_flat_records_against_the_general_form(gpu_lib, n, kind):
    """The mixed anisotropic pass of a mesh in the z = 0 plane (compact records)
    and of the same mesh at z = 1/4 (the general records and products): the same
    qualities to the bit (only products of exact zeros differ), the same marks."""
    import torch
    import core_gb300 as cg
    from core_gb300 import workload
    from core_gb300.mesh import makeMdsBox
    m = makeMdsBox(n, n, 0)
    rng = np.random.default_rng(n)
    inner = np.all((m.coords[:, :2] > 0) & (m.coords[:, :2] < 1), axis=1)
    m.coords[inner, :2] += rng.uniform(-0.2, 0.2, (int(inner.sum()), 2)) / n
    u = workload.boundary_layer_field(m.coords)
    if kind == "odd":  # flat pieces (zero Hessians), values over many orders of magnitude
        u = np.where(m.coords[:, 0] < 0.5, 0.0, u * 10.0 ** rng.integers(-200, 100, m.n_verts))
    elif kind == "nan":
        u[m.n_verts // 2] = np.nan
    got = []
    for z in (0.0, 0.25):
        m.coords[:, 2] = z
        with cg.Context(m, precision="fp32") as c:
            bits = torch.zeros((2, (m.n_edges + 31) // 32), dtype=torch.int32, device="cuda")
            q = torch.zeros(m.n_elems, dtype=torch.float64, device="cuda")
            d_u = torch.from_numpy(u).cuda()
            torch.cuda.synchronize()
            c.aniso_estimate_and_mark_resident(d_u.data_ptr(), 2.0 / n ** 2, 0.05 / n, 4.0 / n, bits[0].data_ptr(),
                                               bits[1].data_ptr(), q.data_ptr())
            torch.cuda.synchronize()
            got.append((bits.cpu().numpy(), q.cpu().numpy()))
    assert np.array_equal(got[0][1], got[1][1], equal_nan=True)
    assert np.array_equal(got[0][0], got[1][0])


@pytest.mark.parametrize("n", [2, 3, 16, 33])
@pytest.mark.parametrize("ratio", [1.0, 30.0, 1e5, 1e7])
@pytest.mark.parametrize("scale", [1.0, 1e40])
def test_rotated_frames_lengths(gpu_lib, n, ratio, scale):
    """The FP64 anisotropic pass's lengths (rotation frames on a plane) against the
    bitwise lengths of the same metric, sizes' ratios up to and past the line
    (2^19) where the sequence itself is taken, lengths inside and outside the
    ordinary range: each form's dot products round to 8 ulps of |d|, which
    counts at most `ratio` times in the length.  Marks: the bitwise lengths'."""
    import torch
    import core_gb300 as cg
    from core_gb300 import workload
    from core_gb300.mesh import makeMdsBox
    m = makeMdsBox(n, n, 0)
    m.coords *= scale
    x = m.coords / scale
    u = workload.boundary_layer_field(x)
    hmin = 0.3 * scale / n
    eps = 0.1 * np.abs(u).max()  # h = sqrt(eps / |lambda|), lambda up to about |u| n^2 / scale^2
    with cg.Context(m) as c:
        bits = torch.zeros((2, (m.n_edges + 31) // 32), dtype=torch.int32, device="cuda")
        d_u = torch.from_numpy(u).cuda()
        torch.cuda.synchronize()
        q = torch.zeros(m.n_elems, dtype=torch.float64, device="cuda")
        c.aniso_estimate_and_mark_resident(d_u.data_ptr(), eps, hmin, hmin * ratio, bits[0].data_ptr(),
                                           bits[1].data_ptr(), q.data_ptr())
        torch.cuda.synchronize()
        L = c.debug_read("L", np.float64, m.n_edges)
        sizes = c.debug_read("sizes3", np.float64, 3 * m.n_verts).reshape(-1, 3)
        frames = c.debug_read("frames9", np.float64, 9 * m.n_verts).reshape(-1, 9)
        want = c.makeSizeField(sizes=sizes, frames=frames).measure()
        want_q = c.measureQuality(sizes=sizes, frames=frames)
    aspect = (sizes[:, :2].max(axis=1) / sizes[:, :2].min(axis=1)).max()
    spread = max(aspect, sizes[:, :2].max() / sizes[:, :2].min())
    assert np.all(np.abs(L - want) <= (32 + 16 * spread) * 2.0 ** -53 * want)
    # a metric edge vector is off by delta = 4 spread ulps of its length at most,
    # 48 A^2 / s^2 <= 1 by 8 delta
    assert np.all(np.abs(q.cpu().numpy() - want_q) <= (32 + 32 * spread) * 2.0 ** -53)
    e = np.arange(m.n_edges)
    b = bits.cpu().numpy().view(np.uint32)
    assert np.array_equal((b[0][e >> 5] >> (e & 31)) & 1, want > 1.5)
    assert np.array_equal((b[1][e >> 5] >> (e & 31)) & 1, want < 0.5)


@pytest.mark.parametrize("n,kind", [(2, "plain"), (3, "plain"), (16, "plain"), (33, "warped"), (9, "fan"), (9, "no memory")])
def test_pass_recovery_on_triangles(gpu_lib, n, kind):
    """The FP64 anisotropic pass's Hessian (refined weights) against the calls'
    (the factors, in absolute coordinates: a recovered value is good to about
    cond(patch) ulps, the vertices' distance from the origin over an element's
    width, below 4 n, a few times over, and the second gradient divides the first
    recovery's error by the width); with a patch too large for the weights, the
    factors' bits."""
    import torch
    import core_gb300 as cg
    from core_gb300 import workload
    from core_gb300.mesh import Mesh, makeMdsBox
    m = makeMdsBox(n, n, 0)
    rng = np.random.default_rng(n)
    inner = np.all((m.coords[:, :2] > 0) & (m.coords[:, :2] < 1), axis=1)
    m.coords[inner, :2] += rng.uniform(-0.2, 0.2, (int(inner.sum()), 2)) / n
    if kind == "warped":
        m.coords[:, 2] = 0.1 * np.sin(3 * m.coords[:, 0])
    elif kind == "fan":  # a wheel of twelve triangles beside the square
        k, V = 12, m.n_verts
        t = np.arange(k) * 2 * np.pi / k
        x = np.zeros((k + 1, 3))
        x[1:, 0], x[1:, 1] = np.cos(t), np.sin(t)
        x[:, 0] += 3.0
        ring = V + 1 + np.arange(k)
        hub = np.full(k, V)
        ev = np.stack([hub, ring, np.roll(ring, -1)], 1)
        ed = np.concatenate([np.stack([hub, ring], 1), np.stack([ring, np.roll(ring, -1)], 1)])
        m = Mesh(2, np.concatenate([m.coords, x]), np.concatenate([m.elem_verts, ev]).astype(np.int32),
                 np.concatenate([m.edge_verts, ed]).astype(np.int32))
    u = workload.boundary_layer_field(m.coords)
    with cg.Context(m) as c:
        ip = c.getGradIPField(u)
        ip2 = c.getGradIPField(c.recoverField(ip))
        want = c.recoverField(ip2)
    with cg.Context(m) as c:
        if kind == "no memory":
            c.test_hooks(alloc_fail_after=3)
        bits = torch.zeros((2, (m.n_edges + 31) // 32), dtype=torch.int32, device="cuda")
        d_u = torch.from_numpy(u).cuda()
        torch.cuda.synchronize()
        try:
            c.aniso_estimate_and_mark_resident(d_u.data_ptr(), 0.1, 0.1 / n, 1.0, bits[0].data_ptr(), bits[1].data_ptr())
        except cg.SprgError:
            assert kind == "no memory"  # the failed allocation was one the pass needs
            return
        torch.cuda.synchronize()
        got = c.debug_read("rec", np.float64, 9 * m.n_verts).reshape(-1, 9)
    if kind == "fan":
        assert np.array_equal(got, want)
    one = 64 * 4 * n * 2.0 ** -53
    assert np.abs(got - want).max() <= one * (np.abs(ip2).max() + 4 * n * np.abs(ip).max())
