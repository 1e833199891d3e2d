"""Device mesh extraction (models/renderer.py:9-34, 353-358): lattice values
against the oracle's extract_fields, vertices against the lattice-edge
crossings every marching-cubes variant produces, and the triangles by their
properties: closed, consistently oriented, outward, Euler characteristic."""
import numpy as np
import pytest
import torch

from oracle import mesh as OMS

pytestmark = pytest.mark.gpu


def _mc(u, thr=0.0, lo=(-1.0, -1.0, -1.0), hi=(1.0, 1.0, 1.0)):
    from supernormal_gb300.mesh import marching_cubes

    v, t = marching_cubes(torch.as_tensor(u, device="cuda"), thr, lo, hi)
    return v.double().cpu().numpy(), t.long().cpu().numpy()


def _topology(v, t, closed=True):
    e = np.concatenate([t[:, [0, 1]], t[:, [1, 2]], t[:, [2, 0]]])
    directed = {tuple(x) for x in e.tolist()}
    assert len(directed) == len(e), "a directed edge appears twice: inconsistent orientation"
    und = np.sort(e, axis=1)
    _, cnt = np.unique(und, axis=0, return_counts=True)
    if closed:
        assert (cnt == 2).all(), "open or non-manifold edges"
    else:                                  # cut by the lattice's box: boundary edges once
        assert (cnt <= 2).all(), "non-manifold edges"
    return len(v) - len(cnt) + len(t)     # Euler characteristic


def _lattice(f, res, lo=-1.0, hi=1.0):
    g = np.linspace(lo, hi, res)
    x, y, z = np.meshgrid(g, g, g, indexing="ij")
    return f(x, y, z).astype(np.float32)


def test_sphere_mesh():
    u = _lattice(lambda x, y, z: 0.5 - np.sqrt(x * x + y * y + z * z), 48)   # -sdf of a sphere
    v, t = _mc(u)
    ref = OMS.edge_crossings(u, 0.0, (-1, -1, -1), (1, 1, 1))
    assert len(v) == len(ref)
    np.testing.assert_allclose(v[np.lexsort(v.T)], ref[np.lexsort(ref.T)], atol=2e-6)
    assert _topology(v, t) == 2
    c = v[t].mean(1)
    n = np.cross(v[t[:, 1]] - v[t[:, 0]], v[t[:, 2]] - v[t[:, 0]])
    assert ((n * c).sum(1) > 0).all()                                    # normals point outward
    assert np.abs(np.linalg.norm(v, axis=1) - 0.5).max() < 0.01


def test_torus_mesh_genus_one():
    def f(x, y, z):
        q = np.sqrt(x * x + y * y) - 0.5
        return 0.2 - np.sqrt(q * q + z * z)
    v, t = _mc(_lattice(f, 64))
    assert _topology(v, t) == 0


@pytest.mark.parametrize("seed", [0, 1, 2])
def test_random_field_is_watertight(seed):
    """Random values (every ambiguous face configuration occurs) inside a
    border that is outside: closed, consistently oriented surfaces."""
    rng = np.random.default_rng(seed)
    u = rng.uniform(-1, 1, (24, 20, 18)).astype(np.float32)
    u[0], u[-1], u[:, 0], u[:, -1], u[:, :, 0], u[:, :, -1] = -1, -1, -1, -1, -1, -1
    v, t = _mc(u, 0.0, (0, 0, 0), (23, 19, 17))
    ref = OMS.edge_crossings(u, 0.0, (0, 0, 0), (23, 19, 17))
    assert len(v) == len(ref) and len(t) > 100
    np.testing.assert_allclose(v[np.lexsort(v.T)], ref[np.lexsort(ref.T)], atol=2e-5)
    _topology(v, t)
    # the host restatement numbers vertices the same way: identical triangles
    hv, ht = OMS.marching_cubes(u, 0.0, (0, 0, 0), (23, 19, 17))
    np.testing.assert_array_equal(t, ht)
    np.testing.assert_allclose(v, hv, atol=2e-5)


@pytest.mark.parametrize("shape", [(2, 2, 2), (3, 2, 31), (2, 3, 32), (5, 4, 33), (4, 7, 64), (3, 5, 65), (9, 120, 97),
                                   (33, 17, 2)])
def test_word_edges_match_host(shape):
    """Rows that end inside, at and past a 32-point word, and more words than
    one tile holds: the same vertices and triangles, in the same order, as the
    host restatement (vertices: float32 arithmetic of coordinates below 128)."""
    rng = np.random.default_rng(sum(shape))
    u = rng.uniform(-1, 1, shape).astype(np.float32)
    u.flat[:: 7] = np.nan                                  # outside, as any comparison with NaN is false
    hi = tuple(float(n - 1) for n in shape)
    v, t = _mc(u, 0.1, (0, 0, 0), hi)
    hv, ht = OMS.marching_cubes(u, 0.1, (0, 0, 0), hi)
    np.testing.assert_array_equal(t, ht)
    np.testing.assert_allclose(v, hv, atol=2e-5)


@pytest.mark.parametrize("res,slab", [((2, 2, 2), 1), ((5, 3, 33), 1), ((33, 7, 31), 500), ((64, 65, 32), 1 << 21),
                                      ((20, 40, 70), 9000)])
def test_lattice_slabs_equal_the_point_queries(built_lib, res, slab):
    """Slabs of any size and rows that end inside a tile: the values of
    extract_fields' point by point query, bit for bit."""
    from supernormal_gb300.fields import SDFNetwork
    from supernormal_gb300.mesh import extract_fields, sdf_lattice

    torch.manual_seed(1)
    net = SDFNetwork(3, 1, 64, 1, skip_in=(-1,), bias=0.5, input_concat=True, encoding_config=dict(
        otype="HashGrid", n_levels=16, n_features_per_level=2, log2_hashmap_size=15, base_resolution=16,
        per_level_scale=1.447))
    net.bindwidth = 16
    net = net.cuda()
    lo, hi = (-1.0, -0.9, -1.1), (1.0, 0.8, 1.2)
    want = extract_fields(lo, hi, res, net.sdf_raw)
    assert torch.equal(sdf_lattice(net, lo, hi, res, slab_points=slab), -want)
    assert torch.equal(sdf_lattice(net, lo, hi, res, negate=False, slab_points=slab), want)


def test_empty_and_capacity():
    from supernormal_gb300._lib import call, stream_handle

    u = torch.full((8, 8, 8), -1.0, device="cuda")
    v, t = _mc(u.cpu().numpy())
    assert v.shape == (0, 3) and t.shape == (0, 3)
    # outputs are written only up to the given capacity; the counts are exact
    uu = torch.as_tensor(_lattice(lambda x, y, z: 0.5 - np.sqrt(x * x + y * y + z * z), 16), device="cuda")
    ws = torch.empty(int(call("sn_marching_cubes_workspace_bytes", 16, 16, 16)), dtype=torch.uint8, device="cuda")
    counts = torch.zeros(2, dtype=torch.int32, device="cuda")
    verts = torch.full((10, 3), 7.0, device="cuda")
    tris = torch.full((5, 3), -7, dtype=torch.int32, device="cuda")
    lo = np.array([-1.0, -1.0, -1.0])
    hi = np.array([1.0, 1.0, 1.0])
    call("sn_marching_cubes", uu, 16, 16, 16, 0.0, lo.ctypes.data, hi.ctypes.data, 10, 5, verts, tris, counts, ws,
         stream_handle())
    n_v, n_t = counts.tolist()
    assert n_v > 10 and n_t > 5 and (tris >= 0).all()


def test_sdf_network_extract_geometry_matches_oracle_lattice(built_lib):
    """NeuSRenderer.extract_geometry: the -sdf lattice of the fused field
    against the oracle's extract_fields with the float64 field, then a mesh
    whose vertices are the crossings of that lattice."""
    from oracle import field as OF
    from supernormal_gb300.fields import SDFNetwork, SingleVarianceNetwork
    from supernormal_gb300.mesh import sdf_lattice
    from supernormal_gb300.renderer import NeuSRenderer

    enc = dict(otype="HashGrid", n_levels=16, n_features_per_level=2, log2_hashmap_size=15,
               base_resolution=16, per_level_scale=1.447)
    torch.manual_seed(0)
    net = SDFNetwork(3, 1, 64, 1, skip_in=(-1,), bias=0.5, encoding_config=enc, input_concat=True)
    with torch.no_grad():
        net.encoding.params.mul_(300.0)
        net.lin0.weight_v[:, 3:].normal_(0.0, 0.05)
    net.bindwidth = 16
    net = net.cuda()
    lo, hi = torch.tensor([-1.0, -1.0, -1.0]), torch.tensor([1.0, 1.0, 1.0])
    u = sdf_lattice(net, lo, hi, 40).cpu().numpy()
    prm = OF.params_from_module(net)
    geom = OF.geometry_from_module(net)
    ref = OMS.extract_fields(lo, hi, 40, lambda p: -OF.sdf_network(p, **prm, geom=geom, active_levels=16,
                                                                    out_cols=1))
    assert np.abs(u - ref).max() < 2e-5 * max(1.0, np.abs(ref).max())
    r = NeuSRenderer(net, SingleVarianceNetwork(0.3).cuda())
    v, t = r.extract_geometry(lo, hi, 40)
    assert v.dtype == np.float64 and t.dtype == np.int64 and len(t) > 100
    crossing = OMS.edge_crossings(u, 0.0, lo.numpy(), hi.numpy())
    assert len(v) == len(crossing)
    _topology(v, t, closed=False)         # this field's zero set reaches the box
    hv, ht = OMS.marching_cubes(u, 0.0, lo.numpy(), hi.numpy())
    np.testing.assert_array_equal(t, ht)


def _small_net():
    from supernormal_gb300.fields import SDFNetwork

    torch.manual_seed(0)
    net = SDFNetwork(3, 1, 64, 1, input_concat=True, encoding_config=dict(
        otype="HashGrid", n_levels=2, n_features_per_level=2, log2_hashmap_size=10, base_resolution=8,
        per_level_scale=1.5)).cuda()
    net.bindwidth = 2
    return net


def test_lattice_asks_a_replaced_sdf_raw(monkeypatch):
    """An sdf_raw of the instance's own, or put in the class' place, is queried."""
    from supernormal_gb300.fields import SDFNetwork
    from supernormal_gb300.mesh import sdf_lattice

    lo, hi, raw = (-1.0,) * 3, (1.0,) * 3, SDFNetwork.sdf_raw
    net = _small_net()
    want = sdf_lattice(net, lo, hi, (5, 6, 7))
    net.sdf_raw = lambda x: 2.0 * raw(net, x)
    assert torch.equal(sdf_lattice(net, lo, hi, (5, 6, 7)), 2.0 * want)
    monkeypatch.setattr(SDFNetwork, "sdf_raw", lambda net, x, count=None: 4.0 * raw(net, x, count))
    assert torch.equal(sdf_lattice(_small_net(), lo, hi, (5, 6, 7)), 4.0 * want)


@pytest.mark.parametrize("res,slab", [((9000, 3, 40), 1 << 12), ((40, 3, 9000), 1 << 12), ((300, 2, 41), 1)])
def test_lattice_memory_is_bounded(res, slab):
    """Rows along x and along z that no slab of slab_points holds: the values of the
    point-by-point query, in no more memory than it takes (its slabs' points and values,
    at most 16 bytes a point and as much again for the weights and the allocator's
    rounding), beside the lattice itself."""
    from supernormal_gb300.mesh import extract_fields, sdf_lattice

    net, lo, hi = _small_net(), (-1.0,) * 3, (1.0,) * 3
    want = extract_fields(lo, hi, res, net.sdf_raw, slab_points=slab)
    torch.cuda.synchronize()
    torch.cuda.reset_peak_memory_stats()
    before = torch.cuda.memory_allocated()
    got = sdf_lattice(net, lo, hi, res, negate=False, slab_points=slab)
    extra = torch.cuda.max_memory_allocated() - before - got.numel() * 4
    assert torch.equal(got, want)
    assert extra <= 2 * 16 * max(slab, res[1] * res[2]) + (1 << 16)


@pytest.mark.parametrize("n", [2_097_120, 2_097_153])
def test_lattice_store_of_long_rows(n):
    """Rows along z and along x up to and past 65,535 tiles of 32 points, the most that a
    grid's second axis holds."""
    from supernormal_gb300._lib import call, stream_handle

    for nx, ny, nz in ((2, 2, n), (n, 2, 2)):
        values = torch.rand(1, nz, nx, device="cuda")
        u = torch.zeros(nx, ny, nz, device="cuda")
        call("sn_lattice_store", 1, 1, nx, ny, nz, 1, values, u, stream_handle())
        assert torch.equal(u[:, 1], -values[0].T) and not u[:, 0].any()


@pytest.mark.parametrize("n", [2, 3, 31, 32, 33, 1023, 1024, 1025, 5000, 100_001])
@pytest.mark.parametrize("rows", [(2, 2), (3, 71), (300, 1001)])
def test_lattice_points_of_long_and_short_rows(n, rows):
    """Rows around the inner axis' pieces and the short rows' limit, few and many: every coordinate is its own
    multiple of 2^-10, exact in double and rounded once."""
    from supernormal_gb300._lib import call, stream_handle

    if n * rows[0] * rows[1] > 1 << 26:
        rows = (rows[0], 7)
    for name, shape, first, count in (("sn_lattice_points", (*rows, n), 1, rows[0] - 1),
                                      ("sn_lattice_points_x", (n, rows[1], rows[0]), 1, rows[1] - 1)):
        lo = np.array([-1.0, 0.5, 3.0])
        hi = lo + (np.array(shape) - 1) * 2.0**-10
        axes = [torch.as_tensor((lo[d] + np.arange(shape[d]) * 2.0**-10).astype(np.float32), device="cuda") for d in range(3)]
        if name == "sn_lattice_points":
            want = torch.cartesian_prod(axes[0][first:], axes[1], axes[2])
        else:
            want = torch.cartesian_prod(axes[1][first:], axes[2], axes[0])[:, [2, 0, 1]]
        x = torch.full((want.shape[0] + 64, 3), 7.0, device="cuda")
        call(name, first, count, *shape, lo.ctypes.data, hi.ctypes.data, x, stream_handle())
        assert torch.equal(x[:-64], want) and bool((x[-64:] == 7.0).all())
