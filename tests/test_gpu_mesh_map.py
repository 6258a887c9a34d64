"""The GPU triangle-mesh distance map (fcdemDistMapFromMesh): at every vertex
of a coarse torus mesh's map, the FP64 oracle's signed distance and closest
point; the config-2 mesh (256 x 64 quads) on the 128-cell map agrees with the
exact torus map within the faceting error."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_mesh_map_matches_fp64_oracle():
    from fullc0ntact_gb300 import dem, scenes
    from oracle import mesh_oracle as mo
    from oracle import oracle as O
    verts, tris = scenes.torus_mesh(0.3, 0.1, 24, 10)
    m = dem.DistanceMap.from_mesh(verts, tris, 24, 0.05)
    v = m.vertices()
    coords = O.lattice_coords(m.vmin, m.cell_size, m.cells).astype(np.float64)
    d, cp = mo.mesh_distance(coords, verts, tris)
    assert np.abs(v[:, 0] - d).max() <= 2e-6
    assert np.all(np.sign(v[np.abs(d) > 1e-5, 0]) == np.sign(d[np.abs(d) > 1e-5]))
    # the contact point is a closest point: |vertex - cp| = |distance|
    gcp = v[:, 1:].astype(np.float64)
    assert np.abs(np.linalg.norm(coords - gcp, axis=1) - np.abs(d)).max() <= 2e-6
    # and lies on the mesh (where several triangles are equally close -- the
    # symmetry planes of the lattice -- it may be another one than the
    # oracle's)
    on, _ = mo.mesh_distance(gcp, verts, tris)
    assert np.abs(on).max() <= 2e-6


def test_torus_mesh_map_matches_exact_torus():
    from fullc0ntact_gb300 import dem, scenes
    R, r = 0.3, 0.1
    verts, tris = scenes.torus_mesh(R, r, 256, 64)
    m = dem.DistanceMap.from_mesh(verts, tris, 128, 0.05)
    t = dem.DistanceMap.torus(R, r, 128, 0.05)
    assert np.allclose(m.vmin, t.vmin, atol=1e-6) and np.allclose(m.vmax, t.vmax, atol=1e-6)
    vm, vt = m.vertices(), t.vertices()
    facet = r * (1 - np.cos(np.pi / 64)) + (R + r) * (1 - np.cos(np.pi / 256))
    assert np.abs(vm[:, 0] - vt[:, 0]).max() <= facet + 1e-5
    far = np.abs(vt[:, 0]) > 2 * facet
    assert np.all(np.sign(vm[far, 0]) == np.sign(vt[far, 0]))


@pytest.mark.parametrize("form", ["closed", "shuffled", "unwelded", "open"])
@pytest.mark.parametrize("nu,nv,cells", [(3, 5, 9), (4, 4, 13), (3, 11, 16), (32, 17, 21)])
def test_mesh_map_forms_match_fp64_oracle(nu, nv, cells, form):
    """Cluster remainders (30, 32, 66 and 1,088 triangles), lattices that are no
    multiple of a brick, triangle order, vertices given once per triangle, and
    a mesh with a boundary: distance, closest point and winding-number sign."""
    from fullc0ntact_gb300 import dem, scenes
    from oracle import mesh_oracle as mo
    from oracle import oracle as O
    verts, tris = scenes.torus_mesh(0.3, 0.1, nu, nv)
    rng = np.random.default_rng(nu * 100 + nv)
    if form == "open":
        tris = tris[: len(tris) * 2 // 3]
    elif form != "closed":
        tris = rng.permutation(tris)
    if form == "unwelded":
        verts, tris = verts[tris.reshape(-1)], np.arange(tris.size, dtype=np.uint32).reshape(-1, 3)
    m = dem.DistanceMap.from_mesh(verts, tris, cells, 0.05)
    v = m.vertices()
    coords = O.lattice_coords(m.vmin, m.cell_size, m.cells).astype(np.float64)
    d, _ = mo.mesh_distance(coords, verts, tris)
    assert np.abs(np.abs(v[:, 0]) - np.abs(d)).max() <= 2e-6
    V = verts.astype(np.float64)
    wind = mo.winding_number(coords, V[tris[:, 0]], V[tris[:, 1]], V[tris[:, 2]])
    sure = (np.abs(d) > 1e-5) & (np.abs(wind - 0.5) > 1e-3)
    assert np.all((v[sure, 0] < 0) == (wind[sure] > 0.5))
    gcp = v[:, 1:].astype(np.float64)
    assert np.abs(np.linalg.norm(coords - gcp, axis=1) - np.abs(d)).max() <= 2e-6
    on, _ = mo.mesh_distance(gcp, verts, tris)
    assert np.abs(on).max() <= 2e-6


@pytest.mark.parametrize("cells", [12, 44, 80])
@pytest.mark.parametrize("nu,nv", [(3, 3), (8, 8), (13, 5), (16, 16), (43, 6)])
def test_meshes_of_few_triangles(nu, nv, cells):
    """18, 128, 130, 512 and 516 triangles on lattices below and above 65,536
    vertices, closed and with a boundary: both kernels' maps against the FP64
    oracle at a sample of the vertices."""
    from fullc0ntact_gb300 import dem, scenes
    from oracle import mesh_oracle as mo
    from oracle import oracle as O
    verts, tris = scenes.torus_mesh(0.3, 0.1, nu, nv)
    for part in (len(tris), len(tris) - 2):
        m = dem.DistanceMap.from_mesh(verts, tris[:part], cells, 0.05)
        dem.check("mesh map")
        coords = O.lattice_coords(m.vmin, m.cell_size, m.cells).astype(np.float64)
        pick = np.random.default_rng(nu).permutation(len(coords))[:4000]
        v, x = m.vertices()[pick], coords[pick]
        d, _ = mo.mesh_distance(x, verts, tris[:part])
        assert np.abs(np.abs(v[:, 0]) - np.abs(d)).max() <= 2e-6
        V = verts.astype(np.float64)[tris[:part]]
        wind = mo.winding_number(x, V[:, 0], V[:, 1], V[:, 2])
        sure = (np.abs(d) > 1e-5) & (np.abs(wind - 0.5) > 1e-3)
        assert np.all((v[sure, 0] < 0) == (wind[sure] > 0.5))
        gap = np.linalg.norm(x - v[:, 1:].astype(np.float64), axis=1) - np.abs(d)
        assert np.abs(gap).max() <= 2e-6


def test_mesh_map_that_leaves_no_room_for_its_roots():
    """Device memory for the map and less than the sign roots' list beside it: the
    same map, every vertex's sign from its own solid angles."""
    import torch
    from fullc0ntact_gb300 import dem, scenes
    verts, tris = scenes.torus_mesh(0.3, 0.1, 24, 10)
    cells = 240
    dem.DistanceMap.from_mesh(verts, tris[: len(tris) * 2 // 3], 24, 0.05)  # loads both ways' kernels
    want = dem.DistanceMap.from_mesh(verts, tris, cells, 0.05).vertices()
    nv = want.shape[0]  # 16 bytes a vertex for the map, 13 for the list and the distances
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    free, _ = torch.cuda.mem_get_info()
    hog = torch.empty(free - nv * 16 - nv * 7, dtype=torch.uint8, device="cuda")
    try:
        if torch.cuda.mem_get_info()[0] >= nv * 29:
            pytest.skip("another process gave memory back")
        m = dem.DistanceMap.from_mesh(verts, tris, cells, 0.05)
        dem.check("mesh map")
        got = m.vertices()
    finally:
        del hog
        torch.cuda.empty_cache()
    np.testing.assert_array_equal(np.abs(got), np.abs(want))
    sure = np.abs(want[:, 0]) > 1e-5
    np.testing.assert_array_equal(got[sure], want[sure])
