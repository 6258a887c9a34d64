"""First calls on a non-blocking stream: buffers that a call has to get and
clear are ready before its kernels use them, whatever the stream."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.fixture
def side():
    """A non-blocking stream as the library's stream."""
    from fullc0ntact_gb300 import dem
    s = torch.cuda.Stream()
    s.wait_stream(torch.cuda.current_stream())
    dem.set_stream(s)
    with torch.cuda.stream(s):
        yield s
    dem.set_stream(None)
    s.synchronize()


def _sort(keys, vals, cells):
    from fullc0ntact_gb300 import dem
    from fullc0ntact_gb300.params import make_params
    P = make_params(len(keys), (2, 2, 2), 0.01)
    P.numCells = cells
    dem.set_parameters(P)
    k = torch.from_numpy(keys.view(np.int32)).cuda()
    v = torch.from_numpy(vals.view(np.int32)).cuda()
    dem.sort_particles(k, v, len(keys))
    dem.check("sortParticles")
    return k.cpu().numpy().view(np.uint32), v.cpu().numpy().view(np.uint32)


@pytest.mark.parametrize("cells", [2 ** 23, 2 ** 22, 5 * 2 ** 18, 2 ** 16 - 1])
def test_first_sort_of_a_cell_count_on_a_side_stream(side, cells):
    rng = np.random.default_rng(cells)
    n = 150_000
    keys = rng.integers(0, cells, n).astype(np.uint32)
    vals = rng.permutation(n).astype(np.uint32)
    o = np.argsort(keys, kind="stable")
    k, v = _sort(keys, vals, cells)
    np.testing.assert_array_equal(k, keys[o])
    np.testing.assert_array_equal(v, vals[o])


@pytest.mark.parametrize("grid", [(256, 256, 128), (32, 64, 128)])
def test_first_update_of_a_cell_count_on_a_side_stream(side, grid):
    from fullc0ntact_gb300 import dem, scenes
    sc = scenes.lattice_scene(30_000)
    sc["params"].gridSize[:] = grid
    sc["params"].numCells = grid[0] * grid[1] * grid[2]
    other = scenes.lattice_scene(2000)
    got = []
    for stream in (side, None):
        dem.set_stream(None)
        dem.DeviceScene(other).update(1)  # another cell count: the next call gets its buffers
        torch.cuda.synchronize()
        ds = dem.DeviceScene(sc)
        torch.cuda.synchronize()
        dem.set_stream(stream)
        ds.update(3)
        torch.cuda.synchronize()
        dem.check("update")
        got.append((ds.pos.cpu().numpy(), ds.vel.cpu().numpy()))
    dem.set_stream(side)
    np.testing.assert_array_equal(got[0][0], got[1][0])
    np.testing.assert_array_equal(got[0][1], got[1][1])


def test_maps_and_networks_made_on_a_side_stream(side):
    """A map's vertices and a network's weights and optimiser state are in place
    when the call that makes them returns."""
    from fullc0ntact_gb300 import dem, scenes, sdf
    m = dem.DistanceMap.torus(0.3, 0.1, 96, 0.05)
    v = m.vertices()
    mesh = dem.DistanceMap.from_mesh(*scenes.torus_mesh(0.3, 0.1, 48, 24), 48, 0.05).vertices()
    a = sdf.SdfNet(3, 64, 3, seed=5).get_params()
    dem.set_stream(None)
    np.testing.assert_array_equal(v, dem.DistanceMap.torus(0.3, 0.1, 96, 0.05).vertices())
    np.testing.assert_array_equal(
        mesh, dem.DistanceMap.from_mesh(*scenes.torus_mesh(0.3, 0.1, 48, 24), 48, 0.05).vertices())
    np.testing.assert_array_equal(a, sdf.SdfNet(3, 64, 3, seed=5).get_params())
    dem.set_stream(side)


def _cpu(keys, vals):
    o = np.argsort(keys, kind="stable")
    return keys[o], vals[o]


def test_sorts_of_alternating_cell_counts():
    """Two grids in one process, and sizes that grow and shrink between them."""
    rng = np.random.default_rng(17)
    for n, cells in [(3000, 2 ** 12), (70_000, 2 ** 20), (3000, 2 ** 20), (300_000, 2 ** 12),
                     (70_000, 2 ** 15), (300_000, 2 ** 20), (10, 2 ** 12), (300_000, 2 ** 12),
                     (300_001, 3 * 2 ** 18), (70_000, 2 ** 20), (5000, 1), (300_000, 2 ** 15)]:
        keys = rng.integers(0, cells, n).astype(np.uint32)
        vals = rng.permutation(n).astype(np.uint32)
        k, v = _sort(keys, vals, cells)
        rk, rv = _cpu(keys, vals)
        np.testing.assert_array_equal(k, rk)
        np.testing.assert_array_equal(v, rv)


@pytest.mark.parametrize("n", [4000, 60_000, 300_000])
@pytest.mark.parametrize("warm", [2 ** 19, 2 ** 14])
def test_captured_sort_outlives_sorts_of_other_cell_counts(side, n, warm):
    """A recorded sortParticles replays correctly after sorts with smaller and
    larger cell counts.  warm = 2^14: the key width is first met (or not) during
    the capture, after a warm-up call at another one."""
    from fullc0ntact_gb300 import dem
    from fullc0ntact_gb300.params import make_params
    cells = 2 ** 19 if n != 4000 else 2 ** 17
    rng = np.random.default_rng(n + warm)
    draw = lambda: (rng.integers(0, cells, n).astype(np.uint32), rng.permutation(n).astype(np.uint32))
    dev = lambda a: torch.from_numpy(a.view(np.int32)).cuda()
    warm = min(warm, cells)
    _sort(rng.integers(0, warm, n).astype(np.uint32), np.arange(n, dtype=np.uint32), warm)
    P = make_params(n, (2, 2, 2), 0.01)
    P.numCells = cells
    dem.set_parameters(P)
    keys, vals = draw()
    k, v = dev(keys), dev(vals)
    side.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g, stream=side):
        dem.sort_particles(k, v, n)
    for other in (2 ** 9, 2 ** 21, cells):
        ok, ov = rng.integers(0, other, n).astype(np.uint32), np.arange(n, dtype=np.uint32)
        gk, gv = _sort(ok, ov, other)
        np.testing.assert_array_equal(gv, _cpu(ok, ov)[1])
        keys, vals = draw()
        k.copy_(dev(keys))
        v.copy_(dev(vals))
        g.replay()
        side.synchronize()
        dem.check("replay")
        rk, rv = _cpu(keys, vals)
        np.testing.assert_array_equal(k.cpu().numpy().view(np.uint32), rk)
        np.testing.assert_array_equal(v.cpu().numpy().view(np.uint32), rv)
