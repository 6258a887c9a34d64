"""The collide kernels give bit-identical results: the per-thread kernel with
global reads, the kernel with shared-memory tiles staged by bulk copies, and
the kernel for crowded neighbourhoods, on scenes that exercise staged tiles,
multi-row tiles, x-wrapping windows, crowded cells, inert particles and the
polydisperse mode."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _run(sc, path, steps):
    from fullc0ntact_gb300 import dem
    dem.lib.fcdemSetCollidePath(path)
    try:
        ds = dem.DeviceScene(sc)
        ds.stages()
        if steps > 1:
            ds.update(steps - 1)
        dem.check("collide path %d" % path)
        return ds.pos.cpu().numpy(), ds.vel.cpu().numpy()
    finally:
        dem.lib.fcdemSetCollidePath(-1)


@pytest.mark.parametrize("case", ["packed", "lattice", "wrap", "random_poly", "sparse"])
def test_tiled_equals_global(case):
    from fullc0ntact_gb300 import scenes
    if case == "packed":
        sc = scenes.packed_scene(200_000, grid=128)
    elif case == "lattice":
        sc = scenes.lattice_scene(16384)
    elif case == "wrap":  # particles across the whole x range: windows wrap
        sc = scenes.random_box(30000, grid=(32, 32, 32), radius=1.0 / 32.0, seed=8)
    elif case == "random_poly":
        sc = scenes.random_box(30000, grid=(64, 64, 64), radius=1.0 / 64.0, seed=9, poly=True)
    else:  # few particles per row: many row groups per tile
        sc = scenes.random_box(3000, grid=(64, 64, 64), radius=1.0 / 64.0, seed=10)
    a = _run(sc, 0, 3)
    b = _run(sc, 1, 3)
    for x, y in zip(a, b):
        np.testing.assert_array_equal(x.view(np.uint32), y.view(np.uint32))


def _run_cull(sc, on, steps):
    from fullc0ntact_gb300 import dem
    dem.lib.fcdemSetCellCulling(int(on))
    try:
        ds = dem.DeviceScene(sc)
        ds.stages()
        if steps > 1:
            ds.update(steps - 1)
        dem.check("cell culling %d" % on)
        return ds.pos.cpu().numpy(), ds.vel.cpu().numpy()
    finally:
        dem.lib.fcdemSetCellCulling(1)


@pytest.mark.parametrize("case", ["packed", "lattice", "wrap", "random_poly", "small_grid"])
def test_cell_culling_is_exact(case):
    from fullc0ntact_gb300 import scenes
    if case == "packed":
        sc = scenes.packed_scene(200_000, grid=128)
    elif case == "lattice":
        sc = scenes.lattice_scene(16384)
    elif case == "wrap":
        sc = scenes.random_box(30000, grid=(32, 32, 32), radius=1.0 / 64.0, seed=8)
    elif case == "random_poly":  # particleRadius bounds the radii in w
        sc = scenes.random_box(30000, grid=(64, 64, 64), radius=1.0 / 64.0, seed=9, poly=True)
    else:  # grid too small for culling: it must switch itself off
        sc = scenes.random_box(2000, grid=(2, 4, 4), radius=0.1, cell=0.5, seed=11)
    a = _run_cull(sc, False, 4)
    b = _run_cull(sc, True, 4)
    for x, y in zip(a, b):
        np.testing.assert_array_equal(x.view(np.uint32), y.view(np.uint32))


def test_radius_bound_violation_is_reported():
    from fullc0ntact_gb300 import _native, dem, scenes
    sc = scenes.random_box(5000, grid=(64, 64, 64), radius=1.0 / 64.0, seed=12, poly=True)
    sc["pos"][17, 3] = 2.0 / 64.0  # above particleRadius
    ds = dem.DeviceScene(sc)
    ds.stages()
    with pytest.raises(_native.FcdemError, match="radius"):
        dem.check()


@pytest.mark.parametrize("n", [5000, 40_000])
def test_every_radius_out_of_bound_is_reported_after_each_clear(n):
    """A scene that reports from every warp and step: the error is there after
    each run, gone once read, and the states are those of the right bound."""
    from fullc0ntact_gb300 import dem, scenes
    sc = scenes.random_box(n, grid=(64, 64, 64), radius=1.0 / 64.0, seed=12, poly=True)
    right, broken = dem.DeviceScene(sc), dem.DeviceScene(sc)
    broken.params.particleRadius /= 4.0
    try:
        for steps in (1, 3):
            right.update(steps)
            assert dem.lib.fcdemGetLastError() == 0
            broken.update(steps)
            assert dem.lib.fcdemGetLastError() == 8  # FCDEM_ERR_RADIUS_BOUND
            assert dem.lib.fcdemGetLastError() == 0
            for a, b in ((right.pos, broken.pos), (right.vel, broken.vel)):
                np.testing.assert_array_equal(a.cpu().numpy(), b.cpu().numpy())
    finally:
        dem.set_radius_mode(False)


def _crowded_scene(kind):
    """Scenes with collapsed cells: thousands of particles in a few cells, the
    cells around them sparse or crowded too."""
    from fullc0ntact_gb300 import scenes
    if kind == "mono":
        sc = scenes.random_box(20000, grid=(16, 16, 16), radius=1.0 / 16.0, seed=21)
    elif kind == "poly":
        sc = scenes.random_box(20000, grid=(16, 16, 16), radius=1.0 / 16.0, seed=22, poly=True)
    else:  # packed polydisperse scene with three collapsed cells
        sc = scenes.packed_scene(100_000, grid=128)
    rng = np.random.default_rng(23)
    cell = float(sc["params"].cellSize[0])
    origin = np.array([sc["params"].worldOrigin[k] for k in range(3)], np.float32)
    n = sc["pos"].shape[0]
    picks = rng.permutation(n)
    start = 0
    for count, c in ((2500, (5, 5, 5)), (700, (6, 5, 5)), (300, (9, 9, 9)), (90, (12, 3, 7))):
        idx = picks[start:start + count]
        start += count
        lo = origin + np.array(c, np.float32) * cell
        sc["pos"][idx, :3] = lo + rng.uniform(0.05, 0.95, (count, 3)).astype(np.float32) * cell
    return sc


def _run_crowd(sc, on, steps, pipeline=1):
    from fullc0ntact_gb300 import dem
    dem.lib.fcdemSetCrowdPath(int(on))
    dem.lib.fcdemSetUpdatePipeline(pipeline)
    try:
        ds = dem.DeviceScene(sc)
        ds.stages()
        if steps > 1:
            ds.update(steps - 1)
        dem.check("crowd path %d" % on)
        return ds.pos.cpu().numpy(), ds.vel.cpu().numpy(), ds.hash.cpu().numpy()
    finally:
        dem.lib.fcdemSetCrowdPath(1)
        dem.lib.fcdemSetUpdatePipeline(1)


@pytest.mark.parametrize("kind", ["mono", "poly", "packed"])
@pytest.mark.parametrize("pipeline", [0, 1])
def test_crowd_path_is_exact(kind, pipeline):
    """The warp-per-group kernel for crowded neighbourhoods gives results
    bit-identical to the one-thread-per-particle kernel, through the
    reference-named stages and both fcdemUpdate pipelines."""
    sc = _crowded_scene(kind)
    a = _run_crowd(sc, True, 3, pipeline)
    b = _run_crowd(sc, False, 3, pipeline)
    for x, y in zip(a, b):
        np.testing.assert_array_equal(x.view(np.uint32), y.view(np.uint32))


def _inert_scene():
    """Packed polydisperse scene with particles that take part in no pair
    term: 3,000 with NaN positions (they share one cell, a crowded
    neighbourhood), 300 with one NaN coordinate, and 40 spheres of equal
    radius at one point (coincident: dist = 0, their normals are NaN)."""
    from fullc0ntact_gb300 import scenes
    sc = scenes.packed_scene(100_000, grid=128)
    rng = np.random.default_rng(31)
    picks = rng.permutation(sc["pos"].shape[0])
    sc["pos"][picks[:3000], :3] = np.float32(np.nan)
    for k, idx in enumerate(np.array_split(picks[3000:3300], 3)):
        sc["pos"][idx, k] = np.float32(np.nan)
    same = picks[3300:3340]
    sc["pos"][same, :3] = np.float32(0.25)
    sc["pos"][same, 3] = np.float32(sc["params"].particleRadius)
    sc["vel"][same, :3] = np.float32(0.0)  # still coincident after the integrate
    return sc


def test_inert_particles_match_oracle():
    """Particles with a NaN coordinate are skipped by collide (their force is
    +0.0 and they give their partners nothing); the oracle walks them like
    every other particle.  One update through the reference-named stages:
    hashes and order bit for bit, new velocities within the 1e-5 bar with
    NaN exactly where the oracle has NaN."""
    from fullc0ntact_gb300 import dem
    from oracle import oracle as O
    from fcdem_testutil import REL_TOL, force_floor, oracle_params, rel_err_vec
    sc = _inert_scene()
    ds = dem.DeviceScene(sc)
    ds.stages()
    dem.check("stages with inert particles")
    st = O.step_stages(oracle_params(bytes(sc["params"])), sc["pos"], sc["vel"], sc["dt"],
                       radius_from_w=True)
    np.testing.assert_array_equal(ds.hash.cpu().numpy().view(np.uint32), st["hash_sorted"])
    np.testing.assert_array_equal(ds.index.cpu().numpy().view(np.uint32), st["index_sorted"])
    out = ds.vel.cpu().numpy()
    np.testing.assert_array_equal(np.isnan(out[:, :3]), np.isnan(st["newVel"][:, :3]))
    assert int(np.isnan(out[:, 0]).sum()) >= 40  # the coincident spheres
    # a particle with a NaN coordinate keeps its velocity (force +0.0)
    inert = np.isnan(st["pos"][:, :3]).any(axis=1)
    assert int(inert.sum()) == 3300
    keep = st["vel_in"][inert, :3] + np.float32(0.0)
    np.testing.assert_array_equal(out[inert, :3].view(np.uint32), keep.view(np.uint32))
    f_ref = st["newVel"][:, :3].astype(np.float64) - st["vel_in"][:, :3]
    f_gpu = out[:, :3].astype(np.float64) - st["vel_in"][:, :3]
    assert rel_err_vec(out, st["newVel"], 1e-6).max() <= REL_TOL
    assert rel_err_vec(f_gpu, f_ref, force_floor(f_ref)).max() <= REL_TOL


@pytest.mark.parametrize("pipeline", [0, 1])
def test_inert_particles_identical_on_every_path(pipeline):
    """Five fused updates of the scene with inert particles: the crowded
    kernel (which skips chunks of inert partners) and the per-thread kernel
    give the same bits."""
    sc = _inert_scene()
    a = _run_crowd(sc, True, 5, pipeline)
    b = _run_crowd(sc, False, 5, pipeline)
    for x, y in zip(a, b):
        np.testing.assert_array_equal(x.view(np.uint32), y.view(np.uint32))


@pytest.mark.parametrize("limit", [128, 2048])
def test_crowd_limit_does_not_change_results(limit):
    """The neighbourhood size above which a particle goes to the crowded
    kernel (fcdemSetCrowdLimit) moves work between the two kernels only:
    three fused updates of the packed scene with crowded cells end in the
    same bits at the default limit (512) and at `limit`."""
    from fullc0ntact_gb300 import dem
    sc = _crowded_scene("packed")
    a = _run_crowd(sc, True, 3)
    dem.lib.fcdemSetCrowdLimit(limit)
    try:
        b = _run_crowd(sc, True, 3)
    finally:
        dem.lib.fcdemSetCrowdLimit(0)
    for x, y in zip(a, b):
        np.testing.assert_array_equal(x.view(np.uint32), y.view(np.uint32))



def test_collide_configurations_give_identical_results():
    """Three fused updates of the packed scene with collapsed cells under
    collide configurations that differ in crowd limit, persistent-grid width
    and row staging: the same bits as the default configuration."""
    from fullc0ntact_gb300 import dem
    sc = _crowded_scene("packed")
    dem.lib.fcdemSetCollideConfig(-1)
    ref = _run_crowd(sc, True, 3)
    try:
        for k in (0, 1, 7, 15, 22, 29):
            dem.lib.fcdemSetCollideConfig(k)
            got = _run_crowd(sc, True, 3)
            for x, y in zip(ref, got):
                np.testing.assert_array_equal(x.view(np.uint32), y.view(np.uint32))
    finally:
        dem.lib.fcdemSetCollideConfig(-1)


def test_collide_autotuner_keeps_the_state_and_the_results():
    """fcdemAutotuneCollide on the packed scene with collapsed cells: it returns
    a configuration index and a step time, puts pos and vel back as they were,
    and the next update under the chosen configuration gives the bits of the
    default one."""
    import torch
    from fullc0ntact_gb300 import dem
    sc = _crowded_scene("packed")
    ds = dem.DeviceScene(sc)
    pos0, vel0 = ds.pos.clone(), ds.vel.clone()
    k, ms = ds.autotune_collide()
    try:
        assert 0 <= k < 30 and ms > 0.0
        assert torch.equal(ds.pos.view(torch.int32), pos0.view(torch.int32))
        assert torch.equal(ds.vel.view(torch.int32), vel0.view(torch.int32))
        ds.update(2)
        dem.check("update after autotune")
        tuned = (ds.pos.cpu().numpy(), ds.vel.cpu().numpy())
    finally:
        dem.lib.fcdemSetCollideConfig(-1)
    ds2 = dem.DeviceScene(sc)
    ds2.update(2)
    dem.check("update, default configuration")
    for x, y in zip(tuned, (ds2.pos.cpu().numpy(), ds2.vel.cpu().numpy())):
        np.testing.assert_array_equal(x.view(np.uint32), y.view(np.uint32))


def _rows_scene(grid, n, poly, kind, many, seed):
    """Scenes at the edges of the row scan: `rows` puts n particles into one
    column of cells (rows of n candidates), `full` spreads them over the whole
    grid and past it, so that the first and last columns wrap.  many: 25,000
    more over the whole grid, above the size up to which nine lanes share a
    particle."""
    from fullc0ntact_gb300 import scenes
    radius = 1.0 / 64.0
    total = n + 25000 if many else n
    sc = scenes.random_box(total, grid=grid, radius=radius, seed=seed, cell=1.0 / 32.0, poly=poly)
    rng = np.random.default_rng(seed + 1)
    ext = np.array(grid) / 32.0
    sc["pos"][:, :3] = np.clip(-1.0 + rng.uniform(-0.02, 1.02, (total, 3)) * ext, -0.98, 0.98)
    if kind == "rows":
        sc["pos"][:n, 0] = rng.uniform(-0.5, -0.5 + 3.0 / 32.0, n)
        sc["pos"][:n, 1:3] = rng.uniform(-0.5, -0.5 + 1.0 / 32.0, (n, 2))
    return sc


@pytest.mark.parametrize("many", [False, True])
@pytest.mark.parametrize("poly", [False, True])
@pytest.mark.parametrize("grid,n,kind", [
    ((64, 64, 64), 1, "rows"), ((64, 64, 64), 3, "rows"), ((64, 64, 64), 4, "rows"),
    ((64, 64, 64), 5, "rows"), ((64, 64, 64), 31, "rows"), ((64, 64, 64), 33, "rows"),
    ((64, 64, 64), 129, "rows"), ((64, 64, 64), 255, "rows"), ((64, 64, 64), 256, "rows"),
    ((64, 64, 64), 700, "rows"), ((4, 4, 4), 300, "full"), ((4, 8, 16), 700, "full"),
    ((8, 2, 4), 200, "full"), ((2, 8, 8), 300, "full"), ((16, 16, 16), 4001, "full")])
def test_row_scan_edges_match_oracle(grid, n, kind, poly, many):
    """One thread per particle (the hit-mask scan and the general loop) and nine
    lanes per particle, on rows of 0 to 700 candidates, wrapped columns and
    aliased axes: bit-exact against the oracle, staged (cellStart/cellEnd) and
    fused (prefix table), with and without the crowded path."""
    from fullc0ntact_gb300 import dem
    from oracle import oracle as O
    sc = _rows_scene(grid, n, poly, kind, many, 100 + n)
    P = O.SimParams.from_buffer_copy(bytes(sc["params"]))
    with O.gpu_arithmetic():
        pos, vel = sc["pos"].copy(), sc["vel"].copy()
        O.update(P, pos, vel, sc["dt"], 1, poly)  # in place
    for crowd in (1, 0):
        dem.lib.fcdemSetCrowdPath(crowd)
        try:
            for fused in (False, True):
                ds = dem.DeviceScene(sc)
                ds.update(1) if fused else ds.stages()
                dem.check("row scan")
                for a, b in ((ds.pos, pos), (ds.vel, vel)):
                    np.testing.assert_array_equal(a.cpu().numpy(), b)
        finally:
            dem.lib.fcdemSetCrowdPath(1)
            dem.set_radius_mode(False)


@pytest.mark.parametrize("poly", [False, True])
@pytest.mark.parametrize("n", [6000, 40_000])
@pytest.mark.parametrize("grid", [(32, 32, 32), (8, 16, 32)])
def test_particles_moved_across_a_face_after_the_sort(grid, n, poly):
    """A staged host may move particles between calcHash and collide: the tables
    then list a particle in a neighbour of the cell that its position gives
    (every row and every part of a wrapped row).  It never meets itself there:
    bit-exact against the oracle, with one thread and with nine lanes per
    particle."""
    from fullc0ntact_gb300 import dem, scenes
    from oracle import oracle as O
    cell = 1.0 / 16.0
    sc = scenes.random_box(n, grid=grid, radius=1.0 / 64.0, seed=n + grid[0], cell=cell, poly=poly)
    rng = np.random.default_rng(5)
    pos, vel = sc["pos"], sc["vel"]
    pos[:, :3] = -1.0 + rng.uniform(0.0, 1.0, (n, 3)) * np.array(grid) * cell
    # a quarter of them just below a face on some axes, the world's edges among the
    # faces, then just above it (by less than the margin of the cell culling)
    some = rng.permutation(n)[: n // 4]
    axes = rng.random((len(some), 3)) < 0.5
    face = -1.0 + rng.integers(0, np.array(grid) + 1, (len(some), 3)) * cell
    step = rng.uniform(1e-7, 1e-6, (2, len(some), 3))
    moved = pos.copy()
    pos[some, :3] = np.where(axes, face - step[0], pos[some, :3])
    moved[some, :3] = np.where(axes, face + step[1], pos[some, :3])
    P = O.SimParams.from_buffer_copy(bytes(sc["params"]))
    with O.gpu_arithmetic():
        h, x = O.sort_pairs(*O.calc_hash(P, pos))
        cs, ce, sp, sv = O.reorder(h, x, moved, vel, P.numCells)
        want = O.collide(P, sp, sv, x, cs, ce, radius_from_w=poly)
    ds = dem.DeviceScene(sc)
    ds.activate()
    try:
        dem.calc_hash(ds.hash, ds.index, ds.pos, n)
        dem.sort_particles(ds.hash, ds.index, n)
        ds.pos.copy_(torch.from_numpy(moved))
        dem.reorder_data_and_find_cell_start(ds.cell_start, ds.cell_end, ds.sorted_pos,
                                             ds.sorted_vel, ds.hash, ds.index, ds.pos, ds.vel, n,
                                             ds.num_cells)
        out = torch.empty_like(ds.vel)
        dem.collide(out, ds.sorted_pos, ds.sorted_vel, ds.index, ds.cell_start, ds.cell_end, n,
                    ds.num_cells)
        dem.check("collide")
    finally:
        dem.set_radius_mode(False)
    assert np.isfinite(want).all()
    np.testing.assert_array_equal(out.cpu().numpy(), want)


@pytest.mark.parametrize("many", [0, 25_000])
def test_crowded_cell_whose_first_members_moved_away(many):
    """Members of a crowded cell that a staged host has moved across a face after
    the sort, the first of many of its groups of 32 among them: every particle
    gets its force, bit-exact against the oracle."""
    from fullc0ntact_gb300 import dem, scenes
    from oracle import oracle as O
    m, cell = 700, 1.0 / 16.0
    n = m + many
    sc = scenes.random_box(n, grid=(32, 32, 32), radius=1.0 / 64.0, seed=3, cell=cell)
    rng = np.random.default_rng(6)
    pos, vel = sc["pos"], sc["vel"]
    pos[m:, 0] = rng.uniform(0.0, 0.99, many)
    pos[:m, :3] = -0.5 + rng.uniform(0.01, 0.99, (m, 3)) * cell
    moved = pos.copy()
    for first, axis in ((0, 0), (5, 1), (7, 2)):
        some = np.arange(first, m, 8)
        pos[some, axis] = -0.5 + cell - rng.uniform(1e-7, 1e-6, len(some))
        moved[some, axis] = -0.5 + cell + rng.uniform(1e-7, 1e-6, len(some))
    P = O.SimParams.from_buffer_copy(bytes(sc["params"]))
    with O.gpu_arithmetic():
        h, x = O.sort_pairs(*O.calc_hash(P, pos))
        cs, ce, sp, sv = O.reorder(h, x, moved, vel, P.numCells)
        want = O.collide(P, sp, sv, x, cs, ce)
    ds = dem.DeviceScene(sc)
    ds.activate()
    dem.calc_hash(ds.hash, ds.index, ds.pos, n)
    dem.sort_particles(ds.hash, ds.index, n)
    ds.pos.copy_(torch.from_numpy(moved))
    dem.reorder_data_and_find_cell_start(ds.cell_start, ds.cell_end, ds.sorted_pos, ds.sorted_vel,
                                         ds.hash, ds.index, ds.pos, ds.vel, n, ds.num_cells)
    out = torch.full_like(ds.vel, float("nan"))
    dem.collide(out, ds.sorted_pos, ds.sorted_vel, ds.index, ds.cell_start, ds.cell_end, n,
                ds.num_cells)
    dem.check("collide")
    assert np.isfinite(want).all()
    np.testing.assert_array_equal(out.cpu().numpy(), want)


@pytest.mark.parametrize("poly", [False, True])
@pytest.mark.parametrize("extra", [0, 1])
def test_crowded_kernel_of_few_and_of_many_groups(extra, poly):
    """The largest scene of the form for few groups and the smallest of the other,
    many of its neighbourhoods crowded: the same bits as without the crowded path."""
    from fullc0ntact_gb300 import dem, scenes
    n = 3 * 256 * torch.cuda.get_device_properties(0).multi_processor_count + extra
    sc = scenes.random_box(n, grid=(64, 64, 64), radius=1.0 / 64.0, seed=1, cell=1.0 / 32.0, poly=poly)
    sc["pos"][:, :3] = np.random.default_rng(n).uniform(-0.3, -0.05, (n, 3))
    got = []
    for on in (1, 0):
        dem.lib.fcdemSetCrowdPath(on)
        try:
            ds = dem.DeviceScene(sc)
            ds.update(2)
            dem.check("update")
            got.append((ds.pos.cpu().numpy(), ds.vel.cpu().numpy()))
        finally:
            dem.lib.fcdemSetCrowdPath(1)
            dem.set_radius_mode(False)
    for a, b in zip(*got):
        np.testing.assert_array_equal(a.view(np.uint32), b.view(np.uint32))
