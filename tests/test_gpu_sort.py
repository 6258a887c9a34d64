"""sortParticles: the onesweep radix sort against a stable CPU sort, on the
key distributions the step produces and on edge cases."""
import ctypes

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _sort_gpu(keys, vals, num_cells):
    from fullc0ntact_gb300 import dem
    from fullc0ntact_gb300.params import make_params
    g = 1
    while g ** 3 < num_cells:
        g *= 2
    P = make_params(len(keys), (g, g, g), 0.01)
    P.numCells = num_cells
    dem.set_parameters(P)
    k = torch.from_numpy(keys.view(np.int32).copy()).cuda()
    v = torch.from_numpy(vals.view(np.int32).copy()).cuda()
    dem.sort_particles(k, v, len(keys))
    dem.check("sortParticles")
    return k.cpu().numpy().view(np.uint32), v.cpu().numpy().view(np.uint32)


def _sort_cpu(keys, vals):
    o = np.argsort(keys, kind="stable")
    return keys[o], vals[o]


@pytest.mark.parametrize("n,num_cells", [
    (2, 8), (3, 64), (255, 256), (256, 256), (257, 2 ** 18), (4095, 2 ** 18), (4096, 2 ** 18),
    (4097, 2 ** 18), (100_000, 2 ** 24), (1_000_003, 2 ** 24), (300_000, 2 ** 12),
    (70_000, 2 ** 30), (50_000, 2 ** 32 - 1)])
def test_random_keys(n, num_cells):
    rng = np.random.default_rng(n)
    keys = rng.integers(0, num_cells, n, dtype=np.uint64).astype(np.uint32)
    vals = rng.permutation(n).astype(np.uint32)
    k, v = _sort_gpu(keys, vals, num_cells)
    rk, rv = _sort_cpu(keys, vals)
    np.testing.assert_array_equal(k, rk)
    np.testing.assert_array_equal(v, rv)


@pytest.mark.parametrize("pattern", ["equal", "sorted", "reversed", "few", "blocks"])
def test_key_patterns(pattern):
    n, cells = 200_000, 2 ** 18
    rng = np.random.default_rng(5)
    if pattern == "equal":
        keys = np.full(n, 12345, np.uint32)
    elif pattern == "sorted":
        keys = np.sort(rng.integers(0, cells, n)).astype(np.uint32)
    elif pattern == "reversed":
        keys = np.sort(rng.integers(0, cells, n))[::-1].astype(np.uint32).copy()
    elif pattern == "few":
        keys = rng.choice(np.array([0, 7, 1 << 17, cells - 1], np.uint32), n)
    else:  # runs of identical keys, as cells of a sorted particle array
        keys = np.repeat(rng.integers(0, cells, n // 50), 50).astype(np.uint32)
    vals = np.arange(n, dtype=np.uint32)
    k, v = _sort_gpu(keys, vals, cells)
    rk, rv = _sort_cpu(keys, vals)
    np.testing.assert_array_equal(k, rk)
    np.testing.assert_array_equal(v, rv)


def test_key_above_grid_is_reported():
    from fullc0ntact_gb300 import _native
    keys = np.arange(1000, dtype=np.uint32)
    keys[500] = 1 << 20
    with pytest.raises(_native.FcdemError, match="key width"):
        _sort_gpu(keys, np.arange(1000, dtype=np.uint32), 4096)


def test_repeated_sorts_reuse_scratch():
    rng = np.random.default_rng(9)
    for n in [10_000, 500_000, 20_000, 500_000]:
        keys = rng.integers(0, 2 ** 24, n).astype(np.uint32)
        vals = np.arange(n, dtype=np.uint32)
        k, v = _sort_gpu(keys, vals, 2 ** 24)
        rk, rv = _sort_cpu(keys, vals)
        np.testing.assert_array_equal(v, rv)


@pytest.mark.parametrize("n", [5000, 300_001])
def test_every_pass_configuration_sorts_identically(n):
    from fullc0ntact_gb300 import dem
    lib = dem.lib
    count = lib.fcdemSetSortConfig(n, -1)
    assert count >= 2
    rng = np.random.default_rng(n + 1)
    keys = rng.integers(0, 2 ** 24, n).astype(np.uint32)
    vals = np.arange(n, dtype=np.uint32)
    rk, rv = _sort_cpu(keys, vals)
    try:
        for k in range(count):
            assert lib.fcdemSetSortConfig(n, k) == count
            gk, gv = _sort_gpu(keys, vals, 2 ** 24)
            np.testing.assert_array_equal(gk, rk)
            np.testing.assert_array_equal(gv, rv)
    finally:
        lib.fcdemSetSortConfig(n, -1)


def test_autotune_picks_a_configuration():
    import ctypes as C
    from fullc0ntact_gb300 import dem
    t = C.c_float()
    best = dem.lib.fcdemAutotuneSort(200_000, 2 ** 24, C.byref(t))
    dem.check("autotune")
    assert best >= 0 and t.value > 0.0
    keys = np.random.default_rng(3).integers(0, 2 ** 24, 200_000).astype(np.uint32)
    vals = np.arange(200_000, dtype=np.uint32)
    gk, gv = _sort_gpu(keys, vals, 2 ** 24)
    rk, rv = _sort_cpu(keys, vals)
    np.testing.assert_array_equal(gv, rv)
    dem.lib.fcdemSetSortConfig(200_000, -1)


def test_lookback_wait_that_runs_out_is_reported_and_recovers():
    """The look-back wait of the radix sort is bounded.  With a limit of zero
    rounds every tile after the first gives up at once: the sort records
    FCDEM_ERR_DEVICE_TIMEOUT, and its writes stay inside the arrays (a
    partial prefix is at most the true one; the guard words around the
    arrays are untouched).  With the default limit restored the next sort is
    correct."""
    from fullc0ntact_gb300 import dem
    from fullc0ntact_gb300.params import make_params
    lib = dem.lib
    n, cells, pad = 300_000, 2 ** 24, 4096  # 74 tiles of 4096 keys, 3 passes
    rng = np.random.default_rng(77)
    keys = rng.integers(0, cells, n).astype(np.uint32)
    vals = np.arange(n, dtype=np.uint32)
    P = make_params(n, (256, 256, 256), 0.01)
    dem.set_parameters(P)
    guard = -123456789
    kb = torch.full((n + 2 * pad,), guard, dtype=torch.int32, device="cuda")
    vb = torch.full((n + 2 * pad,), guard, dtype=torch.int32, device="cuda")
    kb[pad:pad + n] = torch.from_numpy(keys.view(np.int32)).cuda()
    vb[pad:pad + n] = torch.from_numpy(vals.view(np.int32)).cuda()
    assert lib.fcdemGetLastError() == 0
    try:
        lib.fcdemSetSortWaitLimit(0)
        lib.sortParticles(kb.data_ptr() + 4 * pad, vb.data_ptr() + 4 * pad, n)
        code = lib.fcdemGetLastError()
    finally:
        lib.fcdemSetSortWaitLimit(-1)
    assert code == 5, code  # FCDEM_ERR_DEVICE_TIMEOUT
    for b in (kb, vb):
        assert bool((b[:pad] == guard).all()) and bool((b[pad + n:] == guard).all())
    k, v = _sort_gpu(keys, vals, cells)  # the context still works
    rk, rv = _sort_cpu(keys, vals)
    np.testing.assert_array_equal(k, rk)
    np.testing.assert_array_equal(v, rv)


@pytest.mark.parametrize("cells", [1, 2, 4096, 2 ** 18, 3 * 2 ** 17, 2 ** 24, 2 ** 25])
@pytest.mark.parametrize("n", [2, 255, 257, 1024, 1025, 4096, 262_144, 262_145, 2 ** 21, 2 ** 21 + 1])
def test_counting_and_radix_sort_agree(n, cells):
    """sortParticles by default (the counting sort up to its bounds) against the
    CPU's stable sort: sizes around its blocks, its large cells and its
    bounds; uniform keys, one cell for all, and a few crowded cells; values
    that are no permutation.  A forced configuration (the radix sort) gives
    the same arrays."""
    from fullc0ntact_gb300 import dem
    rng = np.random.default_rng(n + cells)
    vals = rng.integers(0, 2 ** 32, n, dtype=np.uint64).astype(np.uint32)
    kinds = [rng.integers(0, cells, n), np.full(n, cells - 1)]
    if n <= 300_000:
        kinds.append(np.where(rng.random(n) < 0.7, rng.integers(0, min(cells, 3), n),
                              rng.integers(0, cells, n)))
    for keys in kinds:
        keys = keys.astype(np.uint32)
        rk, rv = _sort_cpu(keys, vals)
        k, v = _sort_gpu(keys, vals, cells)
        np.testing.assert_array_equal(k, rk)
        np.testing.assert_array_equal(v, rv)
    try:
        dem.lib.fcdemSetSortConfig(n, 0)
        k, v = _sort_gpu(keys, vals, cells)
    finally:
        dem.lib.fcdemSetSortConfig(n, -1)
    np.testing.assert_array_equal(k, rk)
    np.testing.assert_array_equal(v, rv)


@pytest.mark.parametrize("n,cells", [(200_000, 64), (60_000, 4), (300_000, 2 ** 12), (3000, 2),
                                     (100_000, 2 ** 9)])
def test_keys_above_the_width_are_kept(n, cells):
    """Keys with bits above the sorted width are reported, and the pairs come back
    whole, in stable order of their low bits, however large their cells are.
    (The radix sort takes whole bytes of the key: its pairs are whole too.)"""
    from fullc0ntact_gb300 import dem
    from fullc0ntact_gb300.params import make_params
    rng = np.random.default_rng(n)
    keys = rng.integers(0, 2 ** 32, n, dtype=np.uint64).astype(np.uint32)
    if cells == 2 ** 12:  # sparse members of crowded cells among many small ones
        keys = np.where(rng.random(n) < 0.2, keys & np.uint32(0xfff0001f), keys)
    vals = rng.integers(0, 2 ** 32, n, dtype=np.uint64).astype(np.uint32)
    P = make_params(n, (2, 2, 2), 0.01)
    P.numCells = cells
    dem.set_parameters(P)
    width = (cells - 1).bit_length()
    whole = 8 * -(-width // 8)  # the radix sort's bits
    for config in (-1, 0):  # the default and the radix sort
        dem.lib.fcdemSetSortConfig(n, config)
        try:
            k = torch.from_numpy(keys.view(np.int32).copy()).cuda()
            v = torch.from_numpy(vals.view(np.int32).copy()).cuda()
            dem.sort_particles(k, v, n)
            assert dem.lib.fcdemGetLastError() == 6  # FCDEM_ERR_KEY_RANGE
        finally:
            dem.lib.fcdemSetSortConfig(n, -1)
        got = k.cpu().numpy().view(np.uint32), v.cpu().numpy().view(np.uint32)
        orders = [np.argsort(keys & np.uint32((1 << bits) - 1), kind="stable")
                  for bits in ((width, whole) if config < 0 else (whole,))]
        assert any(np.array_equal(got[0], keys[o]) and np.array_equal(got[1], vals[o])
                   for o in orders)


def _launches(n, cells):
    """Kernel launches of one sortParticles of n pairs below cells."""
    from fullc0ntact_gb300 import dem
    dem.lib.fcdemGetLaunchCount.restype = ctypes.c_ulonglong
    keys = np.random.default_rng(n).integers(0, cells, n).astype(np.uint32)
    _sort_gpu(keys, np.arange(n, dtype=np.uint32), cells)  # (buffers)
    before = dem.lib.fcdemGetLaunchCount()
    _sort_gpu(keys, np.arange(n, dtype=np.uint32), cells)
    return dem.lib.fcdemGetLaunchCount() - before


@pytest.mark.parametrize("n,cells", [(200_000, 2 ** 24), (200_000, 2 ** 30), (2 ** 21 + 5, 2 ** 24)])
def test_autotuned_index_names_the_kept_sort(n, cells):
    """Setting the index that the tuner returned changes nothing, and a tuning
    run leaves other key widths of the size class alone."""
    from fullc0ntact_gb300 import dem
    lib = dem.lib
    shapes = lib.fcdemSetSortConfig(n, -1)
    default = _launches(n, 2 ** 20)
    counted = _launches(n, cells) == _launches(n, 2 ** 20) and n <= 2 ** 21
    try:
        t = ctypes.c_float()
        best = lib.fcdemAutotuneSort(n, cells, ctypes.byref(t))
        dem.check("autotune")
        assert 0 <= best <= shapes and (best < shapes or (counted and cells <= 2 ** 24))
        kept = _launches(n, cells)
        assert _launches(n, 2 ** 20) == default
        assert lib.fcdemSetSortConfig(n, best) == shapes
        assert _launches(n, cells) == kept
    finally:
        lib.fcdemSetSortConfig(n, -1)


@pytest.mark.parametrize("n,cells", [(3000, 64), (4096, 2 ** 20), (4097, 256), (5000, 2 ** 13),
                                     (155_649, 2 ** 13), (300_001, 3 * 2 ** 18),
                                     (2 ** 21 - 1, 2 ** 16), (2 ** 21, 2 ** 24)])
def test_crowded_cells(n, cells):
    """Cells on both sides of the sizes at which another kernel takes their pairs
    (1,024 and n / 256 pairs), several of them, and cells of a few hundred, in
    random order and in runs, against the CPU's stable sort."""
    rng = np.random.default_rng(n + cells)
    giant = max(-(-n // 256), 1025)
    kinds = {
        "one cell": np.full(n, cells - 1),
        "half in one": np.where(rng.random(n) < 0.5, 7, rng.integers(0, cells, n)),
        "three cells": rng.integers(0, 3, n) * (cells // 3),
        "256 each": rng.integers(0, max(1, n // 256), n) % cells,
        "257 each, in runs": (np.arange(n) // 257) % cells,
        "as many giants as there can be": np.minimum(rng.permutation(n) // giant, cells - 1),
    }
    for members in {1024, 1025, giant - 1, giant, giant + 1}:
        k = rng.integers(1, cells, n)
        k[rng.permutation(n)[: min(members, n)]] = 0
        kinds[f"a cell of {members}"] = k
    vals = rng.integers(0, 2 ** 32, n, dtype=np.uint64).astype(np.uint32)
    for name, keys in kinds.items():
        keys = keys.astype(np.uint32)
        k, v = _sort_gpu(keys, vals, cells)
        rk, rv = _sort_cpu(keys, vals)
        np.testing.assert_array_equal(k, rk, err_msg=name)
        np.testing.assert_array_equal(v, rv, err_msg=name)
