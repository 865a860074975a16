"""Which insertion kernel a call takes: a pinned id's own kernel at every size,
the default by mode, size and slices; and the kernels that the defaults reach
only at large sizes against the oracle there.

Tolerance of the latter as for the other insertion tests: the taps are the
oracle's, so only the order of FP32 additions differs (2e-6 for the at most
~1e3 additions of a cell here)."""
from __future__ import annotations

import numpy as np
import pytest

from oracle import oracle

PLANE, PIXEL, SCATTER = 5, 6, -2
MODES = ["nearest_neighbor", "gauss_2", "gauss_5", "trilinear"]
RTOL = 2e-6


@pytest.mark.parametrize("mode", MODES)
def test_pinned_ids_run_their_kernel(mode):
    from eman2_b200.batch import insertion_kernel, set_tile
    for N in (16, 384, 700):
        for tile in (0, 3, 4, PLANE, PIXEL):
            want = {("gauss_5", PIXEL): PLANE, ("nearest_neighbor", PLANE): PIXEL}.get((mode, tile), tile)
            set_tile(N, mode, 4, tile)
            try:
                assert insertion_kernel(N, mode, 4, 100) == want
                assert insertion_kernel(N, mode, 4, 3, "gather") == want
            finally:
                set_tile(N, mode, 4, -1)


@pytest.mark.parametrize("mode,N,nsym,n,kernel", [
    ("gauss_5", 1000, 14, 30, PLANE), ("gauss_2", 432, 14, 40, PLANE),
    ("gauss_2", 434, 14, 15, PLANE), ("gauss_2", 434, 14, 16, PIXEL),
    ("gauss_2", 480, 14, 45, PIXEL), ("gauss_2", 480, 14, 46, PLANE),
    ("gauss_2", 640, 1, 2048, PLANE), ("trilinear", 400, 14, 500, PLANE),
    ("trilinear", 402, 14, 14, PLANE), ("trilinear", 402, 14, 15, PIXEL),
    ("trilinear", 640, 14, 500, PIXEL), ("nearest_neighbor", 96, 1, 500, PIXEL)])
def test_default_kernel(mode, N, nsym, n, kernel):
    from eman2_b200.batch import insertion_kernel
    assert insertion_kernel(N, mode, nsym, n, "gather") == kernel


def test_scatter_kernel():
    from eman2_b200.batch import insertion_kernel
    assert insertion_kernel(96, "gauss_2", 1, 63) == SCATTER
    assert insertion_kernel(96, "gauss_2", 1, 64) == PLANE
    assert insertion_kernel(384, "gauss_2", 14, 1) == PLANE
    assert insertion_kernel(96, "gauss_5", 1, 1) == PLANE
    assert insertion_kernel(384, "nearest_neighbor", 1, 1) == SCATTER


def _inputs(N, n):
    from eman2_b200.synth import quaternion_blocks, random_quaternions
    rng = np.random.default_rng(N)
    return (rng.normal(size=(n, N, N + 2)).astype(np.float32),
            quaternion_blocks(random_quaternions(n, rng)),
            rng.uniform(0.5, 1.0, n).astype(np.float32))


def _recon(N, mode, sym):
    from eman2_b200 import Reconstructors
    r = Reconstructors.get("fourier", {"size": [N] * 3, "sym": sym, "mode": mode})
    r.setup()
    return r


@pytest.mark.gpu
@pytest.mark.parametrize("mode", ["gauss_2", "trilinear"])
def test_a_pinned_kernel_is_the_one_launched(gpu, mode):
    """Few slices: the compositions and the plane columns are two launches; the
    pixel-major kernel has one to clear its counter before it and one for the
    face taps after it."""
    import ctypes

    from eman2_b200 import _lib
    from eman2_b200.batch import set_tile
    N, n = 40, 12
    sl, rots, w = _inputs(N, n)
    launches = {}
    for tile in (PLANE, PIXEL):
        r = _recon(N, mode, "c1")
        set_tile(N, mode, 1, tile)
        try:
            st = _lib.fr_stats()
            _lib.check(_lib.load().fr_stats_reset())
            r.insert_slices(sl, rots, w, schedule="gather")
            _lib.check(_lib.load().fr_stats_get(ctypes.byref(st)))
        finally:
            set_tile(N, mode, 1, -1)
        launches[tile] = st.kernel_launches
    assert launches == {PLANE: 2, PIXEL: 4}


@pytest.mark.gpu
@pytest.mark.parametrize("mode,missing", [("gauss_2", None), ("trilinear", None), ("gauss_5", 6),
                                          ("nearest_neighbor", 5)])
def test_autotune_times_each_kernel_once(gpu, mode, missing):
    from eman2_b200.batch import TILE_NAMES, autotune, set_tile
    _, ms = autotune(32, mode, 1, nparticles=64)
    set_tile(32, mode, 1, -1)
    assert [k for k, v in ms.items() if v < 0] == ([TILE_NAMES[missing]] if missing else [])


@pytest.mark.gpu
@pytest.mark.parametrize("mode,N,sym,n,kernel", [
    ("trilinear", 402, "d2", 60, PIXEL), ("gauss_2", 434, "c3", 80, PIXEL),
    ("gauss_2", 434, "d3", 97, PLANE), ("trilinear", 384, "c4", 130, PLANE)])
def test_default_kernels_at_large_sizes(gpu, mode, N, sym, n, kernel):
    """Beyond the sizes of the other insertion tests: the pixel-major kernel, and
    the plane columns through a partial volume of 4 N / 3 slices or more."""
    from eman2_b200.batch import insertion_kernel
    nsym = len(oracle.sym_ops(sym))
    assert insertion_kernel(N, mode, nsym, n, "gather") == kernel
    sl, rots, w = _inputs(N, n)
    r = _recon(N, mode, sym)
    r.insert_slices(sl, rots, w, schedule="gather")
    d, nm = r.get_accumulators()
    o = oracle.OracleVolume(N, "fp32acc64")
    o.insert(sl, rots, w, mode, sym)
    assert np.array_equal(nm != 0, o.norm != 0)
    assert oracle.rel_l2(nm, o.norm) < RTOL and oracle.rel_l2(d, o.data) < RTOL


def test_bench_names_the_kernel_that_runs():
    import bench
    c4, g2 = bench.WORKLOADS["c4"], bench.WORKLOADS["c4g2"]
    assert bench.insertion_kernel_name(c4, 2048) == "k_plane"
    assert bench.insertion_kernel_name(g2, 2048) == "k_plane"
    assert bench.insertion_kernel_name(g2, 1, "scatter") == "k_plane"    # 14 slices of 384^2
    assert bench.insertion_kernel_name(dict(g2, N=96, sym="c1"), 1, "scatter") == "k_scatter"
    assert bench.update_roof_of("k_plane", "gauss_5") is None
    assert bench.update_roof_of("k_plane", "gauss_2") == "smem_rmw"
