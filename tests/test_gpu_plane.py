"""The plane-column insertion kernel where its geometry can go wrong: volumes
of a few cells, planes along the axes and the diagonals, the square pixel set,
matrices that are not rotations, and slice counts on either side of its
workspaces' limits (centre copies from 16 slices, the partial volume from
max(256, 8N/3), turns of 2048).

Tolerance: the taps are the oracle's, so only the order of FP32 additions
differs: a cell's sum is within n eps / 2 of the FP64 sum of n taps in the worst
case and sqrt(n) eps / 2 in the mean, below 2e-6 for the at most ~1e3 additions
of a chain here."""
from __future__ import annotations

import numpy as np
import pytest

from oracle import oracle

pytestmark = pytest.mark.gpu
RTOL = 2e-6


def _rotations(n, seed):
    from eman2_b200.synth import quaternion_blocks, random_quaternions
    r = quaternion_blocks(random_quaternions(n, np.random.default_rng(seed)))
    c, s = np.cos(np.pi / 4), np.sin(np.pi / 4)
    fixed = [np.eye(3), np.eye(3)[[1, 2, 0]], np.eye(3)[[2, 0, 1]], np.diag([-1.0, 1, -1]),
             [[c, s, 0], [-s, c, 0], [0, 0, 1]], [[1, 0, 0], [0, c, s], [0, -s, c]],
             [[c, 0, -s], [0, 1, 0], [s, 0, c]], [[1, 1e-4, 0], [-1e-4, 1, 0], [0, 0, 1]]]
    k = min(n, len(fixed))
    r[:k] = np.asarray(fixed[:k], np.float32)
    return r


def _check(N, mode, sym, rots, corners=False, seed=0, schedule="auto"):
    from eman2_b200 import Reconstructors
    n = len(rots)
    rng = np.random.default_rng(seed)
    sl = rng.normal(size=(n, N, N + 2)).astype(np.float32)
    w = rng.uniform(0.5, 1.0, n).astype(np.float32)
    r = Reconstructors.get("fourier", {"size": [N] * 3, "sym": sym, "mode": mode,
                                       "corners": corners})
    r.setup()
    r.insert_slices(sl, rots, w, schedule=schedule)
    d, nm = r.get_accumulators()
    o = oracle.OracleVolume(N, "fp32acc64")
    o.insert(sl, rots, w, mode, sym, corners=corners)
    assert np.array_equal(nm != 0, o.norm != 0)
    m = o.norm != 0
    assert np.max(np.abs(nm[m] - o.norm[m]) / o.norm[m]) < 1e-4
    assert oracle.rel_l2(nm, o.norm) < RTOL and oracle.rel_l2(d, o.data) < RTOL


@pytest.mark.parametrize("mode", ["gauss_2", "gauss_5", "trilinear"])
@pytest.mark.parametrize("N,n,sym", [(4, 20, "c1"), (6, 20, "c1"), (10, 12, "d2"), (34, 17, "c3"),
                                     (50, 8, "tet"), (96, 257, "c1"), (48, 300, "d4")])
def test_plane_matches_oracle(gpu, mode, N, n, sym):
    _check(N, mode, sym, _rotations(n, N + n))


@pytest.mark.parametrize("mode", ["gauss_2", "gauss_5", "trilinear"])
def test_plane_square_pixel_set(gpu, mode):
    _check(20, mode, "c2", _rotations(40, 3), corners=True)


@pytest.mark.parametrize("mode", ["gauss_2", "gauss_5", "trilinear"])
def test_plane_other_matrices(gpu, mode):
    """Scaled, sheared and flat matrices among rotations: every one inserted
    as the scatter schedule of a per-tap inserter would."""
    r = _rotations(300, 5)
    r[40] *= 0.7
    r[41] *= 1.3
    r[42][1] = r[42][0]
    r[43] = 0
    r[44][0] += 0.2 * r[44][1]
    r[45] *= 1.004
    _check(40, mode, "c1", r, schedule="gather")


@pytest.mark.parametrize("mode", ["gauss_2", "trilinear"])
@pytest.mark.parametrize("N,n,sym", [(4, 70, "c1"), (6, 64, "c1"), (10, 40, "d2"), (34, 64, "c1"),
                                     (50, 8, "tet")])
def test_small_volumes_of_many_slices(gpu, mode, N, n, sym):
    """Enough slices that the two-tap windows take the plane columns too."""
    from eman2_b200.batch import insertion_kernel
    assert insertion_kernel(N, mode, len(oracle.sym_ops(sym)), n) == 5
    _check(N, mode, sym, _rotations(n, N + n))


@pytest.mark.parametrize("mode", ["gauss_2", "gauss_5", "trilinear"])
def test_small_volumes_in_one_launch(gpu, mode):
    """Uneven jobs of few slices each, as segments of one launch.  Against the
    oracle through its own preparation: 2e-5, as for the other FFT paths."""
    from eman2_b200.batch import BatchReconstructor
    from eman2_b200.particles import particle_meta
    shapes = [(4, 1, "c1"), (6, 20, "c1"), (10, 3, "d2"), (34, 17, "c3"), (50, 2, "tet")]
    b = BatchReconstructor([{"size": [N] * 3, "sym": sym, "mode": mode} for N, _, sym in shapes])
    images, metas, parts = [], [], []
    for N, n, sym in shapes:
        rng = np.random.default_rng(N)
        img = rng.normal(size=(n, N, N)).astype(np.float32)
        rots, w = _rotations(n, N), rng.uniform(0.5, 1.0, n).astype(np.float32)
        shifts = rng.uniform(-1, 1, (n, 2)).astype(np.float32)
        images.append(img)
        metas.append(particle_meta(rots, shifts, w))
        parts.append((img, rots, shifts, w))
    b.insert_particles(images, metas)
    for j, ((N, n, sym), (img, rots, shifts, w)) in enumerate(zip(shapes, parts)):
        sl = np.stack([oracle.particle_to_slice(img[i], N, shifts[i], {}) for i in range(n)])
        o = oracle.OracleVolume(N, "fp32acc64")
        o.insert(sl, rots, w, mode, sym)
        d, nm = b.get_accumulators(j)
        assert np.array_equal(nm != 0, o.norm != 0)
        assert oracle.rel_l2(nm, o.norm) < RTOL and oracle.rel_l2(d, o.data) < 2e-5
    b.close()


@pytest.mark.parametrize("tile", [5, 6, -2])
@pytest.mark.parametrize("mode", ["gauss_2", "trilinear"])
def test_matrices_of_no_numbers(gpu, mode, tile):
    """Slices whose first rows hold a NaN or are scaled beyond the integers end
    inside the kernels' tables and volumes: the call returns, and away from the
    origin, where the NaN coordinates' taps go, the sums are the others'."""
    from eman2_b200 import Reconstructors, _lib
    from eman2_b200.batch import set_tile
    N, n = 40, 60
    rng = np.random.default_rng(8)
    sl = rng.normal(size=(n, N, N + 2)).astype(np.float32)
    w = np.ones(n, np.float32)
    rots = _rotations(n, 9)
    bad = rots.copy()
    bad[20, 0, 1] = np.nan
    bad[30, 1, 0] = np.nan
    bad[40, :2] *= 1e9
    bad[50, :2] *= 1e12
    bad[55, 0] = np.inf
    o = oracle.OracleVolume(N, "fp32acc64")
    keep = np.setdiff1d(np.arange(n), [20, 30, 40, 50, 55])
    o.insert(sl[keep], rots[keep], w[keep], mode, "c1")
    r = Reconstructors.get("fourier", {"size": [N] * 3, "sym": "c1", "mode": mode})
    r.setup()
    set_tile(N, mode, 1, tile)
    try:
        r.insert_slices(sl, bad, w, schedule="scatter" if tile == -2 else "gather")
        d, nm = r.get_accumulators()
    finally:
        set_tile(N, mode, 1, -1)
    far = np.ones(nm.shape, bool)
    near = np.r_[0:3, N - 2:N]
    far[np.ix_(near, near, [0, 1, 2])] = False
    assert np.isfinite(nm[far]).all()
    assert oracle.rel_l2(nm[far], o.norm[far]) < RTOL
    cells = nm.shape + (2,)
    assert oracle.rel_l2(d.reshape(cells)[far], o.data.reshape(cells)[far]) < RTOL
