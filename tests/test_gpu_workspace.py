"""The partial volume that large plane-column insertions borrow: one a device
for every handle, lent to one call at a time across streams and threads, given
back when memory runs out, and done without where there is none.

Tolerance as for the other insertion tests: only the order of FP32 additions
differs, 2e-6 for the at most ~1e3 additions of a cell here."""
from __future__ import annotations

import threading
from contextlib import contextmanager, nullcontext

import numpy as np
import pytest

from oracle import oracle

pytestmark = pytest.mark.gpu
RTOL = 2e-6
MB = 1 << 20


def _inputs(N, n, seed=0):
    import torch
    from eman2_b200.synth import quaternion_blocks, random_quaternions
    rng = np.random.default_rng(seed + N)
    sl = rng.normal(size=(n, N, N + 2)).astype(np.float32)
    return (torch.from_numpy(sl).cuda(), sl, quaternion_blocks(random_quaternions(n, rng)),
            rng.uniform(0.5, 1.0, n).astype(np.float32))


def _recon(N, mode="gauss_2"):
    from eman2_b200 import Reconstructors
    r = Reconstructors.get("fourier", {"size": [N] * 3, "sym": "c1", "mode": mode})
    r.setup()
    return r


def _free():
    import torch
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    return torch.cuda.mem_get_info()[0]


@contextmanager
def _left(nbytes):
    """The device's memory taken but for so many bytes."""
    import torch
    hog = torch.empty(_free() - nbytes, dtype=torch.uint8, device="cuda")
    try:
        yield
    finally:
        del hog
        _free()


def _expected(N, sl, rots, w, mode="gauss_2"):
    o = oracle.OracleVolume(N, "fp32acc64")
    o.insert(sl, rots, w, mode, "c1")
    return o


def _check(r, o):
    d, nm = r.get_accumulators()
    assert np.array_equal(nm != 0, o.norm != 0)
    assert oracle.rel_l2(nm, o.norm) < RTOL and oracle.rel_l2(d, o.data) < RTOL


def test_handles_share_one(gpu):
    N, n = 192, 600
    d_sl, _, rots, w = _inputs(N, n)
    recons = [_recon(N) for _ in range(3)]
    recons[0].insert_slices(d_sl, rots, w)
    before = _free()
    for r in recons[1:]:
        r.insert_slices(d_sl, rots, w)
    assert before - _free() < 16 * MB       # one more would be 57 MB each
    for r in recons:
        r.close()


def test_given_back_when_memory_runs_out(gpu):
    """A map that fits only in the partial volume's place."""
    N, n = 256, 800
    d_sl, _, rots, w = _inputs(N, n)
    want = None
    for short in (False, True):
        r = _recon(N)
        r.insert_slices(d_sl, rots, w)
        # the map takes 67 MB, the partial volume 135
        with _left(60 * MB) if short else nullcontext():
            got = r.finish(True).numpy()
        if want is not None:
            assert oracle.rel_l2(got, want) < 2e-5
        want = got
        r.close()


def test_without_room_straight_into_the_sums(gpu):
    N, n = 256, 800
    d_sl, sl, rots, w = _inputs(N, n, 1)
    r = _recon(N)
    r.insert_slices(d_sl[:300], rots[:300], w[:300])    # scratch in place
    r.setup()
    with _left(20 * MB), pytest.raises(Exception):      # takes back an earlier call's volume
        _recon(512)
    with _left(100 * MB):
        before = _free()
        r.insert_slices(d_sl, rots, w)
        assert before - _free() < 16 * MB               # none was taken
    _check(r, _expected(N, sl, rots, w))
    r.close()


def test_a_call_too_large_leaves_a_smaller_volume(gpu):
    """Calls that find no room do not make the others allocate theirs anew."""
    small, large = _inputs(192, 600), _inputs(256, 800)
    recons = [_recon(192), _recon(256)]
    with _left(20 * MB), pytest.raises(Exception):
        _recon(512)
    for r, (d_sl, _, rots, w) in zip(recons, (small, large)):
        r.insert_slices(d_sl[:250], rots[:250], w[:250])    # scratch in place
    recons[0].insert_slices(small[0], small[2], small[3])
    with _left(100 * MB):                                   # 57 MB are lent already, 135 would be
        before = _free()
        for r, (d_sl, _, rots, w) in zip(recons[::-1], (large, small)):
            r.insert_slices(d_sl, rots, w)
        assert abs(before - _free()) < 16 * MB
    for r in recons:
        r.close()


def test_threads_on_their_own_streams(gpu):
    sizes = (96, 160, 128, 192)
    jobs = [(N, *_inputs(N, 530, 2)) for N in sizes]
    recons = [_recon(N, "gauss_2" if k % 2 else "trilinear") for k, N in enumerate(sizes)]
    go = threading.Barrier(len(sizes))

    def run(r, d_sl, rots, w):
        go.wait()
        for _ in range(6):
            r.insert_slices(d_sl, rots, w)

    ts = [threading.Thread(target=run, args=(r, j[1], j[3], j[4])) for r, j in zip(recons, jobs)]
    for t in ts:
        t.start()
    for t in ts:
        t.join()
    for k, (r, (N, _, sl, rots, w)) in enumerate(zip(recons, jobs)):
        o = _expected(N, sl, rots, w, "gauss_2" if k % 2 else "trilinear")
        d, nm = r.get_accumulators()
        assert oracle.rel_l2(nm, 6 * o.norm) < RTOL and oracle.rel_l2(d, 6 * o.data) < RTOL
        r.close()


def test_captured_rounds_beside_calls(gpu):
    """A graph's branches insert through partial volumes of their own while calls
    borrow the device's."""
    import torch
    from eman2_b200 import Reconstructors
    from eman2_b200.batch import InsertGraph, insert_particles_multi
    from eman2_b200.particles import particle_meta
    shapes = [(96, 300, "c1", "gauss_2"), (64, 80, "d2", "gauss_5"), (80, 70, "c4", "trilinear")]
    params = [{"size": [N] * 3, "sym": s, "mode": m} for N, _, s, m in shapes]
    images, metas = [], []
    for N, n, _, _ in shapes:
        _, _, rots, w = _inputs(N, n, 3)
        img = torch.randn(n, N, N, generator=torch.Generator().manual_seed(N))
        images.append(img.cuda())
        metas.append(particle_meta(rots, None, w))

    def handles():
        rs = [Reconstructors.get("fourier", p) for p in params]
        for r in rs:
            r.setup()
        return rs

    alone, mixed = handles(), handles()
    for r, im, m in zip(alone, images, metas):
        for _ in range(3):
            r.insert_particles(im, m)
    g = InsertGraph(mixed, [N for N, *_ in shapes], [n for _, n, *_ in shapes], [False] * 3)
    g.launch(images, metas)
    insert_particles_multi(mixed, images, metas)
    g.launch(images, metas)
    for a, b in zip(alone, mixed):
        (d0, n0), (d1, n1) = a.get_accumulators(), b.get_accumulators()
        assert oracle.rel_l2(n1, n0) < RTOL and oracle.rel_l2(d1, d0) < RTOL
    g.close()
