"""Results into pageable host memory: byte for byte what the device holds, for
sizes around the pieces the copying threads take and from several host threads
at once; and finish() with and without the weight volume asked for."""
from __future__ import annotations

import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _seeded(N, seed):
    from eman2_b200 import Reconstructors
    rng = np.random.default_rng(seed)
    d = rng.normal(size=(N, N, N + 2)).astype(np.float32)
    w = rng.uniform(0.5, 2.0, (N, N, N // 2 + 1)).astype(np.float32)
    r = Reconstructors.get("fourier", {"size": [N] * 3, "sym": "c1", "mode": "gauss_2"})
    r.setup_seedandweights(d, w)
    return r, d, w


@pytest.mark.parametrize("N", [16, 100, 102, 126, 128, 160, 254])
def test_accumulators_round_trip(gpu, N):
    r, d, w = _seeded(N, N)
    gd, gw = r.get_accumulators()
    assert np.array_equal(gd, d) and np.array_equal(gw, w)


def test_round_trips_from_threads(gpu):
    jobs = [_seeded(N, N) for N in (128, 140, 160, 130)]
    bad = []

    def run(r, d, w):
        for _ in range(5):
            gd, gw = r.get_accumulators()
            if not (np.array_equal(gd, d) and np.array_equal(gw, w)):
                bad.append(d.shape)

    ts = [threading.Thread(target=run, args=j) for j in jobs]
    for t in ts:
        t.start()
    for t in ts:
        t.join()
    assert not bad


def test_finish_weights_only_when_asked(gpu, tmp_path):
    from eman2_b200 import EMData
    r, _, _ = _seeded(48, 1)
    plain = r.finish(True).numpy()
    out = EMData(nx=1, ny=1)
    for key, val in (("normout", out), ("savenorm", str(tmp_path / "n.npy"))):
        r, _, _ = _seeded(48, 1)
        r.insert_params({key: val})
        assert np.array_equal(r.finish(True).numpy(), plain)
    assert np.array_equal(out.numpy(), np.load(tmp_path / "n.npy"))
    assert out.numpy().shape == (48, 48, 25)


def _per_thread_stream(r):
    """The handle on the per-thread default stream (cudaStreamPerThread)."""
    from eman2_b200 import _lib
    _lib.check(_lib.load().fr_set_stream(r.handle, 2))


@pytest.mark.parametrize("N", [64, 128, 190])
def test_finish_on_the_per_thread_stream(gpu, N):
    """A map copied out behind work still queued on the per-thread stream,
    whose handle names another stream in every thread, is the one that an
    ordinary stream gives."""
    import torch
    r, d, w = _seeded(N, N)
    want = r.finish(True).numpy()
    r, _, _ = _seeded(N, N)
    _per_thread_stream(r)
    with torch.cuda.stream(torch.cuda.ExternalStream(2)):
        torch.cuda._sleep(50_000_000)
    assert np.array_equal(r.finish(True).numpy(), want)


def test_per_thread_stream_from_two_threads(gpu):
    """Insertions that one thread queued on its per-thread stream are in the map
    that another thread takes from its own."""
    import torch
    from eman2_b200 import Reconstructors
    N, n = 48, 20
    rng = np.random.default_rng(3)
    sl = rng.normal(size=(n, N, N + 2)).astype(np.float32)
    rots = np.stack([np.linalg.qr(rng.normal(size=(3, 3)))[0] for _ in range(n)]).astype(np.float32)

    def inserted(per_thread):
        r = Reconstructors.get("fourier", {"size": [N] * 3, "sym": "c1", "mode": "gauss_2"})
        r.setup()
        if per_thread:
            _per_thread_stream(r)
            with torch.cuda.stream(torch.cuda.ExternalStream(2)):
                torch.cuda._sleep(50_000_000)
        r.insert_slices(sl, rots, np.ones(n, np.float32))
        return r

    want = inserted(False).finish(True).numpy()
    made = []
    t = threading.Thread(target=lambda: made.append(inserted(True)))
    t.start()
    t.join()
    got = made[0].finish(True).numpy()
    assert np.abs(got - want).max() < 1e-5 * np.abs(want).max()
