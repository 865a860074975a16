"""The one-launch particle preparation (fr_slice.cu) over radix pairs of every
kind (equal, unequal, odd with even, the largest image that fits), odd and
oversized boxes, shifts from none to beyond the image, and particles with and
without a phase flip in one call.  FP32 transforms against FP64 ones rounded:
2e-5 as for the other FFT paths (a transform's error is a few eps log2 N)."""
from __future__ import annotations

import numpy as np
import pytest

from oracle import oracle

pytestmark = pytest.mark.gpu
RTOL = 2e-5


def _shifts(n, N, rng):
    s = rng.uniform(-5, 5, (n, 2)).astype(np.float32)
    fixed = [(0, 0), (0, 1.5), (-2.25, 0), (3, -4), (1e-7, -1e-7), (-0.5, 2e-6), (N / 2, 0.25),
             (0.75, -N), (-1.0 * N, 2.0), (-0.999999, 0.999999)]
    s[:len(fixed)] = np.asarray(fixed, np.float32)
    return s


@pytest.mark.parametrize("N", [16, 18, 30, 42, 76, 84, 98, 150, 170, 196, 208, 240])
def test_preprocess_sizes(gpu, N):
    from eman2_b200 import Reconstructors, _lib
    n = 56
    rng = np.random.default_rng(N)
    img = rng.normal(size=(n, N, N)).astype(np.float32)
    inv = _shifts(n, N, rng)
    r = Reconstructors.get("fourier", {"size": [N] * 3, "sym": "c1", "mode": "gauss_2"})
    r.setup()
    out = np.empty((n, N, N + 2), np.float32)
    _lib.check(_lib.load().fr_preprocess_slices(r.handle, _lib.ptr(img), n, _lib.ptr(inv),
                                                _lib.ptr(out)))
    for i in range(n):
        want = oracle.preprocess_slice(img[i], float(inv[i, 0]), float(inv[i, 1]))
        if not want.any():
            assert not out[i].any()
        else:
            assert oracle.rel_l2(out[i], want) < RTOL, i


@pytest.mark.parametrize("box,N", [(11, 16), (64, 96), (101, 150), (33, 32), (70, 60), (128, 192),
                                   (101, 152), (120, 176), (160, 240)])
def test_particles_sizes(gpu, box, N):
    from eman2_b200 import Reconstructors
    from eman2_b200.particles import particle_meta
    from eman2_b200.synth import quaternion_blocks, random_quaternions
    n = 48
    rng = np.random.default_rng(N + 1)
    img = (rng.normal(size=(n, box, box)) + 3.0).astype(np.float32)
    rots = quaternion_blocks(random_quaternions(n, rng))
    shifts = rng.uniform(-3, 3, (n, 2)).astype(np.float32)
    w = rng.uniform(0.5, 1.0, n).astype(np.float32)
    df = rng.uniform(0.8, 2.5, n).astype(np.float32)
    df[::5] = 0.0
    take = np.arange(56) % n   # as many as the one launch asks for
    n, img, rots, shifts, w, df = 56, img[take], rots[take], shifts[take], w[take], df[take]
    ctf = {"dfdiff": 0.1, "dfang": 30.0}
    r = Reconstructors.get("fourier", {"size": [N] * 3, "sym": "c1", "mode": "gauss_2"})
    r.setup()
    r.insert_particles(img, particle_meta(rots, shifts, w, ctf=ctf, defocus=df))
    d, nm = r.get_accumulators()
    sl = np.stack([oracle.particle_to_slice(img[i], N, shifts[i], dict(ctf, defocus=float(df[i])))
                   for i in range(n)])
    o = oracle.OracleVolume(N, "fp32acc64")
    o.insert(sl, rots, w, "gauss_2", "c1")
    assert oracle.rel_l2(nm, o.norm) < 2e-6
    assert oracle.rel_l2(d, o.data) < RTOL


@pytest.mark.parametrize("box,N,n", [(16, 16, 1), (13, 26, 6), (101, 150, 3), (70, 60, 2),
                                     (200, 240, 6), (170, 242, 2), (256, 384, 1), (300, 286, 2),
                                     (150, 224, 40), (90, 252, 47)])
def test_few_particles(gpu, box, N, n):
    """A call of few particles (fr_lines.cu): one to three passes a line, odd
    and oversized boxes, each call's particles with and without a phase flip."""
    from eman2_b200 import Reconstructors
    from eman2_b200.particles import particle_meta
    from eman2_b200.synth import quaternion_blocks, random_quaternions
    rng = np.random.default_rng(N + n)
    for defocus in ([0.0] * n, [1.5 - 1.5 * (i % 2) for i in range(n)]):
        img = (rng.normal(size=(n, box, box)) + 3.0).astype(np.float32)
        rots = quaternion_blocks(random_quaternions(n, rng))
        shifts = rng.uniform(-5, 5, (n, 2)).astype(np.float32)
        fixed = [(2.25, -1.5), (0, 0), (-N, 1), (1e-7, 0), (-0.5, 3), (4, N / 2)][:n]
        shifts[:len(fixed)] = fixed
        w = rng.uniform(0.5, 1.0, n).astype(np.float32)
        ctf = {"dfdiff": 0.1, "dfang": 30.0}
        r = Reconstructors.get("fourier", {"size": [N] * 3, "sym": "c1", "mode": "gauss_2"})
        r.setup()
        r.insert_particles(img, particle_meta(rots, shifts, w, ctf=ctf,
                                              defocus=np.asarray(defocus, np.float32)))
        d, nm = r.get_accumulators()
        sl = np.stack([oracle.particle_to_slice(img[i], N, shifts[i],
                                                dict(ctf, defocus=float(defocus[i])))
                       for i in range(n)])
        o = oracle.OracleVolume(N, "fp32acc64")
        o.insert(sl, rots, w, "gauss_2", "c1")
        assert oracle.rel_l2(nm, o.norm) < 2e-6
        assert oracle.rel_l2(d, o.data) < RTOL


@pytest.mark.parametrize("N,n,shift", [(32, 4, 1), (32, 64, 1), (32, 4, 0), (32, 64, 0),
                                       (242, 2, 1), (242, 2, 0)])
def test_slices_over_images(gpu, N, n, shift):
    """Slices written over the memory of their own images come out as they do
    into memory of their own."""
    import torch
    from eman2_b200 import Reconstructors, _lib
    rng = np.random.default_rng(N + n)
    img = rng.normal(size=(n, N, N)).astype(np.float32)
    inv = rng.uniform(-5, 5, (n, 2)).astype(np.float32)
    want = np.stack([oracle.preprocess_slice(img[i], float(inv[i, 0]), float(inv[i, 1]))
                     for i in range(n)])
    r = Reconstructors.get("fourier", {"size": [N] * 3, "sym": "c1", "mode": "gauss_2"})
    r.setup()
    buf = torch.zeros(n * N * (N + 2) + 2, device="cuda")
    if shift:      # images behind the slices' start, in the slices' memory
        src = buf[2:2 + n * N * N]
    else:
        src = buf[:n * N * N]
    src.copy_(torch.from_numpy(img).reshape(-1))
    d_inv = torch.from_numpy(inv).cuda()
    torch.cuda.synchronize()
    _lib.check(_lib.load().fr_preprocess_slices(r.handle, src.data_ptr(), n, d_inv.data_ptr(),
                                                buf.data_ptr()))
    got = buf[:n * N * (N + 2)].cpu().numpy().reshape(n, N, N + 2)
    for i in range(n):
        assert oracle.rel_l2(got[i], want[i]) < RTOL, i


@pytest.mark.parametrize("N,n", [(32, 64), (32, 3), (170, 30), (242, 3), (52, 60)])
@pytest.mark.parametrize("axis", [(0,), (1,), (0, 1)])
def test_nan_shift_gives_a_nan_slice(gpu, N, n, axis):
    """A shift that is not a number makes its slice so, in each preparation (one
    launch, with the radix 17 too, and lines), and leaves the others alone."""
    from eman2_b200 import Reconstructors, _lib
    rng = np.random.default_rng(N)
    img = rng.normal(size=(n, N, N)).astype(np.float32)
    inv = rng.uniform(-2, 2, (n, 2)).astype(np.float32)
    inv[1, list(axis)] = np.nan
    r = Reconstructors.get("fourier", {"size": [N] * 3, "sym": "c1", "mode": "gauss_2"})
    r.setup()
    out = np.empty((n, N, N + 2), np.float32)
    _lib.check(_lib.load().fr_preprocess_slices(r.handle, _lib.ptr(img), n, _lib.ptr(inv),
                                                _lib.ptr(out)))
    assert np.isnan(out[1]).all()
    for i in (0, n - 1):
        want = oracle.preprocess_slice(img[i], float(inv[i, 0]), float(inv[i, 1]))
        assert i == 1 or oracle.rel_l2(out[i], want) < RTOL, i


@pytest.mark.parametrize("box,N,n", [(200, 300, 57), (290, 432, 49), (330, 500, 3), (512, 768, 1)])
def test_lines_of_many_or_large_images(gpu, box, N, n):
    """The line preparation where several blocks' stages overlap: many particles
    a call and sizes beyond 384, each stage reading what the one before it wrote.
    Without astigmatism, so that no sign hangs on the last place of an angle."""
    from eman2_b200 import Reconstructors
    from eman2_b200.particles import particle_meta
    from eman2_b200.synth import quaternion_blocks, random_quaternions
    rng = np.random.default_rng(N)
    img = (rng.normal(size=(n, box, box)) + 3.0).astype(np.float32)
    rots = quaternion_blocks(random_quaternions(n, rng))
    shifts = rng.uniform(-5, 5, (n, 2)).astype(np.float32)
    df = rng.uniform(0.8, 2.5, n).astype(np.float32)
    df[1::4] = 0.0
    w = rng.uniform(0.5, 1.0, n).astype(np.float32)
    ctf = {"voltage": 300.0, "cs": 2.7}
    r = Reconstructors.get("fourier", {"size": [N] * 3, "sym": "c1", "mode": "nearest_neighbor"})
    r.setup()
    r.insert_particles(img, particle_meta(rots, shifts, w, ctf=ctf, defocus=df))
    d, nm = r.get_accumulators()
    sl = np.stack([oracle.particle_to_slice(img[i], N, shifts[i], dict(ctf, defocus=float(df[i])))
                   for i in range(n)])
    o = oracle.OracleVolume(N, "fp32acc64")
    o.insert(sl, rots, w, "nearest_neighbor", "c1")
    assert oracle.rel_l2(nm, o.norm) < 2e-6
    assert oracle.rel_l2(d, o.data) < RTOL


@pytest.mark.parametrize("box,N,n", [(101, 152, 24), (90, 136, 55), (113, 170, 40), (152, 228, 31)])
def test_radices_17_and_19_from_24_particles(gpu, box, N, n):
    """The one-launch preparation of sizes with a factor 17 or 19, which takes
    over at 24 particles, with and without a phase flip in one call (and without
    astigmatism, so that no sign hangs on the last place of an angle)."""
    from eman2_b200 import Reconstructors
    from eman2_b200.particles import particle_meta
    from eman2_b200.synth import quaternion_blocks, random_quaternions
    rng = np.random.default_rng(N + n)
    img = (rng.normal(size=(n, box, box)) + 3.0).astype(np.float32)
    rots = quaternion_blocks(random_quaternions(n, rng))
    shifts = rng.uniform(-3, 3, (n, 2)).astype(np.float32)
    w = rng.uniform(0.5, 1.0, n).astype(np.float32)
    df = rng.uniform(0.8, 2.5, n).astype(np.float32)
    df[::5] = 0.0
    ctf = {"voltage": 300.0, "cs": 2.7}
    r = Reconstructors.get("fourier", {"size": [N] * 3, "sym": "c1", "mode": "gauss_2"})
    r.setup()
    r.insert_particles(img, particle_meta(rots, shifts, w, ctf=ctf, defocus=df))
    d, nm = r.get_accumulators()
    sl = np.stack([oracle.particle_to_slice(img[i], N, shifts[i], dict(ctf, defocus=float(df[i])))
                   for i in range(n)])
    o = oracle.OracleVolume(N, "fp32acc64")
    o.insert(sl, rots, w, "gauss_2", "c1")
    assert oracle.rel_l2(nm, o.norm) < 2e-6
    assert oracle.rel_l2(d, o.data) < RTOL
