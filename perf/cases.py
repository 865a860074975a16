"""Performance cases of the direct Fourier inversion path: what programs that
reconstruct maps have this library do, each through its public entry points.

``listed()`` names the cases, ``draw(rng)`` gives more of the same ranges,
``prepare(case, seed)`` makes what a program has in hand before the call,
``run(state)`` is one pass, ``work(case)`` the bytes and operations a pass
cannot do without, and ``exact(case, seed)`` the same outputs summed in 64 bits
(the taps are those of the reference's single-precision window and table
rules; every value and sum after that is double).
"""
from __future__ import annotations

import math

import numpy as np
import torch

from eman2_b200 import EMData, Reconstructors, Transform, _lib
from eman2_b200.batch import InsertGraph, insert_particles_multi
from eman2_b200.particles import particle_meta

DEV = "cuda"
CTF = {"voltage": 300.0, "cs": 2.7, "ampcont": 10.0}
WINDOW = {"nearest_neighbor": 1, "gauss_2": 2, "trilinear": 2, "gauss_5": 6}


# ------------------------------------------------------------------ the cases

def listed():
    return [
        # An initial model from class averages: the drop-in loop of a program
        # written for the reference, one preprocess_slice and one insert_slice
        # per image held in host memory, then finish().
        {"name": "initial model, 24 averages", "kind": "loop", "box": 64, "N": 96,
         "mode": "gauss_2", "sym": "c1", "n": 24},
        # The per-particle insertion loop of make3d on a large box, one particle
        # a call, as a program without batching runs it.
        {"name": "one particle a call, 256", "kind": "single", "box": 256, "N": 384,
         "mode": "gauss_5", "sym": "d7", "n": 4, "ctf": True},
        {"name": "one particle a call, 128", "kind": "single", "box": 128, "N": 192,
         "mode": "gauss_2", "sym": "c1", "n": 16, "ctf": True},
        # A whole small reconstruction in one go: setup, every particle, finish.
        {"name": "small job, 2000 particles", "kind": "job", "box": 64, "N": 96,
         "mode": "gauss_2", "sym": "c1", "n": 2000, "ctf": False},
        # One chunk of a CTF-corrected job from a 16-bit stack already in HBM
        # (widened on the device), into the resident volume.
        {"name": "16-bit chunk, box 128", "kind": "chunk", "box": 128, "N": 192,
         "mode": "gauss_2", "sym": "c1", "n": 2048, "ctf": True, "stack": "float16"},
        # Chunks of the large symmetric jobs: the wide and the narrow inserter.
        {"name": "gauss_5 d7 chunk, box 256", "kind": "chunk", "box": 256, "N": 384,
         "mode": "gauss_5", "sym": "d7", "n": 128, "ctf": True, "stack": "float32"},
        {"name": "gauss_2 d7 chunk, box 256", "kind": "chunk", "box": 256, "N": 384,
         "mode": "gauss_2", "sym": "d7", "n": 1024, "ctf": True, "stack": "float32"},
        # A ragged one: an odd box in a padded size that is not 2-3-5-7 smooth.
        {"name": "odd box 101, c4", "kind": "chunk", "box": 101, "N": 152,
         "mode": "trilinear", "sym": "c4", "n": 777, "ctf": True, "stack": "int16"},
        # A tick of the batched form: even/odd pairs of uneven jobs in one call.
        {"name": "batched tick, 8 uneven jobs", "kind": "batch", "jobs": 8, "n": 96,
         "draw": 1},
        # The captured round a server replays for many small requests.
        {"name": "captured round, 6 jobs", "kind": "graph", "jobs": 6, "n": 3,
         "ticks": 8, "draw": 2},
        # The slice-agreement pass that scores a job's particles.
        {"name": "agreement, 384 d7", "kind": "agree", "N": 384, "sym": "d7", "n": 128},
        # The end of a job: normalise, inverse FFT, kernel correction, clip, and
        # the map in host memory.
        {"name": "finish, 384 to 256", "kind": "finish", "box": 256, "N": 384,
         "mode": "gauss_5"},
    ]


def _smooth(n):
    for p in (2, 3, 5, 7):
        while n % p == 0:
            n //= p
    return n == 1


def _pad(rng, box):
    """A padded size about 1.5 box: mostly the next even smooth one, as programs
    pick it, else whatever even size comes out."""
    n = int(math.ceil(1.5 * box))
    n += n % 2
    if rng.random() < 0.75:
        while not _smooth(n):
            n += 2
    return n


def _pixels(N):
    return int(0.5 * math.pi * (N / 2 + 0.5) ** 2 + N)


def _nsym(sym):
    return {"tet": 12, "oct": 24}.get(sym) or (int(sym[1:]) if sym[0] == "c" else 2 * int(sym[1:]))


def _taps(c):
    return _pixels(c["N"]) * WINDOW[c["mode"]] ** 3 * _nsym(c["sym"])


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["loop", "single", "job", "chunk", "chunk", "chunk", "batch", "graph",
                       "agree", "finish"])
    if kind == "batch":
        return {"kind": kind, "jobs": 2 * rng.randint(1, 5), "n": _log(rng, 8, 128),
                "draw": rng.randrange(1 << 20)}
    if kind == "graph":
        return {"kind": kind, "jobs": rng.randint(2, 8), "n": rng.randint(1, 6),
                "ticks": rng.randint(2, 10), "draw": rng.randrange(1 << 20)}
    if kind == "agree":
        N = _pad(rng, _log(rng, 48, 256))
        sym = rng.choice(["c1", "c4", "d7"])
        most = 3e8 / (_nsym(sym) * N * N / 2)
        return {"kind": kind, "N": N, "sym": sym, "n": max(1, min(2048, _log(rng, 1, most)))}
    box = _log(rng, 48, 256)
    c = {"kind": kind, "box": box, "N": _pad(rng, box)}
    if kind == "finish":
        c["mode"] = rng.choice(["gauss_2", "gauss_5"])
        return c
    c["mode"] = rng.choice(["gauss_2", "gauss_2", "gauss_5", "gauss_5", "nearest_neighbor",
                            "trilinear"])
    c["sym"] = rng.choice(["c1", "c1", "c4", "d7", "tet"])
    c["ctf"] = rng.random() < 0.7
    if kind == "loop":
        c.update(box=min(box, 160), sym=rng.choice(["c1", "c4"]), n=rng.randint(6, 48))
        c["N"] = _pad(rng, c["box"])
        del c["ctf"]
        return c
    if kind == "single":
        c["n"] = rng.randint(1, 16) if _taps(c) < 2e7 else rng.randint(1, 4)
        return c
    # a chunk or a job: taps up to those of the largest listed case
    most = 2.0e10 if c["mode"] == "gauss_5" else 5.0e9
    c["n"] = max(1, min(2048, _log(rng, 16, max(17, most / _taps(c)))))
    if kind == "job":
        c["box"], c["N"] = min(c["box"], 160), min(c["N"], 240)
    else:
        c["stack"] = rng.choice(["float32", "float32", "float16", "int16"])
    return c


def _jobs(case):
    """The jobs of a batched case: even/odd pairs of boxes 64 to 160, both
    modes, c1 or d7, log-uniform particle counts about case["n"]."""
    rng = np.random.default_rng(1000 + int(case["draw"]))
    out = []
    for j in range(int(case["jobs"])):
        if j % 2 == 0 or case["kind"] == "graph":
            box = int(rng.choice([64, 96, 128, 160]))
            mode = str(rng.choice(["gauss_2", "gauss_5"]))
            sym = str(rng.choice(["c1", "d7"]))
        n = int(case["n"]) if case["kind"] == "graph" else \
            max(1, int(round(case["n"] * math.exp(rng.uniform(-1.0, 1.0)))))
        out.append({"box": box, "N": box * 3 // 2, "mode": mode, "sym": sym, "n": n, "ctf": True})
    return out


# ------------------------------------------------------------------ inputs

def _rotations(rng, n):
    q = rng.normal(size=(n, 4))
    w, x, y, z = (q / np.linalg.norm(q, axis=1, keepdims=True)).T
    m = np.stack([w * w + x * x - y * y - z * z, 2 * (x * y + w * z), 2 * (x * z - w * y),
                  2 * (x * y - w * z), w * w - x * x + y * y - z * z, 2 * (y * z + w * x),
                  2 * (x * z + w * y), 2 * (y * z - w * x), w * w - x * x - y * y + z * z], axis=1)
    return m.reshape(n, 3, 3).astype(np.float32)


def _particles(job, seed):
    """Projections of a blob phantom with a CTF, in noise: images on the GPU,
    orientations, shifts, weights and defocus values on the host."""
    n, box = int(job["n"]), int(job["box"])
    rng = np.random.default_rng(seed)
    rots = _rotations(rng, n)
    shifts = rng.uniform(-4, 4, (n, 2)).astype(np.float32)
    weights = rng.uniform(0.5, 1.0, n).astype(np.float32)
    defocus = rng.uniform(0.8, 2.5, n).astype(np.float32) if job.get("ctf") else None
    blobs = 12
    c = rng.normal(size=(blobs, 3))
    c *= (0.3 * box * rng.uniform(0, 1, blobs) ** (1 / 3) / np.linalg.norm(c, axis=1))[:, None]
    uv = np.einsum("nij,gj->ngi", rots[:, :2].astype(np.float64), c) + shifts[:, None]
    uv = torch.as_tensor(uv, device=DEV, dtype=torch.float32)
    inv = torch.as_tensor(1 / (2 * rng.uniform(1.5, 3.0, blobs) ** 2), device=DEV,
                          dtype=torch.float32)
    ax = torch.arange(box, device=DEV, dtype=torch.float32) - box // 2
    gen = torch.Generator(device=DEV).manual_seed(int(seed))
    images = torch.empty((n, box, box), device=DEV)
    for a in range(0, n, 256):
        d = ax - uv[a:a + 256, :, :, None]
        e = torch.exp(-d * d * inv[None, :, None, None])
        s = torch.einsum("ngy,ngx->nyx", e[:, :, 1], e[:, :, 0])
        sd = s.std(dim=(1, 2), keepdim=True)
        images[a:a + 256] = s + torch.randn(s.shape, generator=gen, device=DEV) * sd * 5
    return images, rots, shifts, weights, defocus


def _meta(rots, shifts, weights, defocus):
    return particle_meta(rots, shifts, weights, ctf=CTF, defocus=defocus, apix=1.0)


def _recon(job):
    r = Reconstructors.get("fourier", {"size": [job["N"]] * 3, "sym": job["sym"],
                                       "mode": job["mode"]})
    r.setup()
    return r


def _volume(N):
    return (torch.empty((N, N, N + 2), device=DEV), torch.empty((N, N, N // 2 + 1), device=DEV))


def _stored(images, stack):
    """The images as a stack of this type stores them, and as read back."""
    if stack == "float16":
        raw = images.to(torch.float16)
    elif stack == "int16":
        raw = torch.round(images * 256).clamp(-32768, 32767).to(torch.int16)
    else:
        raw = images
    return raw, raw.float()


def _seeds(case, seed):
    return [int(seed) * 64 + j for j in range(len(_jobs(case)))]


def _agree_inputs(case, seed):
    N, n = int(case["N"]), int(case["n"])
    gen = torch.Generator(device=DEV).manual_seed(int(seed))
    rng = np.random.default_rng(seed)
    data = torch.randn((N, N, N + 2), generator=gen, device=DEV)
    norm = torch.rand((N, N, N // 2 + 1), generator=gen, device=DEV) * 4 + 0.5
    norm[torch.rand(norm.shape, generator=gen, device=DEV) < 0.05] = 0   # cells never reached
    data.view(N, N, N // 2 + 1, 2).mul_(norm[..., None])
    slices = torch.randn((n, N, N + 2), generator=gen, device=DEV)
    return data, norm, slices, _rotations(rng, n), rng.uniform(0.5, 1.0, n).astype(np.float32)


def _finish_inputs(case, seed):
    N = int(case["N"])
    gen = torch.Generator(device=DEV).manual_seed(int(seed))
    data = torch.randn((N, N, N + 2), generator=gen, device=DEV)
    norm = torch.rand((N, N, N // 2 + 1), generator=gen, device=DEV) * 4 + 0.1
    data.view(N, N, N // 2 + 1, 2).mul_(norm[..., None])
    cells = torch.view_as_complex(data.view(N, N, N // 2 + 1, 2))
    for x in (0, N // 2):            # these planes hold every tap and its conjugate
        pl = cells[:, :, x]
        cells[:, :, x] = pl + torch.roll(torch.flip(pl, (0, 1)), (1, 1), (0, 1)).conj()
    return data, norm


def prepare(case, seed):
    kind = case["kind"]
    if kind == "loop":
        job = dict(case, box=case["N"], ctf=False)      # class averages, padded by the program
        images, rots, shifts, weights, _ = _particles(job, seed)
        host = images.cpu().numpy()
        xfs = []
        for i in range(case["n"]):
            m = np.zeros((3, 4), np.float32)
            m[:, :3] = rots[i]
            m[:2, 3] = shifts[i]
            xfs.append(Transform(m.reshape(-1).tolist()))
        return {"kind": kind, "recon": _recon(case), "images": [EMData(h) for h in host],
                "xfs": xfs, "weights": [float(w) for w in weights]}
    if kind == "single":
        images, *rest = _particles(case, seed)
        rots, shifts, weights, defocus = rest
        metas = [_meta(rots[i:i + 1], shifts[i:i + 1], weights[i:i + 1],
                       None if defocus is None else defocus[i:i + 1]) for i in range(case["n"])]
        return {"kind": kind, "recon": _recon(case), "images": images, "metas": metas,
                "out": _volume(case["N"])}
    if kind in ("job", "chunk"):
        images, *rest = _particles(case, seed)
        s = {"kind": kind, "recon": _recon(case), "meta": _meta(*rest)}
        if kind == "job":
            s["images"] = images
            return s
        s["raw"], wide = _stored(images, case["stack"])
        s["images"] = torch.empty_like(wide)
        s["mode"] = {"float16": 12, "int16": 1, "float32": 2}[case["stack"]]
        s["out"] = _volume(case["N"])
        return s
    if kind in ("batch", "graph"):
        jobs = _jobs(case)
        recons = [_recon(j) for j in jobs]
        images, metas = [], []
        for j, sd in zip(jobs, _seeds(case, seed)):
            ticks = int(case.get("ticks", 1))
            im, *rest = _particles(dict(j, n=j["n"] * ticks), sd)
            images.append([im[t * j["n"]:(t + 1) * j["n"]] for t in range(ticks)])
            metas.append([_meta(*(a[t * j["n"]:(t + 1) * j["n"]] for a in rest))
                          for t in range(ticks)])
        s = {"kind": kind, "recons": recons, "out": [_volume(j["N"]) for j in jobs],
             "images": list(zip(*images)), "metas": list(zip(*metas))}
        if kind == "graph":
            s["graph"] = InsertGraph(recons, [j["box"] for j in jobs], [j["n"] for j in jobs],
                                     [True] * len(jobs))
        return s
    if kind == "agree":
        data, norm, slices, rots, weights = _agree_inputs(case, seed)
        r = _recon(dict(case, mode="gauss_2"))
        r.setup_seedandweights(data, norm)
        return {"kind": kind, "recon": r, "slices": slices, "rots": rots, "weights": weights}
    data, norm = _finish_inputs(case, seed)
    return {"kind": "finish", "recon": _recon(dict(case, sym="c1")), "data": data, "norm": norm,
            "box": int(case["box"])}


# ------------------------------------------------------------------ one pass

def _accumulators(r, out):
    """The volume's sums, copied to the program's own device buffers (what a
    program that merges partial volumes reads)."""
    _lib.check(_lib.load().fr_get_accumulators(r.handle, _lib.ptr(out[0]), _lib.ptr(out[1])))
    return {"data": out[0], "norm": out[1]}


def run(s):
    kind = s["kind"]
    if kind == "loop":
        r = s["recon"]
        r.setup()
        status = []
        for img, xf, w in zip(s["images"], s["xfs"], s["weights"]):
            status.append(r.insert_slice(r.preprocess_slice(img, xf), xf, w))
        return {"map": r.finish(True).numpy(), "status": status}
    if kind == "single":
        for i, m in enumerate(s["metas"]):
            s["recon"].insert_particles(s["images"][i:i + 1], m)
        return _accumulators(s["recon"], s["out"])
    if kind == "job":
        r = s["recon"]
        r.setup()
        r.insert_particles(s["images"], s["meta"])
        return {"map": r.finish(True).numpy()}
    if kind == "chunk":
        images = s["raw"]
        if s["mode"] != 2:
            images = s["images"]
            _lib.check(_lib.load().fr_decode_images(
                _lib.ptr(s["raw"]), s["mode"], 0, images.numel(), _lib.ptr(images),
                torch.cuda.current_stream().cuda_stream))
        s["recon"].insert_particles(images, s["meta"])
        return _accumulators(s["recon"], s["out"])
    if kind == "batch":
        insert_particles_multi(s["recons"], s["images"][0], s["metas"][0])
        return [_accumulators(r, o) for r, o in zip(s["recons"], s["out"])]
    if kind == "graph":
        for images, metas in zip(s["images"], s["metas"]):
            s["graph"].launch(images, metas)
        return [_accumulators(r, o) for r, o in zip(s["recons"], s["out"])]
    if kind == "agree":
        return s["recon"].slice_agreement(s["slices"], s["rots"], s["weights"])
    r = s["recon"]
    r.setup_seedandweights(s["data"], s["norm"])
    return r.finish_corrected(outsize=s["box"]).numpy()


# ------------------------------------------------------------------ the floor

# Operations of a tap (distance, table index, three multiply-adds), of a pixel
# (three coordinates) and of a value through one 2-D FFT of size N.
_TAP, _PIX = 16, 18


def _insert_work(c):
    N, n = c["N"], c["n"]
    fft = 5.0 * N * N * math.log2(N)          # real transform, both dimensions
    flops = n * (_taps(c) * _TAP + _pixels(N) * _nsym(c["sym"]) * _PIX + fft * (3 if c.get("ctf") else 1))
    size = {"float16": 2, "int16": 2}.get(c.get("stack"), 4)
    return {"bytes": n * c["box"] ** 2 * size, "flops": flops}


def _sums(*parts):
    return {k: float(sum(p[k] for p in parts)) for k in ("bytes", "flops")}


def work(case):
    kind = case["kind"]
    if kind in ("batch", "graph"):
        ticks = int(case.get("ticks", 1))
        return _sums(*({"bytes": w["bytes"] + 4 * 12 * (j["N"] // 2 + 1) * j["N"] ** 2,
                        "flops": w["flops"]}
                       for j in _jobs(case) for w in [_insert_work(dict(j, n=j["n"] * ticks))]))
    N = case["N"]
    cells = (N // 2 + 1) * N * N
    if kind in ("single", "chunk"):
        # the volume read and written by the insertion, and copied out
        return _sums(_insert_work(case), {"bytes": 4 * 12 * cells, "flops": 0})
    if kind in ("loop", "job"):
        c = dict(case, box=N) if kind == "loop" else case
        return _sums(_insert_work(c), {"bytes": 3 * 12 * cells + 12 * N ** 3,
                                       "flops": 7.5 * N ** 3 * math.log2(N)})
    if kind == "agree":
        pix = case["n"] * N * (N // 2 + 2)
        return {"bytes": 12.0 * cells + 8.0 * pix, "flops": 50.0 * pix * _nsym(case["sym"])}
    # finish: the sums in, normalised, transformed, and the clipped map out
    return {"bytes": 2 * 12.0 * cells + 8.0 * cells + 4.0 * N ** 3 + 4.0 * case["box"] ** 3,
            "flops": 7.5 * N ** 3 * math.log2(N)}


# ------------------------------------------------------------------ 64 bits

def _eman(az, alt):
    a, b = math.radians(az), math.radians(alt)
    return [math.cos(a), math.sin(a), 0.0, -math.cos(b) * math.sin(a), math.cos(b) * math.cos(a),
            math.sin(b), math.sin(b) * math.sin(a), -math.sin(b) * math.cos(a), math.cos(b)]


def _eman_phi(az, alt, phi):
    a, b, p = math.radians(az), math.radians(alt), math.radians(phi)
    return [math.cos(p) * math.cos(a) - math.cos(b) * math.sin(a) * math.sin(p),
            math.cos(p) * math.sin(a) + math.cos(b) * math.cos(a) * math.sin(p),
            math.sin(b) * math.sin(p),
            -math.sin(p) * math.cos(a) - math.cos(b) * math.sin(a) * math.cos(p),
            -math.sin(p) * math.sin(a) + math.cos(b) * math.cos(a) * math.cos(p),
            math.sin(b) * math.cos(p),
            math.sin(b) * math.sin(a), -math.sin(b) * math.cos(a), math.cos(b)]


def _operators(sym):
    f = np.float32
    if sym == "tet":
        l1 = f(math.degrees(math.acos(float(f(-1.0) / f(3.0)))))
        ops = [_eman_phi(0, 0, 120.0 * k) for k in range(3)]
        ops += [_eman_phi(120.0 * a, float(l1), 60.0 + 120.0 * k) for a in range(3) for k in range(3)]
    else:
        n = int(sym[1:])
        ops = [_eman(float(f(i) * f(360) / f(n)), alt)
               for alt in ((0.0,) if sym[0] == "c" else (0.0, 180.0)) for i in range(n)]
    return torch.tensor(ops, dtype=torch.float64).float().to(DEV).view(-1, 3, 3)


def _copies(rots, sym):
    """Rotation blocks of every symmetry copy, composed in single precision."""
    a = torch.as_tensor(rots, device=DEV)[:, None, :, :, None]      # n,1,i,k,1
    b = _operators(sym)[None, :, None]                              # 1,q,1,k,j
    p = a * b
    return (p[:, :, :, 0] + p[:, :, :, 1]) + p[:, :, :, 2]          # n,q,i,j


def _edge_mean(im):
    n = im.shape[-1] * 2 + im.shape[-2] * 2
    return (im[:, 0].sum(1) + im[:, -1].sum(1) + im[:, :, 0].sum(1) + im[:, :, -1].sum(1)) / n


def _ctf_signs(N, defocus):
    f = torch.float32
    kv = np.float32(300.0)
    lam = np.float32(12.2639) / np.sqrt(kv * np.float32(1000) + np.float32(0.97845) * kv * kv)
    g1 = np.float32(math.pi / 2 * np.float64(np.float32(2.7)) * 1e7 * np.float64(lam ** np.float32(3)))
    g2 = np.float32(math.pi * np.float64(lam) * 10000.0)
    acac = np.float32(math.pi / 2 - np.float64(np.float32(math.asin(0.1))))
    y = torch.fft.fftfreq(N, 1.0 / N, device=DEV, dtype=torch.float64).round()
    x = torch.arange(N // 2 + 1, device=DEV, dtype=torch.float64)
    s = (x[None] ** 2 + y[:, None] ** 2).sqrt().to(f) * float(np.float32(1.0) / np.float32(N))
    t1 = s * float(-g1) * s * s * s
    k = torch.as_tensor(defocus, device=DEV)[:, None, None] * float(g2)
    gam = t1 + k * s * s
    c = torch.cos((gam - float(acac)).double())
    return torch.where(c < 0, -1.0, 1.0).double()


def _slices(images, N, shifts, defocus):
    """The preprocessed slices (n, N, N/2+1), complex double."""
    n, box = images.shape[0], images.shape[-1]
    im = images.double()
    im = im - _edge_mean(im)[:, None, None]
    p = torch.zeros((n, N, N), device=DEV, dtype=torch.float64)
    o = (N - box + 1) // 2
    p[:, o:o + box, o:o + box] = im
    if defocus is not None:
        p = torch.fft.irfft2(torch.fft.rfft2(p) * _ctf_signs(N, defocus), s=(N, N))
    p = p - _edge_mean(p)[:, None, None]
    return _shifted(p, N, shifts)


def _shifted(p, N, shifts):
    n, h = p.shape[0], N // 2
    t = torch.as_tensor(shifts, device=DEV)
    ax = torch.arange(N, device=DEV)

    def axis(tr):
        q = ((ax - h).float()[None] + tr[:, None]) + float(h)
        inside = (q >= 0) & (q < N)
        i = q.clamp(0, N - 1).to(torch.int32).long()
        return inside, i, (i + 1).clamp(max=N - 1), (q - i.float()).double()

    inx, x0, x1, u = axis(t[:, 0])
    iny, y0, y1, v = axis(t[:, 1])
    b = torch.arange(n, device=DEV)[:, None, None]
    u, v = u[:, None, :], v[:, :, None]

    def at(y, x):
        return p[b, y[:, :, None], x[:, None, :]]

    out = (1 - u) * (1 - v) * at(y0, x0) + u * (1 - v) * at(y0, x1) + \
        (1 - u) * v * at(y1, x0) + u * v * at(y1, x1)
    out = out * (inx[:, None, :] & iny[:, :, None])
    return torch.fft.rfft2(torch.roll(out, (h, h), (1, 2))) * math.sqrt((N + 2) / N)


def _scaled(i, N):
    """float(i) / float(N), single precision division."""
    return torch.as_tensor(i.cpu().numpy().astype(np.float32) / np.float32(N), device=DEV)


def _insert(vol, slices, copies, weights, N, mode):
    """Adds every tap of every copy to vol = (data, norm), double sums."""
    h = N // 2
    y, x = torch.meshgrid(torch.arange(-h, h, device=DEV), torch.arange(0, h + 1, device=DEV),
                          indexing="ij")
    rad = (x * x + y * y).double().sqrt().float()
    keep = (rad + 0.5).to(torch.int32) <= h
    y, x = y[keep], x[keep]
    rx, ry = _scaled(x, N), _scaled(y, N)
    flat = torch.where((x == 0) & (y < 0), -y * (h + 1), torch.where(y < 0, N + y, y) * (h + 1) + x)
    conj = torch.where((x == 0) & (y < 0), -1.0, 1.0).double()
    K = WINDOW[mode]
    table = torch.as_tensor(np.exp(-np.arange(1000) / 50.0).astype(np.float32), device=DEV).double()
    gw = np.float32(4.0 / math.pi ** 2) if mode == "gauss_2" else np.float32(10.4 / math.pi ** 2)
    hh = float(np.float32(1.0) / gw)
    n, q = copies.shape[:2]
    per = max(1, int(1.6e7 // (x.numel() * K ** 3)))
    for p in range(n):
        w = float(weights[p])
        val = slices[p].reshape(-1)[flat]
        re, im = val.real, val.imag * conj
        for a in range(0, q, per):
            M = copies[p, a:a + per][:, None]                    # s,1,3,3
            c = [(rx * M[..., 0, k] + ry * M[..., 1, k]) * float(N) for k in range(3)]
            if mode == "nearest_neighbor":
                st = [torch.floor(v + 0.5) for v in c]
            elif mode == "gauss_5":
                st = [torch.floor(v.double() - 2.5).float() for v in c]
            else:
                st = [torch.floor(v) for v in c]
            off = torch.arange(K, device=DEV, dtype=torch.float32)
            t = [s[..., None] + off for s in st]                 # s,px,K exact integers
            d = [tt - v[..., None] for tt, v in zip(t, c)]       # rounded once
            X, Y, Z = 0, 1, 2

            def grid(fx, fy, fz, op):
                return op(op(fx[..., None, None, :], fy[..., None, :, None]), fz[..., :, None, None])

            if mode in ("gauss_2", "gauss_5"):
                d2 = [v * v for v in d]
                r = grid(d2[X], d2[Y], d2[Z], torch.add)
                f = (-r) * hh
                g = torch.where(f < -19.98, torch.exp(f.double()),
                                table[(f.double() * -50.0 + 0.5).long().clamp(max=999)])
                del r, f
            elif mode == "trilinear":
                o = [1 - v.double().abs() for v in d]
                g = grid(o[X], o[Y], o[Z], torch.mul)
            else:
                g = torch.ones(c[0].shape + (1, 1, 1), device=DEV, dtype=torch.float64)
            g = g * w
            full = g.shape
            ti = [v.long() for v in t]
            i = ti[X][..., None, None, :].expand(full).reshape(-1)
            j = ti[Y][..., None, :, None].expand(full).reshape(-1)
            k = ti[Z][..., :, None, None].expand(full).reshape(-1)
            vre = (g * re[:, None, None, None]).reshape(-1)
            vim = (g * im[:, None, None, None]).reshape(-1)
            _place(vol, N, i, j, k, vre, vim, g.reshape(-1))
    vol[0][0, 0, 1] = 0
    vol[0][0, 0, N + 1] = 0


def _place(vol, N, i, j, k, re, im, w):
    """The Hermitian placement of taps (i, j, k): i < 0 conjugated at the
    mirrored cell, the planes i = 0 and |i| = N/2 at both cells (the mirrored
    copy without weight), the two self-conjugate cells real."""
    h, w2 = N // 2, N // 2 + 1
    ok = (i.abs() <= h) & (j.abs() <= h) & (k.abs() <= h)
    data = torch.view_as_complex(vol[0].view(N, N, w2, 2)).reshape(-1)
    norm = vol[1].reshape(-1)

    def cell(a, b, c):
        return a + torch.where(b < 0, N + b, b) * w2 + torch.where(c < 0, N + c, c) * (w2 * N)

    def add(m, a, b, c, sign, weight):
        at = cell(a[m], b[m], c[m])
        data.index_add_(0, at, torch.complex(re[m], im[m] * sign))
        if weight:
            norm.index_add_(0, at, w[m])

    axis = (j == 0) & (k == 0)
    own = ok & axis & ((i == 0) | (i.abs() == h))
    add(own, i.abs(), j, k, 1.0, True)                 # imaginary part zeroed by the caller
    ok = ok & ~own
    add(ok & (i == 0), i, -j, -k, -1.0, False)
    add(ok & (i.abs() == h), i.abs(), -j, -k, -1.0, False)
    add(ok & (i < 0), -i, -j, -k, -1.0, True)
    add(ok & (i >= 0), i, j, k, 1.0, True)


def _zero(N):
    return (torch.zeros((N, N, N + 2), device=DEV, dtype=torch.float64),
            torch.zeros((N, N, N // 2 + 1), device=DEV, dtype=torch.float64))


def _normalised(vol, N):
    """Weights of the conjugate pairs of planes 0 and N/2 summed (the five
    self-conjugate cells doubled), then data / weight."""
    data, norm = vol[0], vol[1].clone()
    h = N // 2
    for x in (0, h):
        pl = vol[1][:, :, x]
        mirror = torch.roll(torch.flip(pl, (0, 1)), (1, 1), (0, 1))
        norm[:, :, x] = pl + mirror
    norm[0, 0, 0] = vol[1][0, 0, 0]
    norm[0, 0, h] = vol[1][0, 0, h]
    norm[h, h, h] = vol[1][h, h, h]
    d = torch.view_as_complex(data.view(N, N, h + 1, 2))
    return torch.where(norm == 0, torch.zeros_like(d), d / torch.where(norm == 0, 1.0, norm))


def _map(vol, N):
    # a real inverse transform of the half volume: x is the halved axis, and
    # planes 0 and N/2 enter by the real part of their transform
    c = torch.fft.ifft2(_normalised(vol, N), dim=(0, 1))
    return torch.roll(torch.fft.irfft(c, n=N, dim=2), (N // 2,) * 3, (0, 1, 2))


def _exact_job(case, seed):
    images, rots, shifts, weights, defocus = _particles(case, seed)
    if case.get("stack"):
        raw, images = _stored(images, case["stack"])
    vol, N = _zero(case["N"]), case["N"]
    for a in range(0, case["n"], 64):
        b = slice(a, a + 64)
        _insert(vol, _slices(images[b], N, shifts[b], None if defocus is None else defocus[b]),
                _copies(rots[b], case["sym"]), weights[b], N, case["mode"])
    return vol


def _exact_seconds(jobs):
    return sum(j["n"] * (2.3e-3 + 5.6e-10 * _taps(j)) for j in jobs)


def exact(case, seed):
    kind = case["kind"]
    if kind in ("single", "job", "chunk", "loop") and _exact_seconds([case]) > 17:
        return None
    if kind in ("single", "chunk"):
        vol = _exact_job(case, seed)
        return {"data": vol[0], "norm": vol[1]}
    if kind == "job":
        return {"map": _map(_exact_job(case, seed), case["N"])}
    if kind == "loop":
        images, rots, shifts, weights, _ = _particles(dict(case, box=case["N"], ctf=False), seed)
        vol, N = _zero(case["N"]), case["N"]
        sl = _shifted(images.double(), N, -shifts)      # preprocess_slice undoes the transform
        _insert(vol, sl, _copies(rots, case["sym"]), weights, N, case["mode"])
        return {"map": _map(vol, N), "status": None}
    if kind in ("batch", "graph"):
        jobs = [dict(j, n=j["n"] * int(case.get("ticks", 1))) for j in _jobs(case)]
        if _exact_seconds(jobs) > 17:
            return None
        vols = [_exact_job(j, sd) for j, sd in zip(jobs, _seeds(case, seed))]
        return [{"data": v[0], "norm": v[1]} for v in vols]
    if kind == "agree":
        return _exact_agree(case, seed)
    data, norm = _finish_inputs(case, seed)
    N, box = int(case["N"]), int(case["box"])
    m = _map((data.double(), norm.double()), N)
    o = (N - box) // 2
    width = np.float32({"gauss_2": 4.0, "gauss_5": 10.4}[case["mode"]]) / np.float32(N * N)
    ax = (torch.arange(o, o + box, device=DEV, dtype=torch.float64) - N // 2) ** 2
    r2 = ax[:, None, None] + ax[:, None] + ax
    return m[o:o + box, o:o + box, o:o + box] * torch.exp(r2 * float(width))


def _exact_agree(case, seed):
    data, norm, slices, rots, weights = _agree_inputs(case, seed)
    N, n, h = int(case["N"]), int(case["n"]), int(case["N"]) // 2
    copies = _copies(rots, case["sym"])
    if n * copies.shape[1] > 4000:
        return None
    y, x = torch.meshgrid(torch.arange(-h, h, device=DEV), torch.arange(0, h + 2, device=DEV),
                          indexing="ij")
    live = ~((x == 0) & (y == 0))
    y, x = y[live], x[live]
    rx, ry = _scaled(x, N), _scaled(y, N)
    at = 2 * x + (N + 2) * torch.where(y < 0, N + y, y)
    rad = (x * x + y * y).double().sqrt()
    rmax = max(5.0, min(N / 12.0, N / 2 - 1.0))
    low = (rad > 3) & (rad < rmax)
    data, norm = data.double().view(-1, 2), norm.double().view(-1)
    flat = torch.cat([slices.view(n, -1), torch.zeros((n, 2), device=DEV)], 1)
    out = torch.empty((n, 5), device=DEV, dtype=torch.float64)
    for p in range(n):
        d2 = torch.stack([flat[p][at], flat[p][at + 1]], 1).double()
        S = torch.zeros(8, device=DEV, dtype=torch.float64)
        for M in copies[p]:
            c = [rx * M[0, k] + ry * M[1, k] for k in range(3)]
            ok = (c[0].abs() <= 0.5) & (c[1].abs() < 0.5) & (c[2].abs() < 0.5)
            v = [torch.trunc(torch.where(q < 0, q * float(N) - 0.5, q * float(N) + 0.5)).long()
                 for q in c]
            sg = torch.where(v[0] < 0, -1, 1)
            i, j, k = (q * sg for q in v)
            cell = (i + torch.where(j < 0, N + j, j) * (h + 1) +
                    torch.where(k < 0, N + k, k) * (h + 1) * N)
            cell = torch.where(ok, cell, 0)
            inside = ok & (i <= h) & (j.abs() <= h) & (k.abs() <= h)
            nv = torch.where(ok, norm[cell], 0.0)
            ok = nv != 0
            g = torch.where(inside[:, None], data[cell], 0.0)
            g = torch.stack([g[:, 0], g[:, 1] * sg], 1) / torch.where(ok, nv, 1.0)[:, None]
            dot = (g * d2).sum(1) * nv
            pw, pw2 = (g * g).sum(1) * nv, (d2 * d2).sum(1) * nv
            z = [(a * ok * m).sum() for a, m in ((dot, low), (pw, low), (pw2, low))]
            z += [(a * ok).sum() for a in (dot, nv, pw, pw2)] + [ok.sum().double()]
            S += torch.stack(z)
        dl, p1, p2, dot, vw, pw, pw2, cnt = S.tolist()
        dot /= math.sqrt(pw * pw2)
        dl = dl / math.sqrt(p1 * p2) if p1 * p2 > 0 else dl
        rw = float(np.float32(1.0) / weights[p])
        out[p] = torch.tensor([math.sqrt(pw / pw2), dot, dl, dot * rw / ((rw - 1) * dot + 1),
                               vw / cnt])
    return out.cpu().numpy()
