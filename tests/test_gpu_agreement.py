"""The slice-agreement pass over the sizes its blocks split at: fewer rows than
one block takes, a remainder of rows, one slice and several, and the
low-resolution limit at, below and above its clamps.  Sums are FP64 on both
sides over the same FP32 terms, so the attributes agree to float rounding;
the accumulators they are taken from differ by summation order (2e-6)."""
from __future__ import annotations

import numpy as np
import pytest

from oracle import oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("N,n,sym,apix", [(8, 1, "c1", 1.0), (22, 2, "d3", 3.0), (34, 3, "c1", 0.1),
                                          (50, 5, "tet", 2.5), (96, 2, "c4", 1.0)])
def test_agreement_sizes(gpu, N, n, sym, apix):
    from eman2_b200 import Reconstructors
    from eman2_b200.synth import quaternion_blocks, random_quaternions
    rng = np.random.default_rng(N)
    sl = rng.normal(size=(n, N, N + 2)).astype(np.float32)
    rt = quaternion_blocks(random_quaternions(n, rng))
    w = rng.uniform(0.2, 1.0, n).astype(np.float32)
    r = Reconstructors.get("fourier", {"size": [N] * 3, "sym": sym, "mode": "gauss_2"})
    r.setup()
    r.insert_slices(sl, rt, w)
    got = r.slice_agreement(sl, rt, w, apix=apix)
    o = oracle.OracleVolume(N, "fp32")
    o.insert(sl, rt, w, "gauss_2", sym)
    for i in range(n):
        np.testing.assert_allclose(got[i], o.compare(sl[i], rt[i], float(w[i]), sym, apix),
                                   rtol=2e-5, atol=2e-6)


@pytest.mark.parametrize("N,n", [(318, 23), (506, 37)])
def test_agreement_slabs(gpu, N, n):
    """Volumes beyond the L2 cache are taken in two or three slabs when many
    slices are compared at once, whole when few are: the same FP64 sums in
    another order, so the attributes agree to the rounding to float."""
    from eman2_b200 import Reconstructors
    from eman2_b200.synth import quaternion_blocks, random_quaternions
    rng = np.random.default_rng(N)
    sl = rng.normal(size=(n, N, N + 2)).astype(np.float32)
    rt = quaternion_blocks(random_quaternions(n, rng))
    w = rng.uniform(0.2, 1.0, n).astype(np.float32)
    r = Reconstructors.get("fourier", {"size": [N] * 3, "sym": "d7", "mode": "gauss_2"})
    r.setup()
    r.insert_slices(sl, rt, w)
    got = r.slice_agreement(sl, rt, w)
    for i in range(0, n, 7):
        np.testing.assert_allclose(got[i], r.slice_agreement(sl[i:i + 1], rt[i:i + 1], w[i:i + 1])[0],
                                   rtol=3e-7, atol=1e-7)
