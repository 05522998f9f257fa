"""Class bytes of the on-device result counts, path by path (needs a B200), against the counting rule
restated on NumPy arrays: the skip set is replaced by each duplicate set, so which member of a cluster
counts as unique depends on all clusters before it.  Few duplicated paths, more than the sets that a CTA
forms ahead (48), and every path on one point, at the sizes where the kernel changes its form."""
import numpy as np
import pytest

import ghc
from test_gpu_results import _WS

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


def _class_bytes(z, conv, imag_tol, dup_tol):
    """(class byte of every path, number of converged paths with a later path on their point)"""
    n = len(z)
    cls = conv.astype(np.uint8) | (conv & (np.abs(z.imag) <= imag_tol).all(1)).astype(np.uint8) << 1
    skip, clusters = np.zeros(n, bool), 0
    for p in range(n):
        if not conv[p]:
            continue
        d = z[p + 1:] - z[p]
        later = np.zeros(n, bool)
        later[p + 1:] = ((np.abs(d.real) < dup_tol) & (np.abs(d.imag) < dup_tol)).all(1)
        clusters += later.any()
        if skip[p]:
            continue
        if later.any():
            skip = later
        else:
            cls[p] |= 4
    return cls, clusters


@pytest.mark.parametrize("paths,hyp", [(33, 3), (64, 3), (65, 3), (96, 1481), (128, 1481), (129, 3), (583, 3),
                                       (2500, 1), (8193, 1)])
@pytest.mark.parametrize("shared", ["few", "third", "all"])
def test_class_of_every_path(paths, hyp, shared):
    rng = np.random.default_rng(paths)
    N, distinct = 3, min(hyp, 3)
    z = rng.normal(size=(distinct, paths, N)) + 1j * rng.normal(size=(distinct, paths, N))
    for h in range(distinct):
        if shared == "all":
            z[h] = z[h, 0] + 1e-7 * rng.normal(size=(paths, N))
        else:
            moved = rng.permutation(paths)[:max(1, paths // (50 if shared == "few" else 3))]
            z[h, moved] = z[h, rng.integers(0, paths, len(moved))] + 1e-7
    z[:, ::5] = z[:, ::5].real + 0j
    conv = rng.random((distinct, paths)) < 0.8
    inf = ~conv
    want, clusters = zip(*(_class_bytes(z[h], conv[h], 1e-4, 1e-4) for h in range(distinct)))
    if shared != "few" and paths >= 583:
        assert min(clusters) > 48
    tile = np.arange(hyp) % distinct
    counts, cls = ghc.count_results_device(_WS(z[tile], conv[tile], inf[tile]), N, want_class=True)
    counts, cls = counts.cpu().numpy(), cls.cpu().numpy().reshape(hyp, paths)
    for h in range(hyp):
        w = want[tile[h]]
        assert np.array_equal(cls[h], w), h
        assert counts[h].tolist() == [int((w & 1).sum()), int((w >> 1 & 1).sum()), int(inf[tile[h]].sum()),
                                      int((w >> 2).sum())]
