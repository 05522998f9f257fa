"""On-device result counts where the kernel changes its form (needs a B200): a warp per hypothesis up
to 64 paths, a CTA above, first coordinates read in place above 8,192 -- against the host rule, with
clusters that share only their first coordinates and sets that overlap words of 32 paths."""
import numpy as np
import pytest

import ghc
from test_gpu_results import _WS

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("paths,hyp", [(2, 9), (32, 5), (63, 3), (65, 3), (257, 3), (8192, 1), (8193, 1)])
def test_counts_equal_the_host_rule(paths, hyp):
    rng = np.random.default_rng(paths)
    N = 3
    z = rng.normal(size=(hyp, paths, N)) + 1j * rng.normal(size=(hyp, paths, N))
    for h in range(hyp):
        for _ in range(min(200, paths // 3)):
            a, b, c = rng.integers(0, paths, 3)
            z[h, b] = z[h, a] + 1e-7
            z[h, c, 0] = z[h, a, 0]  # the same first coordinate, another point
    z[:, ::5] = z[:, ::5].real + 0j
    conv = rng.random((hyp, paths)) < 0.8
    inf = rng.random((hyp, paths)) < 0.1
    counts, cls = ghc.count_results_device(_WS(z, conv, inf), N, want_class=True)
    counts, cls = counts.cpu().numpy(), cls.cpu().numpy().reshape(hyp, paths)
    for h in range(hyp):
        host = ghc.count_results(z[h], conv[h], inf[h])
        assert [host["converged"], host["real"], host["infinity"], host["unique"]] == counts[h].tolist()
        assert [host["converged"], host["real"], host["unique"]] == [int(((cls[h] >> k) & 1).sum()) for k in range(3)]
