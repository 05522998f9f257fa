"""A mix with a bucket whose coefficient buffers leave no room for it in the shared launch (needs a B200):
the buckets are launched one by one, with the results of their own launches."""
import numpy as np
import pytest

import ghc
import scenes
from test_gpu_spread import _cx

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

N, M, PATHS = 12, 900, 5  # 901 complex coefficients, twice, for each of the CTA's 8 paths: more than 227 KB


def _large(root):
    rng = np.random.default_rng(1)
    d = root / "LARGE_12"
    d.mkdir()
    (d / "gpuhc_settings.yaml").write_text(
        "problem_name: LARGE_12\nGPUHC_Type: P2C\nGPUHC_Max_Steps: 4\nGPUHC_Max_Correction_Steps: 3\n"
        "GPUHC_Num_Of_Steps_to_Increase_Delta_t: 2\nNum_Of_Vars: 12\nNum_Of_Params: 4\nNum_Of_Tracks: %d\n"
        "dHdx_Max_Terms: 2\ndHdx_Max_Parts: 3\ndHdt_Max_Terms: 20\ndHdt_Max_Parts: 4\nMax_Order_Of_T: 1\n"
        "Num_Of_Coeffs_From_Params: %d\n" % (PATHS, M))
    for f in ("start_params.txt", "target_params.txt"):
        (d / f).write_text("1 0\n" * 4)
    (d / "start_sols.txt").write_text("".join("%.4f %.4f\n" % (a, b) for a, b in 0.3 * rng.normal(size=(N * PATHS, 2))))
    hx = np.stack([np.ones(N * N * 2, int), rng.integers(0, M, N * N * 2), rng.integers(0, N + 1, N * N * 2)], 1)
    ht = np.concatenate([np.ones((N * 20, 1), int), rng.integers(0, M, (N * 20, 1)), rng.integers(0, N + 1, (N * 20, 2))], 1)
    (d / "dHdx_indx.txt").write_text(" ".join(map(str, hx.reshape(-1).tolist())) + "\n")
    (d / "dHdt_indx.txt").write_text(" ".join(map(str, ht.reshape(-1).tolist())) + "\n")
    return ghc.Problem("LARGE_12", root=str(root))


def test_mix_of_a_large_bucket_equals_separate_launches(tmp_path):
    rng = np.random.default_rng(2)
    draw = lambda *shape: 0.3 * (rng.normal(size=shape) + 1j * rng.normal(size=shape))  # noqa: E731
    large, p3p = _large(tmp_path), ghc.Problem("P3P_TD")
    s, t = p3p.params()
    st, tg, _ = scenes.targets_for("P3P_TD", 40, 5, s, t)
    hx, ht = p3p.p2c_device(_cx(st), _cx(tg))
    buckets = [(p3p, 40, dict(d_coef_hx=hx, d_coef_ht=ht)),
               (large, 30, dict(d_coef_hx=_cx(draw(30, 2 * (M + 1))), d_coef_ht=_cx(draw(30, M + 1))))]
    fields = ("endpoints", "status", "conv", "inf", "steps", "corr", "t_end")
    alone, mixed = [], []
    for pb, H, kw in buckets:
        ws = ghc.Workspace(pb, H, ghc.PREC_FP64)
        ghc.track(pb, ws, _cx(pb.start_sols()), **kw)
        alone.append({f: getattr(ws, f).cpu().numpy() for f in fields})
        mixed.append((pb, ghc.Workspace(pb, H, ghc.PREC_FP64), _cx(pb.start_sols()), kw))
    ghc.track_mix(mixed)
    for (_, ws, _, _), a in zip(mixed, alone):
        for f in fields:
            b = getattr(ws, f).cpu().numpy()
            assert np.array_equal(a[f], b, equal_nan=b.dtype.kind == "f"), f
