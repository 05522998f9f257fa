"""A launch of few paths gives each its own warp, whose sub-warps share the path's coefficients and its
H_x walk (needs a B200): every size with more than one sub-warp per warp, every walk, against the same
hypothesis inside a batch that is not spread, bit for bit."""
import numpy as np
import pytest

import ghc
import scenes

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


def _cx(a, dtype=torch.float64):
    return torch.view_as_real(torch.from_numpy(np.ascontiguousarray(a, dtype=np.complex128))).to(dtype).cuda()


@pytest.mark.parametrize("prec", [ghc.PREC_FP64, ghc.PREC_FP32, ghc.PREC_MIXED])
@pytest.mark.parametrize("name", ["P3P", "rel_pos_quiver", "dual_reciever_TDOA_5pt", "5pt_rel_pos_alg_form_quat",
                                  "3view_triangulation", "P3P_10x10", "4view_triangulation",
                                  "generalized_3views_4pts", "5pt_rel_pos_full_form_quat"])
def test_spread_equals_batch(name, prec):
    pb = ghc.Problem(name)
    s, t = pb.params()
    H = 700 // pb.paths + 2  # more paths than one per warp of the GPU's first wave
    st, tg, _ = scenes.targets_for(name, H, 5, s, t)
    hx, ht = pb.p2c_device(_cx(st), _cx(tg))
    sols = _cx(pb.start_sols(), torch.float32 if prec == ghc.PREC_FP32 else torch.float64)
    whole = ghc.Workspace(pb, H, prec)
    for walk in (0, 1, 2):
        ghc.set_tuning(pb, prec, 0, walk)
        ghc.track(pb, whole, sols, d_coef_hx=hx, d_coef_ht=ht, max_steps=25)
        for h in (0, H - 1):
            one = ghc.Workspace(pb, 1, prec)
            ghc.track(pb, one, sols, d_coef_hx=hx[h:h + 1].contiguous(), d_coef_ht=ht[h:h + 1].contiguous(), max_steps=25)
            for f in ("endpoints", "status", "steps", "corr", "t_end", "dt_end"):
                a = getattr(one, f).cpu().numpy()
                b = getattr(whole, f)[h * pb.paths:(h + 1) * pb.paths].cpu().numpy()
                assert np.array_equal(a, b, equal_nan=a.dtype.kind == "f"), (walk, h, f)
