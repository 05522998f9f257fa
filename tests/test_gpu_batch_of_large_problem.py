"""More than one wave of paths of problems whose coefficient buffers limit the CTA (needs a B200): 565
coefficients leave no room for 128 threads, 75 take CTAs of more -- each hypothesis of the batch equals
its own launch, bit for bit."""
import numpy as np
import pytest

import ghc
import scenes
from test_gpu_spread import _cx

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("prec", [ghc.PREC_FP64, ghc.PREC_FP32, ghc.PREC_MIXED])
@pytest.mark.parametrize("name,H", [("generalized_3views_6lines", 4), ("5pt_rel_pos_geo_form_quat", 260),
                                    ("dual_reciever_TDOA_5pt", 400), ("3view_triangulation", 400)])
def test_batch_equals_single_launches(name, H, prec):
    pb = ghc.Problem(name)
    s, t = pb.params()
    st, tg, _ = scenes.targets_for(name, H, 9, s, t)
    hx, ht = pb.p2c_device(_cx(st), _cx(tg))
    sols = _cx(pb.start_sols(), torch.float32 if prec == ghc.PREC_FP32 else torch.float64)
    whole, one = ghc.Workspace(pb, H, prec), ghc.Workspace(pb, 1, prec)
    ghc.track(pb, whole, sols, d_coef_hx=hx, d_coef_ht=ht, max_steps=12)
    for h in (0, H // 2, H - 1):
        ghc.track(pb, one, sols, d_coef_hx=hx[h:h + 1].contiguous(), d_coef_ht=ht[h:h + 1].contiguous(), max_steps=12)
        for f in ("endpoints", "status", "steps", "corr"):
            a = getattr(one, f).cpu().numpy()
            b = getattr(whole, f)[h * pb.paths:(h + 1) * pb.paths].cpu().numpy()
            assert np.array_equal(a, b, equal_nan=a.dtype.kind == "f"), (h, f)
