"""Coefficient tables and parameters at 8-byte addresses (needs a B200): the tracker loads whole complex
values only where they are aligned to 16 bytes, and must give the same bits from an odd address, at
every degree of the coefficient polynomials (K = 1, 2 with their own loads, 3 and 4 without) and for
the parameter homotopy."""
import numpy as np
import pytest

import ghc
import scenes

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


def _odd(t):
    """A copy of t that starts 8 bytes past a 16-byte boundary."""
    flat = torch.empty(t.numel() + 3, dtype=t.dtype, device=t.device)
    at = 1 if flat.data_ptr() % 16 == 0 else 0
    out = flat[at:at + t.numel()].view(t.shape)
    out.copy_(t)
    assert out.data_ptr() % 16 == 8
    return out


def _cx(a, dtype=torch.float64):
    return torch.view_as_real(torch.from_numpy(np.ascontiguousarray(a, dtype=np.complex128))).to(dtype).cuda()


@pytest.mark.parametrize("prec", [ghc.PREC_FP64, ghc.PREC_FP32, ghc.PREC_MIXED])
@pytest.mark.parametrize("name", ["P3P_TD", "generalized_3views_4pts", "distorted_2view_triangulation",
                                  "dual_reciever_TDOA_5pt", "trifocal_2op1p_30x30"])
def test_odd_addresses_give_the_same_bits(name, prec):
    pb = ghc.Problem(name)
    s, t = pb.params()
    st, tg, _ = scenes.targets_for(name, 2, 3, s, t)
    d_st, d_tg = _cx(st), _cx(tg)
    if pb.kind == ghc.KIND_P2C:
        hx, ht = pb.p2c_device(d_st, d_tg)
        kw = dict(d_coef_hx=hx, d_coef_ht=ht)
    else:
        kw = dict(d_p_start=d_st, d_p_target=d_tg, d_p_diff=(d_tg - d_st).contiguous())
    sols = _cx(pb.start_sols(), torch.float32 if prec == ghc.PREC_FP32 else torch.float64)
    runs = []
    for move in (lambda v: v, _odd):
        ws = ghc.Workspace(pb, 2, prec)
        ghc.track(pb, ws, sols, max_steps=30, **{k: move(v) for k, v in kw.items()})
        runs.append(ws)
    for f in ("endpoints", "status", "steps", "corr", "t_end", "dt_end"):
        a, b = (getattr(r, f).cpu().numpy() for r in runs)
        assert np.array_equal(a, b, equal_nan=a.dtype.kind == "f"), f
