"""Problems whose term words and path buffers fill a CTA's shared memory (needs a B200): what the
tables leave free holds a path's buffers with two pivot rows, not with all of them, and in mixed precision not
the second form of the H words either.  They are tracked all the same, and equal the oracle bit for bit, at
sizes with four, two and one path in the smallest CTA."""
import numpy as np
import pytest

import ghc
import oracle as O

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

K, COEFS, PATHS, HYP = 1, 20, 3, 2


def _rows(rng, n, N):
    """n terms: scale, coefficient, six variables (mostly the constant N; more than the balanced walk takes)."""
    parts = 8
    t = np.full((n, parts), N, dtype=np.int64)
    t[:, 0] = rng.choice([-2, -1, 1, 2], n)
    t[:, 1] = rng.integers(0, COEFS, n)
    some = rng.random((n, parts - 2)) < 0.25
    t[:, 2:][some] = rng.integers(0, N, int(some.sum()))
    return t


def _write(root, N, Tx, Tt, columns):
    """A problem folder whose H_x rows have `columns` columns of Tx terms and whose H rows have Tt terms."""
    rng = np.random.default_rng(N)
    name = "LARGE_%d" % N
    d = root / name
    d.mkdir()
    (d / "gpuhc_settings.yaml").write_text(
        "problem_name: %s\nGPUHC_Type: P2C\nGPUHC_Max_Steps: 3\nGPUHC_Max_Correction_Steps: 3\n"
        "GPUHC_Num_Of_Steps_to_Increase_Delta_t: 2\nNum_Of_Vars: %d\nNum_Of_Params: %d\nNum_Of_Tracks: %d\n"
        "dHdx_Max_Terms: %d\ndHdx_Max_Parts: 8\ndHdt_Max_Terms: %d\ndHdt_Max_Parts: 8\nMax_Order_Of_T: %d\n"
        "Num_Of_Coeffs_From_Params: %d\n" % (name, N, COEFS, PATHS, Tx, Tt, K, COEFS))
    pairs = "".join("%.3f %.3f\n" % (a, b) for a, b in rng.normal(size=(COEFS, 2)))
    (d / "start_params.txt").write_text(pairs)
    (d / "target_params.txt").write_text(pairs)
    (d / "start_sols.txt").write_text("".join("%.4f %.4f\n" % (a, b) for a, b in 0.3 * rng.normal(size=(N * PATHS, 2))))
    hx = np.zeros((N, N, Tx, 8), dtype=np.int64)
    for r in range(N):
        for c in range(columns):
            hx[r, (r + c) % N] = _rows(rng, Tx, N)
    ht = _rows(rng, N * Tt, N)
    (d / "dHdx_indx.txt").write_text(" ".join(map(str, hx.reshape(-1).tolist())) + "\n")
    (d / "dHdt_indx.txt").write_text(" ".join(map(str, ht.reshape(-1).tolist())) + "\n")
    return name


def _cx(a, dtype=torch.float64):
    return torch.view_as_real(torch.from_numpy(np.ascontiguousarray(a, dtype=np.complex128))).to(dtype).cuda()


# (N, terms per H_x entry, H_x entries per row, terms per row of H)
LARGE = [(5, 800, 5, 1660), (16, 100, 16, 160), (18, 360, 2, 845)]


@pytest.mark.parametrize("prec", [ghc.PREC_FP64, ghc.PREC_FP32, ghc.PREC_MIXED])
@pytest.mark.parametrize("N,Tx,columns,Tt", LARGE)
def test_tables_that_fill_a_cta(tmp_path, N, Tx, columns, Tt, prec):
    name = _write(tmp_path, N, Tx, Tt, columns)
    pb, ob = ghc.Problem(name, root=str(tmp_path)), O.Problem(name, root=str(tmp_path))
    rng = np.random.default_rng(7)
    # (single-precision values, so that every precision and the oracle start from the same numbers)
    draw = lambda *shape: (0.1 * (rng.normal(size=shape) + 1j * rng.normal(size=shape))).astype(np.complex64).astype(  # noqa: E731
        np.complex128)
    hx, ht = draw(HYP, (COEFS + 1) * (K + 1)), draw(HYP, (COEFS + 1) * K)
    sols = ob.start_sols.astype(np.complex64).astype(np.complex128)
    d_sols = _cx(sols, torch.float32 if prec == ghc.PREC_FP32 else torch.float64)
    ws = ghc.Workspace(pb, HYP, prec)
    polish = 0 if prec == ghc.PREC_FP32 else 1
    ghc.track(pb, ws, d_sols, polish_iters=polish, d_coef_hx=_cx(hx), d_coef_ht=_cx(ht))
    ref = O.track(ob, sols, precision={ghc.PREC_FP64: "d", ghc.PREC_FP32: "f", ghc.PREC_MIXED: "mixed"}[prec],
                  polish_iters=polish, hx=hx, ht=ht)
    for f in ("conv", "inf", "status", "steps", "corr", "t_end"):
        assert np.array_equal(getattr(ws, f).cpu().numpy(), ref[f]), f
    z = ws.endpoints.double().cpu().numpy()
    z = z[..., 0] + 1j * z[..., 1]
    fin = np.isfinite(ref["endpoints"])
    assert np.array_equal(np.isfinite(z), fin) and np.array_equal(z[fin], ref["endpoints"][fin])
    assert fin.any()
