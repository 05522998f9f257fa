"""The device LU's column groups vs the oracle, bit for bit (needs a B200): a zero pivot, or a NaN in
a row below it, at every column -- the first, middle and last of each group -- in batches where the
warp's other systems are regular and go on eliminating the column that one of them skips."""
import numpy as np
import pytest

import ghc
import oracle as O
from lu_cases import SIZES
from test_gpu_lu import cx_t

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("prec", [ghc.PREC_FP64, ghc.PREC_FP32])
@pytest.mark.parametrize("N", [n for n in SIZES if n > 3])
def test_skipped_column_in_every_place(N, prec):
    rng = np.random.default_rng(N)
    tt = torch.float64 if prec == ghc.PREC_FP64 else torch.float32
    systems = []
    for i in range(N):
        for odd in ("zero", "nan", None):
            A = rng.normal(size=(N, N)) + 1j * rng.normal(size=(N, N))
            if odd == "zero":
                A[:, i] = 0
            elif odd == "nan":
                A[N - 1, i] = complex(np.nan, 0.5)
            systems.append((A.astype(np.complex64).astype(np.complex128),
                            (rng.normal(size=N) + 1j * rng.normal(size=N)).astype(np.complex64).astype(np.complex128)))
    z = ghc.lu_solve_device(cx_t([a for a, _ in systems], tt), cx_t([b for _, b in systems], tt), prec)
    z = z.double().cpu().numpy()
    z = z[..., 0] + 1j * z[..., 1]
    for s, (a, b) in enumerate(systems):
        ref = O.lu_solve(a, b, "d" if prec == ghc.PREC_FP64 else "f")
        assert np.array_equal(z[s], ref, equal_nan=True), (N, s)
