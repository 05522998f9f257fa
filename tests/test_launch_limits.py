"""Launches of more paths than the 32-bit work counter numbers are refused before any device work (no
GPU; the pointers below are never used)."""
import ctypes

import pytest

import ghc

ERR_RANGE = -4


def _args(n_hyp, paths=0):
    a = ghc.TrackArgs()
    a.n_hyp, a.paths, a.precision = n_hyp, paths, ghc.PREC_FP64
    a.d_start_sols = a.d_endpoints = a.d_coef_hx = a.d_coef_ht = a.d_counter = 256
    return a


def _calls(pb, a):
    yield "track", lambda: ghc.ghc_track(pb.h, ctypes.byref(a), None)
    yield "track_noalloc", lambda: ghc.ghc_track_noalloc(pb.h, ctypes.byref(a), None)
    yield "track_mix", lambda: ghc.ghc_track_mix((ctypes.c_void_p * 1)(pb.h), ctypes.byref(a), 1, None)


@pytest.mark.parametrize("n_hyp,paths", [((1 << 29) + 1, 0), ((1 << 32) + 1, 1), (1 << 62, 0), ((1 << 33), 8)])
def test_more_than_2_to_the_32_paths_are_refused(n_hyp, paths):
    pb = ghc.Problem("P3P_TD")  # 8 paths
    for name, call in _calls(pb, _args(n_hyp, paths)):
        assert call() == ERR_RANGE, name
        assert b"2^32" in ghc.ghc_last_error(), name
    if paths == 0:
        assert ghc.ghc_solve_host(pb.h, ghc.PREC_FP64, n_hyp, 256, 1.0, 0, 256, None, None, None, None,
                                  None) == ERR_RANGE
    assert pb.bound_device() == -1
