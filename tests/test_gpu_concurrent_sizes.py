"""Two host threads that launch one kernel with different shared-memory sizes (needs a B200): neither
may take the other's limit away, so every call is accepted and gives what it gives alone."""
import threading

import numpy as np
import pytest

import ghc
import scenes
from test_gpu_results import _WS
from test_gpu_spread import _cx

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


def _run_together(calls, rounds):
    """Each call `rounds` times on its own thread and stream; raises what a call raised."""
    failed = []
    start = threading.Barrier(len(calls))

    def loop(call):
        try:
            with torch.cuda.stream(torch.cuda.Stream()):
                start.wait(60)
                for _ in range(rounds):
                    call()
                torch.cuda.current_stream().synchronize()
        except Exception as e:  # noqa: BLE001 (reported by the test's own thread)
            failed.append(e)

    threads = [threading.Thread(target=loop, args=(c,)) for c in calls]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not failed, failed[0]


def test_result_counts_of_two_sizes():
    rng = np.random.default_rng(3)
    calls, expect, got = [], [], []
    for paths in (3071, 5344):
        z = rng.normal(size=(1, paths, 3)) + 1j * rng.normal(size=(1, paths, 3))
        z[0, 1::7] = z[0, 0]
        ws = _WS(z, np.ones((1, paths), bool), np.zeros((1, paths), bool))
        out = torch.zeros((1, 4), dtype=torch.int32, device="cuda")
        host = ghc.count_results(z[0], ws.conv.cpu().numpy(), ws.inf.cpu().numpy())
        expect.append([host["converged"], host["real"], host["infinity"], host["unique"]])
        got.append(out)
        calls.append(lambda ws=ws, out=out: ghc.count_results_device(ws, 3, out=out))
    torch.cuda.synchronize()
    _run_together(calls, 3000)
    assert [o.cpu().numpy()[0].tolist() for o in got] == expect


def test_polish_of_two_problems():
    calls, spaces, alone = [], [], []
    for name in ("distorted_2view_triangulation", "dual_reciever_TDOA_5pt"):  # one polish kernel, 24 and 85 coefficients
        pb = ghc.Problem(name)
        s, t = pb.params()
        st, tg, _ = scenes.targets_for(name, 1, 5, s, t)
        hx, ht = pb.p2c_device(_cx(st), _cx(tg))
        sols, ws = _cx(pb.start_sols()), ghc.Workspace(pb, 1, ghc.PREC_FP64)
        call = lambda pb=pb, ws=ws, sols=sols, hx=hx, ht=ht: ghc.track(  # noqa: E731
            pb, ws, sols, d_coef_hx=hx, d_coef_ht=ht, max_steps=2, polish_iters=1)
        call()
        alone.append(ws.endpoints.cpu().numpy().copy())
        spaces.append(ws)
        calls.append(call)
    torch.cuda.synchronize()
    _run_together(calls, 3000)
    for ws, a in zip(spaces, alone):
        assert np.array_equal(ws.endpoints.cpu().numpy(), a, equal_nan=True)
