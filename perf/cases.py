"""The calls that the tracker's speed is judged by, through the Python binding (ghc.py).

Every case is one call sequence of a user's program with its inputs in place:

track   p2c_device (P2C problems) and track on a batch of hypotheses, with or
        without the FP64 polish: what a RANSAC loop runs per batch, and, with
        one hypothesis, the latency that a single solve is quoted by.
mix     track_mix: four problems' batches in one launch (a server's uneven mix).
counts  count_results_device on a tracked batch's endpoints.
host    solve_host: host parameters in, host endpoints out, copies included.

Problems, precisions, step controls and batch sizes are those of the workloads,
the server and the tests; hypotheses come from the seeded scene generators.
"""
import math
import os
import sys

import numpy as np
import torch

PACKAGE = os.path.join(os.getcwd(), "homotopy-continuation-tracker-on-gpu_b200")
if PACKAGE not in sys.path:
    sys.path.insert(0, PACKAGE)

import ghc  # noqa: E402
import scenes  # noqa: E402

PRECISION = {"fp64": ghc.PREC_FP64, "fp32": ghc.PREC_FP32, "mixed": ghc.PREC_MIXED}
P3P, FIVE, GEN, CY, PH30 = ("P3P_TD", "5pt_rel_pos_alg_form_quat", "generalized_3views_4pts",
                            "uncalibrated_trifocal_rel_pos_CY", "trifocal_2op1p_30x30")
MIX = (P3P, FIVE, GEN, PH30)
# per problem: the largest batch of a case; steps and corrector iterations per path under the
# reference's step control (means over seeded batches), for work() alone
LARGEST = {P3P: 24000, FIVE: 4096, GEN: 512, CY: 128, PH30: 48}
STEPS = {P3P: (10, 15), FIVE: (8, 43), GEN: (12, 88), CY: (64, 164), PH30: (64, 128)}


def _track(name, problem, hyp, precision="fp64", polish=0, control="reference"):
    return {"name": name, "call": "track", "problem": problem, "hyp": hyp, "precision": precision, "polish": polish,
            "control": control}


def listed():
    return [
        # one minimal solve with its polish: latency, a few launches
        _track("p3p_one", P3P, 1, polish=2),
        # one solve of the headline problem in the reference's own precision: its quoted latency
        _track("gen_one_fp32", GEN, 1, precision="fp32"),
        # RANSAC on a cheap problem: many tiny systems
        _track("p3p_batch", P3P, 20000),
        # a server's batch of the uneven five-point system
        _track("five_batch", FIVE, 2048),
        # the headline batch
        _track("gen_batch", GEN, 512),
        # the headline's mixed-precision mode, ragged size, polished
        _track("gen_mixed", GEN, 251, precision="mixed", polish=2),
        # RANSAC on the uncalibrated trifocal problem, polished (bench config cy)
        _track("cy_batch", CY, 128, polish=2),
        # the largest system, in both of its modes
        _track("ph30_batch", PH30, 48),
        _track("ph30_mixed", PH30, 37, precision="mixed"),
        # four problems in one launch, in the proportions of the mix workload
        {"name": "mix", "call": "mix", "hyp": 16},
        # the result stage after the headline batch
        {"name": "gen_counts", "call": "counts", "problem": GEN, "hyp": 1024},
        # end to end from and to host memory, as the drop-in solver is called
        {"name": "five_host", "call": "host", "problem": FIVE, "hyp": 200, "precision": "fp64", "polish": 0},
    ]


def _size(rng, most):
    n = int(round(math.exp(rng.uniform(0.0, math.log(most)))))
    return max(1, min(most, n))


def draw(rng):
    call = rng.choice(["track"] * 8 + ["mix", "counts", "counts", "host"])
    if call == "mix":
        return {"call": "mix", "hyp": rng.randint(3, 16)}
    problem = rng.choice([P3P, FIVE, GEN, CY, PH30])
    if call == "counts":
        return {"call": "counts", "problem": problem, "hyp": _size(rng, 2 * LARGEST[problem])}
    precision = rng.choice(["fp64", "fp64", "fp32", "mixed"])
    polish = 0 if precision == "fp32" else rng.choice([0, 2])
    if call == "host":
        return {"call": "host", "problem": problem, "hyp": _size(rng, LARGEST[problem] // 4), "precision": precision,
                "polish": polish}
    control = "path_jump_free" if precision != "fp32" and rng.random() < 0.2 else "reference"
    # the path-jump-free control takes about eight times the steps
    most = LARGEST[problem] // (16 if control == "path_jump_free" else 4 if precision == "fp32" else 1)
    return {"call": "track", "problem": problem, "hyp": _size(rng, max(1, most)), "precision": precision,
            "polish": polish, "control": control}


def _targets(problem, hyp, seed, start, shipped):
    """(start [P+1], targets [hyp, P+1]): distinct seeded scenes, the larger P3P batches as samples
    with noise of at most 256 scenes (the scene generator is a Python loop)."""
    if problem != P3P or hyp <= 256:
        st, tg, _ = scenes.targets_for(problem, hyp, seed, start, shipped)
        return st, tg
    st, tg, _ = scenes.targets_for(problem, 256, seed, start, shipped)
    rng = np.random.default_rng(seed + 1)
    tg = tg[rng.integers(0, 256, size=hyp)]
    tg[:, :-1] *= 1.0 + 1e-3 * rng.normal(size=(hyp, tg.shape[1] - 1))
    return st, tg


def _cx(a, dtype=torch.float64):
    a = np.ascontiguousarray(np.asarray(a, dtype=np.complex128))
    return torch.view_as_real(torch.from_numpy(a)).to(dtype).cuda()


class _Bucket:
    """One problem's batch: its handle, inputs and output buffers."""

    def __init__(self, problem, hyp, seed, precision="fp64", polish=0, control="reference"):
        self.pb = ghc.Problem(problem)
        start, shipped = self.pb.params()
        start, tg = _targets(problem, hyp, seed, start, shipped)
        self.d_start, self.d_tg = _cx(start), _cx(tg)
        self.d_diff = self.d_tg - self.d_start
        prec = PRECISION[precision]
        self.sols = _cx(self.pb.start_sols(), torch.float32 if precision == "fp32" else torch.float64)
        self.ws = ghc.Workspace(self.pb, hyp, prec)
        self.kw = dict(polish_iters=polish)
        if control == "path_jump_free":
            self.kw.update(step=ghc.ROBUST_STEP, max_corr=3, max_steps=2000)

    def inputs(self):
        if self.pb.kind == ghc.KIND_P2C:
            hx, ht = self.pb.p2c_device(self.d_start, self.d_tg)
            return dict(d_coef_hx=hx, d_coef_ht=ht)
        return dict(d_p_start=self.d_start, d_p_target=self.d_tg, d_p_diff=self.d_diff)

    def outputs(self, inputs):
        w = self.ws
        out = dict(endpoints=w.endpoints, status=w.status, conv=w.conv, inf=w.inf, steps=w.steps, corr=w.corr,
                   t_end=w.t_end, dt_end=w.dt_end)
        if self.kw["polish_iters"]:
            out["resid"] = w.resid
        if "d_coef_hx" in inputs:
            out["hx"], out["ht"] = inputs["d_coef_hx"], inputs["d_coef_ht"]
        return out


def _paths(problem):
    return {P3P: 8, FIVE: 40, GEN: 583, CY: 668, PH30: 312}[problem]


def _unknowns(problem):
    return {P3P: 3, FIVE: 6, GEN: 12, CY: 12, PH30: 30}[problem]


class _Endpoints:
    """A tracked batch as the result stage finds it: 85 % converged, about 2 % of the paths on
    another path's root, a tenth of them real."""

    def __init__(self, problem, hyp, seed):
        g = torch.Generator(device="cuda").manual_seed(seed)
        self.paths, self.n_hyp, self.N = _paths(problem), hyp, _unknowns(problem)
        n = hyp * self.paths
        z = torch.randn((hyp, self.paths, self.N, 2), dtype=torch.float64, device="cuda", generator=g)
        real = torch.rand((hyp, self.paths), device="cuda", generator=g) < 0.1
        z[..., 1] *= torch.where(real, 1e-9, 1.0)[..., None]
        if self.paths > 1:
            dup = torch.rand((hyp, self.paths), device="cuda", generator=g) < 0.02
            other = torch.randint(0, self.paths, (hyp, self.paths), device="cuda", generator=g)
            z = torch.where(dup[..., None, None], torch.gather(z, 1, other[..., None, None].expand_as(z)) + 1e-9, z)
        self.endpoints = z.reshape(n, self.N, 2).contiguous()
        u = torch.rand(n, device="cuda", generator=g)
        self.conv = (u < 0.85).to(torch.uint8)
        self.inf = (u > 0.95).to(torch.uint8)


def _mix_sizes(hyp):
    """Hypotheses per problem of the mix workload's 8192 : 4096 : 2048 : 1024."""
    return (8 * hyp, 4 * hyp, 2 * hyp, hyp)


def prepare(case, seed):
    call = case["call"]
    if call == "track":
        return dict(call=call, b=_Bucket(case["problem"], case["hyp"], seed, case["precision"], case["polish"],
                                         case["control"]))
    if call == "mix":
        return dict(call=call, b=[_Bucket(p, h, seed + i) for i, (p, h) in enumerate(zip(MIX, _mix_sizes(case["hyp"])))])
    if call == "counts":
        return dict(call=call, b=_Endpoints(case["problem"], case["hyp"], seed))
    pb = ghc.Problem(case["problem"])
    start, shipped = pb.params()
    _, tg = _targets(case["problem"], case["hyp"], seed, start, shipped)
    return dict(call=call, pb=pb, tg=tg, out=ghc.solve_outputs(pb, case["hyp"]),
                kw=dict(precision=PRECISION[case["precision"]], polish_iters=case["polish"]))


def run(state):
    if state["call"] == "track":
        b = state["b"]
        inputs = b.inputs()
        ghc.track(b.pb, b.ws, b.sols, **inputs, **b.kw)
        return b.outputs(inputs)
    if state["call"] == "mix":
        ins = [b.inputs() for b in state["b"]]
        ghc.track_mix([(b.pb, b.ws, b.sols, dict(i, **b.kw)) for b, i in zip(state["b"], ins)])
        return [b.outputs(i) for b, i in zip(state["b"], ins)]
    if state["call"] == "counts":
        counts, cls = ghc.count_results_device(state["b"], state["b"].N, want_class=True)
        return dict(counts=counts, cls=cls)
    o = ghc.solve_host(state["pb"], targets=state["tg"], out=state["out"], **state["kw"])
    return {k: o[k] for k in ("endpoints", "status", "conv", "inf", "steps")}


def _track_work(problem, hyp, precision="fp64", polish=0, control="reference"):
    """Bytes in and out, and the flops of the evaluations and solves at the mean step counts."""
    pb = ghc.Problem(problem)
    N, paths = pb.N, pb.paths
    n = hyp * paths
    real = 4 if precision == "fp32" else 8
    if pb.kind == ghc.KIND_P2C:
        table = 16 * (pb.M + 1) * (2 * pb.K + 1)
        coef = (pb.M + 1) * 4 * (2 * pb.K - 1)
    else:
        table = 2 * 16 * (pb.P + 1)
        coef = 6 * (pb.P + 1)
    fixed = 8 * N ** 3 / 3 + 8 * N ** 2
    hx = pb.n_hx_terms * (6 * (pb.Px - 2) + 4)
    ht = pb.n_ht_terms * (6 * (pb.Pt - 2) + 4)
    s, c = STEPS[problem]
    if control == "path_jump_free":
        s, c = 8 * s, 8 * c
    flops = n * (4 * s * (coef + hx + ht + fixed) + (c + polish) * (hx + ht + fixed))
    # inputs, endpoints, flags, counters, t and dt, residuals; the coefficient tables are an output of
    # p2c_device and an input of track
    moved = hyp * (16 * (pb.P + 1) + 2 * table) + paths * N * 2 * real
    moved += n * (2 * N * real + 3 + 8 + 16 + (8 if polish else 0))
    return {"bytes": moved, "flops": flops}


def work(case):
    call = case["call"]
    if call == "track":
        return _track_work(case["problem"], case["hyp"], case["precision"], case["polish"], case["control"])
    if call == "host":
        return _track_work(case["problem"], case["hyp"], case["precision"], case["polish"])
    if call == "mix":
        w = [_track_work(p, h) for p, h in zip(MIX, _mix_sizes(case["hyp"]))]
        return {k: sum(x[k] for x in w) for k in ("bytes", "flops")}
    paths, N = _paths(case["problem"]), _unknowns(case["problem"])
    n = case["hyp"] * paths
    # every pair of a hypothesis is told apart by its first component in nearly all cases
    return {"bytes": n * (16 * N + 3) + 16 * case["hyp"], "flops": n * (N + 2 * paths)}


def _p2c_terms(problem):
    rows = [line.split() for line in open(os.path.join(ghc.PROBLEMS, problem, "p2c_terms.txt"))
            if line.strip() and not line.startswith("#")]
    M, K = int(rows[0][0]), int(rows[0][1])
    return M, K, [(int(r[0]), int(r[1]) / int(r[2]), [int(j) for j in r[4:4 + int(r[3])]]) for r in rows[1:]]


def _p2c_exact(problem, hyp, seed):
    """c_k(q + t (p - q)) expanded in t, and its derivative, in complex128."""
    pb = ghc.Problem(problem)
    start, shipped = pb.params()
    q, p = _targets(problem, hyp, seed, start, shipped)
    d = p - q[None, :]
    M, K, terms = _p2c_terms(problem)
    hx = np.zeros((hyp, M + 1, K + 1), dtype=np.complex128)
    for k, scale, factors in terms:
        poly = np.zeros((hyp, K + 1), dtype=np.complex128)
        poly[:, 0] = scale
        for j in factors:
            nxt = poly * q[j]
            nxt[:, 1:] += poly[:, :-1] * d[:, j:j + 1]
            poly = nxt
        hx[:, k] += poly
    hx[:, M, 0] = 1.0
    ht = hx[:, :, 1:] * np.arange(1, K + 1)
    ht[:, M] = 0.0
    ht[:, M, 0] = 1.0
    return {k: torch.view_as_real(torch.from_numpy(np.ascontiguousarray(v.reshape(hyp, -1))))
            for k, v in (("hx", hx), ("ht", ht))}


def exact(case, seed):
    """The coefficient tables in 64 bits.  A tracked endpoint has no value apart from the tracker's
    own arithmetic: under the reference's step control a path may jump, and which root it ends on
    (with its flags and counters) turns on the last bit."""
    if case["call"] == "mix":
        every = [(p, h, seed + i) for i, (p, h) in enumerate(zip(MIX, _mix_sizes(case["hyp"])))]
        return [None if p == PH30 else _p2c_exact(p, h, s) for p, h, s in every]
    if case["call"] == "track" and case["problem"] != PH30:
        return _p2c_exact(case["problem"], case["hyp"], seed)
    return None
