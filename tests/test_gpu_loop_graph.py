"""The CG loop as a graph that repeats itself on the device, against the same
launches without a graph: the same bits, iterations and stop reason for every
solution buffer, after a new set-up, at every stop code that a right-hand side
or the iteration limit can bring, and for a batch."""
import numpy as np
import pytest

from premixfem_b200 import fields
from premixfem_b200.solver import BatchSolver, DarcySolver

pytestmark = pytest.mark.gpu


@pytest.fixture(autouse=True)
def _one_launch_shape(monkeypatch):
    monkeypatch.setenv("PMF_TUNE_FORCE", "0")  # the same bits from every solver


OPTS = "-pmf_sd 3,2,2 -en_lv1 3 -en_lv2 2 -ksp_rtol 1e-10 -pmf_precision mixed"


def _fields(seed):
    return fields.random_box((21, 16, 18), seed=seed, sigma=1.5, dirichlet={"x-": 1.0})


def _run(extra, device=True):
    import torch
    out = []
    s = DarcySolver.from_problem(_fields(1), OPTS + extra)
    keep = []
    for seed in (1, 2):
        prob = _fields(seed)
        k = [np.ascontiguousarray(q).ravel() for q in prob["kappa"]]
        s.set_kappa(*k)
        s.setup()
        b = s.rhs(prob["source"].ravel())
        zero, bad = np.zeros_like(b), b.copy()
        bad[7] = np.nan
        for rhs in (b, 2.0 * b, zero, bad, b):
            if device:
                keep.append(torch.full((b.size + 1,), 3.0, dtype=torch.float64, device="cuda"))
                x, its, rn, reason = s.solve(torch.from_numpy(rhs).cuda(), out=keep[-1][:-1])
                x = x.cpu().numpy()
            else:
                x, its, rn, reason = s.solve(rhs)
            out.append((x, its, rn, reason))
    s.close()
    return out


@pytest.mark.parametrize("extra", ["", " -pmf_pcg_chunk 2", " -ksp_max_it 3", " -ksp_max_it 4", " -ksp_max_it 5",
                                   " -ksp_constant_null_space -ksp_max_it 30", " -use_W_cycle"])
@pytest.mark.parametrize("device", [True, False])
def test_loop_graph_matches_launches(native, extra, device):
    a, b = _run(extra, device), _run(extra + " -pmf_pcg_graph 0", device)
    assert len({r for _, _, _, r in a}) >= 2
    for (xa, ia, ra, fa), (xb, ib, rb, fb) in zip(a, b):
        assert (ia, fa) == (ib, fb)
        assert ra == rb or (np.isnan(ra) and np.isnan(rb))
        assert np.array_equal(xa, xb, equal_nan=True)


def test_misaligned_solution(native):
    """A solution buffer at an odd element takes one cell per load: sums in another order."""
    import torch
    prob = _fields(1)
    s = DarcySolver.from_problem(prob, OPTS)
    s.setup()
    b = torch.from_numpy(s.rhs(prob["source"].ravel())).cuda()
    x, its, _, _ = s.solve(b)
    buf = torch.empty(b.numel() + 1, dtype=torch.float64, device="cuda")
    y, its2, _, reason = s.solve(b, out=buf[1:])
    s.close()
    assert reason == "converged" and abs(its - its2) <= 1
    assert float((x - y).norm() / x.norm()) <= 1e-8


def test_batch_loop_graph(native):
    import torch
    batch = fields.grf_batch(count=3, seed=5, lo=9, hi=20)
    problems = [p for p, _ in batch]
    res = []
    for extra in ("", " -pmf_pcg_graph 0"):
        s = BatchSolver(problems, [fields.tiles(p["mesh"]) for p in problems], "-en_lv1 4 -en_lv2 4" + extra)
        s.set_kappa_problems(problems)
        s.setup()
        outs = []
        for j in range(2):
            b = torch.from_numpy(s.rhs(s.pack([srcs[j] for _, srcs in batch]))).cuda()
            buf = torch.empty_like(b)
            x, its, rn, reasons = s.solve(b, out=buf)
            outs.append((x, list(its), list(rn), list(reasons)))
        res.append([(x.cpu().numpy(), i, r, f) for x, i, r, f in outs])
        s.close()
    for (xa, ia, ra, fa), (xb, ib, rb, fb) in zip(*res):
        assert (ia, ra, fa) == (ib, rb, fb) and np.array_equal(xa, xb)
