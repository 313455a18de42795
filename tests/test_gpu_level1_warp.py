"""The level-1 solve by one warp per subdomain (k_ic_warp, the tuner's last
candidate, forced by PMF_TUNE_FORCE) against the natural-order kernel
(candidate 0): the preconditioner application agrees to 1e-12 in FP64 and 1e-5
in mixed precision (the same operations; products of the backward sweep are
rounded before they are added), PCG takes the same iterations (+-1).

Shapes: full and partial lanes (ny times the planes per group 32, 30, 26, 20),
one plane per group (ny above 16, or lines of 4 cells), a last group with
fewer planes, lines longer than a batch of steps and not a multiple of it,
ragged boxes, several visits a cycle."""
import numpy as np
import pytest

from premixfem_b200 import fields
from premixfem_b200.solver import DarcySolver, options_string

pytestmark = pytest.mark.gpu

CASES = {
    "16x16x16": ((32, 32, 32), (2, 2, 2), ""),
    "8x8x8": ((16, 16, 16), (2, 2, 2), "-si_lv1 2"),
    "10x10x5": ((20, 20, 10), (2, 2, 2), ""),
    "13x13x7": ((26, 26, 14), (2, 2, 2), "-use_W_cycle"),
    "ragged": ((13, 11, 9), (2, 2, 2), ""),
    "ny20": ((10, 40, 10), (2, 2, 2), ""),
    "ny32": ((16, 64, 8), (2, 2, 2), ""),
    "nx4": ((8, 16, 10), (2, 2, 2), ""),
    "nx21": ((42, 12, 14), (2, 2, 2), ""),
    "nx3": ((6, 8, 8), (2, 2, 2), ""),  # too short: the natural kernel either way
}


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("name", list(CASES))
def test_warp_level1_matches_natural(native, monkeypatch, name, precision):
    mesh, sd, extra = CASES[name]
    prob = fields.random_box(mesh, seed=7, sigma=1.5)
    x = np.random.default_rng(3).standard_normal(int(np.prod(mesh)))
    out = []
    for force in ("0", "100"):
        monkeypatch.setenv("PMF_TUNE_FORCE", force)
        s = DarcySolver.from_problem(prob, options_string({"pmf_sd": sd, "en_lv1": 3, "en_lv2": 2,
                                                           "pmf_precision": precision}) + " " + extra)
        s.setup()
        y = s.pc_apply(x)
        _, its, _, reason = s.solve(s.rhs(prob["source"].ravel()))
        s.close()
        assert reason == "converged"
        out.append((y, its))
    rel = np.linalg.norm(out[1][0] - out[0][0]) / np.linalg.norm(out[0][0])
    assert rel <= (1e-12 if precision == "fp64" else 1e-5), rel
    assert abs(out[0][1] - out[1][1]) <= 1


def test_no_room_for_the_step_ordered_factor(native, monkeypatch):
    """The factor's copy is this kernel's alone: where it does not fit beside what the other kernels need, one of them
    runs.  118 MB of copy for 3.3 million FP64 cells, 16 MB left (and what the stream-ordered pools give back)."""
    import torch
    prob = fields.random_box((160, 160, 128), seed=7, sigma=1.5)

    def solve(kernel):
        s = DarcySolver.from_problem(prob, options_string({"pmf_sd": (10, 10, 8), "en_lv1": 3, "en_lv2": 2,
                                                           "pmf_lv1_kernel": kernel}))
        s.setup()
        its = s.solve(s.rhs(prob["source"].ravel()))[1]
        used = free - torch.cuda.mem_get_info()[0]
        s.close()
        return its, used

    monkeypatch.setenv("PMF_TUNE_FORCE", "100")
    free = torch.cuda.mem_get_info()[0]
    solve("natural")  # warms the pools
    free = torch.cuda.mem_get_info()[0]
    its, used = solve("natural")
    its_warp, used_warp = solve("auto")
    assert used_warp - used > 100 << 20
    hog = torch.empty(torch.cuda.mem_get_info()[0] - used - (16 << 20), dtype=torch.uint8, device="cuda")
    free = torch.cuda.mem_get_info()[0]
    try:
        assert abs(solve("auto")[0] - its) <= 1
    finally:
        del hog
        torch.cuda.empty_cache()
    assert abs(its_warp - its) <= 1


@pytest.mark.parametrize("tile,offered", [((4, 4, 4), False), ((4, 8, 8), False), ((8, 8, 8), True)],
                         ids=lambda v: "x".join(map(str, v)) if isinstance(v, tuple) else str(v))
def test_idle_lanes_take_no_memory(native, monkeypatch, tile, offered):
    """A shape that leaves most of a warp's lanes idle would fill its factor's copy with nothing: it is not offered."""
    import torch
    monkeypatch.setenv("PMF_TUNE_FORCE", "100")
    mesh = tuple(64 for _ in tile)
    prob = fields.random_box(mesh, seed=7, sigma=1.0)
    used = []
    for kernel in ("natural", "natural", "auto"):  # the first one warms the pools
        free = torch.cuda.mem_get_info()[0]
        s = DarcySolver.from_problem(prob, options_string({
            "pmf_vranks": (2, 2, 2), "pmf_sd": tuple(32 // t for t in tile), "en_lv1": 2, "en_lv2": 2,
            "pmf_lv1_kernel": kernel}))
        s.setup()
        used.append(free - torch.cuda.mem_get_info()[0])
        s.close()
    # 262 144 cells: 1.6 entries of 32 bytes a cell are 13 MB, 4.9 and 9.5 are 41 and 80; cudaMalloc's blocks are 2 MB
    assert (used[2] - used[1] > 8 << 20) == offered
