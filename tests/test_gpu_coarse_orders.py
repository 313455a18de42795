"""The dense coarse problems at the edges of their tiles: inverses of order 1,
63, 64, 65, 128, 130 and 192 (64-wide panels), the level-3 eigensolve with blocks
of 6, 12 and 16 columns (tensor-core launches) and 18 and 20 (one CTA per rank),
one rank and ragged ranks, a floating rank included.

Level-3 eigenvalues and the preconditioner at 1e-6 against the oracle's level 2
and 3 on the basis that the library computed, so that the local eigensolver's
tolerance is not part of the difference; a block iteration of this kind
needs some tens of steps, so 100 of the 500 allowed mean that it stalled."""
import numpy as np
import pytest

from oracle import pmf_oracle as O
from premixfem_b200 import fields
from premixfem_b200.solver import DarcySolver, options_string

pytestmark = pytest.mark.gpu

CASES = {
    "n1": ((6, 5, 4), (1, 1, 1), (2, 1, 1), 1, 1),
    "n63": ((15, 15, 6), (3, 3, 1), (1, 1, 1), 7, 2),
    "n64": ((16, 16, 16), (4, 4, 4), (1, 1, 1), 1, 4),
    "n65": ((52, 4, 4), (13, 1, 1), (1, 1, 1), 5, 6),
    "n66_wide": ((44, 4, 4), (11, 1, 1), (1, 1, 1), 6, 7),
    "n128": ((16, 16, 8), (4, 4, 2), (1, 1, 1), 4, 4),
    "n130": ((52, 8, 4), (13, 2, 1), (1, 1, 1), 5, 4),
    "n192_wide": ((16, 16, 16), (4, 4, 4), (1, 1, 1), 3, 8),
    "ragged": ((22, 18, 10), (2, 2, 2), (2, 2, 1), 5, 4),
}


@pytest.mark.parametrize("contrast", [1.0, 4.0])
@pytest.mark.parametrize("name", list(CASES))
def test_coarse_orders(native, monkeypatch, name, contrast):
    mesh, sd, vr, k, en2 = CASES[name]
    prob = fields.random_box(mesh, seed=3, sigma=contrast, dirichlet={"x-": 1.0})
    op = O.Operator(prob)
    s = DarcySolver.from_problem(prob, options_string({"pmf_sd": sd, "pmf_vranks": vr, "en_lv1": k, "en_lv2": en2}))
    s.setup()
    phi = s.phi()

    def basis(op, box, o):
        V = phi[O.box_cells(op.mesh, box)]
        return np.zeros(k), V, k, 0.0

    monkeypatch.setattr(O, "local_basis", basis)
    pc = O.Preconditioner(op, O.Options(sd=sd, vranks=vr, en_lv1=k, en_lv2=en2))
    ev, _, its = s.eigen_lv2()
    assert np.max(its) <= 100
    ref = np.stack(list(pc.eigvals_lv2))
    # a rank of one unknown has the eigenvalue zero alone: its scale is the coarse matrix's
    scale = np.maximum(np.abs(ref).max(axis=1, keepdims=True), 1e-3 * np.abs(pc.A2full).max())
    assert (np.abs(ev - ref) / np.maximum(np.abs(ref), 1e-3 * scale)).max() <= 1e-6
    x = np.random.default_rng(2).standard_normal(op.n)
    y, yr = s.pc_apply(x), pc.apply(x)
    s.close()
    assert np.linalg.norm(y - yr) <= 1e-6 * np.linalg.norm(yr)


@pytest.mark.parametrize("contrast", [1.0, 4.0])
def test_floating_ranks_of_one_unknown(native, monkeypatch, contrast):
    """64 ranks of one unknown, most of them floating: their 1 x 1 matrix is the rounding of zero, of either sign, and
    its inverse may drop it as null.  The bars of the test above."""
    monkeypatch.setitem(CASES, "floating", ((16, 16, 16), (1, 1, 1), (4, 4, 4), 1, 1))
    test_coarse_orders(native, monkeypatch, "floating", contrast)


@pytest.mark.parametrize("contrast", [1.0, 4.0])
@pytest.mark.parametrize("vr,en2", [((2, 2, 2), 8), ((3, 3, 3), 8), ((3, 3, 3), 10)])
def test_wide_blocks_of_floating_ranks(native, monkeypatch, vr, en2, contrast):
    """Blocks of 20 and 24 columns on ranks of 36 unknowns, most of which touch no Dirichlet face; the bars of the test
    above."""
    monkeypatch.setitem(CASES, "floating", (tuple(v * n for v, n in zip(vr, (6, 6, 2))), (3, 3, 1), vr, 4, en2))
    test_coarse_orders(native, monkeypatch, "floating", contrast)


@pytest.mark.parametrize("case", [((16, 16, 16), (1, 1, 1), (8, 8, 8), 4, 3), ((48, 24, 8), (3, 3, 1), (8, 4, 4), 4, 8)],
                         ids=["512_ranks_of_4", "128_ranks_of_36"])
def test_many_ranks(native, monkeypatch, case):
    """Level-3 problems of 1 536 and 1 024 unknowns, solved in launches of their own; the bars of the test above."""
    monkeypatch.setitem(CASES, "many", case)
    test_coarse_orders(native, monkeypatch, "many", 1.0)


def test_cost_of_many_ranks(native):
    """4 096 ranks of one subdomain each: the level-3 inverse, 537 MB, is streamed once an iteration (about 0.1 ms), not
    once for every group of rows."""
    s = DarcySolver.from_problem(fields.random_box((128, 128, 128), seed=3), options_string({
        "sd": 1, "pmf_vranks": (16, 16, 16), "en_lv1": 4, "en_lv2": 2, "pmf_precision": "mixed", "pmf_eig_max_it": 2}))
    s.setup()
    s.profile_iteration(5)
    ms = s.profile_iteration(20)["coarse"][0]
    s.close()
    assert ms <= 0.7, ms


@pytest.mark.parametrize("contrast", [1.0, 4.0])
@pytest.mark.parametrize("case", [((16, 4, 4), (4, 1, 1), (1, 1, 1), 4, 16), ((24, 16, 8), (3, 1, 1), (2, 2, 2), 4, 12),
                                  ((24, 12, 12), (3, 1, 1), (3, 3, 3), 3, 9), ((24, 24, 8), (4, 1, 1), (2, 2, 1), 4, 10)],
                         ids=["16_of_16", "12_of_12", "9_of_9", "10_of_16"])
def test_most_of_a_small_rank(native, monkeypatch, case, contrast):
    """More than eight wanted vectors in blocks of at most 16: all or most of the ranks' spaces, floating ranks among
    them; the bars of the test above."""
    monkeypatch.setitem(CASES, "small", case)
    test_coarse_orders(native, monkeypatch, "small", contrast)
