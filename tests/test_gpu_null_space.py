"""-ksp_constant_null_space on the GPU against the oracle.

With the option, PETSc's CG removes the operator's constant null space from
every preconditioned residual (KSP_PCApply -> MatNullSpaceRemove); the
right-hand side is not projected.  The case is the reference's own test.c
problem (src/test.c:7-38): constant k = (2, 1, 0.5), the well source, no
Dirichlet face, so A is singular.  Parity bars as for the other PCG tests:
iterations within +-1 of the oracle with the same option, the solution within
1e-8 relative of the zero-mean direct solve, compared modulo constants.
"""
import numpy as np
import pytest

from oracle import pmf_oracle as O
from premixfem_b200 import fields
from premixfem_b200.solver import DarcySolver, options_string

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_constant_null_space_matches_oracle(native, precision):
    prob = fields.aniso_const(8, 8, 8)
    d = {"sd": 2, "en_lv1": 4, "en_lv2": 4}
    ref = O.solve(prob, O.Options(**d, constant_null_space=True))
    assert ref["reason"] == "converged_rtol"
    s = DarcySolver.from_problem(prob, options_string(dict(d, pmf_precision=precision)) + " -ksp_constant_null_space")
    s.setup()
    b = s.rhs(prob["source"].ravel())
    x, its, rnorm, reason = s.solve(b)
    s.close()
    assert reason == "converged"
    assert abs(its - ref["its"]) <= 1, (its, ref["its"])
    assert rnorm <= 1e-8 * np.linalg.norm(b) * (1 + 1e-6)
    xd = O.direct_solve(ref["op"], ref["b"])
    xd = xd - xd.mean()
    err = np.linalg.norm((x - x.mean()) - xd) / np.linalg.norm(xd)
    assert err <= 1e-8, err


def test_constant_null_space_option_values(native):
    # PETSc boolean option: bare flag or a true/false word; anything else is an argument error
    from premixfem_b200._native import PmfError
    for opt in ("-ksp_constant_null_space", "-ksp_constant_null_space true", "-ksp_constant_null_space 0"):
        DarcySolver((1.0, 1.0, 1.0), (8, 8, 8), "-sd 2 " + opt).close()
    with pytest.raises(PmfError) as e:
        DarcySolver((1.0, 1.0, 1.0), (8, 8, 8), "-sd 2 -ksp_constant_null_space maybe")
    assert e.value.code == 62


@pytest.mark.parametrize("form", [{"pmf_precision": "fp64"}, {"pmf_precision": "mixed"},
                                  {"pmf_precision": "mixed", "pmf_eig_precision": "fp64"}],
                         ids=["fp64", "mixed", "mixed_fp64_basis"])
@pytest.mark.parametrize("seed", [1, 2, 3, 4])
def test_constant_is_in_the_coarse_space(native, seed, form):
    """Channels of contrast 1e6 without a Dirichlet face: every subdomain's first basis vector is the constant to the
    last bits, so that the coarse operator's null vector is the operator's own, and CG gets to 1e-10 of the right-hand
    side."""
    prob = fields.layered(seed=seed, M=30, N=44, P=30, smooth_layers=10)
    s = DarcySolver.from_problem(prob, options_string(dict(form, pmf_vranks=(2, 2, 1), pmf_sd=(2, 2, 6), en_lv1=4,
                                                           en_lv2=4, ksp_constant_null_space=True, ksp_rtol=1e-10,
                                                           ksp_max_it=2000)))
    s.setup()
    phi = s.phi()[:, 0].reshape(prob["kappa"][0].shape)
    boxes, _ = s.subdomains()
    for x0, nx, y0, ny, z0, nz in boxes:
        v = phi[z0:z0 + nz, y0:y0 + ny, x0:x0 + nx]
        assert np.ptp(v) <= 1e-13 * np.abs(v).max()
    _, its, _, reason = s.solve(s.rhs(prob["source"].ravel()))
    s.close()
    assert reason == "converged", its


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("seed", [1, 2, 3, 4])
def test_singular_operator_without_the_option(native, seed, precision):
    """The same channels without -ksp_constant_null_space and with the default shift of the level-3 matrix, which the
    coarse solve multiplies the constant by 1e12 with: a consistent right-hand side is solved to the default 1e-8."""
    prob = fields.layered(seed=seed, M=30, N=44, P=30, smooth_layers=10)
    s = DarcySolver.from_problem(prob, options_string(dict(sd=3, en_lv1=4, en_lv2=4, pmf_precision=precision,
                                                           ksp_max_it=600)))
    s.setup()
    b = s.rhs(prob["source"].ravel())
    x, its, _, reason = s.solve(b)
    r = b - s.apply_A(x)
    s.close()
    assert reason == "converged", its
    assert np.linalg.norm(r) <= 1.1e-8 * np.linalg.norm(b)


@pytest.mark.parametrize("project", [True, False], ids=["null_space", "plain"])
@pytest.mark.parametrize("form", [{"pmf_precision": "fp64"}, {"pmf_precision": "mixed"},
                                  {"pmf_precision": "mixed", "pmf_eig_precision": "fp64"}],
                         ids=["fp64", "mixed", "mixed_fp64_basis"])
@pytest.mark.parametrize("seed", [1, 2, 5])
def test_callers_own_cg_on_a_singular_operator(native, seed, form, project):
    """CG of a caller's own through apply_A and pc_apply on the same channels, with and without the null space taken out
    of z: the 1e-8 that the library's own solve reaches, in its iterations give or take a tenth."""
    prob = fields.layered(seed=seed, M=30, N=44, P=30, smooth_layers=10)
    s = DarcySolver.from_problem(prob, options_string(dict(form, sd=3, en_lv1=4, en_lv2=4, ksp_max_it=600,
                                                           ksp_constant_null_space=project)))
    s.setup()
    b = s.rhs(prob["source"].ravel())
    _, its, _, reason = s.solve(b)
    assert reason == "converged"

    def precondition(r):
        z = s.pc_apply(r)
        return z - z.mean() if project else z

    x, r = np.zeros_like(b), b.copy()
    p = z = precondition(r)
    rz, n = r @ z, 0
    while np.linalg.norm(r) > 1e-8 * np.linalg.norm(b) and n < 1.1 * its:
        w = s.apply_A(p)
        x, r, n = x + rz / (p @ w) * p, r - rz / (p @ w) * w, n + 1
        z = precondition(r)
        rz, old = r @ z, rz
        p = z + rz / old * p
    r = b - s.apply_A(x)
    s.close()
    assert np.linalg.norm(r) <= 1.1e-8 * np.linalg.norm(b), n


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("mesh,sd,seed", [((20, 22, 18), 5, 2), ((20, 22, 18), 5, 8), ((16, 16, 16), 4, 4),
                                          ((30, 28, 26), 6, 3)], ids=lambda v: str(v).replace(", ", "x"))
def test_one_rank_holds_the_singular_problem(native, mesh, sd, seed, precision):
    """A single rank's coarse block is the whole singular operator's: its inverse must not depend on how the rounding of
    its last pivot falls.  Iterations within +-1 of the oracle's."""
    prob = fields.random_box(mesh, seed=seed, sigma=1.5)
    prob["dirichlet"] = {}
    src = np.random.default_rng(seed).standard_normal(prob["kappa"][0].shape)
    prob["source"] = src - src.mean()
    d = {"sd": sd, "en_lv1": 4, "en_lv2": 4}
    ref = O.solve(prob, O.Options(**d, constant_null_space=True))
    s = DarcySolver.from_problem(prob, options_string(dict(d, pmf_precision=precision, ksp_constant_null_space=True,
                                                           ksp_max_it=100)))
    s.setup()
    _, its, _, reason = s.solve(s.rhs(prob["source"].ravel()))
    s.close()
    assert reason == "converged" and abs(its - ref["its"]) <= 1, (its, ref["its"])


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("mesh,vranks,sd,seed", [((24, 24, 24), (2, 2, 1), 2, 1), ((24, 20, 16), (2, 1, 1), 2, 2),
                                                 ((16, 16, 16), (2, 2, 2), 1, 3), ((16, 16, 16), (1, 1, 1), 2, 3)],
                         ids=lambda v: str(v).replace(", ", "x"))
def test_pc_apply_of_a_vector_with_a_sum(native, mesh, vranks, sd, seed, precision):
    """One application to a vector whose sum is not zero, without the shift that would drown it: the oracle's to the 1e-6
    of the other applications (a projection would take part of it away)."""
    prob = fields.random_box(mesh, seed=seed, sigma=1.5)
    prob["dirichlet"] = {}
    d = {"sd": sd, "en_lv1": 4, "en_lv2": 4, "no_shift_A_cc": True}
    x = np.random.default_rng(seed).standard_normal(int(np.prod(mesh)))
    y = O.Preconditioner(O.Operator(prob), O.Options(**d, vranks=vranks)).apply(x)
    s = DarcySolver.from_problem(prob, options_string(dict(d, pmf_vranks=vranks, pmf_precision=precision)))
    s.setup()
    z = s.pc_apply(x)
    s.close()
    assert np.linalg.norm(z - y) <= 1e-6 * np.linalg.norm(y)


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("seed", [1, 3, 5])
def test_batch_of_singular_problems(native, seed, precision):
    """Three channel problems without a Dirichlet face and one with, in one batch (which has no null space option): each
    converges to the default 1e-8."""
    from premixfem_b200.solver import BatchSolver
    probs = [fields.layered(seed=seed * 10 + q, M=18 + 2 * q, N=24, P=16, smooth_layers=5) for q in range(4)]
    probs[2]["dirichlet"] = {"z-": 1.0}
    rng = np.random.default_rng(seed)
    srcs = [v - v.mean() for v in (rng.standard_normal(p["source"].shape) for p in probs)]
    s = BatchSolver(probs, [tuple(-(-n // 8) for n in p["mesh"]) for p in probs],
                    options_string({"en_lv1": 4, "en_lv2": 3, "pmf_precision": precision, "ksp_max_it": 800}))
    s.set_kappa(*[s.pack([p["kappa"][d] for p in probs]) for d in range(3)])
    s.setup()
    _, its, _, reason = s.solve(s.rhs(s.pack(srcs)))
    s.close()
    assert list(reason) == ["converged"] * 4, (its, reason)
