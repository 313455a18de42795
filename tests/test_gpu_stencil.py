"""The z-march of the 7-point operator (32 x 8 tiles, stretches of 1 to 16
planes by the number of tiles) at its edges, the fused CG step built on it, and
the restriction and prolongation for every basis size, against the sparse
operator of the oracle.

Bars: an operator product is a sum of at most seven products per cell, so 1e-13
of its norm; a solve at rtol 1e-11 leaves a true residual within 1e-10."""
import numpy as np
import pytest

from oracle import pmf_oracle as O
from premixfem_b200 import fields
from premixfem_b200.solver import DarcySolver

pytestmark = pytest.mark.gpu

MESHES = [(2, 2, 2), (31, 9, 17), (32, 8, 16), (33, 7, 5), (64, 16, 33), (65, 17, 31), (5, 3, 130), (130, 2, 3),
          (3, 100, 4), (96, 96, 48)]


@pytest.mark.parametrize("mesh", MESHES, ids=lambda m: "x".join(map(str, m)))
def test_operator_and_cg_step(native, mesh):
    prob = fields.random_box(mesh, seed=4, sigma=2.0, dirichlet={"x-": 1.0, "z+": 0.5})
    op = O.Operator(prob)
    sd = tuple(max(1, (n + 7) // 8) for n in mesh)
    s = DarcySolver.from_problem(prob, f"-pmf_sd {sd[0]},{sd[1]},{sd[2]} -en_lv1 1 -en_lv2 1 -ksp_rtol 1e-11")
    s.setup()
    x = np.random.default_rng(1).standard_normal(op.n)
    ref = op.A @ x
    assert np.linalg.norm(s.apply_A(x) - ref) <= 1e-13 * np.linalg.norm(ref)
    b = s.rhs(prob["source"].ravel())
    u, _, _, reason = s.solve(b)
    s.close()
    assert reason == "converged"
    assert np.linalg.norm(b - op.A @ u) <= 1e-10 * np.linalg.norm(b)


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("k", range(1, 9))
def test_basis_sizes(native, k, precision):
    """The W-cycle visits the restriction with an iterate, the V-cycle without; one basis vector more
    never leaves the solve unconverged."""
    prob = fields.random_box((17, 15, 19), seed=5, sigma=1.5)
    op = O.Operator(prob)
    for extra in ("", " -use_W_cycle"):
        s = DarcySolver.from_problem(prob, f"-pmf_sd 2,2,3 -en_lv1 {k} -en_lv2 2 -pmf_precision {precision} "
                                           f"-ksp_rtol 1e-11{extra}")
        s.setup()
        b = s.rhs(prob["source"].ravel())
        u, _, _, reason = s.solve(b)
        s.close()
        assert reason == "converged"
        assert np.linalg.norm(b - op.A @ u) <= 1e-10 * np.linalg.norm(b)


@pytest.mark.parametrize("mesh,tile", [((4, 1024, 1024), (4, 16, 16)), ((8, 512, 1024), (8, 16, 16)),
                                       ((2048, 1, 2048), (16, 1, 16)), ((2048, 3, 704), (16, 3, 16))],
                         ids=["4x1024x1024", "8x512x1024", "2048x1x2048", "2048x3x704"])
def test_thin_meshes_leave_no_threads_idle(native, mesh, tile):
    """Meshes of a few cells in x or y take no longer than a cube of as many cells (4.2 million; 30 % for the box's
    surface and the clock): the operator's call and the CG step."""
    import time

    import torch

    def times(mesh, tile):
        n = [-(-m // t) for m, t in zip(mesh, tile)]
        vr = [1, 1, 1]
        while np.prod([-(-c // v) for c, v in zip(n, vr)]) * 2 > 2000:
            vr[int(np.argmax([c / v for c, v in zip(n, vr)]))] *= 2
        sd = [-(-c // v) for c, v in zip(n, vr)]
        s = DarcySolver((1.0, 1.0, 1.0), mesh, f"-pmf_vranks {vr[0]},{vr[1]},{vr[2]} -pmf_sd {sd[0]},{sd[1]},{sd[2]} "
                                               "-en_lv1 2 -en_lv2 2 -pmf_eig_max_it 3 -pmf_autotune 0")
        k = torch.from_numpy(np.exp(np.random.default_rng(0).standard_normal(int(np.prod(mesh))))).cuda()
        s.set_kappa(k, k, k)
        s.set_dirichlet("x-", 0.0)
        s.setup()
        x, y = torch.ones_like(k), torch.empty_like(k)
        best = []
        for _ in range(5):
            t0 = time.perf_counter()
            for _ in range(20):
                s.apply_A(x, y)
            best.append((time.perf_counter() - t0) / 20)
        s.profile_iteration(10)
        step = s.profile_iteration(20)["cg_p_update_Ap"][0]
        s.close()
        return min(best), step

    ref = times((161, 163, 160), (16, 16, 16))
    got = times(mesh, tile)
    assert got[0] <= 1.3 * ref[0] and got[1] <= 1.3 * ref[1], (got, ref)


def test_a_basis_vector_costs_its_bytes(native):
    """The restriction with five to eight FP32 basis vectors against four, on 4.1 million cells: a cell's bytes are
    those of k + 10 values, and 10 % are left for the clock."""
    import torch
    k0 = torch.from_numpy(np.exp(np.random.default_rng(0).standard_normal(160 ** 3))).cuda()
    us = {}
    for k in range(4, 9):
        s = DarcySolver((1.0, 1.0, 1.0), (160, 160, 160), f"-pmf_vranks 4,2,2 -pmf_sd 3,5,5 -en_lv1 {k} -en_lv2 2 "
                                                          "-pmf_precision mixed -pmf_eig_max_it 3")
        s.set_kappa(k0, k0, k0)
        s.set_dirichlet("x-", 0.0)
        s.setup()
        s.profile_iteration(10)
        us[k] = 1e3 * s.profile_iteration(40)["resid_restrict"][0]
        s.close()
    for k in range(5, 9):
        assert us[k] <= 1.1 * (k + 10) / 14 * us[4], us
