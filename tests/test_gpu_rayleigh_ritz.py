"""The local eigensolves' projected problems (one warp per subdomain) at every
kernel width: en_lv1 + 2 block columns give bases of up to 9, 15, 18, 21, 24, 27
and 30 vectors.  The second box has subdomains of 12 to 27 cells, so the wider
bases exceed the space and dependent vectors leave the basis."""
import numpy as np
import pytest

from oracle import pmf_oracle as O
from premixfem_b200 import fields
from premixfem_b200.solver import DarcySolver, options_string

pytestmark = pytest.mark.gpu

MESHES = {"ragged": (13, 11, 9), "tiny": (6, 5, 5)}


@pytest.mark.parametrize("mesh", list(MESHES))
@pytest.mark.parametrize("k", [1, 3, 4, 5, 6, 7, 8])
def test_local_eigenvalues_at_every_width(native, mesh, k):
    prob = fields.random_box(MESHES[mesh], seed=k, sigma=1.5)
    s = DarcySolver.from_problem(prob, options_string({"sd": 2, "en_lv1": k, "en_lv2": 2}))
    s.setup()
    ev, ks, iters, status = s.eigen_lv1()
    boxes, _ = s.subdomains()
    s.close()
    # four eigenvalues: a scale for the rows whose only wanted one is the constant's, zero
    ref = O.local_eigenvalues(prob, [tuple(b) for b in boxes], max(k, 4), method="dense")
    scale = np.abs(ref).max(axis=1, keepdims=True)
    ref = ref[:, :k]
    err = np.abs(ev - ref) / np.maximum(np.abs(ref), 1e-3 * scale)
    # the FP64 form's stopping residual, 1e-8 of the operator's scale, bounds an eigenvalue's
    # error by its square over the gap; 1e-6 is the bar of the other eigenvalue tests
    assert (ks == k).all() and (status != 1).all()
    assert err.max() <= 1e-6, f"max rel eigen error {err.max():.2e}"


@pytest.mark.parametrize("k", [4, 6, 8])
@pytest.mark.parametrize("tile", [(2, 3, 4), (3, 3, 3), (4, 2, 2), (5, 3, 2), (4, 4, 4), (6, 5, 3)],
                         ids=lambda t: "x".join(map(str, t)))
def test_basis_wider_than_the_space(native, tile, k):
    """Bases that fill or exceed the space of a small subdomain: dependent vectors have to be recognised as
    such, else their Ritz values are noise and the lowest wanted ones are wrong.  27 subdomains of four
    contrasts; the bars of the test above."""
    for seed, sigma in enumerate([0.5, 1.5, 3.0, 4.0]):
        prob = fields.random_box(tuple(3 * n for n in tile), seed=seed, sigma=sigma)
        s = DarcySolver.from_problem(prob, options_string({"sd": 3, "en_lv1": k, "en_lv2": 2}))
        s.setup()
        ev, _, _, status = s.eigen_lv1()
        boxes, _ = s.subdomains()
        s.close()
        ref = O.local_eigenvalues(prob, [tuple(b) for b in boxes], k, method="dense")
        scale = np.abs(ref).max(axis=1, keepdims=True)
        err = np.abs(ev - ref) / np.maximum(np.abs(ref), 1e-3 * scale)
        assert (status != 1).all()
        assert err.max() <= 1e-6, f"max rel eigen error {err.max():.2e}"


@pytest.mark.parametrize("tile,k", [((3, 3, 3), 6), ((5, 3, 2), 6), ((4, 4, 2), 8), ((3, 3, 4), 8)],
                         ids=lambda v: "x".join(map(str, v)) if isinstance(v, tuple) else str(v))
def test_images_belong_to_the_block(native, tile, k):
    """Blocks whose basis takes nearly all of the space: search directions shrink to rounding, and an image that is
    carried along with them instead of computed from them no longer belongs to its vector; the Ritz values are then
    wrong and the block stops converging.  216 subdomains; the bars of the tests above."""
    for seed in range(8):
        prob = fields.random_box(tuple(3 * n for n in tile), seed=seed, sigma=[0.5, 1.5, 3.0, 4.0][seed % 4])
        s = DarcySolver.from_problem(prob, options_string({"sd": 3, "en_lv1": k, "en_lv2": 2}))
        s.setup()
        ev, _, _, status = s.eigen_lv1()
        boxes, _ = s.subdomains()
        s.close()
        ref = O.local_eigenvalues(prob, [tuple(b) for b in boxes], k, method="dense")
        scale = np.abs(ref).max(axis=1, keepdims=True)
        err = np.abs(ev - ref) / np.maximum(np.abs(ref), 1e-3 * scale)
        assert (status != 1).all()
        assert err.max() <= 1e-6, f"max rel eigen error {err.max():.2e}"
