"""The lock-step eigensolver's Gram, update and image kernels where their groups of
cells end: subdomains of 125, 189, 1 309 (a chunk and a ragged rest), 4 096 and
2 x 3 x 4 = 24 cells, blocks of 5, 8 and 10 columns, FP64 and FP32 storage.

Eigenvalues against the dense oracle: 1e-6 in FP64 storage, the bar of the other
eigenvalue tests.  FP32 storage stops where vectors rounded to FP32 stop it, with
a residual near 1e-6 of the largest eigenvalue that the block sees; the final FP64
Rayleigh-Ritz leaves its square over the gap, so 1e-5 holds there."""
import numpy as np
import pytest

from oracle import pmf_oracle as O
from premixfem_b200 import fields
from premixfem_b200.solver import DarcySolver, options_string

pytestmark = pytest.mark.gpu

TILES = [(5, 5, 5), (9, 7, 3), (17, 11, 7), (16, 16, 16), (2, 3, 4)]


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("k", [3, 6, 8])
@pytest.mark.parametrize("tile", TILES, ids=lambda t: "x".join(map(str, t)))
def test_local_eigenvalues_at_group_edges(native, tile, k, precision):
    prob = fields.random_box(tuple(2 * n for n in tile), seed=11, sigma=1.0)
    s = DarcySolver.from_problem(prob, options_string({"pmf_sd": (2, 2, 2), "en_lv1": k, "en_lv2": 2,
                                                       "pmf_precision": precision}))
    s.setup()
    ev, ks, _, status = s.eigen_lv1()
    boxes, _ = s.subdomains()
    s.close()
    ref = O.local_eigenvalues(prob, [tuple(b) for b in boxes], k, method="dense")
    scale = np.abs(ref).max(axis=1, keepdims=True)
    err = np.abs(ev - ref) / np.maximum(np.abs(ref), 1e-3 * scale)
    assert (ks == k).all() and (status != 1).all()
    assert err.max() <= (1e-6 if precision == "fp64" else 1e-5), f"max rel eigen error {err.max():.2e}"
