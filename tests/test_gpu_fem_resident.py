"""The SSAFEM linear solve in one cooperative kernel (csrc/ssa_fem.cu k_cg_resident) where its
blocks and runs begin and end: grids of 255, 256, 257 and 258 nodes, rows longer and shorter than
a block, one, two and more than 32 blocks, periodic and not; and a grid too large for it."""
import numpy as np
import pytest

from pism_b200 import verification as V
from oracle import ssafd_oracle as O
from oracle import ssafem_oracle as F
from tests.test_gpu_ssafem import GOLDEN, gpu_solve, rel_l2, TIGHT

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("build,Mx,My", [("i", 5, 51), ("i", 3, 86), ("i", 3, 41), ("i", 4, 301), ("j", 16, 16),
                                         ("j", 17, 15), ("j", 33, 31), ("j", 3, 259), ("j", 259, 3), ("j", 95, 91)])
def test_against_the_oracle(build, Mx, My):
    """both converged far below it: the tolerance of the SSAFEM tests (1e-8)"""
    g, c, f = V.build_test_i(My=My, Mx=Mx) if build == "i" else V.build_test_j(Mx, My)
    vel, st = gpu_solve(g, c, f, **TIGHT)
    ref, _ = F.SSAFEMOracle(*O.from_case(g, c, f)).solve()
    assert st["converged"] > 0
    assert np.isfinite(vel).all() and rel_l2(vel, ref) < 1e-8


def test_a_grid_beyond_it():
    """281 x 279 nodes take the kernels of an iteration each: closer to the exact shelf than the
    reference's printed error on its finer regression grid"""
    g, c, f = V.build_test_j(281, 279)
    vel, st = gpu_solve(g, c, f)
    assert st["converged"] > 0
    printed = GOLDEN["test_j_fem"]["cases"][1]
    assert printed["Mx"] < 279
    assert V.report(vel, V.exact_velocity_j(g))["prcntavvec"] < printed["prcntavvec"]
