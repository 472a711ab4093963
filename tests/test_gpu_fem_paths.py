"""The SSAFEM linear solve in one cooperative kernel (graphs = 2, csrc/ssa_fem.cu k_cg_resident)
against the three kernels of an iteration (graphs = 0, and 1: replayed batches): the same operations
and the same order of every sum, so one Newton step gives the same iterations and the same velocity bit
for bit, and so does the whole solve.  A wrong neighbour or a stale value at a run's end would
show after one linear solve, where Newton's later steps hide it."""
import numpy as np
import pytest

from pism_b200 import verification as V

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():
    pytest.skip("no CUDA device", allow_module_level=True)

from pism_b200.ssa import SSAFEM  # noqa: E402


def solve(case, graphs, **options):
    g, c, f = case
    s = SSAFEM(g, c.copy(graphs=graphs), **options)
    s.set_inputs(**{k: f[k] for k in ("thickness", "surface", "bed", "mask", "tauc")}, bc_mask=f["bc_mask"],
                 bc_values=f["bc_values"])
    s.set_initial_guess(np.zeros((g.Mx, g.My, 2)))
    v, st = s.solve(), s.stats()
    s.close()
    return v, (st["newton_iterations"], st["ksp_iterations"])


@pytest.mark.parametrize("build,Mx,My", [("i", 5, 51), ("i", 3, 86), ("i", 3, 41), ("i", 4, 301), ("i", 5, 481),
                                         ("j", 16, 16), ("j", 17, 15), ("j", 33, 31), ("j", 3, 259), ("j", 259, 3),
                                         ("j", 95, 91), ("j", 241, 241)])
def test_bitwise(build, Mx, My):
    case = V.build_test_i(My=My, Mx=Mx) if build == "i" else V.build_test_j(Mx, My)
    for options in (dict(snes_rtol=0.999999), {}):   # the first step alone; the whole solve
        ref, its = solve(case, 0, **options)
        assert options == {} or its[0] == 1
        assert np.isfinite(ref).all()
        for graphs in (1, 2):
            v, n = solve(case, graphs, **options)
            assert n == its
            np.testing.assert_array_equal(v, ref)
