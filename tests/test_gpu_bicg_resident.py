"""The block-Jacobi BiCGStab solve in one cooperative kernel (csrc/ssa_kernels.cu
k_bicg_resident, the linear solve of graphs = 2 where the grid's tiles are resident at once)
against the five kernels of an iteration (graphs = 0): the same operations and the same order of
every sum, so the same iterates bit for bit, on grids at the edges of its tiles and of its linear
blocks, narrower than a tile, with fronts, Dirichlet rows and ice-free cells."""
import numpy as np
import pytest

from pism_b200.config import GridDesc, SSAConfig

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():
    pytest.skip("no CUDA device", allow_module_level=True)

from pism_b200.ssa import KSPFailure, SSAFD  # noqa: E402


@pytest.mark.parametrize("cfbc", [False, True])
@pytest.mark.parametrize("Mx,My", [(3, 3), (8, 32), (9, 33), (7, 31), (17, 65), (5, 201), (3, 600), (100, 3), (95, 350),
                                   (96, 400)])
def test_bitwise(Mx, My, cfbc):
    """95 x 350 is 132 tiles, 96 x 400 156: one on each side of what 148 SMs hold"""
    rng = np.random.Generator(np.random.PCG64(100 * Mx + My))
    i, j = np.arange(Mx)[:, None] / Mx, np.arange(My)[None, :] / My
    H = 900.0 + 500.0 * np.sin(7 * i + 3 * j) + rng.uniform(0.0, 100.0, (Mx, My))
    mask = np.where(rng.uniform(size=(Mx, My)) < 0.05, 4.0, np.where(np.sin(5 * i + 4 * j) > 0.3, 3.0, 2.0))
    vel = 1e-5 * np.stack([np.sin(6 * i + j), np.cos(3 * i - 5 * j)], -1)
    f = {"thickness": H, "surface": H, "bed": np.zeros((Mx, My)), "mask": mask,
         "tauc": rng.uniform(1e4, 2e5, (Mx, My)), "melange": np.zeros((Mx, My)),
         "bc_mask": (rng.uniform(size=(Mx, My)) < 0.03).astype(float), "bc_values": vel}
    b = torch.tensor(1e3 * np.stack([np.sin(5 * i + 3 * j), np.cos(4 * i - 2 * j)], -1), device="cuda")
    out = {}
    for graphs in (0, 2):
        s = SSAFD(GridDesc(Mx, My, 5e3 * (Mx - 1), 5e3 * (My - 1)),
                  SSAConfig(flow_law="isothermal_glen", pc_type="bjacobi", ksp_rtol=1e-6, ksp_max_it=60, graphs=graphs,
                            calving_front_stress_boundary_condition=cfbc, ssa_dirichlet_bc=True))
        s.set_inputs(**f)
        s.set_initial_guess(vel)
        s.assemble_rhs()
        s.compute_hardav_staggered()
        s.compute_nuH_staggered(1e13)
        for start in (0.0, 1e-6):
            x = torch.full_like(b, start)
            torch.cuda.synchronize()
            try:
                its = s.linear_solve_rhs(b, x)
            except KSPFailure as e:   # 60 iterations are enough to compare
                its = str(e)
            torch.cuda.synchronize()
            out[graphs, start] = (x.cpu().numpy(), its)
        s.close()
    for start in (0.0, 1e-6):
        assert np.isfinite(out[0, start][0]).all()
        np.testing.assert_array_equal(out[0, start][0], out[2, start][0])
        assert out[0, start][1] == out[2, start][1]
