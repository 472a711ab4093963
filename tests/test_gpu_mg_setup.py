"""The multigrid set-up (csrc/ssa_mg.cu: Galerkin operators of the levels built by a launch each
and by the closing block, and the pivoted inverse of the coarsest one) through one V-cycle,
against the same cycle in 64 bits with dense operators: A probed column by column, R A P by
piecewise-constant aggregation, omega = 0.9, correction 1.2.

Shapes: the coarsest level directly below the grid (7 x 8), levels of odd and even sizes,
aggregation in one direction only, a level just above and just below the closing block's size.

Tolerance: the cycle rounds to FP32 (6e-8 an operation) and the coarsest operator's condition
number, below 1e4 on these grids with basal drag everywhere, may amplify that: 1e-3 relative L2.
A misplaced block or pivot is an O(1) error."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():
    pytest.skip("needs a CUDA device", allow_module_level=True)

from pism_b200.config import GridDesc, SSAConfig  # noqa: E402
from pism_b200.ssa import SSAFD  # noqa: E402


def aggregate(Mx, My):
    ax, ay = (2 if Mx > 4 else 1), (2 if My > 4 else 1)
    cx, cy = -(-Mx // ax), -(-My // ay)
    i, j = torch.meshgrid(torch.arange(Mx, device="cuda"), torch.arange(My, device="cuda"), indexing="ij")
    cell = ((i // ax) * cy + j // ay).reshape(-1)
    P = torch.zeros((2 * Mx * My, 2 * cx * cy), dtype=torch.float64, device="cuda")
    k = torch.arange(Mx * My, device="cuda")
    for q in (0, 1):
        P[2 * k + q, 2 * cell + q] = 1.0
    return P, cx, cy


def smooth(A, b):
    n = A.shape[0] // 2
    k = torch.arange(n, device="cuda")
    D = A.reshape(n, 2, n, 2)[k, :, k, :]
    return 0.9 * torch.linalg.solve(D, b.reshape(n, 2)).reshape(-1)


def vcycle(A, b, Mx, My):
    if Mx <= 4 and My <= 4:
        return torch.linalg.solve(A, b)
    P, cx, cy = aggregate(Mx, My)
    x = smooth(A, b)
    x = x + 1.2 * (P @ vcycle(P.T @ A @ P, P.T @ (b - A @ x), cx, cy))
    return x + smooth(A, b - A @ x)


@pytest.mark.parametrize("Mx,My", [(7, 8), (9, 13), (3, 40), (31, 30), (45, 50), (43, 44)])
def test_vcycle_matches_dense_galerkin_operators(Mx, My):
    rng = np.random.Generator(np.random.PCG64(100 * Mx + My))
    i, j = np.arange(Mx)[:, None] / Mx, np.arange(My)[None, :] / My
    mask = np.where(rng.uniform(size=(Mx, My)) < 0.05, 0.0, 2.0)
    f = {"thickness": 900.0 + 500.0 * np.sin(7 * i + 3 * j), "surface": 900.0 + 200.0 * np.cos(4 * i - j),
         "bed": np.zeros((Mx, My)), "mask": mask, "tauc": rng.uniform(2e4, 2e5, (Mx, My)),
         "melange": np.zeros((Mx, My))}
    vel = 1e-5 * np.stack([np.sin(6 * i + j), np.cos(3 * i - 5 * j)], -1)
    s = SSAFD(GridDesc(Mx, My, 5e3 * (Mx - 1), 5e3 * (My - 1)), SSAConfig(flow_law="isothermal_glen", pc_type="mg"))
    s.set_inputs(**f)
    s.set_initial_guess(vel)
    s.assemble_rhs()
    s.compute_hardav_staggered()
    s.compute_nuH_staggered(1e13)
    n = 2 * Mx * My
    A = torch.empty((n, n), dtype=torch.float64, device="cuda")
    x = torch.zeros((Mx, My, 2), dtype=torch.float64, device="cuda")
    y = torch.empty_like(x)
    for c in range(n):
        x.zero_()
        x.view(-1)[c] = 1.0
        torch.cuda.synchronize()
        s.apply(x, y)
        torch.cuda.synchronize()
        A[:, c] = y.view(-1)
    r = torch.tensor(1e3 * np.stack([np.sin(5 * i + 3 * j), np.cos(4 * i - 2 * j)], -1), device="cuda")
    z = torch.zeros_like(r)
    torch.cuda.synchronize()
    s.apply_preconditioner(r, z)
    torch.cuda.synchronize()
    s.close()
    ref = vcycle(A, r.reshape(-1), Mx, My)
    assert float(torch.linalg.norm(z.reshape(-1) - ref) / torch.linalg.norm(ref)) < 1e-3
