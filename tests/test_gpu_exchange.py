"""What the one-kernel Krylov solves do when a block's wait runs out (csrc/ssa_exchange.cuh): no
block may take a sum with a part missing for a sum, so a solve whose waits gave up ends with an
error and never as converged.  Grids of at most 32 blocks add their slots in one trip, larger ones
in two."""
import os
import shutil
import subprocess

import numpy as np
import pytest

from pism_b200 import _capi, verification as V
from pism_b200.config import GridDesc, SSAConfig

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():
    pytest.skip("no CUDA device", allow_module_level=True)

from pism_b200.ssa import SSAFD, SSAFEM, KSPFailure  # noqa: E402

REPO = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
SHORT = 2000   # reads: about 2 ms


@pytest.fixture(scope="module")
def driver(tmp_path_factory):
    if shutil.which("nvcc") is None:
        pytest.skip("needs nvcc")
    exe = str(tmp_path_factory.mktemp("exchange") / "check")
    subprocess.run(["nvcc", "-gencode", "arch=compute_100a,code=sm_100a", "-O3", "-std=c++17", "-I",
                    os.path.join(REPO, "include"), "-I", os.path.join(REPO, "pismv0.7.3_b200", "csrc"),
                    os.path.join(REPO, "tests", "exchange_check.cu"), "-o", exe], check=True)
    return exe


def ask(driver, *line):
    out = subprocess.run([driver], input=" ".join(str(v) for v in line) + "\n", capture_output=True, text=True,
                         check=True, timeout=60).stdout.split()
    return [int(v) for v in out[:3]], out[3] == "1"


@pytest.mark.parametrize("one", [0, 1])
@pytest.mark.parametrize("blocks", [1, 2, 31, 32, 33, 64, 65, 148])
def test_sums(driver, blocks, one):
    assert ask(driver, blocks, -1, 1 << 20, one) == ([blocks] * 3, True)


@pytest.mark.parametrize("one", [0, 1])
@pytest.mark.parametrize("blocks,absent", [(2, 0), (2, 1), (32, 0), (32, 31), (33, 32), (33, 0), (64, 40), (64, 1), (148, 147),
                                           (148, 70)])
def test_a_block_that_never_posts(driver, blocks, absent, one):
    """no block finishes a round without it"""
    assert ask(driver, blocks, absent, SHORT, one)[0] == [0, 0, 0]


@pytest.mark.parametrize("limit", [1, 4, 16, 64])
@pytest.mark.parametrize("Mx,My", [(5, 201), (40, 201), (95, 350)])
def test_bicgstab_gives_up_or_solves(Mx, My, limit):
    """7, 35 and 132 blocks: an error or the answer (a few blocks may find every word at the first
    read); with one read and more than 32 blocks the error"""
    i, j = np.arange(Mx)[:, None] / Mx, np.arange(My)[None, :] / My
    H = 900.0 + 500.0 * np.sin(7 * i + 3 * j)
    f = {"thickness": H, "surface": H, "bed": np.zeros((Mx, My)), "mask": np.full((Mx, My), 2.0),
         "tauc": np.full((Mx, My), 5e4), "melange": np.zeros((Mx, My))}
    s = SSAFD(GridDesc(Mx, My, 5e3 * (Mx - 1), 5e3 * (My - 1)),
              SSAConfig(flow_law="isothermal_glen", pc_type="bjacobi", ksp_rtol=1e-6, ksp_max_it=2000, graphs=2))
    s.set_inputs(**f)
    s.set_initial_guess(1e-5 * np.stack([np.sin(6 * i + j), np.cos(3 * i - 5 * j)], -1))
    s.assemble_rhs()
    s.compute_hardav_staggered()
    s.compute_nuH_staggered(1e13)
    b = torch.tensor(1e3 * np.stack([np.sin(5 * i + 3 * j), np.cos(4 * i - 2 * j)], -1), device="cuda")
    ref = torch.zeros_like(b)
    torch.cuda.synchronize()
    s.linear_solve_rhs(b, ref)
    assert s.lib.pism_gpu_ssa_set_wait_limit(s._h, limit) == _capi.OK
    for _ in range(3):
        x = torch.zeros_like(b)
        torch.cuda.synchronize()
        try:
            s.linear_solve_rhs(b, x)
        except KSPFailure as e:
            assert "reason -11" in str(e)
        else:
            assert torch.equal(x, ref) and (limit > 1 or Mx * My < 32 * 256)
    s.close()


@pytest.mark.parametrize("limit", [1, 4, 16, 64])
@pytest.mark.parametrize("Mx,My", [(16, 32), (91, 95), (241, 241)])
def test_cg_gives_up_or_solves(Mx, My, limit):
    """2, 34 and 227 blocks, as above"""
    g, c, f = V.build_test_j(Mx, My)
    s = SSAFEM(g, c)
    s.set_inputs(**{k: f[k] for k in ("thickness", "surface", "bed", "mask", "tauc")}, bc_mask=f["bc_mask"],
                 bc_values=f["bc_values"])
    zero = np.zeros((Mx, My, 2))
    s.set_initial_guess(zero)
    ref = s.solve()
    assert s.lib.pism_gpu_ssa_set_wait_limit(s._h, limit) == _capi.OK
    for _ in range(3):
        s.set_initial_guess(zero)
        try:
            v = s.solve()
        except KSPFailure as e:
            assert "gave up waiting" in str(e)
            np.testing.assert_array_equal(s.velocity(), zero)   # a failed solve leaves the velocity
        else:
            assert np.array_equal(v, ref) and (limit > 1 or Mx * My < 32 * 256)
    s.close()


def test_limit_is_checked():
    s = SSAFD(GridDesc(5, 5, 1e4, 1e4), SSAConfig(flow_law="isothermal_glen"))
    for reads in (0, -1, (1 << 20) + 1):
        assert s.lib.pism_gpu_ssa_set_wait_limit(s._h, reads) == _capi.EINVAL
    assert s.lib.pism_gpu_ssa_set_wait_limit(s._h, 1 << 20) == _capi.OK
    s.close()
