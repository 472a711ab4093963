"""The resident small-level cycle: its layout on CPU (csrc/ssa_small_plan.h's resident_plan,
compiled with g++, on the level chains mg_plan builds), and on the GPU its results against the
cycle that holds every level in the cluster's shared memory, bit for bit."""
import os
import shutil
import subprocess

import numpy as np
import pytest

from tests.test_small_plan import mg_chain

REPO = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

# (Mx, My): wide = the first small level is spread over a cluster; the long thin ones do not fit
SHAPES = [((801, 801), 1), ((401, 401), 1), ((1601, 1601), 1), ((201, 131), 1), ((130, 97), 1), ((128, 128), 1),
          ((127, 129), 1), ((45, 44), 0), ((64, 64), 0), ((63, 65), 1), ((61, 61), 0), ((7, 7), None), ((5, 9), 0),
          ((5, 201), 0), ((33, 17), 0), ((67, 67), 1), ((5, 4000), None), ((3, 1000), None), ((1000, 3), None)]


@pytest.fixture(scope="module")
def checker(tmp_path_factory):
    gxx = shutil.which("g++")
    if gxx is None:
        pytest.skip("no g++")
    exe = str(tmp_path_factory.mktemp("resident") / "resident_plan_check")
    subprocess.run([gxx, "-O1", "-std=c++17", "-I", os.path.join(REPO, "pismv0.7.3_b200", "csrc"),
                    os.path.join(REPO, "tests", "resident_plan_check.cc"), "-o", exe], check=True)
    return exe


@pytest.mark.parametrize("shape,wide", SHAPES)
def test_layout(checker, shape, wide):
    lev, first = mg_chain(*shape)
    line = f"{first} {len(lev)} " + " ".join(f"{a} {b} {c} {d}" for a, b, c, d in lev) + "\n"
    out = subprocess.run([checker], input=line, capture_output=True, text=True, check=True).stdout.split()
    assert out[0] == ("none" if wide is None else "ok"), out
    if wide is not None:
        assert int(out[1]) == wide, out


@pytest.mark.gpu
@pytest.mark.parametrize("Mx,My", [(801, 801), (401, 401), (130, 97), (127, 129), (63, 65), (7, 7), (5, 9), (5, 201),
                                   (67, 67), (3, 1000)])
def test_cycle_bitwise(Mx, My):
    """z = M^-1 r with mg_small_kernel 0 (the resident cycle where the levels fit) and 1 (every
    level a block per CTA in shared memory): the same arithmetic per cell in the same order"""
    import torch
    from pism_b200.config import GridDesc, SSAConfig
    from pism_b200.ssa import SSAFD
    rng = np.random.Generator(np.random.PCG64(Mx * 1000 + My))
    H = rng.uniform(200.0, 2000.0, (Mx, My))
    f = {"thickness": H, "surface": H, "bed": np.zeros((Mx, My)), "mask": rng.choice([0.0, 2.0, 3.0, 4.0], (Mx, My)),
         "tauc": rng.uniform(1e4, 2e5, (Mx, My)), "melange": np.zeros((Mx, My))}
    vel = rng.normal(0.0, 1e-5, (Mx, My, 2))
    # a smooth residual: the coarse correction carries most of z
    i, j = np.arange(Mx)[:, None] / Mx, np.arange(My)[None, :] / My
    wave = np.sin(5.0 * i + 3.0 * j + rng.uniform()) + 0.1 * rng.normal(0.0, 1.0, (Mx, My))
    r = torch.tensor(1e3 * np.stack([wave, wave[::-1, ::-1]], axis=-1).copy(), device="cuda")
    g = GridDesc(Mx, My, 5e3 * (Mx - 1), 5e3 * (My - 1))
    z = {}
    for k in (0, 1):
        s = SSAFD(g, SSAConfig(flow_law="isothermal_glen", pc_type="mg", mg_small_kernel=k))
        s.set_inputs(**f)
        s.set_initial_guess(vel)
        s.assemble_rhs()
        s.compute_hardav_staggered()
        s.compute_nuH_staggered(1e13)
        z[k] = torch.zeros_like(r)
        torch.cuda.synchronize()
        s.apply_preconditioner(r, z[k])
        torch.cuda.synchronize()
        z[k] = z[k].cpu().numpy()
        s.close()
    assert np.isfinite(z[0]).all() and np.abs(z[0]).max() > 0.0
    np.testing.assert_array_equal(z[0], z[1])
