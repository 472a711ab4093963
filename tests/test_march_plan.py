"""The marching fine-level passes' division of a grid (CPU, csrc/ssa_march_plan.h compiled with g++):
every cell is some warp's, and the partial sums of the fused pass, two a block, fit what a handle
allocates for them whatever the device's SMs (eight a resident block was too little for a grid of
many columns on a small device)."""
import os
import shutil
import subprocess

import numpy as np
import pytest

REPO = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.fixture(scope="module")
def driver(tmp_path_factory):
    if shutil.which("g++") is None:
        pytest.skip("needs g++")
    exe = str(tmp_path_factory.mktemp("march") / "check")
    subprocess.run(["g++", "-std=c++17", "-O1", "-Wall", "-I", os.path.join(REPO, "pismv0.7.3_b200", "csrc"),
                    os.path.join(REPO, "tests", "march_plan_check.cc"), "-o", exe], check=True)
    return exe


def shapes():
    rng = np.random.Generator(np.random.PCG64(7))
    out = [(3, 262144), (3, 265217), (3, 66001), (4096, 262144), (262144, 3), (801, 801), (3, 3), (7, 27), (7, 28), (7, 29)]
    for _ in range(300):
        out.append((int(np.exp(rng.uniform(np.log(3), np.log(4000)))), int(np.exp(rng.uniform(np.log(3), np.log(262144))))))
    return out


@pytest.mark.parametrize("sms", [148, 132, 40, 16, 1])
def test_cover_and_partials(driver, sms):
    cases = shapes()
    text = "".join(f"{Mx} {My} {sms}\n" for Mx, My in cases)
    rows = subprocess.run([driver], input=text, capture_output=True, text=True, check=True).stdout.split("\n")
    for (Mx, My), row in zip(cases, rows):
        v = [int(x) for x in row.split()]
        for q, (W, align) in enumerate(((30, 2), (30, 1), (28, 1))):
            strips, R, chunks, blocks = v[4 * q:4 * q + 4]
            assert strips * W >= My > (strips - 1) * W
            assert R >= 1 and R % align == 0 and chunks * R >= Mx > (chunks - 1) * R
            assert 4 * blocks >= strips * chunks
        # what pism_gpu_ssa_create allocates
        assert max(4 * sms * 8, v[12]) >= 2 * v[11], (Mx, My, sms)
