"""The refinement's end on the device (csrc/ssa_state.h refine_more, CPU): a refinement that skips
the pass whose inner solve would find the tolerance met leaves the same state as one that takes it,
and the state of the host loop (linear_solve_mixed), over seeded scenarios with every kind of end."""
import os
import shutil
import subprocess

import numpy as np
import pytest

from tests.test_picard_control import (KSP_BREAKDOWN, KSP_MAXIT, KSP_NAN, KSP_OK, KSP_OUTER_DONE, KSP_STALLED,
                                       host_mixed)

REPO = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.fixture(scope="module")
def driver(tmp_path_factory):
    if shutil.which("g++") is None:
        pytest.skip("needs g++")
    exe = str(tmp_path_factory.mktemp("refine") / "check")
    subprocess.run(["g++", "-std=c++17", "-O1", "-Wall", "-I", os.path.join(REPO, "include"), "-I",
                    os.path.join(REPO, "pismv0.7.3_b200", "csrc"),
                    os.path.join(REPO, "tests", "refine_more_check.cc"), "-o", exe], check=True)
    return exe


def scenario(rng, kind):
    """rtol, max_refine, inner outcomes, norms: enough records for the loop to end by itself"""
    n, rtol, b2 = 12, 10.0 ** rng.uniform(-8, -1), 10.0 ** rng.uniform(-3, 6)
    ends = int(rng.integers(1, 9))   # the record that ends it
    max_refine = ends if kind == "limit" else 60
    rec = [(int(rng.integers(1, 9)), KSP_MAXIT if rng.uniform() < 0.2 else KSP_OK) for _ in range(n)]
    big = [(b2 * (rtol * 10.0 ** rng.uniform(0.1, 3)) ** 2, b2) for _ in range(n + 1)]
    norms = list(big)
    if kind == "met":
        norms[ends] = (b2 * (rtol * 0.5) ** 2, b2)
    elif kind == "nan":
        norms[ends] = (float("nan"), b2)
    elif kind == "inf":
        norms[ends] = (float("inf"), b2)
    elif kind == "zero_b":
        norms = [(r2, 0.0) for r2, _ in norms]
    elif kind == "equal":
        norms[ends] = (b2, b2)
        rtol = 1.0
        norms = [(4.0 * b2, b2) if q < ends else v for q, v in enumerate(norms)]
    elif kind == "inner":
        rec[ends] = (3, KSP_NAN if rng.uniform() < 0.5 else KSP_STALLED)
    elif kind == "stuck":
        rec[ends] = (0, KSP_BREAKDOWN)
    return rtol, max_refine, rec, norms


@pytest.mark.parametrize("kind", ["met", "limit", "nan", "inf", "zero_b", "equal", "inner", "stuck"])
def test_same_state_without_the_last_pass(driver, kind):
    rng = np.random.Generator(np.random.PCG64(sum(map(ord, kind))))
    cases = [scenario(rng, kind) for _ in range(50)]
    text = "".join(" ".join(repr(v) if isinstance(v, float) else str(v) for v in
                            (rtol, most, len(rec), *(x for r in rec for x in r), *(x for q in norms for x in q))) + "\n"
                   for rtol, most, rec, norms in cases)
    out = subprocess.run([driver], input=text, capture_output=True, text=True, check=True).stdout.splitlines()
    assert len(out) == 2 * len(cases)
    skipped = 0
    for q, (rtol, most, rec, norms) in enumerate(cases):
        full, less = out[2 * q].split(), out[2 * q + 1].split()
        assert less[:8] == full[:8]                            # the state
        assert full[8] == full[9] and less[8] == less[9]       # the passes counted are those taken
        assert int(full[9]) - int(less[9]) in (0, 1)
        skipped += int(full[9]) - int(less[9])
        records = []
        for (it, st), (r2, b2) in zip(rec, norms):
            met = not (r2 ** 0.5 > rtol * b2 ** 0.5) or b2 == 0.0
            records.append((0, KSP_OUTER_DONE, r2, b2) if met else (it, st, r2, b2))
        inner, status, steps, final, _ = host_mixed(records, most)
        assert (int(less[3]), int(less[4]), int(less[5])) == (inner, status, steps)
        assert less[7] == full[7] and (float(less[7]) == final or (final != final and less[7] in ("nan", "-nan")))
    # the ends that refine_more decides are those by the residual
    assert skipped == (len(cases) if kind in ("met", "nan", "equal") else 0)
