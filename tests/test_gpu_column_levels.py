"""The 3-D fields' kernel (csrc/ssa_column.cu) where its tile can go wrong: one warp's 32 columns cut
by the grid's end, levels around the warp width, and the flow laws of its two forms (one
exponential a level for GPBLD and Paterson-Budd, the general hardness for the others), with cold,
warm and temperate ice.

Tolerance 1e-12 of the largest value: FP64 throughout, exponents up to 61 carry 61 roundings of
1.1e-16, a factor 100 below it."""
import numpy as np
import pytest

from test_gpu_stress_balance import gpu_fields, oracle_fields, random_columns, relmax

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():
    pytest.skip("no CUDA device", allow_module_level=True)


@pytest.mark.parametrize("Mx,My,Mz,law", [(3, 11, 2, "gpbld"), (5, 13, 31, "gpbld"), (4, 8, 32, "pb"), (7, 5, 33, "pb"),
                                          (6, 43, 64, "gpbld"), (5, 7, 41, "arr"), (5, 7, 40, "hooke"),
                                          (3, 3, 101, "isothermal_glen")])
def test_column_fields_match_the_oracle(Mx, My, Mz, law):
    g, c, f, vel = random_columns(Mx + 10 * Mz, Mx, My, Mz, law)
    if f["enthalpy"] is not None:   # 231 K to temperate with more water than the laws admit
        rng = np.random.default_rng(Mz)
        f["enthalpy"] = rng.uniform(1.6e4, 1.1e5, (Mx, My, Mz))
    bmr = np.random.default_rng(1).normal(0.0, 1e-9, (Mx, My))
    ref, got = oracle_fields(g, c, f, vel, bmr), gpu_fields(g, c, f, vel, bmr, True)
    for k in ref:
        assert np.array_equal(got[k], ref[k]) if k in ("u", "v") else relmax(got[k], ref[k]) < 1e-12, k
