"""The strain heating's rounding under the Paterson-Budd laws (csrc/ssa_column.cu): its error against
long double is no larger than that of pow(A exp(-Q / RT), -1/n) with the same device functions,
what the kernel evaluated before it took one exponential a level.  Columns whose top level is at
the ice surface, where the pressure is 0 and the temperature the same in every evaluation; the
factor D^(1/n + 1) comes from the isothermal law with softness 1."""
import numpy as np
import pytest

from pism_b200.config import GridDesc, SSAConfig

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():
    pytest.skip("no CUDA device", allow_module_level=True)

from pism_b200.ssa import SSAFD  # noqa: E402

M, TOP = 512, 1000.0


def heating(law, E, vel, **cfg):
    z = np.array([0.0, TOP, 2.0 * TOP])
    H = np.full((M, M), TOP)
    s = SSAFD(GridDesc(M, M, 1e6, 1e6, z=z), SSAConfig(flow_law=law, **cfg))
    s.set_inputs(thickness=H, surface=H, bed=np.zeros((M, M)), mask=np.full((M, M), 2.0), tauc=np.full((M, M), 5e4),
                 melange=np.zeros((M, M)), **({} if E is None else {"enthalpy": np.repeat(E[..., None], 3, axis=2)}))
    s.set_initial_guess(vel)
    out = s.stress_balance_3d()["strain_heating"][..., 1]
    s.close()
    return out


@pytest.mark.parametrize("law,kind", [("pb", "cold"), ("gpbld", "cold"), ("gpbld", "temperate")])
def test_error_against_long_double(law, kind):
    L = np.longdouble
    rng = np.random.Generator(np.random.PCG64(11))
    c = SSAConfig()
    vel = rng.normal(0.0, 1e-5, (M, M, 2))
    D2e = 0.5 * heating("isothermal_glen", None, vel, ice_softness=1.0)
    cap, T0, Tm = c.ice_specific_heat_capacity, c.enthalpy_converter_reference_temperature, c.water_melting_point_temperature
    Es = cap * (Tm - T0)
    E = rng.uniform(cap * (230.0 - T0), Es, (M, M)) if kind == "cold" else Es + rng.uniform(0.0, 3300.0, (M, M))
    got = heating(law, E, vel)
    # what every evaluation shares: the rounded temperature, its exponent and the water's factor
    T = np.where(E < Es, E / cap + T0, Tm) - Tm + Tm
    cold = T < c.Paterson_Budd_critical_temperature
    A = np.where(cold, c.Paterson_Budd_A_cold, c.Paterson_Budd_A_warm)
    x = np.where(cold, c.Paterson_Budd_Q_cold, c.Paterson_Budd_Q_warm) / (c.ideal_gas_constant * T)
    omega = np.minimum(np.where(E <= Es, 0.0, (E - Es) / c.water_latent_heat_fusion), c.gpbld_water_frac_observed_limit)
    water = 1.0 + c.gpbld_water_frac_coeff * omega if law == "gpbld" else np.ones((M, M))
    p = 1.0 / c.ssa_Glen_exponent
    true = L(2.0) * (L(1.0) * A * np.exp(-L(1.0) * x) * water) ** (-L(p)) * D2e
    t = lambda a: torch.tensor(a, device="cuda")   # noqa: E731
    plain = (2.0 * torch.pow(t(A) * torch.exp(-t(x)) * t(water), -p) * t(D2e)).cpu().numpy()
    rms = lambda v: float(np.sqrt(np.mean(((v - true) / true).astype(np.float64) ** 2)))   # noqa: E731
    print(law, kind, "here", rms(got), "pow(exp())", rms(plain))
    assert rms(got) <= rms(plain)
