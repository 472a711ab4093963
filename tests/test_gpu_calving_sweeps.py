"""The calving front's kernels where their launches can go wrong (csrc/ssa_calving.cu): a last block
and a last warp cut by the grid's end, tongues that need more than one batch of sweeps, a caller's
mask with fractions, and outputs that start off a 16-byte boundary.

Masks, thicknesses and strain rates equal the oracle's bit for bit; the stresses go through pow(),
whose last bit may differ from the host's: 1e-13."""
import numpy as np
import pytest

from oracle import ssafd_oracle as O
from pism_b200 import _capi
from test_gpu_calving import handle, random_front, relmax

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():
    pytest.skip("no CUDA device", allow_module_level=True)


@pytest.mark.parametrize("Mx,My,offset", [(3, 3, 1), (5, 51, 0), (16, 16, 1), (3, 86, 0), (70, 41, 1)])
def test_fronts_on_cut_blocks(Mx, My, offset):
    g, f, vel, Href = random_front(Mx + My, Mx, My)
    G, K = O.Grid(g.Mx, g.My, g.Lx, g.Ly), 1e14
    M = f["mask"].copy()
    if Mx == 70:   # a tongue that goes cell by cell from its tip at the smallest i: sixty sweeps at most
        M[2:66, 17:24] = 4.0
        M[4:66, 20] = 3.0
    H = np.where((M == 2) | (M == 3), 300.0, 0.0)
    ref_m, ref_href, ref_h = O.eigen_calving(G, M, Href, H, vel, 1e7, K)
    ref_e, ref_s = O.principal_strain_rates(G, M, vel), O.deviatoric_stresses_2d(G, O.Config(), M, vel)
    dt, rmax, _, count = O.eigen_calving_max_timestep(G, M, vel, K)
    s = handle(g, f, vel)
    try:
        m = torch.tensor(M + np.random.default_rng(0).uniform(-0.4, 0.4, M.shape), device="cuda")
        buf = torch.full((5 * Mx * My + 3,), 7.0, dtype=torch.float64, device="cuda")
        edot, stress = buf[offset:], buf[offset + 2 * Mx * My:]
        for _ in range(2):   # a second call finds what the first left in the handle
            assert s.lib.pism_gpu_ssa_strain_rates(s._h, ptr(m), ptr(edot), ptr(stress), _capi.MEM_DEVICE) == 0
            out = s.eigen_calving(1e7, K, m, torch.tensor(Href, device="cuda"), torch.tensor(H, device="cuda"))
            step = s.eigen_calving_max_timestep(K, m)
        b = buf.cpu().numpy()
    finally:
        s.close()
    n = Mx * My
    np.testing.assert_array_equal(b[offset:offset + 2 * n].reshape(Mx, My, 2), ref_e)
    assert relmax(b[offset + 2 * n:offset + 5 * n].reshape(Mx, My, 3), ref_s) < 1e-13
    assert np.all(b[:offset] == 7.0) and np.all(b[offset + 5 * n:] == 7.0)
    np.testing.assert_array_equal(out["mask"].cpu().numpy(), ref_m)
    np.testing.assert_array_equal(out["Href"].cpu().numpy(), ref_href)
    np.testing.assert_array_equal(out["thickness"].cpu().numpy(), ref_h)
    assert step["max_rate"] == rmax and step["count"] == count and step["dt"] == pytest.approx(dt, rel=1e-14)


def ptr(t):
    import ctypes
    return ctypes.cast(t.data_ptr(), ctypes.POINTER(ctypes.c_double))
