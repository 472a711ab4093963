"""CUDA tensors that the Python interface makes itself (eigen_calving's copies, a batch's zero guess, the
outputs in memory torch used before) are filled and released on torch's current stream; the
handle works on a stream of its own.  Each test keeps torch's stream busy for some milliseconds
before the call and compares with a call on an idle device."""
import numpy as np
import pytest

from pism_b200 import synthetic as S
from pism_b200.config import GridDesc, SSAConfig

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():
    pytest.skip("no CUDA device", allow_module_level=True)

from pism_b200.ssa import SSAFD  # noqa: E402

NAMES = ("thickness", "surface", "bed", "mask", "tauc", "melange")


def busy(work):
    """some milliseconds of matrix products on torch's stream"""
    for _ in range(20):
        torch.mm(work, work)


@pytest.fixture(scope="module")
def work():
    return torch.ones((4096, 4096), device="cuda")


@pytest.fixture(scope="module")
def front():
    M = 201
    i, j = np.arange(M)[:, None] / M, np.arange(M)[None, :] / M
    H = 600.0 + 300.0 * np.sin(9 * i + 4 * j)
    mask = np.where(np.sin(7 * i + 5 * j) > 0.5, 4.0, np.where(np.sin(3 * i - 8 * j) > 0.0, 3.0, 2.0))
    s = SSAFD(GridDesc(M, M, 1e6, 1e6), SSAConfig(flow_law="isothermal_glen"))
    s.set_inputs(thickness=H, surface=H, bed=np.zeros((M, M)), mask=mask, tauc=np.full((M, M), 5e4),
                 melange=np.zeros((M, M)))
    s.set_initial_guess(1e-5 * np.stack([np.sin(6 * i + j), np.cos(3 * i - 5 * j)], -1))
    d = {"mask": torch.tensor(mask, device="cuda"), "H": torch.tensor(H, device="cuda"),
         "Href": torch.tensor(np.where(mask == 4.0, 20.0, 0.0), device="cuda")}
    yield s, d
    s.close()


@pytest.mark.parametrize("side", [False, True])
def test_eigen_calving_copies(front, work, side):
    s, d = front
    args = (3e6, 1e17, d["mask"], d["Href"], d["H"])
    torch.cuda.synchronize()
    ref = {k: v.clone() for k, v in s.eigen_calving(*args).items()}
    assert not torch.equal(ref["Href"], d["Href"])
    stream = torch.cuda.Stream() if side else torch.cuda.current_stream()
    with torch.cuda.stream(stream):
        for _ in range(3):
            # the copies are given memory that holds other values
            junk = [torch.full_like(d["H"], 1e30) for _ in range(3)]
            torch.cuda.synchronize()
            del junk
            busy(work)
            out = s.eigen_calving(*args)
            torch.cuda.synchronize()
            for k in ref:
                assert torch.equal(out[k], ref[k]), k


def test_outputs_in_memory_still_read(front, work):
    """an output tensor takes the place of one that queued work still reads"""
    s, d = front
    shapes = {"strain": lambda: s.strain_rates(d["mask"], stresses=False, device=True)["edot"],
              "mass": lambda: s.mass_continuity_step(1e6, d["Href"])["thickness"]}
    for name, call in shapes.items():
        for _ in range(3):
            torch.cuda.synchronize()
            out = call()
            torch.cuda.synchronize()
            out.fill_(7.0)
            torch.cuda.synchronize()
            busy(work)
            seen = out + 0.0   # queued behind the products
            del out            # its memory is the next call's
            call()
            torch.cuda.synchronize()
            assert bool((seen == 7.0).all()), name


def test_zero_guess_of_a_batch(work):
    M = 41
    g, c, f, _ = S.build_synthetic(M, 4000e3 / (M - 1), seed=3)
    m = {k: torch.tensor(f[k], device="cuda") for k in NAMES}
    s = SSAFD(g, c.copy(pc_type="mg", precision="mixed", ksp_rtol=1e-6))
    torch.cuda.synchronize()
    ref = s.solve_batch([m])[0][0].clone()
    for _ in range(3):
        junk = torch.full_like(ref, 1e30)
        torch.cuda.synchronize()
        del junk
        busy(work)
        assert torch.equal(s.solve_batch([m])[0][0], ref)
    s.close()


def test_inputs_and_guess_still_being_written(front, work):
    """tensors given right after the operations that make them"""
    s, d = front
    vel = 1e-5 * torch.stack([torch.sin(6 * d["H"]), torch.cos(3 * d["H"])], -1)
    torch.cuda.synchronize()
    for _ in range(3):
        busy(work)
        guess = 2.0 * vel
        s.set_initial_guess(guess)
        got = s.velocity(out=torch.empty_like(vel))
        torch.cuda.synchronize()
        assert torch.equal(got, 2.0 * vel)
        busy(work)
        H = d["H"] + 1.0
        s.set_inputs(thickness=H, surface=H, bed=torch.zeros_like(H), mask=d["mask"], tauc=torch.full_like(H, 5e4),
                     melange=torch.zeros_like(H))
        s.assemble_rhs()
        got = s.driving_stress()
        torch.cuda.synchronize()
        s.set_inputs(thickness=H, surface=H, bed=torch.zeros_like(H), mask=d["mask"], tauc=torch.full_like(H, 5e4),
                     melange=torch.zeros_like(H))
        s.assemble_rhs()
        np.testing.assert_array_equal(got, s.driving_stress())
        s.set_inputs(thickness=d["H"], surface=d["H"], bed=torch.zeros_like(H), mask=d["mask"],
                     tauc=torch.full_like(H, 5e4), melange=torch.zeros_like(H))
