"""The U-Net's kernel forms by shape (csrc/unet.cu): convolution tiles of 16 x 16 and 8 x 16
pixels, one and several channel slices, and the weight gradient's blocks of 32 x 32, 16 x 32
and 16 x 16 channels, at images whose edges cut the tiles.

The forward of a batch equals that of its images alone bit for bit: an output adds the same
products in the same order in every tile.  Gradients: the bounds of tests/test_gpu_unet.py
(6e-2 a layer, 3e-2 on average, relative L2) for the reason given there."""
import numpy as np
import pytest

from oracle import unet_oracle as U

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():
    pytest.skip("needs a CUDA device", allow_module_level=True)

from pism_b200 import learned as Lr  # noqa: E402

DEV = torch.device("cuda", 0)


@pytest.mark.parametrize("B,H,W", [(150, 8, 8), (40, 24, 40), (9, 72, 88), (2, 200, 8)])
def test_batched_forward_equals_single_images(B, H, W):
    rng = np.random.Generator(np.random.PCG64(B))
    x = torch.tensor(rng.standard_normal((B, H, W, 8)).astype(np.float32), device=DEV)
    p = U.init_params(B)
    net, one = Lr.UNet(B, H, W, params=p), Lr.UNet(1, H, W, params=p)
    y = net.forward(x).cpu().numpy()
    for b in (0, B // 2, B - 1):
        assert np.array_equal(y[b], one.forward(x[b:b + 1].contiguous()).cpu().numpy()[0])
    net.close()
    one.close()


@pytest.mark.parametrize("B,H,W", [(3, 104, 136), (5, 24, 56)])
def test_gradients_match_the_oracle(B, H, W):
    rng = np.random.Generator(np.random.PCG64(B + H + W))
    p = U.init_params(B)
    x = rng.standard_normal((B, H, W, 8)).astype(np.float32)
    t = rng.standard_normal((B, H, W, 2)).astype(np.float32)
    o = U.UNetOracle(p, bf16=True)
    o.forward(x)
    _, ref = o.backward(t, np.ones((B, H, W), np.float32))
    net = Lr.UNet(B, H, W, params=p)
    g = torch.empty(U.param_count(), dtype=torch.float32, device=DEV)
    net.forward(torch.tensor(x, device=DEV))
    net.backward(torch.tensor(t, device=DEV), grad_out=g)
    g = g.cpu().numpy()
    net.close()
    offs, head = U.layout()
    pairs = [(a, b) for (_, cout, _), (wo, bo) in zip(U.LAYERS, offs) for a, b in ((wo, bo), (bo, bo + cout))]
    errs = [np.linalg.norm(g[a:b] - ref[a:b]) / np.linalg.norm(ref[a:b]) for a, b in pairs + [(head, g.size)]]
    assert max(errs) < 6e-2 and np.mean(errs) < 3e-2, np.round(errs, 4)
