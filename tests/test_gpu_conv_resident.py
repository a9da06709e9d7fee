"""Convolutions whose weights stay in shared memory (conv_vol_kernel<.., RESIDENT>: at most six steps a tile), one to five tiles a pair of
CTAs, and short layers that write a split volume (conv_short_kernel<.., VOL>), against float64.

Tolerance: as in test_gpu_conv_vol.py, 2^-20 of the result's 2-norm for every layer."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

import fortis_b200
from fortis_b200.model import write_blob

TOL = 2.0 ** -20
_keep = []      # weights of the memref entries are constants of the program, told apart by their address


# a pair's tiles are 252 rows (256 with a tap a step), a row a position of the grid, 74 pairs on the device; 2, 3, 6 and 5 steps, 9 do not fit
@pytest.mark.parametrize("C,K", [(43, (1, 1, 3)), (16, (1, 3, 3)), (65, (1, 1, 3)), (40, (1, 3, 3)), (130, (1, 1, 1)), (20, (3, 3, 3))])
@pytest.mark.parametrize("F,H", [(32, 90), (64, 100), (1, 188), (40, 290), (31, 390)])
def test_tiles_per_pair(C, K, F, H):
    from tests.test_gpu_conv import _conv_entry
    from tests.test_gpu_f32tc import memref, randn
    pad = tuple(k // 2 for k in K)
    D = 1 if K[0] == 1 else 3
    x, w = randn((1, C, D, H // D, 200), 1), randn((F, C) + K, 2)
    _keep.append(w)
    want = torch.nn.functional.conv3d(x.double(), w.double(), padding=pad)
    y = torch.full(want.shape, float("nan"), device="cuda")
    torch.cuda.synchronize()                                  # the library runs on a stream of its own
    h = fortis_b200.Host()
    h.reset()
    h.option("test_conv_route", 1)
    before = h.L.fortis_debug_launches(b"conv_vol_kernel")
    for _ in range(2):
        _conv_entry(h.L, "fortis_conv3d", 5)(*memref(x), *memref(w), *memref(y), 1, C, D, H // D, 200, F, *K, *want.shape[2:], 1, 1, 1, *pad)
    h.sync()
    assert h.L.fortis_device_status() == 0 and h.L.fortis_debug_launches(b"conv_vol_kernel") == before + 2
    assert float((y.double() - want).norm() / want.norm()) < TOL
    h.reset()


@pytest.mark.parametrize("ci,co", [(1, 3), (3, 8), (4, 20), (3, 32), (2, 64), (1, 100)])
@pytest.mark.parametrize("H,W", [(5, 9), (61, 130)])
def test_short_layer_writes_the_volume(ci, co, H, W):
    """conv_short_kernel at every number of channels a thread, rows turned in shared memory."""
    rng = np.random.default_rng(3)
    layers = [dict(op="conv2d", W=(rng.standard_normal((b, a, 3, 3)) / np.sqrt(9 * a)).astype(np.float32), b=rng.uniform(-0.1, 0.1, b).astype(np.float32), stride=1, pad=1,
                   act=act, slope=0.1) for a, b, act in ((ci, co, "leaky"), (co, 40, "relu"), (40, 5, "none"))]
    x = torch.randn((2, ci, H, W), device="cuda", generator=torch.Generator(device="cuda").manual_seed(1))
    want = x.double()
    for l in layers:
        want = torch.nn.functional.conv2d(want, torch.from_numpy(l["W"]).cuda().double(), torch.from_numpy(l["b"]).cuda().double(), padding=1)
        want = want.clamp_min(0) if l["act"] == "relu" else torch.where(want > 0, want, want * float(np.float32(0.1))) if l["act"] == "leaky" else want
    h = fortis_b200.Host()
    h.reset()
    h.load_model(write_blob(layers))
    h.option("test_conv_route", 1)
    h.option("conv_shape", "2,1,%d,%d" % (H, W))
    y = torch.full((2, 5, H, W), float("nan"), device="cuda")
    torch.cuda.synchronize()
    h.forward(x, y)
    h.sync()
    assert float((y.double() - want).norm() / want.norm()) < len(layers) * TOL
    h.reset()
