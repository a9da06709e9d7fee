"""2-D operator networks whose convolutions write the next one's split volume: rows that move to another grid, phases of strided layers,
channels that are not multiples of 32, short first layers, extents that change, against float64.

Tolerance: as in test_gpu_conv_vol.py, 2^-20 of the result's 2-norm for every layer on the tensor cores; sums of fewer than 128 products
on the FFMA kernels stay below that."""
import math

import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

import fortis_b200
from fortis_b200.model import write_blob

_rng = np.random.default_rng(3)


def conv(ci, co, k, stride=1, pad=0, act="leaky"):
    kh, kw = k if isinstance(k, tuple) else (k, k)
    return dict(op="conv2d", W=_rng.normal(0.0, math.sqrt(2.0 / (kh * kw * ci)), size=(co, ci, kh, kw)).astype(np.float32),
                b=_rng.uniform(-0.1, 0.1, co).astype(np.float32), stride=stride, pad=pad, act=act, slope=0.1)


NETS = {
    "short, same grid, stride 2, 1x1": [conv(3, 32, 3, 1, 1), conv(32, 33, 3, 1, 1), conv(33, 64, 3, 2, 1), conv(64, 20, 1)],
    "stride 3 after 5x5, no padding": [conv(16, 40, 5, 1, 2), conv(40, 40, 3, 3, 0), conv(40, 7, 3, 1, 1, "none")],
    "a line kernel feeds taps": [conv(20, 48, 3, 1, 1, "relu"), conv(48, 30, (2, 4), 1, 0), conv(30, 33, 2, 2, 1, "none")],
    "stride beyond the kernel": [conv(32, 36, 3, 1, 1), conv(36, 50, 2, 3, 0), conv(50, 10, 3, 1, 1, "none")],
}


def exact(layers, x):
    for l in layers:
        x = torch.nn.functional.conv2d(x, torch.from_numpy(l["W"]).cuda().double(), torch.from_numpy(l["b"]).cuda().double(), stride=l["stride"], padding=l["pad"])
        x = x.clamp_min(0) if l["act"] == "relu" else torch.where(x > 0, x, x * float(np.float32(l["slope"]))) if l["act"] == "leaky" else x
    return x


@pytest.mark.parametrize("route", [0, 1, 2])
@pytest.mark.parametrize("name", NETS)
def test_layers_write_the_next_ones_volume(name, route):
    layers = NETS[name]
    h = fortis_b200.Host()
    h.reset()
    h.load_model(write_blob(layers))
    h.option("test_conv_route", route)
    for N, H, W in ((1, 13, 9), (3, 40, 131), (2, 21, 64), (3, 40, 131)):
        x = torch.randn((N, layers[0]["W"].shape[1], H, W), device="cuda", generator=torch.Generator(device="cuda").manual_seed(N * H))
        want = exact(layers, x.double())
        h.option("conv_shape", "%d,1,%d,%d" % (N, H, W))
        for _ in range(2):
            y = torch.full(want.shape, float("nan"), device="cuda")
            h.forward(x, y)
            h.sync()
            assert h.L.fortis_device_status() == 0
            assert float((y.double() - want).norm()) <= len(layers) * 2.0 ** -20 * float(want.norm())
    h.reset()


def test_without_memory_for_the_volumes():
    layers = NETS["short, same grid, stride 2, 1x1"]
    x = torch.randn((1, 3, 40, 131), device="cuda", generator=torch.Generator(device="cuda").manual_seed(1))
    want = exact(layers, x.double())
    h = fortis_b200.Host()
    for limit in (1, 1 << 20, 0):
        h.reset()
        h.option("test_volume_limit", limit)
        h.load_model(write_blob(layers))
        h.option("conv_shape", "1,1,40,131")
        for _ in range(2):
            y = torch.full(want.shape, float("nan"), device="cuda")
            h.forward(x, y)
            h.sync()
            assert float((y.double() - want).norm()) <= len(layers) * 2.0 ** -20 * float(want.norm())
    h.reset()
