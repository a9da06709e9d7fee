"""fp32 convolutions over split volumes (fortis_conv3d_f32.cu) at the edges of their tiles, stages, phases and grids, against
float64.

Tolerance: every product keeps 21 bits of each operand and drops lo.lo, at most 2^-21 + 2^-22 of the product; the sums add 4 or 8
truncations per 32 or 64 k and one rounding per chunk, at most 8 * 2^-23 of the partial sums.  With zero-mean data both stay below
2^-20 = 9.5e-7 of the result's 2-norm; a network of L layers adds them up: L * 2^-20.
"""
import os
import re

import numpy as np
import pytest

torch = pytest.importorskip("torch")

import fortis_b200
from fortis_b200.model import write_blob

TOL = 2.0 ** -20
_keep = []      # weights of the memref entries are constants of the program, told apart by their address


@pytest.fixture()
def host():
    h = fortis_b200.Host()
    h.reset()
    yield h
    h.reset()


def rel(a, b):
    a, b = a.double(), b.double()
    return float((a - b).norm() / b.norm())


def on_device(host, route):
    host.option("test_conv_route", {"volume": 1, "loads": 2}[route])
    return lambda: host.L.fortis_debug_launches(b"conv_vol_kernel")


# (N, C, F, D, H, W), kernel, stride, padding: one line's taps a step (three wide, stride 1, padding 0 and 1) and a tap a step (others);
# stages of a plane, of a line (wide volumes), of a tap (strides); phases; padding of K and more; rows 126, 127, 252, 253 of a tile and
# a pair; channels 8 to 100 in blocks of 32, features 1 to 130 in tiles of 32 and 64; lines of one and two positions.  Every case
# runs on both kernels, whatever the estimate would choose; sums of fewer than 128 products run on neither
@pytest.mark.gpu
@pytest.mark.parametrize("route", ["volume", "loads"])
@pytest.mark.parametrize("shape,K,stride,pad", [
    ((1, 32, 64, 3, 6, 7), (3, 3, 3), (1, 1, 1), (1, 1, 1)),
    ((1, 16, 1, 1, 1, 126), (1, 3, 3), (1, 1, 1), (0, 1, 1)),
    ((1, 48, 33, 1, 1, 127), (1, 1, 3), (1, 1, 1), (0, 0, 1)),
    ((1, 64, 32, 1, 2, 126), (1, 3, 3), (1, 1, 1), (0, 1, 1)),
    ((1, 43, 64, 1, 1, 253), (1, 1, 3), (1, 1, 1), (0, 0, 1)),
    ((2, 8, 130, 5, 4, 6), (3, 3, 3), (1, 1, 1), (0, 0, 0)),
    ((2, 100, 40, 4, 5, 3), (3, 3, 3), (1, 1, 1), (1, 0, 1)),
    ((1, 9, 65, 7, 6, 1), (3, 3, 3), (1, 1, 1), (1, 1, 1)),
    ((1, 24, 20, 6, 6, 2), (3, 3, 3), (1, 1, 1), (1, 1, 1)),
    ((1, 16, 64, 9, 10, 11), (3, 3, 3), (2, 2, 1), (1, 1, 1)),
    ((2, 32, 64, 9, 8, 13), (3, 3, 3), (2, 2, 2), (1, 1, 1)),
    ((1, 20, 17, 9, 10, 11), (5, 5, 5), (1, 1, 1), (2, 2, 2)),
    ((1, 8, 64, 12, 11, 10), (5, 3, 4), (3, 1, 2), (1, 2, 0)),
    ((1, 64, 64, 1, 5, 300), (1, 3, 3), (1, 1, 1), (0, 1, 1)),
    ((1, 32, 32, 1, 6, 300), (1, 5, 5), (1, 1, 1), (0, 2, 2)),
    ((1, 130, 31, 4, 4, 5), (1, 1, 1), (1, 1, 1), (0, 0, 0)),
    ((1, 130, 12, 4, 4, 5), (1, 1, 1), (2, 1, 2), (1, 2, 3)),
    ((1, 32, 16, 3, 3, 3), (2, 2, 3), (1, 1, 1), (3, 2, 4)),
    ((1, 40, 64, 1, 7, 200), (1, 3, 3), (1, 2, 1), (0, 1, 0)),
    ((1, 48, 20, 1, 1, 126), (1, 3, 3), (1, 1, 1), (0, 1, 1)),
    ((1, 16, 65, 7, 6, 1), (3, 3, 3), (1, 1, 1), (1, 1, 1)),
    ((2, 24, 30, 9, 9, 12), (3, 3, 3), (2, 2, 2), (1, 1, 1)),
    ((1, 33, 96, 10, 7, 9), (3, 3, 3), (3, 2, 2), (0, 1, 2)),
    ((1, 32, 32, 11, 5, 6), (4, 1, 2), (2, 1, 3), (1, 0, 1)),
    ((2, 64, 64, 33, 33, 33), (3, 3, 3), (1, 1, 1), (1, 1, 1)),
])
def test_layers(host, shape, K, stride, pad, route):
    from tests.test_gpu_conv import _conv_entry
    from tests.test_gpu_f32tc import memref, randn
    N, C, F, D, H, W = shape
    x, w = randn((N, C, D, H, W), 1), randn((F, C) + K, 2)
    _keep.append(w)
    want = torch.nn.functional.conv3d(x.double(), w.double(), stride=stride, padding=pad)
    y = torch.full(want.shape, float("nan"), device="cuda")
    torch.cuda.synchronize()                                  # the library runs on a stream of its own
    launches = on_device(host, route)
    before = launches()
    _conv_entry(host.L, "fortis_conv3d", 5)(*memref(x), *memref(w), *memref(y), N, C, D, H, W, F, *K, *want.shape[2:], *stride, *pad)
    host.sync()
    assert rel(y, want) < TOL
    products = C * min(K[0], D) * min(K[1], H) * min(K[2], W)
    assert launches() - before == (route == "volume" and products >= 128)


def conv3d_layer(rng, ci, co, k, act="none", **flags):
    return dict(W=(rng.standard_normal((co, ci, k, k, k)) / np.sqrt(ci * k ** 3)).astype(np.float32),
                b=(0.1 * rng.standard_normal(co)).astype(np.float32), pad=k // 2, act=act, slope=0.2, **flags)


# widths that are no multiples of 32, kernels of one and two widths, a first layer that is short and one that is not, residuals
@pytest.mark.gpu
@pytest.mark.parametrize("route", ["volume", "loads"])
@pytest.mark.parametrize("spec", [
    [(3, 24, 3), (24, 24, 3), (24, 5, 3)],
    [(6, 40, 3), (40, 40, 5), (40, 40, 3), (40, 2, 3)],
    [(2, 70, 5), (70, 70, 3), (70, 33, 3)],
    [(130, 20, 1), (20, 36, 3), (36, 36, 5), (36, 3, 3)],
])
def test_networks_change_their_extents(host, spec, route):
    """Volumes of other extents in the same buffers: the padding is zero again, whatever lay there before."""
    launches = on_device(host, route)
    before = launches()
    rng = np.random.default_rng(3)
    layers = [conv3d_layer(rng, ci, co, k, "leaky" if l < len(spec) - 1 else "none") for l, (ci, co, k) in enumerate(spec)]
    layers[0]["save"] = True
    if spec[1][1] == spec[0][1]: layers[1]["add"] = True
    host.load_model(write_blob(layers))
    for shape in [(2, 7, 6, 9), (1, 4, 9, 5), (2, 7, 6, 9)]:
        host.option("conv_shape", "%d,%d,%d,%d" % shape)
        x = rng.standard_normal(shape + (spec[0][0],)).astype(np.float32)
        y = np.zeros(shape + (spec[-1][1],), np.float32)
        host.forward(x, y)
        v, skip = torch.from_numpy(x).double().permute(0, 4, 1, 2, 3), None
        for l in layers:
            v = torch.nn.functional.conv3d(v, torch.from_numpy(l["W"]).double(), torch.from_numpy(l["b"]).double(), padding=l["pad"])
            if l.get("add"): v = v + skip
            if l["act"] == "leaky": v = torch.where(v > 0, v, v * float(np.float32(0.2)))
            if l.get("save"): skip = v
        assert rel(torch.from_numpy(y), v.permute(0, 2, 3, 4, 1)) < len(layers) * TOL
    on_volumes = sum(ci * min(k, 6) ** 3 >= 128 for ci, _, k in spec)
    assert launches() - before == (3 * on_volumes if route == "volume" else 0)


# few channels with many taps, 1x1x1 layers: volumes pad channels to 32, and the general kernel is up to three times as fast
@pytest.mark.gpu
@pytest.mark.parametrize("width,k,cin,extents,over_volumes", [
    (8, 5, 3, (1, 20, 20, 20), False), (8, 5, 8, (2, 33, 33, 33), False), (24, 5, 3, (1, 8, 9, 10), False), (160, 1, 3, (2, 33, 33, 33), False),
    (32, 3, 3, (1, 20, 20, 20), True), (64, 3, 3, (2, 12, 13, 14), True), (64, 3, 64, (1, 8, 9, 10), True), (128, 5, 128, (1, 8, 9, 10), True),
])
def test_networks_run_over_volumes_where_that_is_faster(host, width, k, cin, extents, over_volumes):
    rng = np.random.default_rng(3)
    host.load_model(write_blob([conv3d_layer(rng, ci, co, k) for ci, co in [(cin, width), (width, width), (width, width), (width, 3)]]))
    host.option("conv_shape", "%d,%d,%d,%d" % extents)
    x = torch.randn(extents + (cin,), device="cuda", generator=torch.Generator(device="cuda").manual_seed(1))
    y, general = [torch.zeros(extents + (3,), device="cuda") for _ in range(2)]
    torch.cuda.synchronize()
    before = host.L.fortis_debug_launches(b"conv_vol_kernel")
    host.forward(x, y)
    launched = host.L.fortis_debug_launches(b"conv_vol_kernel") - before
    assert launched == (3 + (cin * k ** 3 >= 128) if over_volumes else 0)
    host.option("test_conv_route", 2)
    host.forward(x, general)
    assert rel(y, general) < 2 * 4 * TOL


@pytest.mark.gpu
@pytest.mark.parametrize("H,W", [(17, 23), (64, 50)])
def test_pooling_and_upsampling_on_the_way_into_a_convolution(host, H, W):
    rng = np.random.default_rng(5)

    def conv(ci, co, k, act="none", stride=1):
        return dict(op="conv2d", W=(rng.standard_normal((co, ci, k, k)) / np.sqrt(ci * k * k)).astype(np.float32),
                    b=(0.1 * rng.standard_normal(co)).astype(np.float32), stride=stride, pad=k // 2, act=act, slope=0.1)
    layers = [conv(3, 20, 3, "leaky"), dict(op="maxpool2d", channels=20, k=3, stride=2), conv(20, 36, 3, "relu"), dict(op="upsample2d", channels=36, scale=3),
              conv(36, 17, 5, "leaky"), dict(op="maxpool2d", channels=17, k=2, stride=2), dict(op="upsample2d", channels=17, scale=2), conv(17, 4, 3)]
    host.load_model(write_blob(layers))
    host.option("conv_shape", "2,1,%d,%d" % (H, W))
    x = rng.standard_normal((2, 3, H, W)).astype(np.float32)
    v = torch.from_numpy(x).double()
    for l in layers:
        if l["op"] == "conv2d":
            v = torch.nn.functional.conv2d(v, torch.from_numpy(l["W"]).double(), torch.from_numpy(l["b"]).double(), stride=l["stride"], padding=l["pad"])
            v = v.clamp_min(0) if l["act"] == "relu" else torch.where(v > 0, v, v * float(np.float32(0.1))) if l["act"] == "leaky" else v
        elif l["op"] == "maxpool2d":
            v = torch.nn.functional.max_pool2d(v, l["k"], l["stride"])
        else:
            v = torch.nn.functional.interpolate(v, scale_factor=l["scale"], mode="nearest")
    y = np.zeros(v.shape, np.float32)
    host.forward(x, y)
    assert rel(torch.from_numpy(y), v) < 4 * TOL


def test_launch_order_rules_in_the_source():
    """As tests/test_kernel_source_cpu.py checks of the other programmatically launched kernels: dependents are released after the
    tensor memory is allocated, and what the grid in front may write is not read as constant memory."""
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    text = open(os.path.join(root, "fortis_b200", "csrc", "fortis_conv3d_f32.cu")).read()
    start = text.index("conv_vol_kernel(const __grid_constant__")
    body = re.sub(r"//[^\n]*", "", text[start:text.index("\n}\n", start)])
    alloc, release = body.index("tcgen05.alloc"), body.index("griddepcontrol.launch_dependents")
    assert alloc < release and "__syncthreads()" in body[alloc:release] and "cluster_sync_all()" in body[alloc:release]
    assert "ld.global.nc" not in text
    for line in body.splitlines():
        assert not ("__ldg" in line and any(w in line for w in ["P.skip", "P.res", "src"])), line.strip()


def test_register_split_adds_up():
    """setmaxnreg draws on the registers the block was launched with: the warpgroups' shares are what 512 threads of 128 have."""
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    text = open(os.path.join(root, "fortis_b200", "csrc", "fortis_conv3d_f32.cu")).read()
    dec, inc = [int(v) for v in re.findall(r"setmaxnreg\.dec\.sync\.aligned\.u32 (\d+)", text)], [int(v) for v in re.findall(r"setmaxnreg\.inc\.sync\.aligned\.u32 (\d+)", text)]
    assert len(dec) == 2 and len(inc) == 1 and 128 * sum(dec) + 256 * inc[0] <= 128 * 512
