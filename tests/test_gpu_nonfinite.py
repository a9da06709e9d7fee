"""NaN and infinite inputs through the activations of every kernel: what the oracle's definitions (np.maximum for ReLU and
max pooling) give, NaN and infinity by infinity."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

import fortis_b200
from fortis_b200 import descriptors as D
from oracle import fortis_oracle as fo


@pytest.fixture()
def host():
    h = fortis_b200.Host()
    h.reset()
    yield h
    h.reset()


def same_specials(got, want):
    got, want = np.asarray(got), np.asarray(want)
    assert np.array_equal(np.isnan(got), np.isnan(want)) and np.array_equal(np.isinf(got), np.isinf(want))
    assert np.isnan(want).any() and np.isfinite(want).any()


@pytest.mark.parametrize("precision,rows,act,mask", [("fp32", 300, "relu", False), ("fp32", 700, "relu", False), ("fp32", 700, "leaky", True),
                                                     ("fp32", 300, "leaky", True), ("bf16", 700, "relu", True), ("bf16", 4000, "relu", True)])
def test_mlp(host, precision, rows, act, mask):
    """Both sides of the fp32 kernels' row limit and of the 16-bit kernels'; `mask`: a final ReLU on some outputs."""
    layers = fortis_b200.mlp_layers([40, 64, 64, 24], seed=3, act=act, slope=0.1)
    m = (np.arange(24) % 2).astype(np.float32) if mask else None
    x = np.random.default_rng(1).standard_normal((rows, 40)).astype(np.float32)
    x[5, 7], x[rows - 1, 39], x[200, 3] = np.nan, np.nan, np.inf
    y = np.zeros((rows, 24), np.float32)
    host.load_model(fortis_b200.write_blob(layers, relu_mask=m))
    host.option("precision", precision)
    host.L.fortis_begin(rows)
    host.forward_batched(x, y)
    with np.errstate(invalid="ignore"):
        same_specials(y, fo.mlp_forward(layers, x, relu_mask=m))


@pytest.mark.parametrize("dims", [[27, 20, 20, 3], [27, 20, 3]])
@pytest.mark.parametrize("fuse", ["0", "1"])
def test_stencil_nets(host, dims, fuse):
    G, S, Lp, K = D.stencil(20, 12, 2)
    layers = fortis_b200.mlp_layers(dims, seed=4, init="uniform", act="relu", bias="uniform")
    rng = np.random.default_rng(2)
    gin = [np.asfortranarray(rng.standard_normal((22, 14, 2)).astype(np.float32)) for _ in range(3)]
    gin[1][5, 6, 1] = np.nan
    out, want = ([np.zeros((22, 14, 2), np.float32, order="F") for _ in range(3)] for _ in range(2))
    host.configure(gather=G, scatter=S, loop=Lp, kdist=K)
    host.load_model(fortis_b200.write_blob(layers))
    host.option("fuse", fuse)
    host.step(gin, out)
    fo.full_step(G, S, Lp, K, layers, gin, want)
    same_specials(np.stack(out), np.stack(want))


@pytest.mark.parametrize("channels", [2, 24])
def test_conv_and_pooling(host, channels):
    """Few channels and many: the two kernels a convolution may take."""
    rng = np.random.default_rng(7)
    conv = lambda ci, co, act: dict(op="conv2d", W=rng.standard_normal((co, ci, 3, 3)).astype(np.float32), b=np.zeros(co, np.float32),
                                    stride=1, pad=1, act=act, slope=0.1)
    layers = [conv(channels, 24, "relu"), dict(op="maxpool2d", channels=24, k=2, stride=2), conv(24, 5, "relu")]
    x = rng.standard_normal((1, channels, 40, 36)).astype(np.float32)
    x[0, 1, 17, 20] = np.nan
    y = np.zeros((1, 5, 20, 18), np.float32)
    host.load_model(fortis_b200.write_blob(layers))
    host.option("conv_shape", "1,1,40,36")
    host.forward(x, y)
    h = np.maximum(fo.conv2d_nchw(x, layers[0]["W"], stride=(1, 1), pad=(1, 1)), 0)
    h = np.maximum(np.maximum(h[:, :, ::2, ::2], h[:, :, 1::2, ::2]), np.maximum(h[:, :, ::2, 1::2], h[:, :, 1::2, 1::2]))
    same_specials(y, np.maximum(fo.conv2d_nchw(h, layers[2]["W"], stride=(1, 1), pad=(1, 1)), 0))


def same_specials64(got, want):
    """Against float64 on the device: too many rows for the oracle."""
    got, want = got.cpu().numpy(), want.cpu().numpy()
    same_specials(got, want)


@pytest.mark.parametrize("pair", [1, 2])
def test_mlp_of_many_rows(host, pair):
    """The kernel on pairs of CTAs and the one that it stands in for."""
    layers = fortis_b200.mlp_layers([40, 768, 300, 24], seed=3, act="relu")
    x = torch.randn((3000, 40), device="cuda", generator=torch.Generator(device="cuda").manual_seed(1))
    x[5, 7], x[2999, 39], x[200, 3], x[1283, 0] = float("nan"), float("nan"), float("inf"), -float("inf")
    y = torch.zeros((3000, 24), device="cuda")
    host.load_model(fortis_b200.write_blob(layers))
    host.option("test_mlp_pair", pair)
    host.L.fortis_begin(3000)
    torch.cuda.synchronize()
    host.forward_batched(x, y)
    v = x.double()
    for l in layers:
        v = v @ torch.from_numpy(l["W"]).cuda().double().T + torch.from_numpy(l["b"]).cuda().double()
        if l.get("act") == "relu": v = torch.where(v < 0, 0.0, v)             # NaN stays NaN
    same_specials64(y, v)


@pytest.mark.parametrize("route", [1, 2])
@pytest.mark.parametrize("act", ["relu", "leaky"])
def test_conv_network(host, route, act):
    """Over split volumes, through the exchange of rows between a tile's warps (line ends, rows 31 and 32) and through a split residual, and
    on the kernel that loads the taps."""
    rng = np.random.default_rng(7)
    conv = lambda ci, co, a, **kw: dict(W=(rng.standard_normal((co, ci, 3, 3, 3)) / np.sqrt(27 * ci)).astype(np.float32), b=np.zeros(co, np.float32), pad=1, act=a, slope=0.1, **kw)
    layers = [conv(5, 40, act, save=True), conv(40, 40, act), conv(40, 40, "none", add=True), conv(40, 3, act)]
    x = rng.standard_normal((1, 14, 11, 40, 5)).astype(np.float32)
    x[0, 1, 5, 39, 2], x[0, 12, 9, 0, 4], x[0, 12, 1, 31, 0] = np.nan, np.nan, np.inf
    y = np.zeros((1, 14, 11, 40, 3), np.float32)
    host.load_model(fortis_b200.write_blob(layers))
    host.option("test_conv_route", route)
    host.option("conv_shape", "1,14,11,40")
    host.forward(x, y)
    v, skip = torch.from_numpy(x).double().permute(0, 4, 1, 2, 3), None
    for l in layers:
        v = torch.nn.functional.conv3d(v, torch.from_numpy(l["W"]).double(), padding=1)
        if l.get("add"): v = v + skip
        if l["act"] == "relu": v = torch.where(v < 0, 0.0, v)
        elif l["act"] == "leaky": v = torch.where(v < 0, v * float(np.float32(0.1)), v)
        if l.get("save"): skip = v
    same_specials64(torch.from_numpy(y), v.permute(0, 2, 3, 4, 1))
