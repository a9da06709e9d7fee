"""fp32 convolutions where the device has no room for split volumes: the kernels that need none run, the results are right, and a
network does not free and allocate on every call.  A test option refuses the allocations; no memory is filled up.

Tolerance: as tests/test_gpu_conv_vol.py derives it, 2^-20 of the result's 2-norm per layer."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

import fortis_b200
from fortis_b200.model import write_blob
from tests.test_gpu_conv_vol import TOL, conv3d_layer, rel


@pytest.fixture()
def host():
    h = fortis_b200.Host()
    h.reset()
    yield h
    h.reset()


def network64(layers, x):
    v = torch.from_numpy(x).double().permute(0, 4, 1, 2, 3)
    for l in layers:
        v = torch.nn.functional.conv3d(v, torch.from_numpy(l["W"]).double(), torch.from_numpy(l["b"]).double(), padding=l["pad"])
        if l["act"] == "leaky": v = torch.where(v > 0, v, v * float(np.float32(0.2)))
    return v.permute(0, 2, 3, 4, 1)


# a short first layer; a first layer whose input would be packed
@pytest.mark.parametrize("graph", [0, 1])
@pytest.mark.parametrize("cin", [3, 40])
def test_network_without_room_for_split_volumes(host, cin, graph):
    rng = np.random.default_rng(3)
    layers = [conv3d_layer(rng, ci, co, 3, a) for ci, co, a in [(cin, 32, "leaky"), (32, 32, "leaky"), (32, 5, "none")]]
    host.load_model(write_blob(layers))
    host.option("test_conv_route", 1)
    host.option("graph", graph)
    allocs = lambda: host.L.fortis_debug_launches(b"volume_allocs")

    def call(shape):
        host.option("conv_shape", "%d,%d,%d,%d" % shape)
        x = rng.standard_normal(shape + (cin,)).astype(np.float32)
        y = [np.zeros(shape + (5,), np.float32) for _ in range(4)]
        host.forward(x, y[0])
        before = allocs()
        for v in y[1:]:
            host.forward(x, v)
        assert allocs() == before                              # nothing is tried again
        assert rel(torch.from_numpy(y[0]), network64(layers, x)) < 3 * TOL
        assert all(v.tobytes() == y[0].tobytes() for v in y[1:])
    call((1, 6, 7, 8))
    launches = host.L.fortis_debug_launches(b"conv_vol_kernel")
    host.option("test_volume_limit", 1)
    call((2, 12, 11, 13))
    assert host.L.fortis_debug_launches(b"conv_vol_kernel") == launches
    call((1, 6, 7, 8))                                         # fits what there is
    call((2, 12, 11, 13))


def layer(host, x, w, pad):
    from tests.test_gpu_f32tc import conv_call
    y = torch.full([x.shape[0], w.shape[0]] + [n + 2 * p - k + 1 for n, p, k in zip(x.shape[2:], pad, w.shape[2:])], float("nan"), device="cuda")
    torch.cuda.synchronize()
    conv_call(host, x, w, y, (1, 1, 1), pad)
    host.sync()
    return y


# a kernel that the split-TF32 kernel takes, and one of more taps in a row than that has tables for
@pytest.mark.parametrize("K", [(3, 3, 3), (1, 1, 40)])
@pytest.mark.parametrize("limit", [1, 1 << 19])                # no room for the weights; room for them, not for the volume
def test_layer_without_room_for_a_split_volume(host, K, limit):
    from tests.test_gpu_f32tc import conv64, randn
    pad = tuple(min(1, k // 2) for k in K)
    x, w = randn((1, 32, 9, 33, 60), 1), randn((8, 32) + K, 2)
    host.option("test_conv_route", 1)
    host.option("test_volume_limit", limit)
    launches = host.L.fortis_debug_launches(b"conv_vol_kernel")
    y = layer(host, x, w, pad)
    assert host.L.fortis_debug_launches(b"conv_vol_kernel") == launches
    # sums of up to 1280 products: on the FFMA kernel one rounding each, at random 2^-24 * sqrt(1280 / 3) of the 2-norm = 1.2e-6
    assert rel(y, conv64(x, w, (1, 1, 1), pad)) < 2 * TOL
    assert host.L.fortis_last_error() == 0


def test_model_without_room_for_split_volume_weights(host):
    rng = np.random.default_rng(4)
    layers = [conv3d_layer(rng, ci, co, 3, a) for ci, co, a in [(3, 32, "leaky"), (32, 32, "leaky"), (32, 5, "none")]]
    host.option("test_volume_limit", 1)
    host.load_model(write_blob(layers))
    host.option("conv_shape", "1,6,7,8")
    x, y = rng.standard_normal((1, 6, 7, 8, 3)).astype(np.float32), np.zeros((1, 6, 7, 8, 5), np.float32)
    host.forward(x, y)
    assert rel(torch.from_numpy(y), network64(layers, x)) < 3 * TOL


def test_weights_are_kept_once_per_form_that_calls_take(host):
    """A layer called with one stride and padding packs one form of its weights for split volumes, and repeats nothing."""
    from tests.test_gpu_f32tc import conv64, randn
    x, w = randn((1, 32, 9, 10, 11), 1), randn((64, 32, 3, 3, 3), 2)
    host.option("test_conv_route", 1)
    allocs = lambda: host.L.fortis_debug_launches(b"volume_allocs")
    layer(host, x, randn((64, 32, 3, 3, 3), 3), (1, 1, 1))      # sizes the workspace
    before = allocs()
    for _ in range(3):
        y = layer(host, x, w, (1, 1, 1))
    assert allocs() == before + 1
    assert rel(y, conv64(x, w, (1, 1, 1), (1, 1, 1))) < TOL


def test_weights_and_volumes_are_not_padded_beyond_use(host):
    """One channel, 33^3 taps: padded to 32 channels and features the weights would be 294 MB for 144 KB."""
    from tests.test_gpu_f32tc import conv64, randn
    x, w = randn((1, 1, 36, 37, 38), 1), randn((1, 1, 33, 33, 33), 2)
    host.option("test_conv_route", 1)
    allocs, launches = host.L.fortis_debug_launches(b"volume_allocs"), host.L.fortis_debug_launches(b"conv_vol_kernel")
    y = layer(host, x, w, (0, 0, 0))
    assert host.L.fortis_debug_launches(b"volume_allocs") == allocs and host.L.fortis_debug_launches(b"conv_vol_kernel") == launches
    # 35,937 products on the FFMA kernel, one rounding each of up to 2^-24: at random 6.5e-6 of the 2-norm
    assert rel(y, conv64(x, w, (1, 1, 1), (0, 0, 0))) < 35937 ** 0.5 * 2.0 ** -24


def device_free():
    torch.cuda.synchronize()
    return torch.cuda.mem_get_info()[0]


def workspace_goes_back(graph):
    from tests.test_gpu_f32tc import randn
    host = fortis_b200.Host()
    rng = np.random.default_rng(6)
    host.option("test_conv_route", 1)
    x, w = [randn((1, 32, d, 64, 64), 1) for d in (63, 255)], randn((8, 32, 3, 3, 3), 2)
    layer(host, x[0][:, :, :5].contiguous(), w, (1, 1, 1))
    host.reset()
    torch.cuda.empty_cache()
    before = device_free()
    host.option("test_conv_route", 1)
    if graph:                                                  # one layer, 32 channels: its input is packed into the workspace
        host.load_model(write_blob([conv3d_layer(rng, 32, 3, 3)]))
        host.option("conv_shape", "1,63,64,64")
        host.option("graph", 1)
        xn = rng.standard_normal((1, 63, 64, 64, 32)).astype(np.float32)
        yn = [np.zeros((1, 63, 64, 64, 3), np.float32) for _ in range(3)]
        host.forward(xn, yn[0])
        host.forward(xn, yn[1])                                # captured
    y = [layer(host, v, w, (1, 1, 1)) for v in x]
    if graph:
        host.forward(xn, yn[2])                                # replayed: in the buffer that was outgrown
        assert yn[1].tobytes() == yn[0].tobytes() and yn[2].tobytes() == yn[0].tobytes()
    held = before - device_free()
    assert held > (260 + 65 * graph) << 20, held
    host.reset()
    del y
    torch.cuda.empty_cache()
    kept = before - device_free()                              # the pool keeps the network's input and output, 36 MB, for the next model
    assert kept < 48 << 20, kept


@pytest.mark.parametrize("graph", [0, 1])
def test_the_workspace_of_single_layers_goes_back_to_the_device(graph):
    """A layer's split volume (65 MB) is given back by a reset; one that a graph of the library addresses, also after it was outgrown by
    a larger layer (260 MB), with the graph.  In a process of its own: the library pools memory."""
    import os, subprocess, sys
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    subprocess.run([sys.executable, "-c", "import tests.test_gpu_conv_memory as t; t.workspace_goes_back(%d)" % graph], cwd=root, check=True, timeout=300)
