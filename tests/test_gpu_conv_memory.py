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
