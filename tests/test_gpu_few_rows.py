"""16-bit MLPs of few rows run layer by layer (fortis_mlp_f32tc.cu, the 16-bit forms): the fused kernel's results bit for
bit, at the edges of tiles, widths that are not multiples of anything, and every precision."""
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

import fortis_b200
from fortis_b200 import descriptors as D


@pytest.fixture()
def host():
    h = fortis_b200.Host()
    h.reset()
    yield h
    h.reset()


def randn(shape, seed):
    return torch.randn(shape, device="cuda", generator=torch.Generator(device="cuda").manual_seed(seed))


@pytest.mark.parametrize("precision", ["bf16", "fp16", "fp8w"])
@pytest.mark.parametrize("dims,rows", [([244, 768, 768, 128], 1), ([244, 768, 768, 128], 129), ([100, 650, 701, 577, 33], 1000),
                                       ([256, 768, 768, 1], 3072), ([244, 768, 768, 128], 3073), ([100, 300, 65, 33], 300)])
def test_few_rows_layer_by_layer_gives_the_fused_kernels_bits(host, precision, dims, rows):
    layers = fortis_b200.mlp_layers(dims, seed=3, act="leaky", slope=0.15, bias="uniform", scale=0.1)
    G, S, Lp, K = D.identity(dims[0], dims[-1], rows)
    x = randn((rows, dims[0]), 10)
    outs, sums = [], []
    for pair in ("1", "default"):
        host.reset()
        host.configure(gather=G, scatter=S, loop=Lp)
        host.option("tc_pair", pair)
        host.option("precision", precision)
        host.option("checksum", 1)
        host.load_model(fortis_b200.write_blob(layers))
        y = torch.full((rows, dims[-1]), float("nan"), device="cuda")
        host.step([x], [y])
        z = torch.full((rows, dims[-1]), float("nan"), device="cuda")
        host.L.mlp_forward_batched(x.data_ptr(), z.data_ptr())       # row-major arrays instead of the descriptors
        host.check()
        assert host.L.fortis_device_status() == 0
        outs.append((y, z))
        sums.append(host.step_checksum())
    assert torch.equal(outs[0][0], outs[1][0]) and torch.equal(outs[0][1], outs[1][1]) and torch.equal(outs[0][0], outs[0][1])
    assert abs(sums[0] - sums[1]) <= 1e-12 * float(outs[0][0].double().abs().sum())     # the same values in another order
