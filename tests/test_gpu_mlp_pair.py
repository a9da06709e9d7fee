"""fp32 MLP steps on pairs of CTAs (fortis_mlp_pair.cu) and on the split-TF32 kernel: the same sums, so a row's outputs are the same bits
on either and however many rows are in the call.  The edges of the pairs' tiles (128 and 256 rows, 128 and 256 features, 32 k and chunks of
128), both kinds of input and output, all activations.  A test option says which kernel runs, a counter that it did."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

import fortis_b200
from fortis_b200 import descriptors as D
from fortis_b200.model import mlp_layers, write_blob


@pytest.fixture()
def host():
    h = fortis_b200.Host()
    h.reset()
    yield h
    h.reset()


def forward(host, x, n_out):
    y = torch.full((x.shape[0], n_out), float("nan"), device="cuda")
    torch.cuda.synchronize()
    host.L.fortis_begin(x.shape[0])
    host.forward_batched(x, y)
    return y


def pairs(host, on):
    host.option("test_mlp_pair", 1 if on else 2)
    return host.L.fortis_debug_launches(b"mlp_pair_kernel")


@pytest.mark.parametrize("dims,rows,act", [
    ([40, 32, 5], 513, "leaky"), ([31, 130, 64, 257], 1000, "relu"), ([64, 96, 128, 1], 2049, "leaky"),
    ([33, 768, 1], 9217, "leaky"), ([244, 800, 768, 130], 9344, "relu"), ([1, 1023, 1025, 256], 7000, "leaky"), ([768, 768, 300], 9343, "leaky"),
    ([129, 2049, 31], 3500, "relu"),
])
def test_rows_have_the_same_bits_in_calls_of_any_size(host, dims, rows, act):
    layers = mlp_layers(dims, seed=2, act=act, bias="uniform")
    in_div = np.linspace(0.5, 2.0, dims[0]).astype(np.float32)
    out_mul = np.linspace(-1.0, 3.0, dims[-1]).astype(np.float32)
    host.load_model(write_blob(layers, in_div=in_div, out_mul=out_mul))
    x = torch.randn((rows, dims[0]), device="cuda", generator=torch.Generator(device="cuda").manual_seed(1))
    before = pairs(host, True)
    y = forward(host, x, dims[-1])
    assert pairs(host, False) - before == len(dims) - 1
    assert torch.equal(y, forward(host, x, dims[-1]))
    assert pairs(host, False) - before == len(dims) - 1
    if rows > 1500:
        parts = torch.cat([forward(host, x[r:r + 1500].contiguous(), dims[-1]) for r in range(0, rows - 1500, 1500)])
        assert torch.equal(y[:parts.shape[0]], parts)
    v = x.double() / torch.from_numpy(in_div).cuda().double()
    for k, l in enumerate(layers):
        v = v @ torch.from_numpy(l["W"]).cuda().double().T + torch.from_numpy(l["b"]).cuda().double()
        if l.get("act") == "relu": v = v.clamp_min(0)
        elif l.get("act") == "leaky": v = torch.where(v > 0, v, v * float(np.float32(l["slope"])))
    v = v * torch.from_numpy(out_mul).cuda().double()
    assert float((y.double() - v).norm() / v.norm()) < 1e-5


def test_gathered_step_and_its_checksum(host):
    """The column step over device arrays: inputs through the slot table, outputs scattered, the checksum folded in the launch."""
    ncol = 9601
    G, S, L, K = D.column(ncol, 60)
    host.configure(gather=G, scatter=S, loop=L, kdist=K)
    layers = mlp_layers([244, 768, 768, 128], seed=0)
    host.load_model(write_blob(layers))
    g = torch.Generator(device="cuda").manual_seed(3)
    gin = [torch.randn((60, ncol), device="cuda", generator=g) for _ in range(4)] + [torch.randn(ncol, device="cuda", generator=g) for _ in range(4)]
    out = [torch.zeros((60, ncol), device="cuda") for _ in range(2)] + [torch.zeros(ncol, device="cuda") for _ in range(8)]
    host.option("checksum", "1")
    torch.cuda.synchronize()
    pairs(host, False)
    host.step(gin, out)
    host.sync()
    checksum, general = host.step_checksum(), [v.clone() for v in out]
    for v in out:
        v.zero_()
    torch.cuda.synchronize()
    before = pairs(host, True)
    host.step(gin, out)
    host.sync()
    assert pairs(host, True) - before == 3
    assert all(torch.equal(a, b) for a, b in zip(out, general))
    x = torch.cat([f.T for f in gin[:4]] + [v[:, None] for v in gin[4:]], dim=1).double()
    for l in layers:
        x = x @ torch.from_numpy(l["W"]).cuda().double().T + torch.from_numpy(l["b"]).cuda().double()
        if l.get("act") == "leaky": x = torch.where(x > 0, x, x * float(np.float32(l["slope"])))
    y = torch.cat([out[0].T, out[1].T] + [v[:, None] for v in out[2:]], dim=1)
    assert float((y.double() - x).norm() / x.norm()) < 1e-5
    bound = 1e-12 * float(y.double().abs().sum())
    assert abs(host.step_checksum() - float(y.double().sum())) <= bound and abs(checksum - float(y.double().sum())) <= bound


# where pairs are faster, and widths and rows whose tiles they would mostly pad or leave a round mostly empty
@pytest.mark.parametrize("dims,rows,on", [([244, 768, 768, 768, 768, 128], 30011, True), ([129, 2049, 31], 3500, True), ([244, 768, 768, 768, 128], 9345, True),
                                          ([244, 896, 896, 896, 128], 8000, False), ([500, 768, 3], 11400, False), ([244, 1024, 1024, 1024, 128], 7000, False),
                                          ([244, 767, 128], 30011, False)])
def test_pairs_run_where_they_are_faster(host, dims, rows, on):
    host.load_model(write_blob(mlp_layers(dims, seed=2, act="leaky", bias="uniform")))
    x = torch.randn((rows, dims[0]), device="cuda", generator=torch.Generator(device="cuda").manual_seed(1))
    before = host.L.fortis_debug_launches(b"mlp_pair_kernel")
    forward(host, x, dims[-1])
    assert host.L.fortis_debug_launches(b"mlp_pair_kernel") - before == (len(dims) - 1 if on else 0)


def staged_step():
    import fortis_b200
    ncol = 20000
    h = fortis_b200.Host()
    G, S, L, K = D.column(ncol, 60)
    h.configure(gather=G, scatter=S, loop=L, kdist=K)
    h.load_model(write_blob(mlp_layers([244, 768, 768, 128], seed=0)))
    rng = np.random.default_rng(1)
    gin = [np.asfortranarray(rng.standard_normal((ncol, 60)).astype(np.float32)) for _ in range(4)] + [rng.standard_normal(ncol).astype(np.float32) for _ in range(4)]
    out = [np.zeros((ncol, 60), np.float32, order="F") for _ in range(2)] + [np.zeros(ncol, np.float32) for _ in range(8)]
    torch.cuda.synchronize()
    before = torch.cuda.mem_get_info()[0]
    for _ in range(3):
        h.step(gin, out)
    used = before - torch.cuda.mem_get_info()[0]
    # staged inputs and outputs 30 MB, the model's 30, weights 15; activations of a chunk of up to 6784 columns two times 21 (of all 20,000,
    # split, two times 123); 32 MB for what the runtime allocates with the first launches
    assert used < (30 + 30 + 15 + 42 + 32) << 20, used >> 20
    assert np.isfinite(out[0]).all() and np.abs(out[0]).max() > 0


def test_a_staged_step_holds_activations_for_its_chunks():
    """Of a step over host arrays the chunks decide which kernel runs and how much lies between the layers, not the whole call.  In a
    process of its own: the library pools memory."""
    import os, subprocess, sys
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    subprocess.run([sys.executable, "-c", "import tests.test_gpu_mlp_pair as t; t.staged_step()"], cwd=root, check=True, timeout=300)
