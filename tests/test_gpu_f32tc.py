"""The split-TF32 tensor-core kernel (fp32 Linear layers and convolutions) at the edges of its tiles, steps and dispatch
rules, against float64.

Tolerance: every product keeps 21 bits of each operand and drops lo.lo, at most 2^-21 + 2^-22 of the
product; the sums add 8 truncations per 64 k and one rounding per chunk, at most 8 * 2^-23 of the partial sums.  With
zero-mean data both stay below 2^-20 = 9.5e-7 of the result's 2-norm.
"""
import ctypes
import hashlib
import os
import subprocess
import sys

import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

import fortis_b200
from fortis_b200 import descriptors

TOL = 2.0 ** -20


@pytest.fixture()
def host():
    h = fortis_b200.Host()
    h.reset()
    yield h
    h.reset()


def rel(a, b):
    a, b = a.double(), b.double()
    return float((a - b).norm() / b.norm())


def memref(t):
    return (t.data_ptr(), t.data_ptr(), 0) + tuple(t.shape) + tuple(t.stride())


def randn(shape, seed, scale=1.0):
    return torch.randn(shape, device="cuda", generator=torch.Generator(device="cuda").manual_seed(seed)) * scale


_keep = []      # weights of the memref entries are constants of the program, told apart by their address


@pytest.mark.parametrize("B,N,K", [(512, 1, 1), (512, 32, 32), (513, 33, 31), (640, 64, 33), (641, 65, 64), (1000, 96, 65), (767, 129, 130),
                                   (2000, 257, 100), (19000, 200, 36)])
def test_gemm_tile_and_step_edges(host, B, N, K):
    A, W = randn((B, K), 1), randn((N, K), 2)
    C = torch.full((B, N), float("nan"), device="cuda")
    _keep.append(W)
    f = host.L.fortis_gemm
    f.argtypes, f.restype = ([ctypes.c_void_p] * 2 + [ctypes.c_long] * 5) * 3 + [ctypes.c_long] * 3, None
    f(*memref(A), *memref(W), *memref(C), B, N, K)
    host.sync()
    assert rel(C, A.double() @ W.double().T) < TOL
    assert host.L.fortis_device_status() == 0


def conv_entry(host, x, w, y, stride, pad):
    conv_call(host, x, w, y, stride, pad)
    host.sync()


def conv_call(host, x, w, y, stride, pad):
    f = host.L.fortis_conv3d
    f.argtypes, f.restype = ([ctypes.c_void_p] * 2 + [ctypes.c_long] * 11) * 3 + [ctypes.c_long] * 18, None
    _keep.append(w)
    f(*memref(x), *memref(w), *memref(y), x.shape[0], x.shape[1], *x.shape[2:], w.shape[0], *w.shape[2:], *y.shape[2:], *stride, *pad)


def conv64(x, w, stride, pad):
    return torch.nn.functional.conv3d(x.cpu().double(), w.cpu().double(), stride=stride, padding=pad).cuda()


@pytest.mark.parametrize("C,F,K,stride,pad,shape", [
    (1, 1, (1, 1, 1), (1, 1, 1), (0, 0, 0), (1, 3, 4, 5)),           # one tap, one channel
    (7, 31, (3, 3, 3), (1, 1, 1), (1, 1, 1), (2, 5, 6, 7)),          # channels one by one
    (8, 33, (2, 3, 4), (1, 2, 3), (0, 1, 3), (1, 6, 9, 11)),         # one group of channels, other extents per axis
    (16, 64, (3, 3, 3), (2, 2, 2), (1, 1, 1), (1, 9, 9, 17)),
    (17, 65, (3, 3, 3), (1, 1, 1), (2, 2, 2), (1, 4, 5, 6)),         # a ragged group; padding wider than K / 2
    (39, 96, (1, 5, 5), (1, 1, 1), (0, 0, 0), (2, 1, 12, 9)),
    (3, 130, (7, 1, 1), (1, 1, 1), (3, 0, 0), (1, 5, 8, 40)),
    (64, 64, (3, 3, 3), (1, 1, 1), (1, 1, 1), (2, 8, 9, 10)),
    (2, 3, (33, 1, 1), (1, 1, 1), (16, 0, 0), (1, 40, 3, 3)),        # more taps on an axis than the kernel takes: FFMA
])
def test_conv_groups_taps_and_strides(host, C, F, K, stride, pad, shape):
    x, w = randn((shape[0], C) + shape[1:], 3), randn((F, C) + K, 4)
    want = conv64(x, w, stride, pad)
    y = torch.full(want.shape, float("nan"), device="cuda")
    conv_entry(host, x, w, y, stride, pad)
    assert rel(y, want) < TOL
    assert host.L.fortis_device_status() == 0


def test_conv_infinities_nans_and_the_largest_values(host):
    """Where fp32 arithmetic gives an infinity or NaN so does the split form, and nowhere else; values that round past
    the largest TF32 value stay finite."""
    x, w = randn((1, 8, 6, 7, 40), 5), randn((5, 8, 3, 3, 3), 6)
    w[0, 0, 0, 0, 0] = 0.5                                            # its low half is exactly zero
    x[0, 1, 2, 3, 4], x[0, 2, 4, 5, 20], x[0, 3, 1, 1, 30] = float("inf"), float("-inf"), float("nan")
    want = conv64(x, w, (1, 1, 1), (1, 1, 1))
    y = torch.zeros(want.shape, device="cuda")
    conv_entry(host, x, w, y, (1, 1, 1), (1, 1, 1))
    assert torch.equal(torch.isnan(y), torch.isnan(want)) and torch.equal(torch.isinf(y), torch.isinf(want))
    inf = torch.isinf(want)
    assert torch.equal(torch.sign(y[inf]).double(), torch.sign(want[inf]))
    fine = torch.isfinite(want)
    assert rel(y[fine], want[fine]) < TOL
    big = torch.full((1, 1, 1, 1, 4), 3.4028234e38, device="cuda")
    w1 = torch.full((1, 1, 1, 1, 1), 0.25, device="cuda")
    y1 = torch.zeros_like(big)
    conv_entry(host, big, w1, y1, (1, 1, 1), (0, 0, 0))
    assert rel(y1, big.double() * 0.25) < TOL


def test_conv_net_whose_last_layer_adds_a_skip(host):
    """Volumes between layers are channel-major, the program's arrays are channels-last: a skip added by the last layer
    is read in the one layout and the result stored in the other."""
    rng = np.random.default_rng(8)
    conv = lambda ci, co: (0.2 * rng.standard_normal((co, ci, 3, 3, 3))).astype(np.float32)
    layers = [dict(W=conv(5, 12), b=rng.standard_normal(12).astype(np.float32), act="leaky", slope=0.1, pad=1, save=True),
              dict(W=conv(12, 20), b=np.zeros(20, np.float32), act="relu", pad=1),
              dict(W=conv(20, 12), b=np.ones(12, np.float32), act="none", pad=1, add=True)]
    x = randn((2, 5, 6, 7, 5), 9)
    y = torch.zeros((2, 5, 6, 7, 12), device="cuda")
    host.load_model(fortis_b200.write_blob(layers))
    host.option("conv_shape", "2,5,6,7")
    host.forward(x, y)
    h, skip = x.double().permute(0, 4, 1, 2, 3), None
    for L in layers:
        h = conv64(h, torch.from_numpy(L["W"]), 1, 1) + torch.from_numpy(L["b"]).double().cuda().reshape(1, -1, 1, 1, 1)
        if L.get("add"):
            h = h + skip
        h = {"none": lambda v: v, "relu": lambda v: v.clamp_min(0), "leaky": lambda v: torch.where(v > 0, v, v * 0.1)}[L["act"]](h)
        if L.get("save"):
            skip = h
    assert rel(y, h.permute(0, 2, 3, 4, 1)) < 3 * TOL                # three layers


@pytest.mark.parametrize("dims,rows", [([244, 768, 128], 511), ([244, 768, 128], 512), ([33, 65, 31, 7], 513), ([64, 1000, 5], 700), ([5, 3], 640)])
def test_mlp_on_either_side_of_the_row_limit(host, dims, rows):
    """Through the descriptors and through row-major arrays; below 512 rows on the FFMA kernels."""
    layers = fortis_b200.mlp_layers(dims, seed=3, act="relu", bias="uniform", scale=0.1)
    G, S, Lp, K = descriptors.identity(dims[0], dims[-1], rows)
    x = randn((rows, dims[0]), 10)
    host.configure(gather=G, scatter=S, loop=Lp)
    host.load_model(fortis_b200.write_blob(layers))
    y, z = (torch.full((rows, dims[-1]), float("nan"), device="cuda") for _ in range(2))
    host.step([x], [y])
    host.L.mlp_forward_batched(x.data_ptr(), z.data_ptr())
    host.check()
    want = x.double()
    for i, L in enumerate(layers):
        want = want @ torch.from_numpy(L["W"]).double().cuda().T + torch.from_numpy(L["b"]).double().cuda()
        if i + 1 < len(layers):
            want = want.clamp_min(0)
    # MLP steps keep all three products in one accumulator for 128 k: 48 truncations instead of 8, under 4 * TOL per layer
    assert rel(y, want) < 4 * TOL * len(layers) and rel(z, want) < 4 * TOL * len(layers)
    assert host.L.fortis_device_status() == 0


def chains():
    """Checksums of chains of layers whose launches may overlap: conv networks that rotate three volumes and add skips, an
    fp32 MLP and a 16-bit one of few rows, each called three times on other inputs."""
    h, out = fortis_b200.Host(), []
    for precision, shape in (("fp32", (1, 9, 10, 33)), ("fp32", (2, 17, 19, 21)), ("bf16", (1, 9, 10, 33))):
        h.reset()
        h.load_model(fortis_b200.write_blob(fortis_b200.conv_layers(3, 64, 3, nblocks=3, seed=6)))
        h.option("precision", precision)
        h.option("conv_shape", "%d,%d,%d,%d" % shape)
        for call in range(3):
            x = randn(shape + (3,), call)
            y = torch.zeros_like(x)
            h.forward(x, y)
            out.append(y)
    for precision, dims, rows in (("fp32", [33, 65, 31, 40, 7], 1300), ("bf16", [100, 200, 64, 96, 33], 700)):
        h.reset()
        h.load_model(fortis_b200.write_blob(fortis_b200.mlp_layers(dims, seed=3, act="leaky", slope=0.2, scale=0.2)))
        h.option("precision", precision)
        h.L.fortis_begin(rows)
        for call in range(3):
            x, y = randn((rows, dims[0]), call), torch.zeros((rows, dims[-1]), device="cuda")
            h.forward_batched(x, y)
            out.append(y)
    assert h.L.fortis_device_status() == 0
    h.reset()
    return hashlib.sha256(b"".join(t.cpu().numpy().tobytes() for t in out)).hexdigest()


def in_child(code, **env):
    return subprocess.run([sys.executable, "-c", "from tests import test_gpu_f32tc as t; " + code], check=True, text=True, stdout=subprocess.PIPE,
                          env=dict(os.environ, **env), cwd=os.path.dirname(os.path.dirname(os.path.abspath(__file__)))).stdout


def test_layers_that_overlap_give_the_bits_of_layers_run_one_by_one():
    assert chains() == in_child("print(t.chains())", FORTIS_NO_PDL="1").split()[-1]


def test_biases_of_a_layer_with_more_feature_tiles_than_sms(host):
    """A CTA then has several tiles whose rows are partly behind the last one, each with a bias table of its own."""
    rng = np.random.default_rng(12)
    C, F = 64, 19100
    W, b = rng.standard_normal((F, C, 1, 1)).astype(np.float32), (10 * rng.standard_normal(F)).astype(np.float32)
    x, y = randn((1, C, 10, 13), 13), torch.zeros((1, F, 10, 13), device="cuda")
    host.load_model(fortis_b200.write_blob([dict(op="conv2d", W=W, b=b, stride=1, pad=0, act="none")]))
    host.option("conv_shape", "1,1,10,13")
    host.forward(x, y)
    want = torch.from_numpy(W[:, :, 0, 0]).double().cuda() @ x.double().reshape(C, 130) + torch.from_numpy(b).double().cuda()[:, None]
    assert rel(y.reshape(F, 130), want) < TOL


@pytest.mark.parametrize("C,K", [(1, (1, 1, 1)), (8, (1, 1, 1)), (27, (1, 1, 1)), (1, (3, 3, 3)), (14, (3, 3, 1)), (15, (3, 3, 1)), (128, (1, 1, 1)), (64, (3, 3, 3))])
@pytest.mark.parametrize("clamp", [False, True])
def test_a_convolution_is_no_less_exact_than_its_fp32_sums(host, C, K, clamp):
    """Against 64 bits, the error of a chain of fp32 fused multiply-adds over the same products (channels inside taps), for
    reductions on both sides of the limit below which operands are not split.  5 % for the sample of 20,000 outputs."""
    x, w = randn((1, C, 8, 10, 12), 14), randn((32, C) + K, 15)
    if clamp:
        x = x.clamp_min(0)
    want = conv64(x, w, (1, 1, 1), (0, 0, 0))
    y = torch.full(want.shape, float("nan"), device="cuda")
    conv_entry(host, x, w, y, (1, 1, 1), (0, 0, 0))
    chain = torch.zeros(want.shape, device="cuda")
    D, H, W = want.shape[2:]
    for kd, kh, kw in np.ndindex(K):
        for c in range(C):          # a product of two fp32 values is exact in 64 bits: one fp32 rounding a step, as in an FMA
            win = x[:, c, None, kd:kd + D, kh:kh + H, kw:kw + W].double()
            chain = (chain.double() + win * w[None, :, c, kd, kh, kw, None, None, None].double()).float()
    assert rel(y, want) <= 1.05 * rel(chain, want)


@pytest.mark.parametrize("dims", [[244, 128], [244, 64, 128]])
def test_host_vectors_updated_in_place(host, dims):
    """Column vectors that a step reads and writes stay in the host's pages; one layer's feature tiles must not read what
    another tile has stored."""
    rows, nlev = 9000, 60
    G, S, Lp, K = descriptors.column(rows, nlev)
    rng = np.random.default_rng(17)
    fields = [np.asfortranarray(rng.standard_normal((rows, nlev)).astype(np.float32)) for _ in range(4)]
    vectors = [rng.standard_normal(rows).astype(np.float32) for _ in range(8)]
    blob = fortis_b200.write_blob(fortis_b200.mlp_layers(dims, seed=3, act="relu"))
    got = []
    for in_place in (False, True):
        host.reset()
        host.configure(gather=G, scatter=S, loop=Lp)
        host.load_model(blob)
        gin = [v.copy() for v in vectors[:4]]
        out = [np.zeros((rows, nlev), np.float32, order="F") for _ in range(2)] + [v if in_place else v.copy() for v in gin] + [v.copy() for v in vectors[4:]]
        host.step(fields + gin, out)
        got.append([a.copy(order="F") for a in out])
    for a, b in zip(*got):
        assert np.array_equal(a, b)


@pytest.mark.parametrize("xe,we", [(-117, 100), (-121, 100), (100, -117), (-60, -55), (120, -120)])
def test_small_and_large_values_keep_their_low_halves(host, xe, we):
    """The tensor core takes subnormal operands as zero; a value's low half is 2^-12 of it and its last bit 2^-23."""
    x, w = randn((1, 64, 5, 8, 8), 24, 2.0 ** xe), randn((32, 64, 3, 3, 3), 25, 2.0 ** we)
    want = conv64(x, w, (1, 1, 1), (0, 0, 0))
    y = torch.full(want.shape, float("nan"), device="cuda")
    conv_entry(host, x, w, y, (1, 1, 1), (0, 0, 0))
    assert rel(y, want) < TOL


def test_captured_calls_keep_their_weights(host):
    """The memref entries keep the prepared weights of 64 layers by address; a graph that holds such an address is replayed
    after more layers than that have been called."""
    f = host.L.fortis_gemm
    f.argtypes, f.restype = ([ctypes.c_void_p] * 2 + [ctypes.c_long] * 5) * 3 + [ctypes.c_long] * 3, None
    gemm = lambda A, W, C: f(*memref(A), *memref(W), *memref(C), A.shape[0], W.shape[0], W.shape[1])
    one, pad = (1, 1, 1), (1, 1, 1)
    shapes = [(20, 16), (3, 5)]                                       # on the tensor cores, on the FFMA kernel
    x = [randn((1, c, 4, 5, 6), 20) for c, _ in shapes]
    w = [randn((o, c, 3, 3, 3), 21) for c, o in shapes]
    y = [torch.zeros((1, o, 4, 5, 6), device="cuda") for _, o in shapes]
    A, B, C = randn((600, 40), 22), randn((24, 40), 23), torch.zeros((600, 24), device="cuda")
    _keep.append(B)
    def calls():
        for i in range(2):
            conv_call(host, x[i], w[i], y[i], one, pad)
        gemm(A, B, C)
    calls()
    host.sync()
    host.L.mgpuStreamCreate.restype = ctypes.c_void_p
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.stream(torch.cuda.ExternalStream(host.L.mgpuStreamCreate())):
        graph.capture_begin(capture_error_mode="relaxed")
        calls()
        graph.capture_end()
        other = [torch.zeros_like(y[0]), torch.zeros_like(y[1]), torch.zeros_like(C)]
        for seed in range(70):
            for i in range(2):
                conv_call(host, x[i], randn(w[i].shape, 100 + seed), other[i], one, pad)
            W = randn(B.shape, 300 + seed)
            _keep.append(W)
            gemm(A, W, other[2])
        for t in x + [A]:
            t.normal_()
        for t in y + [C]:
            t.zero_()
        graph.replay()
        torch.cuda.current_stream().synchronize()
    for i in range(2):
        assert rel(y[i], conv64(x[i], w[i], one, pad)) < TOL
    assert rel(C, A.double() @ B.double().T) < TOL
    assert host.L.fortis_device_status() == 0


def very_many_rows():
    rows, host = 2 ** 31 - 100, fortis_b200.Host()
    layers = fortis_b200.mlp_layers([1, 2, 1], seed=3, act="relu", bias="uniform")
    host.load_model(fortis_b200.write_blob(layers))
    host.L.fortis_begin(rows)
    x, y = torch.empty(rows, device="cuda").uniform_(-1, 1), torch.zeros(rows, device="cuda")
    host.forward_batched(x, y)
    for part in (slice(0, 1000), slice(rows - 1000, rows)):
        want = x[part, None].double()
        for i, L in enumerate(layers):
            want = want @ torch.from_numpy(L["W"]).double().cuda().T + torch.from_numpy(L["b"]).double().cuda()
            want = want if i else want.clamp_min(0)
        assert rel(y[part], want[:, 0]) < TOL


def test_more_rows_than_32_bit_tile_coordinates_hold():
    """Such an MLP call runs on the FFMA kernels.  52 GB on the device, in a process of its own: the library pools memory."""
    if torch.cuda.mem_get_info()[0] < 70e9:
        pytest.skip("needs 70 GB of device memory")
    in_child("t.very_many_rows()")
