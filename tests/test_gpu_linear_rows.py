"""fp32 layers of few rows (linear_rows_kernel) at the edges of their tiles, chunks of K and rounds, with rows on and off sixteen bytes,
against float64.

Tolerance: an output is one sum of K products in the order of the inputs, every step rounded once: |error| <= (K + 2) 2^-24 sum |a||w|,
element by element (twice that with the division by the input norms in front).  Where the order is exact arithmetic, small whole numbers,
there is no error at all."""
import ctypes

import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

import fortis_b200


def memref(t):
    return (t.data_ptr(), t.data_ptr(), 0) + tuple(t.shape) + tuple(t.stride())


def bound(a, w, K):
    return (K + 2) * 2.0 ** -24 * (a.double().abs() @ w.double().abs().T) + 1e-30


@pytest.mark.parametrize("off", [0, 1])
@pytest.mark.parametrize("M,N,K", [(1, 1, 1), (1, 768, 768), (8, 8, 32), (9, 9, 33), (7, 300, 255), (16, 16, 256), (17, 15, 257), (50, 768, 768),
                                   (33, 31, 130), (300, 768, 768), (511, 97, 499), (511, 768, 8), (320, 513, 20), (200, 2048, 64)])
def test_gemm_entry(M, N, K, off):
    L = fortis_b200.Host().L
    vp, cl = ctypes.c_void_p, ctypes.c_long
    L.fortis_gemm.argtypes, L.fortis_gemm.restype = ([vp, vp] + [cl] * 5) * 3 + [cl] * 3, None
    g = torch.Generator(device="cuda").manual_seed(M + N + K)
    buf = [torch.randn(n * K + off, device="cuda", generator=g) for n in (M, N)]
    a, w = buf[0][off:].view(M, K), buf[1][off:].view(N, K)
    c = torch.full((M + 1, N), 7.0, device="cuda")
    L.fortis_gemm(*memref(a), *memref(w), *memref(c[:M]), M, N, K)
    L.fortis_sync()
    assert bool(((c[:M].double() - a.double() @ w.double().T).abs() <= bound(a, w, K)).all())
    assert bool((c[M] == 7.0).all())
    a.round_(), w.round_()
    torch.cuda.synchronize()                                  # the library runs on a stream of its own
    L.fortis_gemm(*memref(a), *memref(w), *memref(c[:M]), M, N, K)
    L.fortis_sync()
    assert bool((c[:M].double() == a.double() @ w.double().T).all())


@pytest.mark.parametrize("rows", [1, 65, 511])
def test_norms_activation_and_mask(rows):
    dims = [45, 130, 33]
    layers = fortis_b200.mlp_layers(dims, seed=3, act="leaky", slope=1.5, bias="uniform")
    rng = np.random.default_rng(1)
    in_div, out_mul = (rng.uniform(0.5, 2.0, n).astype(np.float32) for n in (dims[0], dims[-1]))
    mask = (np.arange(dims[-1]) % 3 == 0).astype(np.float32)
    h = fortis_b200.Host()
    h.reset()
    h.load_model(fortis_b200.write_blob(layers, in_div=in_div, out_mul=out_mul, relu_mask=mask))
    h.L.fortis_begin(rows)
    x = torch.randn((rows, dims[0]), device="cuda", generator=torch.Generator(device="cuda").manual_seed(rows))
    y = torch.full((rows, dims[-1]), float("nan"), device="cuda")
    h.forward_batched(x, y)
    h.sync()
    v, slack = x.double() / torch.from_numpy(in_div).cuda().double(), 0.0
    for i, l in enumerate(layers):
        W, b = torch.from_numpy(l["W"]).cuda(), torch.from_numpy(l["b"]).cuda().double()
        K = W.shape[1]
        slack = 1.5 * (2 * bound(v, W, K) + (slack @ W.double().abs().T if i else 0.0) + 2.0 ** -22 * b.abs())
        v = v @ W.double().T + b
        if l["act"] == "leaky":
            v = torch.where(v > 0, v, 1.5 * v)
    v, slack = v * torch.from_numpy(out_mul).cuda().double(), slack * 2.0 + 2.0 ** -22 * v.abs()
    m = torch.from_numpy(mask).cuda().bool()
    v = torch.where(m, v.clamp_min(0), v)
    assert bool(((y.double() - v).abs() <= slack).all())
    h.reset()
