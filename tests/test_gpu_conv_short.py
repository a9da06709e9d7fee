"""Convolutions of few products per output (the CUDA-core kernel that keeps them in one pass) at the edges of its voxel and
channel groups, against float64.

Tolerance: K fused multiply-adds one after another round K times, each by at most 2^-24 of a partial sum, so an output is
within K * 2^-24 * 1.01 of sum |x||w|, element by element.
"""
import ctypes

import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

import fortis_b200
from tests.test_gpu_f32tc import memref, randn

_keep = []      # weights of the memref entries are constants of the program, told apart by their address


@pytest.fixture()
def host():
    h = fortis_b200.Host()
    h.reset()
    yield h
    h.reset()


# (N, C, F, D, H, W), kernel, stride, padding.  One voxel, a ragged warp, every group of channels (1, 4, 5, 8, 9, 16, 17, 33, 65),
# every number of voxels a thread takes with 4, 8 and 16 channels (one; two from 3552 warps of 32 voxels and one group of channels on; four
# from 7104), one and two with 32
@pytest.mark.parametrize("shape,K,stride,pad", [
    ((1, 1, 1, 1, 1, 1), (1, 1, 1), (1, 1, 1), (0, 0, 0)),
    ((2, 3, 64, 5, 7, 9), (3, 3, 3), (1, 1, 1), (1, 1, 1)),
    ((1, 3, 33, 6, 11, 13), (3, 3, 3), (2, 2, 2), (1, 0, 1)),
    ((1, 1, 17, 9, 8, 7), (5, 5, 5), (1, 2, 1), (2, 2, 2)),
    ((1, 100, 5, 3, 5, 17), (1, 1, 1), (1, 1, 1), (0, 0, 0)),
    ((3, 2, 9, 1, 12, 31), (1, 10, 6), (1, 1, 3), (0, 9, 5)),
    ((1, 1, 65, 4, 4, 4), (2, 3, 4), (1, 1, 1), (1, 2, 3)),
    ((2, 3, 64, 33, 33, 33), (3, 3, 3), (1, 1, 1), (1, 1, 1)),
    ((1, 32, 2, 1, 340, 340), (1, 1, 1), (1, 1, 1), (0, 0, 0)),
    ((1, 4, 8, 1, 500, 500), (1, 3, 3), (1, 1, 1), (0, 1, 1)),
    ((1, 4, 4, 4, 239, 239), (1, 2, 2), (1, 1, 1), (0, 0, 0)),
    ((1, 3, 16, 30, 60, 65), (1, 3, 3), (1, 1, 1), (0, 1, 1)),
    ((1, 4, 4, 4, 241, 241), (1, 2, 2), (1, 1, 1), (0, 0, 0)),
    ((1, 2, 7, 1, 340, 345), (1, 3, 3), (1, 1, 1), (0, 1, 1)),
    ((1, 3, 16, 30, 90, 91), (1, 3, 3), (1, 1, 1), (0, 1, 1)),
])
def test_short_sums(host, shape, K, stride, pad):
    N, C, F, D, H, W = shape
    x, w = randn((N, C, D, H, W), 1), randn((F, C) + K, 2)
    _keep.append(w)
    want = torch.nn.functional.conv3d(x.double(), w.double(), stride=stride, padding=pad)
    bound = torch.nn.functional.conv3d(x.double().abs(), w.double().abs(), stride=stride, padding=pad) * (C * K[0] * K[1] * K[2] * 1.01 * 2.0 ** -24)
    y = torch.full(want.shape, float("nan"), device="cuda")
    torch.cuda.synchronize()                                  # the library runs on a stream of its own
    f = host.L.fortis_conv3d
    f.argtypes, f.restype = ([ctypes.c_void_p] * 2 + [ctypes.c_long] * 11) * 3 + [ctypes.c_long] * 18, None
    f(*memref(x), *memref(w), *memref(y), N, C, D, H, W, F, *K, *want.shape[2:], *stride, *pad)
    host.sync()
    assert bool(((y.double() - want).abs() <= bound).all())
