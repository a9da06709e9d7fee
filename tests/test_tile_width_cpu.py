"""Tile widths of fortis_gemm on the tensor cores, 148 SMs: measured products (B, N, K) and the widths within 3 % of the fastest."""
import pytest

import fortis_b200


# few inputs and one feature more than a tile holds, stored element by element; many inputs; rows that fill tiles of 128; rows off 16 bytes
@pytest.mark.parametrize("B,N,K,widths", [
    (19000, 129, 32, [32]), (19000, 65, 64, [32]), (8192, 257, 32, [32]), (12000, 65, 32, [32]), (40000, 160, 32, [32]), (19000, 96, 32, [32]),
    (8192, 768, 768, [128]), (40000, 256, 512, [128]), (19000, 129, 33, [32]), (40000, 129, 130, [64]),
])
def test_widths(B, N, K, widths):
    assert fortis_b200.load().fortis_debug_tile_width(B, N, K) in widths
