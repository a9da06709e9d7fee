"""Which form a 16-bit step of few rows takes, against device times of both forms (B200, us: fused, layer by layer)."""
import ctypes

import pytest

import fortis_b200

MEASURED = [
    ([244, 768, 768, 768, 768, 128], False, 1000, 60.3, 34.1), ([244, 768, 768, 768, 768, 128], False, 3072, 59.0, 42.1),
    ([16, 16, 14], False, 1, 14.7, 9.2), ([16] * 8 + [14], False, 3072, 31.5, 28.9), ([64] * 8 + [38], False, 1000, 32.9, 29.4),
    ([244] + [256] * 4 + [128], False, 1000, 27.3, 25.6), ([244] + [256] * 7 + [128], False, 1000, 35.9, 38.0),
    ([244] + [256] * 7 + [128], False, 3072, 35.0, 37.4), ([244] + [256] * 7 + [128], True, 1000, 42.4, 38.7),
    ([244] + [512] * 7 + [128], False, 3072, 59.3, 56.8), ([244, 256, 512, 256, 512, 256, 512, 256, 128], False, 1000, 45.1, 40.7),
    ([244, 256, 512, 256, 512, 256, 512, 256, 128], False, 3072, 44.1, 50.0), ([244, 512, 256, 512, 256, 512, 256, 512, 128], False, 3072, 46.2, 52.2),
    ([244, 768, 256, 768, 256, 768, 256, 768, 128], False, 128, 61.6, 44.3), ([244] + [768] * 7 + [128], True, 128, 112.3, 51.5),
]


@pytest.mark.parametrize("widths,fp8w,rows,fused,layers", MEASURED)
def test_the_faster_form_runs(widths, fp8w, rows, fused, layers):
    L = fortis_b200.load()
    form = L.fortis_debug_few_rows((ctypes.c_int * len(widths))(*widths), len(widths) - 1, int(fp8w), ctypes.c_long(rows))
    assert (layers if form else fused) <= 1.02 * min(fused, layers)


def test_larger_calls_and_single_layers_run_fused():
    L = fortis_b200.load()
    for widths, rows in (([244, 768, 768, 768, 768, 128], 3073), ([244, 128], 100)):
        assert not L.fortis_debug_few_rows((ctypes.c_int * len(widths))(*widths), len(widths) - 1, 0, ctypes.c_long(rows))
