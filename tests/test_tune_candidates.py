"""What the autotuner offers are launches that differ: no value of a knob is clamped
to another one's launch, the library's own choices are among them, and the table
takes each."""
import os
import sys

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
sys.path.insert(0, os.path.join(ROOT, "bc250-vaapi_b200"))
from b200enc import autotune  # noqa: E402


@pytest.mark.parametrize("mbh", [1, 2, 4, 5, 9, 30, 45, 68, 135])
def test_intra_ctas_differ(mbh):
    all_ctas = 2 * -(-mbh // 4)  # the launch's own number and its limit (csrc/intra.cu)
    c = autotune.candidates("intra_ctas", mbh)
    assert len({min(v, all_ctas) for v in c}) == len(c) == 2 and all_ctas in c


def test_library_tile_shapes_are_offered():
    for name in ("deblock_tile_w", "deblock_tile_h"):
        assert {3, 4, 8} <= set(autotune.candidates(name, 68))  # csrc/deblock.cu, by picture size


def test_table_takes_every_candidate():
    import b200enc
    L = b200enc.load_library()
    try:
        for name, key in autotune.KEYS.items():
            for f in (autotune.candidates, autotune.throughput_candidates):
                assert all(L.b200enc_tune_set(key, v) == 0 for v in f(name, 68)), name
    finally:
        for key in autotune.KEYS.values():
            L.b200enc_tune_set(key, 0)
