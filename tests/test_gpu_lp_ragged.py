"""The layer kernels of the proposal network's training (csrc/lp_train.cu) where the
rows end inside a warp of the last tile: every layer's count of rows is odd, or
leaves one row, or one short of a warp. Some of a warp's lanes then store and add
between its loads of the accumulators. Checks and tolerances are those of
test_gpu_lp_layers.py.
"""
import pytest

import test_gpu_lp_layers as layers

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mbw,mbh", [(5, 1), (9, 7), (11, 3), (19, 5), (13, 9), (23, 7)])
def test_rows_end_inside_a_warp(gpu, mbw, mbh):
    layers.test_layers_at_tile_edges(gpu, mbw, mbh)
