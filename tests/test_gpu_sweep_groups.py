"""The fused sweep's launches with both groups of planes full: planes above 110 KB (one CTA
an SM) and below, tensor-core and CUDA-core commutators in each, a grid of 1024+
points below.  Every handle here has enough planes to keep whole-plane kernels alone, and
is too large for one launch of its own, so the fused launches take all of them (the
counts say so: they are counted on the first handle) and results equal stepping alone
bit for bit.
"""
import pytest

from test_gpu_sweep_forms import check, make

pytestmark = pytest.mark.gpu

SHAPES = [  # nb, grid, batch
    (5, (96, 96, 1), 6),   # 147 KB planes, CUDA cores
    (25, (90, 84, 1), 1),  # 121 KB planes, tensor cores (beyond the TMA-fed commutator's 24 bands)
    (14, (24, 24, 1), 1),  # small planes, tensor cores
    (7, (36, 36, 1), 4),   # small planes of 1296 points, CUDA cores
]


@pytest.mark.parametrize("steps", [2, 33])
def test_both_plane_groups(pkg, po, tmp_path, steps):
    pairs = make(pkg, po, tmp_path, SHAPES)
    # four stages of planes, tensor-core and CUDA-core commutators, in two groups
    check(pkg, pairs, steps, [24 * steps, 0, 0, 0], fused=True)
