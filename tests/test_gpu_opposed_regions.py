"""Regions of suspected cells, at the sizes where their linking changes over.

Cells are linked in 2x2 blocks first and then block to block with as few links
as the neighbours allow; a thread dilates 4 x 4 cells, a block of threads 512 x
4, and lists of cells, tiles and sites are filled a block at a time. The masks
run from single sites to just joined labyrinths and full areas. Region labels,
counts and statistics equal the oracle's, samples agree to the bound of the
existing comparison (1e-4).
"""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("density", [0.001, 0.02, 0.08, 0.3])
@pytest.mark.parametrize("size", [(9, 7), (64, 50), (1023, 37), (1026, 34), (1032, 131)])
def test_masks(stages, oracle, size, density):
    w, h = size
    rng = np.random.default_rng(w + int(1000 * density))
    m = rng.uniform(0.05, 0.9, (h, w)).astype(np.float32)
    m[rng.random((h, w)) < density / 4] = 1.1
    m[h // 2, w // 2] = 1.2
    det = (0.987,) * 3
    ours, stats, labels, count = stages.opposed(m, "GBRG", det, None)
    ref, ref_stats, ref_labels, ref_count = oracle.opposed(m, 3, det, None)
    assert count == ref_count and np.array_equal(labels, ref_labels)
    assert stats.tolist() == ref_stats.tolist()
    assert float(np.max(np.abs(ours - ref))) <= 1e-4


def test_long_regions(stages, oracle):
    # Rows, columns and a comb: links in a chain as long as the image.
    m = np.random.default_rng(1).uniform(0.1, 0.8, (700, 600)).astype(np.float32)
    m[10:690, 40:60] = 1.1
    m[30:34, 80:590] = 1.2
    m[100:600:24, 100:560] = 1.3
    m[100:600, 556:560] = 1.3
    det = (0.987,) * 3
    ours, stats, labels, count = stages.opposed(m, "RGGB", det, None)
    ref, ref_stats, ref_labels, ref_count = oracle.opposed(m, 0, det, None)
    assert count == ref_count and np.array_equal(labels, ref_labels)
    assert stats.tolist() == ref_stats.tolist()
    assert float(np.max(np.abs(ours - ref))) <= 1e-4
