"""The byte model of the counting sort's kernels (cryo_roofline.py): what each
reads and writes per particle and per cell, the sentinel's cell included."""
import pytest

import cryo_roofline as rf


@pytest.mark.parametrize("kernel,particle,cell", [("k_cell_scan", 0, 16), ("k_cell_scatter", 16, 8),
                                                  ("k_cell_order", 12, 4)])
def test_bytes_of_the_cell_sort(kernel, particle, cell):
    assert rf.per_particle(kernel, {}, False) == (particle, particle)
    assert rf.kernel_bytes(kernel, {}, 1000, 500, False, num_cells=99) == 1500 * particle + 100 * cell
