"""Cells of more LEFs than a genome's longest chromosome has, every epoch against the CPU oracle: move adjustment in more
than one group of 32 units per worker thread (from 16,385 LEFs), rankings at and above 65,535 units, where the merge
that packs ranks into 16 bits gives way to a sort of all units; crowded, so that pushes run across the groups."""

import pytest

from modlefork_gb300 import genome
from test_gpu_parity import compare_cell, small_genome

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nl,length", [(16_384, 250_000_000), (16_385, 30_000_000), (33_000, 60_000_000),
                                       (65_535, 250_000_000), (65_536, 250_000_000), (70_001, 120_000_000)])
def test_cell_of_many_lefs(nl, length):
    cfg = genome.genome_config(num_cells=4, skip_burnin=1, seed=nl)
    chrom, bars = small_genome(cfg, length, 500, seed=nl, occupancy="beta")
    compare_cell(cfg, chrom, bars, nl=nl, target=3 * nl)
