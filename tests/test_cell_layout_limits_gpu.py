"""What a cell's layout accepts: histories and barrier bits up to a block's whole shared memory (they go to the global
slot where they do not fit beside the ring), budgets down to what these need."""

import pytest

from modlefork_gb300 import engine, genome
from test_gpu_parity import compare_cell, small_genome

pytestmark = pytest.mark.gpu

FIXED = 256 + 8192  # what a budget counts besides history and bits


def _cfg(history):
    return genome.genome_config(num_cells=4, burnin_history_length=history, burnin_smoothing_window_size=5,
                                burnin_target_epochs_for_lef_activation=30, min_burnin_epochs=5, max_burnin_epochs=60,
                                seed=2)


# 16 bytes of history per epoch: 13,900 leave 1 KB of the 227 KB that a block may have, 13,500 fit with the ring's 8 KB
@pytest.mark.parametrize("history", [13_000, 13_500, 13_900])
def test_long_histories(history):
    cfg = _cfg(history)
    chrom, bars = small_genome(cfg, 5_000_000, 20, seed=1, occupancy="beta")
    compare_cell(cfg, chrom, bars, nl=40, target=100)


def test_refusals_stay():
    cfg = _cfg(14_100)
    chrom, bars = small_genome(cfg, 5_000_000, 20, seed=1, occupancy="beta")
    with engine.Engine(cfg, 0) as eng:
        cid = eng.upload_chrom(chrom, bars)
        with pytest.raises(engine.EngineError, match="shared memory"):
            eng.trace_cell(cid, 1, 100, 0, 40, max_epochs=100)
    cfg = _cfg(200)
    with engine.Engine(cfg, 0) as eng:
        cid = eng.upload_chrom(chrom, bars)
        need = FIXED + 16 * 200 + 16
        for budget, ok in ((need, True), (need - 1, False)):
            eng.set_debug_flags(0, budget)
            if ok:
                assert eng.trace_cell(cid, 1, 100, 0, 40, max_epochs=1000)[0].status == 0
            else:
                with pytest.raises(engine.EngineError, match="shared memory"):
                    eng.trace_cell(cid, 1, 100, 0, 40, max_epochs=1000)
