"""The autotuner can leave every knob as it was given: the choice is never slower than the default."""
import pytest

from gasatt import _lib
from gasatt.tune import DEFAULT_CHUNKS, knob_candidates
from gasatt.workload import config


def test_chunk_by_population_is_a_candidate():
    cfg = config(32, 64, 5e-6, 1e-14, 1.0, precision=_lib.FP32_SPLIT)
    assert cfg.pass_chunk == 0 and 0 in knob_candidates(cfg)["pass_chunk"] and DEFAULT_CHUNKS[0] == 0


@pytest.mark.gpu
def test_a_small_population_keeps_it():
    """4,000 electrons fill three or four blocks with chunks of 1024 and more."""
    from gasatt.sim import births
    from gasatt.tune import tune
    cfg = config(32, 64, 5e-6, 1e-14, 300.0, precision=_lib.FP32_SPLIT, capacity=20000, seed=7)
    parts = births(2000, 8.0, 64 * 5e-6, seed=3, sigma_r=30e-6, Rp=32 * 5e-6)
    best, table = tune(cfg, parts, knobs={"pass_chunk": knob_candidates(cfg)["pass_chunk"]}, steps=400)
    t = table["pass_chunk"]
    assert best.pass_chunk == 0 and t[0] < 0.9 * min(v for k, v in t.items() if k)
