"""Host logic of the tuner: genome handling and configuration validity, no GPU needed."""

import ctypes
import random

import pytest

from tuna_b200 import _lib, make_configs, tuner


def test_genomes_stay_inside_the_search_space():
    rng = random.Random(0)
    for path in ("stream", "tstream", "umma"):
        space = tuner.space_for(path)
        g = tuner.random_genome(rng, path)
        for _ in range(50):
            g = tuner.mutate(rng, tuner.crossover(rng, g, tuner.random_genome(rng, path)), path)
            assert set(g) == set(space)
            assert all(g[k] in space[k] for k in g)


def test_validity_filter_matches_the_launcher(tuna_lib):
    ok = tuner.to_config("stream", 16, dict(rows_per_warp=1, warps_m=16, warps_k=1, k_steps=8))
    assert tuner.is_valid(tuna_lib, 4096, 16, 4096, ok)
    too_many_warps = tuner.to_config("stream", 16, dict(rows_per_warp=1, warps_m=16, warps_k=2, k_steps=8))
    assert not tuner.is_valid(tuna_lib, 4096, 16, 4096, too_many_warps)
    bad_steps = tuner.to_config("stream", 16, dict(rows_per_warp=1, warps_m=16, warps_k=1, k_steps=4))
    assert not tuner.is_valid(tuna_lib, 4096, 16, 4096, bad_steps)
    umma = tuner.to_config("umma", 256, dict(row_blocks=1, stages_w=4, stages_x=4, stages_a=4, dequant_warps=16, k_accs=1))
    assert tuner.is_valid(tuna_lib, 4096, 2048, 4096, umma)
    umma_bad = tuner.to_config("umma", 256, dict(row_blocks=2, stages_w=4, stages_x=4, stages_a=4, dequant_warps=16, k_accs=1))
    assert not tuner.is_valid(tuna_lib, 4096, 2048, 4096, umma_bad)
    # combinations no GPU test exercises are refused by the launcher
    for bad in (dict(dequant_warps=12), dict(k_accs=2), dict(stages_w=2), dict(row_blocks=3)):
        g = dict(row_blocks=1, stages_w=4, stages_x=4, dequant_warps=16, k_accs=1)
        g.update(bad)
        assert not tuner.is_valid(tuna_lib, 4096, 2048, 4096, tuner.to_config("umma", 64, g))


@pytest.mark.parametrize("n,tile_tok,fields,fits", [
    (2048, 0, dict(row_blocks=4), False),      # 4 x 256 accumulator columns
    (100, 0, dict(row_blocks=2), True),
    (1, 0, dict(stages_x=4), False),           # four row blocks of 16 tokens: two accumulators leave three A-slot stages
    (16, 16, dict(row_blocks=1, stages_x=15), True),
    (16, 16, dict(row_blocks=1, stages_x=16), False),
    (256, 256, dict(row_blocks=1, stages_w=4, stages_x=5), True),
    (256, 256, dict(row_blocks=1, stages_w=9, stages_x=5), False),  # shared memory: 32 + 36 + 160 KB
    (128, 128, dict(row_blocks=2, stages_w=6, stages_x=4), True),
    (128, 128, dict(row_blocks=2, stages_w=6, stages_x=5), False),
])
def test_umma_fields_that_do_not_fit_one_sm_are_refused(tuna_lib, n, tile_tok, fields, fits):
    assert tuner.is_valid(tuna_lib, 4096, n, 4096, tuner.to_config("umma", tile_tok, fields)) == fits


@pytest.mark.parametrize("n", [16, 25, 40, 64])
def test_fields_without_a_kernel_mean_the_weight_streaming_one(tuna_lib, n):
    """Up to 64 tokens: its own fields steer it, those of the other kernels do not count."""
    for fields, fits in ((dict(row_blocks=1, k_steps=8), True), (dict(row_blocks=1, k_steps=16), False), (dict(row_blocks=4, tile_tok=32), False),
                         (dict(row_blocks=1, k_accs=2), True), (dict(dequant_warps=4), True), (dict(stages_w=3), True)):
        assert tuner.is_valid(tuna_lib, 4096, n, 4096, _lib.TunaConfig(**fields)) == fits, fields
    assert tuner.is_valid(tuna_lib, 4096, n, 4096, _lib.TunaConfig())


def test_config_fields_round_trip():
    cfg = tuner.to_config("umma", 64, dict(row_blocks=2, stages_w=6, stages_x=4, stages_a=8, dequant_warps=8, k_accs=1))
    d = cfg.as_dict()
    assert d["path"] == _lib.PATH_UMMA and d["tile_tok"] == 64 and d["row_blocks"] == 2 and d["k_accs"] == 1
    assert all(v == (0,) for v in tuner.UMMA_SPACE.values())  # the pair kernel: its own choices only


def test_path_is_part_of_the_search():
    assert tuner.candidate_paths(16) == ("tstream", "stream")
    assert "umma" in tuner.candidate_paths(64) and "tstream" in tuner.candidate_paths(64)
    assert tuner.candidate_paths(2048) == ("tstream", "umma")
    assert tuner.tile_tok_for("tstream", 9) == 16 and tuner.tile_tok_for("tstream", 40) == 64
    assert tuner.tile_tok_for("tstream", 65) == 128 and tuner.tile_tok_for("tstream", 2048) == 128
    assert tuner.tile_tok_for("stream", 8) == 8 and tuner.tile_tok_for("umma", 2048) == 256


def test_the_default_kernel_is_always_among_the_candidates(tuna_lib):
    """What the library chooses by shape can be found by a search, with the tile it chooses itself."""
    names = {v: k for k, v in tuner.PATH_IDS.items()}
    for m, k in ((4096, 4096), (57344, 8192), (512, 512)):
        for n in (1, 9, 16, 17, 24, 25, 32, 33, 64, 65, 256, 300, 2048):
            chosen = _lib.TunaConfig()
            assert tuna_lib.tuna_lookup_config(m, n, k, ctypes.byref(chosen)) == 0
            assert names[chosen.path] in tuner.candidate_paths(n), n
    genome = tuner.random_genome(random.Random(1), "umma")
    assert tuner.to_config("umma", tuner.tile_tok_for("umma", 256), genome).tile_tok == 0


def test_only_a_faster_configuration_becomes_an_entry():
    umma = tuner.random_genome(random.Random(1), "umma")
    results = [(12.0, "tstream", {"row_blocks": 1, "k_steps": 8}), (10.0, "umma", umma)]
    entry = tuner.table_entry(32, results, 11.0)
    assert entry["path"] == "umma" and entry["tile_tok"] == 0 and entry["us"] == 10.0
    make_configs.validate({"4096_32_4096": entry})
    assert tuner.table_entry(32, results, 10.0) is None  # the default is as fast
    assert tuner.table_entry(32, results, 10.05) is None
    assert tuner.table_entry(32, results, None)["path"] == "umma"  # the default could not be timed


def test_token_counts_of_one_bucket_are_measured_apart(tuna_lib, tmp_path):
    class FakeBench:
        def __init__(self, us):
            self.us = us

        def time_us(self, cfg):
            return self.us

    for n, us in ((24, 10.0), (32, 12.0)):
        assert tuner.tune_shape(4096, n, 4096, "umma", 1, 4, 0, tmp_path / "state.json", log=lambda s: None, bench=FakeBench(us))[1] == us


def test_tstream_validity(tuna_lib):
    ok = tuner.to_config("tstream", 16, dict(row_blocks=2, k_steps=8))
    assert tuner.is_valid(tuna_lib, 4096, 16, 4096, ok)
    too_wide = tuner.to_config("tstream", 64, dict(row_blocks=2, k_steps=8))  # 2 x 64 accumulator columns > 64
    assert not tuner.is_valid(tuna_lib, 4096, 64, 4096, too_wide)
    bad_steps = tuner.to_config("tstream", 16, dict(row_blocks=1, k_steps=16))
    assert not tuner.is_valid(tuna_lib, 4096, 16, 4096, bad_steps)
    # 128-token tiles: one row block and 128-column slots only
    assert tuner.is_valid(tuna_lib, 4096, 300, 4096, tuner.to_config("tstream", 128, dict(row_blocks=1, k_steps=4)))
    assert not tuner.is_valid(tuna_lib, 4096, 300, 4096, tuner.to_config("tstream", 128, dict(row_blocks=2, k_steps=4)))
    assert not tuner.is_valid(tuna_lib, 4096, 300, 4096, tuner.to_config("tstream", 128, dict(row_blocks=1, k_steps=8)))
