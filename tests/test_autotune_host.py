"""The autotuner's own candidates run on one stream: the times of overlapped ones (a sixth entry) differ from
run to run by more than the candidates do, so a choice between them does not hold."""
from water_flow_simulation_b200 import autotune


def test_default_candidates_run_on_one_stream():
    lists = (autotune.SINGLE_FP32, autotune.SINGLE_FP16, autotune.BATCH_FP16)
    assert all(len(tile) == 5 for tiles in lists for tile in tiles)
    assert all(len(set(tiles)) == len(tiles) >= 5 for tiles in lists)
