"""Into how many pieces an MLX affine-4 GEMM of up to 64 rows cuts its contraction (spl_debug_q4_plan): host arithmetic, no GPU.

A cut tile's blocks are a cluster and have to find room in one GPC together: a cut that would fit the SMs in one wave of blocks may not fit in clusters."""
import pytest

from splosh_b200.engine import EngineError, debug_q4_plan

B200 = (148, 74, 45, 33, 26, 22, 15, 15)


def test_a_cut_of_one_wave_fits_in_clusters():
    for tiles in range(1, 149):
        for stages in list(range(1, 25)) + [32, 35, 48, 68, 100]:
            pieces = debug_q4_plan(128 * tiles, 256 * stages)
            assert 1 <= pieces <= min(8, stages)
            if pieces > 1:
                assert -(-stages // -(-stages // pieces)) == pieces          # no piece is empty
                if tiles * pieces <= 148:
                    assert tiles <= B200[pieces - 1], (tiles, stages, pieces)


def test_the_cut_of_tensors_in_use():
    """The 27B shape's mixer outputs and MLP, the tiny hybrid's, a drafter's query and key projections, and a tensor whose sevens would not fit."""
    shapes = [(5120, 6144), (5120, 17408), (34816, 5120), (1024, 2816), (1024, 1024), (4096, 5120), (1024, 5120), (2048, 5120), (128, 4096)]
    assert [debug_q4_plan(n, k) for n, k in shapes] == [3, 3, 1, 6, 1, 4, 7, 5, 8]


def test_a_device_without_room_for_large_clusters():
    for n, k in [(128, 4096), (1024, 5120), (1024, 17408)]:
        assert debug_q4_plan(n, k, clusters=(148, 74, 45, 33, 0, 0, 0, 0)) == 4


def test_bad_arguments_are_refused():
    for n, k, sms in ((0, 256, 148), (128, 0, 148), (128, 100, 148), (128, 256, 0)):
        with pytest.raises(EngineError):
            debug_q4_plan(n, k, sms)
