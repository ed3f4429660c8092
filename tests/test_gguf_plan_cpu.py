"""The launch a GGUF GEMM takes for a step of `rows` rows (spl_debug_gguf_plan): host arithmetic, no GPU.

A weight is formed once a block, so blocks of 128 rows convert half of what blocks of 64 do, but each takes longer (about 1.25 to 1.5 times): they
are right where they save more than that in waves of blocks, and never where they save no wave."""
import os
import re

import pytest

from splosh_b200.engine import EngineError, debug_gguf_plan

KINDS = ["Q4_K", "Q5_K", "Q6_K"]
# (columns, contraction): the 27B shape's mixer inputs (gated-delta, attention), gate|up, out, down and head; the GGUF tests' shape; odd ones.
SHAPES = [(16480, 5120), (14336, 5120), (34816, 5120), (5120, 6144), (5120, 17408), (248320, 5120), (1024, 256), (256, 512), (130, 1024), (2000, 2560)]


def waves(n, rows, block, pieces, sms):
    return -(-(-(-n // 128) * -(-rows // block) * pieces) // sms)


@pytest.mark.parametrize("sms", [148, 132, 20])
@pytest.mark.parametrize("kind", KINDS)
def test_blocks_of_128_rows_only_where_they_save_waves(kind, sms):
    for n, k in SHAPES:
        for rows in list(range(1, 66)) + list(range(65, 600, 7)) + [128, 129, 192, 193, 256, 257, 384, 385, 448, 2048]:
            block, pieces = debug_gguf_plan(kind, n, k, rows, sms)
            assert 1 <= pieces <= k // 256
            if rows <= 64:
                assert block == (16 if rows <= 16 else 32 if rows <= 32 else 64)
                continue
            narrow, wide = waves(n, rows, 64, pieces, sms), waves(n, rows, 128, pieces, sms)
            assert block in (64, 128)
            if wide == narrow:
                assert block == 64, (n, k, rows)
            if 1.6 * wide <= narrow:
                assert block == 128, (n, k, rows)


@pytest.mark.parametrize("kind", KINDS)
def test_the_cut_of_the_27b_tensors(kind):
    """The pieces do not depend on the rows a block holds (outputs stay the same to the bit): a 64-row block's cut."""
    rows = (65, 128, 129, 192, 193, 200, 256, 400)
    assert [debug_gguf_plan(kind, 5120, 6144, r)[1] for r in rows] == [3, 3, 1, 1, 2, 2, 2, 1]
    assert [debug_gguf_plan(kind, 5120, 17408, r) for r in rows] == [(128, 3), (128, 3), (64, 1), (64, 1), (128, 4), (128, 4), (128, 4), (64, 1)]
    assert debug_gguf_plan(kind, 34816, 5120, 200) == (128, 1)
    assert debug_gguf_plan(kind, 34816, 5120, 129) == (64 if kind == "Q6_K" else 128, 1)


def test_bad_arguments_are_refused():
    for n, k, rows, sms in ((0, 256, 1, 148), (128, 0, 1, 148), (128, 100, 1, 148), (128, 256, 0, 148), (128, 256, 1, 0)):
        with pytest.raises(EngineError):
            debug_gguf_plan("Q4_K", n, k, rows, sms)


def skips_a_phase(stages, sets):
    """The weight ring's schedule: dequant set s takes the half-stage units s, s + sets, ... A set that comes to a slot for phase p
    has to have waited for phase p - 1 itself, or never have been due there before: its barrier tells two phases apart, no more."""
    for s in range(sets):
        last = {}
        for unit in range(s, 24 * stages * sets, sets):
            slot, phase = unit // 2 % stages, unit // 2 // stages
            if phase not in (last.get(slot, -1), last.get(slot, -1) + 1):
                return True
            last[slot] = phase
    return False


def test_no_dequant_set_skips_a_phase_of_the_weight_ring():
    path = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "splosh_b200", "csrc", "spl_gemm_gguf.cuh")
    define = dict(re.findall(r"#define (SPL_GG_SETS|SPL_GG_CSTAGES) (\d+)", open(path).read()))
    assert not skips_a_phase(int(define["SPL_GG_CSTAGES"]), int(define["SPL_GG_SETS"]))
    assert skips_a_phase(2, 3) and skips_a_phase(4, 3) and skips_a_phase(5, 3) and not skips_a_phase(6, 3)
