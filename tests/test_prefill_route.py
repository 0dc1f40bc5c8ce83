"""Which kernel takes a step's prompt portions (csrc/prefill_attn.cu): host arithmetic, no GPU.  0: 16-token tiles, 1: tensor memory,
2: both."""
import ctypes as C
import os
import subprocess
import sys

import pytest

from llmq_b200 import lib

HEADS = {64: (32, 8), 128: (32, 8), 256: (16, 8)}
ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def route(D, portions=None, n_seqs=0, n_tiles=None, columns=512, window=0, heads=None):
    n_q, n_kv = heads or HEADS[D]
    if portions is None:
        return lib.load().b200q_prefill_attn_route(None, 0, n_seqs, n_tiles, columns, n_q, n_kv, D, window)
    flat = [x for i, (past, n) in enumerate(portions) for x in (0, n, past, i)]
    return lib.load().b200q_prefill_attn_route((C.c_int32 * len(flat))(*flat), len(portions), n_seqs, sum((n + 15) // 16 for _, n in portions),
                                               columns, n_q, n_kv, D, window)


SHORT = [(0, 8 + 7 * i % 33) for i in range(200)]


@pytest.mark.parametrize("columns", [8, 40, 512])
def test_known_portions_decide_alone(columns):
    """a longer sequence of the same step (a wider table) changes nothing for the portions"""
    for D in (64, 128, 256):
        for portions in (SHORT, [(0, 16)] * 32, [(42, 10 + i % 22) for i in range(27)], [(0, 64)], [(0, 5)]):
            assert route(D, portions, columns=columns) == 0, (D, portions[:2])
        for portions in ([(0, 2000)], [(0, 1000)] * 8, [(0, 4400)], [(0, 2000)] + [(0, 20)] * 20, [(0, 600)] * 4):
            assert route(D, portions, columns=columns) == 1, (D, portions[:2])
    for portions in ([(0, 128)] * 36, [(0, 128)] * 16, [(0, 200)] * 20, [(0, 300)] * 14, [(1500, 40)]):
        assert route(128, portions, columns=columns) == 1


def test_tiles_alone():
    for D in (64, 128, 256):
        assert route(D, n_tiles=400, columns=8) == 0                      # no room for long ones
        assert route(D, n_tiles=400, columns=512) == 2                    # 400 of 16 tokens, or one of 6400
        assert route(D, n_seqs=3, n_tiles=240, columns=128) == 1          # at least 1280 tokens each on average
        assert route(D, n_seqs=200, n_tiles=300, columns=4) == 0
        assert route(D, n_seqs=500, n_tiles=300, columns=512) == 2
        assert route(D, n_seqs=1, n_tiles=3, columns=96) == 1             # 40 tokens behind 1500
    assert route(64, n_seqs=1, n_tiles=3, columns=32) == 0                # ... behind 400
    assert route(128, n_seqs=36, n_tiles=288, columns=8) == 1             # 36 prompts of 128 tokens
    assert route(128, n_seqs=0, n_tiles=0) == 0


def test_a_window_bounds_the_work():
    assert route(256, [(0, 3000)], window=256) == 1 and route(256, [(3000, 16)] * 4, window=64) == 0


def test_batch_invariant_runs_take_one_kernel():
    code = ("import sys; sys.path.insert(0, %r); from tests.test_prefill_route import route; "
            "assert route(128, [(0, 2000)]) == 0 and route(256, n_tiles=400) == 0" % ROOT)
    subprocess.run([sys.executable, "-c", code], env=dict(os.environ, B200Q_BATCH_INVARIANT="1"), cwd=ROOT, check=True, timeout=120)
