"""Which sequences of a step run by chunks of tokens, and in how wide slices of a head's state: the rules, on the CPU."""
import ctypes

import numpy as np
import pytest
import torch

from prelude_b200.engine.batch import StepBatch
from prelude_b200.ops import kernels as K


def _batch(lens, room=None, **more):
    empty = torch.zeros(0, dtype=torch.int32)
    cu = np.zeros((room or len(lens)) + 1, np.int32)
    cu[1:len(lens) + 1] = np.cumsum(lens)
    return StepBatch(n_tokens=sum(lens), n_seqs=len(lens), token_ids=empty, positions=empty, token_seq=empty, cu_q=torch.from_numpy(cu),
                     q_start=empty, kv_len=empty, state_slots=empty, logit_rows=empty, block_tables={}, status=empty,
                     q_lens=np.asarray(lens, np.int32), **more)


RULES = {"state space": (32, 2, 2, 2), "gated delta rule": (64, 16, 4, 128), "gated linear attention": (256,)}


@pytest.mark.parametrize("kind,lens,want", [
    ("gated delta rule", [500], (1, 0, 0, 1, 0, True)), ("gated delta rule", [1, 15, 15, 15, 700], (1, 0, 0, 5, 0, True)),
    ("gated delta rule", [63], None), ("gated delta rule", [1] * 60 + [8], None), ("gated delta rule", [1] * 60 + [127], None),
    ("gated delta rule", [1] * 60 + [128, 127], (128, 0, 0, 1, 61, True)), ("gated delta rule", [15] * 5 + [128], (128, 0, 0, 1, 5, True)),
    ("gated delta rule", [16] * 5, (1, 0, 0, 5, 0, True)), ("state space", [1] * 60 + [8], (2, 0, 0, 1, 60, True)),
    ("state space", [1, 1, 30], (1, 0, 0, 3, 0, True)), ("state space", [1] * 40, None), ("state space", [2] * 16, (1, 0, 0, 16, 0, True)),
    ("state space", [31], None), ("gated linear attention", [1] * 60 + [196], (1, 0, 0, 61, 0, True)), ("gated linear attention", [255], None)])
def test_sequences_go_by_their_own_length(kind, lens, want):
    """One token each beside a portion: however many tokens the step has, only a sequence that is long itself goes by chunks, where
    chunks do not pay for many short ones."""
    assert K._split(_batch(lens), sum(lens), *RULES[kind]) == want


@pytest.mark.parametrize("kind,tokens,want", [
    ("state space", 32, (2, 2, 2, 18, 32, False)), ("state space", 1024, (2, 2, 2, 256, 256, False)), ("state space", 31, None),
    ("gated delta rule", 64, (16, 4, 128, 8, 64, False)), ("gated delta rule", 1024, (16, 4, 128, 68, 256, False)), ("gated delta rule", 32, None),
    ("gated linear attention", 256, (1, 0, 0, 256, 0, False)), ("gated linear attention", 224, None)])
def test_a_recorded_step_allows_for_every_spread_of_its_tokens(kind, tokens, want):
    """It has room for 256 requests and is replayed with other lengths: neither its rows nor the lengths at hand count."""
    assert K._split(_batch([tokens], room=256, extras={"recorder": object()}), tokens, *RULES[kind]) == want


def test_the_rules_are_those_of_the_kernels():
    assert RULES == {"state space": (K.SCAN_CHUNKED_MIN_TOKENS, *K.SCAN_CHUNKED_LENGTHS), "gated linear attention": (K.GLA_CHUNKED_MIN_TOKENS,),
                     "gated delta rule": (K.DELTA_CHUNKED_MIN_TOKENS, *K.DELTA_CHUNKED_LENGTHS)}


def test_a_decode_step_has_no_chunks():
    assert K._split(_batch([1] * 400, decode_only=True), 400, 1) is None


def _launches(*args):
    from prelude_b200.ops import library
    out = (ctypes.c_int * 16)()
    n = library.library().pb_walk_launches(*args, ctypes.addressof(out))
    return [tuple(out[4 * i:4 * i + 4]) for i in range(n)]


@pytest.mark.parametrize("narrowest,widest", [(16, 64), (16, 32), (32, 32)])
@pytest.mark.parametrize("cols", [16, 32, 48, 64, 96, 128, 192])
@pytest.mark.parametrize("heads", [1, 2, 16, 30, 32, 60, 64, 119, 128, 200])
def test_slices_follow_the_sequences_there_are(heads, cols, narrowest, widest):
    """The widest slices that give four fifths of the multiprocessors a block - of the sequences that walk, not of the rows that a
    recorded step has room for: that one has a launch for every width, and for any number of sequences exactly one of them works, the
    one that a step with this number picks."""
    if cols % narrowest:
        pytest.skip("not taken")
    picked = {}
    for n in range(1, 257):
        (width, rows, lo, hi), = _launches(heads, cols, narrowest, widest, n, 1)
        assert rows == n and cols % width == 0 and narrowest <= width <= widest
        picked[n] = width
        if not torch.cuda.is_available():                   # without a device the rule counts 148 multiprocessors
            full = [w for w in (64, 32, 16) if narrowest <= w <= widest and cols % w == 0 and heads * (cols // w) * n >= 119]
            assert width == (full[0] if full else narrowest)
    for most in (1, 2, 7, 256):
        ranges = _launches(heads, cols, narrowest, widest, most, 0)
        for n in range(1, most + 1):
            (width, rows), = [(w, r) for w, r, lo, hi in ranges if lo <= n <= hi]
            assert width == picked[n] and 1 <= rows <= most
    assert _launches(heads, cols, narrowest, widest, 0, 0) == [] == _launches(heads, cols, narrowest, widest, 0, 1)
